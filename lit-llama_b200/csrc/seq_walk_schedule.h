// The order in which the tensor-core walk (seq_scan_mma.cuh) takes its operands, apart from the waits and copies themselves, so that a program on the host can run
// it with others in their place.
#pragma once
#ifdef __CUDACC__
#define B2L_WALK_FN __host__ __device__ __forceinline__
#else
#define B2L_WALK_FN inline
#endif

namespace b2l {

// Chunk n goes through stage n % STAGES, its copy STAGES - 1 chunks ahead of the one that is handed over:
//   copy(n)    starts the copy of chunk n
//   wait(n)    waits for it; false once a wait has run out, then and ever after
//   hand(n)    named barrier: the walk may read chunk n
//   freed(n)   named barrier: the outputs of the chunk that was in n's stage before are read out
//   drain(n)   waits for a copy whose wait ran out, with a limit of its own
// After a wait that ran out no copy starts: its stage may have one in flight, and its barrier a phase that is incomplete.  The named barriers have no limit,
// so they are met for every chunk all the same; what is handed over then is lost, and the kernel's end says so.
template <int STAGES, class Copy, class Wait, class Hand, class Freed, class Drain>
B2L_WALK_FN void walk_operands(int n_chunks, Copy copy, Wait wait, Hand hand, Freed freed, Drain drain) {
  int ahead = 0, copied = 0;
  for (; ahead < STAGES - 1 && ahead < n_chunks; ++ahead) copy(ahead);
  copied = ahead;
  bool ok = true;
  for (int n = 0; n < n_chunks; ++n) {
    ok = wait(n);
    hand(n);
    if (ahead < n_chunks) {
      if (ahead >= STAGES) freed(ahead);
      if (ok) {
        copy(ahead);
        copied = ahead + 1;
      }
      ++ahead;
    }
  }
  if (!ok)
    for (int n = copied > STAGES ? copied - STAGES : 0; n < copied; ++n) drain(n);      // no copy outlives the CTA
}

// Where the walk leaves its state: in scratch memory for the form that takes columns with infinities or NaN again, unless operands were lost, which takes nothing
// again: the state itself then becomes NaN.
B2L_WALK_FN bool walk_state_to_scratch(bool redo, bool gone) { return redo && !gone; }

}  // namespace b2l
