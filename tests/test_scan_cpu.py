"""CPU: what the host can check of the recurrences' kernels: the order of the walk's copies when a wait runs out, the space that a portion asks for, and what it
does with less."""
import ctypes as C
import os
import subprocess
import types

import pytest
import torch

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

SCHEDULE = r"""
#include <cstdio>
#include <cstdlib>
#include <vector>
#include "seq_walk_schedule.h"
#define REQUIRE(x) do { if (!(x)) { std::printf("line %d: %s (chunks %d, fails %d)\n", __LINE__, #x, chunks, fails); return 1; } } while (0)
constexpr int STAGES = 4;
// One CTA's operand warp: barriers of one arrival a phase, named barriers by their arrivals, the copy of chunk `fails` and of those after it never complete.
static int run(int chunks, int fails) {
  std::vector<int> phase(STAGES, 0), open(STAGES, -1), arrived(STAGES, 0), met(STAGES, 0), drained;      // completed phases, copy in flight, EMPTY's two sides
  int handed = 0;
  bool dead = false;
  b2l::walk_operands<STAGES>(
      chunks,
      [&](int n) {
        if (dead) std::printf("copy of chunk %d after a wait ran out\n", n), std::exit(1);
        if (open[n % STAGES] >= 0 || phase[n % STAGES] != n / STAGES) std::printf("copy of chunk %d into a stage in use\n", n), std::exit(1);
        open[n % STAGES] = n;
      },
      [&](int n) {
        if (dead) return false;
        if (open[n % STAGES] != n || n >= fails) dead = true;
        else open[n % STAGES] = -1, ++phase[n % STAGES];
        return !dead;
      },
      [&](int n) {
        if (n != handed++) std::exit(2);
        ++arrived[n % STAGES];      // the walk takes the chunk and its outputs are read out: they arrive without a wait on this warp
      },
      [&](int n) { ++met[n % STAGES]; }, [&](int n) { drained.push_back(n); });
  REQUIRE(handed == chunks);
  for (int s = 0; s < STAGES; ++s) REQUIRE(met[s] == (arrived[s] > 0 ? arrived[s] - 1 : 0));      // all but a stage's last arrivals are met
  std::vector<int> in_flight;
  for (int n = 0; n < chunks; ++n)
    if (open[n % STAGES] == n) in_flight.push_back(n);
  for (int n : in_flight) {
    bool found = false;
    for (int d : drained) found |= d == n;
    REQUIRE(found);
  }
  REQUIRE(fails < chunks || drained.empty());
  for (int d : drained) REQUIRE(open[d % STAGES] == d || phase[d % STAGES] > d / STAGES);          // never a copy that was not started
  return 0;
}
int main() {
  for (int chunks = 1; chunks <= 19; ++chunks)
    for (int fails = 0; fails <= chunks; ++fails)
      if (run(chunks, fails)) return 1;
  for (int redo = 0; redo < 2; ++redo)
    for (int gone = 0; gone < 2; ++gone)
      if (b2l::walk_state_to_scratch(redo, gone) != (redo == 1 && gone == 0)) return 1;
  return 0;
}
"""


def test_walk_starts_no_copy_after_a_wait_that_ran_out(tmp_path):
    """The operand warp's own loop against barriers of the host: after the first wait that runs out no copy starts (its stage may hold one, its barrier an
    incomplete phase), every named barrier is still met, and each copy in flight is waited for; lost operands never leave the state as it was."""
    src, exe = tmp_path / "schedule.cpp", tmp_path / "schedule"
    src.write_text(SCHEDULE)
    subprocess.run(["g++", "-std=c++17", "-O1", "-I", os.path.join(ROOT, "lit-llama_b200", "csrc"), str(src), "-o", str(exe)], check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout


def _space(T, heads, qk_heads, K, V, per_channel, delta, vscale=0):
    from lit_llama_b200 import _seqlib as S

    n_chunks, least = C.c_int(0), C.c_longlong(-1)
    n = S.lib().b2l_seq_scan_space(T, heads, qk_heads, K, V, per_channel, delta, 0, vscale, C.byref(n_chunks), C.byref(least))
    return n, least.value, n_chunks.value


def test_scan_space_is_what_the_form_writes():
    """Floats: 2 matrices of 16 x 16 a chunk and head for the form in f32; for the tensor cores a chunk's operands, 6 (12 with the delta rule: W and Q) 16-bit words a
    key channel and token for W | Q and 6 for the decayed keys, the decays, and 384 words for every 16 value columns (400 with one decay per head)."""
    from lit_llama_b200 import _seqlib as S

    def ops(K, delta):
        return 16 * K * 3 // 2 * (2 if delta else 1) + 16 * K * 3 // 2 + K

    assert _space(2048, 16, 16, 64, 128, 1, 1) == (128 * 16 * 512, 0, 1)                                  # the delta rule with 64 keys stays in f32
    assert _space(300, 16, 16, 128, 256, 1, 1) == (19 * 16 * 512, 0, 1)                                   # more value columns than the tensor cores' form takes
    assert _space(2048, 16, 16, 128, 128, 1, 1) == (128 * 16 * (ops(128, 1) + 8 * 384), 128 * 16 * 512, 1)
    assert _space(512, 32, 1, 128, 64, 0, 0, 1) == (32 * (ops(128, 0) + 32 * 4 * 400), 32 * 32 * 512, 1)      # operands of q and k once for all heads
    assert _space(4096, 160, 160, 128, 16, 1, 1)[0] == 12 * 160 * (ops(128, 1) + 384)                     # twelve chunks of 160 heads a segment
    assert _space(2048, 4, 4, 128, 128, 1, 0) == (16 * 4 * 128 * 128, 0, 16) and _space(31, 4, 4, 128, 128, 1, 1) == (0, 0, 1)
    for T in (33, 64, 79, 512, 2047, 40000):
        for H in (1, 4, 18, 65, 160, 256):
            for K, V, per_channel, delta in ((64, 16, 1, 0), (128, 128, 1, 1), (128, 48, 0, 0), (128, 64, 1, 0), (64, 64, 1, 1)):
                n, least, n_chunks = _space(T, H, H, K, V, per_channel, delta)
                assert n_chunks > 1 or (least < max(n, 1) and n <= S.lib().b2l_seq_scan_work_floats(T, H))


def test_scan_space_for_the_most_serves_all():
    from lit_llama_b200 import _seqlib as S

    f = S.lib().b2l_seq_scan_work_floats
    for T in (31, 32, 63, 64, 500, 2048, 30000):
        n = [f(T, H) for H in range(1, 257)]
        assert n == sorted(n)
    for H in (1, 7, 65, 100, 256):
        n = [f(T, H) for T in range(16, 6000, 5)]
        assert n == sorted(n)


def test_scan_within_refuses_what_the_scan_refuses():
    from lit_llama_b200 import _seqlib as S

    lib, said = S.lib(), lambda: S.lib().b2l_seq_last_error()
    assert lib.b2l_seq_scan_within(None, 10, None) == -1 and b"null argument block" in said()
    a = S.ScanArgs(T=512, heads=2, qk_heads=2, K=64, V=64, n_chunks=4)
    assert lib.b2l_seq_scan_within(C.byref(a), 4 * 2 * 64 * 64 - 1, None) == -1 and b"end states" in said()
    assert lib.b2l_seq_scan_within(C.byref(a), 4 * 2 * 64 * 64, None) == -1 and b"null pointer" in said()
    a = S.ScanArgs(T=0, heads=2, qk_heads=2, K=64, V=64, n_chunks=1, q=64, k=64, v=64, decay=64, state=64, meta=64, out=64)
    assert lib.b2l_seq_scan_within(C.byref(a), 0, None) == 0 and lib.b2l_seq_scan(C.byref(a), None) == 0       # no tokens: no launch


@pytest.mark.parametrize("delta,T,H,memory,want", [(1, 2048, 16, "all", "fast"), (1, 2048, 16, "little", "least"), (1, 2048, 16, "none", "none"), (1, 70, 2, "little", "fast"),
                                                   (0, 2048, 4, "none", "raises")])
def test_scan_without_memory_takes_the_form_that_fits(monkeypatch, delta, T, H, memory, want):
    """No room for the tensor cores' operands: the walk in f32 has what it needs; without that, token by token.  A portion that was to run in chunks says so."""
    from lit_llama_b200 import _seqlib as S, mixers as X

    K = V = 128
    fast, least, _ = _space(T, H, H, K, V, 1, delta)
    limit = {"all": fast, "little": max(least, H * 3000), "none": 100}[memory]
    real, asked, calls = torch.empty, [], []

    def empty(shape, **kw):
        n = 1
        for d in shape:
            n *= d
        asked.append(n)
        if n > limit:
            raise torch.OutOfMemoryError("no memory (the test's)")
        return real((n,), dtype=kw["dtype"], device="meta")

    monkeypatch.setattr(X, "_p", lambda t, offset=0: None if t is None else 64)
    monkeypatch.setattr(X.torch, "empty", empty)
    lib = types.SimpleNamespace(b2l_seq_scan_space=S.lib().b2l_seq_scan_space, b2l_seq_scan_within=lambda a, floats, stream: calls.append((a._obj.work_state, a._obj.n_chunks, floats)) or 0)
    monkeypatch.setattr(S, "lib", lambda: lib)
    ctx = types.SimpleNamespace(T=T, meta=None, act=0, stream=None)

    def scan():
        X._scan(ctx, q=64, ldq=H * K, k=64, ldk=H * K, v=64, ldv=H * V, q_mult=1.0, decay=64, ldd=H * K, per_channel=True, state=types.SimpleNamespace(device="meta"), out=64,
                ldo=H * V, heads=H, qk_heads=H, K=K, V=V, beta=64 if delta else None, ldb=H)

    if want == "raises":
        with pytest.raises(torch.OutOfMemoryError):
            scan()
        assert not calls
        return
    scan()
    floats = {"fast": fast, "least": least, "none": 0}[want]
    assert calls == [(64 if floats else None, 1, floats)] and asked[0] == fast and asked[-1] == (floats or least)


def test_slots_are_zeroed_on_the_pools_device(monkeypatch):
    """The zeroing is a kernel: a pool in host memory is refused before it starts and loses no slot, one on another device than the current one is zeroed there."""
    from lit_llama_b200 import _seqlib as S, state as P

    pool = P.SequenceStatePool({"S": P.StateSpec((4, 8), torch.float32)}, 3, torch.device("cpu"))
    monkeypatch.setattr(S, "lib", lambda: pytest.fail("no launch"))
    with pytest.raises(RuntimeError, match="tensor on cpu"):
        pool.acquire("r")
    assert pool.free_slots() == 3 and not pool.has("r")
    current, calls = [0], []

    class Device:
        def __init__(self, device):
            self.device = device

        def __enter__(self):
            self.before, current[0] = current[0], self.device.index

        def __exit__(self, *exc):
            current[0] = self.before

    monkeypatch.setattr(P.torch.cuda, "device", Device)
    monkeypatch.setattr(P.torch._C, "_cuda_getDevice", lambda: current[0], raising=False)
    monkeypatch.setattr(S, "stream_ptr", lambda: 100 + current[0])
    monkeypatch.setattr(S, "lib", lambda: types.SimpleNamespace(
        b2l_seq_zero_slots=lambda p, n, k, slot, stream: calls.append((current[0], list(p), list(n), k, slot, stream)) or 0))
    for index in (1, 0):
        pool.tensors = {"S": types.SimpleNamespace(is_cuda=True, device=torch.device("cuda", index), nbytes=3 * 128, data_ptr=lambda: 4096)}
        slot = pool.acquire(index)
        assert calls.pop() == (index, [4096], [128], 1, slot, 100 + index) and current[0] == 0
