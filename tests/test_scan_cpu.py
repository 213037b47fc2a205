"""CPU: what the host can check of the recurrences' kernels: the order of the walk's copies when a wait runs out."""
import os
import subprocess

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
