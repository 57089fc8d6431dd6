"""What a kernel that gives up waits for, against a model of the barriers' phases, on the CPU."""
import os
import subprocess

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

PROGRAM = r"""
#include <cstdio>
#include <vector>
#include "ring_drain.cuh"
// a barrier's completed phases; a wait for a parity passes unless the phase at work has it
struct Bar { int done = 0; bool passes(unsigned parity) const { return (done & 1) != (int)parity; } };
// one place, `steps` fills of it, the copy of step `slow` (if any) landing only behind the end: whether an
// arrival met an open phase (the barrier takes one a phase) or the end did not wait for that copy
static bool one_place(int steps, int slow, bool heeds) {
  OnePlace copies; Bar bar;
  int flying = 0, bad = 0; bool gave_up = false;
  for (int i = 0; i < steps; ++i) {
    copies.fill(heeds && gave_up, [&] { bad += flying; ++flying; });
    if (flying && i != slow && !gave_up) { --flying; ++bar.done; }
    if (!bar.passes(i & 1)) gave_up = true;                          // the wait runs out
  }
  copies.drain([&](int s, unsigned parity) {
    bad += s != 0 || bar.passes(parity) == (flying > 0);
    if (flying) { --flying; ++bar.done; }
    bad += !bar.passes(parity);
  });
  return bad || flying;
}
int main() {
  int cases = 0;
  for (int steps = 0; steps < 9; ++steps)
    for (int slow = 0; slow <= steps; ++slow) {
      if (one_place(steps, slow, true)) { std::printf("one place %d %d\\n", steps, slow); return 1; }
      if (one_place(steps, slow, false) != (slow + 1 < steps)) return 1;       // (the model sees it)
    }
  for (int stages = 1; stages <= 8; ++stages)
    for (int fills = 0; fills <= 3 * stages + 1; ++fills)
      for (unsigned flying = 0; flying < 1u << (fills < stages ? fills : stages); ++flying) {
        std::vector<Bar> bars(stages);
        std::vector<bool> in_flight(stages, false);
        int stage = 0; unsigned phase = 0;              // as the kernels' copying threads count
        for (int n = 0; n < fills; ++n) {
          // (a stage is filled again once its fill before is complete; of the last ones some are not)
          const int back = fills - 1 - n;
          if (back < stages && flying >> back & 1) in_flight[stage] = true;
          else ++bars[stage].done;
          if (++stage == stages) { stage = 0; phase ^= 1; }
        }
        int asked = 0; bool right = true;
        ring_drain(stages, stage, phase, [&](int s, unsigned parity) {
          ++asked;
          right &= bars[s].passes(parity) == !in_flight[s];          // waits for it, and for nothing else
          right &= bars[s].passes(0) || bars[s].passes(1);           // (either: always passed)
          ++bars[s].done;
          right &= !in_flight[s] || bars[s].passes(parity);          // and ends when it lands
        });
        if (asked != stages || !right) { std::printf("%d %d %u\n", stages, fills, flying); return 1; }
        ++cases;
      }
  std::printf("%d\n", cases);
}
"""


def test_the_last_fill_of_every_stage_and_no_other(tmp_path):
    src, exe = tmp_path / "drain.cpp", tmp_path / "drain"
    src.write_text(PROGRAM)
    subprocess.run(["g++", "-std=c++17", "-O1", "-I", os.path.join(ROOT, "binfer_b200", "csrc"), str(src),
                    "-o", str(exe)], check=True)
    out = subprocess.run([str(exe)], capture_output=True, text=True)
    assert out.returncode == 0 and int(out.stdout) > 1000, out.stdout
