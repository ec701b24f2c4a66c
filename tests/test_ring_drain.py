"""After a wait that ran out, a kernel waits for the copies that it still has in flight: the rule (``csrc/drain.h``) against a model
of the barriers, compiled for the host."""

import os
import re
import subprocess

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "dryft_b200", "csrc")

MODEL = r"""
#include "drain.h"
#include <cstdio>
#include <random>
#include <vector>
int main() {
  std::mt19937 rng(5);
  for (int trial = 0; trial < 20000; ++trial) {
    const int stages = 1 + rng() % 5, issued = rng() % 40, used = issued > 0 ? issued - (int)(rng() % (stages + 1)) : 0;
    // copies before `used` have landed (their stages were filled again, or could be); the rest land in any order, slowly
    std::vector<int> ended(stages, 0);                 // phases that a stage's barrier has completed
    std::vector<int> flying;
    for (int i = 0; i < issued; ++i)
      if (i < used || i < issued - stages) ended[i % stages] = i / stages + 1; else flying.push_back(i);
    int polls = 0;
    const bool stuck = trial % 7 == 0 && !flying.empty();      // nothing lands any more
    auto landed = [&](int s, unsigned parity) {
      ++polls;
      if (!stuck && !flying.empty() && rng() % 3 == 0) {
        const size_t k = rng() % flying.size();
        ended[flying[k] % stages] = flying[k] / stages + 1;
        flying.erase(flying.begin() + k);
      }
      return (unsigned)((ended[s] - 1) & 1) == parity;   // what the hardware answers: the phase before the current one has this parity
    };
    const bool done = ring_drain(issued, stages, landed, [&] { return polls > 5000; });
    if (done != !stuck || (done && !flying.empty())) { printf("trial %d: done %d, %zu copies in flight\n", trial, done, flying.size()); return 1; }
  }
  return 0;
}
"""


def test_every_copy_has_landed_when_the_wait_ends(tmp_path):
    src, exe = tmp_path / "model.cc", tmp_path / "model"
    src.write_text(MODEL)
    subprocess.run(["g++", "-std=c++17", "-O1", "-I", CSRC, str(src), "-o", str(exe)], check=True)
    out = subprocess.run([str(exe)], capture_output=True, text=True, timeout=60)
    assert out.returncode == 0, out.stdout


@pytest.mark.parametrize("name", sorted(f for f in os.listdir(CSRC) if f.endswith((".cu", ".cuh", ".h"))))
def test_no_wait_asks_for_either_parity(name):
    """A barrier always answers yes to one of the two parities: asking for both waits for nothing."""
    text = open(os.path.join(CSRC, name)).read()
    assert not re.search(r"try_wait\(([^;]*?), 0\) && !mbar_try_wait\(\1, 1\)", text)
