"""Which copies of a shared-memory ring may still be in flight (csrc/lla_ring.h), against a
ring that is played step by step and abandoned at every point."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

HARNESS = r"""
#include <cstdio>
#include <random>
#include <vector>
#include "lla_ring.h"
int main() {
    std::mt19937 g(3);
    long bad = 0;
    for (uint32_t S = 1; S <= 9; ++S)
        for (int trial = 0; trial < 4000; ++trial) {
            std::vector<long> done(S, 0);          // completed phases of a stage's barrier
            uint64_t issued = 0, read = 0;         // copies; stages handed back by the reader
            std::vector<uint64_t> flight;          // copies that have not landed
            for (int step = (int)(g() % 60); step > 0; --step) {
                const unsigned what = g() % 3;
                if (what == 0 && issued < read + S) flight.push_back(issued++);
                if (what == 1 && !flight.empty()) {  // any copy may land first
                    const size_t k = g() % flight.size();
                    ++done[flight[k] % S];
                    flight.erase(flight.begin() + k);
                }
                if (what == 2 && read < issued && done[read % S] > (long)(read / S)) ++read;
            }
            // given up here: the stages and parities to wait for are those of the copies in flight
            std::vector<bool> waits(S, false);
            for (uint32_t s = 0; s < S; ++s) {
                uint32_t parity = 7;
                const bool had = lla::ring_last_phase(issued, S, s, parity);
                if (had != (issued > s)) ++bad;
                // a wait on a parity ends once the phase of the other parity is the current one
                if (had) waits[s] = (uint32_t)(done[s] & 1) == parity;
                if (!had && done[s]) ++bad;
            }
            std::vector<bool> want(S, false);
            for (uint64_t f : flight) want[f % S] = true;
            if (want != waits) ++bad;
        }
    std::printf("%ld\n", bad);
    return bad != 0;
}
"""


@pytest.mark.skipif(not shutil.which("g++"), reason="needs a host compiler")
def test_ring_last_phase(tmp_path):
    src = tmp_path / "ring.cpp"
    src.write_text(HARNESS)
    exe = str(tmp_path / "ring")
    subprocess.run(["g++", "-O1", "-std=c++17", "-I", os.path.join(ROOT, "linfa-linalg_gb300", "csrc"), str(src), "-o", exe],
                   check=True)
    r = subprocess.run([exe], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout
