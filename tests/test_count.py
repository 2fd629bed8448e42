"""The meeting count of tf_solve_bsr_static's thread blocks across its 32-bit wrap."""
import os
import subprocess

from tissuefolding_paperversion_gb300 import build

PROBE = r"""
#include <cstdio>
#include <initializer_list>
#include "tf_count.h"
// grid blocks arrive one by one at meetings whose goals pass 2^32: a block may
// leave a meeting only once all have arrived
int main() {
    int wrong = 0;
    for (unsigned grid : {1u, 2u, 33u, 152u, 512u})
        for (unsigned start : {0u, 0xffffffffu, 0xffffffffu - 3 * grid, 0x7fffffffu, 0x80000000u - grid}) {
            unsigned seen = start, goal = start;
            for (int meeting = 0; meeting < 8; ++meeting) {
                goal += grid;
                for (unsigned k = 0; k < grid; ++k) {
                    wrong += tf::count_reached(seen, goal);
                    ++seen;
                }
                wrong += !tf::count_reached(seen, goal);
                wrong += !tf::count_reached(seen + grid - 1, goal);  // others already at the next one
            }
        }
    std::printf("%d\n", wrong);
}
"""


def test_meeting_count_across_its_wrap(tmp_path):
    src, exe = tmp_path / "probe.cpp", tmp_path / "probe"
    src.write_text(PROBE)
    subprocess.run(["g++", "-std=c++17", "-I", build.CSRC, str(src), "-o", str(exe)], check=True)
    assert subprocess.run([str(exe)], capture_output=True, text=True, check=True).stdout == "0\n"
