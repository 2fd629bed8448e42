"""Which FP64 matrices the Krylov products read past L2."""
import subprocess

import pytest

from tissuefolding_paperversion_gb300 import build

PROBE = r"""
#include <cstdio>
#include <cstdlib>
#include "tf_stream.h"
int main(int, char** a) { std::printf("%d\n", tf::stream_matrix(std::atoll(a[1]), std::atoi(a[2]), std::atoll(a[3]))); }
"""
NODE_BYTES = 1377  # of the matrix, on the layered sheets
L2 = 129 << 20


@pytest.fixture(scope="module")
def rule(tmp_path_factory):
    d = tmp_path_factory.mktemp("stream")
    src, exe = d / "probe.cpp", d / "probe"
    src.write_text(PROBE)
    subprocess.run(["g++", "-std=c++17", "-I", build.CSRC, str(src), "-o", str(exe)], check=True)

    def ask(nbytes, multigrid, l2=L2):
        out = subprocess.run([str(exe), str(nbytes), str(int(multigrid)), str(l2)], capture_output=True, text=True)
        return out.stdout == "1\n"
    return ask


@pytest.mark.parametrize("multigrid,kept,streamed", [(False, 61605, 92480), (True, 28880, 36980)])
def test_matrices_that_an_iteration_finds_in_l2_are_kept_there(rule, multigrid, kept, streamed):
    """The sizes between which the measured times cross."""
    assert not rule(kept * NODE_BYTES, multigrid) and rule(streamed * NODE_BYTES, multigrid)
    assert not rule(147 * NODE_BYTES, multigrid) and not rule(0, multigrid)


def test_the_rule_at_its_line_and_at_the_largest_matrix(rule):
    assert not rule(2 << 20, False, 3 << 20) and rule((2 << 20) + 1, False, 3 << 20)
    assert not rule(1 << 20, True, 3 << 20) and rule((1 << 20) + 1, True, 3 << 20)
    assert rule(9 << 31, True) and rule(9 << 31, False)  # past 32 bits
