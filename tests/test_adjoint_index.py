"""The adjoint-source kernel's (receiver, shot) index on the host: the last
pairs of a call and the first item beyond it, at sizes around 2^31 and 2^32
pairs, where a 32-bit product of the two counts wraps and every thread would
drop out."""
import os
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CUDA_INC = "/usr/local/cuda/include"

MAIN = r"""
#include <cstdio>
#include <cstdlib>
#include "adjoint_index.hpp"
int main(int, char **v) {
    const int ns = std::atoi(v[1]), ntr = std::atoi(v[2]);
    const size_t last = (size_t)ns * ntr - 1;
    for (size_t t : {(size_t)0, (size_t)ns, last, last + 1}) {
        const gm::AdjointItem a = gm::adjoint_item(t, ns, ntr);
        std::printf("%d %d %d\n", a.receiver, a.shot, (int)a.in);
    }
}
"""


@pytest.fixture(scope="module")
def program(tmp_path_factory):
    d = tmp_path_factory.mktemp("adjoint")
    (d / "main.cpp").write_text(MAIN)
    exe = str(d / "main")
    subprocess.run(["g++", "-std=c++17", "-I", CUDA_INC, "-I", os.path.join(ROOT, "germaine_b200", "csrc"),
                    str(d / "main.cpp"), "-o", exe], check=True)
    return exe


@pytest.mark.parametrize("ns,ntr", [(1, 1), (1, 7), (100, 801), (2048, (1 << 20) - 1), (2048, 1 << 20),
                                    (2049, (1 << 20) + 3), (65537, 65539)])
def test_pairs_beyond_32_bits(program, ns, ntr):
    out = subprocess.run([program, str(ns), str(ntr)], check=True, capture_output=True, text=True).stdout
    rows = [tuple(int(v) for v in ln.split()) for ln in out.split("\n") if ln]
    first, second, last, beyond = rows
    assert first == (0, 0, 1)
    assert second == (1, 0, int(ntr > 1))
    assert last == (ntr - 1, ns - 1, 1)
    assert beyond == (ntr, 0, 0)
