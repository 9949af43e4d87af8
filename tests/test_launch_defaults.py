"""The argument blocks of the kernels start empty: a pointer that the host does not
set is null, and is refused or built, not followed.  CPU only."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CUDA = "/usr/local/cuda/include"

pytestmark = pytest.mark.skipif(shutil.which("g++") is None or not os.path.isdir(CUDA), reason="needs g++ and CUDA's headers")

SOURCE = r"""
#include <cstdio>
#include <cstring>
#include <new>
#include "xjpcg_internal.hpp"
using namespace xjpcg;
template <typename T>
T* made() {  // default-initialised, on memory that held something else
    static unsigned char room[sizeof(T)] __attribute__((aligned(16)));
    std::memset(room, 0xa5, sizeof room);
    return new (room) T;
}
#define NONE(x, f) if (x->f) { std::printf("%s\n", #f); bad = 1; }
int main() {
    int bad = 0;
    BatchLaunch* b = made<BatchLaunch>();
    NONE(b, sysRow) NONE(b, order) NONE(b, rowptr) NONE(b, col) NONE(b, val) NONE(b, val32) NONE(b, b) NONE(b, diag)
    NONE(b, x) NONE(b, r) NONE(b, Ap) NONE(b, J) NONE(b, r32) NONE(b, d32) NONE(b, Ap32) NONE(b, J32) NONE(b, pGlobal)
    NONE(b, p32Global) NONE(b, res) NONE(b, queue) NONE(b, sliceBase) NONE(b, sliceOff) NONE(b, sval) NONE(b, sval32)
    NONE(b, scol) NONE(b, patLen) NONE(b, patOff) NONE(b, meta) NONE(b, sysPat)
    BatchClusterArgs* c = made<BatchClusterArgs>();
    NONE(c, sysRow) NONE(c, order) NONE(c, width) NONE(c, rowptr) NONE(c, col) NONE(c, val) NONE(c, b) NONE(c, diag)
    NONE(c, x) NONE(c, res)
    LoopArgs* l = made<LoopArgs>();
    NONE(l, sliceOff) NONE(l, sval) NONE(l, col32) NONE(l, col16) NONE(l, patLen) NONE(l, patIdx) NONE(l, patOff)
    NONE(l, genOff) NONE(l, pat) NONE(l, gcol) NONE(l, x) NONE(l, p) NONE(l, r) NONE(l, J) NONE(l, state)
    NONE(l, counters) NONE(l, posts)
    return bad;
}
"""


def test_argument_blocks_start_empty(tmp_path):
    src, exe = tmp_path / "defaults.cpp", tmp_path / "defaults"
    src.write_text(SOURCE)
    subprocess.run(["g++", "-std=c++17", "-O1", "-I" + CUDA, "-I" + os.path.join(ROOT, "include"),
                    "-I" + os.path.join(ROOT, "hpc_gb300", "csrc"), str(src), "-o", str(exe)], check=True)
    run = subprocess.run([str(exe)], capture_output=True, text=True)
    assert run.returncode == 0, "not null: " + run.stdout
