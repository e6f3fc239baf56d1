"""The shared memory of the scatter order's counting pass (csrc/sorttiles.h), compiled
for the host: on every grid that the library takes, the counts of its sort tiles fit
what the kernel is opted in to, which a block of this GPU can have (227 KB); and every
bin's tile lies inside the counts."""
import os
import shutil
import subprocess

import pytest

from conftest import ROOT

SRC = r'''
#include <cstdio>
#include "sorttiles.h"
using namespace erp;
int main() {
    int bad = 0, grids = 0;
    for (int m = kGridMin; m <= kGridMax; m *= 2)
        for (int n = kGridMin; n <= kGridMax; n *= 2, ++grids) {
            const size_t need = sort_count_smem(m, n);
            const int nty = (n + kSortTile - 1) / kSortTile;
            const size_t last = 4 * ((size_t)((m - 1) / kSortTile) * nty + (n - 1) / kSortTile + 1);
            if (need > kSortCountSmem || need > 227 * 1024 || last > need) { printf("%d x %d: %zu\n", m, n, need); ++bad; }
        }
    printf("%s %d %d %d\n", bad ? "FAIL" : "ok", grids, kGridMin, kGridMax);
    return bad != 0;
}
'''


def test_counts_fit_on_every_grid(tmp_path):
    if not shutil.which("g++"):
        pytest.skip("no host C++ compiler")
    src, exe = tmp_path / "t.cpp", tmp_path / "t"
    src.write_text(SRC)
    csrc = os.path.join(ROOT, "reda_erplacer_gb300", "csrc")
    subprocess.run(["g++", "-O2", "-std=c++17", "-I", csrc, str(src), "-o", str(exe)], check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True, timeout=60)
    assert r.returncode == 0 and r.stdout.split() == ["ok", "81", "16", "4096"], r.stdout
    # the kernel that takes more than 48 KB is opted in, to that amount
    src = open(os.path.join(csrc, "k_place.cu")).read()
    assert "cudaFuncSetAttribute(k_sort_count, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kSortCountSmem)" in src
