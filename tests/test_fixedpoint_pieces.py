"""The density scatter's split of a contribution into pieces (csrc/fixedpoint.h),
compiled for the host: recombined it is rint(x), the integer the oracle's replay
adds, and every piece is below its plane's bound.  Exhaustive over the exponents
where rounding, the carry between pieces and the first integers lie."""
import os
import shutil
import subprocess

import pytest

from conftest import ROOT

SRC = r'''
#include <cstdio>
#include <cstdint>
#include <cstring>
#include "fixedpoint.h"
using namespace erp;
static float from_bits(uint32_t b) { float v; memcpy(&v, &b, 4); return v; }
static long long bad = 0, n = 0;
template <int B> void check2(float x) {
    uint32_t s0, s1;
    fxp_split2<B>(x, s0, s1);
    ++n;
    if (((uint64_t)s1 << B) + s0 != fxp_rint_u64(x) || s0 >> B || s1 >> B) { if (bad++ < 5) printf("%d %a: %u %u\n", B, x, s0, s1); }
}
int main() {
    for (uint32_t e = 0; e < 190; ++e) {
        const uint32_t step = (e >= 124 && e <= 151) ? 1 : 997;
        for (uint32_t m = 0; m < (1u << 23); m += step) {
            const float x = from_bits((e << 23) | m);
            if (x < 4398046511104.0f) check2<21>(x);
            if (x < 70368744177664.0f) check2<23>(x);
            uint32_t s0, s1, s2;
            fxp_split3(x, s0, s1, s2);
            ++n;
            if (((uint64_t)s2 << 42) + ((uint64_t)s1 << 21) + s0 != fxp_rint_u64(x) || s0 >> 21 || s1 >> 21 || s2 >> 21) { if (bad++ < 5) printf("3 %a\n", x); }
        }
    }
    printf("%s %lld\n", bad ? "FAIL" : "ok", n);
    return bad != 0;
}
'''


def test_pieces_recombine_to_rint(tmp_path):
    if not shutil.which("g++"):
        pytest.skip("no host C++ compiler")
    src, exe = tmp_path / "p.cpp", tmp_path / "p"
    src.write_text(SRC)
    subprocess.run(["g++", "-O2", "-std=c++17", "-ffp-contract=off", "-I",
                    os.path.join(ROOT, "reda_erplacer_gb300", "csrc"), str(src), "-o", str(exe)], check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0 and r.stdout.startswith("ok"), r.stdout[-2000:]
