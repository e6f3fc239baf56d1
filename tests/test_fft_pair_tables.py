"""The stage tables and index arithmetic of the pair FFT (csrc/fft_pair.cuh): the
host part of the header gives every twiddle's angle, and the transform that its
split describes, restated here step by step, is the discrete Fourier transform."""
import os
import shutil
import subprocess

import numpy as np
import pytest

from conftest import ROOT

SRC = r'''
#include <cstdio>
#define __host__
#define __device__
#include "fft_pair.cuh"
using namespace erp;
int main() {
    for (int n = 64; n <= 4096; n *= 2) {
        std::printf("%d %d %d %d %d", n, fft_r1(n), fft_r2(n), fft_r3(n), fft_tw_len(n));
        for (int k = 0; k < fft_tw_len(n); ++k) std::printf(" %d", fft_tw_num(n, k));
        std::printf("\n");
    }
}
'''


@pytest.fixture(scope="module")
def tables(tmp_path_factory):
    if not shutil.which("g++"):
        pytest.skip("no g++")
    d = tmp_path_factory.mktemp("fftpair")
    src, exe = d / "t.cpp", d / "t"
    src.write_text(SRC)
    subprocess.run(["g++", "-O1", "-std=c++17", "-I", os.path.join(ROOT, "reda_erplacer_gb300", "csrc"), str(src),
                    "-o", str(exe)], check=True)
    rows = subprocess.run([str(exe)], check=True, capture_output=True, text=True).stdout.splitlines()
    return [list(map(int, r.split())) for r in rows]


def test_split_is_the_dft(tables):
    assert [r[0] for r in tables] == [64, 128, 256, 512, 1024, 2048, 4096]
    for n, r1, r2, r3, length, *num in tables:
        assert r1 * r2 * r3 == n and r1 % r2 == 0 and r1 % r3 == 0 and length == len(num) <= n
        m = n // r1
        w = np.exp(-2j * np.pi * np.array(num) / n)
        w1 = np.vstack([np.ones(m), w[:(r1 - 1) * m].reshape(r1 - 1, m)])
        w2 = np.vstack([np.ones(r3), w[(r1 - 1) * m:].reshape(r2 - 1, r3)])
        rng = np.random.default_rng(n)
        z = rng.standard_normal(n) + 1j * rng.standard_normal(n)
        a = np.fft.fft(z.reshape(r1, m), axis=0) * w1                       # (q1, t)
        b = np.fft.fft(a.reshape(r1, r2, r3), axis=1) * w2[None]            # (q1, q2, o)
        c = np.fft.fft(b, axis=2)                                           # (q1, q2, q3)
        out = np.empty(n, complex)
        q1, q2, q3 = np.meshgrid(np.arange(r1), np.arange(r2), np.arange(r3), indexing="ij")
        out[q1 + r1 * (q2 + r2 * q3)] = c
        np.testing.assert_allclose(out, np.fft.fft(z), rtol=0, atol=1e-10)
