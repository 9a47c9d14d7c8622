"""The draws that a slot's prepared generator state has behind it, by the
expressions of the kernels compiled for the host (CPU): two for each masked
position before the first valid one, in whole blocks of 624, for scans up to
the largest accepted one (2^31 - 1 positions, nearly 2^32 draws)."""
import ctypes
import os
import subprocess

import pytest

from conftest import ROOT

SOURCE = """
#include "qsk_internal.h"
extern "C" long long draws(int nd, const int *fft, const int *lo, int k) {
    qsk::Geom g = {};
    g.nd = nd;
    g.N = 1;
    long long nvalid = 1;
    for (int d = 0; d < nd; ++d) {
        g.fft[d] = g.src[d] = fft[d];
        g.sstride[d] = g.N;
        g.N *= fft[d];
        nvalid *= fft[d] - lo[d];
    }
    const int kept = int(qsk::skipped_blocks(g, lo, nvalid, k));   // the field beside the state
    return qsk::skipped_draws(kept);
}
"""


@pytest.fixture(scope="module")
def draws(tmp_path_factory):
    d = tmp_path_factory.mktemp("draws")
    (d / "draws.cpp").write_text(SOURCE)
    so = str(d / "draws.so")
    subprocess.run(["g++", "-std=c++17", "-shared", "-fPIC", "-I", os.path.join(ROOT, "g2s_b200", "csrc"), "-I",
                    "/usr/local/cuda/include", str(d / "draws.cpp"), "-o", so], check=True)
    f = ctypes.CDLL(so).draws
    f.restype = ctypes.c_longlong
    return lambda fft, lo, k: f(len(fft), (ctypes.c_int * 4)(*fft), (ctypes.c_int * 4)(*lo), k)


@pytest.mark.parametrize("fft,lo", [
    ((100,), (0,)), ((100,), (99,)), ((2000,), (312,)), ((2000,), (313,)), ((50, 40), (7, 5)), ((30, 20, 10), (3, 4, 5)),
    ((2**30 + 700,), (2**30 - 1,)), ((2**30 + 700,), (2**30,)), ((2**30 + 700,), (2**30 + 500,)),
    ((2**31 - 1,), (2**31 - 2,)), ((46340, 46340), (40000, 30000)), ((1290, 1290, 1290), (900, 700, 1280)),
])
def test_skipped_draws(draws, fft, lo):
    # the first valid position in scan order, and the valid ones before it: none
    first, stride = 0, 1
    for f, l in zip(fft, lo):
        first += l * stride
        stride *= f
    n = 2 * first
    assert draws(fft, lo, 1) == (0 if n <= 624 else (n - 1) // 624 * 624)
    assert draws(fft, lo, 2**31 - 1) == 0   # fewer valid positions than k: none are skipped
