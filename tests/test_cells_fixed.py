"""The integer conversion of shifts (cells) to fixed-point phase slopes
(csrc/cells_fixed.h) against exact integer arithmetic: v / N cycles in units
of 2^-64, rounded half to even, modulo one cycle."""
import ctypes
import math
import os
import subprocess

import numpy as np
import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "isar_imaging_cuda_gb300", "csrc")

SRC = r"""
#include <cstring>
#include "cells_fixed.h"
extern "C" void convert(const double* v, int64_t* out, long n, int lg)
{
    for (long i = 0; i < n; ++i) {
        uint64_t b;
        std::memcpy(&b, &v[i], 8);
        out[i] = isar::cells_to_fixed(b, lg);
    }
}
"""


def exact_fixed(v, lg):
    """v / 2^lg cycles in units of 2^-64, rounded half to even, as a signed
    64-bit number modulo one cycle; in integers."""
    m, e = math.frexp(v)
    n, k = int(m * (1 << 53)), e - 53 + 64 - lg
    if k >= 0:
        r = n << k
    else:
        q, rem = divmod(n, 1 << -k)
        twice = 2 * rem - (1 << -k)
        r = q + (1 if twice > 0 or (twice == 0 and q & 1) else 0)
    r &= (1 << 64) - 1
    return r - (1 << 64) if r >> 63 else r


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    d = tmp_path_factory.mktemp("cells")
    (d / "t.cpp").write_text(SRC)
    so = str(d / "t.so")
    subprocess.run(["g++", "-O2", "-ffp-contract=off", "-shared", "-fPIC", "-I", CSRC, str(d / "t.cpp"), "-o", so],
                   check=True)
    m = ctypes.CDLL(so)
    m.convert.argtypes = [ctypes.c_void_p, ctypes.c_void_p, ctypes.c_long, ctypes.c_int]
    return m


@pytest.mark.parametrize("lg", [9, 10, 11, 12, 13])
def test_cells_to_fixed_is_exact(lib, lg):
    rng = np.random.default_rng(lg)
    N = float(1 << lg)
    f32 = (rng.standard_normal(20000) * N).astype(np.float32).astype(np.float64)
    vals = [f32, np.cumsum(f32[:2000]), rng.uniform(-4 * N, 4 * N, 20000),
            rng.standard_normal(20000) * 10.0 ** rng.uniform(-30, 4, 20000),
            np.ldexp(rng.integers(1, 1 << 20, 4000).astype(np.float64), rng.integers(-90, 0, 4000)),   # ties of the rounding
            np.array([0.0, -0.0, 0.5, -0.5, N / 2, -N / 2, N, -N, np.nextafter(N / 2, 0), 2.0 ** -52, -2.0 ** -60, 1e-310])]
    v = np.ascontiguousarray(np.concatenate(vals + [-x for x in vals]))
    got = np.empty(v.size, np.int64)
    lib.convert(v.ctypes.data, got.ctypes.data, v.size, lg)
    assert got.tolist() == [exact_fixed(x, lg) for x in v.tolist()]


def test_no_number_is_half_a_cycle(lib):
    v = np.array([np.nan, -np.nan, np.inf, -np.inf])
    got = np.empty(v.size, np.int64)
    lib.convert(v.ctypes.data, got.ctypes.data, v.size, 13)
    assert got.tolist() == [-(1 << 63)] * 4
