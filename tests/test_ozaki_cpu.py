"""Digit slicing of the tensor-core FP64 Euler stage
(hopefoam_gb300/csrc/ozaki.cuh, euler_fp64_tc.cuh), compiled for the host.

Bounds: a value's seven digits restore it to half a unit of the seventh,
2^-56 of the row's bound 2^E, plus the 2^-63 that the shift into the 64-bit
fixed-point word drops; an integer converts to FP64 within half a unit
in the last place; a sliced dot product (exact accumulators, digit pairs
i + j <= 6 or 7) differs from the exact one by the two roundings to digits and
the dropped pairs, together below K (2 + 8) 2^-55 of the rows' bounds."""
import ctypes
import os
import subprocess

import numpy as np
import pytest

from hopefoam_gb300.mesh import load_cubature

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(HERE, "..", "hopefoam_gb300", "csrc")

SRC = r'''
#include <cmath>
#include "euler_fp64_tc.cuh"
extern "C" int row_bound(double v) { return oz::row_bound(oz::mag_hi(v)); }
extern "C" void digits(const double* v, int n, int eb, int* out) {
    for (int i = 0; i < n; i++) {
        const uint64_t y = oz::biased(v[i], eb);
        for (int s = 0; s < 7; s++) out[7 * i + s] = oz::digit(y, s);
    }
}
extern "C" double from_fixed(long long z, int ex) { return oz::from_fixed(z, ex); }
extern "C" double combine7(const int* d, int eb) { return oz::combine7(d[0], d[1], d[2], d[3], d[4], d[5], d[6], eb); }
extern "C" double combine8(const int* d, int eb) { return oz::combine8(d, eb); }
extern "C" int half_bits(int d) { return oz::half_bits(d); }
template <int N> static int img(const double* cub, int n, int smem_limit) {
    dgb::RefOps o;
    if (!dgb::build_ref_ops(N, cub, n, o).empty()) return -1;
    const dgk::OzImage im = dgk::oz_build<N>(o);
    return im.exact && dgk::OzDims<N>::SMEM <= smem_limit && im.bytes.size() == dgk::OzDims<N>::piece_off(dgk::OzDims<N>::PIECES);
}
extern "C" int image(int N, const double* cub, int n, int lim) {
    switch (N) {
        case 1: return img<1>(cub, n, lim); case 2: return img<2>(cub, n, lim); case 3: return img<3>(cub, n, lim);
        case 4: return img<4>(cub, n, lim); case 5: return img<5>(cub, n, lim); case 6: return img<6>(cub, n, lim);
        default: return img<7>(cub, n, lim);
    }
}
'''


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    d = tmp_path_factory.mktemp("ozaki")
    src, so = d / "t.cpp", d / "t.so"
    src.write_text(SRC)
    r = subprocess.run(["g++", "-O2", "-std=c++17", "-shared", "-fPIC", "-I", CSRC, "-I", "/usr/local/cuda/include", str(src),
                        os.path.join(CSRC, "dg_basis.cpp"), "-o", str(so)], capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    L = ctypes.CDLL(str(so))
    for f in (L.from_fixed, L.combine7, L.combine8):
        f.restype = ctypes.c_double
    L.from_fixed.argtypes = [ctypes.c_longlong, ctypes.c_int]
    L.row_bound.argtypes = [ctypes.c_double]
    return L


def _dp(a):
    return a.ctypes.data_as(ctypes.POINTER(ctypes.c_double))


def _ip(a):
    return a.ctypes.data_as(ctypes.POINTER(ctypes.c_int))


def _digits(L, v):
    v = np.ascontiguousarray(v, np.float64)
    eb = L.row_bound(float(np.abs(v).max()))
    out = np.zeros((v.size, 7), np.int32)
    L.digits(_dp(v), v.size, eb, _ip(out))
    return out, eb


def test_digits_restore_values(lib):
    rng = np.random.default_rng(0)
    edge = np.ldexp(np.array([1 - 2.0 ** -53, 1 - 2.0 ** -8, 1 - 2.0 ** -7, 0.5, 0.50390625, 1.0, -1.0, 0.0]), 3)
    for v in (rng.standard_normal(4000) * np.exp2(rng.integers(-70, 5, 4000)), edge, -edge):
        d, eb = _digits(lib, v)
        assert d.min() >= -128 and d.max() <= 127
        w = np.exp2(np.longdouble(eb - 1022) - 7 - 8 * np.arange(7).astype(np.longdouble))
        err = np.abs((d.astype(np.longdouble) * w).sum(1) - v.astype(np.longdouble))
        assert float(err.max()) <= 2.0 ** (eb - 1022 - 56) + 2.0 ** (eb - 1022 - 63)
    # a value that sets its own row's bound
    for x in rng.uniform(1, 2, 2000):
        d, _ = _digits(lib, np.array([x, -x]))
        assert d.min() >= -128 and d.max() <= 127
    # digits as FP16
    for k in range(-128, 128):
        assert np.array([lib.half_bits(k)], np.uint16).view(np.float16)[0] == k


def test_integers_round_to_fp64(lib):
    rng = np.random.default_rng(1)
    for z in [0, 1, -1, (1 << 62) - 1, -(1 << 62)] + [int(t) for t in rng.integers(-2 ** 62, 2 ** 62, 3000) >> rng.integers(0, 61, 3000)]:
        got, want = lib.from_fixed(z, -40), np.longdouble(z) * np.exp2(np.longdouble(-40))
        assert abs(np.longdouble(got) - want) <= np.longdouble(2.0) ** -53 * abs(want)


@pytest.mark.parametrize("K,groups", [(3, 7), (36, 7), (33, 8), (263, 8)])
def test_sliced_products(lib, K, groups):
    """Smallest and largest reduction lengths of the stage's two kinds of product."""
    rng = np.random.default_rng(K)
    for trial in range(200):
        a = rng.standard_normal(K) * np.exp2(rng.integers(-6, 6)) + (trial % 3)
        b = rng.uniform(-1, 1, K) * np.exp2(rng.integers(-4, 3, K).astype(float))
        da, ea = _digits(lib, a)
        db, eb = _digits(lib, b)
        D = np.zeros(8, np.int64)
        for i in range(7):
            for j in range(7):
                if i + j < groups:
                    D[i + j] += (da[:, i].astype(np.int64) * db[:, j]).sum()
        assert np.abs(D).max() < (1 << 22 if groups == 7 else 1 << 24)
        got = (lib.combine7 if groups == 7 else lib.combine8)(_ip(D.astype(np.int32)), ea + eb)
        want = (a.astype(np.longdouble) * b.astype(np.longdouble)).sum()
        scale = 2.0 ** (ea + eb - 2044)
        assert abs(float(np.longdouble(got) - want)) <= K * 10 * 2.0 ** -55 * scale + 2.0 ** -53 * abs(float(want))


@pytest.mark.parametrize("N", range(1, 8))
def test_operator_images_are_exact(lib, N):
    """The largest possible accumulators of every order stay below 2^22 (interpolation) and 2^24 (weak derivative and lift)."""
    cub = np.ascontiguousarray(load_cubature(3 * (N + 1)))
    assert lib.image(N, _dp(cub), len(cub), 232448) == 1
