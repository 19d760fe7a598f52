"""The collect step of the multilevel correction in the iteration that stops the
solve: every row of z and of its FP32 mirror belongs to that iteration, although
the blocks that sum r.z mark the solve as done while later blocks have not
started.  The correction is called as the iteration calls it, with more row
blocks than the device holds at once."""
import ctypes
import os
import subprocess

import numpy as np
import pytest

import preload

pytestmark = pytest.mark.gpu

SRC = '''
#include <algorithm>
#include <vector>
#include "mg.hpp"
using namespace dgk;
template <typename T>
static T* up(const std::vector<T>& h) {
    T* d = nullptr;
    if (cudaMalloc(&d, std::max<size_t>(h.size(), 1) * sizeof(T)) != cudaSuccess) return nullptr;
    cudaMemcpy(d, h.data(), h.size() * sizeof(T), cudaMemcpyHostToDevice);
    return d;
}
// K elements of Np nodes on nv vertices (element k: k, k + 1, k + 2 mod nv), V the identity; z and dz of one correction
// whose r.r is below the stop limit (first call), or in an iteration after that (second call: nothing may change)
extern "C" int correction(int K, int Np, int nv, const double* lam, const double* r, const double* zb, double* z, float* dz, int* done) {
    std::vector<int> etov(3 * (size_t)K), vptr(nv + 1, 0), vinc(3 * (size_t)K);
    for (int k = 0; k < K; k++)
        for (int c = 0; c < 3; c++) vptr[(etov[3 * k + c] = (k + c) % nv) + 1]++;
    for (int v = 0; v < nv; v++) vptr[v + 1] += vptr[v];
    std::vector<int> fill(vptr.begin(), vptr.end() - 1);
    for (int q = 0; q < 3 * K; q++) vinc[fill[etov[q]]++] = q;
    std::vector<double> V((size_t)nv * nv, 0.0);
    for (int v = 0; v < nv; v++) V[(size_t)v * nv + v] = 1.0;
    const size_t n = (size_t)K * Np;
    MgLevels m;
    m.nl = 1;
    m.lv[0].n = nv;
    m.lv[0].r = up(std::vector<double>(nv, 0.0));
    m.lv[0].x = up(std::vector<double>(nv, 0.0));
    m.V = up(V);
    m.K = K;
    m.Np = Np;
    m.etov = up(etov);
    m.lam = up(std::vector<double>(lam, lam + 3 * Np));
    m.vptr = up(vptr);
    m.vinc = up(vinc);
    double* d_r = up(std::vector<double>(r, r + n));
    double* d_zb = up(std::vector<double>(zb, zb + n));
    double* d_z = up(std::vector<double>(n, -1.0));
    float* d_dz = up(std::vector<float>(n, 0.f));
    double* part = up(std::vector<double>(3 * 4096, 0.0));
    PcgScalars h{};
    h.tol2 = 2.0;
    h.rr = h.rz = h.rzb = 1.0;
    PcgScalars* S = up(std::vector<PcgScalars>(1, h));
    for (int call = 0; call < 2; call++)
        if (launch_mg_correction(m, d_r, d_zb, d_z, d_dz, 3, true, S, part, 1216, nullptr) != cudaSuccess) return 1;
    if (cudaMemcpy(z, d_z, n * sizeof(double), cudaMemcpyDeviceToHost) != cudaSuccess) return 2;
    cudaMemcpy(dz, d_dz, n * sizeof(float), cudaMemcpyDeviceToHost);
    cudaMemcpy(&h, S, sizeof(h), cudaMemcpyDeviceToHost);
    done[0] = h.done;
    done[1] = h.it;
    for (const void* p : {(const void*)m.lv[0].r, (const void*)m.lv[0].x, (const void*)m.V, (const void*)m.etov, (const void*)m.lam,
                          (const void*)m.vptr, (const void*)m.vinc, (const void*)d_r, (const void*)d_zb, (const void*)d_z,
                          (const void*)d_dz, (const void*)part, (const void*)S})
        cudaFree(const_cast<void*>(p));
    return 0;
}
'''


@pytest.fixture(scope="module")
def lib(gpu_lib, tmp_path_factory):
    from hopefoam_gb300 import build as B

    d = tmp_path_factory.mktemp("collect")
    (d / "t.cu").write_text(SRC)
    r = subprocess.run([B.NVCC, *B.ARCH, "-std=c++17", "-Xcompiler", "-fPIC", "-shared", "-I", preload.CSRC, str(d / "t.cu"),
                        "-o", str(d / "t.so"), B.LIB, "-Xlinker", "-rpath=" + os.path.dirname(B.LIB)], capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    return ctypes.CDLL(str(d / "t.so"))


@pytest.mark.parametrize("Np", [3, 15, 36])
def test_rows_of_the_stopping_iteration(lib, Np):
    K, nv = 12_000_000 // (Np * 8) // 3 * 3 + 1, 97
    rng = np.random.default_rng(Np)
    lam = rng.uniform(0, 1, (Np, 3))
    r, zb = 1e-3 * rng.standard_normal((K, Np)), rng.standard_normal((K, Np))
    z, dz, done = np.zeros((K, Np)), np.zeros((K, Np), np.float32), np.zeros(2, np.int32)
    p = lambda a: a.ctypes.data_as(ctypes.c_void_p)
    assert lib.correction(K, Np, nv, p(lam), p(r), p(zb), p(z), p(dz), p(done)) == 0
    assert tuple(done) == (1, 1)
    etov = (np.arange(K)[:, None] + np.arange(3)) % nv
    x = np.zeros(nv)
    np.add.at(x, etov.reshape(-1), (r @ lam).reshape(-1))
    c = x[etov] @ lam.T
    # round-off of sums of K 3 / nv products of the size of r (in another order), and of FP32 for the mirror
    assert np.abs(z - (zb + c)).max() < 1e-10
    assert np.abs(dz - (c - c[:, :1])).max() < 1e-5 * np.abs(c).max()
