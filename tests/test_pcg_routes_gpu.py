"""Routes of the PCG that a solve takes only where something is missing: the
cooperative launch does not fit (fewer SMs than the device reports), or there is
no memory for the assembled rows.  The function that says so is replaced in a
child process."""
import os
import subprocess

import pytest

import preload

pytestmark = pytest.mark.gpu

TOO_LARGE = '''
#include <dlfcn.h>
#include <cuda_runtime.h>
#include "ipdg.hpp"
static int tried = 0, iterations = 0, fits = 1;
extern "C" int tries() { return tried; }
extern "C" int launched() { return iterations; }
extern "C" void set_fits(int f) { fits = f; }
namespace dgk {
bool persist_fits(const IpdgArgs&, const PcgVecs&, bool) { return fits; }
cudaError_t launch_pcg_persistent(const IpdgArgs&, const PcgVecs&, bool, const void*, double*, void*, unsigned long long*, int, int, cudaStream_t) {
    tried++;
    return cudaErrorCooperativeLaunchTooLarge;
}
cudaError_t launch_pcg_iteration(const IpdgArgs& a, const PcgVecs& v, bool fp32, int parity, const LpcNet* n, const LpcFeatArgs* f, cudaStream_t s) {
    static void* lib = dlopen("LIBRARY", RTLD_NOW | RTLD_NOLOAD);
    static auto real = (decltype(&launch_pcg_iteration))dlsym(lib, "SYMBOL");
    iterations++;
    return real(a, v, fp32, parity, n, f, s);
}
}
'''

FALLBACK = '''
import ctypes, sys
import numpy as np
from hopefoam_gb300 import _lib as L
from hopefoam_gb300.mesh import delaunay_square
from hopefoam_gb300.poisson import PressureSolver
shim = ctypes.CDLL(sys.argv[1])
m = delaunay_square(400, seed=3)
b = np.random.default_rng(0).standard_normal(m.K * 6)
for pc in (L.DG_PC_BLOCK_JACOBI, L.DG_PC_MULTILEVEL):
    for precision in (L.DG_PREC_FP64, L.DG_PREC_SPLIT):
        got = []
        for fits in (0, 1):  # the general iterations from the start; after a launch that does not fit
            shim.set_fits(fits)
            ps = PressureSolver(m, 2, tau_coef=1.0)
            t0 = shim.tries()
            for solve in range(2):
                n0 = shim.launched()
                x, st = ps.solve(b, rtol=1e-10, maxit=20000, pc=pc, precision=precision)
                got.append((x, st["iterations"], shim.launched() - n0))
            assert shim.tries() - t0 == fits, "the launch is tried once"
            ps.ctx.close()
        for x, it, n in got[1:]:
            assert np.array_equal(x, got[0][0]) and it == got[0][1]
        # first solve after the other: the same batches (one more set of launches where a graph is captured)
        assert got[0][2] == got[2][2], (pc, precision, [g[1:] for g in got])
print("same")
'''


def test_cooperative_launch_does_not_fit(gpu_lib, tmp_path):
    from hopefoam_gb300 import build as B

    names = subprocess.run(["nm", "-D", "--defined-only", B.LIB], capture_output=True, text=True, check=True).stdout.split()
    symbol, = [n for n in names if "launch_pcg_iteration" in n]
    so = preload.compile_host(TOO_LARGE.replace("LIBRARY", os.path.realpath(B.LIB)).replace("SYMBOL", symbol), tmp_path / "too_large.so", "-ldl")
    assert "same" in preload.run(so, FALLBACK, so)


NO_ROWS = '''
#include "ipdg.hpp"
namespace dgk { size_t block_rows_size(int, int) { return (size_t)1 << 60; } }
'''

MATRIX_FREE = '''
import sys
import numpy as np
from hopefoam_gb300 import _lib as L
from hopefoam_gb300.mesh import delaunay_square
from hopefoam_gb300.poisson import PressureSolver
N = int(sys.argv[1])
for n in (60, 1500):
    m = delaunay_square(n, seed=3)
    ps = PressureSolver(m, N, tau_coef=20.0)
    b = np.random.default_rng(N).standard_normal(m.K * ps.Np)
    for pc in (L.DG_PC_BLOCK_JACOBI, L.DG_PC_MULTILEVEL):
        for precision in (L.DG_PREC_FP64, L.DG_PREC_SPLIT):
            x, st = ps.solve(b, rtol=1e-10, maxit=20000, pc=pc, precision=precision)
            r = b - ps.apply(x)
            assert st["rel_residual"] <= 1e-10 and np.linalg.norm(r) < 1.001e-10 * np.linalg.norm(b), (n, pc, precision)
    ps.ctx.close()
print("solved")
'''


@pytest.mark.parametrize("N", range(1, 8))
def test_no_memory_for_rows(gpu_lib, tmp_path, N):
    """The matrix-free apply inside the solves, and the general iterations of small problems, every order: the residual of
    the result with the operator's own apply, which the operator tests hold against the oracle (the same kernel as in the
    solve: the stopping tolerance, and round-off of the norm)."""
    so = preload.compile_host(NO_ROWS, tmp_path / "no_rows.so")
    assert "solved" in preload.run(so, MATRIX_FREE, N)


def test_solves_beside_each_other(gpu_lib):
    """Two solvers whose iterations run in one cooperative launch, and Euler steps of a third context, from a host thread
    each: every solve has the bits that it has alone."""
    import concurrent.futures

    import numpy as np

    from hopefoam_gb300 import _lib as L
    from hopefoam_gb300 import euler
    from hopefoam_gb300.mesh import delaunay_square, periodic_square
    from hopefoam_gb300.poisson import PressureSolver

    def solver(n, N, seed):
        m = delaunay_square(n, seed=seed)
        return PressureSolver(m, N, tau_coef=1.0), np.random.default_rng(seed).standard_normal(m.K * (N + 1) * (N + 2) // 2)

    jobs = [(*solver(2000, 3, 1), dict(pc=L.DG_PC_BLOCK_JACOBI, precision=L.DG_PREC_SPLIT)),
            (*solver(900, 3, 2), dict(pc=L.DG_PC_MULTILEVEL, precision=L.DG_PREC_FP64))]
    want = [ps.solve(b, rtol=1e-9, maxit=20000, **kw)[0] for ps, b, kw in jobs]
    m = periodic_square(60, 60, 10.0, 10.0, perturb=0.1, seed=1)
    ops = euler.reference_operators(4)
    q = euler.isentropic_vortex(*euler.node_coords(m, ops["r"], ops["s"]), x0=5.0, y0=5.0)
    ctx = euler.EulerContext(m, 4)
    ctx.upload(q)
    ctx.lserk4(1e-4, 60, precision=L.DG_PREC_SPLIT)
    want_q = ctx.download()

    def solve(ps, b, kw, x):
        for _ in range(6):
            assert np.array_equal(ps.solve(b, rtol=1e-9, maxit=20000, **kw)[0], x), kw

    def step():
        for _ in range(6):
            ctx.upload(q)
            ctx.lserk4(1e-4, 60, precision=L.DG_PREC_SPLIT)
            assert np.array_equal(ctx.download(), want_q), "steps"

    with concurrent.futures.ThreadPoolExecutor(3) as pool:
        for f in [pool.submit(solve, *j, x) for j, x in zip(jobs, want)] + [pool.submit(step)]:
            f.result()
    for ps, _, _ in jobs:
        ps.ctx.close()
    ctx.close()
