"""Right-hand sides of the tensor-core FP64 stage (euler_fp64_tc.cu) and of the
plain FP64 stage (euler_fp64.cu) against the same formulas in extended
precision, on elements in which density, pressure or both vary strongly, and
between neighbours of different density: the tensor-core stage has to be as
exact as the plain one, also where the digits of a row share one exponent.

The plain stage runs in a child process in which no operator is taken to be
exact in digits (its setup function replaced).  Both take the library's own
fused operators, as the extended-precision one does, so that only the stage's
arithmetic differs.  The criterion, over the elements of one state and order: the median of
err_tc / err_plain (L2 over the nodes, each variable against its own norm) at most 1.25, the
ratio of the root mean squares at most 2.  Emulated on the host the medians are 0.5 to 1.03; the median of
72 ratios that scatter by a factor of 1.5 moves by 0.07, the mean squares hang on a few elements."""
import ctypes

import numpy as np
import pytest

import preload
from conftest import rel_l2

pytestmark = pytest.mark.gpu

LD = np.longdouble
GAMMA = LD(1.4)

NO_DIGITS = '''
#include "dg_internal.hpp"
namespace dgk { cudaError_t setup_euler_fp64_tc(int, const dgb::RefOps&, int, OzPlan&) { return cudaSuccess; } }
'''

OPS = '''
#include <cstring>
#include "dg_basis.hpp"
extern "C" int ops(int N, const double* cub, int n, int* sizes, int* ring, double* Vg, double* If, double* Sr, double* Ss, double* Lift) {
    dgb::RefOps o;
    if (!dgb::build_ref_ops(N, cub, n, o).empty()) return 1;
    const int s[4] = {o.Np, o.Ng, o.Nfp, o.Nfq};
    memcpy(sizes, s, sizeof(s));
    if (!Vg) return 0;
    memcpy(ring, o.ring.data(), o.Np * sizeof(int));
    auto put = [](double* d, const std::vector<double>& v) { memcpy(d, v.data(), v.size() * sizeof(double)); };
    put(Vg, o.dVg); put(If, o.If); put(Sr, o.dSr); put(Ss, o.dSs); put(Lift, o.dLift);
    return 0;
}
'''

PLAIN = '''
import sys
import numpy as np
from hopefoam_gb300 import euler
from hopefoam_gb300.mesh import periodic_square
N, path = int(sys.argv[1]), sys.argv[2]
q = np.load(path + "_q.npy")
ctx = euler.EulerContext(periodic_square(6, 6, 10.0, 10.0, perturb=0.1, seed=N), N)
out = []
for state in q:
    ctx.upload(state)
    out.append([ctx.rhs(flux=f) for f in (0, 1)])
np.save(path + "_r.npy", np.array(out))
'''


@pytest.fixture(scope="module")
def libs(tmp_path_factory):
    import os

    d = tmp_path_factory.mktemp("precision")
    return (preload.compile_host(NO_DIGITS, d / "nodigits.so"),
            ctypes.CDLL(preload.compile_host(OPS, d / "ops.so", os.path.join(preload.CSRC, "dg_basis.cpp"))), d)


def _operators(lib, N):
    from hopefoam_gb300.mesh import load_cubature

    cub = np.ascontiguousarray(load_cubature(3 * (N + 1)))
    p = lambda a: a.ctypes.data_as(ctypes.c_void_p)
    sz = np.zeros(4, np.int32)
    assert lib.ops(N, p(cub), len(cub), p(sz), *[None] * 6) == 0
    Np, Ng, Nfp, Nfq = map(int, sz)
    ring = np.zeros(Np, np.int32)
    A = [np.zeros(s) for s in ((Ng, Np), (Nfq, Nfp), (Np, Ng), (Np, Ng), (Np, 3 * Nfq))]
    assert lib.ops(N, p(cub), len(cub), p(sz), p(ring), *map(p, A)) == 0
    return ring, [a.astype(LD) for a in A]


def _primitive(q):
    u, v = q[1] / q[0], q[2] / q[0]
    return u, v, (GAMMA - 1) * (q[3] - (q[1] * u + q[2] * v) / 2)


def _flux(q):
    u, v, p = _primitive(q)
    return (np.stack([q[1], u * q[1] + p, u * q[2], u * (q[3] + p)]), np.stack([q[2], v * q[1], v * q[2] + p, v * (q[3] + p)]))


def _roe(nx, ny, a, b):
    """Flux of euler_flux.cuh's roe_flux, owner a, neighbour b."""
    rot = lambda q: (nx * q[1] + ny * q[2], nx * q[2] - ny * q[1])
    (mO, tO), (mN, tN) = rot(a), rot(b)
    uM, uP, vM, vP = mO / a[0], mN / b[0], tO / a[0], tN / b[0]
    pM, pP = ((GAMMA - 1) * (q[3] - (m * u + t * v) / 2) for q, m, t, u, v in ((a, mO, tO, uM, vM), (b, mN, tN, uP, vP)))
    HM, HP = (a[3] + pM) / a[0], (b[3] + pP) / b[0]
    sM, sP = np.sqrt(a[0]), np.sqrt(b[0])
    u, v, H = ((sM * x + sP * y) / (sM + sP) for x, y in ((uM, uP), (vM, vP), (HM, HP)))
    c2 = (GAMMA - 1) * (H - (u * u + v * v) / 2)
    c, rhob = np.sqrt(np.abs(c2)), sM * sP
    d1, d4 = ((s * rhob * (uP - uM) / c / 2 + (pP - pM) / c2 / 2) * np.abs(u + s * c) for s in (-1, 1))
    d2, d3 = ((b[0] - a[0]) - (pP - pM) / c2) * np.abs(u), rhob * (vP - vM) * np.abs(u)
    fr = (mO + mN - d1 - d2 - d4) / 2
    fu = (mO * uM + pM + mN * uP + pP - d1 * (u - c) - d2 * u - d4 * (u + c)) / 2
    fv = (tO * uM + tN * uP - d1 * v - d2 * v - d3 - d4 * v) / 2
    fe = (uM * (a[3] + pM) + uP * (b[3] + pP) - d1 * (H - u * c) - d2 * (u * u + v * v) / 2 - d3 * v - d4 * (H + u * c)) / 2
    return np.stack([fr, nx * fu - ny * fv, ny * fu + nx * fv, fe])


def _reference(m, N, ring, ops, q, flux):
    """Right-hand side in extended precision, reference node order."""
    Vg, If, Sr, Ss, Lift = ops
    nfp, nfq, nb = N + 1, If.shape[0], 3 * N
    v = np.asarray(m.VXY, np.float64)
    xr, yr, xs, ys = 0.5 * (v[:, 1, 0] - v[:, 0, 0]), 0.5 * (v[:, 1, 1] - v[:, 0, 1]), 0.5 * (v[:, 2, 0] - v[:, 0, 0]), 0.5 * (v[:, 2, 1] - v[:, 0, 1])
    J = xr * ys - xs * yr
    rx, sx, ry, sy = (t.astype(LD) for t in (ys / J, -yr / J, -xs / J, xr / J))
    w = q[:, :, ring].astype(LD)
    fx, fy = _flux(w @ Vg.T)
    R = (rx[:, None] * fx + ry[:, None] * fy) @ Sr.T + (sx[:, None] * fx + sy[:, None] * fy) @ Ss.T
    j = np.arange(nfp)
    pos = lambda f: (f * N + j) % nb
    for f in range(3):
        gx, gy = ((-sx, -sy), (rx + sx, ry + sy), (-rx, -ry))[f]
        s = np.sqrt(gx * gx + gy * gy)
        nx, ny = (gx / s)[:, None], (gy / s)[:, None]
        nbr = np.empty(w.shape[:2] + (nfp,), LD)
        for k in range(m.K):
            k2, f2 = m.EToE[k, f], m.EToF[k, f]
            nbr[:, k] = w[:, k2][:, pos(f2)[::-1] if m.ROT[k, f] & 1 else pos(f2)]
        a, b = w[:, :, pos(f)] @ If.T, nbr @ If.T
        if flux == 1:
            F = _roe(nx, ny, a, b)
        else:
            speed = lambda q: (lambda u, v, p: np.abs(u * nx + v * ny) + np.sqrt(np.abs(GAMMA * p / q[0])))(*_primitive(q))
            lam = np.maximum(speed(a), speed(b)).max(1)[:, None]
            (ax, ay), (bx, by) = _flux(a), _flux(b)
            F = ((ax + bx) * nx + (ay + by) * ny + lam * (a - b)) / 2
        R -= (s[:, None] * F) @ Lift[:, f * nfq:(f + 1) * nfq].T
    out = np.empty_like(R)
    out[:, :, ring] = R
    return out


def _states(m, N, kind, C):
    """Per element linear in a random direction, from 1 to C."""
    from hopefoam_gb300 import euler

    ops = euler.reference_operators(N)
    rng = np.random.default_rng(100 * N + int(C))
    th = rng.uniform(0, 2 * np.pi, m.K)[:, None]
    t = np.cos(th) * ops["r"] + np.sin(th) * ops["s"]
    t = (t - t.min(1, keepdims=True)) / (t.max(1, keepdims=True) - t.min(1, keepdims=True))
    s, one = 1 + (C - 1) * t, np.ones_like(t)
    u, v, p = (rng.uniform(a, b, m.K)[:, None] * one for a, b in ((-1.5, 1.5), (-1.5, 1.5), (0.5, 2)))
    if kind == "velocity":  # constant velocity and pressure
        return np.stack([s, s * u, s * v, p / 0.4 + 0.5 * s * (u * u + v * v)])
    if kind == "momentum":  # constant momentum and energy
        return np.stack([s, u, v, p / 0.4 + 3 * one])
    if kind == "pressure":
        return np.stack([one, u, v, s * p / 0.4 + 0.5 * (u * u + v * v)])
    scale = C ** rng.uniform(-0.5, 0.5, m.K)[:, None]  # neighbours
    rho = 1 + 0.2 * t
    return scale * np.stack([rho, rho * u, rho * v, p / 0.4 + 0.5 * rho * (u * u + v * v)])


KINDS = ("velocity", "momentum", "pressure", "neighbours")
CONTRASTS = (1.5, 10.0, 25.0, 100.0, 900.0)


@pytest.mark.parametrize("N", range(1, 8))
def test_as_exact_as_the_plain_stage(gpu_lib, libs, N):
    from hopefoam_gb300 import euler
    from hopefoam_gb300.mesh import periodic_square

    so, lib, tmp = libs
    ring, ops = _operators(lib, N)
    m = periodic_square(6, 6, 10.0, 10.0, perturb=0.1, seed=N)
    names = [(k, C) for k in KINDS for C in CONTRASTS]
    q = np.array([_states(m, N, k, C) for k, C in names])
    np.save(tmp / f"{N}_q.npy", q)
    preload.run(so, PLAIN, N, tmp / str(N))
    plain = np.load(tmp / f"{N}_r.npy")
    ctx = euler.EulerContext(m, N)
    rows, ok = [], True
    for i, name in enumerate(names):
        ctx.upload(q[i])
        for flux in (0, 1):
            ref = _reference(m, N, ring, ops, q[i], flux)
            norm = np.sqrt((ref ** 2).sum(2))
            err = [np.sqrt((((g - ref) ** 2).sum(2) / norm ** 2).sum(0)).astype(float) for g in (ctx.rhs(flux=flux), plain[i, flux])]
            med, rms = np.median(err[0] / err[1]), np.linalg.norm(err[0]) / np.linalg.norm(err[1])
            rows.append((*name, flux, float(np.median(err[1])), float(med), float(rms)))
            ok &= med <= 1.25 and rms <= 2.0
    for r in rows:
        print("%-10s %5g flux %d: plain %.1e, median ratio %.2f, rms ratio %.2f" % r)
    assert ok, [r for r in rows if r[4] > 1.25 or r[5] > 2.0]
    ctx.close()


@pytest.mark.parametrize("N", range(1, 8))
@pytest.mark.parametrize("flux", [0, 1])
def test_plain_stage(gpu_lib, libs, N, flux):
    """The plain kernel, which serves operators that are not exact in digits, against the oracle."""
    so, _, tmp = libs
    preload.run(so, '''
import sys
import numpy as np
from conftest import rel_l2
from test_euler_gpu import TOL_RHS, _setup, _vertex_ulp_sensitivity
from hopefoam_gb300 import euler
from hopefoam_gb300.mesh import periodic_square
N, flux = int(sys.argv[1]), int(sys.argv[2])
m = periodic_square(6, 5, 10.0, 10.0, perturb=0.1, seed=N)
ctx, orc, x, y = _setup(m, N)
q = euler.isentropic_vortex(x, y, x0=5.0, y0=5.0, uinf=0.7, vinf=0.2)
ctx.upload(q)
g = ctx.rhs(flux=flux)
r = orc.euler_rhs(q.reshape(-1), flux=flux).reshape(g.shape)
assert rel_l2(g, r) < max(TOL_RHS, 10 * _vertex_ulp_sensitivity(m, N, q, flux, r))
''', N, flux)
