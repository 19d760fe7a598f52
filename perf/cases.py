"""Performance cases: what users of this package have it do, through its public entry points.

Four families, over the sizes that the tests, the tutorials' meshes and bench.py use:

* ``euler``    time steps of the compressible Euler solver (``EulerContext``): device state in, one LSERK4 or
               SSP-RK2 step, device state out; FP64 (the default) and split precision, LF and Roe, orders 1..7;
* ``batch``    many independent vortex cases of mixed orders advanced together (``EulerBatch``);
* ``shock``    one limited SSP-RK2 step of the double-Mach tutorial (walls, limiter, moving-shock data);
* ``poisson``  one pressure solve (``PressureSolver.solve``): block Jacobi or multilevel, mixed or FP64;
* ``chorin``   two incompressible steps (``ChorinSolver``: BDF1 start, then BDF2) of the Pearson vortex.

Time steps are short enough (``cfl``) that one split-precision step stays near FP64 accuracy on the coarse
meshes too; the work of a step does not depend on its length.
"""
import functools
import math
import os

import numpy as np
import torch

from hopefoam_gb300 import _lib as L
from hopefoam_gb300 import euler
from hopefoam_gb300.batch import EulerBatch, batch_cases
from hopefoam_gb300.ins import ChorinSolver, PearsonVortex, pearson_mesh
from hopefoam_gb300.mesh import Mesh, connect, delaunay_square, periodic_square
from hopefoam_gb300.poisson import PressureSolver
from hopefoam_gb300.shock import DoubleMach

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
GAMMA = 1.4
BOX = 10.0
FLUX = {"lf": L.DG_FLUX_LF, "roe": L.DG_FLUX_ROE}
PREC = {"fp64": L.DG_PREC_FP64, "split": L.DG_PREC_SPLIT}
PC = {"bj": L.DG_PC_BLOCK_JACOBI, "multilevel": L.DG_PC_MULTILEVEL}


def listed():
    return [
        # the smallest runs: the tutorial-sized vortex (reference loop: Roe, SSP-RK2, FP64), launches and latency
        dict(name="vortex-512-n2-roe-fp64", kind="euler", order=2, nx=16, ny=16, flux="roe", scheme="ssprk2", prec="fp64", cfl=0.2),
        # the CPU-sized verification run: K = 3200, N = 3, plain FP64
        dict(name="vortex-3200-n3-lf-fp64", kind="euler", order=3, nx=40, ny=40, flux="lf", scheme="lserk4", prec="fp64", cfl=0.5),
        # an ordinary FP64 production run at the headline order
        dict(name="vortex-32768-n5-lf-fp64", kind="euler", order=5, nx=128, ny=128, flux="lf", scheme="lserk4", prec="fp64", cfl=0.5),
        # the highest order in FP64, ragged element count (tiles never come out even)
        dict(name="vortex-9794-n7-roe-fp64", kind="euler", order=7, nx=71, ny=69, flux="roe", scheme="lserk4", prec="fp64", cfl=0.5),
        # the headline workload: split precision, N = 5, K = 131072
        dict(name="vortex-131072-n5-lf-split", kind="euler", order=5, nx=256, ny=256, flux="lf", scheme="lserk4", prec="split", cfl=0.2),
        # a large high-order split run (working set far above L2)
        dict(name="vortex-320000-n7-roe-split", kind="euler", order=7, nx=400, ny=400, flux="roe", scheme="lserk4", prec="split", cfl=0.2),
        # parameter sweep: uneven cases of orders 2..6 in one graph launch
        dict(name="batch-24-n2to6-split", kind="batch", n=24, kmin=800, kmax=20000, cfl=0.02),
        # shock tutorial: limited SSP-RK2 step, walls, FP64
        dict(name="doublemach-5390-n4-fp64", kind="shock", order=4, prec="fp64", dt=1e-5),
        # a small pressure solve with the plain preconditioner (host arrays, the default options)
        dict(name="poisson-4k-n4-bj-split", kind="poisson", order=4, n=2000, pc="bj", prec="split"),
        # the large pressure solve with the multilevel preconditioner
        dict(name="poisson-101k-n4-ml-split", kind="poisson", order=4, n=50000, pc="multilevel", prec="split"),
        # incompressible steps: a small tutorial-sized mesh, and a refined one (FP64, the default)
        dict(name="chorin-1152-n3-fp64", kind="chorin", order=3, n=24, prec="fp64", rtol=1e-11),
        dict(name="chorin-32768-n2-fp64", kind="chorin", order=2, n=128, prec="fp64", rtol=1e-11),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["euler", "euler", "euler", "batch", "shock", "poisson", "chorin"])
    if kind == "euler":
        prec = rng.choice(["fp64", "split"])
        order = rng.randint(1, 7)
        # nodes: 3e3 .. 7e5 (FP64: 53 ms a step at the top), .. 4e6 (split)
        nodes = _log_int(rng, 3000, 700000 if prec == "fp64" else 4000000)
        m = max(12, int(math.sqrt(nodes / ((order + 1) * (order + 2)))))
        return dict(kind=kind, order=order, nx=m + rng.randint(0, 3), ny=m + rng.randint(-3, 3),
                    flux=rng.choice(["lf", "roe"]), scheme=rng.choice(["lserk4", "lserk4", "ssprk2"]), prec=prec,
                    cfl=0.5 if prec == "fp64" else 0.02)
    if kind == "batch":
        return dict(kind=kind, n=rng.randint(5, 30), kmin=800, kmax=_log_int(rng, 2000, 20000), cfl=0.02)
    if kind == "shock":
        return dict(kind=kind, order=rng.randint(2, 6), prec=rng.choice(["fp64", "fp64", "split"]),
                    dt=rng.uniform(2e-6, 1e-5))
    if kind == "poisson":
        pc = rng.choice(["bj", "multilevel"])
        return dict(kind=kind, order=rng.randint(2, 5), n=_log_int(rng, 500, 3000 if pc == "bj" else 20000), pc=pc,
                    prec=rng.choice(["split", "fp64"]))
    order = rng.randint(2, 4)
    return dict(kind=kind, order=order, n=_log_int(rng, 12, 100 if order == 2 else 48), prec=rng.choice(["fp64", "split"]),
                rtol=1e-11)


# ---------------------------------------------------------------------------
# inputs


@functools.lru_cache(maxsize=8)
def _periodic(nx, ny):
    return periodic_square(nx, ny, BOX, BOX, perturb=0.1, seed=nx)


@functools.lru_cache(maxsize=8)
def _delaunay(n):
    return delaunay_square(n, seed=3)


@functools.lru_cache(maxsize=2)
def _double_mach():
    d = np.load(os.path.join(ROOT, "tests", "golden", "doublemach.npz"))
    EToE, EToF, ROT, BC = connect(d["EToV"])
    m = Mesh(d["EToV"], d["VXY"], EToE, EToF, ROT, BC, name="doublemach")
    m.patch, m.patch_names = d["patch"], tuple(str(x) for x in d["patch_names"])
    m.patch_first_face = d["patch_first_face"]
    return m


def _dev(a):
    return torch.as_tensor(np.ascontiguousarray(a), device="cuda")


def _coords(mesh, r, s):
    """Node coordinates x(r, s), y(r, s) of every element, (K, Np) each, on the GPU."""
    v, r, s = _dev(mesh.VXY), _dev(r), _dev(s)
    w = torch.stack([-(r + s) / 2, (1 + r) / 2, (1 + s) / 2])
    return v[:, :, 0] @ w, v[:, :, 1] @ w


def _vortex(x, y, seed):
    """Isentropic vortex in a free stream, strength and stream drawn from the seed, plus a smooth disturbance."""
    rng = np.random.default_rng(seed)
    beta, mach, ang = rng.uniform(3.0, 5.0), rng.uniform(0.3, 0.8), rng.uniform(0, 2 * np.pi)
    uinf, vinf = mach * math.sqrt(GAMMA) * math.cos(ang), mach * math.sqrt(GAMMA) * math.sin(ang)
    dx, dy = x - BOX / 2, y - BOX / 2
    r2 = dx * dx + dy * dy
    rho = (1 - (GAMMA - 1) * beta ** 2 * torch.exp(2 * (1 - r2)) / (16 * GAMMA * math.pi ** 2)) ** (1 / (GAMMA - 1))
    u = uinf - beta * torch.exp(1 - r2) * dy / (2 * math.pi)
    v = vinf + beta * torch.exp(1 - r2) * dx / (2 * math.pi)
    p = rho ** GAMMA
    k = 2 * math.pi / BOX
    a, b = rng.uniform(0, 2 * np.pi, 2)
    rho = rho * (1 + 0.02 * torch.sin(k * (x + 2 * y) + a) * torch.cos(k * (2 * x - y) + b))
    return torch.stack([rho, rho * u, rho * v, p / (GAMMA - 1) + 0.5 * rho * (u * u + v * v)]).contiguous()


def _cfl_dt(mesh, q, order, cfl):
    rho, u, v = q[0], q[1] / q[0], q[2] / q[0]
    p = (GAMMA - 1) * (q[3] - 0.5 * rho * (u * u + v * v))
    smax = float((torch.sqrt(u * u + v * v) + torch.sqrt(GAMMA * p / rho)).max())
    return cfl * mesh.min_h() / ((order + 1) ** 2 * smax)


def _modes(x, y, seed, kmax=16):
    """Pressure source on [0, 2 pi]^2: Taylor-Green terms plus random Fourier modes, amplitudes ~ N(0, 1/|k|^2)."""
    rng = np.random.default_rng(seed)
    f = torch.cos(2 * x) + torch.cos(2 * y)
    for kx in range(-kmax, kmax + 1):
        for ky in range(0, kmax + 1):
            k2 = kx * kx + ky * ky
            if k2 == 0 or k2 > kmax * kmax or (ky == 0 and kx < 0) or rng.random() > 0.15:
                continue
            a, b = rng.standard_normal(2) / math.sqrt(k2)
            ph = kx * x + ky * y
            f = f + a * torch.cos(ph) + b * torch.sin(ph)
    return f


def _euler_inputs(case, seed, r, s):
    mesh = _periodic(case["nx"], case["ny"])
    q = _vortex(*_coords(mesh, r, s), seed)
    return mesh, q, _cfl_dt(mesh, q, case["order"], case["cfl"])


def _poisson_inputs(case, seed, r, s, mass):
    mesh = _delaunay(case["n"])
    x, y = _coords(mesh, r, s)
    v = _dev(mesh.VXY)
    a, b = v[:, 1] - v[:, 0], v[:, 2] - v[:, 0]
    J = 0.25 * (a[:, 0] * b[:, 1] - a[:, 1] * b[:, 0])
    return mesh, J[:, None] * (_modes(x, y, seed) @ _dev(mass).T)


def _batch_list(case, seed):
    """Orders and meshes by the case alone, vortex strengths and Mach numbers by the seed."""
    rng = np.random.default_rng(seed)
    return [dict(c, beta=float(rng.uniform(1, 6)), mach=float(rng.uniform(0.1, 0.8)))
            for c in batch_cases(case["n"], seed=case["n"], kmin=case["kmin"], kmax=case["kmax"])]


# ---------------------------------------------------------------------------


def prepare(case, seed):
    kind = case["kind"]
    if kind == "euler":
        ops = euler.reference_operators(case["order"])
        mesh, q, dt = _euler_inputs(case, seed, ops["r"], ops["s"])
        ctx = euler.EulerContext(mesh, case["order"])
        return dict(case=case, ctx=ctx, q=q, out=torch.empty_like(q), dt=dt)
    if kind == "batch":
        b = EulerBatch(_batch_list(case, seed), cfl=case["cfl"])
        q = []
        for g in b.groups:
            t = torch.empty((4, g["ctx"].K, g["ctx"].Np), dtype=torch.float64, device="cuda")
            g["ctx"].download_device(t.data_ptr())
            q.append(t)
        torch.cuda.synchronize()
        return dict(case=case, batch=b, q=q, out=[torch.empty_like(t) for t in q])
    if kind == "shock":
        mesh = _double_mach()
        dm = DoubleMach(mesh, case["order"])
        ctx = euler.EulerContext(mesh, case["order"])
        q = dm.initial_state()
        q = q * (1 + 1e-3 * np.random.default_rng(seed).standard_normal(q.shape))  # a flow that has developed
        ctx.set_boundary_traces(dm.bdata(0.0))
        ctx.set_boundary_kinds(dm.kinds, dm.gref)
        q = _dev(q)
        return dict(case=case, ctx=ctx, q=q, out=torch.empty_like(q), bdata=dm.bdata(0.0), bdata1=dm.bdata(case["dt"]))
    if kind == "poisson":
        ops = euler.reference_operators(case["order"])
        mesh, b = _poisson_inputs(case, seed, ops["r"], ops["s"], ops["Mref"])
        return dict(case=case, ps=PressureSolver(mesh, case["order"], tau_coef=1.0), b=b.cpu().numpy().reshape(-1))
    nu = 0.01
    cs = ChorinSolver(pearson_mesh(case["n"]), case["order"], nu=nu, dt=1e-3,
                      precision=None if case["prec"] == "fp64" else PREC[case["prec"]])
    pv = PearsonVortex(cs)
    t0 = float(np.random.default_rng(seed).uniform(0, 0.5))
    U, p = pv.initial_state(t0)
    return dict(case=case, cs=cs, U=U, p=p, bd=[pv.bdata(t0), pv.bdata(t0 + cs.dt)])


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "euler":
        ctx = state["ctx"]
        ctx.upload_device(state["q"].data_ptr())
        step = ctx.lserk4 if case["scheme"] == "lserk4" else ctx.ssprk2
        step(state["dt"], 1, flux=FLUX[case["flux"]], precision=PREC[case["prec"]])
        ctx.download_device(state["out"].data_ptr())
        return state["out"]
    if kind == "batch":
        b = state["batch"]
        for g, q in zip(b.groups, state["q"]):
            g["ctx"].upload_device(q.data_ptr())
        b.run(1)
        for g, o in zip(b.groups, state["out"]):
            g["ctx"].download_device(o.data_ptr())
        return state["out"]
    if kind == "shock":
        ctx = state["ctx"]
        ctx.upload_device(state["q"].data_ptr())
        ctx.set_boundary_traces(state["bdata"])
        ctx.limited_ssprk2(case["dt"], state["bdata1"], precision=PREC[case["prec"]])
        ctx.download_device(state["out"].data_ptr())
        return state["out"]
    if kind == "poisson":
        x, _ = state["ps"].solve(state["b"], rtol=1e-10, pc=PC[case["pc"]], precision=PREC[case["prec"]])
        return x
    cs = state["cs"]
    cs.set_state(state["U"], state["p"])
    for bd in state["bd"]:
        cs.step(bd, rtol=case["rtol"])
    return cs.get_state()


def _euler_work(K, N, stages):
    """Per stage: state read and written once, metrics and neighbour words; the interpolation, volume, lift and
    trace contractions (2 flops a multiply-add)."""
    Np, Nfp, Nfq = (N + 1) * (N + 2) // 2, N + 1, N + 2
    Ng = [0, 12, 19, 36, 54, 73, 93, 118][N]
    flops = 2 * 4 * (3 * Ng * Np + 3 * Nfq * Np + 2 * 3 * Nfq * Nfp)
    return dict(bytes=K * (64 * Np + 44) * stages, flops=K * flops * stages)


def work(case):
    kind = case["kind"]
    if kind == "euler":
        return _euler_work(2 * case["nx"] * case["ny"], case["order"], 5 if case["scheme"] == "lserk4" else 2)
    if kind == "batch":
        k = (case["kmax"] - case["kmin"]) / math.log(case["kmax"] / case["kmin"])  # mean of the log-uniform counts
        per = [_euler_work(case["n"] * k / 5, N, 5) for N in (2, 3, 4, 5, 6)]
        return dict(bytes=sum(p["bytes"] for p in per), flops=sum(p["flops"] for p in per))
    if kind == "shock":
        return _euler_work(5390, case["order"], 2)
    # solves: the data once and the operator once per unit of the iteration counts that conjugate gradients need
    # (plain block Jacobi: about the inverse mesh width times the order)
    N = case["order"]
    Np, Nfp, Nfq = (N + 1) * (N + 2) // 2, N + 1, N + 2
    op = 2 * (3 * Np * Np + 2 * 3 * Nfq * (2 * Np + Nfp))
    if kind == "poisson":
        K = 2 * case["n"]
        its = 150 if case["pc"] == "multilevel" else 8 * N * math.sqrt(case["n"])
        return dict(bytes=16.0 * K * Np, flops=K * op * its)
    K = 2 * case["n"] ** 2
    return dict(bytes=2 * 48.0 * K * Np, flops=2 * K * op * 150)


# ---------------------------------------------------------------------------
# the same in plain 64-bit torch, from the published method (nodal DG, Hesthaven & Warburton)


def _jacobi(x, a, b, n):
    """Orthonormal Jacobi polynomial of degree n."""
    g0 = 2 ** (a + b + 1) / (a + b + 1) * math.gamma(a + 1) * math.gamma(b + 1) / math.gamma(a + b + 1)
    p = [np.full_like(x, 1 / math.sqrt(g0))]
    if n == 0:
        return p[0]
    g1 = (a + 1) * (b + 1) / (a + b + 3) * g0
    p.append(((a + b + 2) * x / 2 + (a - b) / 2) / math.sqrt(g1))
    old = 2 / (2 + a + b) * math.sqrt((a + 1) * (b + 1) / (a + b + 3))
    for i in range(1, n):
        h = 2 * i + a + b
        new = 2 / (h + 2) * math.sqrt((i + 1) * (i + 1 + a + b) * (i + 1 + a) * (i + 1 + b) / (h + 1) / (h + 3))
        p.append(((x + (a * a - b * b) / h / (h + 2)) * p[-1] - old * p[-2]) / new)
        old = new
    return p[n]


def _djacobi(x, a, b, n):
    return np.zeros_like(x) if n == 0 else math.sqrt(n * (n + a + b + 1)) * _jacobi(x, a + 1, b + 1, n - 1)


def _gauss(n):
    return np.polynomial.legendre.leggauss(n)


def _gll(N):
    if N == 1:
        return np.array([-1.0, 1.0])
    c = np.polynomial.legendre.Legendre.basis(N).deriv()
    x = np.sort(np.real(c.roots()))
    for _ in range(4):
        x = x - c(x) / c.deriv()(x)
    return np.concatenate([[-1.0], x, [1.0]])


def _vander(N, r, s, grad=False):
    a = np.where(np.abs(1 - s) > 1e-13, 2 * (1 + r) / np.where(np.abs(1 - s) > 1e-13, 1 - s, 1) - 1, -1.0)
    out, dr, ds = [], [], []
    for i in range(N + 1):
        for j in range(N + 1 - i):
            fa, gb = _jacobi(a, 0, 0, i), _jacobi(s, 2 * i + 1, 0, j)
            out.append(math.sqrt(2) * fa * gb * (1 - s) ** i)
            dfa, dgb = _djacobi(a, 0, 0, i), _djacobi(s, 2 * i + 1, 0, j)
            w = (0.5 * (1 - s)) ** (i - 1) if i > 0 else np.ones_like(s)
            d_r = dfa * gb * w
            t = dgb * (0.5 * (1 - s)) ** i
            if i > 0:
                t = t - 0.5 * i * gb * w
            d_s = dfa * gb * 0.5 * (1 + a) * w + fa * t
            dr.append(2 ** (i + 0.5) * d_r)
            ds.append(2 ** (i + 0.5) * d_s)
    return tuple(np.stack(m, 1) for m in ((out, dr, ds) if grad else (out,)))


@functools.lru_cache(maxsize=8)
def _element(N):
    """Warp-and-blend nodes and the operators on them, as numpy arrays."""
    alpha = [0, 0, 0, 1.4152, 0.1001, 0.2751, 0.98, 1.0999][N]
    lam = [(1 - i / N - j / N, j / N, i / N) for i in range(N + 1) for j in range(N + 1 - i)]
    l3, l1 = np.array([x[1] for x in lam]), np.array([x[2] for x in lam])
    l1, l2, l3 = l1, 1 - l1 - l3, l3  # l1: top vertex, l2: (-1,-1), l3: (1,-1)
    x, y = -l2 + l3, (2 * l1 - l2 - l3) / math.sqrt(3)
    gll, eq = _gll(N), np.linspace(-1, 1, N + 1)

    def warp(t):
        V = np.stack([_jacobi(eq, 0, 0, i) for i in range(N + 1)], 1)
        Pm = np.stack([_jacobi(t, 0, 0, i) for i in range(N + 1)], 1)
        w = Pm @ np.linalg.solve(V, gll - eq)
        inside = np.abs(t) < 1 - 1e-10
        return w / np.where(inside, 1 - t * t, 1) + w * (np.where(inside, 1, 0) - 1)

    w1 = 4 * l2 * l3 * warp(l3 - l2) * (1 + (alpha * l1) ** 2)
    w2 = 4 * l1 * l3 * warp(l1 - l3) * (1 + (alpha * l2) ** 2)
    w3 = 4 * l1 * l2 * warp(l2 - l1) * (1 + (alpha * l3) ** 2)
    x = x + w1 + math.cos(2 * math.pi / 3) * w2 + math.cos(4 * math.pi / 3) * w3
    y = y + math.sin(2 * math.pi / 3) * w2 + math.sin(4 * math.pi / 3) * w3
    L1, L2, L3 = (math.sqrt(3) * y + 1) / 3, (-3 * x - math.sqrt(3) * y + 2) / 6, (3 * x - math.sqrt(3) * y + 2) / 6
    r, s = -L2 + L3 - L1, -L2 - L3 + L1
    V, Vr, Vs = _vander(N, r, s, True)
    Vi = np.linalg.inv(V)
    M = Vi.T @ Vi
    with open(os.path.join(ROOT, "hopefoam_gb300", "data", "tri_cubature.txt")) as f:
        rows = [x for x in f.read().split("\n") if x and not x.startswith("#")]
    i = 0
    while True:
        _, strength, n = rows[i].split()
        if int(strength) == 3 * (N + 1):
            cub = np.array([[float(t) for t in x.split()] for x in rows[i + 1:i + 1 + int(n)]])
            break
        i += int(n) + 1
    G, Gr, Gs = (m @ Vi for m in _vander(N, cub[:, 0], cub[:, 1], True))
    fn = np.zeros((3, N + 1), np.int64)
    fn[0], fn[1, 0], fn[2, 0] = np.arange(N + 1), N, len(r) - 1
    for i in range(1, N + 1):
        fn[1, i], fn[2, i] = fn[1, i - 1] + N + 1 - i, fn[2, i - 1] - i - 1
    xg, wg = _gauss(N + 2)
    If = np.stack([_jacobi(xg, 0, 0, i) for i in range(N + 1)], 1) @ np.linalg.inv(
        np.stack([_jacobi(r[fn[0]], 0, 0, i) for i in range(N + 1)], 1))
    return dict(r=r, s=s, M=M, Mi=V @ V.T, G=G, Gr=Gr, Gs=Gs, w=cub[:, 2], Dr=Vr @ Vi, Ds=Vs @ Vi, fn=fn, If=If, wf=wg)


class _Geo:
    def __init__(self, mesh):
        v = _dev(mesh.VXY)
        xr, xs = (v[:, 1] - v[:, 0]) / 2, (v[:, 2] - v[:, 0]) / 2
        self.J = xr[:, 0] * xs[:, 1] - xr[:, 1] * xs[:, 0]
        self.rx, self.ry = xs[:, 1] / self.J, -xs[:, 0] / self.J
        self.sx, self.sy = -xr[:, 1] / self.J, xr[:, 0] / self.J
        e = torch.roll(v, -1, 1) - v  # edge f from vertex f to f + 1
        ln = e.norm(dim=2)
        self.nx, self.ny = e[:, :, 1] / ln, -e[:, :, 0] / ln
        self.sJ = ln / 2
        self.nb, self.nf = _dev(mesh.EToE).long(), _dev(mesh.EToF).long()
        self.inside = self.nb >= 0
        self.nb, self.nf = self.nb.clamp(min=0), self.nf.clamp(min=0)


def _prim(q):
    u, v = q[1] / q[0], q[2] / q[0]
    return u, v, (GAMMA - 1) * (q[3] - 0.5 * (q[1] * u + q[2] * v))


def _roe(nx, ny, a, b):
    """Roe flux through the face, states a (inside) and b (outside), in the face frame."""
    def frame(q):
        m, t = nx * q[1] + ny * q[2], nx * q[2] - ny * q[1]
        u, v = m / q[0], t / q[0]
        p = (GAMMA - 1) * (q[3] - 0.5 * (m * u + t * v))
        return q[0], u, v, p, (q[3] + p) / q[0], torch.stack([m, m * u + p, t * u, u * (q[3] + p)])
    ra, ua, va, pa, Ha, Fa = frame(a)
    rb, ub, vb, pb, Hb, Fb = frame(b)
    sa, sb = torch.sqrt(ra), torch.sqrt(rb)
    rho = sa * sb
    u, v, H = ((sa * x + sb * y) / (sa + sb) for x, y in ((ua, ub), (va, vb), (Ha, Hb)))
    c2 = (GAMMA - 1) * (H - 0.5 * (u * u + v * v))
    c = torch.sqrt(c2.abs())
    w1 = (-0.5 * rho * (ub - ua) / c + 0.5 * (pb - pa) / c2) * (u - c).abs()
    w2 = (rb - ra - (pb - pa) / c2) * u.abs()
    w3 = rho * (vb - va) * u.abs()
    w4 = (0.5 * rho * (ub - ua) / c + 0.5 * (pb - pa) / c2) * (u + c).abs()
    F = 0.5 * (Fa + Fb) - 0.5 * torch.stack([w1 + w2 + w4, w1 * (u - c) + w2 * u + w4 * (u + c), (w1 + w2 + w4) * v + w3,
                                             w1 * (H - u * c) + w2 * (u * u + v * v) / 2 + w3 * v + w4 * (H + u * c)])
    return torch.stack([F[0], nx * F[1] - ny * F[2], ny * F[1] + nx * F[2], F[3]])


def _euler_rhs(q, N, g, flux):
    E = _element(N)
    qg = q @ _dev(E["G"]).T
    u, v, p = _prim(qg)
    Fx = torch.stack([qg[1], qg[1] * u + p, qg[2] * u, (qg[3] + p) * u])
    Fy = torch.stack([qg[2], qg[1] * v, qg[2] * v + p, (qg[3] + p) * v])
    del u, v, p, qg
    Sr, Ss = (_dev(E["Mi"] @ (E[m] * E["w"][:, None]).T) for m in ("Gr", "Gs"))
    R = (g.rx[:, None] * Fx + g.ry[:, None] * Fy) @ Sr.T + (g.sx[:, None] * Fx + g.sy[:, None] * Fy) @ Ss.T
    del Fx, Fy
    If = _dev(E["If"])
    tr = q[:, :, _dev(E["fn"])] @ If.T  # (4, K, 3, Nfq), along each face
    a, b = tr, tr[:, g.nb, g.nf].flip(-1)
    nx, ny = g.nx[:, :, None], g.ny[:, :, None]
    if flux == "roe":
        F = _roe(nx, ny, a, b)
    else:
        def normal(w):
            u, v, p = _prim(w)
            un = nx * u + ny * v
            return torch.stack([w[0] * un, w[1] * un + nx * p, w[2] * un + ny * p, (w[3] + p) * un]), un.abs() + torch.sqrt(GAMMA * p / w[0])
        (Fa, la), (Fb, lb) = normal(a), normal(b)
        lam = torch.maximum(la, lb).amax(-1, keepdim=True)
        F = 0.5 * (Fa + Fb) + 0.5 * lam * (a - b)
    F = F * (g.sJ / g.J[:, None])[:, :, None] * _dev(E["wf"])
    for f in range(3):
        lift = E["Mi"][:, E["fn"][f]] @ E["If"].T
        R = R - F[:, :, f] @ _dev(lift).T
    return R


RK4A = [0.0, -567301805773.0 / 1357537059087.0, -2404267990393.0 / 2016746695238.0, -3550918686646.0 / 2091501179385.0, -1275806237668.0 / 842570457699.0]
RK4B = [1432997174477.0 / 9575080441755.0, 5161836677717.0 / 13612068292357.0, 1720146321549.0 / 2090206949498.0, 3134564353537.0 / 4481467310338.0, 2277821191437.0 / 14882151754819.0]


def _euler_step(q, dt, N, g, flux, scheme):
    if scheme == "ssprk2":
        q1 = q + dt * _euler_rhs(q, N, g, flux)
        return 0.5 * q + 0.5 * (q1 + dt * _euler_rhs(q1, N, g, flux))
    res = torch.zeros_like(q)
    for a, b in zip(RK4A, RK4B):
        res = a * res + dt * _euler_rhs(q, N, g, flux)
        q = q + b * res
    return q


def _sipg_solve(mesh, N, b, tau_coef, tol):
    """Block-Jacobi conjugate gradients on the interior-penalty Laplacian (homogeneous Dirichlet), in 64 bits."""
    E, g = _element(N), _Geo(mesh)
    W = E["w"][:, None]
    Srr, Sss = _dev(E["Gr"].T @ (W * E["Gr"])), _dev(E["Gs"].T @ (W * E["Gs"]))
    Srs = _dev(E["Gr"].T @ (W * E["Gs"]) + E["Gs"].T @ (W * E["Gr"]))
    Np = Srr.shape[0]
    T = np.zeros((3, N + 2, Np))
    for f in range(3):
        T[f][:, E["fn"][f]] = E["If"]
    Drf, Dsf, T = _dev(T @ E["Dr"]), _dev(T @ E["Ds"]), _dev(T)
    crr, css, crs = g.rx ** 2 + g.ry ** 2, g.sx ** 2 + g.sy ** 2, g.rx * g.sx + g.ry * g.sy
    ar = g.nx * g.rx[:, None] + g.ny * g.ry[:, None]
    as_ = g.nx * g.sx[:, None] + g.ny * g.sy[:, None]
    h = g.sJ / g.J[:, None]
    other = h[g.nb, g.nf]
    tau = tau_coef * (N + 1) ** 2 * torch.where(g.inside, torch.maximum(h, other), h)[:, :, None]
    wJ = g.sJ[:, :, None] * _dev(E["wf"])
    ins = g.inside[:, :, None]
    nf3, J1 = 3 * (N + 2), g.J[:, None]
    face = torch.cat([T.reshape(nf3, Np), Drf.reshape(nf3, Np), Dsf.reshape(nf3, Np)]).T.contiguous()
    vol = torch.cat([Srr, Srs, Sss]).T.contiguous()

    def apply(u):
        t = (u @ face).reshape(-1, 3, 3, N + 2)
        um, dm = t[:, 0], ar[:, :, None] * t[:, 1] + as_[:, :, None] * t[:, 2]
        up, dp = um[g.nb, g.nf].flip(-1), -dm[g.nb, g.nf].flip(-1)
        jump, dp = torch.where(ins, um - up, 2 * um), torch.where(ins, dp, dm)
        c1, c2 = wJ * (tau / 2 * jump - 0.5 * (dm + dp)), -0.5 * wJ * jump
        c = torch.cat([c1, c2 * ar[:, :, None], c2 * as_[:, :, None]], 1).reshape(-1, 3 * nf3)
        y = (u @ vol).reshape(-1, 3, Np)
        return J1 * (crr[:, None] * y[:, 0] + crs[:, None] * y[:, 1] + css[:, None] * y[:, 2]) + c @ face.T

    Dn = ar[:, :, None, None] * Drf + as_[:, :, None, None] * Dsf
    jm, sg = torch.where(ins, 1.0, 2.0)[..., None], torch.where(ins, 0.5, 1.0)[..., None]
    w4, t4 = wJ[..., None], tau[..., None]
    B = J1[:, :, None] * (crr[:, None, None] * Srr + crs[:, None, None] * Srs + css[:, None, None] * Sss)
    B = B + torch.einsum("fgi,kfgj->kij", T, w4 * (t4 / 2 * jm * T - sg * Dn)) + torch.einsum("kfgi,kfgj->kij", Dn, -0.5 * w4 * jm * T)
    P = torch.linalg.inv(B)
    del Dn, B
    x, r = torch.zeros_like(b), b.clone()
    z = torch.bmm(P, r[:, :, None])[:, :, 0]
    p, rz = z.clone(), (r * z).sum()
    stop = float(b.square().sum()) * tol * tol
    for it in range(30000):
        Ap = apply(p)
        al = rz / (p * Ap).sum()
        x += al * p
        if it % 50 == 49:
            r = b - apply(x)
            if float(r.square().sum()) <= stop:
                break
        else:
            r -= al * Ap
        z = torch.bmm(P, r[:, :, None])[:, :, 0]
        new = (r * z).sum()
        p = z + (new / rz) * p
        rz = new
    return x


def exact(case, seed):
    kind = case["kind"]
    if kind == "euler":
        E = _element(case["order"])
        mesh, q, dt = _euler_inputs(case, seed, E["r"], E["s"])
        return _euler_step(q, dt, case["order"], _Geo(mesh), case["flux"], case["scheme"])
    if kind == "batch":
        cases, out = _batch_list(case, seed), []
        for N in sorted({c["order"] for c in cases}):
            E, qs = _element(N), []
            for c in cases:
                if c["order"] != N:
                    continue
                mesh = periodic_square(c["m"], c["m"], BOX, BOX, perturb=0.1, seed=c["seed"])
                x, y = _coords(mesh, E["r"], E["s"])
                q = _dev(euler.isentropic_vortex(x.cpu().numpy(), y.cpu().numpy(), 0.0, beta=c["beta"], x0=BOX / 2,
                                                 y0=BOX / 2, uinf=c["mach"] * math.sqrt(GAMMA), gamma=GAMMA))
                qs.append(_euler_step(q, _cfl_dt(mesh, q, N, case["cfl"]), N, _Geo(mesh), "lf", "lserk4"))
            out.append(torch.cat(qs, 1))
        return out
    if kind == "poisson":
        E = _element(case["order"])
        mesh, b = _poisson_inputs(case, seed, E["r"], E["s"], E["M"])
        return _sipg_solve(mesh, case["order"], b, 1.0, 1e-12).reshape(-1)
    # the limited step and the projection step have no short closed form: None
    return None
