"""Block-Jacobi PCG with the multilevel coarse-space correction
(DG_PC_MULTILEVEL) on the SIPG pressure operator, through the C ABI:
same solution as block Jacobi (both to rtol 1e-10: the solutions agree to
1e-8 relative), iteration counts that do not grow with the mesh, both
arithmetic modes, and the mixed boundary types / Helmholtz form of the
incompressible step."""
import numpy as np
import pytest

from conftest import rel_l2

pytestmark = pytest.mark.gpu


def _solver(n_interior, N, tau):
    from hopefoam_gb300.mesh import delaunay_square
    from hopefoam_gb300.poisson import PressureSolver, poisson_rhs

    m = delaunay_square(n_interior, seed=1)
    ps = PressureSolver(m, N, tau_coef=tau)
    b, _ = poisson_rhs(m, N, seed=3)
    return ps, b


@pytest.mark.parametrize("N,tau", [(4, 1.0), (2, 20.0), (7, 1.0)])
def test_multilevel_matches_block_jacobi(gpu_lib, N, tau):
    from hopefoam_gb300 import _lib as L

    ps, b = _solver(3000, N, tau)
    x_bj, st_bj = ps.solve(b, rtol=1e-10, pc=L.DG_PC_BLOCK_JACOBI, precision=L.DG_PREC_FP64)
    x_mg, st_mg = ps.solve(b, rtol=1e-10, pc=L.DG_PC_MULTILEVEL, precision=L.DG_PREC_FP64)
    x_mx, st_mx = ps.solve(b, rtol=1e-10, pc=L.DG_PC_MULTILEVEL, precision=L.DG_PREC_SPLIT)
    print("N=%d tau=%g K=%d: block Jacobi %d its %.1f ms, multilevel %d its %.1f ms (mixed %d its %.1f ms)" %
          (N, tau, ps.mesh.K if hasattr(ps, "mesh") else -1, st_bj["iterations"], st_bj["ms"], st_mg["iterations"],
           st_mg["ms"], st_mx["iterations"], st_mx["ms"]))
    assert st_mg["rel_residual"] <= 1e-10 and st_mx["rel_residual"] <= 1e-10
    assert rel_l2(x_mg, x_bj) < 1e-8 and rel_l2(x_mx, x_bj) < 1e-8
    assert st_mg["iterations"] * 4 < st_bj["iterations"]


def test_multilevel_iterations_do_not_grow(gpu_lib):
    from hopefoam_gb300 import _lib as L

    its = []
    for n in (2000, 8000, 32000):
        ps, b = _solver(n, 4, 1.0)
        _, st = ps.solve(b, rtol=1e-10, pc=L.DG_PC_MULTILEVEL, precision=L.DG_PREC_FP64)
        its.append(st["iterations"])
    print("multilevel iterations at 2k / 8k / 32k interior points:", its)
    assert max(its) < 1.6 * min(its)


def _cycle(A, r, omega=0.6, coarsest=500):
    """One V(1,1) cycle as mg.hpp defines it, on scipy matrices."""
    import scipy.sparse as sp

    n = A.shape[0]
    if n <= coarsest:
        return np.linalg.solve(A.toarray(), r)
    agg = -np.ones(n, np.int64)
    na = 0
    for i in range(n):
        if agg[i] >= 0:
            continue
        agg[i] = na
        nb = A.indices[A.indptr[i]:A.indptr[i + 1]]
        agg[nb[agg[nb] < 0]] = na
        na += 1
    P = sp.csr_matrix((np.ones(n), (np.arange(n), agg)), shape=(n, na))
    d = omega / A.diagonal()
    x = d * r
    x = x + P @ _cycle((P.T @ A @ P).tocsr(), P.T @ (r - A @ x), omega, coarsest)
    return x + d * (r - A @ x)


@pytest.mark.parametrize("n_interior", [4, 60, 300, 450, 1200, 3000, 12000])
def test_one_application_against_its_definition(gpu_lib, n_interior):
    """z = B r + P V(P^T r) of the first iteration (its solution is a multiple of z) against the cycle written out
    level by level: only the dense inverse (20, 96 and some 300 unknowns: part of a block, whole blocks, a remainder);
    the cycle as one dense matrix; one and two sparse levels above it.
    Tolerance: round-off (1e-15) times the condition number of the P1 operator (about 1e5 at 12000 vertices), with a
    factor of 100 for the differently formed coarse operators."""
    import scipy.sparse as sp

    from hopefoam_gb300 import _lib as L
    from hopefoam_gb300.euler import reference_operators
    from hopefoam_gb300.mesh import delaunay_square, load_cubature
    from hopefoam_gb300.poisson import PressureSolver, poisson_rhs
    from oracle.oracle import Oracle

    N = 2
    m = delaunay_square(n_interior, seed=1)
    ps = PressureSolver(m, N, tau_coef=1.0)
    b, _ = poisson_rhs(m, N, seed=3)
    x, st = ps.solve(b, rtol=1e-14, maxit=1, pc=L.DG_PC_MULTILEVEL, precision=L.DG_PREC_FP64, raise_on_fail=False)
    assert st["status"] == L.DG_ERR_NOT_CONVERGED and st["iterations"] == 1
    ops = reference_operators(N)
    orc = Oracle(m, N, load_cubature(3 * (N + 1)))
    diag, off, _ = orc.ipdg_blocks(tau_coef=1.0)
    K, Np = m.K, ps.Np
    lam = np.stack([-(ops["r"] + ops["s"]) / 2, (1 + ops["r"]) / 2, (1 + ops["s"]) / 2], 1)
    rows = np.repeat(np.arange(K * Np), 3)
    nv = int(m.EToV.max()) + 1
    P = sp.csr_matrix((np.tile(lam, (K, 1)).reshape(-1), (rows, np.repeat(m.EToV, Np, axis=0).reshape(-1))), shape=(K * Np, nv))
    i, j = np.meshgrid(np.arange(Np), np.arange(Np), indexing="ij")
    k = np.arange(K)
    blocks = [(k, k, -diag)] + [(k[m.EToE[:, f] >= 0], m.EToE[m.EToE[:, f] >= 0, f], -off[m.EToE[:, f] >= 0, f])
                                for f in range(3)]
    S = sum(sp.csr_matrix((v.reshape(-1), ((kr[:, None, None] * Np + i).reshape(-1), (kc[:, None, None] * Np + j).reshape(-1))),
                          shape=(K * Np, K * Np)) for kr, kc, v in blocks)
    pattern = sp.csr_matrix((np.ones(9 * K), (np.repeat(m.EToV, 3, axis=1).reshape(-1), np.tile(m.EToV, (1, 3)).reshape(-1))),
                            shape=(nv, nv))
    A1 = (P.T @ S @ P).multiply(pattern > 0).tocsr()
    A1.sort_indices()
    z = np.linalg.solve(-diag, b.reshape(K, Np, 1)).reshape(-1) + P @ _cycle(A1, P.T @ b)
    alpha = (b @ z) / (z @ (S @ z))
    assert rel_l2(x, alpha * z) < 1e-8


@pytest.mark.parametrize("N", [1, 3, 5, 6])
def test_every_order_matches_block_jacobi(gpu_lib, N):
    """The orders that test_multilevel_matches_block_jacobi leaves out (every order has its own layout of elements in
    warps), with sparse levels above the dense one, both arithmetic modes: both solves to 1e-10, the solutions agree
    to 1e-8 as there."""
    from hopefoam_gb300 import _lib as L

    ps, b = _solver(3000, N, 1.0)
    x_bj, _ = ps.solve(b, rtol=1e-10, pc=L.DG_PC_BLOCK_JACOBI, precision=L.DG_PREC_FP64)
    for precision in (L.DG_PREC_FP64, L.DG_PREC_SPLIT):
        x, st = ps.solve(b, rtol=1e-10, pc=L.DG_PC_MULTILEVEL, precision=precision)
        assert st["rel_residual"] <= 1e-10 and rel_l2(x, x_bj) < 1e-8


@pytest.mark.parametrize("N,n_interior", [(2, 3000), (4, 12000)])
def test_repeated_solves_follow_the_operator(gpu_lib, N, n_interior):
    """Solves that alternate arithmetic, preconditioner and Helmholtz coefficient on one solver, the batches of
    iterations kept between them, against one solver per solve: the same launches in the same order, so the same bits."""
    from hopefoam_gb300 import _lib as L

    ps, b = _solver(n_interior, N, 1.0)
    ml, bj = L.DG_PC_MULTILEVEL, L.DG_PC_BLOCK_JACOBI
    seq = [(0.0, ml, 1), (0.0, ml, 1), (0.0, ml, 0), (50.0, ml, 1), (50.0, bj, 1), (50.0, ml, 1), (0.0, ml, 1), (50.0, ml, 0)]
    fresh = {}
    for mass, pc, precision in seq:
        assert ps.ctx.lib.dg_ipdg_set_mass(ps.ctx.h, mass) == L.DG_OK
        x, _ = ps.solve(b, rtol=1e-10, pc=pc, precision=precision)
        if (mass, pc, precision) not in fresh:
            p2, _ = _solver(n_interior, N, 1.0)
            assert p2.ctx.lib.dg_ipdg_set_mass(p2.ctx.h, mass) == L.DG_OK
            fresh[mass, pc, precision] = p2.solve(b, rtol=1e-10, pc=pc, precision=precision)[0]
            p2.ctx.close()
        assert np.array_equal(x, fresh[mass, pc, precision])


@pytest.mark.parametrize("N,n_interior,precision", [(3, 300, 0), (3, 300, 1), (2, 3000, 0), (4, 6000, 1)])
def test_boundary_types_change_between_solves(gpu_lib, N, n_interior, precision):
    """Boundary types and the Helmholtz coefficient changed after solves, when the assembled rows, the levels and a batch of
    iterations are kept already (small problems in one launch, larger ones in batches): the bits of a fresh solver."""
    from hopefoam_gb300 import _lib as L

    ps, b = _solver(n_interior, N, 1.0)
    nb = ps.ctx.n_bfaces
    types = [np.zeros(nb, np.int32), (np.arange(nb) % 3 == 0).astype(np.int32), np.where(np.arange(nb) % 2, 2, 0).astype(np.int32)]

    def prepare(p, t, mass):
        assert p.ctx.lib.dg_ipdg_set_boundary_types(p.ctx.h, L.iptr(types[t])) == L.DG_OK
        assert p.ctx.lib.dg_ipdg_set_mass(p.ctx.h, mass) == L.DG_OK

    for t, mass, pc in ((0, 0.0, "MULTILEVEL"), (1, 0.0, "MULTILEVEL"), (1, 20.0, "BLOCK_JACOBI"), (2, 20.0, "MULTILEVEL"),
                        (0, 0.0, "BLOCK_JACOBI"), (0, 0.0, "MULTILEVEL")):
        prepare(ps, t, mass)
        kw = dict(rtol=1e-8, maxit=20000, pc=getattr(L, "DG_PC_" + pc), precision=precision)
        x, st = ps.solve(b, **kw)
        fresh, _ = _solver(n_interior, N, 1.0)
        prepare(fresh, t, mass)
        y, st2 = fresh.solve(b, **kw)
        fresh.ctx.close()
        assert st["iterations"] == st2["iterations"] and np.array_equal(x, y), (t, mass, pc)
    ps.ctx.close()
