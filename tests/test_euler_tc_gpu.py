"""FP64 Euler stage on the tensor cores (euler_fp64_tc.cu) where its tiles and
routes change, against the CPU oracle.  Tolerance as for every FP64 right-hand
side: 1e-11 relative L2 (or ten times the oracle's one-ulp sensitivity); an
element taken by the plain FP64 route is held to the same."""
import numpy as np
import pytest

from conftest import rel_l2
from test_euler_gpu import TOL_RHS, _setup, _vertex_ulp_sensitivity

pytestmark = pytest.mark.gpu


def _state(x, y, L):
    k = 2 * np.pi / L
    rho = 1 + 0.2 * np.sin(k * x) * np.cos(k * y)
    u, v = 0.6 + 0.3 * np.cos(k * y), -0.2 + 0.4 * np.sin(k * x)
    p = 1 + 0.1 * np.cos(k * (x + y))
    return np.stack([rho, rho * u, rho * v, p / 0.4 + 0.5 * rho * (u * u + v * v)])


def _against_oracle(ctx, orc, m, N, q, flux):
    ctx.upload(q)
    g = ctx.rhs(flux=flux)
    r = orc.euler_rhs(q.reshape(-1), flux=flux).reshape(g.shape)
    assert rel_l2(g, r) < max(TOL_RHS, 10 * _vertex_ulp_sensitivity(m, N, q, flux, r))
    return g


@pytest.mark.parametrize("N,nx,ny", [(1, 4, 4), (2, 3, 5), (3, 11, 3), (4, 4, 12), (5, 3, 3), (6, 4, 4), (7, 5, 7),
                                     (1, 49, 51), (3, 50, 49)])
@pytest.mark.parametrize("flux", [0, 1])
def test_tile_edges(gpu_lib, N, nx, ny, flux):
    """K = 32 n, 32 n - 2, 32 n + 2 and less than a tile; with more tiles than SMs (K = 4900, 4998) too."""
    from hopefoam_gb300.mesh import periodic_square

    m = periodic_square(nx, ny, 10.0, 10.0, perturb=0.1, seed=N)
    ctx, orc, x, y = _setup(m, N)
    _against_oracle(ctx, orc, m, N, _state(x, y, 10.0), flux)
    ctx.close()


@pytest.mark.parametrize("N", [1, 3, 5, 7])
@pytest.mark.parametrize("flux", [0, 1])
def test_plain_route(gpu_lib, N, flux):
    """Elements outside the digit range (a density dip between nodes that no nodal bound foresees, values beyond the
    FP32 exponents, not finite) take the plain FP64 route, and no other element's result changes."""
    from hopefoam_gb300.mesh import periodic_square

    m = periodic_square(6, 6, 10.0, 10.0, perturb=0.1, seed=N)
    ctx, orc, x, y = _setup(m, N)
    q = _state(x, y, 10.0)
    base = _against_oracle(ctx, orc, m, N, q, flux)
    touched = lambda k: np.unique(np.r_[k, m.EToE[k]])
    # near-vacuum at one node: the interpolated density nearly vanishes or changes sign at some points
    dip = q.copy()
    dip[0, 40, 1] = 1e-3
    ctx.upload(dip)
    g = ctx.rhs(flux=flux)
    r = orc.euler_rhs(dip.reshape(-1), flux=flux).reshape(g.shape)
    ok = np.isfinite(r).all((0, 2))
    assert np.array_equal(np.isfinite(g).all((0, 2)), ok)
    rest = np.setdiff1d(np.arange(m.K), touched(40))
    assert np.array_equal(g[:, rest], base[:, rest])
    # one element and its neighbours 2^150 larger (outside FP32): values scale with it
    big = q.copy()
    big[:, 10] *= 2.0 ** 150
    ctx.upload(big)
    g = ctx.rhs(flux=flux)
    r = orc.euler_rhs(big.reshape(-1), flux=flux).reshape(g.shape)
    near = touched(10)
    assert rel_l2(g[:, near], r[:, near]) < 1e-10
    rest = np.setdiff1d(np.arange(m.K), near)
    assert np.array_equal(g[:, rest], base[:, rest])
    # the stage update of such elements: q + dt R
    from hopefoam_gb300 import _lib as L

    dt = 1e-4
    ctx.upload(big)
    assert ctx.lib.dg_forward_euler_stage(ctx.h, dt, flux, L.DG_PREC_FP64) == L.DG_OK
    s = ctx.download()
    assert rel_l2(s[:, near], big[:, near] + dt * r[:, near]) < 1e-12
    assert rel_l2(s[:, rest], q[:, rest] + dt * base[:, rest]) < 1e-15
    for bad in (np.nan, np.inf):
        w = q.copy()
        w[3, 20, 0] = bad
        ctx.upload(w)
        g = ctx.rhs(flux=flux)
        assert not np.isfinite(g[:, 20]).all()
        rest = np.setdiff1d(np.arange(m.K), touched(20))
        assert np.array_equal(g[:, rest], base[:, rest])
    ctx.close()


@pytest.mark.parametrize("N,nx,ny", [(2, 19, 16), (4, 61, 5), (1, 33, 18), (3, 37, 22), (5, 46, 20)])
def test_tiles_of_fewer_groups(gpu_lib, N, nx, ny):
    """K = 608, 610, 1188, 1628, 1840: on 152 SMs tiles of 1, 2, 2, 3 and 4 groups of 8 elements, with whole and
    ragged last tiles.  The last element once more with values that leave it and its neighbours to the plain route."""
    from hopefoam_gb300.mesh import periodic_square

    m = periodic_square(nx, ny, 10.0, 10.0, perturb=0.1, seed=N)
    ctx, orc, x, y = _setup(m, N)
    q = _state(x, y, 10.0)
    base = _against_oracle(ctx, orc, m, N, q, N % 2)
    big = q.copy()
    big[:, -1] *= 2.0 ** 150
    near = np.unique(np.r_[m.K - 1, m.EToE[-1]])
    ctx.upload(big)
    g = ctx.rhs(flux=N % 2)
    r = orc.euler_rhs(big.reshape(-1), flux=N % 2).reshape(g.shape)
    assert rel_l2(g[:, near], r[:, near]) < 1e-10
    rest = np.setdiff1d(np.arange(m.K), near)
    assert np.array_equal(g[:, rest], base[:, rest])
    ctx.close()


@pytest.mark.parametrize("N,nx,ny", [(1, 3, 3), (2, 5, 5), (3, 3, 7), (4, 3, 11), (1, 35, 35), (1, 49, 50), (2, 71, 70)])
@pytest.mark.parametrize("flux", [0, 1])
def test_route_changes_between_launches(gpu_lib, N, nx, ny, flux):
    """Elements that take the plain route in one launch and not in the next, on contexts whose flags no launch has written
    yet and over many launches: one to three tiles per block, last groups of two and four elements (K = 18, 50, 42, 66, 2450,
    4900, 9940), where three of a group's four warps have little or nothing to update.  Each launch gives the bits that
    its state has on a context of its own; the scaled state against the oracle as in test_plain_route."""
    from hopefoam_gb300.mesh import periodic_square

    m = periodic_square(nx, ny, 10.0, 10.0, perturb=0.1, seed=N)
    ctx, orc, x, y = _setup(m, N)
    q = _state(x, y, 10.0)
    big = q.copy()
    big[:, -1] *= 2.0 ** 150  # the last element: with its neighbours beyond the FP32 exponents
    every = q * 2.0 ** 150
    want = []
    for w in (q, big, every):
        c, _, _, _ = _setup(m, N)
        c.upload(w)
        want.append(c.rhs(flux=flux))
        c.close()
    for j in (1, 0, 2, 0, 1, 2, 1) * 4:
        ctx.upload((q, big, every)[j])
        assert np.array_equal(ctx.rhs(flux=flux), want[j])
    r = orc.euler_rhs(every.reshape(-1), flux=flux).reshape(want[2].shape)
    assert rel_l2(want[2], r) < 1e-10
    ctx.close()


@pytest.mark.parametrize("N", range(1, 8))
@pytest.mark.parametrize("element_dt", [False, True])
def test_steps_of_plain_route_elements(gpu_lib, N, element_dt):
    """LSERK4 and SSP-RK2 steps, with one step size and with one per element, where some elements take the plain route
    (a density 100 times lower at one end) and the others do not: against
    the same updates written out with the right-hand sides of the library.  Only round-off of the updates differs (ten
    stages, each a few units in the last place of the state, and of the step folded into the metrics): 1e-14 of the state's norm."""
    from hopefoam_gb300 import _lib as L
    from hopefoam_gb300.mesh import periodic_square
    from oracle.oracle import lserk4_coeffs

    m = periodic_square(5, 7, 10.0, 10.0, perturb=0.1, seed=N)
    ctx, orc, x, y = _setup(m, N)
    q = _state(x, y, 10.0)
    near = np.array([0, 9, 33, 50, 51, 69])
    rest = np.setdiff1d(np.arange(m.K), near)
    for k in near:
        t = (x[k] - x[k].min()) / (x[k].max() - x[k].min())
        u, v = q[1, k] / q[0, k], q[2, k] / q[0, k]
        q[0, k] = 1 + 99 * t
        q[1, k], q[2, k], q[3, k] = q[0, k] * u, q[0, k] * v, 60 + 0.5 * q[0, k] * (u * u + v * v)
    factor = np.random.default_rng(N).uniform(0.5, 1.5, m.K) if element_dt else np.ones(m.K)
    assert ctx.lib.dg_set_element_dt(ctx.h, L.dptr(factor) if element_dt else None) == L.DG_OK
    dt = 1e-4
    step = dt * factor[None, :, None]

    def rhs(w):
        ctx.upload(w)
        return ctx.rhs(flux=N % 2)

    w, res = q.copy(), np.zeros_like(q)
    a, b = lserk4_coeffs()[:2]
    for _ in range(2):
        for ai, bi in zip(a, b):
            res = ai * res + step * rhs(w)
            w = w + bi * res
    ctx.upload(q)
    ctx.lserk4(dt, 2, flux=N % 2)
    g = ctx.download()
    assert rel_l2(g[:, near], w[:, near]) < 1e-14 and rel_l2(g[:, rest], w[:, rest]) < 1e-14
    w = q.copy()
    for _ in range(2):
        w1 = w + step * rhs(w)
        w = 0.5 * (w + (w1 + step * rhs(w1)))
    ctx.upload(q)
    ctx.ssprk2(dt, 2, flux=N % 2)
    g = ctx.download()
    assert rel_l2(g[:, near], w[:, near]) < 1e-14 and rel_l2(g[:, rest], w[:, rest]) < 1e-14
    ctx.close()
