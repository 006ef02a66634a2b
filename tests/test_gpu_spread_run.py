"""The spreading and interpolation kernels on their own (plan.spread,
plan.interp) against the FP64 oracle, for every kernel support and at the sizes
where they can go wrong: oversampled grids down to 16 cells (windows that wrap
around the grid), numbers of points around a warp's batch, points on bin and
grid edges, a clustered set (one bin), and values that are not finite.

Tolerances: single precision, the Horner evaluation of degree D = W + 3 <= 11
and the product of the weights round at most 2 (2 D + 2) 2^-24 = 3e-6 relative
to the largest weights; double, the polynomial coefficients of planner and
oracle agree to about 1e-11.
"""
import numpy as np
import pytest

from ducc_b200 import nufft
from oracle import nufft_oracle as O

pytestmark = pytest.mark.gpu


def _force(W, single, nover, ndim):
    """(kernel row, oversampled shape) with support W."""
    for k, row in enumerate(O.kernel_db()):
        if row[0] == W and row[6] == single and row[5] == ndim:
            return k, nover
    pytest.skip("no kernel of this support")


def _coords(kind, M, nover, rng):
    ndim = len(nover)
    if kind == "uniform":
        return rng.uniform(-np.pi, np.pi, (M, ndim))
    if kind == "bin":      # all in a few cells
        return rng.uniform(0.3, 0.3 + 3 * 2 * np.pi / max(nover), (M, ndim))
    # cell edges, the first and the last cells of the period included
    n = np.array(nover)
    return rng.integers(-n, n, (M, ndim)) * (2 * np.pi / n)


def _case(W, single, shape, nover, M, kind, seed=1):
    rng = np.random.default_rng(seed)
    ct = np.float32 if single else np.float64
    coord = _coords(kind, M, nover, rng).astype(ct)
    vals = (rng.standard_normal(M) + 1j * rng.standard_normal(M)).astype(
        np.complex64 if single else np.complex128)
    k, nov = _force(W, single, nover, len(shape))
    p = O.Params(shape, 1e-3, single, M, True, force=(k, nov))
    return p, k, nov, coord, vals


GRIDS2 = [((5, 6), (16, 16)), ((9, 40), (18, 88)), ((30, 13), (64, 28)), ((50, 60), (110, 126))]


def _run(W, single, shape, nover, M, kind):
    import torch
    p, k, nov, coord, vals = _case(W, single, shape, nover, M, kind)
    plan = nufft.plan(nu2u=True, coord=torch.from_numpy(coord).cuda(), grid_shape=shape,
                      epsilon=1e-3, force_kernel=k, force_nover=nov, spreader="plain")
    got = plan.spread(points=torch.from_numpy(vals).cuda())
    tol = 3e-6 if single else 1e-10
    assert O.l2error(got.cpu().numpy(), O.spread(p, coord, vals)) < tol
    rng = np.random.default_rng(5)
    grid = (rng.standard_normal(nov) + 1j * rng.standard_normal(nov)).astype(vals.dtype)
    out = plan.interp(grid=torch.from_numpy(grid).cuda())
    assert O.l2error(out.cpu().numpy(), O.interpolate(p, grid, coord)) < tol


@pytest.mark.parametrize("W", range(4, 9))
@pytest.mark.parametrize("shape,nover", GRIDS2)
@pytest.mark.parametrize("M,kind", [(1, "uniform"), (33, "edges"), (300, "bin"), (2500, "uniform")])
def test_2d_single(W, shape, nover, M, kind):
    _run(W, True, shape, nover, M, kind)


@pytest.mark.parametrize("W", range(4, 17))
@pytest.mark.parametrize("shape,nover", GRIDS2)
@pytest.mark.parametrize("M,kind", [(1, "uniform"), (17, "edges"), (300, "bin"), (2500, "uniform")])
def test_2d_double(W, shape, nover, M, kind):
    _run(W, False, shape, nover, M, kind)


GRIDS3 = [((3, 4, 5), (16, 16, 16)), ((10, 5, 20), (22, 18, 44)), ((15, 20, 9), (36, 48, 20))]


@pytest.mark.parametrize("W", range(4, 9))
@pytest.mark.parametrize("shape,nover", GRIDS3)
@pytest.mark.parametrize("M,kind", [(1, "uniform"), (129, "edges"), (300, "bin"), (1500, "uniform")])
def test_3d_single(W, shape, nover, M, kind):
    _run(W, True, shape, nover, M, kind)


@pytest.mark.parametrize("W", range(4, 17))
@pytest.mark.parametrize("shape,nover", GRIDS3)
@pytest.mark.parametrize("M,kind", [(1, "uniform"), (65, "edges"), (300, "bin"), (900, "uniform")])
def test_3d_double(W, shape, nover, M, kind):
    _run(W, False, shape, nover, M, kind)


@pytest.mark.parametrize("single", [True, False])
@pytest.mark.parametrize("shape,nover", [((50, 60), (110, 126)), ((15, 20, 9), (36, 48, 20))])
def test_nonfinite_value_stays_in_its_footprint(single, shape, nover):
    import torch
    W = 6
    p, k, nov, coord, vals = _case(W, single, shape, nover, 200, "uniform")
    vals[77] = np.inf
    plan = nufft.plan(nu2u=True, coord=torch.from_numpy(coord).cuda(), grid_shape=shape,
                      epsilon=1e-3, force_kernel=k, force_nover=nov, spreader="plain")
    got = plan.spread(points=torch.from_numpy(vals).cuda()).cpu().numpy()
    i0, _ = O.getpix(p, coord[77:78])
    bad = np.zeros(nov, bool)
    bad[np.ix_(*[(i0[0, d] + np.arange(W)) % nov[d] for d in range(len(nov))])] = True
    assert np.array_equal(~np.isfinite(got), bad)
    vals[77] = 0
    ref = O.spread(p, coord, vals)
    assert O.l2error(got[~bad], ref[~bad]) < (3e-6 if single else 1e-10)


@pytest.mark.parametrize("single,W,shape,nover", [(False, 6, (50, 60), (110, 126)),
                                                  (False, 6, (15, 20, 9), (36, 48, 20)),
                                                  (True, 6, (15, 20, 9), (36, 48, 20)),
                                                  (True, 8, (15, 20, 9), (36, 48, 20))])
def test_nonfinite_cell_reaches_its_points_only(single, W, shape, nover):
    import torch
    p, k, nov, coord, vals = _case(W, single, shape, nover, 400, "uniform")
    plan = nufft.plan(nu2u=True, coord=torch.from_numpy(coord).cuda(), grid_shape=shape,
                      epsilon=1e-3, force_kernel=k, force_nover=nov)
    rng = np.random.default_rng(6)
    grid = (rng.standard_normal(nov) + 1j * rng.standard_normal(nov)).astype(vals.dtype)
    ref = O.interpolate(p, grid, coord)
    cell = tuple(n // 3 for n in nov)
    grid[cell] = np.nan
    got = plan.interp(grid=torch.from_numpy(grid).cuda()).cpu().numpy()
    i0, _ = O.getpix(p, coord)
    hit = np.all((np.array(cell) - i0) % np.array(nov) < W, axis=1)
    assert 0 < hit.sum() < 400 and np.array_equal(~np.isfinite(got), hit)
    assert O.l2error(got[~hit], ref[~hit]) < (3e-6 if single else 1e-10)


@pytest.mark.parametrize("ndim", [2, 3])
@pytest.mark.parametrize("single,W", [(True, w) for w in range(4, 9)] +
                         [(False, w) for w in range(4, 17)])
def test_smallest_grids(single, W, ndim):
    """Oversampled axes of 2 nsafe cells, the shortest that are accepted: the
    windows go around them more than once."""
    n = 2 * ((W + 1) // 2)
    _run(W, single, (2, 3, 2)[:ndim], (n, n, n + 2 if n + 2 != 14 else n)[:ndim], 200, "edges")
    _run(W, single, (2, 3, 2)[:ndim], (n,) * ndim, 200, "uniform")


@pytest.mark.parametrize("W,nover,M", [(8, (36, 48, 20), 4500), (9, (36, 48, 20), 4500),
                                       (10, (20, 40, 36), 4500), (11, (30, 40, 36), 45000),
                                       (11, (110, 120, 126), 17000), (12, (126, 120, 128), 17000),
                                       (13, (72, 70, 80), 17000), (14, (72, 70, 80), 17000),
                                       (15, (90, 88, 80), 17000)])
def test_3d_double_direct(W, nover, M):
    """3D double-precision interpolation cell by cell (few points per bin, small
    supports, and W = 11 with many points per bin)."""
    _run(W, False, tuple(n // 2 - 3 for n in nover), nover, M, "uniform")
    if M < 5000:
        _run(W, False, tuple(n // 2 - 3 for n in nover), nover, M, "edges")


@pytest.mark.parametrize("single,shape,M", [(True, (20, 24, 18), 3000), (True, (500,), 3000),
                                            (False, (20, 24, 18), 3000),
                                            (False, (20, 24, 18), 6000), (False, (40, 36), 3000)])
@pytest.mark.parametrize("eps", [1e-2, 1e-5])
def test_strided_unplanned(single, shape, M, eps):
    """Unplanned calls read unsorted coordinates through their strides; values and
    results may be strided as well."""
    import torch
    rng = np.random.default_rng(8)
    ct = torch.complex64 if single else torch.complex128
    nd = len(shape)
    coord = rng.uniform(-np.pi, np.pi, (M, nd)).astype(np.float32 if single else np.float64)
    vals = torch.from_numpy(rng.standard_normal((M, 2))).cuda().to(ct) + 1j
    grid = torch.from_numpy(rng.standard_normal(shape)).cuda().to(ct) + 1j
    c = torch.from_numpy(coord).cuda()
    cs = torch.from_numpy(np.ascontiguousarray(coord.T)).cuda().T[:, :]
    assert nd == 1 or not cs.is_contiguous()
    kw = dict(forward=True, epsilon=eps)
    ref = nufft.u2nu(grid=grid, coord=c, **kw)
    out = torch.zeros((M, 3), dtype=ct, device="cuda")
    nufft.u2nu(grid=grid, coord=cs, out=out[:, 1], **kw)
    assert torch.equal(out[:, 1], ref) and not out[:, ::2].any()
    u0 = nufft.nu2u(points=vals[:, 0].contiguous(), coord=c,
                    out=torch.empty(shape, dtype=ct, device="cuda"), **kw)
    u1 = nufft.nu2u(points=vals[:, 0], coord=cs,
                    out=torch.empty(shape, dtype=ct, device="cuda"), **kw)
    # (sums in another order)
    assert torch.linalg.vector_norm(u1 - u0) <= 2 * eps * torch.linalg.vector_norm(u0)


@pytest.mark.parametrize("kind", ["uniform", "bin"])
@pytest.mark.parametrize("W", range(4, 17))
@pytest.mark.parametrize("single", [True, False])
def test_1d(single, W, kind):
    """1D: several points at a time (single precision, spread points) and one."""
    if single and W > 8:
        pytest.skip("no kernel of this support")
    for M in (1, 70, 3000):
        _run(W, single, (400,), (900,), M, kind)


@pytest.mark.parametrize("shape,nover,W", [((400,), (900,), 7), ((3000,), (6480,), 5),
                                           ((30, 40), (64, 90), 6)])
def test_many_chunks_of_one_tile(shape, nover, W):
    """Most points in one tile (some fifty chunks) and a few all over the grid."""
    import torch
    rng = np.random.default_rng(9)
    M = 50000
    coord = np.where(rng.random((M, 1)) < 0.99, rng.uniform(0.1, 0.12, (M, len(shape))),
                     rng.uniform(-np.pi, np.pi, (M, len(shape)))).astype(np.float32)
    p, k, nov, _, vals = _case(W, True, shape, nover, M, "uniform")
    plan = nufft.plan(nu2u=True, coord=torch.from_numpy(coord).cuda(), grid_shape=shape,
                      epsilon=1e-3, force_kernel=k, force_nover=nov)
    grid = (rng.standard_normal(nov) + 1j * rng.standard_normal(nov)).astype(np.complex64)
    out = plan.interp(grid=torch.from_numpy(grid).cuda()).cpu().numpy()
    assert O.l2error(out, O.interpolate(p, grid, coord)) < 3e-6
    got = plan.spread(points=torch.from_numpy(vals).cuda()).cpu().numpy()
    # 5e4 values of size 1 summed in one order or another in a few cells
    assert O.l2error(got, O.spread(p, coord, vals)) < 3e-6 + 50000 ** 0.5 * 2 ** -23
