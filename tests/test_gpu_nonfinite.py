"""Coordinates that are not finite: the other points' results stay what they
are, the point's own results and a type-1 output are not finite, and the next
call is not affected.  (That every cell such a point touches lies on the grid is
shown on the host, in test_fold_cpu.py.)"""
import numpy as np
import pytest

from ducc_b200 import nufft

pytestmark = pytest.mark.gpu

SHAPES = [(2500,), (128, 144), (5, 6), (40, 44, 48)]
BAD = (0, 17, 1000, 1001, 2999)


def _inputs(shape, single, seed=3):
    import torch
    rng = np.random.default_rng(seed)
    M, rt = 3000, (np.float32 if single else np.float64)
    ct = np.complex64 if single else np.complex128
    coord = rng.uniform(-np.pi, np.pi, (M, len(shape))).astype(rt)
    for k, j in enumerate(BAD):
        coord[j] = 0
    broken = coord.copy()
    for k, j in enumerate(BAD):
        broken[j, k % len(shape)] = (np.nan, np.inf, -np.inf)[k % 3]
    broken[BAD[0]] = np.nan
    vals = (rng.standard_normal(M) + 1j * rng.standard_normal(M)).astype(ct)
    grid = (rng.standard_normal(shape) + 1j * rng.standard_normal(shape)).astype(ct)
    good = np.ones(M, bool)
    good[list(BAD)] = False
    return [torch.from_numpy(x).cuda() for x in (coord, broken, vals, grid)] + [good]


def _eps(single):
    return 1e-5 if single else 1e-9


def _close(a, b, single):
    # both within epsilon of the exact transform; a point in the wrong place
    # would show as 1 / sqrt(3000)
    a, b = a.cpu().numpy(), b.cpu().numpy()
    return np.linalg.norm(a - b) <= 2 * _eps(single) * np.linalg.norm(b)


@pytest.mark.parametrize("single", [True, False])
@pytest.mark.parametrize("shape", SHAPES)
@pytest.mark.parametrize("planned", [False, True])
def test_type2_and_type1(shape, single, planned):
    import torch
    coord, broken, vals, grid, good = _inputs(shape, single)
    eps = _eps(single)

    def both(c):
        out = torch.empty(shape, dtype=vals.dtype, device="cuda")
        if planned:
            p = nufft.plan(nu2u=True, coord=c, grid_shape=shape, epsilon=eps)
            return (p.u2nu(grid=grid, forward=True), p.nu2u(points=vals, forward=True, out=out),
                    p.u2nu_dcoord(grid=grid, weights=vals, forward=True))
        return (nufft.u2nu(grid=grid, coord=c, forward=True, epsilon=eps),
                nufft.nu2u(points=vals, coord=c, forward=True, epsilon=eps, out=out),
                nufft.u2nu_dcoord(grid=grid, coord=c, weights=vals, forward=True, epsilon=eps))

    ref = both(coord)
    got = both(broken)
    assert not torch.isfinite(got[0][~good]).any() and torch.isfinite(got[0][good]).all()
    assert _close(got[0][good], ref[0][good], single)
    assert not torch.isfinite(got[1]).any()
    assert torch.isfinite(got[2][good]).all() and _close(got[2][good], ref[2][good], single)
    again = both(coord)
    assert all(_close(a, b, single) for a, b in zip(again, ref))


def test_tensor_core_spreader():
    import torch
    shape = (128, 144)
    coord, broken, vals, _, _ = _inputs(shape, True)
    res = []
    for c in (coord, broken, coord):
        out = torch.empty(shape, dtype=vals.dtype, device="cuda")
        res.append(nufft.plan(nu2u=True, coord=c, grid_shape=shape, epsilon=1e-5, spreader="tc")
                   .nu2u(points=vals, forward=True, out=out))
    assert not torch.isfinite(res[1]).any() and _close(res[2], res[0], True)


@pytest.mark.parametrize("single", [True, False])
def test_batch(single):
    import torch
    from ducc_b200 import batch
    shape = (128, 144)
    coord, broken, vals, grid, good = _inputs(shape, single)
    eps = _eps(single)
    out = []
    for c in (coord, broken):
        p = [nufft.plan(nu2u=True, coord=x, grid_shape=shape, epsilon=eps) for x in (coord, c)]
        b = batch.Batch(p)
        uni = [torch.empty(shape, dtype=vals.dtype, device="cuda") for _ in p]
        pts = [torch.empty_like(vals) for _ in p]
        b.nu2u(points=[vals, vals], out=uni, forward=True)
        b.u2nu(grids=[grid, grid], out=pts, forward=True)
        out.append((uni, pts))
    (u0, p0), (u1, p1) = out
    assert _close(u1[0], u0[0], single) and not torch.isfinite(u1[1]).any()
    assert _close(p1[0], p0[0], single) and _close(p1[1][good], p0[1][good], single)
    assert not torch.isfinite(p1[1][~good]).any()
