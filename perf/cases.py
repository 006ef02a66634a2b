"""Performance cases of the library's main paths, at its public entry points.

``listed()`` gives the named cases, ``draw(rng)`` another case of the same
ranges, ``prepare`` / ``run`` one pass of a case, ``work`` the bytes and
operations that a pass cannot do without, ``tolerance`` how far two correct
implementations may differ, and ``exact`` the same outputs in 64 bits from
plain torch.

Kinds of case:
  nufft     type 1 (``nu2u``) and type 2 (``u2nu``) at the same points, planned
            or by the one-call functions, 1D / 2D / 3D, on tensors or on numpy
            arrays
  batch     many uneven 2D plans through ``batch.Batch``, both types
  autograd  differentiable type 2 at moving coordinates: plan, forward and
            backward with the gradients of image and coordinates
  wgrid     radio-interferometric gridding and degridding with w-stacking
  sphere    spherical-harmonic synthesis at arbitrary points and its adjoint
"""
import math

import numpy as np
import torch

from ducc_b200 import autograd, batch, nufft, sht, wgridder

C_LIGHT = 299792458.


# ------------------------------------------------------------------ cases
def _nufft(shape, npoints, dtype, eps, points, planned, host=False, fft_order=False):
    n = list(shape) + [1] * (3 - len(shape))
    return {"kind": "nufft", "ndim": len(shape), "n0": n[0], "n1": n[1], "n2": n[2],
            "npoints": npoints, "dtype": dtype, "eps": eps, "points": points,
            "planned": planned, "host": host, "fft_order": fft_order}


def listed():
    named = [
        # a DUCC script's small call on numpy arrays, nothing planned: latency
        # and launches are all there is
        ("small_host_2d", _nufft((64, 72), 4000, "c64", 1e-5, "uniform", False, host=True)),
        # a time series at uneven sampling times in double precision
        ("series_1d_c128", _nufft((3001,), 1_000_000, "c128", 1e-9, "uniform", True)),
        # a CG iteration's normal operator on a mid-size image: the
        # library's headline workload (16 Gaussian clusters, planned)
        ("clustered_2d_c64", _nufft((4096, 4096), 50_000_000, "c64", 1e-6, "clustered", True)),
        # coordinates that change with every call: index, spreading and
        # interpolation of a ragged image, few points per mode
        ("once_2d_c64", _nufft((1001, 1430), 400_000, "c64", 1e-5, "uniform", False,
                               fft_order=True)),
        # double precision at a tight tolerance, as DUCC's default arrays give it
        ("planned_2d_c128", _nufft((2000, 2048), 5_000_000, "c128", 1e-10, "uniform", True)),
        # a 3D volume in single precision (particles on a mesh, MRI volumes)
        ("volume_3d_c64", _nufft((256, 256, 256), 10_000_000, "c64", 1e-5, "uniform", True)),
        # the same in double precision at a tight tolerance
        ("volume_3d_c128", _nufft((90, 96, 100), 1_000_000, "c128", 1e-10, "uniform", True)),
        # a stack of images of different sizes and point sets, some with several
        # transforms over the same points
        ("uneven_batch", {"kind": "batch", "instances": 24, "side_min": 64, "side_max": 1024,
                          "m_min": 1000, "m_max": 1_000_000}),
        # a training step of a learned radial MRI trajectory
        ("radial_autograd", {"kind": "autograd", "side": 1024, "spokes": 2048, "samples": 2048,
                             "eps": 1e-6}),
        # a major cycle of radio imaging: residual visibilities to an image and
        # a model image to visibilities
        ("imaging_wgrid", {"kind": "wgrid", "npix": 2048, "rows": 200_000, "channels": 16,
                           "dtype": "c64", "eps": 1e-5, "fov_deg": 2.0, "weights": True}),
        # lensing a CMB temperature map: a field at displaced positions, and the adjoint
        ("sphere_spin0_c64", {"kind": "sphere", "lmax": 2047, "npoints": 10_000_000, "spin": 0,
                              "dtype": "c64", "eps": 1e-5}),
        # detector pointings on a polarised sky in double precision
        ("sphere_spin2_c128", {"kind": "sphere", "lmax": 767, "npoints": 1_000_000, "spin": 2,
                               "dtype": "c128", "eps": 1e-9}),
    ]
    return [dict(c, name=name) for name, c in named]


def _log(rng, a, b):
    return int(round(math.exp(rng.uniform(math.log(a), math.log(b)))))


def draw(rng):
    kind = rng.choice(["2d", "2d", "2d", "1d", "3d", "3d", "batch", "autograd", "wgrid", "sphere"])
    dtype = rng.choice(["c64", "c128"])
    if kind in ("1d", "2d", "3d"):
        eps = rng.choice([1e-3, 1e-4, 1e-5, 1e-6] if dtype == "c64" else [1e-5, 1e-7, 1e-9, 1e-11])
        if kind == "1d":
            shape, m = (_log(rng, 64, 3000),), _log(rng, 1000, 5_000_000)
        elif kind == "2d":
            big = 3000 if dtype == "c64" else 2000
            shape = (_log(rng, 48, big), _log(rng, 48, big))
            m = _log(rng, 1000, 20_000_000 if dtype == "c64" else 5_000_000)
        else:
            shape = tuple(_log(rng, 16, 160 if dtype == "c64" else 96) for _ in range(3))
            m = _log(rng, 1000, 5_000_000 if dtype == "c64" else 1_000_000)
        points = rng.choice(["uniform", "clustered"]) if kind == "2d" else "uniform"
        host = m <= 100_000 and rng.random() < 0.3
        return _nufft(shape, m, dtype, eps, points, rng.random() < 0.6, host=host,
                      fft_order=rng.random() < 0.3)
    if kind == "batch":
        return {"kind": "batch", "instances": rng.randint(4, 24), "side_min": 64,
                "side_max": _log(rng, 200, 1024), "m_min": 1000, "m_max": _log(rng, 10_000, 1_000_000)}
    if kind == "autograd":
        return {"kind": "autograd", "side": _log(rng, 128, 1024), "spokes": _log(rng, 100, 2048),
                "samples": _log(rng, 256, 2048), "eps": rng.choice([1e-4, 1e-5, 1e-6])}
    if kind == "wgrid":
        return {"kind": "wgrid", "npix": 2 * _log(rng, 64, 1024), "rows": _log(rng, 2000, 200_000),
                "channels": rng.randint(1, 16), "dtype": dtype,
                "eps": rng.choice([1e-3, 1e-4, 1e-5] if dtype == "c64" else [1e-5, 1e-7, 1e-9]),
                "fov_deg": rng.choice([1.0, 2.0, 5.0]), "weights": rng.random() < 0.5}
    return {"kind": "sphere", "lmax": _log(rng, 63, 1535 if dtype == "c64" else 767),
            "npoints": _log(rng, 10_000, 5_000_000 if dtype == "c64" else 1_000_000),
            "spin": rng.choice([0, 0, 2]), "dtype": dtype,
            "eps": rng.choice([1e-3, 1e-5]) if dtype == "c64" else rng.choice([1e-5, 1e-9])}


# ------------------------------------------------------------------ inputs
_CT = {"c64": torch.complex64, "c128": torch.complex128}
_RT = {"c64": torch.float32, "c128": torch.float64}


def _gen(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(int(seed))
    return g


def _randn(g, shape, dtype):
    return torch.randn(shape, generator=g, dtype=dtype, device="cuda")


def _rand(g, shape, dtype=torch.float64):
    return torch.rand(shape, generator=g, dtype=dtype, device="cuda")


def _points(g, m, ndim, how, dtype):
    """(m, ndim) coordinates in [-pi, pi): uniform, or 16 Gaussian clusters of
    sigma 0.3 (wrapped)."""
    if how == "uniform":
        x = (_rand(g, (m, ndim), dtype) * 2 - 1) * math.pi
    else:
        centres = (_rand(g, (16, ndim), dtype) * 2 - 1) * math.pi
        which = torch.randint(0, 16, (m,), generator=g, device="cuda")
        x = centres[which] + 0.3 * _randn(g, (m, ndim), dtype)
        x = torch.remainder(x + math.pi, 2 * math.pi) - math.pi
    return x.contiguous()


def _shape(case):
    return tuple(case["n%d" % d] for d in range(case["ndim"]))


def _nufft_inputs(case, seed):
    g = _gen(seed)
    ct, rt = _CT[case["dtype"]], _RT[case["dtype"]]
    coord = _points(g, case["npoints"], case["ndim"], case["points"], rt)
    return coord, _randn(g, (case["npoints"],), ct), _randn(g, _shape(case), ct)


def _batch_inputs(case, seed):
    # sizes belong to the case, values to the seed
    r = np.random.default_rng(1000 + case["instances"])
    g = _gen(seed)
    res = []
    for _ in range(case["instances"]):
        side = 2 * int(round(np.exp(r.uniform(np.log(case["side_min"]),
                                              np.log(case["side_max"]))) / 2))
        m = int(np.exp(r.uniform(np.log(case["m_min"]), np.log(case["m_max"]))))
        nt = int(r.choice([1, 4]))
        eps = float(r.choice([1e-4, 1e-6]))
        res.append((side, eps, nt, _points(g, m, 2, "uniform", torch.float32),
                    _randn(g, (nt, m), torch.complex64),
                    _randn(g, (nt, side, side), torch.complex64)))
    return res


def _autograd_inputs(case, seed):
    g = _gen(seed)
    ns, nr = case["spokes"], case["samples"]
    ang = math.pi * (torch.arange(ns, device="cuda", dtype=torch.float64)
                     + 0.1 * _randn(g, (ns,), torch.float64)) / ns
    rad = -math.pi + 2 * math.pi * torch.arange(nr, device="cuda", dtype=torch.float64) / nr
    coord = torch.stack([torch.outer(ang.cos(), rad).ravel(),
                         torch.outer(ang.sin(), rad).ravel()], 1).to(torch.float32).contiguous()
    n = case["side"]
    return coord, _randn(g, (n, n), torch.complex64), _randn(g, (ns * nr,), torch.complex64)


def _wgrid_inputs(case, seed):
    g = _gen(seed)
    rows, nch, npix = case["rows"], case["channels"], case["npix"]
    ps = case["fov_deg"] * math.pi / 180 / npix
    freq = 1.0e9 + torch.arange(nch, device="cuda", dtype=torch.float64) * (0.45e9 / nch)
    umax = 0.45 / ps * C_LIGHT / float(freq[-1])
    r = umax * _rand(g, (rows,)).sqrt()
    phi = 2 * math.pi * _rand(g, (rows,))
    w = (2 * _rand(g, (rows,)) - 1) * umax / 3
    uvw = torch.stack([r * phi.cos(), r * phi.sin(), w], 1).contiguous()
    vis = _randn(g, (rows, nch), _CT[case["dtype"]])
    wgt = (0.5 + _rand(g, (rows, nch), _RT[case["dtype"]])) if case["weights"] else None
    dirty = _randn(g, (npix, npix), _RT[case["dtype"]])
    return ps, freq, uvw, vis, wgt, dirty


def _sphere_inputs(case, seed):
    g = _gen(seed)
    lmax, m, spin = case["lmax"], case["npoints"], case["spin"]
    ncomp = 1 if spin == 0 else 2
    nalm = (lmax + 1) * (lmax + 2) // 2
    ab = _rand(g, (ncomp, nalm, 2)) * 2 - 1
    ab[:, :lmax + 1, 1] = 0           # a_l0 are real
    alm = torch.complex(ab[..., 0], ab[..., 1])
    if spin:                          # no l < spin
        for mm in range(spin):
            first = mm * (2 * lmax + 1 - mm) // 2
            alm[:, first + mm:first + spin] = 0
    loc = torch.stack([torch.acos(_rand(g, (m,)) * 2 - 1), 2 * math.pi * _rand(g, (m,))],
                      1).contiguous()
    mp = _rand(g, (ncomp, m), _RT[case["dtype"]]) - 0.5
    return alm.to(_CT[case["dtype"]]), loc, mp


# ------------------------------------------------------------------ prepare and run
def prepare(case, seed):
    kind = case["kind"]
    if kind == "nufft":
        coord, vals, grid = _nufft_inputs(case, seed)
        s = {"case": case, "coord": coord, "vals": vals, "grid": grid}
        if case["host"]:
            for k in ("coord", "vals", "grid"):
                s[k] = s[k].cpu().numpy()
            s["uni"] = np.empty(_shape(case), s["vals"].dtype)
        else:
            s["uni"] = torch.empty_like(grid)
        if case["planned"]:
            s["plan"] = nufft.plan(nu2u=True, coord=s["coord"], grid_shape=_shape(case),
                                   epsilon=case["eps"], fft_order=case["fft_order"])
            s["pout"] = np.empty_like(s["vals"]) if case["host"] else torch.empty_like(vals)
        return s
    if kind == "batch":
        inst = _batch_inputs(case, seed)
        plans = [nufft.plan(nu2u=True, coord=c, grid_shape=(side, side), epsilon=eps,
                            spreader="plain") for side, eps, _, c, _, _ in inst]
        return {"case": case, "batch": batch.Batch(plans, ntrans=[i[2] for i in inst]),
                "vals": [i[4] for i in inst], "grids": [i[5] for i in inst],
                "uni": [torch.empty_like(i[5]) for i in inst],
                "pout": [torch.empty_like(i[4]) for i in inst]}
    if kind == "autograd":
        coord, img, gout = _autograd_inputs(case, seed)
        return {"case": case, "coord": coord.requires_grad_(), "img": img.requires_grad_(),
                "gout": gout}
    if kind == "wgrid":
        ps, freq, uvw, vis, wgt, dirty = _wgrid_inputs(case, seed)
        return {"case": case, "vis": vis, "dirty": dirty,
                "kw": dict(uvw=uvw, freq=freq, wgt=wgt, pixsize_x=ps, pixsize_y=ps,
                           epsilon=case["eps"], do_wgridding=True, nthreads=16)}
    alm, loc, mp = _sphere_inputs(case, seed)
    return {"case": case, "alm": alm, "map": mp,
            "kw": dict(spin=case["spin"], lmax=case["lmax"], loc=loc, epsilon=case["eps"],
                       nthreads=16)}


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "nufft":
        if case["planned"]:
            p = state["plan"]
            return (p.nu2u(points=state["vals"], forward=True, out=state["uni"]),
                    p.u2nu(grid=state["grid"], forward=False, out=state["pout"]))
        kw = dict(coord=state["coord"], epsilon=case["eps"], fft_order=case["fft_order"])
        return (nufft.nu2u(points=state["vals"], forward=True, out=state["uni"], **kw),
                nufft.u2nu(grid=state["grid"], forward=False, **kw))
    if kind == "batch":
        b = state["batch"]
        return (b.nu2u(points=state["vals"], out=state["uni"], forward=True),
                b.u2nu(grids=state["grids"], out=state["pout"], forward=False))
    if kind == "autograd":
        state["img"].grad = None
        state["coord"].grad = None
        y = autograd.u2nu(state["img"], state["coord"], epsilon=case["eps"])
        y.backward(state["gout"])
        return y.detach(), state["img"].grad, state["coord"].grad
    if kind == "wgrid":
        n = case["npix"]
        return (wgridder.vis2dirty(vis=state["vis"], npix_x=n, npix_y=n, **state["kw"]),
                wgridder.dirty2vis(dirty=state["dirty"], **state["kw"]))
    return (sht.synthesis_general(alm=state["alm"], **state["kw"]),
            sht.adjoint_synthesis_general(map=state["map"], **state["kw"]))


# ------------------------------------------------------------------ work
def _nufft_work(shape, m, cbytes, eps):
    """Both types: coordinates, values and the uniform array once each per
    type; per type W^d multiply-adds of a complex value per point (W about
    log10(1/eps) + 2) and an FFT of twice the size per axis."""
    d, cells = len(shape), math.prod(2 * n for n in shape)
    w = math.ceil(math.log10(1 / eps)) + 2
    byts = 2 * (m * (d * cbytes // 2 + cbytes) + math.prod(shape) * cbytes)
    return byts, 2 * (4. * m * w ** d + 5. * cells * math.log2(cells))


def work(case):
    kind = case["kind"]
    cb = 16 if case.get("dtype") == "c128" else 8
    if kind == "nufft":
        b, f = _nufft_work(_shape(case), case["npoints"], cb, case["eps"])
    elif kind == "batch":
        b = f = 0
        r = np.random.default_rng(1000 + case["instances"])
        for _ in range(case["instances"]):
            side = 2 * int(round(np.exp(r.uniform(np.log(case["side_min"]),
                                                  np.log(case["side_max"]))) / 2))
            m = int(np.exp(r.uniform(np.log(case["m_min"]), np.log(case["m_max"]))))
            nt, eps = int(r.choice([1, 4])), float(r.choice([1e-4, 1e-6]))
            bb, ff = _nufft_work((side, side), m, cb, eps)
            b, f = b + nt * bb, f + nt * ff
    elif kind == "autograd":   # type 2, its adjoint and two derivative transforms
        b, f = _nufft_work((case["side"],) * 2, case["spokes"] * case["samples"], cb, case["eps"])
        b, f = 2 * b, 2 * f
    elif kind == "wgrid":
        nvis = case["rows"] * case["channels"]
        w = math.ceil(math.log10(1 / case["eps"])) + 2
        cells = (2 * case["npix"]) ** 2
        b = 2 * (nvis * (cb + (cb // 2 if case["weights"] else 0)) + case["rows"] * 24
                 + case["npix"] ** 2 * cb // 2)
        # W planes' footprints per visibility, and at least 2 W planes
        f = 2 * (4. * nvis * w ** 3 + 2 * w * 5. * cells * math.log2(cells))
    else:
        lmax, m = case["lmax"], case["npoints"]
        nc = 1 if case["spin"] == 0 else 2
        nalm = (lmax + 1) * (lmax + 2) // 2
        b, f = _nufft_work((2 * lmax + 1, nc * (lmax + 1)), m, cb, case["eps"])
        b = 2 * (m * (16 + nc * cb // 2) + nalm * nc * cb)
        f += 2 * 8. * nc * nalm * lmax   # one recurrence step and sum per (l, m, ring)
    return {"bytes": float(b), "flops": float(f)}


def tolerance(case):
    """Relative difference of two implementations with the same kernel and
    oversampled grid: rounding.  Single precision: spreading in another order
    differs by up to 9e-7 and the outputs lie up to 7e-7 (requested accuracy
    1e-5 and below) from 64 bits; double precision: 1e-13 and 2e-12 for the
    long recurrences of the sphere."""
    return {"rel": 1e-11 if case.get("dtype") == "c128" else 4e-6}


# ------------------------------------------------------------------ exact
_W = 16   # window cells per axis of the 64-bit transforms below (double grid)


def _window(z):
    return torch.where(z.abs() < 1, torch.exp(2.30 * _W * (torch.sqrt((1 - z * z).clamp(min=0)) - 1)),
                       torch.zeros_like(z))


def _window_ft(n, ngrid):
    """Fourier transform of the window at modes -(n/2) .. (n-1)/2."""
    x, wq = np.polynomial.legendre.leggauss(120)
    x, wq = torch.from_numpy(x).cuda(), torch.from_numpy(wq).cuda()
    k = torch.arange(-(n // 2), n - n // 2, device="cuda", dtype=torch.float64)
    a = k * (math.pi * _W / ngrid)
    return (_W / 2) * (torch.cos(a[:, None] * x) * (_window(x) * wq)).sum(1)


def _first_cells(x, ngrid):
    """First cell of each point's window and the window argument there."""
    t = torch.remainder(x / (2 * math.pi), 1.0) * ngrid
    i0 = torch.ceil(t - _W / 2)
    return i0.to(torch.int64), (i0 - t) / (_W / 2)


def _taps(coord, grid_shape):
    """For every cell of the W^d window: flat grid index and weight of each point."""
    ax = [_first_cells(coord[:, d], n) for d, n in enumerate(grid_shape)]

    def rec(d, idx, wt):
        if d == len(grid_shape):
            yield idx, wt
            return
        i0, z0 = ax[d]
        for a in range(_W):
            i = torch.remainder(i0 + a, grid_shape[d])
            w = _window(z0 + a * (2 / _W))
            yield from rec(d + 1, i if idx is None else idx * grid_shape[d] + i,
                           w if wt is None else wt * w)

    yield from rec(0, None, None)


def _centred(n, ngrid):
    """Grid indices of the modes -(n/2) .. (n-1)/2."""
    return torch.remainder(torch.arange(-(n // 2), n - n // 2, device="cuda"), ngrid)


def _kept(big, shape, grid_shape):
    for d, (n, m) in enumerate(zip(shape, grid_shape)):
        big = big.index_select(d, _centred(n, m))
    return big


def _corrected(u, shape, grid_shape):
    for d, (n, m) in enumerate(zip(shape, grid_shape)):
        u = u / _window_ft(n, m).reshape([-1 if e == d else 1 for e in range(len(shape))])
    return u


def _grid_shape(shape):
    return [max(2 * n, 2 * _W) for n in shape]


def _type1(coord, vals, shape, forward):
    """sum_j vals_j exp(-+ i k x_j) for centred modes k, in complex128."""
    coord, vals = coord.to(torch.float64), vals.to(torch.complex128)
    gs = _grid_shape(shape)
    re = torch.zeros(math.prod(gs), dtype=torch.float64, device="cuda")
    im = torch.zeros_like(re)
    for idx, w in _taps(coord, gs):
        re.index_add_(0, idx, w * vals.real)
        im.index_add_(0, idx, w * vals.imag)
    big = torch.complex(re, im).reshape(gs)
    big = torch.fft.fftn(big) if forward else torch.fft.ifftn(big, norm="forward")
    return _corrected(_kept(big, shape, gs), shape, gs)


def _type2(coord, uni, forward):
    """sum_k uni_k exp(-+ i k x_j) over centred modes k, in complex128."""
    coord, shape = coord.to(torch.float64), list(uni.shape)
    gs = _grid_shape(shape)
    u = _corrected(uni.to(torch.complex128), shape, gs)
    for d, (n, m) in enumerate(zip(shape, gs)):
        pad = list(u.shape)
        pad[d] = m
        u = torch.zeros(pad, dtype=torch.complex128, device="cuda").index_copy_(
            d, _centred(n, m), u)
    u = (torch.fft.fftn(u) if forward else torch.fft.ifftn(u, norm="forward")).reshape(-1)
    out = torch.zeros(coord.shape[0], dtype=torch.complex128, device="cuda")
    for idx, w in _taps(coord, gs):
        out += w * u[idx]
    return out


def _exact_nufft(case, seed):
    if case["npoints"] * 16. ** case["ndim"] > 2e10:
        return None   # over about 20 seconds
    coord, vals, grid = _nufft_inputs(case, seed)
    shape = _shape(case)
    uni = _type1(coord, vals, shape, True)
    if case["fft_order"]:
        uni = torch.fft.ifftshift(uni)
        grid = torch.fft.fftshift(grid)
    return uni, _type2(coord, grid, False)


def _exact_batch(case, seed):
    uni, pts = [], []
    for side, _, nt, coord, vals, grids in _batch_inputs(case, seed):
        uni.append(torch.stack([_type1(coord, vals[t], (side, side), True) for t in range(nt)]))
        pts.append(torch.stack([_type2(coord, grids[t], False) for t in range(nt)]))
    return uni, pts


def _exact_autograd(case, seed):
    coord, img, gout = _autograd_inputs(case, seed)
    n = case["side"]
    k = torch.arange(-(n // 2), n - n // 2, device="cuda", dtype=torch.float64)
    g = gout.to(torch.complex128)
    grad = [(g.conj() * _type2(coord, -1j * kk * img.to(torch.complex128), True)).real
            for kk in (k[:, None], k[None, :])]
    return (_type2(coord, img, True), _type1(coord, gout, (n, n), False), torch.stack(grad, 1))


def _exact_wgrid(case, seed):
    npix, nvis = case["npix"], case["rows"] * case["channels"]
    if npix ** 2 * float(nvis) > 5e10:
        return None   # direct sums: over about 20 seconds
    ps, freq, uvw, vis, wgt, dirty = _wgrid_inputs(case, seed)
    f = freq / C_LIGHT
    u, v, w = (torch.outer(uvw[:, a], f).reshape(-1) for a in range(3))
    wt = torch.ones_like(vis.real) if wgt is None else wgt
    c = (vis * wt).to(torch.complex128).reshape(-1)
    p = (torch.arange(npix, device="cuda", dtype=torch.float64) - npix / 2) * ps
    x, y = (a.reshape(-1) for a in torch.meshgrid(p, p, indexing="ij"))
    nm1 = torch.sqrt(1 - x * x - y * y) - 1
    image = torch.empty_like(x)
    out = torch.zeros_like(c)
    src = dirty.to(torch.float64).reshape(-1) / (nm1 + 1)
    step = max(1, (1 << 27) // nvis)
    for a in range(0, x.numel(), step):
        s = slice(a, a + step)
        ph = 2 * math.pi * torch.remainder(
            torch.outer(x[s], u) + torch.outer(y[s], v) - torch.outer(nm1[s], w), 1.0)
        re, im = ph.cos(), ph.sin()
        image[s] = re @ c.real - im @ c.imag
        out += torch.complex(src[s] @ re, -(src[s] @ im))
    return ((image / (nm1 + 1)).reshape(npix, npix),
            out.reshape(case["rows"], case["channels"]) * wt)


def _harmonics(lmax, spin, theta):
    """For l = 0, 1, ..: sqrt((2l+1)/(4 pi)) d^l_{m,-spin}(theta) as (m, theta)
    for m = 0..lmax (spin 0: with the Condon-Shortley sign) or -lmax..lmax, by
    the three-term recurrence in l from the single term at l = max(|m|, spin)."""
    m = torch.arange(0 if spin == 0 else -lmax, lmax + 1, device="cuda", dtype=torch.float64)
    l0 = m.abs().clamp(min=spin)
    lc, ls = torch.cos(theta / 2).clamp(min=0).log(), torch.sin(theta / 2).clamp(min=0).log()

    def power(e, lg):   # e * lg, 0 where e == 0 (lg may be -inf)
        return torch.where(e[:, None] == 0, 0., e[:, None] * lg[None, :])

    # exponents of cos and sin of theta/2 and sign of the single term (n = -spin)
    top, bottom = m >= spin, m <= -spin
    ec = torch.where(top, l0 - spin, torch.where(bottom, l0 + spin, spin - m))
    es = torch.where(top, l0 + spin, torch.where(bottom, l0 - spin, spin + m))
    odd = torch.where(top, m + spin, torch.where(bottom, 0 * m, m + spin))
    lognorm = 0.5 * (torch.lgamma(2 * l0 + 1) - torch.lgamma(ec + 1) - torch.lgamma(es + 1))
    # carried times e^300, so that sin^m theta stays in range for lmax to 2047
    start = torch.exp(300 + lognorm[:, None] + power(ec, lc) + power(es, ls))
    start = start * (1 - 2 * torch.remainder(odd, 2))[:, None]
    ct = torch.cos(theta)[None, :]
    cur, prev = torch.zeros_like(start), torch.zeros_like(start)
    for l in range(lmax + 1):
        # d^l from d^(l-1), d^(l-2)
        if l >= 1:
            k = l - 1
            den = torch.sqrt(((l * l - m * m) * (l * l - spin * spin)).clamp(min=0)) * max(k, 1)
            a = (2 * k + 1) * (k * (k + 1) * ct + (m * spin)[:, None])
            if k == 0:
                a = (ct + 0 * m[:, None])
            b = l * torch.sqrt(((k * k - m * m) * (k * k - spin * spin)).clamp(min=0))
            ok = ((l0 < l) & (den > 0))[:, None]
            den = torch.where(den > 0, den, torch.ones_like(den))[:, None]
            new = torch.where(ok, (a * cur - b[:, None] * prev) / den, torch.zeros_like(cur))
            prev, cur = cur, new
        cur = torch.where((l0 == l)[:, None], start, cur)
        yield l, m.to(torch.int64), math.sqrt((2 * l + 1) / (4 * math.pi)) * (math.exp(-300) * cur)


def _rings(case):
    lmax = case["lmax"]
    nr = 2 * lmax + 2                       # equidistant rings of the full circle
    theta = 2 * math.pi * torch.arange(lmax + 2, device="cuda", dtype=torch.float64) / nr
    return nr, theta                        # the rings 0 .. pi


def _mirrored(f, m, spin):
    """Values on the rings 0 .. pi, continued to the full circle (rings last)."""
    sign = (1 - 2 * torch.remainder(m + spin, 2)).to(torch.float64)
    return torch.cat([f, sign[:, None] * f[:, 1:-1].flip(1)], 1)


def _alm_index(lmax, l, m):
    return m * (2 * lmax + 1 - m) // 2 + l


def _exact_sphere(case, seed):
    alm, loc, mp = _sphere_inputs(case, seed)
    lmax, spin = case["lmax"], case["spin"]
    if case["npoints"] * 256. > 2e10:
        return None
    alm = alm.to(torch.complex128)
    nr, theta = _rings(case)
    nm = (lmax + 1) if spin == 0 else (2 * lmax + 1)
    sg = -1. if spin % 2 == 0 else 1.       # (-1)^(spin+1)
    ring = torch.zeros((nm, theta.numel()), dtype=torch.complex128, device="cuda")
    for l, m, lam in _harmonics(lmax, spin, theta):
        i = _alm_index(lmax, l, m.abs().clamp(max=l))
        if spin == 0:
            co = alm[0, i]
        else:
            par = (1 - 2 * torch.remainder(m, 2)).to(torch.float64)
            e, b = alm[0, i], alm[1, i]
            co = sg * (torch.where(m < 0, par * e.conj(), e) + 1j * torch.where(m < 0, par * b.conj(), b))
        ring += torch.where(m.abs() <= l, co, 0)[:, None] * lam
    # theta modes (centred) by the DFT of the full circle; mode order (theta, m)
    full = torch.fft.fft(_mirrored(ring, m, spin), dim=1) / nr
    modes = full.index_select(1, _centred(2 * lmax + 1, nr)).T.contiguous()
    if spin == 0:   # real field: m > 0 counts twice
        wide = torch.zeros((2 * lmax + 1, 2 * lmax + 1), dtype=torch.complex128, device="cuda")
        wide[:, lmax:] = modes
        wide[:, lmax + 1:] *= 2
        modes = wide
    f = _type2(loc, modes, False)
    out_map = f.real[None] if spin == 0 else torch.stack([f.real, f.imag])
    # adjoint
    q = mp[0].to(torch.complex128) if spin == 0 else torch.complex(mp[0].double(), mp[1].double())
    gm = _type1(loc, q, (2 * lmax + 1, 2 * lmax + 1), True)
    if spin == 0:
        gm = gm[:, lmax:]
    big = torch.zeros((nr, nm), dtype=torch.complex128, device="cuda")
    big.index_copy_(0, _centred(2 * lmax + 1, nr), gm)
    h = torch.fft.ifft(big, dim=0).T        # (m, rings): the 1/nr is ifft's
    sign = (1 - 2 * torch.remainder(m + spin, 2)).to(torch.float64)[:, None]
    half = h[:, :lmax + 2].clone()
    half[:, 1:-1] += sign * h[:, lmax + 2:].flip(1)
    out_alm = torch.zeros_like(alm)
    for l, m, lam in _harmonics(lmax, spin, theta):
        wl = (lam * half).sum(1)
        if spin == 0:
            k = m[:l + 1]
            out_alm[0, _alm_index(lmax, l, k)] = wl[:l + 1]
        elif l >= spin:
            k = torch.arange(l + 1, device="cuda")
            par = (1 - 2 * torch.remainder(k, 2)).to(torch.float64)
            wp, wm = wl[lmax:lmax + l + 1], par * wl[lmax - l:lmax + 1].flip(0).conj()
            out_alm[0, _alm_index(lmax, l, k)] = sg * (wp + wm) / 2
            out_alm[1, _alm_index(lmax, l, k)] = -1j * sg * (wp - wm) / 2
    return out_map, out_alm


def exact(case, seed):
    return {"nufft": _exact_nufft, "batch": _exact_batch, "autograd": _exact_autograd,
            "wgrid": _exact_wgrid, "sphere": _exact_sphere}[case["kind"]](case, seed)
