"""Shared device constants: unplanned calls upload theirs once, whatever plans a
program makes; plans stay right when the table has given their entry up."""
import threading

import numpy as np
import pytest

from ducc_b200 import nufft

pytestmark = pytest.mark.gpu


def _problem(shape, M=400, seed=0):
    import torch
    rng = np.random.default_rng(seed)
    coord = torch.from_numpy(rng.uniform(-np.pi, np.pi, (M, len(shape)))).cuda()
    vals = torch.from_numpy(rng.standard_normal(M) + 1j * rng.standard_normal(M)).cuda()
    return coord, vals


def _uploads(f):
    import torch
    from torch.profiler import ProfilerActivity, profile
    f()
    torch.cuda.synchronize()
    with profile(activities=[ProfilerActivity.CUDA]) as p:
        f()
        torch.cuda.synchronize()
    names = [e.name for e in p.events()]
    if not any("k_spread" in n for n in names):
        pytest.skip("no kernel records from the profiler")
    return sum("HtoD" in n for n in names)


def test_unplanned_call_uploads_once_after_many_plans():
    import torch
    plans = []
    for i in range(70):
        shape = (20 + 2 * i, 16 + i)
        coord, _ = _problem(shape, 50)
        plans.append(nufft.plan(nu2u=True, coord=coord, grid_shape=shape, epsilon=1e-7))
    del plans
    shape = (31, 77)
    coord, vals = _problem(shape)
    out = torch.empty(shape, dtype=torch.complex128, device="cuda")
    assert _uploads(lambda: nufft.nu2u(points=vals, coord=coord, forward=True, epsilon=1e-7,
                                       out=out)) == 0


def test_plans_outlive_their_place_in_the_table():
    import torch
    shape = (40, 52)
    coord, vals = _problem(shape, seed=1)
    out = [torch.empty(shape, dtype=torch.complex128, device="cuda") for _ in range(2)]
    plan = nufft.plan(nu2u=True, coord=coord, grid_shape=shape, epsilon=1e-9)
    twin = nufft.plan(nu2u=True, coord=coord, grid_shape=shape, epsilon=1e-9)
    plan.nu2u(points=vals, forward=True, out=out[0])
    del twin

    def churn(k):
        for i in range(40):
            s = (10 + 2 * i, 12 + 2 * k)
            c, v = _problem(s, 60, seed=k)
            p = nufft.plan(nu2u=True, coord=c, grid_shape=s, epsilon=1e-9)
            o = torch.empty(s, dtype=torch.complex128, device="cuda")
            p.nu2u(points=v, forward=True, out=o)
            q = torch.empty(s, dtype=torch.complex128, device="cuda")
            nufft.nu2u(points=v, coord=c, forward=True, epsilon=1e-9, out=q)
            ok.append(bool(torch.linalg.vector_norm(o - q) <= 2e-9 * torch.linalg.vector_norm(q)))
            del p

    ok = []
    threads = [threading.Thread(target=churn, args=(k,)) for k in range(4)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert len(ok) == 160 and all(ok)
    plan.nu2u(points=vals, forward=True, out=out[1])
    # (sums in another order)
    assert torch.linalg.vector_norm(out[1] - out[0]) <= 2e-9 * torch.linalg.vector_norm(out[0])
