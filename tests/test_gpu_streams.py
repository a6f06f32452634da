"""Calls on streams other than the default one, which do not wait for it."""
import numpy as np
import pytest

from test_gpu_parity import check_interp, check_spread, dev, plan_for

pytestmark = pytest.mark.gpu


# 1,728 bins scanned by the count kernel, 13,824 by kernels of their own, and
# the binning of few points by one block
@pytest.mark.parametrize("cells,n", [(32, 5000), (64, 5000), (64, 700)])
def test_first_call_on_a_side_stream(ibk, oracle, cuda, cells, n):
    """A fresh plan's first calls find its scratch cleared, although the
    default stream is still busy with work queued before."""
    import torch
    L = [cells / 40.0] * 3
    rng = np.random.default_rng(cells + n)
    g = oracle.geometry(3, L, [0, 0, 0], oracle.TAG_MAC, cells)
    x = np.concatenate([rng.uniform(0, l, n) for l in L])
    f = rng.normal(size=3 * n)
    ue = [rng.normal(size=int(g.size[c])) for c in range(3)]
    plan = plan_for(ibk, 3, L, [0, 0, 0], 0, cells, 0, 3)
    xd, fd, ued = dev(x, cuda), dev(f, cuda), [dev(u, cuda) for u in ue]
    fe = [torch.full((s,), np.nan, dtype=torch.float64, device=cuda) for s in plan.sizes()]
    ul = torch.full((3 * n,), np.nan, dtype=torch.float64, device=cuda)
    torch.cuda.synchronize()
    side = torch.cuda.Stream()
    busy = torch.ones(1 << 28, dtype=torch.float64, device=cuda)
    for _ in range(40):                  # about 25 ms of copies
        busy.mul_(1.0)
    with torch.cuda.stream(side):
        plan.spread(n, xd, fd, fe)
        plan.interpolate(n, xd, ued, ul)
    torch.cuda.synchronize()
    plan.check()
    want_fe, fa = oracle.spread(g, x, f, with_abs=True)
    want, ua = oracle.interpolate(g, x, ue, with_abs=True)
    check_spread([t.cpu().numpy() for t in fe], want_fe, fa)
    check_interp(ul.cpu().numpy(), want, ua)


@pytest.mark.parametrize("first", ["spread", "interpolate"])
def test_captured_spread_takes_the_points_of_any_call_before(ibk, cuda, first):
    """Scratch grown by an interpolation of many points also serves a captured
    FP32C spread of as many, when spreads have only had a few points so far."""
    import torch
    rng = np.random.default_rng(2)
    n, few, L = 5000, 100, [1.6, 1.6, 1.6]
    plan = plan_for(ibk, 3, L, [0, 0, 0], 0, 64, 0, 3, ibk.FP32C)
    x, f = (dev(a, cuda) for a in (rng.uniform(0, 1.6, 3 * n), rng.normal(size=3 * n)))
    xs, fs = (dev(a, cuda) for a in (rng.uniform(0, 1.6, 3 * few), rng.normal(size=3 * few)))
    ue = [dev(rng.normal(size=s), cuda) for s in plan.sizes()]
    ul = torch.empty_like(x)
    fe, want = ([torch.zeros(s, dtype=torch.float64, device=cuda) for s in plan.sizes()] for _ in range(2))
    calls = [lambda: plan.spread(few, xs, fs, fe), lambda: plan.interpolate(n, x, ue, ul)]
    for call in calls if first == "spread" else calls[::-1]:
        call()
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        plan.spread(n, x, f, fe)
    graph.replay()
    plan_for(ibk, 3, L, [0, 0, 0], 0, 64, 0, 3, ibk.FP32C).spread(n, x, f, want)
    torch.cuda.synchronize()
    assert all(torch.equal(a, b) for a, b in zip(fe, want))
