"""The binning's two forms (one block for few points, else count, scan and
scatter), the FP32C spread's CTA sizes and the folded form's copies of the
accumulators, at the sizes where the rules between them lie, through the C
ABI against the oracle."""
import numpy as np
import pytest

from test_gpu_parity import FP32C_TOL, check_interp, check_spread, device_interp, device_spread, normwise, plan_for

pytestmark = pytest.mark.gpu


# 16^3 tiles of 64^3 in FP32C: 1,728 bins (scanned by the count kernel above one
# point a thread); 8^3 in FP64: 13,824 bins; 160^3: 27,000, more than the block holds
@pytest.mark.parametrize("n", [1, 33, 1023, 1024, 1025, 3071, 3072, 3073])
@pytest.mark.parametrize("cells,precision", [(64, 0), (64, 1), (160, 1)])
def test_few_points(ibk, oracle, cuda, n, cells, precision):
    L = [cells / 40.0] * 3
    rng = np.random.default_rng(n + cells)
    g = oracle.geometry(3, L, [0, 1, 0], oracle.TAG_MAC, cells)
    plan = plan_for(ibk, 3, L, [0, 1, 0], 0, cells, 0, 3, precision)
    x = np.concatenate([rng.uniform(-0.01, l + 0.01, n) for l in L])
    f = rng.normal(size=3 * n)
    ue = [rng.normal(size=int(g.size[c])) for c in range(3)]
    want_fe, fa = oracle.spread(g, x, f, with_abs=True)
    want, ua = oracle.interpolate(g, x, ue, with_abs=True)
    fe, ul = device_spread(plan, x, f, cuda), device_interp(plan, x, ue, cuda)
    if precision == 0:
        check_spread(fe, want_fe, fa)
        check_interp(ul, want, ua)
        return
    for c in range(3):
        assert normwise(fe[c], want_fe[c]) <= FP32C_TOL
        assert normwise(ul[c * n:(c + 1) * n], want[c * n:(c + 1) * n]) <= FP32C_TOL


# four, two and one copy of the accumulators, and tiles on both sides of the
# rule for CTAs of 512 threads (at most two tiles per SM)
@pytest.mark.parametrize("tiles", [(16, 16, 16), (32, 24, 16), (32, 32, 12), (8, 8, 8)])
def test_folded_copies(ibk, oracle, cuda, tiles):
    L = [1.6, 1.6, 1.6]
    rng = np.random.default_rng(sum(tiles))
    g = oracle.geometry(3, L, [0, 0, 0], oracle.TAG_MAC, 64)
    plan = plan_for(ibk, 3, L, [0, 0, 0], 0, 64, 0, 3, ibk.FP32C)
    plan.set_tiles(tiles, (16, 16, 16))
    n = 40001
    # most points within a few cells of one corner of a tile, the rest anywhere
    x = np.concatenate([np.concatenate([rng.normal(0.8, 0.05, n - 4000), rng.uniform(0, 1.6, 4000)]) for _ in range(3)])
    f = rng.normal(size=3 * n)
    want_fe = oracle.spread(g, x, f)
    a, b = device_spread(plan, x, f, cuda), device_spread(plan, x, f, cuda)
    for c in range(3):
        assert normwise(a[c], want_fe[c]) <= FP32C_TOL
        assert np.array_equal(a[c], b[c])
