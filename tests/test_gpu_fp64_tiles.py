"""The FP64 spread's tiles (two owning warps a tile, candidates prepared in
chunks of 32) and the exact weights, at the edges of both, through the C ABI
against the oracle: spread within 1e-12 of the sum of |terms| per face (the
summation order differs), interpolation and sort keys bit for bit."""
import numpy as np
import pytest

from test_gpu_parity import check_interp, check_spread, device_interp, device_keys, device_spread, plan_for

pytestmark = pytest.mark.gpu


def _run(ibk, oracle, cuda, x, L, solid, ref, delta=("bspline", 3), tiles=None, seed=3):
    dims = len(L)
    rng = np.random.default_rng(seed)
    kind = oracle.DELTA_NAMES[delta[0]]
    g = oracle.geometry(dims, L, solid, oracle.TAG_MAC, ref, kind, delta[1])
    plan = plan_for(ibk, dims, L, solid, 0, ref, kind, delta[1])
    if tiles is not None:
        plan.set_tiles(tiles, tiles)
    f = rng.normal(size=x.size)
    ue = [rng.normal(size=int(g.size[c])) for c in range(dims)]
    want_fe, fa = oracle.spread(g, x, f, with_abs=True)
    check_spread(device_spread(plan, x, f, cuda), want_fe, fa)
    want, ua = oracle.interpolate(g, x, ue, with_abs=True)
    check_interp(device_interp(plan, x, ue, cuda), want, ua)
    return g, plan


# candidates of the one crowded tile around the chunk size and its warps
@pytest.mark.parametrize("n", [1, 31, 32, 33, 63, 64, 65, 128, 129, 1000])
def test_chunk_edges(ibk, oracle, cuda, n):
    rng = np.random.default_rng(n)
    x = np.concatenate([rng.uniform(0.55, 0.85, n) for _ in range(3)])
    _run(ibk, oracle, cuda, x, [1.6, 1.6, 1.6], [0, 1, 0], 64)


# tile extents that are odd, smaller and larger than the default, and one
# whose accumulators are not padded; the two owners split the last axis
@pytest.mark.parametrize("tiles", [(4, 4, 4), (5, 7, 9), (17, 13, 11), (20, 20, 20), (64, 16, 5), (32, 24, 18)])
def test_tile_extents(ibk, oracle, cuda, tiles):
    rng = np.random.default_rng(sum(tiles))
    x = np.concatenate([rng.uniform(-0.05, 1.65, 4000) for _ in range(3)])
    _run(ibk, oracle, cuda, x, [1.6, 1.6, 1.6], [0, 1, 0], 64, tiles=tiles)


@pytest.mark.parametrize("delta", [("bspline", 1), ("bspline", 4), ("bspline", 5), ("peskin", 0), ("roma", 0)])
@pytest.mark.parametrize("L,solid,ref", [([1.6, 0.8], [0, 1], 24), ([0.75, 0.5, 0.875], [0, 0, 0], 2)])
def test_other_widths(ibk, oracle, cuda, delta, L, solid, ref):
    """Stencils of 2 to 6 nodes (one to seven rounds of a warp), in two
    dimensions and where every axis is one wrapping tile."""
    rng = np.random.default_rng(ref)
    x = np.concatenate([rng.uniform(0, l, 700) for l in L])
    _run(ibk, oracle, cuda, x, L, solid, ref, delta=delta)


def test_points_on_and_next_to_nodes(ibk, oracle, cuda):
    """Offsets of exactly 0 and within rounding of 0, 1/2 and 1 of a cell (the
    reference's own recursion jumps there), and positions far outside."""
    h, n = 1.0 / 64, 600
    rng = np.random.default_rng(8)
    axes = []
    for _ in range(3):
        v = rng.integers(4, 60, n) * h + rng.choice([0.0, 0.5 * h], n)
        for k in range(1, 4):
            v[k::8] = np.nextafter(v[k::8], rng.choice([-1.0, 2.0], v[k::8].size))
        v[4::8] += rng.choice([-1, 1], v[4::8].size) * 2.0 ** -rng.integers(45, 60, v[4::8].size)
        axes.append(v)
    x = np.concatenate(axes)
    g, plan = _run(ibk, oracle, cuda, x, [1.0, 1.0, 1.0], [0, 0, 0], 64)
    far = np.concatenate([rng.choice([-1.0, 1.0], 500) * 10.0 ** rng.uniform(-320, 7, 500) for _ in range(3)])
    for c, got in enumerate(device_keys(plan, far, cuda)):
        assert np.array_equal(got, oracle.sort_keys(g, c, far))


@pytest.mark.parametrize("tiles", [None, (16, 16, 16)])
def test_positions_beyond_the_index_range(ibk, oracle, cuda, tiles):
    """Positions more than 2^31 cells past a wall, where the stencil's index
    saturates: the delta function is 0 there, so they leave the grid as it is
    and take no velocity."""
    rng = np.random.default_rng(12)
    L, solid, n, far = [1.6, 1.6, 1.6], [0, 1, 0], 300, 40
    g = oracle.geometry(3, L, solid, oracle.TAG_MAC, 64)
    plan = plan_for(ibk, 3, L, solid, 0, 64, 0, 3)
    if tiles is not None:
        plan.set_tiles(tiles, tiles)
    near = [rng.uniform(0, l, n) for l in L]
    f = [rng.normal(size=n) for _ in range(3)]
    away = [rng.uniform(0, 1.6, far), 10.0 ** rng.uniform(8, 25, far) * rng.choice([-1, 1], far), rng.uniform(0, 1.6, far)]
    x = np.concatenate([np.concatenate([a, b]) for a, b in zip(near, away)])
    fl = np.concatenate([np.concatenate([a, rng.normal(size=far)]) for a in f])
    want_fe, fa = oracle.spread(g, np.concatenate(near), np.concatenate(f), with_abs=True)
    check_spread(device_spread(plan, x, fl, cuda), want_fe, fa)
    ue = [rng.normal(size=int(g.size[c])) for c in range(3)]
    ul = device_interp(plan, x, ue, cuda).reshape(3, n + far)
    assert np.array_equal(ul[:, n:], np.zeros((3, far)))
    want, ua = oracle.interpolate(g, np.concatenate(near), ue, with_abs=True)
    check_interp(np.ascontiguousarray(ul[:, :n]).reshape(-1), want, ua)


# both forms of the cubic B-spline's spread on either side of the rules between
# them, at tiles that split unevenly, are not padded or wrap: (cells, tiles, points)
@pytest.mark.parametrize("cells,tiles,n", [
    ((24, 24, 24), None, 60000),                    # few full tiles: split candidates
    ((24, 24, 24), None, 8000), ((24, 24, 24), None, 9000),                 # 27 tiles, below and above the limit of few
    ((128, 128, 128), None, 30000), ((128, 128, 128), None, 34000),         # 512 of 16^3, likewise
    ((128, 128, 128), (20, 20, 20), 24000), ((128, 128, 128), (32, 24, 18), 24000),
    ((128, 128, 128), (13, 11, 13), 3000), ((16, 128, 128), (16, 8, 8), 3000), ((16, 16, 16), (16, 16, 16), 9000)])
def test_cubic_forms(ibk, oracle, cuda, cells, tiles, n):
    rng = np.random.default_rng(n)
    L = [c / 40.0 for c in cells]
    x = np.concatenate([rng.uniform(-0.01, l + 0.01, n) for l in L])
    _run(ibk, oracle, cuda, x, L, [0, 1, 0], min(cells), tiles=tiles)
