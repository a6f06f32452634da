"""The Chebyshev-preconditioned diffusion loop (two kernels an iteration, tiles
of columns with recomputed halos) against the oracle, at grids on the edges
of its tiles: fewer faces than a halo reaches around, one more or less than
a tile is wide, runs of planes that do not divide the axis, and for both
tile sizes blocks that reach no wall, walls along y only, and others.

Both solves stop at |d| <= 1e-10, which bounds what a different rounding (or
one iteration more) can change; 1e-10 of the largest value is above that."""
import math

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

ROBIN = [((1.0, 0.0), (0.0, 1.0)), ((2.0, 0.5), (1.0, 0.0)), ((1.0, 0.0), (1.0, 0.0))]
CASES = [((3, 6, 12), (0, 0, 0), 0), ((3, 6, 12), (0, 1, 0), 1), ((4, 8, 4), (1, 1, 1), 2),
         ((26, 13, 52), (0, 1, 0), 0), ((27, 27, 27), (1, 0, 1), 1), ((59, 59, 118), (0, 1, 0), 0),
         ((59, 118), (0, 1), 0), ((174, 87, 87), (0, 0, 0), 2), ((174, 87, 87), (0, 1, 0), 1),
         ((174, 87, 87), (1, 1, 1), 0),
         # few faces along x: tiles of 10 x 26
         ((4, 400, 40), (1, 0, 1), 0), ((8, 400, 40), (0, 1, 0), 1),
         # two dimensions: tiles of 26 x 10 faces, more than 2 per SM of those: of 58 x 26
         ((3, 3), (0, 0), 0), ((4, 8), (1, 1), 0), ((26, 52), (0, 0), 1), ((27, 54), (1, 0), 1), ((348, 232), (0, 0), 0),
         ((348, 232), (1, 1), 1), ((464, 232), (0, 1), 0)]


@pytest.mark.parametrize("cells,solid,comp", CASES)
def test_step_matches_oracle(ibk, cuda, oracle, cells, solid, comp):
    import torch
    lengths, dims = [float(c) for c in cells], len(cells)
    tag = math.gcd(*cells)
    dom = ibk.Domain(*[ibk.Dimension(l, ibk.SOLID if s else ibk.PERIODIC) for l, s in zip(lengths, solid)])
    plan = ibk.Plan(ibk.Mac(tag), dom, ibk.Bspline(3), ibk.FP64)
    fg = oracle.FluidGrid(oracle.geometry(dims, lengths, list(solid), tag=oracle.TAG_MAC, refinement=tag), comp, ROBIN)
    dt, mu, tol = 3.2, 1.0, 1e-10
    d = ibk.Diffusion(plan, comp, dt, mu, tolerance=tol, robin=ROBIN)
    assert d.size == fg.size
    rng = np.random.default_rng(sum(cells) + comp)
    u, rhs, f = (rng.normal(size=fg.size) for _ in range(3))
    U, R, F = (torch.from_numpy(a).to(cuda) for a in (u, rhs, f))
    want, it = oracle.diffusion_step(fg, dt, mu, tol, 10000, 1.0, u, rhs, f)
    got = d.step(U, R, F)
    assert abs(d.iterations - it) <= 1
    assert np.abs(got.cpu().numpy() - want).max() <= 1e-10 * np.abs(want).max()
    # the same bits from one call to the next
    assert torch.equal(d.step(U, R, F), got)
