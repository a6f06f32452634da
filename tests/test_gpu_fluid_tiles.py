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
         # as few points along the marched axis as its halo reaches
         ((12, 6, 3), (0, 0, 0), 0), ((6, 12, 3), (0, 1, 0), 1), ((6, 12, 3), (0, 0, 0), 2),
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


@pytest.mark.parametrize("cells", [(8, 8, 8), (24, 24)])
@pytest.mark.parametrize("pc", [0, 1])
def test_nothing_to_solve(ibk, cuda, cells, pc):
    """A right-hand side of zero on a walled grid: converged before the first
    iteration, the field unchanged."""
    import torch
    dom = ibk.Domain(*[ibk.Dimension(float(c), ibk.SOLID) for c in cells])
    plan = ibk.Plan(ibk.Mac(cells[0]), dom, ibk.Bspline(3), ibk.FP64)
    d = ibk.Diffusion(plan, 0, 3.2, 1.0, tolerance=1e-10, preconditioner=pc)
    zero = torch.zeros(d.size, dtype=torch.float64, device=cuda)
    assert torch.equal(d.step(zero, zero, zero), zero) and d.iterations == 0


@pytest.mark.parametrize("cells", [(8, 8, 8), (24, 24)])
@pytest.mark.parametrize("pc", [0, 1])
def test_bail_out(ibk, cuda, oracle, cells, pc):
    """Without viscosity H is the corrected identity, below 1 at walls: a force
    on one corner face gives a direction d with |d| above the tolerance and
    <d, H d> below its square, where the loop ends without an update."""
    import torch
    dims = len(cells)
    dom = ibk.Domain(*[ibk.Dimension(float(c), ibk.SOLID) for c in cells])
    plan = ibk.Plan(ibk.Mac(cells[0]), dom, ibk.Bspline(3), ibk.FP64)
    robin = [((1.0, 0.0), (1.0, 0.0))] * 3
    geometry = oracle.geometry(dims, [float(c) for c in cells], [1] * dims, tag=oracle.TAG_MAC, refinement=cells[0])
    fg = oracle.FluidGrid(geometry, 0, robin)
    f = np.zeros(fg.size)
    f[0] = 1.0
    corner = oracle.diffusion_apply(fg, 1, f, lam=0.0)[0]
    assert 0.0 < corner < 0.9
    # d = p(H) r, and p(H) is close to 1 / H: |d| is about the force, <d, H d> about corner
    tol = math.sqrt(math.sqrt(corner))
    u = np.random.default_rng(4).normal(size=fg.size)
    zero = np.zeros(fg.size)
    want, it = oracle.diffusion_step(fg, 1.0, 0.0, tol, 100, 1.0, zero, zero, f, precond=pc)
    assert it == 0 and np.array_equal(want, zero)      # the oracle bails out
    d = ibk.Diffusion(plan, 0, 1.0, 0.0, tolerance=tol, robin=robin, preconditioner=pc)
    got = d.step(*(torch.from_numpy(a).to(cuda) for a in (u, zero, f)))
    assert d.iterations == 0 and np.array_equal(got.cpu().numpy(), u)
    assert not np.array_equal(oracle.diffusion_step(fg, 1.0, 0.0, 1e-3 * tol, 100, 1.0, zero, zero, f, precond=pc)[0], zero)


def test_two_handles_on_two_streams_at_once(ibk, cuda):
    import threading
    import torch
    cells = (64, 64, 64)
    dom = ibk.Domain(*[ibk.Dimension(float(c)) for c in cells])
    plan = ibk.Plan(ibk.Mac(64), dom, ibk.Bspline(3), ibk.FP64)
    solvers = [ibk.Diffusion(plan, c, 3.2, 1.0, tolerance=1e-10) for c in range(2)]
    fields = [[torch.randn(s.size, dtype=torch.float64, device=cuda) for _ in range(3)] for s in solvers]
    want = [s.step(*a).clone() for s, a in zip(solvers, fields)]
    torch.cuda.synchronize()
    got, streams = [None, None], [torch.cuda.Stream() for _ in range(2)]

    def work(i):
        with torch.cuda.stream(streams[i]):
            for _ in range(20):
                got[i] = solvers[i].step(*fields[i])
            streams[i].synchronize()
    threads = [threading.Thread(target=work, args=(i,)) for i in range(2)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert all(torch.equal(a, b) for a, b in zip(got, want))
