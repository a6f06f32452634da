"""The framework's work as a user has it do it, one case per kind and size.

A case is a dict of plain values.  ``listed`` names the fixed ones, ``draw``
gives more of the same ranges; ``prepare`` makes what a simulation holds
before the call (plans, positions, forces, grids on the GPU), ``run`` is one
pass through the public entry points, ``exact`` the same outputs from plain
torch in 64 bits and ``work`` what one pass cannot do without.

Units follow the library's workloads: length unit 10 um, grid spacing
0.25 um, forces in pN and velocities in um/s.
"""
import importlib.util
import math
import os
import sys

import torch

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def _package():
    if "ib_cu_b200" not in sys.modules:
        folder = os.path.join(ROOT, "ib.cu_b200")
        spec = importlib.util.spec_from_file_location(
            "ib_cu_b200", os.path.join(folder, "__init__.py"), submodule_search_locations=[folder])
        module = importlib.util.module_from_spec(spec)
        sys.modules["ib_cu_b200"] = module
        spec.loader.exec_module(module)
    return sys.modules["ib_cu_b200"]


UM, PN, UM_PER_S = 0.1, 1e-4, 1e-4      # internal units per um, pN, um/s
H = 0.25 * UM                           # grid spacing
STEP_DT, STEP_K = 1e-3, 1e-3            # 1 us; 1 pN/um
TIMESTEP, VISCOSITY, TOLERANCE = 1e-3, 1.0, 1e-11
SHEAR, BULK, BENDING, VISCOUS = 0.25, 25.0, 1.0, 0.25


def listed():
    return [
        # One red cell in a periodic box, in the library's default precision:
        # a spread and an interpolation as two calls.  Launch latency.
        dict(name="rbc-pair-fp64", kind="couple", scene="box", nx=64, ny=64, nz=64, wall=False, rbc=1, plt=0,
             rbc_points=2210, plt_points=605, delta="bspline3", precision="fp64", call="two"),
        # Platelet outlines in a walled two-dimensional channel, with the
        # 3-point delta of two-dimensional runs.
        dict(name="outlines-2d-fp64", kind="couple", scene="plane", nx=240, ny=120, nz=0, wall=True, rbc=0, plt=24,
             rbc_points=0, plt_points=160, delta="roma", precision="fp64", call="two"),
        # The 32 x 16 x 32 um channel: the force half of a step alone ...
        dict(name="channel-spread-fp32c", kind="couple", scene="channel", nx=128, ny=64, nz=128, wall=True, rbc=40,
             plt=60, rbc_points=2210, plt_points=605, delta="bspline3", precision="fp32c", call="spread"),
        # ... and the velocity half alone, bit-exact precision.
        dict(name="channel-interp-fp64", kind="couple", scene="channel", nx=128, ny=64, nz=128, wall=True, rbc=40,
             plt=60, rbc_points=2210, plt_points=605, delta="bspline3", precision="fp64", call="interp"),
        # A box whose axes are no multiples of a tile, finely sampled cells
        # that overlap each other.
        dict(name="ragged-pair-fp32c", kind="couple", scene="box", nx=90, ny=75, nz=105, wall=False, rbc=9, plt=7,
             rbc_points=8832, plt_points=1552, delta="bspline3", precision="fp32c", call="pair"),
        # The 64 x 32 x 64 um channel in FP64, both operators at one position.
        dict(name="medium-pair-fp64", kind="couple", scene="channel", nx=256, ny=128, nz=256, wall=True, rbc=412,
             plt=750, rbc_points=2210, plt_points=605, delta="bspline3", precision="fp64", call="pair"),
        # The 128 x 64 x 128 um channel at 30 % haematocrit: the headline run.
        dict(name="large-pair-fp32c", kind="couple", scene="channel", nx=512, ny=256, nz=512, wall=True, rbc=3300,
             plt=6000, rbc_points=2210, plt_points=605, delta="bspline3", precision="fp32c", call="pair"),
        # Independent uneven simulations in one graph-captured launch.
        dict(name="ensemble-pair-fp32c", kind="batch", members=24, members_seed=3, most_cells=50, call="pair",
             precision="fp32c"),
        # The serving request: interpolate, advect, spring, spread, with the
        # members' arrays bound for the step.
        dict(name="ensemble-step-fp32c", kind="batch", members=16, members_seed=8, most_cells=12, call="step",
             precision="fp32c"),
        # The implicit diffusion step of one velocity component, small box
        # and large channel.
        dict(name="diffusion-64", kind="diffusion", nx=64, ny=64, nz=64, wall=False, component=0),
        dict(name="diffusion-large", kind="diffusion", nx=512, ny=256, nz=512, wall=True, component=0),
        # The red-cell force set on RBF surfaces: 2500 data sites, 10000
        # samples per shape.
        dict(name="membrane-16", kind="membrane", data_side=50, sample_side=100, shapes=16),
    ]


def draw(rng):
    def spread_over(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    kind = rng.choice(["couple", "couple", "couple", "plane", "batch", "diffusion", "membrane"])
    if kind == "couple":
        # the axes are powers of two apart: the grid spacing is the greatest
        # common divisor of floating-point lengths
        scene = rng.choice(["box", "channel"])
        if scene == "box":
            base = spread_over(24, 110)
            sides = [base * rng.choice([1, 1, 2]) for _ in range(3)]
            cells = spread_over(1, 120)
            rbc = (cells + 1) // 2
            plt = cells - rbc
        else:
            base = 32 * rng.randint(2, 7)
            sides = [base * rng.choice([1, 2]), base, base * rng.choice([1, 2])]
            slots = (sides[0] // 32) * ((sides[1] - 4) // 13) * (sides[2] // 32)
            rbc = max(1, int(slots * rng.uniform(0.1, 0.5)))
            plt = int(8 * (slots - rbc) * rng.uniform(0.0, 0.3))
        return dict(kind="couple", scene=scene, nx=sides[0], ny=sides[1], nz=sides[2], wall=scene == "channel",
                    rbc=rbc, plt=plt, rbc_points=rng.choice([864, 2210, 8832] if scene == "box" else [864, 2210]),
                    plt_points=rng.choice([386, 605, 1552]),
                    delta=rng.choice(["bspline3"] * 5 + ["bspline2", "peskin", "roma", "cosine"]),
                    precision=rng.choice(["fp64", "fp32c"]), call=rng.choice(["two", "pair", "spread", "interp"]))
    if kind == "plane":
        side = spread_over(40, 600)
        return dict(kind="couple", scene="plane", nx=side * rng.choice([1, 2, 4]), ny=side, nz=0,
                    wall=rng.random() < 0.5, rbc=0, plt=spread_over(1, 200), rbc_points=0,
                    plt_points=spread_over(40, 400), delta=rng.choice(["roma", "bspline3", "peskin"]),
                    precision=rng.choice(["fp64", "fp32c"]), call=rng.choice(["two", "pair"]))
    if kind == "batch":
        return dict(kind="batch", members=spread_over(3, 40), members_seed=rng.randrange(1 << 30),
                    most_cells=spread_over(3, 50), call=rng.choice(["pair", "step"]),
                    precision=rng.choice(["fp32c", "fp32c", "fp64"]))
    if kind == "diffusion":
        base = spread_over(24, 140)
        sides = [base * rng.choice([1, 2]) for _ in range(3)]
        return dict(kind="diffusion", nx=sides[0], ny=sides[1], nz=sides[2], wall=rng.random() < 0.6,
                    component=rng.randrange(3))
    side = rng.choice([16, 24, 32, 50])
    return dict(kind="membrane", data_side=side, sample_side=rng.choice([side, side + 6, 2 * side]),
                shapes=spread_over(1, 40))


# ------------------------------------------------------------------ scenes
def _generator(seed):
    gen = torch.Generator(device=_device())
    gen.manual_seed(seed)
    return gen


def _device():
    return torch.device("cuda" if torch.cuda.is_available() else "cpu")


def _normal(gen, *size):
    return torch.randn(*size, generator=gen, dtype=torch.float64, device=gen.device)


def _uniform(gen, *size):
    return torch.rand(*size, generator=gen, dtype=torch.float64, device=gen.device)


def _sphere(n, device):
    """n points of a Fibonacci sphere, (n, 3)."""
    i = torch.arange(n, dtype=torch.float64, device=device) + 0.5
    z = 1.0 - 2.0 * i / n
    rho = torch.sqrt(torch.clamp(1.0 - z * z, min=0.0))
    phi = i * (math.pi * (3.0 - math.sqrt(5.0)))
    return torch.stack([rho * torch.cos(phi), rho * torch.sin(phi), z], dim=1)


def _rbc(n, device):
    """Evans-Fung biconcave disc of radius 3.91 um."""
    s = _sphere(n, device)
    r2 = torch.clamp(s[:, 0] ** 2 + s[:, 1] ** 2, max=1.0)
    h = 0.5 * 3.91 * torch.sqrt(1.0 - r2) * (0.2072 + 2.0026 * r2 - 1.1228 * r2 * r2)
    return torch.stack([3.91 * s[:, 0], 3.91 * s[:, 1], torch.sign(s[:, 2]) * h], dim=1)


def _platelet(n, device):
    return _sphere(n, device) * torch.tensor([1.8, 1.8, 0.5], dtype=torch.float64, device=device)


def _rotations(gen, n):
    q = _normal(gen, n, 4)
    w, x, y, z = (q / q.norm(dim=1, keepdim=True)).unbind(1)
    return torch.stack([1 - 2 * (y * y + z * z), 2 * (x * y - z * w), 2 * (x * z + y * w),
                        2 * (x * y + z * w), 1 - 2 * (x * x + z * z), 2 * (y * z - x * w),
                        2 * (x * z - y * w), 2 * (y * z + x * w), 1 - 2 * (x * x + y * y)], dim=1).view(n, 3, 3)


def _flat_rotations(gen, n):
    """Local z to the wall normal y with at most 5 degrees of tilt, then a full turn about y."""
    tilt = _uniform(gen, n) * math.radians(5.0)
    turn, spin = (_uniform(gen, n) * (2 * math.pi) for _ in range(2))
    zero, one = torch.zeros_like(tilt), torch.ones_like(tilt)

    def about_y(a):
        return torch.stack([a.cos(), zero, a.sin(), zero, one, zero, -a.sin(), zero, a.cos()], dim=1).view(n, 3, 3)

    tilted = torch.stack([one, zero, zero, zero, tilt.cos(), -tilt.sin(), zero, tilt.sin(), tilt.cos()],
                         dim=1).view(n, 3, 3)
    to_y = torch.tensor([[1.0, 0, 0], [0, 0, 1], [0, -1, 0]], dtype=torch.float64, device=gen.device)
    return about_y(spin) @ tilted @ about_y(turn) @ to_y


def _placed(body, rotations, centres):
    return (body[None] @ rotations.transpose(1, 2) + centres[:, None, :]).reshape(-1, body.shape[1])


def _channel_points(case, gen):
    """Non-overlapping cells in slots of 8 x 3.2 x 8 um at least 0.5 um off the
    walls: one red cell or a 2 x 2 x 2 stack of platelets per slot."""
    size = [0.25 * case[k] for k in ("nx", "ny", "nz")]
    nx, ny, nz = int(size[0] // 8.0), int((size[1] - 1.0) // 3.2), int(size[2] // 8.0)
    y0 = 0.5 * (size[1] - 3.2 * ny)
    order = torch.randperm(nx * ny * nz, generator=gen, device=gen.device)
    corner = torch.stack([(order % nx) * 8.0, y0 + (order // nx % ny) * 3.2, (order // (nx * ny)) * 8.0], dim=1)
    rbc, stacks = case["rbc"], (case["plt"] + 7) // 8
    parts = []

    def jitter(n, slack):
        return (2 * _uniform(gen, n, 3) - 1) * torch.tensor(slack, dtype=torch.float64, device=gen.device)

    half = torch.tensor([4.0, 1.6, 4.0], dtype=torch.float64, device=gen.device)
    parts.append(_placed(_rbc(case["rbc_points"], gen.device), _flat_rotations(gen, rbc),
                         corner[:rbc] + half + jitter(rbc, [0.08, 0.04, 0.08])))
    if case["plt"]:
        k = torch.arange(8, device=gen.device)
        place = torch.stack([0.5 + (k & 1), 0.5 + (k >> 1 & 1), 0.5 + (k >> 2)], dim=1).to(torch.float64) * half
        centres = (corner[rbc:rbc + stacks, None, :] + place[None]).reshape(-1, 3)[:case["plt"]]
        parts.append(_placed(_platelet(case["plt_points"], gen.device), _flat_rotations(gen, case["plt"]),
                             centres + jitter(case["plt"], [0.18, 0.12, 0.18])))
    return torch.cat(parts)


def _box_points(sides, groups, gen):
    """Cells at random centres and rotations in a periodic box; they may overlap and cross the boundary."""
    size = 0.25 * torch.tensor(sides, dtype=torch.float64, device=gen.device)
    parts = []
    for body, count in groups:
        if count:
            parts.append(_placed(body, _rotations(gen, count), _uniform(gen, count, 3) * size))
    return torch.cat(parts)


def _plane_points(case, gen):
    """Elliptic outlines (1.8 x 0.5 um) at random in a two-dimensional channel, clear of walls."""
    n, count = case["plt_points"], case["plt"]
    s = torch.arange(n, dtype=torch.float64, device=gen.device) * (2 * math.pi / n)
    body = torch.stack([1.8 * s.cos(), 0.5 * s.sin()], dim=1)
    a = _uniform(gen, count) * (2 * math.pi)
    turn = torch.stack([a.cos(), -a.sin(), a.sin(), a.cos()], dim=1).view(count, 2, 2)
    size = 0.25 * torch.tensor([case["nx"], case["ny"]], dtype=torch.float64, device=gen.device)
    margin = torch.tensor([0.0, 2.0 if case["wall"] else 0.0], dtype=torch.float64, device=gen.device)
    return _placed(body, turn, margin + _uniform(gen, count, 2) * (size - 2 * margin))


def _couple_points(case, gen):
    if case["scene"] == "channel":
        return _channel_points(case, gen)
    if case["scene"] == "plane":
        return _plane_points(case, gen)
    groups = [(_rbc(case["rbc_points"], gen.device), case["rbc"]),
              (_platelet(case["plt_points"], gen.device), case["plt"])]
    return _box_points([case["nx"], case["ny"], case["nz"]], groups, gen)


def _sides(case):
    return [case["nx"], case["ny"]] + ([case["nz"]] if case["nz"] else [])


def _operators(ibk, sides, wall):
    unit = math.gcd(*sides)
    dimensions = [ibk.Dimension(s * H, ibk.SOLID if wall and d == 1 else ibk.PERIODIC) for d, s in enumerate(sides)]
    return ibk.Mac(unit), ibk.Domain(*dimensions)


def _grid_points(sides, wall, c):
    return [s - (1 if wall and d == 1 and c == 1 else 0) for d, s in enumerate(sides)]


def _grids(sides, wall):
    return [math.prod(_grid_points(sides, wall, c)) for c in range(len(sides))]


_DELTAS = {"bspline2": ("Bspline", 2, 3), "bspline3": ("Bspline", 3, 4), "peskin": ("Peskin", None, 4),
           "roma": ("Roma", None, 3), "cosine": ("Cosine", None, 4)}


def _delta(ibk, name):
    cls, order, _ = _DELTAS[name]
    return getattr(ibk, cls)() if order is None else getattr(ibk, cls)(order)


def _couple_inputs(case, seed):
    gen = _generator(seed)
    sides = _sides(case)
    x = (_couple_points(case, gen) * UM).t().contiguous().view(-1)
    f = _normal(gen, x.numel()) * PN
    u = [_normal(gen, s) * UM_PER_S for s in _grids(sides, case["wall"])]
    if case["wall"]:
        # a Poiseuille profile along x of at most 100 um/s over the noise
        y = (torch.arange(sides[1], dtype=torch.float64, device=gen.device) + 0.5) / sides[1]
        u[0].view(-1, sides[1], sides[0]).add_((400.0 * UM_PER_S * y * (1 - y))[None, :, None])
    return x, f, u


MEMBER_SIDES = (32, 48, 64, 96, 128)
MEMBER_CELLS = (("rbc", 864), ("rbc", 2210), ("rbc", 8832), ("plt", 386), ("plt", 1552))


def _members(case):
    """(side, {(kind, points): count}) of each member: the shape of the case, whatever the inputs' seed."""
    gen = torch.Generator()
    gen.manual_seed(case["members_seed"])

    def pick(n):
        return int(torch.randint(n, (1,), generator=gen))

    members = []
    for _ in range(case["members"]):
        side = MEMBER_SIDES[pick(len(MEMBER_SIDES))]
        cells = {}
        for _ in range(1 + pick(case["most_cells"])):
            which = MEMBER_CELLS[pick(len(MEMBER_CELLS))]
            cells[which] = cells.get(which, 0) + 1
        members.append((side, cells))
    return members


def _member_inputs(case, seed):
    gen = _generator(seed)
    out = []
    for side, cells in _members(case):
        groups = [((_rbc if kind == "rbc" else _platelet)(n, gen.device), count)
                  for (kind, n), count in sorted(cells.items())]
        x = (_box_points([side] * 3, groups, gen) * UM).t().contiguous().view(-1)
        # a step finds the springs stretched by about a tenth of a grid cell
        out.append((side, x, _normal(gen, x.numel()) * PN, [_normal(gen, side ** 3) * UM_PER_S for _ in range(3)],
                    x + 0.1 * H * _normal(gen, x.numel())))
    return out


def _diffusion_inputs(case, seed):
    gen = _generator(seed)
    n = math.prod(_grid_points(_sides(case), case["wall"], case["component"]))
    return tuple(_normal(gen, n) for _ in range(3))


def _fourier(ns, nd, device):
    """Evaluation, first and second derivative (ns x nd) of a trigonometric
    interpolant on nd equispaced sites (nd even), at ns equispaced samples."""
    a = 2 * math.pi * (torch.arange(ns, dtype=torch.float64, device=device)[:, None] / ns
                       - torch.arange(nd, dtype=torch.float64, device=device)[None, :] / nd)
    ops = [torch.full_like(a, 1.0 / nd), torch.zeros_like(a), torch.zeros_like(a)]
    for k in range(1, nd // 2 + 1):
        w = (2.0 if k < nd // 2 else 1.0) / nd
        ops[0] += w * torch.cos(k * a)
        if k < nd // 2:
            ops[1] -= w * k * torch.sin(k * a)
        ops[2] -= w * k * k * torch.cos(k * a)
    return ops


def _surface_operators(ns, nd, device):
    """The six operators of the periodic (u, v) grid, u fastest."""
    e, d, dd = _fourier(ns, nd, device)
    return [torch.kron(e, e), torch.kron(e, d), torch.kron(d, e), torch.kron(e, dd), torch.kron(d, d),
            torch.kron(dd, e)]


def _surface_weights(side, device):
    return torch.full((side * side,), (2 * math.pi / side) ** 2, dtype=torch.float64, device=device)


def _membrane_inputs(case, seed):
    """Rest and deformed positions and the velocity at the data sites of tori about the size of a red cell."""
    gen = _generator(seed)
    side, nc = case["data_side"], case["shapes"]
    t = 2 * math.pi * torch.arange(side, dtype=torch.float64, device=gen.device) / side
    v, u = (a.reshape(-1) for a in torch.meshgrid(t, t, indexing="ij"))
    big, small = 0.28 + 0.02 * _uniform(gen, nc, 1), 0.10 + 0.01 * _uniform(gen, nc, 1)
    rho = big + small * torch.cos(v)
    rest = torch.stack([rho * torch.cos(u), rho * torch.sin(u), small * torch.sin(v)])
    stretch = torch.eye(3, dtype=torch.float64, device=gen.device) + 0.05 * _normal(gen, nc, 3, 3)
    moved = torch.einsum("mij,jms->ims", stretch, rest)
    bump = torch.stack([torch.sin(v), torch.cos(2 * u), torch.sin(u + v)])
    moved = moved + 0.01 * _uniform(gen, 1, nc, 1) * bump[:, None, :]
    velocity = torch.einsum("mij,jms->ims", 0.01 * _normal(gen, nc, 3, 3), moved) + 1e-3 * bump[:, None, :]
    return rest.reshape(-1), moved.reshape(-1), velocity.reshape(-1)


# ---------------------------------------------------------- prepare and run
def prepare(case, seed):
    ibk = _package()
    ibk.lib()
    return {"couple": _prepare_couple, "batch": _prepare_batch, "diffusion": _prepare_diffusion,
            "membrane": _prepare_membrane}[case["kind"]](ibk, case, seed)


def run(state):
    return state["run"](state)


def _precision(ibk, case):
    return ibk.FP32C if case["precision"] == "fp32c" else ibk.FP64


def _prepare_couple(ibk, case, seed):
    x, f, u = _couple_inputs(case, seed)
    sides = _sides(case)
    tag, domain = _operators(ibk, sides, case["wall"])
    delta, precision = _delta(ibk, case["delta"]), _precision(ibk, case)
    n = x.numel() // len(sides)
    state = dict(n=n, x=x, f=f, u=u, fe=[torch.zeros_like(c) for c in u], ul=torch.zeros_like(x))
    if case["call"] == "pair":
        state.update(plan=ibk.Plan(tag, domain, delta, precision), run=_run_pair)
        state["plan"].reserve(n)
    if case["call"] in ("two", "spread"):
        state["spread"] = ibk.Spread(tag, domain, delta, precision)
    if case["call"] in ("two", "interp"):
        state["interpolate"] = ibk.Interpolate(tag, domain, delta, precision)
    state.setdefault("run", {"two": _run_two, "spread": _run_spread, "interp": _run_interp}.get(case["call"]))
    return state


def _run_pair(s):
    s["plan"].spread_interpolate(s["n"], s["x"], s["f"], s["fe"], s["u"], s["ul"])
    return s["fe"] + [s["ul"]]


def _run_two(s):
    s["spread"](s["n"], s["x"], s["f"], s["fe"])
    s["interpolate"](s["n"], s["x"], s["u"], s["ul"])
    return s["fe"] + [s["ul"]]


def _run_spread(s):
    s["spread"](s["n"], s["x"], s["f"], s["fe"])
    return s["fe"]


def _run_interp(s):
    return s["interpolate"](s["n"], s["x"], s["u"], s["ul"])


def _prepare_batch(ibk, case, seed):
    inputs = _member_inputs(case, seed)
    instances = [ibk.Instance(*_operators(ibk, [side] * 3, False)) for side, *_ in inputs]
    total = sum(x.numel() // 3 for _, x, *_ in inputs)
    batch = ibk.Batch(instances, ibk.Bspline(3), _precision(ibk, case), max_points=total)
    # the members' results lie back to back in one buffer per field
    results = dict(fe=3 * sum(side ** 3 for side, *_ in inputs))
    results.update(dict(xn=3 * total, fs=3 * total) if case["call"] == "step" else dict(ul=3 * total))
    results = {key: torch.zeros(n, dtype=torch.float64, device=inputs[0][1].device) for key, n in results.items()}
    fe = results["fe"].split([side ** 3 for side, *_ in inputs for _ in range(3)])
    points = {key: buffer.split([x.numel() for _, x, *_ in inputs]) for key, buffer in results.items() if key != "fe"}
    io = []
    for i, (_, x, f, u, xref) in enumerate(inputs):
        io.append(dict(n=x.numel() // 3, x=x, fe=fe[3 * i:3 * i + 3], ue=u, **{key: p[i] for key, p in points.items()}))
        io[-1].update(dict(xref=xref) if case["call"] == "step" else dict(fl=f))
    if case["call"] == "step":
        batch.set_step(STEP_DT, STEP_K)
        op, go = ibk.OP_STEP, _run_batch_step
    else:
        op, go = ibk.OP_SPREAD_INTERPOLATE, _run_batch_pair
    batch.bind(io)
    batch.capture(op)
    return dict(batch=batch, io=io, op=op, results=list(results.values()), run=go)


def _run_batch_pair(s):
    s["batch"].run(s["op"])
    return s["results"]


def _run_batch_step(s):
    # a simulation swaps its position buffers every step, so it binds every step
    s["batch"].bind(s["io"])
    s["batch"].run(s["op"])
    return s["results"]


def _prepare_diffusion(ibk, case, seed):
    u, rhs, f = _diffusion_inputs(case, seed)
    tag, domain = _operators(ibk, _sides(case), case["wall"])
    plan = ibk.Plan(tag, domain, ibk.Bspline(3), ibk.FP64)
    solver = ibk.Diffusion(plan, case["component"], TIMESTEP, VISCOSITY, tolerance=TOLERANCE, max_iterations=5000)
    return dict(plan=plan, solver=solver, u=u, rhs=rhs, f=f, run=_run_diffusion)


def _run_diffusion(s):
    return s["solver"].step(s["u"], s["rhs"], s["f"], gamma=1.0)


def _prepare_membrane(ibk, case, seed):
    rest, moved, velocity = _membrane_inputs(case, seed)
    nd, ns, nc = case["data_side"], case["sample_side"], case["shapes"]
    samples = ibk.SurfacePlan(_surface_operators(ns, nd, rest.device), _surface_weights(ns, rest.device))
    sites = ibk.SurfacePlan([None] + _surface_operators(nd, nd, rest.device)[1:], _surface_weights(nd, rest.device))
    return dict(ibk=ibk, samples=samples, sites=sites, rest=samples.geometry(rest, nc), x=moved, v=velocity, nc=nc,
                run=_run_membrane)


def _run_membrane(s):
    ibk, nc = s["ibk"], s["nc"]
    current = s["samples"].geometry(s["x"], nc)
    return [current[key] for key in ("position", "tu", "tv", "tuu", "tuv", "tvv", "normal", "sigma")] + [
            ibk.membrane_tension(ibk.SKALAK, SHEAR, BULK, s["rest"], current),
            ibk.membrane_bending(s["sites"], s["samples"], BENDING, False, None, s["x"], None, current, nc),
            ibk.membrane_dissipation(s["samples"], VISCOUS, s["v"], current, nc)]


# -------------------------------------------------------------------- exact
def exact(case, seed):
    return {"couple": _exact_couple, "batch": _exact_batch, "diffusion": _exact_diffusion,
            "membrane": _exact_membrane}[case["kind"]](case, seed)


def _phi(name, r):
    s = r.abs()

    def root(v):
        return torch.sqrt(torch.clamp(v, min=0.0))

    if name.startswith("bspline"):
        def spline(n, t):
            if n == 0:
                return ((t >= -0.5) & (t < 0.5)).to(t.dtype)
            b = (n + 1.0) / (2.0 * n)
            return (b + t / n) * spline(n - 1, t + 0.5) + (b - t / n) * spline(n - 1, t - 0.5)
        return spline(int(name[-1]), r)
    if name == "peskin":
        near = (3 - 2 * s + root(1 + 4 * s - 4 * s * s)) / 8
        far = (5 - 2 * s - root(-7 + 12 * s - 4 * s * s)) / 8
        return torch.where(s < 1, near, far)
    if name == "roma":
        near = (1 + root(1 - 3 * s * s)) / 3
        far = (5 - 3 * s - root(1 - 3 * (1 - s) ** 2)) / 6
        return torch.where(s < 0.5, near, torch.where(s < 1.5, far, torch.zeros_like(s)))
    return (1 + torch.cos(0.5 * math.pi * r)) / 4


def _stencils(x, sides, wall, c, delta):
    """Per axis: first node, weights (one per node) and the axis' grid size of component c's stencils."""
    width = _DELTAS[delta][2]
    out = []
    for d, pts in enumerate(_grid_points(sides, wall, c)):
        shift = (1.0 if wall and d == 1 else 0.0) if d == c else 0.5
        t = x[d] / H - shift
        first = torch.floor(t + 0.5 * (width & 1)) - (width - 1) // 2
        out.append((first.long(), [_phi(delta, first + m - t) for m in range(width)], pts, wall and d == 1))
    return out


def _nodes(stencils):
    """Every stencil entry: weight, clamped flat index and whether the node is on the grid."""
    def walk(d):
        if d < 0:
            yield None, 0, None
            return
        first, weights, pts, solid = stencils[d]
        for w, index, inside in walk(d - 1):
            stride = math.prod(s[2] for s in stencils[:d])
            for m, wm in enumerate(weights):
                j = first + m
                on = None
                if solid:
                    on = (j >= 0) & (j < pts)
                    j = j.clamp(0, pts - 1)
                else:
                    j = j % pts
                both = inside if on is None else (on if inside is None else on & inside)
                yield (wm if w is None else w * wm), index + j * stride, both
    return walk(len(stencils) - 1)


def _exact_pair(x, f, u, sides, wall, delta):
    """Force grids (when f is given) and point velocities (when u is)."""
    dims = len(sides)
    x = x.view(dims, -1)
    spread, velocity = [], []
    for c in range(dims):
        stencils = _stencils(x, sides, wall, c, delta)
        grid = torch.zeros(math.prod(s[2] for s in stencils), dtype=x.dtype, device=x.device)
        at = torch.zeros_like(x[c])
        for w, index, inside in _nodes(stencils):
            if f is not None:
                term = w * f.view(dims, -1)[c] / H ** dims
                grid.index_add_(0, index, term if inside is None else torch.where(inside, term, 0.0))
            if u is not None:
                at += w * u[c][index]
        spread.append(grid)
        velocity.append(at)
    return spread if f is not None else None, torch.cat(velocity) if u is not None else None


def _exact_couple(case, seed):
    x, f, u = _couple_inputs(case, seed)
    call = case["call"]
    fe, ul = _exact_pair(x, None if call == "interp" else f, None if call == "spread" else u, _sides(case),
                         case["wall"], case["delta"])
    return ul if call == "interp" else fe if call == "spread" else fe + [ul]


def _exact_batch(case, seed):
    grids, points = [], []
    for side, x, f, u, xref in _member_inputs(case, seed):
        if case["call"] == "pair":
            fe, ul = _exact_pair(x, f, u, [side] * 3, False, "bspline3")
            points.append((ul,))
        else:
            _, ul = _exact_pair(x, None, u, [side] * 3, False, "bspline3")
            xn = x + STEP_DT * ul
            fs = -STEP_K * (xn - xref)
            fe, _ = _exact_pair(xn, fs, None, [side] * 3, False, "bspline3")
            points.append((xn, fs))
        grids += fe
    return [torch.cat(grids)] + [torch.cat(p) for p in zip(*points)]


def _exact_diffusion(case, seed):
    """(I - lambda L)^-1 through the generalised eigenvectors of each axis:
    V' I V = 1, V' L V = D turn it into a division."""
    u, rhs, f = _diffusion_inputs(case, seed)
    pts = _grid_points(_sides(case), case["wall"], case["component"])
    lap, ident, vecs, vals = [], [], [], []
    for d, n in enumerate(pts):
        i = torch.arange(n, device=u.device)
        m = torch.zeros(n, n, dtype=u.dtype, device=u.device)
        m[i, i] = -2.0
        m[i[1:], i[:-1]] = 1.0
        m[i[:-1], i[1:]] = 1.0
        w = torch.ones(n, dtype=u.dtype, device=u.device)
        if not (case["wall"] and d == 1):
            m[0, -1] += 1.0
            m[-1, 0] += 1.0
        elif case["component"] != 1:
            # Dirichlet walls half a cell off the first and last faces
            m[0, 0] -= 1.0
            m[-1, -1] -= 1.0
            w[0] -= 0.25
            w[-1] -= 0.25
        m /= H * H
        s = w.rsqrt()
        e, v = torch.linalg.eigh(s[:, None] * m * s[None, :])
        lap.append(m)
        ident.append(w)
        vals.append(e)
        vecs.append(s[:, None] * v)

    def along(a, q, d):                 # the matrix q along axis d of the grid (x fastest)
        n0, n1, n2 = pts
        if d == 0:
            return (a.view(-1, n0) @ q.t()).view(-1)
        if d == 1:
            return torch.matmul(q, a.view(n2, n1, n0)).reshape(-1)
        return (q @ a.view(n2, -1)).view(-1)

    def scaled(a, axes):
        a = a.view(pts[2], pts[1], pts[0])
        for d in axes:
            a = a * ident[d].view([-1 if 2 - k == d else 1 for k in range(3)])
        return a.reshape(-1)

    lu = scaled(along(u, lap[0], 0), (1, 2)) + scaled(along(u, lap[1], 1), (0, 2)) + scaled(along(u, lap[2], 2), (0, 1))
    b = TIMESTEP * scaled(f, (0, 1, 2)) + TIMESTEP * VISCOSITY * (lu + rhs)
    for d in range(3):
        b = along(b, vecs[d].t().contiguous(), d)
    total = vals[2][:, None, None] + vals[1][None, :, None] + vals[0][None, None, :]
    b = (b.view(pts[2], pts[1], pts[0]) / (1.0 - 0.5 * TIMESTEP * VISCOSITY * total)).view(-1)
    for d in range(3):
        b = along(b, vecs[d], d)
    return u + b


def _dot(a, b):
    return (a * b).sum(0)


def _metric(g):
    """First fundamental form (e, f, g), its u and v derivatives, and the same of its determinant."""
    tu, tv, tuu, tuv, tvv = g
    e = (_dot(tu, tu), _dot(tu, tv), _dot(tv, tv))
    eu = (2 * _dot(tuu, tu), _dot(tuu, tv) + _dot(tuv, tu), 2 * _dot(tuv, tv))
    ev = (2 * _dot(tuv, tu), _dot(tuv, tv) + _dot(tvv, tu), 2 * _dot(tvv, tv))
    det = e[0] * e[2] - e[1] ** 2

    def rate(r):
        return r[0] * e[2] + e[0] * r[2] - 2 * e[1] * r[1]
    return e, eu, ev, det, rate(eu), rate(ev)


def _divergence(stress, stress_u, stress_v, g, det, det_u, det_v):
    """c_u t_u + c_v t_v + s^ij t_ij with c_j = d_i s^ij - s^ij d_i det / (2 det), s = (uu, uv, vv)."""
    cu = stress_u[0] + stress_v[1] - (det_u * stress[0] + det_v * stress[1]) / (2 * det)
    cv = stress_u[1] + stress_v[2] - (det_u * stress[1] + det_v * stress[2]) / (2 * det)
    tu, tv, tuu, tuv, tvv = g
    return cu * tu + cv * tv + stress[0] * tuu + 2 * stress[1] * tuv + stress[2] * tvv


def _adj(m):
    return (m[2], -m[1], m[0])


def _exact_membrane(case, seed):
    rest, moved, velocity = _membrane_inputs(case, seed)
    nd, ns, nc = case["data_side"], case["sample_side"], case["shapes"]
    ops = _surface_operators(ns, nd, rest.device)
    site_ops = _surface_operators(nd, nd, rest.device)

    def apply(q, y, rows):              # operator q on [component][shape][site] values
        return (y.view(-1, nd * nd) @ q.t()).view(-1, nc * rows * rows)

    def normal(g):
        c = torch.linalg.cross(g[0], g[1], dim=0)
        return c / c.norm(dim=0), c.norm(dim=0)

    weights = _surface_weights(ns, rest.device).repeat(nc)
    g0 = [apply(q, rest, ns) for q in ops[1:]]
    g1 = [apply(q, moved, ns) for q in ops[1:]]
    n1, area = normal(g1)
    sigma0, sigma1 = weights * normal(g0)[1], weights * area

    # Skalak tension: s = w1 adj(rest metric) + w2 adj(current metric), over
    # the rest metric's determinant
    m0, m0u, m0v, d0, d0u, d0v = _metric(g0)
    m1, m1u, m1v, d1, d1u, d1v = _metric(g1)

    def mixed(a, b):
        return a[0] * b[2] + a[2] * b[0] - 2 * a[1] * b[1]

    i1, i2 = mixed(m1, m0) / d0, d1 / d0
    i1r = [(mixed(mr, m0) + mixed(m1, m0r) - i1 * d0r) / d0 for mr, m0r, d0r in ((m1u, m0u, d0u), (m1v, m0v, d0v))]
    i2r = [(d1r - i2 * d0r) / d0 for d1r, d0r in ((d1u, d0u), (d1v, d0v))]
    w1, w2 = SHEAR * (i1 - 1), BULK * (i2 - 1) - SHEAR
    stress = [w1 * a + w2 * b for a, b in zip(_adj(m0), _adj(m1))]
    rates = []
    for r, (m0r, m1r) in enumerate(((m0u, m1u), (m0v, m1v))):
        rates.append([SHEAR * i1r[r] * a + w1 * ar + BULK * i2r[r] * b + w2 * br
                      for a, ar, b, br in zip(_adj(m0), _adj(m0r), _adj(m1), _adj(m1r))])
    tension = sigma0 / d0 * _divergence(stress, rates[0], rates[1], g1, d0, d0u, d0v)

    # bending: the surface Laplacian of the mean curvature and its cubic terms
    def curvature(g, nrm):
        e, k = (_dot(g[0], g[0]), _dot(g[0], g[1]), _dot(g[1], g[1])), [_dot(t, nrm) for t in g[2:]]
        det = e[0] * e[2] - e[1] ** 2
        return (k[0] * e[2] + k[2] * e[0] - 2 * k[1] * e[1]) / (2 * det), (k[0] * k[2] - k[1] ** 2) / det

    sites = [apply(q, moved, nd) for q in site_ops[1:]]
    mean = curvature(sites, normal(sites)[0])[0]
    hu, hv, huu, huv, hvv = (apply(q, mean, ns).view(-1) for q in ops[1:])
    e, f, g = m1
    laplacian = (((-d1u * g + d1v * f) / (2 * d1) + m1u[2] - m1v[1]) / d1 * hu
                 + ((d1u * f - d1v * e) / (2 * d1) - m1u[1] + m1v[0]) / d1 * hv
                 + (g * huu - 2 * f * huv + e * hvv) / d1)
    h, k = curvature(g1, n1)
    bending = -4 * sigma1 * BENDING * (laplacian + 2 * h * (h * h - k)) * n1

    # dissipation: the stress g^-1 g' adj(g) = adj(g) g' adj(g) / det of the metric's rate g'
    v = [apply(q, velocity, ns) for q in ops[1:]]
    su, sv, suu, suv, svv = v
    tu, tv, tuu, tuv, tvv = g1
    rate = (2 * _dot(tu, su), _dot(tu, sv) + _dot(su, tv), 2 * _dot(tv, sv))

    def both(a, b, c, d):
        return _dot(a, b) + _dot(c, d)

    rate_u = (2 * both(suu, tu, tuu, su), both(suu, tv, tuu, sv) + both(suv, tu, tuv, su), 2 * both(suv, tv, tuv, sv))
    rate_v = (2 * both(suv, tu, tuv, su), both(suv, tv, tuv, sv) + both(svv, tu, tvv, su), 2 * both(svv, tv, tvv, sv))

    def full(a):
        return [[a[0], a[1]], [a[1], a[2]]]

    def product(a, b):
        return [[sum(a[i][k] * b[k][j] for k in range(2)) for j in range(2)] for i in range(2)]

    adj, adj_u, adj_v = (full(_adj(m)) for m in (m1, m1u, m1v))

    def sandwich(a, b, c):
        p = product(product(a, b), c)
        return (p[0][0], 0.5 * (p[0][1] + p[1][0]), p[1][1])

    raw = sandwich(adj, full(rate), adj)
    pif = [s / d1 for s in raw]
    pif_rates = []
    for adj_r, rate_r, d1r in ((adj_u, rate_u, d1u), (adj_v, rate_v, d1v)):
        parts = (sandwich(adj_r, full(rate), adj), sandwich(adj, full(rate_r), adj), sandwich(adj, full(rate), adj_r))
        pif_rates.append([(a + b + c - p * d1r) / d1 for a, b, c, p in zip(*parts, pif)])
    dissipation = sigma1 * VISCOUS / d1 * _divergence(pif, pif_rates[0], pif_rates[1], g1, d1, d1u, d1v)
    outs = [apply(ops[0], moved, ns)] + g1 + [n1, sigma1, tension, bending, dissipation]
    return [t.reshape(-1) for t in outs]


# --------------------------------------------------------------------- work
def _coupling_work(n, faces, dims, width, spreads, interpolations):
    """Positions once, forces and velocities per point and every face once;
    a product and an addition per stencil entry and component, and the weights' products."""
    nodes = width ** dims
    return (8 * (dims * n * (1 + spreads + interpolations) + faces * (spreads + interpolations)),
            n * dims * 3 * nodes * (spreads + interpolations))


def work(case):
    if case["kind"] == "couple":
        sides = _sides(case)
        n = case["rbc"] * case["rbc_points"] + case["plt"] * case["plt_points"]
        spreads, interpolations = {"spread": (1, 0), "interp": (0, 1)}.get(case["call"], (1, 1))
        b, f = _coupling_work(n, sum(_grids(sides, case["wall"])), len(sides), _DELTAS[case["delta"]][2], spreads,
                              interpolations)
    elif case["kind"] == "batch":
        b = f = 0
        for side, cells in _members(case):
            n = sum(points * count for (_, points), count in cells.items())
            mb, mf = _coupling_work(n, 3 * side ** 3, 3, 4, 1, 1)
            # a step reads positions and rest positions and writes new positions and forces
            b += mb + (8 * 3 * n if case["call"] == "step" else 0)
            f += mf
    elif case["kind"] == "diffusion":
        n = math.prod(_grid_points(_sides(case), case["wall"], case["component"]))
        # u, rhs, f and the result; one operator and one degree-4 polynomial
        # of it per iteration, about a dozen iterations
        b, f = 32 * n, 12 * (4 * 13 + 12) * n
    else:
        nd, ns, nc = case["data_side"] ** 2, case["sample_side"] ** 2, case["shapes"]
        f = 2 * nd * nc * (ns * (6 * 3 + 5 + 5 * 3) + nd * 5 * 3)
        b = 8 * (6 * ns * nd + 5 * nd * nd + nc * (2 * 3 * nd + ns * (22 + 16 + 9)))
    return {"bytes": b, "flops": f}
