"""What a user of this package has it do on the GPU, as cases that can be timed and compared: the model step of single runs,
ensembles and uneven batches in each microphysics configuration, the host round trip, the serving loop, and the field
solves beside the step (the storm's electric potential, the terrain's projection and transport faces).

Sizes are the repository's own: the standard 40x32x50, large 80x64x50 and stress 320x256x80 grids, the 64-member
ensemble, the uneven batch of a regime grid, and ragged grids between them. Runs start from seeded mature storms written
down analytically (updraught cores, cloud, rain, snow, graupel and hail with compact support, a cold pool, noise), so the
microphysics, the sedimentation and the transport meet what they meet fifteen to thirty minutes into a run. A pass of a
step case writes the runs' states from pinned host memory, advances them a few steps and reads them back: each pass does
the same work on the same inputs.

``exact`` gives the 64-bit values of the field solves (numpy, no code of this package). A whole model step has no such
short restatement: its outputs are compared between versions only.
"""
import math

import numpy as np
import torch

from meteolab_gb300.environment import Environment, SliderConfig
from meteolab_gb300.grid import GridOptions, create_grid
from meteolab_gb300.runtime import Context, ElectricSolver, MaskedProjection, Server, TerrainFaces
from meteolab_gb300.scenarios import (CARRIED, CHARGES, ICE2M, RunSpec, Switches, baseline_profile, exponential_ice_moments,
                                      marshall_palmer_number)

DT = 3.0
HEIGHT = 18_900.0
STANDARD, LARGE, STRESS = "40x32x50", "80x64x50", "320x256x80"


def listed():
    return [
        # One storm stepped for a viewer: the smallest step, bound by launches and the latency of its kernels.
        dict(name="single_standard", kind="step", grids=STANDARD, dx=1200.0, steps=4, moments=1, lightning=0),
        # The 64-member ensemble on the standard grid: the throughput configuration.
        dict(name="ensemble64_standard", kind="step", grids=STANDARD + "*64", dx=1200.0, steps=4, moments=1, lightning=0),
        # The large domain of one run.
        dict(name="single_large", kind="step", grids=LARGE, dx=1200.0, steps=4, moments=1, lightning=0),
        # The bandwidth stress grid: 6.6 million nodes at 300 m, the row path of the spectral solves.
        dict(name="single_stress", kind="step", grids=STRESS, dx=300.0, steps=2, moments=1, lightning=0),
        # An uneven batch in one set of launches: the regime grid's two sizes and two ragged ones.
        dict(name="uneven_batch", kind="step", grids=STANDARD + "*12," + LARGE + "*4,36x45x40*2,50x42x33*2", dx=1200.0, steps=3,
             moments=1, lightning=0),
        # An ensemble in the two-moment configuration (rain, graupel and hail numbers and volumes).
        dict(name="ensemble32_two_moment", kind="step", grids=STANDARD + "*32", dx=1200.0, steps=2, moments=2, lightning=0),
        # Electrified storms whose charge breaks down: the charging, and the flashes after each step.
        dict(name="electrified16", kind="step", grids=STANDARD + "*16", dx=1200.0, steps=2, moments=1, lightning=1),
        # The reference engine's host round trip every step, for the ensemble (the members in four pipelined groups).
        dict(name="round_trips64", kind="round_trips", grids=STANDARD + "*64", dx=1200.0, steps=4, groups=4),
        # The serving loop: four requests of uneven sizes and lengths, admitted, stepped, collected and retired.
        dict(name="serve4", kind="serve", grids=STANDARD + "*2," + LARGE + ",36x45x40", dx=1200.0, steps=6, quantum=4),
        # The electric potential of one charge distribution (a lightning viewer's field), host arrays in and out.
        dict(name="electric_standard", kind="electric", grids=STANDARD, dx=1200.0),
        # The terrain's pressure projection of one stage over a hill on the large domain.
        dict(name="projection_large", kind="projection", grids=LARGE, dx=1200.0, form="hill", height=1.0, width=5.0),
        # The transport's face fluxes over a hill on the standard domain.
        dict(name="faces_standard", kind="faces", grids=STANDARD, dx=1200.0, form="hill", height=1.0, width=5.0),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    """One more case of the listed ones' ranges: every kind, sizes from a few thousand nodes to 4 million, odd ones too."""
    kind = rng.choice(["step", "step", "step", "step", "round_trips", "serve", "electric", "projection", "faces"])
    nx, ny, nz = _log_int(rng, 16, 160), _log_int(rng, 12, 128), rng.randint(20, 80)
    dx = rng.choice([1200.0, 600.0, 300.0])
    if kind == "step":
        lightning = int(rng.random() < .2)
        moments = rng.choice([1, 1, 2])
        most = 600_000 if lightning else 2_000_000 if moments == 2 else 4_000_000
        runs = max(1, min(_log_int(rng, 1, 64), 8 if lightning else 64, most // (nx * ny * nz)))
        return dict(kind=kind, grids=f"{nx}x{ny}x{nz}*{runs}", dx=dx, steps=1 if lightning else rng.randint(1, 4), moments=moments,
                    lightning=lightning)
    if kind == "round_trips":
        runs = max(1, min(_log_int(rng, 1, 64), 4_000_000 // (nx * ny * nz)))
        return dict(kind=kind, grids=f"{nx}x{ny}x{nz}*{runs}", dx=dx, steps=rng.randint(1, 4), groups=rng.choice([1, 2, 4]))
    if kind == "serve":
        other = f"{_log_int(rng, 16, 80)}x{_log_int(rng, 12, 64)}x{rng.randint(20, 60)}"
        return dict(kind=kind, grids=f"{min(nx, 80)}x{min(ny, 64)}x{min(nz, 60)}*2,{other}", dx=dx, steps=rng.randint(3, 10), quantum=rng.randint(1, 4))
    if kind == "electric":
        return dict(kind=kind, grids=f"{nx}x{ny}x{nz}", dx=dx)
    form = rng.choice(["hill", "ridge", "plateau", "schar"])
    nx, ny, nz = min(nx, 80), min(ny, 64), min(nz, 50)
    return dict(kind=kind, grids=f"{nx}x{ny}x{nz}", dx=1200.0, form=form, height=round(rng.uniform(.3, 1.0), 2), width=round(rng.uniform(4.0, 8.0), 1))


# ------------------------------------------------------------------------------------------------ inputs
_ctx = None


def _context():
    """The process's one device context, as a user's program keeps it."""
    global _ctx
    if _ctx is None:
        _ctx = Context()
    return _ctx


def _grids(case):
    out = []
    for part in case["grids"].split(","):
        dims, _, count = part.partition("*")
        nx, ny, nz = (int(v) for v in dims.split("x"))
        dx = case["dx"]
        grid = create_grid(GridOptions(nx, ny, nz, nx * dx, ny * dx * .9375, HEIGHT, 100.0))
        out += [grid] * int(count or 1)
    return out


def _qsat(t, p):
    es = 611.2 * torch.exp(17.67 * t / (t + 243.5))
    return .622 * es / (p - es).clamp(min=1.0)


def _storm(grid, env, gen, rng, moments, lightning):
    """A mature storm on `grid` in the environment `env`: one or two cells per 50 km square, each an updraught core with
    its cloud and precipitation shafts, an anvil and a cold pool. Fields as float32 host arrays by name."""
    nx, ny, nz = grid.nx, grid.ny, grid.nz
    dev, f64 = "cuda", torch.float64
    level = lambda a: torch.as_tensor(np.asarray(a), dtype=f64, device=dev).reshape(nz, 1, 1)
    z = level(grid.zs)
    rho, exner, p = level(env.rho), level(env.exner), level(env.p)
    theta0, q0 = level(env.theta), level(env.q)
    x = (torch.arange(nx, device=dev, dtype=f64) * grid.dx).reshape(1, 1, nx)
    y = (torch.arange(ny, device=dev, dtype=f64) * grid.dy).reshape(1, ny, 1)
    zero = torch.zeros((nz, ny, nx), device=dev, dtype=f64)
    f = {k: zero.clone() for k in CARRIED}
    f["theta"] += theta0
    f["q"] += q0
    f["u"] += level(env.u)
    f["v"] += level(env.v)
    charge = zero.clone()

    def bump(a, lo, mid, hi):   # a cosine hump over the heights lo..hi, 1 at mid
        s = torch.where(a < mid, (a - mid) / (mid - lo), (a - mid) / (hi - mid)).clamp(-1, 1)
        return torch.cos(.5 * math.pi * s) ** 2

    cells = max(1, min(12, round(grid.width * grid.depth / 50_000.0 ** 2 * rng.uniform(1, 2))))
    for _ in range(cells):
        cx, cy = rng.uniform(0, grid.width), rng.uniform(0, grid.depth)
        # the core's radius, at most an eighth of the domain and at least two grid lengths
        radius = max(2 * grid.dx, min(rng.uniform(3_000, 6_000), .125 * max(grid.width, grid.depth)))
        strength, lean = rng.uniform(.5, 1.0), rng.uniform(.1, .4)

        def disc(shift, r):  # a cosine disc of radius r, leaning downshear, periodic
            dx = x - cx - shift
            dy = y - cy
            dx = dx - grid.width * torch.round(dx / grid.width)
            dy = dy - grid.depth * torch.round(dy / grid.depth)
            return torch.cos(.5 * math.pi * (torch.sqrt(dx * dx + dy * dy) / r).clamp(max=1.0)) ** 2
        core, shaft = disc(lean * z, radius), disc(lean * z + .6 * radius, 1.2 * radius)
        anvil, pool = disc(1.5 * lean * z, 2.2 * radius), disc(radius, 2.5 * radius)
        f["w"] += strength * (22 * core * bump(z, 0, 6_500, 13_500) - 4 * shaft * bump(z, 0, 1_500, 4_500))
        f["theta"] += strength * (4 * core * bump(z, 1_000, 6_500, 12_500) - 4 * pool * bump(z, -1_800, 0, 1_800))
        f["cold"] += 4 * strength * pool * bump(z, -1_500, 0, 1_500)
        f["cloud"] += strength * 1.8e-3 * core * bump(z, 900, 4_000, 9_000)
        f["rain"] += strength * 2.5e-3 * shaft * bump(z, -2_500, 1_200, 5_500)
        f["snow"] += strength * 1.2e-3 * anvil * bump(z, 4_200, 8_500, 12_500)
        f["graupel"] += strength * 3.0e-3 * (.5 * core + .5 * shaft) * bump(z, 2_500, 6_000, 10_500)
        f["hail"] += strength * 1.5e-3 * shaft * bump(z, -500, 4_000, 8_500)
        f["ice"] += strength * 3.0e-4 * anvil * bump(z, 5_500, 10_000, 13_000)
        f["iceNumber"] += strength * 6.0e5 * anvil * bump(z, 5_500, 10_000, 13_000)
        t = f["theta"] * exner - 273.15
        wet = core * bump(z, 300, 4_000, 11_000)
        f["q"] = f["q"] + (wet > 0) * (.5 + .5 * wet) * (1.005 * _qsat(t, p) - f["q"]).clamp(min=0.0) * (wet > .05)
        f["u"] += strength * 5 * pool * bump(z, -1_500, 0, 1_500) * torch.sin(2 * math.pi * (x - cx) / grid.width)
        swirl = core * bump(z, 500, 4_500, 9_000) * strength * 9
        f["u"] -= swirl * torch.sin(2 * math.pi * (y - cy) / grid.depth).clamp(-.5, .5) * 2
        f["v"] += swirl * torch.sin(2 * math.pi * (x - cx) / grid.width).clamp(-.5, .5) * 2
        charge += strength * core * (2.4 * bump(z, 7_800, 9_500, 11_200) - 3.0 * bump(z, 5_000, 6_500, 8_000)) * 1e-9
    noise = lambda s: s * (torch.rand((nz, ny, nx), generator=gen, device=dev, dtype=f64) - .5)
    f["theta"] += noise(.2) * (z < 1_500)
    for k in ("u", "v"):
        f[k] += noise(.6)
    f["w"] += noise(.2)
    f["w"][0] = 0
    f["w"][-1] = 0
    if lightning:   # a tripole's upper two charges, positive on the ice crystals and negative on the graupel
        per = charge / rho
        f["chargeIce"], f["chargeGraupel"] = per.clamp(min=0.0), per.clamp(max=0.0)
        f["chargeRain"], f["chargeAir"] = zero.clone(), zero.clone()
    out = {k: v.reshape(-1).to(torch.float32).cpu().numpy() for k, v in f.items()}
    if moments == 2:
        air = np.repeat(np.asarray(env.rho), grid.layer)
        out["rainNumber"] = marshall_palmer_number(out["rain"], air)
        for kind in ("graupel", "hail"):
            out[kind + "Number"], out[kind + "Volume"] = exponential_ice_moments(out[kind], air, kind)
    return out


def _specs(case, seed):
    rng = np.random.default_rng(seed)
    gen = torch.Generator(device="cuda")
    gen.manual_seed(int(seed))
    moments, lightning = case.get("moments", 1), case.get("lightning", 0)
    out = []
    for k, grid in enumerate(_grids(case)):
        profile = baseline_profile(rng.uniform(.011, .016), rng.uniform(0.0, 30.0) / math.tanh(2.0), rng.uniform(0.0, 90.0))
        env = Environment(SliderConfig(), grid, profile)
        sw = Switches(dt=DT, rain_moments=moments, ice_moments=moments, lightning=lightning)
        out.append(RunSpec(grid, env, sw, _storm(grid, env, gen, rng, moments, lightning), k, f"run{k}"))
    return out


def _pinned(count):
    return torch.empty(count, dtype=torch.float32, pin_memory=True).numpy()


class _Runs:
    """The device runs of a case, their host states in pinned memory, and where the states come back to."""

    def __init__(self, case, seed):
        self.ctx = _context()
        specs = _specs(case, seed)
        self.steps = case["steps"]
        self.runs = [self.ctx.create(s) for s in specs]
        extra = (CHARGES if case.get("lightning") else ()) + (("rainNumber",) + ICE2M if case.get("moments") == 2 else ())
        total = sum(s.grid.n for s in specs)
        self.start, self.end = _pinned(total * len(CARRIED)), _pinned(total * len(CARRIED))
        more = _pinned(total * max(1, len(extra))), _pinned(total * max(1, len(extra)))
        self.extra_in, self.extra_out, self.views = [], [], {k: [] for k in CARRIED + extra}
        at = more_at = 0
        for s in specs:
            n = s.grid.n
            for k in CARRIED:
                self.start[at:at + n] = s.fields[k]
                self.views[k].append(self.end[at:at + n])
                at += n
            into, back = {}, {}
            for k in extra:
                into[k], back[k] = (m[more_at:more_at + n] for m in more)
                into[k][:] = s.fields[k]
                self.views[k].append(back[k])
                more_at += n
            self.extra_in.append(into)
            self.extra_out.append(back)
            s.fields = {}   # (the host copies live in the packed buffers)
        # one array a field over runs of one size; a list of arrays, run by run and field after field, else
        sizes = {s.grid.n for s in specs}
        if len(sizes) == 1:
            n = sizes.pop()
            whole = torch.from_numpy(self.end).view(len(specs), len(CARRIED), n)
            self.out = {k: whole[:, j] for j, k in enumerate(CARRIED)}
            if extra:
                rest = torch.from_numpy(more[1]).view(len(specs), len(extra), n)
                self.out.update({k: rest[:, j] for j, k in enumerate(extra)})
        else:
            ends = np.cumsum([s.grid.n * len(CARRIED) for s in specs])
            groups, first = [], 0
            for j, s in enumerate(specs):   # runs of the same grid that lie together
                if j + 1 == len(specs) or specs[j + 1].grid is not s.grid:
                    block = torch.from_numpy(self.end[(ends[first - 1] if first else 0):ends[j]])
                    groups.append(block.view(j + 1 - first, len(CARRIED), s.grid.n))
                    first = j + 1
            self.out = [{k: g[:, j] for j, k in enumerate(CARRIED)} for g in groups]

    def __del__(self):
        for r in getattr(self, "runs", []):
            r.retire()


class _Requests:
    def __init__(self, case, seed):
        self.ctx = _context()
        self.specs = _specs(case, seed)
        rng = np.random.default_rng(seed + 1)
        self.lengths = [int(v) for v in rng.integers(max(1, case["steps"] // 2), case["steps"] + 1, len(self.specs))]
        self.server = Server(self.ctx, max_active=8)
        self.server.set_quantum(case["quantum"])

    def __del__(self):
        if getattr(self, "server", None):
            self.server.close()


def _ground(case, grid):
    """Ground heights, m, of a hill, ridge, plateau or Schar ridges at the domain's centre, the lowest column at 0."""
    top, a = case["height"] * 1000.0, max(case["width"] * 1000.0, 2 * grid.dx)
    x = (np.arange(grid.nx) + .5)[None, :] * grid.dx - grid.width / 2
    y = (np.arange(grid.ny) + .5)[:, None] * grid.dy - grid.depth / 2
    if case["form"] == "hill":
        h = top / (1 + (x * x + y * y) / (a * a)) ** 1.5
    elif case["form"] == "ridge":
        h = top / (1 + (x * x) / (a * a)) + 0 * y
    elif case["form"] == "plateau":
        h = top / (1 + np.exp((np.maximum(abs(x), abs(y)) - a) / (.25 * a)))
    else:
        h = top * np.exp(-x * x / (a * a)) * np.cos(math.pi * x / 8_000.0) ** 2 + 0 * y
    return (h - h.min()).astype(np.float32).ravel()


def _winds(grid, seed):
    """A westerly with storm-like gusts: u, v, w as float32, and a first-guess pressure."""
    rng = np.random.default_rng(seed)
    n = grid.n
    u = (12 + rng.normal(0, 3, n)).astype(np.float32)
    v = rng.normal(0, 3, n).astype(np.float32)
    w = rng.normal(0, 1, n).astype(np.float32)
    return u, v, w, rng.normal(0, 20, grid.layer * (grid.nz - 1))


def _density(grid):
    return 1.2 * np.exp(-np.asarray(grid.zs) / 9000)


class _Solve:
    def __init__(self, case, seed):
        self.ctx, self.grid = _context(), _grids(case)[0]
        g = self.grid
        if case["kind"] == "electric":
            self.solver, self.rho = ElectricSolver(self.ctx, g), _charge(g, seed)
        else:
            make = MaskedProjection if case["kind"] == "projection" else TerrainFaces
            self.solver = make(self.ctx, g, _density(g), _ground(case, g))
            self.winds = _winds(g, seed)
            self.work = [a.copy() for a in self.winds]

    def __del__(self):
        if getattr(self, "solver", None):
            self.solver.close()


def _charge(grid, seed):
    """A storm's charge density, C/m3: a few layers of either sign over two cores, and small-scale scatter."""
    rng = np.random.default_rng(seed)
    z = np.asarray(grid.zs)[:, None, None]
    x = (np.arange(grid.nx) * grid.dx)[None, None, :]
    y = (np.arange(grid.ny) * grid.dy)[None, :, None]
    rho = rng.normal(0, 2e-11, (grid.nz, grid.ny, grid.nx))
    for _ in range(2):
        cx, cy = rng.uniform(0, grid.width), rng.uniform(0, grid.depth)
        for h, peak in ((10_000, 2e-9), (6_500, -3e-9), (3_500, 1e-9)):
            rho += rng.uniform(.5, 1) * peak * np.exp(-((x - cx) ** 2 + (y - cy) ** 2) / 2_500.0 ** 2 - ((z - h) / 700.0) ** 2)
    return rho.ravel()


def prepare(case, seed):
    if case["kind"] in ("step", "round_trips"):
        state = _Runs(case, seed)
        if case["kind"] == "round_trips":
            state.end[:] = state.start
            state.groups = case["groups"]
        state.kind = case["kind"]
        return state
    state = _Requests(case, seed) if case["kind"] == "serve" else _Solve(case, seed)
    state.kind = case["kind"]
    return state


# ------------------------------------------------------------------------------------------------ one pass
def run(state):
    if state.kind == "step":
        ctx, runs = state.ctx, state.runs
        ctx.write_packed(runs, state.start)
        for r, extra in zip(runs, state.extra_in):
            if extra:
                r.write(extra)
        ctx.batch_step(runs, state.steps)
        ctx.read_packed(runs, state.end)
        for r, extra in zip(runs, state.extra_out):
            if extra:
                r.read(list(extra), extra)
        return state.out
    if state.kind == "round_trips":   # (the buffer goes on from where the last pass left it, as the engine's does)
        state.ctx.batch_round_trips(state.runs, state.end, steps=state.steps, groups=state.groups)
        return state.out
    if state.kind == "serve":
        out = {}
        for tag, (spec, steps) in enumerate(zip(state.specs, state.lengths)):
            state.server.submit(spec, steps, tag)
        while len(out) < len(state.specs):
            done, _, _ = state.server.iterate()
            for tag in done:
                out[tag] = state.server.collect(tag, state.specs[tag].grid.n)
        return out
    if state.kind == "electric":
        return state.solver.solve(state.rho)
    if state.kind == "projection":   # the stage's winds arrive in the work arrays the projection changes
        for a, b in zip(state.work, state.winds):
            np.copyto(a, b)
        state.solver.project(*state.work[:3], DT, state.work[3])
        return dict(zip(("u", "v", "w", "pressure"), state.work))
    # (the fluxes; the fourth array, the divergence they leave, is at the solve's tolerance: rounding of the fluxes)
    return dict(zip(("mx", "my", "mz"), state.solver.set_velocity_masked(*state.winds[:3])))


def work(case):
    """Step cases: per step and node the 13 fields read and written once (22 in the two-moment and electrified
    configurations' field sets as far as they are carried), and some 5,500 operations a node (WENO and upwind transport of
    three stages about 4,500, the rest the projections, the microphysics and the mixing). Solves: the host arrays in and out;
    transforms of 5 n log2 n a layer, 10 a node for the vertical recurrences, 100 a node for the cut-cell operators, for
    the iterations a hill takes."""
    grids = _grids(case)
    nodes = sum(g.n for g in grids)
    if case["kind"] in ("step", "round_trips", "serve"):
        fields = len(CARRIED) + (5 if case.get("moments") == 2 else 0) + (4 if case.get("lightning") else 0)
        return {"bytes": case["steps"] * nodes * 8.0 * fields, "flops": case["steps"] * nodes * 5500.0}
    transform = 10 * math.log2(grids[0].layer) + 10
    if case["kind"] == "electric":
        return {"bytes": 16.0 * nodes, "flops": nodes * transform}
    if case["kind"] == "projection":
        return {"bytes": 40.0 * nodes, "flops": 30 * nodes * (transform + 100)}
    return {"bytes": 44.0 * nodes, "flops": 12 * nodes * (transform + 50)}


# ------------------------------------------------------------------------------------------------ 64-bit values
def _thomas(lower, diag, upper, rhs):
    """Tridiagonal solves along the first axis (every other axis a system)."""
    n = len(rhs)
    cp, d = np.zeros_like(diag), np.zeros_like(rhs)
    for k in range(n):
        piv = diag[k] - (lower[k] * cp[k - 1] if k else 0)
        cp[k] = upper[k] / piv
        d[k] = (rhs[k] - (lower[k] * d[k - 1] if k else 0)) / piv
    for k in range(n - 2, -1, -1):
        d[k] -= cp[k] * d[k + 1]
    return d


def _exact_electric(grid, rho):
    nx, ny, nz = grid.nx, grid.ny, grid.nz
    dz, h = np.asarray(grid.dzs), np.asarray(grid.hz)
    spec = np.fft.rfft2(-rho.reshape(nz, ny, nx)[1:-1] / 8.8541878128e-12)
    lam = 4 * np.sin(np.pi * np.arange(nx // 2 + 1) / nx)[None, :] ** 2 / grid.dx ** 2 + 4 * np.sin(np.pi * np.arange(ny) / ny)[:, None] ** 2 / grid.dy ** 2
    lo, up = 1 / (h[1:-1] * dz[:-1]), 1 / (h[1:-1] * dz[1:])
    diag = -(lo + up)[:, None, None] - lam
    col = lambda a: np.broadcast_to(a[:, None, None], diag.shape).copy()
    lo, up = col(lo), col(up)
    lo[0] = up[-1] = 0
    phi = np.zeros((nz, ny, nx))
    phi[1:-1] = np.fft.irfft2(_thomas(lo, diag, up, spec), s=(ny, nx))
    return phi.ravel()


class _Cut:
    """The cut cells of a ground in a grid: solid nodes, and each node's height above the ground, m."""

    def __init__(self, grid, ground):
        self.nz, self.ny, self.nx = grid.nz, grid.ny, grid.nx
        self.zs, self.dz, self.hz = (np.asarray(a, np.float64)[:, None, None] for a in (grid.zs, grid.dzs, grid.hz))
        self.g = ground.astype(np.float64).reshape(1, self.ny, self.nx)
        self.top = self.zs.copy()
        self.top[:-1] += self.dz / 2
        buried = self.top - self.g < .2 * self.hz
        buried[-2:] = False
        self.solid = np.logical_and.accumulate(buried, axis=0)
        level = self.solid.sum(axis=0, keepdims=True)
        z = np.arange(self.nz)[:, None, None]
        self.height = np.where(self.solid, 0, np.where(z == level, self.top - self.g, self.hz + 0 * self.g))


def _conjugate_gradients(b, start, apply, precondition, tolerance, most, first):
    """Preconditioned conjugate gradients to `tolerance` of |b|, the residual tested before each iteration (`first`: the
    start's own residual counts too)."""
    q = start.copy()
    r = b - apply(q) if first else b.copy()
    z = precondition(r)
    d, rz, bb = z.copy(), float((r * z).sum()), float((b * b).sum())
    rr = float((r * r).sum())
    for _ in range(most):
        if rr <= tolerance ** 2 * bb:
            break
        s = apply(d)
        ds = float((d * s).sum())
        if not ds > 0:
            break
        alpha = rz / ds
        q += alpha * d
        r -= alpha * s
        rr = float((r * r).sum())
        z = precondition(r)
        new = float((r * z).sum())
        d = z + new / rz * d
        rz = new
    return q


def _exact_projection(grid, ground, u, v, w, first_guess):
    """The masked projection: the node mass flux made divergence-free over the dual cells, conjugate gradients to 1e-6
    around the flat spectral solve."""
    c = _Cut(grid, ground)
    nx, ny, nz, dx, dy = c.nx, c.ny, c.nz, grid.dx, grid.dy
    rho = _density(grid)[:, None, None]
    east, north = lambda a: np.roll(a, -1, 2), lambda a: np.roll(a, -1, 1)
    west, south = lambda a: np.roll(a, 1, 2), lambda a: np.roll(a, 1, 1)
    half, middle = c.dz / 2, c.zs[:-1] + c.dz / 2
    low = np.clip((middle - np.maximum(c.g, c.zs[:-1])) / half, 0, 1)
    high = np.clip((c.zs[1:] - np.maximum(c.g, middle)) / half, 0, 1)
    blocked = high == 0
    dropped = blocked & east(blocked) & north(blocked) & east(north(blocked))
    wall = ~c.solid & (c.zs <= c.g)
    inverse = np.where(c.solid, 0, 1 / np.where(c.solid, 1, rho * c.height))
    lower_share = np.where(c.solid[:-1], 0, rho[:-1] / 4 * low) * (high > 0)
    upper_share = rho[1:] / 4 * (high + np.where(c.solid[:-1], low, 0)) * (high > 0)

    def divergence(a, b, e):
        fu, fv = (lower_share * f[:-1] + upper_share * f[1:] for f in (a, b))
        fz = rho[1:] / 4 * e[1:] - rho[:-1] / 4 * e[:-1]
        out = ((east(fu) + east(north(fu)) - fu - north(fu)) / dx + (north(fv) + east(north(fv)) - fv - east(fv)) / dy +
               (fz + east(fz) + north(fz) + east(north(fz))) / c.dz)
        return np.where(dropped, 0, out)

    def gradient(phi):
        gu, gv, gw = (np.zeros((nz, ny, nx)) for _ in range(3))
        p = phi * c.dz
        a, b, e, d = west(south(p)), south(p), west(p), p
        x_, y_, s = (a - b + e - d) / dx, (a + b - e - d) / dy, (a + b + e + d) / c.dz
        under = rho[:-1] / 4 * low
        over = rho[1:] / 4 * (high + np.where(c.solid[:-1], low, 0))
        gu[:-1] += under * x_
        gv[:-1] += under * y_
        gw[:-1] -= rho[:-1] / 4 * s
        gu[1:] += over * x_
        gv[1:] += over * y_
        gw[1:] += rho[1:] / 4 * s
        gw[wall] = 0
        gw[0] = gw[-1] = 0
        return gu * inverse, gv * inverse, gw * inverse

    nc = nz - 1
    snap = lambda t: np.where(t < 1e-12, 0, np.where(t > 1 - 1e-12, 1, t))
    m, n = np.arange(nx // 2 + 1)[None, :], np.arange(ny)[:, None]
    sx, cx = snap(np.sin(np.pi * m / nx) ** 2), snap(np.cos(np.pi * m / nx) ** 2)
    sy, cy = snap(np.sin(np.pi * n / ny) ** 2), snap(np.cos(np.pi * n / ny) ** 2)
    al, be = 4 * (sx * cy / dx ** 2 + cx * sy / dy ** 2), cx * cy
    null, pinned = (al == 0) & (be == 0), al == 0
    r0, dz, hz = rho[:, 0, 0], c.dz[:, 0, 0], c.hz[:, 0, 0]
    lo, di, up = (np.zeros((nc, ny, nx // 2 + 1)) for _ in range(3))
    for k in range(nc):
        di[k] = -al / 2 * (r0[k] * dz[k] / (2 * hz[k]) + r0[k + 1] * dz[k] / (2 * hz[k + 1]))
        if k:
            t = be * r0[k] / (hz[k] * dz[k])
            lo[k] = -al / 2 * r0[k] * dz[k - 1] / (2 * hz[k]) + t
            di[k] -= t
        if k < nc - 1:
            t = be * r0[k + 1] / (hz[k + 1] * dz[k])
            up[k] = -al / 2 * r0[k + 1] * dz[k + 1] / (2 * hz[k + 1]) + t
            di[k] -= t
    di[0][pinned], up[0][pinned], lo[1][pinned] = 1, 0, 0
    for a, value in ((lo, 0), (di, 1), (up, 0)):
        a[:, null] = value

    def precondition(r):
        s = np.fft.rfft2(-r)
        s[0][pinned] = 0
        s[:, null] = 0
        return np.where(dropped, 0, np.fft.irfft2(_thomas(lo, di, up, s), s=(ny, nx)) * c.dz)

    def apply(x):
        return divergence(*gradient(np.where(dropped, 0, x / c.dz)))

    def mask(a, b, e):
        for f in (a, b, e):
            f[c.solid] = 0
        e[wall] = 0
        e[0] = e[-1] = 0

    a, b, e = (f.astype(np.float64).reshape(nz, ny, nx) for f in (u, v, w))
    mask(a, b, e)
    start = np.where(dropped, 0, first_guess.reshape(nc, ny, nx) * DT * c.dz)
    q = _conjugate_gradients(-divergence(a, b, e), start, apply, precondition, 1e-6, 200, True)
    phi = q / c.dz
    for f, g in zip((a, b, e), gradient(phi)):
        f += g
    mask(a, b, e)
    return dict(zip(("u", "v", "w", "pressure"), (t.ravel() for t in (a, b, e, phi / DT))))


def _exact_faces(grid, ground, u, v, w):
    """The transport's face fluxes over the ground, conjugate gradients to 1e-10 around the flat face solve."""
    c = _Cut(grid, ground)
    nx, ny, nz, dx, dy = c.nx, c.ny, c.nz, grid.dx, grid.dy
    rho = _density(grid)[:, None, None]
    rup = (rho[:-1] + rho[1:]) / 2
    east, north = lambda a: np.roll(a, -1, 2), lambda a: np.roll(a, -1, 1)
    west, south = lambda a: np.roll(a, 1, 2), lambda a: np.roll(a, 1, 1)
    open_x, open_y, open_z = ~(c.solid | east(c.solid)), ~(c.solid | north(c.solid)), ~(c.solid[:-1] | c.solid[1:])

    def aperture(other, shut):   # a face's open heights; what a shut face has open goes to the next open one above
        face = (c.g + other(c.g)) / 2
        bottom = np.concatenate([np.zeros((1, 1, 1)), c.top[:-1]])
        opening = np.where(face <= bottom, c.hz, np.maximum(0, c.top - face))
        out, carry = np.zeros((nz, ny, nx)), np.zeros((ny, nx))
        for k in range(nz):
            out[k] = np.where(shut[k], 0, opening[k] + carry)
            carry = np.where(shut[k], carry + opening[k], 0)
        return out
    ax, ay = aperture(east, ~open_x), aperture(north, ~open_y)

    def divergence(fx, fy, fz):
        out = (ax * fx - west(ax * fx)) / dx + (ay * fy - south(ay * fy)) / dy
        out[:-1] += fz
        out[1:] -= fz
        return out

    def gradient(p):
        return (np.where(open_x, rho * (east(p) - p) / dx, 0), np.where(open_y, rho * (north(p) - p) / dy, 0),
                np.where(open_z, rup * (p[1:] - p[:-1]) / c.dz, 0))

    m, n = np.arange(nx // 2 + 1)[None, :], np.arange(ny)[:, None]
    lam = 4 * np.sin(np.pi * m / nx) ** 2 / dx ** 2 + 4 * np.sin(np.pi * n / ny) ** 2 / dy ** 2
    face = (rup / c.dz)[:, 0, 0]
    lo, up = np.zeros((nz, ny, nx // 2 + 1)), np.zeros((nz, ny, nx // 2 + 1))
    lo[1:] += face[:, None, None]
    up[:-1] += face[:, None, None]
    di = -rho * c.hz * lam - lo - up
    di[0, 0, 0], up[0, 0, 0], lo[1, 0, 0] = 1, 0, 0

    def precondition(r):
        s = np.fft.rfft2(-r / c.hz) * c.hz
        s[0, 0, 0] = 0
        return np.fft.irfft2(_thomas(lo, di, up, s), s=(ny, nx))

    a, b, e = (f.astype(np.float64).reshape(nz, ny, nx) for f in (u, v, w))
    mx = np.where(open_x, rho * (a + east(a)) / 2, 0)
    my = np.where(open_y, rho * (b + north(b)) / 2, 0)
    mz = np.where(open_z, rup * (e[:-1] + e[1:]) / 2, 0)
    q = _conjugate_gradients(-divergence(mx, my, mz), np.zeros((nz, ny, nx)), lambda p: -divergence(*gradient(p)), precondition, 1e-10, 400, False)
    gx, gy, gz = gradient(q)
    return dict(mx=(mx - gx).ravel(), my=(my - gy).ravel(), mz=np.concatenate([mz - gz, np.zeros((1, ny, nx))]).ravel())


def exact(case, seed):
    """The 64-bit values of the field solves; a whole model step has none (see above)."""
    if case["kind"] not in ("electric", "projection", "faces"):
        return None
    grid = _grids(case)[0]
    if case["kind"] == "electric":
        return _exact_electric(grid, _charge(grid, seed))
    ground, winds = _ground(case, grid), _winds(grid, seed)
    if case["kind"] == "projection":
        return _exact_projection(grid, ground, *winds)
    return _exact_faces(grid, ground, *winds[:3])
