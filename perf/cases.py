"""Performance cases of the framework: what its users run, over the sizes they run it at.

A case is a dict of plain values; ``kind`` names the path:

* ``steps``      fused advect -> bin -> pair -> interact steps of one ensemble, plain or as a CUDA graph
* ``ensembles``  the same steps for many independent ensembles in one context
* ``records``    the advection phase alone, every step's positions recorded (the two-phase workflow)
* ``pairs``      fixed-radius pair query of host positions
* ``count``      pair count of clustered host positions
* ``adjoint``    differentiable advection, forward and backward
* ``histogram``  pairwise distance histograms per species

``listed()`` gives the fixed cases, ``draw(rng)`` one more of the same ranges, ``prepare`` the inputs
and the handle that a program keeps, ``run`` one pass through the public API, ``work`` the bytes and
operations a pass cannot do without, ``exact`` its computed outputs in float64 without this package.
"""

import math

import numpy as np
import torch

import lagrangian_microbes_gb300 as lm
from lagrangian_microbes_gb300 import adjoint, engine, fields
from lagrangian_microbes_gb300 import pairwise_distance_histogram as histograms

# The benchmark's geometry: a 1/12 degree hourly field over 190-215E x 15-40N, hourly steps, and about
# 19,600 microbes per square degree (490,000 on 5 x 5 degrees) paired within 0.01 degrees.
BOX = (190.0, 215.0, 15.0, 40.0)
RESOLUTION = 1.0 / 12.0
DT = 3600.0
DENSITY = 19600.0
METRES_PER_DEGREE = 1852.0 * 60.0
BATCH_BOX = (195.0, 215.0, 20.0, 35.0)
MAX_COST = 12e6  # microbe-steps of the largest fused case


def listed():
    return [
        # an interactive user's small run: one step at a time, the state read back after each
        dict(name="step_10k", kind="steps", n=10000, layout="lattice", steps=1, form="plain", radius=0.01, norm="2",
             kh=0.0, census=False),
        # the README-scale run: one simulated day of the fresh 700 x 700 lattice as one graph launch
        dict(name="day_490k_lattice", kind="steps", n=490000, layout="lattice", steps=24, form="graph", radius=0.01,
             norm="2", kh=0.0, census=False),
        # the same run once the flow has mixed it, plain steps with diffusion and a species census per step
        dict(name="steps_490k_mixed", kind="steps", n=490000, layout="mixed", steps=12, form="plain", radius=0.01,
             norm="2", kh=1e-8, census=True),
        # a large single ensemble, a ragged count
        dict(name="steps_2m_mixed", kind="steps", n=2000003, layout="mixed", steps=4, form="plain", radius=0.01,
             norm="2", kh=0.0, census=False),
        # a parameter sweep: ensembles of very different sizes and densities, own field and seed each
        dict(name="ensembles_32", kind="ensembles", ensembles=32, n_min=1000, n_max=200000, steps=6, form="graph",
             radius=0.01),
        # the advection phase of the two-phase workflow: a day of positions recorded into page-locked arrays
        dict(name="records_202k", kind="records", n=202500, layout="lattice", steps=24, kh=0.0),
        # neighbour pairs of positions from elsewhere, e.g. a stored step
        dict(name="pairs_150k", kind="pairs", n=150001, layout="mixed", radius=0.01, norm="2"),
        # pair statistics of strongly clustered positions, too many pairs to list
        dict(name="count_3m_clustered", kind="count", n=3000000, clusters=400, radius=0.01, norm="2"),
        # gradients at three scales and in the three working precisions
        dict(name="adjoint_5k_f64", kind="adjoint", n=5000, steps=24, precision="f64", checkpoint_every=8),
        dict(name="adjoint_100k_f32", kind="adjoint", n=100003, steps=48, precision="f32", checkpoint_every=16),
        dict(name="adjoint_1m_ds", kind="adjoint", n=1000000, steps=24, precision="ds", checkpoint_every=32),
        # distance histograms of the README-scale lattice, one per species
        dict(name="histogram_490k", kind="histogram", n=490000, layout="lattice", bins=70),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["steps", "steps", "steps", "ensembles", "records", "pairs", "count", "adjoint", "adjoint",
                       "histogram"])
    layout = rng.choice(["lattice", "mixed"])
    radius = rng.choice([0.008, 0.01, 0.0125])
    if kind == "steps":
        n = _log_int(rng, 3000, 2000000)
        steps = max(1, min(_log_int(rng, 1, 24), int(MAX_COST // n)))
        return dict(kind=kind, n=n, layout=layout, steps=steps, form=rng.choice(["plain", "graph"]), radius=radius,
                    norm=rng.choice(["2", "2", "1", "inf"]), kh=rng.choice([0.0, 0.0, 1e-8]),
                    census=rng.choice([False, True]))
    if kind == "ensembles":
        return dict(kind=kind, ensembles=rng.randint(2, 40), n_min=1000, n_max=_log_int(rng, 20000, 150000),
                    steps=rng.randint(1, 6), form=rng.choice(["plain", "graph"]), radius=rng.choice([0.008, 0.01]))
    if kind == "records":
        n = _log_int(rng, 5000, 490000)
        return dict(kind=kind, n=n, layout=layout, steps=max(2, min(24, int(5e6 // n))), kh=rng.choice([0.0, 1e-8]))
    if kind == "pairs":
        return dict(kind=kind, n=_log_int(rng, 1000, 490000), layout=layout, radius=radius,
                    norm=rng.choice(["2", "2", "1", "inf"]))
    if kind == "count":
        n = _log_int(rng, 30000, 3000000)
        return dict(kind=kind, n=n, clusters=max(4, n // rng.randint(4000, 9000)), radius=rng.choice([0.008, 0.01]),
                    norm=rng.choice(["2", "2", "1", "inf"]))
    if kind == "adjoint":
        precision = rng.choice(["ds", "ds", "f32", "f64"])
        n = _log_int(rng, 2000, 100000 if precision == "f64" else 1000000)
        return dict(kind=kind, n=n, steps=max(4, min(rng.randint(8, 48), int(2e7 // n))), precision=precision,
                    checkpoint_every=rng.choice([8, 16, 32]))
    return dict(kind=kind, n=_log_int(rng, 5000, 490000), layout=layout, bins=rng.choice([65, 70, 71]))


# ---- inputs ----

def _device():
    return torch.device("cuda" if torch.cuda.is_available() else "cpu")


def _field_arrays(box, frames, rng, modes=32):
    """(lon, lat, times, u, v): a seeded 32-mode streamfunction flow, wavelengths log-uniform in 50-500 km,
    0.2 m/s rms, phases turning once in ten days; float32 m/s, made on the device."""
    nx = int(round((box[1] - box[0]) / RESOLUTION)) + 1
    ny = int(round((box[3] - box[2]) / RESOLUTION)) + 1
    lon = box[0] + RESOLUTION * np.arange(nx)
    lat = box[2] + RESOLUTION * np.arange(ny)
    mid = 0.5 * (box[2] + box[3])
    x = (lon - lon.mean()) * METRES_PER_DEGREE * math.cos(math.radians(mid))
    y = (lat - mid) * METRES_PER_DEGREE
    k = 2 * math.pi / np.exp(rng.uniform(math.log(50e3), math.log(500e3), modes))
    theta, phase = rng.uniform(0, 2 * math.pi, modes), rng.uniform(0, 2 * math.pi, modes)
    dev = _device()
    put = lambda a: torch.as_tensor(a, dtype=torch.float64, device=dev)
    kx, ky = put(k * np.cos(theta)), put(k * np.sin(theta))
    ex = torch.polar(torch.ones(modes, nx, dtype=torch.float64, device=dev), kx[:, None] * put(x) + put(phase)[:, None])
    ey = torch.polar(torch.ones(modes, ny, dtype=torch.float64, device=dev), ky[:, None] * put(y))
    wave = torch.einsum("my,mx->myx", ey, ex)
    amp = 0.2 / math.sqrt(modes / 2)
    times = DT * np.arange(frames)
    turn = torch.polar(torch.ones(frames, dtype=torch.float64, device=dev), put(times) * (2 * math.pi / (10 * 86400.0)))
    u = torch.einsum("t,yx->tyx", turn, torch.einsum("m,myx->yx", (amp * put(np.sin(theta))).to(wave.dtype), wave)).imag
    v = torch.einsum("t,yx->tyx", turn, torch.einsum("m,myx->yx", (-amp * put(np.cos(theta))).to(wave.dtype), wave)).imag
    return lon, lat, times, u.float().contiguous(), v.float().contiguous()


def _velocity_field(arrays):
    lon, lat, times, u, v = arrays
    return fields.VelocityField(lon, lat, times, u.cpu().numpy(), v.cpu().numpy())


def _lattice(n, lat0, lon0, side):
    """n positions of a square-ish lattice (its last column may be short), latitude varying fastest."""
    rows = max(1, int(round(math.sqrt(n))))
    cols = -(-n // rows)
    lons = np.repeat(np.linspace(lon0, lon0 + side, cols), rows)[:n]
    lats = np.tile(np.linspace(lat0, lat0 + side, rows), cols)[:n]
    return lons, lats


def _positions(case, rng):
    """Float64 positions at the benchmark's density: the fresh lattice, or the well-mixed state of a long run."""
    side = math.sqrt(case["n"] / DENSITY)
    lat0, lon0 = 25.0 + 0.3 * rng.random(), 200.0 + 0.3 * rng.random()
    if case["layout"] == "lattice":
        return _lattice(case["n"], lat0, lon0, side)
    return lon0 + side * rng.random(case["n"]), lat0 + side * rng.random(case["n"])


def _clusters(case, rng):
    """Gaussian clusters (3 km) with rank-size Zipf(1.2) populations, as float32 positions."""
    n, k = case["n"], case["clusters"]
    w = np.arange(1, k + 1, dtype=np.float64) ** -1.2
    sizes = np.floor(n * w / w.sum()).astype(np.int64)
    sizes[0] += n - sizes.sum()
    lon = np.repeat(rng.uniform(200.0, 210.0, k), sizes) + 0.03 * rng.standard_normal(n)
    lat = np.repeat(rng.uniform(25.0, 35.0, k), sizes) + 0.03 * rng.standard_normal(n)
    return lon.astype(np.float32), lat.astype(np.float32)


def _norm(case):
    return {"1": 1, "2": 2, "inf": math.inf}[case["norm"]]


def _ensemble_inputs(case, seed):
    rng = np.random.default_rng(seed)
    shape = np.random.default_rng(case["ensembles"] + case["n_max"])  # a sweep's sizes are set, its flows are not
    flows, members = [], []
    for _ in range(case["ensembles"]):
        n = int(round(math.exp(shape.uniform(math.log(case["n_min"]), math.log(case["n_max"])))))
        side = shape.uniform(0.5, 3.0)
        lons, lats = _lattice(n, rng.uniform(BATCH_BOX[2] + 0.5, BATCH_BOX[3] - 0.5 - side),
                              rng.uniform(BATCH_BOX[0] + 0.5, BATCH_BOX[1] - 0.5 - side), side)
        members.append((lons, lats, rng.integers(1, 4, n).astype(np.int8)))
        flows.append(_field_arrays(BATCH_BOX, case["steps"] + 2, rng))
    probabilities = rng.uniform(0.5, 0.9, case["ensembles"])
    seeds = rng.integers(0, 2 ** 62, case["ensembles"])
    return flows, members, probabilities, seeds


def _adjoint_inputs(case, seed):
    rng = np.random.default_rng(seed)
    flow = _field_arrays(BOX, case["steps"] + 1, rng)
    side = 5.0
    lons, lats = _lattice(case["n"], 25.0 + 0.3 * rng.random(), 200.0 + 0.3 * rng.random(), side)
    km = 1.0 / 111.32
    target_lon = lons + rng.normal(0.0, 20.0 * km, case["n"]) / np.cos(np.deg2rad(lats))
    target_lat = lats + rng.normal(0.0, 20.0 * km, case["n"])
    put = lambda a, dt: torch.as_tensor(a, dtype=dt, device=_device())
    return (flow, put(lons, torch.float32), put(lats, torch.float32), put(target_lon, torch.float64),
            put(target_lat, torch.float64))


def prepare(case, seed):
    rng = np.random.default_rng(seed)
    kind = case["kind"]
    if kind in ("steps", "records"):
        flow = _field_arrays(BOX, case["steps"] + 2, rng)
        lons, lats = _positions(case, rng)
        species = rng.integers(1, 4, case["n"]).astype(np.int8)
        radius, norm = (case["radius"], _norm(case)) if kind == "steps" else (0.0, 2)
        sim = engine.Simulation(_velocity_field(flow), lons, lats, species, radius=radius, norm=norm, p_rs=0.7,
                                p_pr=0.7, p_sp=0.7, seed=seed, kh=case["kh"])
        sim.snapshot()
        if kind == "records":
            return dict(case=case, sim=sim, out=sim.record_buffers(case["steps"]))
        if case["form"] == "graph":
            sim.capture(0.0, DT, case["steps"], census=case["census"])
        return dict(case=case, sim=sim)
    if kind == "ensembles":
        flows, members, p, seeds = _ensemble_inputs(case, seed)
        sim = engine.EnsembleSimulation([_velocity_field(f) for f in flows], members, radius=case["radius"], p_rs=p,
                                        p_pr=p, p_sp=p, seeds=seeds)
        sim.snapshot()
        if case["form"] == "graph":
            sim.capture(0.0, DT, case["steps"])
        return dict(case=case, sim=sim)
    if kind == "pairs":
        # one point set per case, numbered from another point for every seed: the pairs are others, their
        # number is the same
        lons, lats = _positions(case, np.random.default_rng(case["n"]))
        shift = int(rng.integers(1, case["n"]))
        return dict(case=case, query=engine.PairQuery(case["radius"], _norm(case)),
                    lon=np.roll(lons.astype(np.float32), shift), lat=np.roll(lats.astype(np.float32), shift))
    if kind == "count":
        lon, lat = _clusters(case, rng)
        return dict(case=case, query=engine.PairQuery(case["radius"], _norm(case)), lon=lon, lat=lat)
    if kind == "adjoint":
        (lon, lat, times, u, v), lon0, lat0, target_lon, target_lat = _adjoint_inputs(case, seed)
        leaves = [t.requires_grad_(True) for t in (lon0, lat0, u, v)]
        return dict(case=case, tape=adjoint.AdjointTape(precision=case["precision"]), leaves=leaves,
                    axes=(lon, lat, times), targets=(target_lon, target_lat))
    lons, lats = _positions(case, rng)
    return dict(case=case, ctx=lm._lib.Context(), lon=lons.astype(np.float32), lat=lats.astype(np.float32),
                species=rng.integers(1, 4, case["n"]).astype(np.int8))


# ---- one pass ----

def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind in ("steps", "ensembles", "records"):
        sim = state["sim"]
        sim.restore()  # every pass starts from the prepared state, as a rewound run does
        if kind == "records":
            rec = sim.step(0.0, DT, case["steps"], interact=False, record=True, out=state["out"])
            return {k: rec[k] for k in ("lon", "lat", "species")}
        census = case.get("census", False)
        if case["form"] == "graph":
            sim.run_graph(1)
            got = {"census": sim.census()} if census else {}
        else:
            got = sim.step(0.0, DT, case["steps"], census=census)
        lon, lat, species, status = sim.state()
        return {"lon": lon, "lat": lat, "species": species, "status": status, **got}
    if kind == "pairs":
        i, j = state["query"].pairs(state["lon"], state["lat"])
        return {"i": i, "j": j}
    if kind == "count":
        return {"pairs": state["query"].count(state["lon"], state["lat"])}
    if kind == "adjoint":
        lon0, lat0, u, v = state["leaves"]
        lon, lat = adjoint.advect_rk4(lon0, lat0, u, v, *state["axes"], 0.0, DT, case["steps"],
                                      checkpoint_every=case["checkpoint_every"], tape=state["tape"])
        loss = adjoint.mean_squared_distance(lon, lat, *state["targets"])
        grads = torch.autograd.grad(loss, state["leaves"])
        return {"lon": lon.detach(), "lat": lat.detach(), "loss": loss.detach(),
                **dict(zip(("g_lon0", "g_lat0", "g_u", "g_v"), grads))}
    by = histograms.species_distance_histograms(state["lon"], state["lat"], state["species"], case["bins"],
                                                ctx=state["ctx"])
    return {"counts": np.stack([by[k][0] for k in by]), "overflow": np.array([by[k][1] for k in by])}


# ---- what a pass cannot do without ----

def _mean_degree(case, density):
    area = {"2": math.pi, "1": 2.0, "inf": 4.0}[case.get("norm", "2")] * case["radius"] ** 2
    return density * area


def work(case):
    kind, n = case["kind"], case.get("n", 0)
    frame = 8.0 * (round((BOX[1] - BOX[0]) / RESOLUTION) + 1) * (round((BOX[3] - BOX[2]) / RESOLUTION) + 1)
    advect_flops = 4 * 45.0
    if kind in ("steps", "records"):
        # per step: the state in and out (position 8 B, species and status 1 B each) and the part of two
        # frames under the microbes; per pair a distance test, an order hash and a draw; the state read back
        s = case["steps"]
        covered = min(1.0, n / DENSITY / ((BOX[1] - BOX[0]) * (BOX[3] - BOX[2])))
        pairs = 0.5 * n * _mean_degree(case, DENSITY) if kind == "steps" else 0.0
        out = 10.0 * n if kind == "steps" else 9.0 * n * s
        return {"bytes": s * (19.0 * n + covered * frame) + out, "flops": s * (advect_flops * n + 120.0 * pairs)}
    if kind == "ensembles":
        lo, hi, e, s = case["n_min"], case["n_max"], case["ensembles"], case["steps"]
        total = e * (hi - lo) / math.log(hi / lo)  # the mean of a log-uniform count
        # the sides are uniform in 0.5-3 degrees, so the mean of 1 / area is 1 / 1.5
        pairs = 0.5 * e * (hi * hi - lo * lo) / (2 * math.log(hi / lo)) / 1.5 * math.pi * case["radius"] ** 2
        return {"bytes": s * (19.0 * total + e * 8.0 * 3.6 / RESOLUTION ** 2) + 10.0 * total,
                "flops": s * (advect_flops * total + 120.0 * pairs)}
    if kind == "pairs":
        pairs = 0.5 * n * _mean_degree(case, DENSITY)
        return {"bytes": 8.0 * n + 16.0 * pairs, "flops": 8.0 * pairs}
    if kind == "count":
        # a pair count needs the positions once; a test per pair is what enumeration would cost
        return {"bytes": 8.0 * n, "flops": 30.0 * n}
    if kind == "adjoint":
        # forward and backward read the frames and write their gradient; a checkpoint per interval; about
        # four evaluations forward, four recomputed and four transposed per step
        s, word = case["steps"], 4.0 if case["precision"] == "f32" else 8.0
        marks = -(-s // case["checkpoint_every"])
        return {"bytes": (s + 1) * 3.0 * frame + 2 * word * n * (2 * marks + 4), "flops": s * n * 12 * 60.0}
    return {"bytes": 9.0 * n + 24.0 * (case["bins"] + 1), "flops": 100.0 * n}


# ---- the computed outputs in float64 ----

class _Flow64:
    """Bilinear in space, linear in time, m/s to degrees/s on a sphere: the advection's right-hand side."""

    def __init__(self, lon, lat, u, v):
        self.x0, self.y0 = float(lon[0]), float(lat[0])
        self.dx = (lon[-1] - lon[0]) / (len(lon) - 1)
        self.dy = (lat[-1] - lat[0]) / (len(lat) - 1)
        self.u, self.v = u, v

    def __call__(self, t, x, y):
        nt, ny, nx = self.u.shape
        k = min(int(t // DT), nt - 1)
        w = t / DT - k
        fx, fy = (x - self.x0) / self.dx, (y - self.y0) / self.dy
        i = fx.detach().floor().long().clamp(0, nx - 2)
        j = fy.detach().floor().long().clamp(0, ny - 2)
        a, b = fx - i, fy - j
        at = j * nx + i

        def sample(f):
            g = f.reshape(-1)
            return ((1 - a) * (1 - b) * g[at] + a * (1 - b) * g[at + 1] + (1 - a) * b * g[at + nx]
                    + a * b * g[at + nx + 1])

        def blend(f):
            return sample(f[k]) if w == 0 else (1 - w) * sample(f[k]) + w * sample(f[k + 1])

        return (blend(self.u) / (METRES_PER_DEGREE * torch.cos(y * (math.pi / 180.0))), blend(self.v) / METRES_PER_DEGREE)

    def step(self, t, x, y):
        k1 = self(t, x, y)
        k2 = self(t + DT / 2, x + DT / 2 * k1[0], y + DT / 2 * k1[1])
        k3 = self(t + DT / 2, x + DT / 2 * k2[0], y + DT / 2 * k2[1])
        k4 = self(t + DT, x + DT * k3[0], y + DT * k3[1])
        return tuple(p + DT / 6 * (a + 2 * b + 2 * c + d) for p, a, b, c, d in zip((x, y), k1, k2, k3, k4))


def _advect64(flow, lons, lats, steps):
    """Positions after each step, from float64 positions through a float32 field."""
    lon, lat, _, u, v = flow
    f = _Flow64(lon, lat, u.double(), v.double())
    x = torch.as_tensor(lons, dtype=torch.float64, device=u.device)
    y = torch.as_tensor(lats, dtype=torch.float64, device=u.device)
    out = []
    for s in range(steps):
        x, y = f.step(s * DT, x, y)
        out.append((x, y))
    return out


def _great_circle(lon1, lat1, lon2, lat2):
    r = math.pi / 180.0
    h = (torch.sin((lat2 - lat1) * r / 2) ** 2
         + torch.cos(lat1 * r) * torch.cos(lat2 * r) * torch.sin((lon2 - lon1) * r / 2) ** 2)
    return 2 * 6371.228e3 * torch.asin(torch.sqrt(h.clamp(max=1.0)))


def exact(case, seed):
    rng = np.random.default_rng(seed)
    kind = case["kind"]
    if kind in ("steps", "records"):
        if case["kh"] > 0:
            return None  # the kicks are random draws, and the recorded positions follow them
        flow = _field_arrays(BOX, case["steps"] + 2, rng)
        path = _advect64(flow, *_positions(case, rng), case["steps"])
        if kind == "records":
            return {"lon": torch.stack([p[0] for p in path]), "lat": torch.stack([p[1] for p in path]), "species": None}
        more = {"census": None} if case["census"] else {}
        return {"lon": path[-1][0], "lat": path[-1][1], "species": None, "status": None, **more}
    if kind == "ensembles":
        flows, members, _, _ = _ensemble_inputs(case, seed)
        ends = [_advect64(f, m[0], m[1], case["steps"])[-1] for f, m in zip(flows, members)]
        return {"lon": torch.cat([p[0] for p in ends]), "lat": torch.cat([p[1] for p in ends]), "species": None,
                "status": None}
    if kind != "adjoint":
        return None  # whole numbers
    (lon, lat, _, u, v), lon0, lat0, target_lon, target_lat = _adjoint_inputs(case, seed)
    leaves = [t.double().requires_grad_(True) for t in (lon0, lat0, u, v)]
    f = _Flow64(lon, lat, leaves[2], leaves[3])
    path = [(leaves[0], leaves[1])]
    for s in range(case["steps"]):
        with torch.no_grad():
            path.append(f.step(s * DT, *path[-1]))
    end = [t.detach().requires_grad_(True) for t in path[-1]]
    d = _great_circle(*end, target_lon, target_lat)
    loss = (d * d).mean()
    gx, gy = torch.autograd.grad(loss, end)
    g_u, g_v = torch.zeros_like(leaves[2]), torch.zeros_like(leaves[3])
    for s in reversed(range(case["steps"])):  # a step's graph at a time: the whole run's would not fit
        here = [t.detach().requires_grad_(True) for t in path[s]]
        frames = [t.detach()[s:s + 2].clone().requires_grad_(True) for t in leaves[2:]]
        local = _Flow64(lon, lat, *frames)
        x, y = local.step(0.0, *here)
        gx, gy, gu, gv = torch.autograd.grad((x, y), here + frames, (gx, gy))
        g_u[s:s + 2] += gu
        g_v[s:s + 2] += gv
    return {"lon": end[0].detach(), "lat": end[1].detach(), "loss": loss.detach(), "g_lon0": gx, "g_lat0": gy,
            "g_u": g_u, "g_v": g_v}
