"""The work that users of this framework have it do, as cases that can be timed and checked.

Every case goes through the public Python interface, as a user's program does: a DEM case sets
the start of a new run (positions, velocities and spins from page-locked host memory, contact
history and forces cleared), advances it and reads the new state; a bonded run goes on from pass
to pass; the surrogate's cases call its network on device arrays.

Kinds of cases and the ranges that `draw` spreads over:

  reference  the reference's own loop (createSolverDEM, a new neighbour list in every step) on the
             sizes of its example programs: 2 to 64 impacting spheres
  cloud      the same loop on a dense cloud over a floor, 200 to 12,000 spheres
  gas        spheres moving in a walled box, Verlet lists, 1,000 to 65,000, FP64 or mixed
  lattice    polydisperse spheres on a loosely packed lattice in a box, few in contact at a time,
             70,000 to 2,000,000, FP64 or mixed
  column     a quasi-2D column of disks in flow, most of them in contact, 70,000 to 200,000,
             FP64 or mixed
  bonded     a bonded bar pulled at its ends, 1,000 to 131,072 spheres, FP64 or mixed
  scenes     a batch of independent clusters fired at their walls, 32 to 256 scenes of 2 to 8,192
             spheres, FP64 or mixed
  predict    one stride of the learned surrogate on a column, 2,000 to 200,000 disks
  train      loss and gradient of the surrogate on a batch of frames, 1 to 4 frames of 2,000 to
             12,000 disks
"""
from __future__ import annotations

import json
import math
import os

import numpy as np
import torch

import cabanadem_b200
from cabanadem_b200 import _lib, api, scenarios as S, surrogate as SG
from cabanadem_b200.inputs import Inputs

DATA = os.path.join(os.path.dirname(os.path.abspath(cabanadem_b200.__file__)), "data")
WEIGHTS = os.path.join(DATA, "dam_break_surrogate.npz")
FIELDS = ("x", "u", "omega", "force", "torque", "tng_count")


# ---------------------------------------------------------------------------------------
# the cases
# ---------------------------------------------------------------------------------------
def listed():
    return [
        # two spheres in a head-on impact above a wall: the reference's first example program
        dict(name="reference_2", kind="reference", n=2, steps=1000),
        # a cloud of spheres in the reference's loop: the size of a laboratory set-up
        dict(name="cloud_3000", kind="cloud", n=3000, steps=200),
        # 4,096 spheres in a walled box: the small configuration, bound by latency
        dict(name="gas_4096", kind="gas", n=4096, steps=1000, mixed=False),
        # an odd size in between, forces in FP32
        dict(name="gas_30011_mixed", kind="gas", n=30011, steps=500, mixed=True),
        # 2,000,000 spheres: the headline configuration, half of its 2,000 steps
        dict(name="lattice_2m", kind="lattice", n=2_000_000, steps=1000, mixed=False),
        # 200,000 disks in dense flow, most of them in contact
        dict(name="column_200k", kind="column", n=200_000, steps=300, mixed=False),
        # the same regime at an odd size, forces in FP32
        dict(name="column_90001_mixed", kind="column", n=90_001, steps=300, mixed=True),
        # the bonded configuration's bar
        dict(name="bonded_131072", kind="bonded", nx=256, ny=64, nz=8, steps=256, mixed=False),
        # a small specimen with odd sides, bond history in FP32
        dict(name="bonded_3003_mixed", kind="bonded", nx=39, ny=11, nz=7, steps=100, mixed=True),
        # a batch of independent scenes of very different sizes
        dict(name="scenes_256", kind="scenes", scenes=256, steps=300, mixed=True),
        # inference and training of the surrogate
        dict(name="predict_200k", kind="predict", n=200_000),
        dict(name="train_4x10000", kind="train", n=10_000, frames=4),
    ]


def draw(rng):
    def log(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    kind = rng.choice(("reference", "cloud", "gas", "lattice", "column", "bonded", "scenes", "predict", "train"))
    mixed = rng.random() < 0.5
    if kind == "reference":
        return dict(kind=kind, n=log(2, 64), steps=log(200, 2000))
    if kind == "cloud":
        return dict(kind=kind, n=log(200, 12_000), steps=log(50, 400))
    if kind == "gas":
        return dict(kind=kind, n=log(1000, 65_000), steps=log(200, 1000), mixed=mixed)
    if kind == "lattice":
        return dict(kind=kind, n=log(70_000, 2_000_000), steps=log(100, 1000), mixed=mixed)
    if kind == "column":
        return dict(kind=kind, n=log(70_000, 200_000), steps=log(100, 300), mixed=mixed)
    if kind == "bonded":
        ny, nz = rng.randint(3, 64), rng.randint(3, 8)
        # the damping's sign makes the bar chaotic: mixed runs stay short enough to be compared
        return dict(kind=kind, nx=max(8, min(256, log(1000, 131_072) // (ny * nz))), ny=ny, nz=nz,
                    steps=log(50, 120) if mixed else log(100, 256), mixed=mixed)
    if kind == "scenes":
        return dict(kind=kind, scenes=log(32, 256), steps=log(100, 300), mixed=mixed)
    if kind == "predict":
        return dict(kind=kind, n=log(2000, 200_000))
    return dict(kind=kind, n=log(2000, 12_000), frames=rng.randint(1, 4))


def count(case):
    return case["nx"] * case["ny"] * case["nz"] if case["kind"] == "bonded" else case.get("n", 0)


def work(case):
    """Inputs read once and outputs written once; per step the integration of every particle and
    the contact or bond law of the pairs that act."""
    kind = case["kind"]
    if kind in ("predict", "train"):
        n = case["n"] * case.get("frames", 1)
        edges, h = 6.0 * n, 128
        node = 2 * (16 * h + h * h) + 3 * 2 * (2 * h * h + 2 * h * h + h * h) + 2 * (h * h + 2 * h)
        edge = 2 * (6 * h + h * h) + 3 * 2 * (h * h + h * h)
        flops = n * node + edges * edge
        if kind == "predict":
            return dict(bytes=n * (24 + 24 + 8 + 24), flops=flops)
        return dict(bytes=n * (3 * 24 + 8 + 4) + 4 * 401_552, flops=3.0 * flops)
    if kind == "scenes":
        n = case["scenes"] * 915.0   # mean of a log-uniform size in [2, 8192]
    else:
        n = count(case)
    pairs = dict(reference=1.0, cloud=0.3, gas=0.1, lattice=0.001, column=2.3, bonded=5.5, scenes=0.5)[kind]
    law = 260.0 if kind == "bonded" else 220.0
    return dict(bytes=n * (72 + 72 + 48 + 4 + 72.0), flops=case["steps"] * n * (30.0 + law * pairs))


# ---------------------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------------------
def _glass(rad):
    m = 4. / 3. * math.pi * rad ** 3 * S.GLASS["rho"]
    E, nu = S.GLASS["E"], S.GLASS["nu"]
    return dict(rad=rad, m=m, I=0.4 * m * rad * rad, rho=np.full_like(rad, S.GLASS["rho"]),
                E=np.full_like(rad, E), nu=np.full_like(rad, nu), G=np.full_like(rad, E / (2 * (1 + nu))))


def _walls(points, normals, E, nu):
    return dict(x=np.array(points, float).reshape(-1, 3), normal=np.array(normals, float).reshape(-1, 3),
                E=np.full(len(points), E), nu=np.full(len(points), nu),
                G=np.full(len(points), E / (2 * (1 + nu))))


def _box(lo, hi):
    points, normals = [], []
    for d in range(3):
        for at, sign in ((lo, 1.0), (hi, -1.0)):
            points.append(at)
            normals.append([sign if k == d else 0.0 for k in range(3)])
    return _walls(points, normals, S.GLASS["E"], S.GLASS["nu"])


def _cubic(n, pitch, rng, room):
    """n sites of a cubic lattice, each moved by up to `room` along every axis."""
    m = int(math.ceil(n ** (1.0 / 3.0)))
    k = np.arange(n)
    x = np.stack([k % m, (k // m) % m, k // (m * m)], axis=1) * pitch + 0.5 * pitch
    return x + rng.uniform(-room, room, size=(n, 3)), m * pitch


def _relaxed_column(n, rng):
    """n disks of r ~ U[0.9, 1.1] mm against the wall x = 0 on the floor y = 0, close to jamming: a
    tight hexagonal lattice relaxed until the overlaps are those of a dense flow (micrometres).
    Elementwise on the device, in a fixed order: the same disks for the same seed."""
    pitch, aspect = 2.06e-3, 2.0
    rowh = pitch * math.sqrt(3.0) / 2.0
    ncol = max(2, int(round(math.sqrt(n * rowh / pitch / aspect))))
    nrow = -(-n // ncol)
    k = np.arange(nrow * ncol)
    row, col = k // ncol, k % ncol
    rad = rng.uniform(0.9e-3, 1.1e-3, size=k.size)
    xy = np.stack([(col + 0.5 * (row % 2)) * pitch + 1.0e-3, row * rowh + 1.0e-3]) + rng.uniform(-5e-5, 5e-5, (2, k.size))
    rad[n:], xy[:, n:] = 0.0, 1e3 + k[n:]          # unused sites touch nothing
    q = torch.from_numpy(xy.reshape(2, nrow, ncol)).cuda()
    r = torch.from_numpy(rad.reshape(nrow, ncol)).cuda()
    odd = (torch.arange(nrow, device="cuda") % 2)[:, None]
    used = r > 0
    shifts = [(0, 1), (0, -1), (1, 0), (-1, 0), (1, 1), (-1, 1), (1, -1), (-1, -1)]

    def moved(a, dr, dc, fill):
        out = torch.full_like(a, fill)
        H, W = a.shape[-2:]
        out[..., max(0, -dr):H - max(0, dr), max(0, -dc):W - max(0, dc)] = \
            a[..., max(0, dr):H + min(0, dr), max(0, dc):W + min(0, dc)]
        return out

    rs = [moved(r, dr, dc, 0.0) for dr, dc in shifts]
    for sweep in range(300):
        step = torch.zeros_like(q)
        for (dr, dc), rj in zip(shifts, rs):
            d = moved(q, dr, dc, -1e3) - q
            dist = torch.sqrt(d[0] * d[0] + d[1] * d[1])
            live = used & (rj > 0)
            if dr:                                  # the far one of the two sites in the row beside
                live = live & ((dc >= 0) if dc == 0 else ((odd == 1) if dc == 1 else (odd == 0)))
            excess = torch.where(live, torch.clamp(r + rj - dist, min=0.0), torch.zeros_like(dist))
            step -= 0.3 * excess * d / dist
        q = q + step
        q = torch.where(used, torch.maximum(q, r.expand_as(q)), q)
    xy = q.reshape(2, -1)[:, :n].cpu().numpy()
    x = np.zeros((n, 3))
    x[:, 0], x[:, 1] = xy
    return x, rad[:n].copy(), float(x[:, 0].max()), float(x[:, 1].max())


def make(case, seed):
    """The start of a DEM case as host arrays: particles, walls, the laws' parameters and the list's."""
    kind, rng = case["kind"], np.random.default_rng(seed)
    n = case["n"]
    if kind == "reference":
        r, v = 0.01, 10.0
        x, u, w = np.zeros((n, 3)), np.zeros((n, 3)), rng.uniform(-20.0, 20.0, (n, 3))
        k = np.arange(n)
        x[:, 0] = np.where(k % 2 == 0, -1.0, 1.0) * r * (1.0 + rng.uniform(0.002, 0.01, n))
        x[:, 1] = r * (1.0 + rng.uniform(0.0005, 0.002, n))
        x[:, 2] = (k // 2) * 4.0 * r + rng.uniform(-0.1, 0.1, n) * r
        u[:, 0] = np.where(k % 2 == 0, v, -v) * rng.uniform(0.5, 1.0, n)
        u[:, 1] = -rng.uniform(1.0, 3.0, n)
        rad = np.full(n, r)
        m = 4. / 3. * math.pi * rad ** 3 * 2800.0
        props = dict(rad=rad, m=m, I=0.4 * m * rad * rad, rho=np.full(n, 2800.0), E=np.full(n, 48e9),
                     nu=np.full(n, 0.2), G=np.full(n, 2e10))
        walls = _walls([(0, 0, 0)], [(0, 1, 0)], 380e9, 0.23)
        return dict(x=x, u=u, omega=w, props=props, walls=walls, cor=0.8, mu=0.3, dt=1e-7, delta=3 * r, skin=0.0,
                    gravity=(0., 0., 0.), max_cnts=6)
    if kind == "cloud":
        r = 1e-3
        x, _ = _cubic(n, 2.1 * r, rng, 0.05 * r)
        x[:, 1] += r - x[:, 1].min()
        u = rng.uniform(-0.5, 0.5, (n, 3))
        u[:, 1] -= 1.0
        props = _glass(np.full(n, r))
        return dict(x=x, u=u, omega=rng.uniform(-50., 50., (n, 3)), props=props,
                    walls=_walls([(0, 0, 0)], [(0, 1, 0)], S.GLASS["E"], S.GLASS["nu"]), cor=0.8, mu=0.3, dt=1e-7,
                    delta=3 * r, skin=0.0, gravity=(0., 0., 0.), max_cnts=16)
    if kind == "gas":
        r = 1e-3
        x, side = _cubic(n, 2.2 * r, rng, 0.1 * r)
        return dict(x=x, u=rng.uniform(-0.5, 0.5, (n, 3)), omega=rng.uniform(-50., 50., (n, 3)),
                    props=_glass(np.full(n, r)), walls=_box((0., 0., 0.), (side,) * 3), cor=0.8, mu=0.3, dt=1e-7,
                    delta=0.0, skin=0.1 * r, gravity=(0., 0., -9.81), max_cnts=16)
    if kind == "lattice":
        rmin, rmax = 0.8e-3, 1.2e-3
        a = 2 * rmax
        side = (n * a ** 3 / math.sqrt(2.0)) ** (1. / 3.)
        nx, ny = max(1, round(side / a)), max(1, round(side / (a * math.sqrt(3.0) / 2.0)))
        k = np.arange(n)
        ix, iy, iz = k % nx, (k // nx) % ny, k // (nx * ny)
        rad = rng.uniform(rmin, rmax, n)
        x = np.stack([a * (ix + 0.5 * ((iy + iz) % 2)), a * math.sqrt(3.0) / 2.0 * (iy + (iz % 2) / 3.0),
                      a * math.sqrt(2.0 / 3.0) * iz], axis=1) + a
        x += rng.uniform(-1., 1., (n, 3)) * (0.05 * (a / 2 - rad))[:, None]
        return dict(x=x, u=rng.uniform(-0.1, 0.1, (n, 3)), omega=np.zeros((n, 3)), props=_glass(rad),
                    walls=_box((0., 0., 0.), tuple(x.max(axis=0) + a)), cor=0.8, mu=0.3, dt=5e-8, delta=0.0,
                    skin=0.1 * 0.5 * (rmin + rmax), gravity=(0., 0., -9.81), max_cnts=16)
    x, rad, width, height = _relaxed_column(n, rng)         # column
    u = np.zeros((n, 3))
    u[:, 0] = 0.4 * x[:, 1] / height + rng.uniform(-0.05, 0.05, n)
    u[:, 1] = -0.3 * x[:, 0] / width + rng.uniform(-0.05, 0.05, n)
    w = np.zeros((n, 3))
    w[:, 2] = rng.uniform(-50., 50., n)
    D = S.DAM
    m = 4. / 3. * math.pi * rad ** 3 * D["rho"]
    props = dict(rad=rad, m=m, I=0.4 * m * rad * rad, rho=np.full(n, D["rho"]), E=np.full(n, D["E"]),
                 nu=np.full(n, D["nu"]), G=np.full(n, D["E"] / (2 * (1 + D["nu"]))))
    walls = _walls([(0, 0, 0), (0, 0, 0), (8 * width, 0, 0)], [(0, 1, 0), (1, 0, 0), (-1, 0, 0)], D["E"], D["nu"])
    return dict(x=x, u=u, omega=w, props=props, walls=walls, cor=D["cor"], mu=D["mu"], dt=D["dt"], delta=0.0,
                skin=0.4e-3, gravity=(0., -9.81, 0.), max_cnts=12, release=4.0)   # m/s that an overlap's energy gives


def make_bar(case, seed):
    rng = np.random.default_rng(seed)
    c = S.bonded_bar(nx=case["nx"], ny=case["ny"], nz=case["nz"])
    st = c["state"]
    st.x[:] += rng.uniform(-5e-6, 5e-6, st.x.shape)
    st.u[:] += rng.uniform(-0.01, 0.01, st.u.shape)
    st.omega[:] = rng.uniform(-5., 5., st.omega.shape)
    return c


def make_scenes(case, seed):
    sc, rng = S.batched_scenes(nscenes=case["scenes"]), np.random.default_rng(seed)
    st, scene = sc.state, sc.extra["scene"]      # the scenes' sizes stay; shots, spins and gaps are the seed's
    theta, speed = np.deg2rad(rng.uniform(0., 90., case["scenes"])), rng.uniform(1., 5., case["scenes"])
    st.u[:, 0], st.u[:, 1] = (speed * np.sin(theta))[scene], (-speed * np.cos(theta))[scene]
    st.x[:] += rng.uniform(-5e-6, 5e-6, st.x.shape)
    st.omega[:] = rng.uniform(-50., 50., st.omega.shape)
    return sc


def make_frames(case, seed):
    """Positions of a flowing column at the last, the current and the next stride, per frame."""
    rng = np.random.default_rng(seed)
    T = SG.STRIDE * S.DAM["dt"]
    out = []
    for _ in range(case.get("frames", 1)):
        x, rad, width, height = _relaxed_column(case["n"], rng)
        d = np.zeros_like(x)
        d[:, 0] = (0.8 * x[:, 1] / height + rng.normal(0., 0.02, len(x))) * T
        d[:, 1] = (-0.6 * x[:, 0] / width + rng.normal(0., 0.02, len(x))) * T
        a = np.zeros_like(x)
        a[:, :2] = rng.normal(0., 2e-6, (len(x), 2))
        out.append((x - d, x, x + d + a, rad))
    frame = np.repeat(np.arange(len(out), dtype=np.int32), case["n"])
    return [np.concatenate(v) for v in zip(*out)] + [frame]


def surrogate_params(case):
    meta = json.loads(str(np.load(WEIGHTS)["meta"]))
    sc = S.dam_break(n=64, aspect=2.0)
    frames = case.get("frames", 1)
    prm = SG.params_for(sc, sigma_a=meta["sigma_a"], max_nodes=case["n"] * frames, max_frames=frames,
                        radius_graph=meta["radius_graph"], sigma_d=meta["sigma_d"], wall_clip=meta["wall_clip"])
    return prm, np.load(WEIGHTS)["params"]


# ---------------------------------------------------------------------------------------
# a user's program: what it keeps, and one pass
# ---------------------------------------------------------------------------------------
def _pinned(a):
    t = torch.empty(a.shape, dtype=torch.float64, pin_memory=True)
    t.copy_(torch.from_numpy(np.ascontiguousarray(a)))
    return t.numpy()


def _outputs(n):
    return {f: torch.empty((n,) if f == "tng_count" else (n, 3), device="cuda",
                           dtype=torch.int32 if f == "tng_count" else torch.float64) for f in FIELDS}


def _stream(ctx):
    return torch.cuda.ExternalStream(ctx.stream_ptr())


def prepare(case, seed):
    kind = case["kind"]
    prec = _lib.DEM_MIXED if case.get("mixed") else _lib.DEM_FP64
    if kind == "bonded":
        b = api.bonded_from_case(make_bar(case, seed), precision=prec)
        p = b.solver.particles
        return dict(case=case, bonds=b, p=p, out=_outputs(p.n), stream=_stream(p.ctx))
    if kind == "scenes":
        sc = make_scenes(case, seed)
        r = api.BatchRunner(sc, precision=prec)
        parts = []
        for q in r.parts:
            st, p = q["scenario"].state, q["solver"].particles
            parts.append(dict(p=p, start={f: _pinned(getattr(st, f)) for f in ("x", "u", "omega")},
                              out=_outputs(p.n), stream=_stream(p.ctx)))
        return dict(case=case, runner=r, parts=parts)
    if kind in ("predict", "train"):
        prev, cur, nxt, rad, frame = make_frames(case, seed)
        prm, w = surrogate_params(case)
        sg = SG.Surrogate(api.default_context(), prm)
        sg.set_params(w)
        with torch.cuda.stream(sg.stream):
            t = [torch.from_numpy(np.ascontiguousarray(a)).cuda() for a in (prev, cur, nxt, rad, frame)]
        return dict(case=case, sg=sg, t=t)
    d = make(case, seed)
    n, W = case["n"], d["walls"]
    p = api.Particles(n, d["max_cnts"], len(W["x"]))
    for f, v in d["props"].items():
        p.set(f, v)
    start = {f: _pinned(d[f]) for f in ("x", "u", "omega")}
    for f, v in start.items():
        p.set(f, v)
    w = api.Wall(len(W["x"]))
    zero = np.zeros_like(W["x"])
    for f, v in dict(W, u=zero, omega=zero).items():
        w.set(f, v)
    force = api.Force(d["cor"], d["cor"], d["mu"], d["mu"])
    if kind in ("reference", "cloud"):
        # the reference's loop takes int(final_time / timestep) + 1 steps
        inp = Inputs({"timestep": {"value": d["dt"]}, "output_frequency": {"value": case["steps"]},
                      "final_time": {"value": d["dt"] * (case["steps"] - 0.5)}})
        s = api.createSolverDEM(inp, p, w, force, d["delta"])
    else:
        s = api.SolverDEM(p, w, force, d["dt"], delta=d["delta"], skin=d["skin"], gravity=d["gravity"], precision=prec)
    return dict(case=case, p=p, wall=w, solver=s, start=start, out=_outputs(n), stream=_stream(p.ctx))


def _start_run(p, start):
    for f, v in start.items():
        p.set(f, v)
    p.clear_contacts()
    p.clear_forces()


def _read(p, out, stream):
    now = torch.cuda.current_stream()
    stream.wait_stream(now)
    for f, t in out.items():
        p.get_device(f, t)
    now.wait_stream(stream)
    return out


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "bonded":
        state["bonds"].run_steps(case["steps"])
        return _read(state["p"], state["out"], state["stream"])
    if kind == "scenes":
        for q in state["parts"]:
            _start_run(q["p"], q["start"])
        state["runner"].run_steps(case["steps"])
        return [_read(q["p"], q["out"], q["stream"]) for q in state["parts"]]
    if kind == "predict":
        prev, cur, _, rad, _ = state["t"]
        return state["sg"].predict(prev, cur, rad)
    if kind == "train":
        prev, cur, nxt, rad, frame = state["t"]
        loss, grad = state["sg"].loss_grad(prev, cur, nxt, rad, frame, case["frames"])
        return dict(loss=loss, grad=grad)
    _start_run(state["p"], state["start"])
    if kind in ("reference", "cloud"):
        state["solver"].run()
        return {f: state["p"].get(f) for f in FIELDS}        # the reference's slices are host views
    state["solver"].run_steps(case["steps"])
    return _read(state["p"], state["out"], state["stream"])


# ---------------------------------------------------------------------------------------
# the same results in plain torch, float64
# ---------------------------------------------------------------------------------------
def _cuda(a):
    return torch.from_numpy(np.ascontiguousarray(a)).cuda()


def _pairs(x, reach, group=None):
    """Directed pairs (i, j), i != j, closer than reach (and of one group)."""
    n = x.shape[0]
    lo = x.min(dim=0).values
    cell = ((x - lo) / reach).floor().long() + 1
    dims = cell.max(dim=0).values + 2
    key = (cell[:, 0] * dims[1] + cell[:, 1]) * dims[2] + cell[:, 2]
    if group is not None:
        key = key + group.long() * (dims[0] * dims[1] * dims[2])
    key, order = key.sort()
    everyone = torch.arange(n, device=x.device)
    pi, pj = [], []
    for dx in (-1, 0, 1):
        for dy in (-1, 0, 1):
            for dz in (-1, 0, 1):
                want = key + (dx * dims[1] + dy) * dims[2] + dz
                a = torch.searchsorted(key, want)
                cnt = torch.searchsorted(key, want, right=True) - a
                i = torch.repeat_interleave(everyone, cnt)
                j = torch.arange(i.numel(), device=x.device) - torch.repeat_interleave(cnt.cumsum(0) - cnt, cnt) + a[i]
                i, j = order[i], order[j]
                near = (i != j) & ((x[i] - x[j]).square().sum(1) < reach * reach)
                pi.append(i[near])
                pj.append(j[near])
    i, j = torch.cat(pi), torch.cat(pj)
    s = (i * n + j).argsort()
    return i[s], j[s]


def _dot(a, b):
    return (a * b).sum(1)


def _cross(a, b):
    return torch.linalg.cross(a, b, dim=1)


def _damping(cor):
    t = torch.log(cor)
    return -2. * math.sqrt(5. / 6.) * t / torch.sqrt(t * t + math.pi ** 2)


def _moduli(E1, nu1, G1, E2, nu2, G2):
    return (1. / ((1 - nu1 ** 2) / E1 + (1 - nu2 ** 2) / E2), 1. / ((2 - nu1) / G1 + (2 - nu2) / G2))


def exact_dem(d, steps, scene=None, scene_params=None):
    """The reference's step (Hertz-Mindlin pairs and walls, velocity Verlet) with its default quirks."""
    x, u, w = (_cuda(d[f]) for f in ("x", "u", "omega"))
    P = {k: _cuda(v) for k, v in d["props"].items()}
    W = {k: _cuda(v) for k, v in d["walls"].items()}
    n, dt, h = x.shape[0], d["dt"], 0.5 * d["dt"]
    rad, m, I = P["rad"], P["m"], P["I"]
    one = torch.ones(n, dtype=torch.float64, device="cuda")
    cor = cor_w = d["cor"] * one
    mu = mu_w = d["mu"] * one
    if scene is not None:
        scene = _cuda(scene).long()
        sp = torch.tensor(scene_params, dtype=torch.float64, device="cuda")
        cor, cor_w, mu, mu_w = (sp[scene, k] for k in range(4))
    Kn, Knw = _damping(cor), _damping(cor_w)
    g = torch.tensor(d["gravity"], dtype=torch.float64, device="cuda")
    travel = (3.0 * float(u.norm(dim=1).max()) + d.get("release", 0.0)) * steps * dt + 0.5 * float(g.norm()) * (steps * dt) ** 2
    margin = 2.0 * travel + 0.02 * float(rad.max())
    pi, pj = _pairs(x, 2.0 * float(rad.max()) + margin, scene)
    near = (x[pi] - x[pj]).norm(dim=1) < rad[pi] + rad[pj] + margin
    pi, pj = pi[near], pj[near]
    Ee, Ge = _moduli(P["E"][pi], P["nu"][pi], P["G"][pi], P["E"][pj], P["nu"][pj], P["G"][pj])
    R = 1. / (1. / rad[pi] + 1. / rad[pj])
    me = 1. / (1. / m[pi] + 1. / m[pj])
    hist = torch.zeros(pi.numel(), 3, dtype=torch.float64, device="cuda")
    was = torch.zeros(pi.numel(), dtype=torch.bool, device="cuda")
    nw = 1 if scene is not None else len(W["x"])
    wh = [torch.zeros(n, 3, dtype=torch.float64, device="cuda") for _ in range(nw)]
    x0 = x.clone()
    x = x + dt * u
    for step in range(steps):
        F, T = torch.zeros_like(x), torch.zeros_like(x)
        r = x[pi] - x[pj]
        act = ((rad[pi] + rad[pj] - r.norm(dim=1)) > 0).nonzero().squeeze(1)
        live = torch.zeros_like(was)
        live[act] = True
        hist = torch.where((live & was)[:, None], hist, torch.zeros_like(hist))
        was = live
        if act.numel():
            i, j, d_ij = pi[act], pj[act], r[act]
            dist = d_ij.norm(dim=1)
            ov = rad[i] + rad[j] - dist
            nrm = d_ij / dist[:, None]
            uj = torch.stack([u[j, 0], u[i, 1], u[i, 2]], dim=1)     # the reference's vel_j
            v = u[i] + _cross(w[i], nrm) * (rad[i] - ov / 2)[:, None] - (uj - _cross(w[j], nrm) * (rad[j] - ov / 2)[:, None])
            vdn = _dot(v, nrm)[:, None]
            vt = v - vdn * nrm
            Rc, mc, sro = R[act], me[act], torch.sqrt(R[act] * ov)
            eta = Kn[i] * torch.sqrt(2. * Ee[act] * sro * mc)
            fn = (4. / 3. * Ee[act] * torch.sqrt(Rc) * ov * torch.sqrt(ov))[:, None] * nrm - eta[:, None] * vdn * nrm
            kt = (8. * Ge[act] * sro)[:, None]
            ts = vt.norm(dim=1, keepdim=True)
            t = torch.where(ts > 1e-12, vt / ts, torch.zeros_like(vt))
            dl = _dot(hist[act] + v * dt, t)[:, None] * t
            lim = (mu[i] * fn.norm(dim=1))[:, None]
            ft = -torch.minimum((kt * dl).norm(dim=1, keepdim=True), lim) * t
            new = -ft / kt
            ln = new.norm(dim=1, keepdim=True)
            new = torch.where(ln > 1e-12, new / ln, torch.zeros_like(new))
            still = v.norm(dim=1, keepdim=True) < 1e-12
            hist[act] = torch.where(still, torch.zeros_like(new), new)
            F.index_add_(0, i, fn + torch.where(still, torch.zeros_like(ft), ft))
        for k in range(nw):
            wid = scene if scene is not None else torch.full((1,), k, dtype=torch.long, device="cuda")
            nrm = W["normal"][wid].expand(n, 3)
            ov = rad - _dot(x - W["x"][wid], nrm)
            hit = (ov > 0).nonzero().squeeze(1)
            keep = torch.zeros(n, 1, dtype=torch.bool, device="cuda")
            keep[hit] = True
            wh[k] = torch.where(keep, wh[k], torch.zeros_like(wh[k]))
            if not hit.numel():
                continue
            nr, o, ri, mi = nrm[hit], ov[hit], rad[hit], m[hit]
            ws = wid[hit] if scene is not None else wid.expand(hit.numel())
            Ew, Gw = _moduli(P["E"][hit], P["nu"][hit], P["G"][hit], W["E"][ws], W["nu"][ws], W["G"][ws])
            a = (ri - o / 2)[:, None]
            v = u[hit] + _cross(w[hit], nr) * a
            vdn = _dot(v, nr)[:, None]
            vt = v - vdn * nr
            sro = torch.sqrt(ri * o)
            eta = Knw[hit] * torch.sqrt(2. * Ew * sro * mi)
            fn = (4. / 3. * Ew * torch.sqrt(ri) * o * torch.sqrt(o))[:, None] * nr - eta[:, None] * vdn * nr
            kt = (8. * Gw * sro)[:, None]
            f = -kt * (wh[k][hit] + vt * dt)
            size = torch.sqrt(f[:, 0] ** 2 + f[:, 1] ** 2 + f[:, 2] * f[:, 1])[:, None]   # as the reference has it
            t = torch.where(size > 1e-12, f / size, torch.zeros_like(f))
            lim = (mu_w[hit] * fn.norm(dim=1))[:, None]
            ft = torch.where(size < lim, size, lim) * t
            still = v.norm(dim=1, keepdim=True) < 1e-12
            ft = torch.where(still, torch.zeros_like(ft), ft)
            wh[k][hit] = torch.where(still, torch.zeros_like(ft), -ft / kt)
            F[hit] += fn + ft
            T[hit] += _cross(nr, ft) * a
        F = F + m[:, None] * g
        u, w = u + h * F / m[:, None], w + h * T / I[:, None]
        if step + 1 < steps:
            u, w = u + h * F / m[:, None], w + h * T / I[:, None]
            x = x + dt * u
    if float((x - x0).norm(dim=1).max()) > 0.5 * margin:
        return None
    return dict(x=x, u=u, omega=w, force=F, torque=T, tng_count=None)


def exact_bar(c, steps):
    st, bp = c["state"], c["bparams"]
    x, u, w, rad, m, I = (_cuda(getattr(st, f)) for f in ("x", "u", "omega", "rad", "m", "I"))
    fix = _cuda(c["fix_flags"]).bool()
    dt, h, n = c["dt"], 0.5 * c["dt"], x.shape[0]
    i, j = _pairs(x, c["search_cutoff"])
    L0 = (x[i] - x[j]).norm(dim=1)
    bonded = L0 < c["bond_factor"] * rad[i]
    i, j, L0 = i[bonded], j[bonded], L0[bonded]
    ft, tn, tt = (torch.zeros(i.numel(), 3, dtype=torch.float64, device="cuda") for _ in range(3))
    rb = torch.minimum(rad[i], rad[j]) * bp["radius_factor"]
    A, J = math.pi * rb ** 2, math.pi * rb ** 4 / 4
    ktor, kben = (bp["kt"] * 2 * J / A)[:, None], (bp["kn"] * J / A)[:, None]
    beta, broken = bp["beta"], torch.zeros(i.numel(), 1, dtype=torch.bool, device="cuda")

    def sign(v):
        return torch.where(v >= 0, torch.ones_like(v), -torch.ones_like(v))

    x = x + dt * u
    for step in range(steps):
        r = x[i] - x[j]
        dist = r.norm(dim=1)
        broken = broken | (((dist - L0) / L0 > bp["break_strain"])[:, None])
        nrm = r / dist[:, None]
        gap = dist - rad[i] - rad[j]
        uj = torch.stack([u[j, 0], u[i, 1], u[i, 2]], dim=1)
        v = u[i] + _cross(w[i], nrm) * (rad[i] + gap / 2)[:, None] - (uj - _cross(w[j], nrm) * (rad[j] + gap / 2)[:, None])
        vn = _dot(v, nrm)[:, None] * nrm
        vt = v - vn
        wr = w[i] - w[j]
        wn = _dot(wr, nrm)[:, None] * nrm
        wt = wr - wn
        fn = (-bp["kn"] * (dist - L0))[:, None] * nrm
        fd = fn + beta * fn.abs() * sign(vn)
        ft = ft - _dot(ft, nrm)[:, None] * nrm - vt * (bp["kt"] * dt)
        ft = ft - beta * ft.abs() * sign(vt)
        tn = _dot(tn, nrm)[:, None] * nrm - wn * (ktor * dt)
        tn = tn - beta * tn.abs() * sign(wn)
        tt = tt - _dot(tt, nrm)[:, None] * nrm - wt * (kben * dt)
        tt = tt - beta * tt.abs() * sign(wt)
        zero = torch.zeros_like(fd)
        F = torch.zeros_like(x).index_add_(0, i, torch.where(broken, zero, fd + ft))
        T = torch.zeros_like(x).index_add_(0, i, torch.where(broken, zero, tn + tt))
        F[fix], T[fix] = 0., 0.
        u, w = u + h * F / m[:, None], w + h * T / I[:, None]
        if step + 1 < steps:
            u, w = u + h * F / m[:, None], w + h * T / I[:, None]
            x = x + dt * u
    return dict(x=x, u=u, omega=w, force=F, torque=T, tng_count=None)


SHAPES = [(16, 128), (16, 128), (384, 128), (256, 128), (384, 128), (256, 128), (384, 128), (256, 128), (128, 16)]


def _network(flat, prm, prev, cur, rad, frame):
    """The surrogate's network in float64: the decoder's output, the displacement and the graph."""
    layers, o = [], 0
    for kin, nout in SHAPES:
        sizes = ((128, kin), (128,), (nout, 128), (nout,))
        layers.append([])
        for s in sizes:
            layers[-1].append(flat[o:o + math.prod(s)].reshape(s))
            o += math.prod(s)

    def mlp(l, v):
        w1, b1, w2, b2 = layers[l]
        return torch.relu(v @ w1.t() + b1) @ w2.t() + b2

    flat2 = cur.clone()
    flat2[:, 2] = 0.
    recv, send = _pairs(flat2, prm.radius_graph * (1 + 1e-12), frame)
    disp = (cur - prev)[:, :2]
    n = cur.shape[0]
    xn = torch.zeros(n, 16, dtype=torch.float64, device="cuda")
    xn[:, :2] = disp / prm.sigma_d
    for k in range(prm.nwalls):
        at, nr = (torch.tensor(list(v)[:2], dtype=torch.float64, device="cuda") for v in (prm.wall_x[k], prm.wall_n[k]))
        xn[:, 2 + k] = (((cur[:, :2] - at) @ (nr / nr.norm()) - rad) / prm.wall_clip).clamp(-1., 1.)
    xn[:, 6] = (rad - prm.r_mean) / prm.r_std
    xe = torch.zeros(recv.numel(), 16, dtype=torch.float64, device="cuda")
    dx = cur[send, :2] - cur[recv, :2]
    dist = dx.norm(dim=1)
    xe[:, :2] = dx / prm.radius_graph
    xe[:, 2] = dist / prm.radius_graph
    xe[:, 3] = (dist - rad[recv] - rad[send]) / prm.r_mean
    xe[:, 4:6] = (disp[send] - disp[recv]) / prm.sigma_d
    hn, e = mlp(0, xn), mlp(1, xe)
    for l in (2, 4, 6):
        w1, b1, w2, b2 = layers[l]
        z = e @ w1[:, :128].t() + b1 + (hn @ w1[:, 128:256].t())[recv] + (hn @ w1[:, 256:].t())[send]
        e = e + torch.relu(z) @ w2.t() + b2
        agg = torch.zeros_like(hn).index_add(0, recv, e)
        hn = hn + mlp(l + 1, torch.cat([hn, agg], dim=1))
    return mlp(8, hn), disp, recv, send


def exact_predict(prm, w, prev, cur, rad):
    with torch.no_grad():
        out, disp, recv, send = _network(_cuda(w).double(), prm, prev, cur, rad, None)
    q = cur[:, :2] + disp + prm.sigma_a * out[:, :2]

    def out_of_walls(q):
        for k in range(prm.nwalls):
            at, nr = (torch.tensor(list(v)[:2], dtype=torch.float64, device="cuda") for v in (prm.wall_x[k], prm.wall_n[k]))
            nr = nr / nr.norm()
            q = q - ((q - at) @ nr - rad).clamp(max=0.)[:, None] * nr
        return q

    q, mass = out_of_walls(q), rad ** 3
    for _ in range(prm.project_iters):
        d = q[send] - q[recv]
        dist = d.norm(dim=1)
        excess = rad[recv] + rad[send] - dist - prm.project_allow * torch.minimum(rad[recv], rad[send])
        share = 0.5 * mass[send] / (mass[recv] + mass[send]) * excess.clamp(min=0.) / dist
        q = out_of_walls(q - torch.zeros_like(q).index_add_(0, recv, share[:, None] * d))
    return torch.cat([q, cur[:, 2:]], dim=1)


def exact(case, seed):
    kind = case["kind"]
    if kind == "bonded":
        if count(case) * case["steps"] > 150_000_000:
            return None
        return exact_bar(make_bar(case, seed), case["steps"])
    if kind == "scenes":
        sc = make_scenes(case, seed)
        outs = []
        for _, sub, _ in S.split_scenes(sc):
            st, wl = sub.state, sub.walls
            d = dict(x=st.x, u=st.u, omega=st.omega, cor=1.0, mu=0.0, dt=sub.dt, gravity=(0., 0., 0.),
                     props={f: getattr(st, f) for f in ("rad", "m", "I", "E", "nu", "G")},
                     walls={f: getattr(wl, f) for f in ("x", "normal", "E", "nu", "G")})
            outs.append(exact_dem(d, case["steps"], sub.extra["scene"], sub.extra["scene_params"]))
        return outs
    if kind in ("predict", "train"):
        prm, w = surrogate_params(case)
        prev, cur, nxt, rad, frame = (_cuda(a) for a in make_frames(case, seed))
        if kind == "predict":
            return exact_predict(prm, w, prev, cur, rad)
        flat = _cuda(w).double().requires_grad_(True)
        out, disp, _, _ = _network(flat, prm, prev, cur, rad, frame)
        loss = (out[:, :2] - ((nxt - cur)[:, :2] - disp) / prm.sigma_a).square().sum() / (2.0 * len(cur))
        return dict(loss=float(loss), grad=torch.autograd.grad(loss, flat)[0])
    return exact_dem(make(case, seed), case["steps"])
