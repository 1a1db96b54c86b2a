"""Timed cases of this framework's main paths, each through a call that a
user's program makes.

  sim2d     ``Sim2D.advance`` (and ``advance_record``): one active
            multi-phase-field system, from one step of a 16-cell lattice to
            the 2048^2 lattice of 1,024 cells;
  ens2d     ``Ensemble2D.advance``: independent systems of mixed size, one
            launch per step;
  sim3d     ``Sim3D.advance`` in the periodic, substrate-slab and hard-wall
            channel geometries;
  predict,  ``Surrogate2D.predict`` and ``Surrogate2D.train_step``: the
  train     relaxation network, forward and forward + backward + update.

Systems start from seeded random centres and have taken ``age`` steps before
the timed call. Outputs are views of the system's own device buffers (fields,
Q5.27 aggregate, cell records). ``exact`` restates each path in 64-bit torch
from the same centres, weights and crops.
"""
from __future__ import annotations

import math
import sys
from pathlib import Path

import numpy as np
import torch

PACKAGE = Path(__file__).resolve().parents[1] / "phase-field-gh200_b200"
if str(PACKAGE) not in sys.path:
    sys.path.insert(0, str(PACKAGE))

import pfb200  # noqa: E402

LAMBDA, DT, KAPPA, MU, XI, TAU, V_A = 7.0, 0.01, 10.0, 1.0, 1500.0, 1.0e4, 1.0e-2
TILE = 288         # side of a 2D cell tile
WINDOW = 144       # active window of a round cell inside its tile
WINDOW_AT = 64     # its first row and column
CROP = 64          # side of the network's crops
LAYERS = ((16, 32), (32, 32), (32, 32), (32, 32), (32, 32), (32, 32), (32, 32), (32, 16))
STORAGE = {"binary32": (0, torch.float32, 4), "binary16": (1, torch.float16, 2),
           "bfloat16": (2, torch.bfloat16, 2)}
ENSEMBLE_SIDES = (256, 384, 512, 768, 1024)
LARGEST_VOXELS = 512 * 64 ** 3  # brick voxels of the largest 3D case


def listed():
    return [
        # one step of a small system between two looks at it: latency
        dict(name="2d_one_step_16_cells", kind="sim2d", L=256, cells=16, radius=12.0, gap=24.0,
             storage="binary32", steps=1, record=0, age=24),
        # the smallest published configuration: fewer cells than SMs
        dict(name="2d_512_64_cells", kind="sim2d", L=512, cells=64, radius=12.0, gap=24.0,
             storage="binary32", steps=12, record=0, age=24),
        # the benchmark's system
        dict(name="2d_2048_1024_cells", kind="sim2d", L=2048, cells=1024, radius=12.0, gap=24.0,
             storage="binary32", steps=6, record=0, age=24),
        # the solver's default parameters: 288 cells of radius 49 at packing 0.9,
        # whose side is not a multiple of four and whose cells fill their windows
        dict(name="2d_default_288_cells", kind="sim2d", L=1554, cells=288, radius=49.0, gap=49.0,
             storage="binary32", steps=6, record=0, age=24),
        # 16-bit pools: the same arithmetic on half the bytes
        dict(name="2d_binary16_400_cells", kind="sim2d", L=1024, cells=400, radius=12.0, gap=24.0,
             storage="binary16", steps=6, record=0, age=24),
        # a recorded run: a trajectory frame of every step into page-locked memory
        dict(name="2d_recorded_400_cells", kind="sim2d", L=1024, cells=400, radius=12.0, gap=24.0,
             storage="binary32", steps=12, record=1, age=24),
        # a batch of replicas of mixed size
        dict(name="2d_ensemble_32", kind="ens2d", systems=32, mix=1234, radius=12.0, steps=6, age=24),
        # the 3D benchmark's periodic system
        dict(name="3d_periodic_512_cells", kind="sim3d", geometry="periodic", side=256, height=256,
             cells=512, radius=10.0, brick=64, gap=20.0, steps=2, age=6),
        # a monolayer on a substrate
        dict(name="3d_slab_187_cells", kind="sim3d", geometry="slab", side=256, height=128,
             cells=187, radius=10.0, brick=80, gap=10.0, steps=2, age=6),
        # a few cells between two walls
        dict(name="3d_channel_12_cells", kind="sim3d", geometry="channel", side=128, height=40,
             cells=12, radius=10.0, brick=64, gap=20.0, steps=4, age=6),
        # the network on every cell of a 400-cell system, and one training batch
        dict(name="surrogate_predict_400", kind="predict", batch=400),
        dict(name="surrogate_train_256", kind="train", batch=256),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["sim2d"] * 5 + ["ens2d"] * 2 + ["sim3d"] * 4 + ["predict", "train"])
    if kind == "sim2d":
        radius = round(math.exp(rng.uniform(math.log(10.0), math.log(49.0))), 2)
        cells = _log_int(rng, 4, 1024)
        density = rng.uniform(0.1, 0.9)
        L = max(288, math.ceil(math.sqrt(cells * math.pi * radius * radius / density)))
        while L > 2300:  # no larger than the largest listed lattice by much
            cells = cells * 3 // 4
            L = max(288, math.ceil(math.sqrt(cells * math.pi * radius * radius / density)))
        steps = rng.choice([1, 3, 6, 7])
        return dict(kind=kind, L=L, cells=cells, radius=radius, gap=round(radius, 1),
                    storage=rng.choice(["binary32"] * 4 + ["binary16", "bfloat16"]), steps=steps,
                    record=rng.choice([0, 0, 0, 1, 2]) if steps > 2 else 0,
                    age=rng.randint(0, 48))
    if kind == "ens2d":
        while True:
            case = dict(kind=kind, systems=rng.randint(2, 32), mix=rng.randint(0, 10 ** 6), radius=12.0,
                        steps=rng.choice([1, 6]), age=rng.randint(0, 48))
            if work(case)["bytes"] <= work(listed()[6])["bytes"]:
                return case
    if kind == "sim3d":
        geometry = rng.choice(["periodic", "slab", "channel"])
        radius = round(rng.uniform(8.0, 16.0), 1)
        k = math.sqrt(7.5) / LAMBDA
        tail = math.log(1.0 / 1.0e-5 - 1.0) / (2.0 * k)
        brick = 8 * math.ceil((2.0 * (radius + 0.5 / k + tail) + 16.0) / 8)
        cells = min(_log_int(rng, 4, 400), LARGEST_VOXELS // brick ** 3)
        gap = round(2.0 * radius, 1)
        if geometry == "periodic":
            height = side = max(brick + 9, math.ceil((cells * 6.0 * gap ** 3) ** (1.0 / 3.0)))
        else:
            side = max(brick + 9, math.ceil(math.sqrt(cells * 3.0) * gap))
            height = brick + rng.randint(4, 40) if geometry == "slab" else math.ceil(
                2.0 * radius) + rng.randint(16, 32)
        return dict(kind=kind, geometry=geometry, side=side, height=height, cells=cells,
                    radius=radius, brick=brick, gap=gap, steps=rng.choice([1, 2, 3]),
                    age=rng.randint(0, 6))
    return dict(kind=kind, batch=_log_int(rng, 1, 400 if kind == "predict" else 256))


# ---------------------------------------------------------------------------
# Inputs
# ---------------------------------------------------------------------------
def _place(seed, n, extent, periodic, gap):
    """n random points in the box `extent`, at least `gap` apart (nearest
    image along the periodic axes)."""
    rng = np.random.default_rng(seed)
    extent, wrap = np.asarray(extent, np.float64), np.asarray(periodic)
    out = np.zeros((n, len(extent)))
    have = tries = 0
    while have < n:
        tries += 1
        if tries > 200000:
            raise ValueError("the centres do not fit")
        c = rng.random(len(extent)) * extent
        d = out[:have] - c
        d -= np.where(wrap, extent * np.round(d / np.where(extent > 0, extent, 1.0)), 0.0)
        if have and np.min((d * d).sum(1)) < gap * gap:
            continue
        out[have] = c
        have += 1
    return out


def _centres2d(L, n, gap, seed):
    c = _place(seed, n, (L, L), (True, True), gap).astype(np.float32)
    return np.ascontiguousarray(c[:, 0]), np.ascontiguousarray(c[:, 1])


def _ensemble_systems(case):
    """(side, cells) of each system: sides of the ensemble benchmark, 16 to 400
    cells at packing 0.5 to 0.9."""
    rng = np.random.default_rng(case["mix"])
    out = []
    for _ in range(case["systems"]):
        L = int(rng.choice(ENSEMBLE_SIDES))
        n = round(rng.uniform(0.5, 0.9) * L * L / (math.pi * case["radius"] ** 2))
        out.append((L, int(min(400, max(16, n)))))
    return out


def _centres3d(case, seed):
    side, gap = case["side"], case["gap"]
    if case["geometry"] == "periodic":
        return _place(seed, case["cells"], (side, side, side), (True, True, True), gap)
    if case["geometry"] == "slab":
        c = _place(seed, case["cells"], (side, side), (True, True), gap)
        return np.concatenate([c, np.full((len(c), 1), -0.5)], 1)
    free = case["height"] - 2 * CHANNEL_PAD - 2.0 * case["radius"]
    c = _place(seed, case["cells"], (side, side, max(free, 0.0)), (True, True, False), gap)
    c[:, 2] += 0.5 * (case["height"] - 2 * CHANNEL_PAD - max(free, 0.0))
    return c


CHANNEL_PAD, WALL_KAPPA, WALL_WIDTH = 4, 5.0, 7.0


def _params3d(case, seed):
    p = pfb200.SimParams3D(Nx=case["side"], Ny=case["side"], Nz=case["height"],
                           geometry=case["geometry"], num_cells=case["cells"], B=case["brick"],
                           target_radius=case["radius"], lambda_=LAMBDA, seed=seed)
    if case["geometry"] == "channel":
        p.channel_padding, p.channel_height = CHANNEL_PAD, case["height"] - 2 * CHANNEL_PAD
        p.wall_kappa, p.wall_width = WALL_KAPPA, WALL_WIDTH
    return p


def _device():
    return torch.device("cuda" if torch.cuda.is_available() else "cpu")


def _weights(seed):
    """Flat network parameters: per layer weights [out][in][3][3], then the
    bias; the first layer has 3 real input channels, the last one real output."""
    rng = np.random.default_rng(seed)
    parts = []
    for i, (ci, co) in enumerate(LAYERS):
        rin, rout = (3 if i == 0 else ci), (1 if i == 7 else co)
        w = np.zeros((co, ci, 3, 3), np.float32)
        w[:rout, :rin] = rng.standard_normal((rout, rin, 3, 3)) * math.sqrt(2.0 / (9.0 * rin))
        b = np.zeros(co, np.float32)
        b[:rout] = 0.05 * rng.standard_normal(rout)
        parts += [w.ravel(), b]
    return np.concatenate(parts)


def _crops(n, seed):
    """n crops as the relaxation driver cuts them: a cell's profile, its
    neighbours' aggregate and its recent rate; and increments to learn."""
    dev = _device()
    g = torch.Generator().manual_seed(seed)
    u = torch.rand((n, 12), generator=g).to(dev)
    noise = torch.randn((n, CROP, CROP), generator=g).to(dev)
    y, x = torch.meshgrid(torch.arange(CROP, device=dev), torch.arange(CROP, device=dev),
                          indexing="ij")
    k = math.sqrt(7.5) / LAMBDA

    def disc(cx, cy, r):
        d = torch.hypot(x[None] - cx[:, None, None], y[None] - cy[:, None, None])
        return 0.5 * (1.0 - torch.tanh(k * (d - r[:, None, None])))

    cx, cy, r = 30 + 4 * u[:, 0], 30 + 4 * u[:, 1], 11.0 + 2.5 * u[:, 2]
    phi = disc(cx, cy, r)
    other = torch.zeros_like(phi)
    for j in range(3):
        a = 2 * math.pi * (u[:, 3 + 3 * j] + j) / 3
        dist = 22.0 + 8.0 * u[:, 4 + 3 * j]
        other += disc(cx + dist * torch.cos(a), cy + dist * torch.sin(a), 12 + u[:, 5 + 3 * j]) ** 2
    rate = phi * (1 - phi) * (12.0 - r)[:, None, None] * 0.1 - 0.2 * phi * other
    crops = torch.zeros((n, CROP + 2, CROP + 2, 16), dtype=torch.bfloat16, device=dev)
    for ch, v in enumerate((phi, other, rate)):
        crops[:, 1:-1, 1:-1, ch] = v.to(torch.bfloat16)
    target = (rate + 0.01 * phi * noise).float()
    return crops.reshape(n, -1, 16), target.contiguous()


# ---------------------------------------------------------------------------
# States
# ---------------------------------------------------------------------------
class _Buffer:
    """A device buffer of a system as a CUDA array; keeps the system alive."""

    def __init__(self, owner, ptr, shape, typestr, strides=None):
        self.owner = owner
        self.__cuda_array_interface__ = dict(shape=tuple(shape), typestr=typestr,
                                             data=(int(ptr), False), strides=strides, version=3)


def _view(owner, ptr, shape, typestr, strides=None):
    return torch.as_tensor(_Buffer(owner, ptr, shape, typestr, strides), device="cuda")


def _views2d(owner, sim, storage):
    """The buffers that hold the state after step k, by k % 6."""
    a, k0, n = sim.step_args(), sim.step, sim.num_cells
    dtype = STORAGE[storage][1]
    pools, slots = [None, None], [None, None, None]
    for j, ptr in enumerate((a.phi_in, a.phi_out)):
        pools[(k0 + j) % 2] = _view(owner, ptr, (n, TILE, TILE),
                                    "<f4" if dtype is torch.float32 else "<i2")
    pools = [p if dtype is torch.float32 else p.view(dtype) for p in pools]
    for j, ptr in enumerate((a.S_rd, a.S_sc, a.S_cl)):
        slots[(k0 + j) % 3] = _view(owner, ptr, (sim.side, sim.pitch), "<i4")
    at = {f: v[1] for f, v in pfb200.CELL_DTYPE.fields.items()}
    size = pfb200.CELL_DTYPE.itemsize
    rest = dict(moments=_view(owner, a.cell + at["V"], (n, 3), "<f8", (size, 8)),
                velocity=_view(owner, a.cell + at["vx"], (n, 2), "<f4", (size, 4)))
    return [dict(phi=pools[k % 2], S=slots[k % 3], **rest) for k in range(6)]


def prepare(case, seed):
    kind = case["kind"]
    if kind == "sim2d":
        p = pfb200.SimParams2D(L=case["L"], num_cells=case["cells"], target_radius=case["radius"],
                               seed=seed, phi_storage=STORAGE[case["storage"]][0])
        sim = pfb200.Sim2D(p, *_centres2d(case["L"], case["cells"], case["gap"], seed))
        sim.advance(case["age"])
        sim.sync()
        state = dict(kind=kind, sim=sim, steps=case["steps"], record=case["record"],
                     views=_views2d(sim, sim, case["storage"]))
        if case["record"]:
            frames = case["steps"] // case["record"]
            pinned = torch.zeros((frames, case["cells"], 12), dtype=torch.float32, pin_memory=True)
            state["pinned"] = pinned
            state["ring"] = pinned.numpy().view(pfb200.TRAJ_DTYPE).reshape(frames, case["cells"])
        return state
    if kind == "ens2d":
        systems = [(L, n, seed * 1000 + r) for r, (L, n) in enumerate(_ensemble_systems(case))]
        ps = [pfb200.SimParams2D(L=L, num_cells=n, target_radius=case["radius"], seed=s)
              for L, n, s in systems]
        ens = pfb200.Ensemble2D(ps, [_centres2d(L, n, case["radius"], s) for L, n, s in systems])
        ens.advance(case["age"])
        ens.sync()
        return dict(kind=kind, ens=ens, steps=case["steps"],
                    views=[_views2d(ens, ens.system(r), "binary32") for r in range(len(ens))])
    if kind == "sim3d":
        sim = pfb200.Sim3D(_params3d(case, seed), _centres3d(case, seed))
        sim.advance(case["age"])
        u, L, n, B = sim.update_args(), sim.layout, case["cells"], case["brick"]
        at = {f: v[1] for f, v in pfb200.CELL3D_DTYPE.fields.items()}
        size = pfb200.CELL3D_DTYPE.itemsize
        views = {p: _view(sim, p, (n, B, B, B), "<f4") for p in (u.phi_in, u.phi_out)}
        views.update({p: _view(sim, p, (L.nz, L.ny, L.pitch_x), "<i4") for p in (u.S_in, u.S_out)})
        return dict(kind=kind, sim=sim, steps=case["steps"], views=views,
                    volume=_view(sim, u.cells + at["V"], (n,), "<f8", (size,)),
                    velocity=_view(sim, u.cells + at["velocity_x"], (n, 3), "<f4", (size, 4)))
    n = case["batch"]
    net = pfb200.Surrogate2D(max_batch=n, seed=1)
    net.set_params(_weights(seed))
    x, t = _crops(n, seed)
    state = dict(kind=kind, net=net, x=x, t=t, batch=n)
    if kind == "predict":
        state["out"] = torch.zeros((n, CROP, CROP), device=x.device)
    else:
        g = torch.Generator().manual_seed(seed)
        state["idx"] = torch.randperm(n, generator=g).to(torch.int32).to(x.device)
    return state


def run(state):
    kind = state["kind"]
    if kind == "sim2d":
        sim = state["sim"]
        if not state["record"]:
            sim.advance(state["steps"])
            return state["views"][sim.step % 6]
        ring = state["ring"]
        sim.advance_record(state["steps"], state["record"], ring)
        sim.sync()  # the frames are read on the host
        return dict(state["views"][sim.step % 6], volume=ring["volume"], vx=ring["vx"],
                    vy=ring["vy"], cx=ring["cx"], cy=ring["cy"])
    if kind == "ens2d":
        ens = state["ens"]
        ens.advance(state["steps"])
        k = ens.step % 6
        return [v[k]["phi"] for v in state["views"]]
    if kind == "sim3d":
        sim, views = state["sim"], state["views"]
        sim.advance(state["steps"])
        u = sim.update_args()
        return dict(phi=views[u.phi_in], S=views[u.S_in], V=state["volume"],
                    velocity=state["velocity"])
    net = state["net"]
    if kind == "predict":
        net.predict(state["x"], state["out"], state["batch"])
        return state["out"]
    loss = net.train_step(state["x"], state["t"], state["idx"], 5e-4)
    return dict(loss=loss, params=net.get_params())


# ---------------------------------------------------------------------------
# Work and tolerance
# ---------------------------------------------------------------------------
def work(case):
    """Each field value read and written once per step, and each aggregate
    word; 60 operations a 2D site, 90 a 3D voxel. The network: its inputs,
    targets, results and parameters, and its multiply-adds on real pixels and
    channels (three times over for a training step)."""
    kind = case["kind"]
    if kind == "sim2d":
        sites = case["cells"] * WINDOW * WINDOW * case["steps"]
        return dict(bytes=sites * 2 * STORAGE[case["storage"]][2] + case["L"] ** 2 * 8 * case["steps"],
                    flops=60.0 * sites)
    if kind == "ens2d":
        systems = _ensemble_systems(case)
        sites = sum(n for _, n in systems) * WINDOW * WINDOW * case["steps"]
        area = sum(L * L for L, _ in systems) * case["steps"]
        return dict(bytes=8 * (sites + area), flops=60.0 * sites)
    if kind == "sim3d":
        v = case["cells"] * case["brick"] ** 3 * case["steps"]
        s = case["side"] ** 2 * case["height"] * case["steps"]
        return dict(bytes=8 * (v + s), flops=90.0 * v)
    n, px = case["batch"], CROP * CROP
    macs = n * 9 * (px * (3 * 32 + 4 * 32 * 32 + 32) + (px // 4) * 2 * 32 * 32)
    params = 4 * sum(9 * a * b + b for a, b in LAYERS)
    if kind == "predict":
        return dict(bytes=n * ((CROP + 2) ** 2 * 32 + px * 4) + params, flops=2.0 * macs)
    return dict(bytes=n * ((CROP + 2) ** 2 * 32 + px * 4) + 8 * params, flops=6.0 * macs)


def tolerance(case):
    """Fields and records of a binary32 path: steps of 1e-7-size rounding on
    values of order one. 16-bit pools round every stored value. The network
    keeps activations in bfloat16, and an update moves a weight by the sign of
    its gradient where that is small."""
    if case["kind"] == "predict":
        return dict(rel=2e-2, max=0.5)
    if case["kind"] == "train":
        return dict(rel=1.5e-3, max=0.1)
    if case["kind"] == "sim2d" and case["storage"] != "binary32":
        return dict(rel=2e-2 if case["storage"] == "bfloat16" else 3e-3, max=0.2, differ=1e-3)
    return dict(rel=4e-6, max=4e-4, differ=1e-3)


# ---------------------------------------------------------------------------
# The same in 64 bits
# ---------------------------------------------------------------------------
def _philox(c0, c1, c2, c3, key):
    """Philox4x32-10 of counter arrays; four uint64 arrays of 32-bit words."""
    m32 = np.uint64(0xFFFFFFFF)
    c = [np.asarray(v, np.uint64) & m32 for v in np.broadcast_arrays(c0, c1, c2, c3)]
    k0, k1 = key & 0xFFFFFFFF, (key >> 32) & 0xFFFFFFFF
    for _ in range(10):
        a, b = c[0] * np.uint64(0xD2511F53), c[2] * np.uint64(0xCD9E8D57)
        c = [(b >> np.uint64(32)) ^ c[1] ^ np.uint64(k0), b & m32,
             (a >> np.uint64(32)) ^ c[3] ^ np.uint64(k1), a & m32]
        k0, k1 = (k0 + 0x9E3779B9) & 0xFFFFFFFF, (k1 + 0xBB67AE85) & 0xFFFFFFFF
    return c


def _u53(hi, lo):
    return (((hi << np.uint64(32)) | lo) >> np.uint64(11)).astype(np.float64) * 2.0 ** -53


P_TUMBLE = -math.expm1(-DT / TAU)
BULK, INTER = 30.0 / LAMBDA ** 2, 60.0 * KAPPA / LAMBDA ** 2
MOTILITY = INTER / XI
STEEP = math.sqrt(7.5) / LAMBDA


def _exact2d(L, n, radius, cx, cy, seed, steps, frames_from=None, every=0):
    """Fields, moments and velocities after `steps` steps from fresh discs (all
    cells in the round window), and records of every `every`-th step after
    step `frames_from`."""
    dev, f8, W = _device(), torch.float64, WINDOW
    gx0 = torch.tensor(np.rint(cx - np.float32(71.5)).astype(np.int64) % L, device=dev)
    gy0 = torch.tensor(np.rint(cy - np.float32(71.5)).astype(np.int64) % L, device=dev)
    w = torch.arange(W, device=dev)
    ids = np.arange(n)
    d = []
    for g, c in ((gx0, cx), (gy0, cy)):
        v = (g[:, None] + w).remainder(L).to(f8) - torch.tensor(c.astype(np.float64), device=dev)[:, None]
        d.append(v - L * torch.round(v / L))
    r = torch.sqrt(d[0][:, None, :] ** 2 + d[1][:, :, None] ** 2)
    phi = 0.5 * (1.0 - torch.tanh(STEEP * (r - (radius + 0.5 / STEEP))))
    del r
    words = _philox(ids, 2, 0, 0, seed)
    theta = 2.0 * math.pi * _u53(words[0], words[1])
    A0 = math.pi * radius * radius
    frames = []

    def moments():
        sq = phi * phi
        row, col = sq.sum(2), sq.sum(1)
        return row.sum(1), (col * w).sum(1), (row * w).sum(1), sq

    V, Cx, Cy, sq = moments()
    vel = torch.zeros((n, 2), dtype=f8, device=dev)
    for s in range(steps):
        gx, gy = (gx0[:, None] + w).remainder(L), (gy0[:, None] + w).remainder(L)
        at = gy[:, :, None] * L + gx[:, None, :]
        S = torch.zeros(L * L, dtype=f8, device=dev)
        S.index_add_(0, at.reshape(-1), sq.reshape(-1))
        other = S[at] - sq
        p = torch.nn.functional.pad(phi, (1, 1, 1, 1))
        east, west, north, south = p[:, 1:-1, 2:], p[:, 1:-1, :-2], p[:, 2:, 1:-1], p[:, :-2, 1:-1]
        dx, dy = 0.5 * (east - west), 0.5 * (north - south)
        lap = (4.0 * (east + west + north + south) + p[:, 2:, 2:] + p[:, 2:, :-2] + p[:, :-2, 2:]
               + p[:, :-2, :-2] - 20.0 * phi) / 6.0
        words = _philox(s & 0xFFFFFFFF, s >> 32, ids, 0xA5A5A5A5, seed)
        hit = _u53(words[0], words[1]) < P_TUMBLE
        theta = np.where(hit, 2.0 * math.pi * _u53(words[2], words[3]), theta)
        heading = torch.tensor(np.stack([np.cos(theta), np.sin(theta)], 1), device=dev)
        force = torch.stack([(phi * dx * other).sum((1, 2)), (phi * dy * other).sum((1, 2))], 1)
        vel = V_A * heading + MOTILITY * force
        sx = torch.clamp(torch.round(Cx / V - 71.5), -4, 4).to(torch.int64)
        sy = torch.clamp(torch.round(Cy / V - 71.5), -4, 4).to(torch.int64)
        grow = (2.0 * MU / A0) * (A0 - V)
        phi = phi + DT * (lap - BULK * phi * (1 - phi) * (1 - 2 * phi) + grow[:, None, None] * phi
                          - INTER * phi * other - vel[:, 0, None, None] * dx - vel[:, 1, None, None] * dy)
        for i in torch.nonzero((sx != 0) | (sy != 0)).flatten().tolist():
            a, b = int(sx[i]), int(sy[i])
            f = torch.nn.functional.pad(phi[i], (4, 4, 4, 4))
            phi[i] = f[4 + b:4 + b + W, 4 + a:4 + a + W]
        gx0, gy0 = (gx0 + sx).remainder(L), (gy0 + sy).remainder(L)
        del p, dx, dy, lap, other, S, at
        V, Cx, Cy, sq = moments()
        if frames_from is not None and s >= frames_from and (s + 1 - frames_from) % every == 0:
            frames.append(torch.stack([V, vel[:, 0], vel[:, 1], (gx0 + Cx / V).remainder(L),
                                       (gy0 + Cy / V).remainder(L)]))
    full = torch.zeros((n, TILE, TILE), dtype=f8, device=dev)
    full[:, WINDOW_AT:WINDOW_AT + W, WINDOW_AT:WINDOW_AT + W] = phi
    return full, torch.stack([V, Cx, Cy], 1), vel, frames


def _seed_radius(radius, brick):
    """Radius of the tanh sphere whose discrete phi^2 sum in the brick is the
    ball's volume."""
    x = (np.arange(brick) - 0.5 * (brick - 1)) ** 2
    r = np.sqrt(x[:, None, None] + x[:, None] + x)
    values, counts = np.unique(r, return_counts=True)
    target, lo, hi = 4.0 * math.pi * radius ** 3 / 3.0, 0.0, float(brick)
    for _ in range(60):
        mid = 0.5 * (lo + hi)
        v = np.sum(counts * (0.5 * (1.0 - np.tanh(STEEP * (values - mid)))) ** 2)
        lo, hi = (mid, hi) if v < target else (lo, mid)
    return 0.5 * (lo + hi)


def _direction(words, more, planar):
    azimuth = 2.0 * math.pi * _u53(more[0], more[1])
    z = np.zeros(len(azimuth)) if planar else 2.0 * _u53(words[0], words[1]) - 1.0
    r = np.sqrt(1.0 - z * z)
    return np.stack([r * np.cos(azimuth), r * np.sin(azimuth), z], 1)


def _exact3d(case, seed):
    dev, f8 = _device(), torch.float64
    n, B, side, nz = case["cells"], case["brick"], case["side"], case["height"]
    periodic, slab = case["geometry"] == "periodic", case["geometry"] == "slab"
    ctr = _centres3d(case, seed)
    wall = torch.zeros(nz, dtype=f8, device=dev)
    if case["geometry"] == "channel":
        ctr[:, 2] = (ctr[:, 2].astype(np.float32) + np.float32(CHANNEL_PAD - 0.5)).astype(np.float64)
        k = math.sqrt(7.5) / WALL_WIDTH
        z = np.arange(nz) + 0.5
        fluid = 0.25 * (1 + np.tanh(k * (z - CHANNEL_PAD))) * (1 - np.tanh(k * (z - (nz - CHANNEL_PAD))))
        wall = torch.tensor(WALL_KAPPA / KAPPA * (1 - fluid) ** 2, device=dev)
    org = torch.tensor(np.rint(ctr - 0.5 * (B - 1)).astype(np.int64), device=dev)
    b = torch.arange(B, device=dev)
    c8 = torch.tensor(ctr, device=dev)
    radius = _seed_radius(case["radius"], B)
    volume0 = 4.0 * math.pi * case["radius"] ** 3 / 3.0 * (0.5 if slab else 1.0)
    ids = np.arange(n)
    words = _philox(ids & 0xFFFFFFFF, ids >> 32, 0x504F4C49, 0, seed)
    heading = _direction(words, words[2:], slab)

    def inside(o):  # planes of the brick inside the domain
        z = o[:, 2, None] + b
        return torch.ones_like(z, dtype=torch.bool) if periodic else (z >= 0) & (z < nz)

    def lattice(o):  # flat lattice index of every voxel (clamped planes outside)
        x, y, z = (o[:, i, None] + b for i in range(3))
        z = z.remainder(nz) if periodic else z.clamp(0, nz - 1)
        return ((z[:, :, None, None] * side + y.remainder(side)[:, None, :, None]) * side
                + x.remainder(side)[:, None, None, :])

    def padded(f, o):  # f with its stencil neighbours: reflected planes at walls, else zeros
        if periodic:
            return torch.nn.functional.pad(f, (1, 1, 1, 1, 1, 1))
        z = o[:, 2, None] + torch.arange(-1, B + 1, device=dev)
        src = torch.where(z == -1, 0, z)
        if not slab:
            src = torch.where(src == nz, nz - 1, src)
        ok = (src >= 0) & (src < nz)
        src = src - o[:, 2, None]
        ok &= (src >= 0) & (src < B)
        g = torch.gather(f, 1, src.clamp(0, B - 1)[:, :, None, None].expand(-1, -1, B, B))
        return torch.nn.functional.pad(g * ok[:, :, None, None], (1, 1, 1, 1))

    chunks = [slice(i, min(n, i + max(1, 2 ** 25 // B ** 3))) for i in
              range(0, n, max(1, 2 ** 25 // B ** 3))]
    phi = torch.zeros((n, B, B, B), dtype=f8, device=dev)
    for ch in chunks:
        x, y, z = ((org[ch, i, None] + b).to(f8) - c8[ch, i, None] for i in range(3))
        r = torch.sqrt(z[:, :, None, None] ** 2 + y[:, None, :, None] ** 2 + x[:, None, None, :] ** 2)
        phi[ch] = 0.5 * (1 - torch.tanh(STEEP * (r - radius))) * inside(org[ch])[:, :, None, None]
    V = torch.zeros(n, dtype=f8, device=dev)
    vel = torch.zeros((n, 3), dtype=f8, device=dev)
    for s in range(case["age"] + case["steps"]):
        S = torch.zeros(side * side * nz, dtype=f8, device=dev)
        for ch in chunks:
            S.index_add_(0, lattice(org[ch]).reshape(-1), (phi[ch] ** 2).reshape(-1))
        key = _philox(s & 0xFFFFFFFF, s >> 32, ids & 0xFFFFFFFF, 0x54554D45, seed)
        hit = _u53(key[0], key[1]) < P_TUMBLE
        more = _philox(s & 0xFFFFFFFF, s >> 32, ids & 0xFFFFFFFF, 0x54554D56, seed)
        heading = np.where(hit[:, None], _direction(key[2:], more, slab), heading)
        shift = torch.zeros((n, 3), dtype=torch.int64, device=dev)
        for ch in chunks:
            f, o = phi[ch], org[ch]
            live = inside(o)[:, :, None, None]
            sq = f * f
            other = (S[lattice(o)] - sq).clamp_(min=0.0)
            if case["geometry"] == "channel":
                other += wall[(o[:, 2, None] + b).clamp(0, nz - 1)][:, :, None, None]
            p = padded(f, o)
            g = [0.5 * (p[:, 1:-1, 1:-1, 2:] - p[:, 1:-1, 1:-1, :-2]),
                 0.5 * (p[:, 1:-1, 2:, 1:-1] - p[:, 1:-1, :-2, 1:-1]),
                 0.5 * (p[:, 2:, 1:-1, 1:-1] - p[:, :-2, 1:-1, 1:-1])]
            V[ch] = sq.sum((1, 2, 3))
            for i in range(3):
                force = (f * g[i] * other).sum((1, 2, 3))
                vel[ch, i] = V_A * torch.tensor(heading[ch, i], device=dev) + MOTILITY * force
                if slab and i == 2:
                    vel[ch, i] = 0.0
                axes = [a for a in (1, 2, 3) if a != 3 - i]
                mean = (sq.sum(axes) * b).sum(1) / V[ch]
                support = (f.abs() > 1e-5).amax(axes)
                lo = torch.where(support, b, B).amin(1)
                hi = torch.where(support, b, -1).amax(1)
                step = torch.clamp(torch.round(mean - 0.5 * (B - 1)).to(torch.int64), -4, 4)
                shift[ch, i] = torch.maximum(torch.minimum(step, lo), hi - (B - 1))
            lap = -128.0 * f
            for dz in range(3):
                for dy in range(3):
                    for dx in range(3):
                        far = (dz != 1) + (dy != 1) + (dx != 1)
                        if far:
                            lap += (14.0, 3.0, 1.0)[far - 1] * p[:, dz:dz + B, dy:dy + B, dx:dx + B]
            grow = (2.0 * MU / volume0) * (volume0 - V[ch])
            new = lap / 30.0 - BULK * f * (1 - f) * (1 - 2 * f) + grow[:, None, None, None] * f \
                - INTER * f * other
            for i in range(3):
                new -= vel[ch, i, None, None, None] * g[i]
            new = (f + DT * new) * live
            for i in torch.nonzero(shift[ch].any(1)).flatten().tolist():
                a = shift[ch.start + i].tolist()
                q = torch.nn.functional.pad(new[i], (4, 4, 4, 4, 4, 4))
                new[i] = q[4 + a[2]:4 + a[2] + B, 4 + a[1]:4 + a[1] + B, 4 + a[0]:4 + a[0] + B]
            phi[ch] = new
        org = org + shift
    return dict(phi=phi, S=None, V=V, velocity=vel)


def _exact_net(weights, x):
    """The network's output channel on padded crops x; `weights` per layer."""
    conv = torch.nn.functional.conv2d
    relu, pool = torch.relu, torch.nn.functional.avg_pool2d

    def layer(i, v):
        return conv(v, weights[i][0], weights[i][1], padding=1)

    a2 = relu(layer(1, relu(layer(0, x))))
    a4 = relu(layer(3, relu(layer(2, pool(a2, 2)))))
    v = a4.repeat_interleave(2, 2).repeat_interleave(2, 3) + a2
    for i in (4, 5, 6):
        v = relu(layer(i, v))
    return layer(7, v)[:, 0]


def _exact_surrogate(case, seed):
    dev, n = _device(), case["batch"]
    flat = _weights(seed)
    x, t = _crops(n, seed)
    x = x.reshape(n, CROP + 2, CROP + 2, 16)[:, 1:-1, 1:-1].permute(0, 3, 1, 2).double()
    weights, at = [], 0
    for ci, co in LAYERS:
        w = torch.from_numpy(flat[at:at + 9 * ci * co].reshape(co, ci, 3, 3)).to(dev)
        at += 9 * ci * co
        bias = torch.from_numpy(flat[at:at + co]).to(dev)
        at += co
        weights.append((w.bfloat16().double().requires_grad_(), bias.double().requires_grad_()))
    if case["kind"] == "predict":
        with torch.no_grad():
            return torch.cat([_exact_net(weights, x[i:i + 32]) for i in range(0, n, 32)])
    loss = 0.0
    for i in range(0, n, 32):
        part = ((_exact_net(weights, x[i:i + 32]) - t[i:i + 32].double()) ** 2).sum() / t.numel()
        part.backward()
        loss += float(part.detach())
    grad = torch.cat([g.grad.reshape(-1) for w in weights for g in w])
    # the first Adam step: bias-corrected moments are the gradient and its square
    step = 5e-4 * grad / (grad.abs() + 1e-8)
    return dict(loss=loss, params=torch.from_numpy(flat).to(dev).double() - step)


def exact(case, seed):
    kind = case["kind"]
    if kind == "sim2d":
        cx, cy = _centres2d(case["L"], case["cells"], case["gap"], seed)
        phi, moments, vel, frames = _exact2d(case["L"], case["cells"], case["radius"], cx, cy, seed,
                                             case["age"] + case["steps"], case["age"],
                                             case["record"] or 1)
        out = dict(phi=phi, S=None, moments=moments, velocity=vel)
        if case["record"]:
            rec = torch.stack(frames).permute(1, 0, 2)
            out.update(zip(("volume", "vx", "vy", "cx", "cy"), rec))
        return out
    if kind == "ens2d":
        out = []
        for r, (L, n) in enumerate(_ensemble_systems(case)):
            s = seed * 1000 + r
            out.append(_exact2d(L, n, case["radius"], *_centres2d(L, n, case["radius"], s), s,
                                case["age"] + case["steps"])[0])
        return out
    if kind == "sim3d":
        return _exact3d(case, seed)
    return _exact_surrogate(case, seed)
