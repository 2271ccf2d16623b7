"""Performance cases: the calls a user of soilb200 makes, over the sizes they are made at.

A case is one pass through the public entry points, from the inputs that a
program holds to the outputs that it takes back:

* ``path``    an episode of the plain terrain step (``PlainPath``): the terrain is put
              back to its start, a bucket (or a site's many buckets) cuts it for a number of
              1/60 s physics steps, and the fields and labels are read out;
* ``mobile``  an episode of the production Mobile V2 operator
              (``B200ProductionMobileV2Solver.step_resident``) on a terrain under a moving layer;
* ``solver``  one call of the drop-in solver (``B200MobileV2Solver.step``) on host arrays;
* ``batch``   an episode of many uneven patches stepped together (``B200PatchBatch``);
* ``relax``   the drop-in repose relaxation of a host height map (``relax_critical_slope``);
* ``settle``  the repose relaxation of a terrain that stays on the GPU
              (``LearnedRelaxation``), with the learned proposals or with the plain sweep alone;
* ``train``   one training step's loss and gradients of the proposal network.

Fields of the fixed-point precision are read out as float32 tensors on the
GPU, which is what a learner or a renderer takes (momentum is held in float32,
heights in 32-bit quanta); those of the double precision as float64.
"""

from __future__ import annotations

import math

import numpy as np
import torch

import soilb200
from soilb200 import bulk_state, learned, pipeline
from soilb200.train_repose import DEFAULT_WEIGHTS

DX = 0.05          # cell size of every workload, m
DT = 1.0 / 60.0    # physics step, s
DEV = "cuda"

# material of the 701^2 cut: density, repose, ..., start / stop angle, mobile friction
START_DEG, STOP_DEG, FRICTION, DENSITY = 38.0, 30.0, 0.55, 1600.0
REPOSE = math.tan(math.radians(35.0))


def listed():
    return [
        # one robot's small test pit: every launch and host round trip counts
        dict(name="path_96", kind="path", ny=96, nx=96, cuts=1, steps=60, tile=32,
             residual="gated", precision="fx32"),
        # a larger one whose loose pile settles under the repose frontier meanwhile
        dict(name="path_192_residual", kind="path", ny=192, nx=192, cuts=1, steps=30, tile=64,
             residual="always", precision="fx32"),
        # the headline workload: a 35 m pile under one bucket cut, one second
        dict(name="path_701", kind="path", ny=701, nx=701, cuts=1, steps=60, tile=64,
             residual="gated", precision="fx32"),
        # a 205 m site worked by 64 machines at once, one second
        dict(name="path_4096_site", kind="path", ny=4096, nx=4096, cuts=64, steps=60, tile=64,
             residual="gated", precision="fx32"),
        # a large terrain that moves everywhere (run-out of a fluidised slope)
        dict(name="mobile_4096", kind="mobile", ny=4096, nx=4096, steps=32, precision="fx32"),
        # the double-precision arithmetic of the reference, an odd medium grid
        dict(name="mobile_301x517_fp64", kind="mobile", ny=301, nx=517, steps=16,
             precision="fp64"),
        # the drop-in solver call on host arrays, as the reference's own gate makes it
        dict(name="solver_256_fp64", kind="solver", ny=256, nx=256, precision="fp64",
             external=False),
        # parallel environments: uneven patches, two seconds of simulation
        dict(name="batch_128", kind="batch", patches=128, steps=120, cfl=0.25),
        # the drop-in relaxation of a cut pile given as a host array
        dict(name="relax_701_fp64", kind="relax", ny=701, nx=701, precision="fp64",
             tolerance=1e-8),
        # a resident terrain settled after the cut, learned proposals + sweeps
        dict(name="settle_701_learned", kind="settle", ny=701, nx=701, schedule="learned"),
        # a large resident terrain settled by the plain sweep alone
        dict(name="settle_2048_plain", kind="settle", ny=2048, nx=2048, schedule="plain"),
        # one training step of the proposal network at its default batch
        dict(name="train_32x128", kind="train", batch=32, n=128),
    ]


def _log_int(rng, lo: int, hi: int) -> int:
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["path", "path", "mobile", "mobile", "solver", "batch", "relax", "settle",
                       "settle", "train"])
    if kind == "path":
        ny = _log_int(rng, 96, 2048)
        nx = max(64, min(2048, int(ny * rng.uniform(0.7, 1.4))))
        residual = "always" if ny <= 256 and rng.random() < 0.5 else "gated"
        return dict(kind=kind, ny=ny, nx=nx, cuts=max(1, ny * nx // 262144), residual=residual,
                    steps=rng.randint(20, 60), tile=rng.choice([32, 64]),
                    precision="fp64" if ny <= 512 and rng.random() < 0.2 else "fx32")
    if kind == "mobile":
        precision = "fp64" if rng.random() < 0.3 else "fx32"
        ny = _log_int(rng, 96, 1024 if precision == "fp64" else 3072)
        nx = max(64, int(ny * rng.uniform(0.7, 1.33)))
        return dict(kind=kind, ny=ny, nx=nx, steps=rng.randint(8, 32), precision=precision)
    if kind == "solver":
        ny = _log_int(rng, 64, 512)
        nx = max(48, int(ny * rng.uniform(0.6, 1.5)))
        return dict(kind=kind, ny=ny, nx=nx, precision=rng.choice(["fp64", "fx32"]),
                    external=rng.random() < 0.5)
    if kind == "batch":
        return dict(kind=kind, patches=_log_int(rng, 8, 128), steps=rng.randint(30, 90),
                    cfl=rng.choice([0.18, 0.25, 0.4]))
    if kind == "relax":
        ny = _log_int(rng, 64, 701)
        nx = max(48, int(ny * rng.uniform(0.7, 1.4)))
        return dict(kind=kind, ny=ny, nx=nx, precision=rng.choice(["fp64", "fx32"]),
                    tolerance=rng.choice([1e-8, 1e-6]))
    if kind == "settle":
        ny = _log_int(rng, 128, 2000)
        nx = max(96, min(2000, int(ny * rng.uniform(0.7, 1.4))))
        return dict(kind=kind, ny=ny, nx=nx, schedule=rng.choice(["learned", "plain"]))
    return dict(kind=kind, batch=rng.randint(2, 32), n=rng.choice([64, 96, 128, 160]))


# ---------------------------------------------------------------------------
# inputs (from the seed alone)
# ---------------------------------------------------------------------------
def _noise(ny: int, nx: int, cells: int, gen) -> torch.Tensor:
    """Lattice value noise in [0, 1] with quintic interpolation."""
    lat = torch.rand(cells + 2, cells + 2, generator=gen, device=DEV, dtype=torch.float64)
    n = max(ny, nx)
    u = (torch.arange(nx, device=DEV, dtype=torch.float64) + 0.5) * cells / n
    v = (torch.arange(ny, device=DEV, dtype=torch.float64) + 0.5) * cells / n
    iu, iv = u.long(), v.long()
    fu, fv = u - iu, v - iv
    su = (fu ** 3 * (fu * (fu * 6 - 15) + 10))[None, :]
    sv = (fv ** 3 * (fv * (fv * 6 - 15) + 10))[:, None]
    iv, iu = iv[:, None], iu[None, :]
    top = lat[iv, iu] + (lat[iv, iu + 1] - lat[iv, iu]) * su
    bot = lat[iv + 1, iu] + (lat[iv + 1, iu + 1] - lat[iv + 1, iu]) * su
    return top + (bot - top) * sv


def _pile(ny: int, nx: int, seed: int) -> torch.Tensor:
    """A dumped pile: parabolic envelope times six octaves of value noise; a small
    part of the cells stands above repose.  Up to 701 cells the pile is a scaled
    one (12 base cells across it; small ones are steeper), beyond it has more
    features of that size."""
    gen = torch.Generator(device=DEV).manual_seed(int(seed))
    n = max(ny, nx)
    acc = torch.zeros(ny, nx, device=DEV, dtype=torch.float64)
    total, amp = 0.0, 1.0
    for o in range(6):
        acc += amp * _noise(ny, nx, max(12, round(12 * n / 701)) * 2 ** o, gen)
        total += amp
        amp *= 0.5
    y = (torch.arange(ny, device=DEV, dtype=torch.float64) - (ny - 1) / 2) / (0.5 * ny)
    x = (torch.arange(nx, device=DEV, dtype=torch.float64) - (nx - 1) / 2) / (0.5 * nx)
    env = (1.0 - y[:, None] ** 2 - x[None, :] ** 2).clamp(0.0, 1.0)
    return min(2.0, n / 200) * env * (0.25 + 0.75 * acc / total)


def _cut_windows(case, seed: int, pile: np.ndarray, travel: float):
    """Per bucket: the cells that it can reach and their place along and across
    its path (1.8 m wide footprint, 0.3 m long, cutting 0.4 m deep at 0.5 m/s)."""
    ny, nx = pile.shape
    rng = np.random.default_rng([seed, 7])
    scale = min(1.0, min(ny, nx) / 350)
    width, length, depth = 1.8 * scale, 0.3 * max(scale, 0.5), 0.4 * scale
    out = []
    for _ in range(case["cuts"]):
        # a machine digs where the face is steep: the best of 16 places (drop over 0.5 m)
        at = rng.uniform(0.2, 0.8, (16, 2)) * (ny - 12, nx - 12)
        r, c = at.astype(int).T + 1
        drop = np.hypot(pile[r + 10, c] - pile[r, c], pile[r, c + 10] - pile[r, c])
        k = int(np.argmax(drop))
        sx, sy = (c[k] + 5) * DX, (r[k] + 5) * DX
        ang = rng.uniform(0.0, 2 * np.pi)
        reach = travel + width + length
        c0, c1 = max(0, int((sx - reach) / DX) - 1), min(nx, int((sx + reach) / DX) + 2)
        r0, r1 = max(0, int((sy - reach) / DX) - 1), min(ny, int((sy + reach) / DX) + 2)
        rows, cols = np.indices((r1 - r0, c1 - c0))
        rows, cols = (rows + r0).ravel(), (cols + c0).ravel()
        px, py = cols * DX - sx, rows * DX - sy
        along = px * np.cos(ang) + py * np.sin(ang)
        across = -px * np.sin(ang) + py * np.cos(ang)
        near = (np.abs(across) <= 0.5 * width) & (along >= -length) & (along <= travel)
        flat = (rows * nx + cols)[near]
        out.append((flat, along[near], pile.reshape(-1)[flat] - depth, length))
    return out


def _cut_schedule(case, seed: int, pile: np.ndarray):
    """(cells, target surfaces) of each step: every cell once, at its lowest target."""
    steps = case["steps"]
    windows = _cut_windows(case, seed, pile, 0.5 * steps * DT)
    sched = []
    for k in range(steps):
        s = 0.5 * (k + 1) * DT
        idx, tgt = [], []
        for flat, along, target, length in windows:
            inside = (along <= s) & (along >= s - length)
            idx.append(flat[inside])
            tgt.append(target[inside])
        idx, tgt = np.concatenate(idx), np.concatenate(tgt)
        order = np.lexsort((tgt, idx))
        idx, tgt = idx[order], tgt[order]
        first = np.ones(idx.size, bool)
        first[1:] = idx[1:] != idx[:-1]
        sched.append((np.ascontiguousarray(idx[first].astype(np.int32)),
                      np.ascontiguousarray(tgt[first])))
    return sched


def _cut_pile(ny: int, nx: int, seed: int) -> torch.Tensor:
    """A pile after a whole 6 m cut: the steep walls that repose relaxation works on."""
    b = _pile(ny, nx, seed)
    host = b.cpu().numpy()
    travel = min(6.0, 0.25 * min(ny, nx) * DX)
    flat = b.reshape(-1)
    for idx, _, tgt, _ in _cut_windows(dict(cuts=max(1, ny * nx // 491401)), seed, host, travel):
        at = torch.from_numpy(idx).to(DEV)
        flat[at] = torch.minimum(flat[at], torch.from_numpy(tgt).to(DEV))
    return b.clamp_min(0.0)


def _moving_layer(ny: int, nx: int, seed: int):
    """A 10 degree slope with swells under 5 to 25 cm of moving material."""
    rng = np.random.default_rng([seed, 11])
    p = rng.uniform(0.0, 2 * np.pi, 4)
    x = torch.arange(nx, device=DEV, dtype=torch.float64)[None, :]
    y = torch.arange(ny, device=DEV, dtype=torch.float64)[:, None]
    b = (math.tan(math.radians(10.0)) * (nx - 1 - x) * DX
         + 0.2 * torch.sin(x / 37 + p[0]) * torch.cos(y / 29 + p[1]))
    h = 0.15 + 0.1 * torch.cos(x / 53 + p[2]) * torch.sin(y / 41 + p[3])
    return b, h, 0.8 * h, 0.3 * h


def _mound(ny: int, nx: int, rng):
    """A tilted, bumpy patch with a freshly dumped heap, steeper than repose, on it."""
    x = torch.arange(nx, device=DEV, dtype=torch.float64)[None, :] * DX
    y = torch.arange(ny, device=DEV, dtype=torch.float64)[:, None] * DX
    z = math.tan(math.radians(10.0)) * x + 0.0 * y
    for _ in range(8):
        a, s = rng.uniform(0.05, 0.3), rng.uniform(0.2, 1.0)
        cx, cy = rng.uniform(0, nx * DX), rng.uniform(0, ny * DX)
        z = z + a * torch.exp(-((x - cx) ** 2 + (y - cy) ** 2) / (2 * s * s))
    sm = min(rng.uniform(0.35, 0.6), 0.12 * min(ny, nx) * DX)
    mx, my = rng.uniform(0.2, 0.8) * (nx - 1) * DX, rng.uniform(0.2, 0.8) * (ny - 1) * DX
    h = 1.3 * sm * torch.exp(-((x - mx) ** 2 + (y - my) ** 2) / (2 * sm * sm))
    return z, h


SIDES = (64, 96, 128, 192, 256, 384, 512)


def _patches(case, seed: int):
    """Uneven patches (aspect at most 2:1): the scene's sizes are the case's, its
    terrains the seed's."""
    sizes = np.random.default_rng([case["patches"], 17])
    rng = np.random.default_rng([seed, 13])
    out = []
    for _ in range(case["patches"]):
        ny = int(sizes.choice(SIDES))
        nx = int(sizes.choice([s for s in SIDES if max(s, ny) <= 2 * min(s, ny)]))
        out.append(_mound(ny, nx, rng))
    return out


def _train_inputs(case, seed: int):
    """(weights, heights before, wanted height change): steep noise patches and
    a diffused version of them."""
    n = case["n"]
    gen = torch.Generator().manual_seed(int(seed))
    weights = []
    for li, ((ci, co), (ri, ro)) in enumerate(zip(learned.LAYERS, learned.REAL)):
        w = torch.zeros(3, 3, ci, co)
        w[:, :, :ri, :ro] = torch.randn(3, 3, ri, ro, generator=gen) * math.sqrt(2 / (9 * ri))
        weights.append(w)
    dgen = torch.Generator(device=DEV).manual_seed(int(seed) + 1)
    pre = torch.stack([sum(0.5 ** o * _noise(n, n, 3 * 2 ** o, dgen) for o in range(4))
                       for _ in range(case["batch"])])
    steep = torch.stack([pre.diff(dim=1).abs().amax((1, 2)), pre.diff(dim=2).abs().amax((1, 2))])
    pre = pre * (math.tan(math.radians(52.0)) * DX / steep.amax(0))[:, None, None]
    post = torch.nn.functional.avg_pool2d(
        torch.nn.functional.pad(pre[:, None], (2, 2, 2, 2), mode="replicate"), 5, 1)[:, 0]
    return weights, pre.contiguous(), (post - pre).to(torch.float32).contiguous()


# ---------------------------------------------------------------------------
# prepare
# ---------------------------------------------------------------------------
def _pin(t: torch.Tensor) -> torch.Tensor:
    return t.cpu().contiguous().pin_memory()


def _material(friction=FRICTION):
    return soilb200.MaterialScenario("soil", DENSITY, 35.0, 0.0, 0.5, START_DEG, STOP_DEG,
                                     friction)


class _State:
    pass


def prepare(case, seed):
    s = _State()
    s.case = case
    kind = case["kind"]
    if kind in ("path", "mobile"):
        s.shape = (case["ny"], case["nx"])
        s.read = {k: torch.empty(s.shape, dtype=torch.float64, pin_memory=True)
                  for k in ("b_eff", "mobile", "momentum_x", "momentum_y")}
    if kind == "path":
        pile = _pile(*s.shape, seed)
        s.reset = {"b_eff": _pin(pile)}
        zero = torch.zeros(s.shape, dtype=torch.float64, pin_memory=True)
        s.reset.update(mobile=zero, momentum_x=zero, momentum_y=zero)
        s.zero_i32 = torch.zeros(s.shape, dtype=torch.int32, pin_memory=True).numpy()
        host = s.reset["b_eff"].numpy()
        s.cuts = _cut_schedule(case, seed, host)
        # with the frontier always on, the pile's body starts out disturbed
        s.seeds = np.flatnonzero(host > 0.25 * host.max()) if case["residual"] == "always" else None
        s.path = pipeline.PlainPath(host, np.zeros(s.shape), dx=DX, material=_material(),
                                    tile_size=case["tile"], residual=case["residual"],
                                    precision=case["precision"])
        s.grid = s.path.grid
    elif kind == "mobile":
        b, h, qx, qy = _moving_layer(*s.shape, seed)
        s.reset = {"mobile": _pin(h), "momentum_x": _pin(qx), "momentum_y": _pin(qy)}
        s.state = bulk_state.B200BulkState(s.shape, DX, DX, b.cpu().numpy(),
                                           precision=case["precision"], mobile_headroom_m=1.0)
        s.grid = s.state.grid
        # a fluidised layer: friction below the slope's own pull
        cfg = soilb200.MobileV2Config(dx_m=DX, dy_m=DX, basal_friction_coefficient=0.15)
        s.solver = bulk_state.B200ProductionMobileV2Solver(config=cfg)
        s.solver.bind_device_state(s.state, _material(0.15))
    elif kind == "solver":
        z, h = _mound(case["ny"], case["nx"], np.random.default_rng([seed, 13]))
        z, h = z.cpu().numpy(), h.cpu().numpy()
        q = np.stack((0.3 * h, -0.2 * h), axis=-1)
        s.state = soilb200.MobileV2State(z, h, q)
        s.external = np.array([0.4, -0.3]) if case["external"] else None
        s.solver = soilb200.B200MobileV2Solver(soilb200.MobileV2Config.unchecked(
            dx_m=DX, dy_m=DX, basal_friction_coefficient=REPOSE, cfl=0.4),
            precision=case["precision"])
    elif kind == "batch":
        parts = _patches(case, seed)
        s.count = sum(h.numel() for _, h in parts)
        s.read = {k: np.empty(s.count, np.float32) for k in ("mobile", "momentum_x", "momentum_y")}
        states = [soilb200.MobileV2State(z.cpu().numpy(), h.cpu().numpy(),
                                         np.zeros(tuple(h.shape) + (2,))) for z, h in parts]
        s.start = [_pin(h).numpy() for _, h in parts]
        s.zero = [np.zeros(h.shape) for h in s.start]
        s.batch = soilb200.B200PatchBatch(states, soilb200.MobileV2Config.unchecked(
            dx_m=DX, dy_m=DX, basal_friction_coefficient=REPOSE, cfl=case["cfl"]))
    elif kind == "relax":
        s.height = _cut_pile(case["ny"], case["nx"], seed).cpu().numpy()
    elif kind == "settle":
        s.shape = (case["ny"], case["nx"])
        s.start = _pin(_cut_pile(*s.shape, seed))
        s.read = torch.empty(s.shape, dtype=torch.float64, pin_memory=True)
        k, datum = soilb200.choose_quantization(s.start.numpy())
        s.grid = soilb200.DeviceGrid(s.shape, DX, DX, precision="fx32", height_exponent=k,
                                     datum_m=datum)
        s.relaxation = learned.LearnedRelaxation(s.grid, learned.ReposeNet.load(DEFAULT_WEIGHTS),
                                                 35.0)
    else:
        weights, s.pre, s.target = _train_inputs(case, seed)
        s.net = learned.ReposeNet(weights=weights)
    return s


# ---------------------------------------------------------------------------
# run
# ---------------------------------------------------------------------------
def _read_out(s) -> dict:
    """The fields as the program takes them: float32 tensors on the GPU for
    the fixed-point precision, the float64 host arrays for the double one."""
    out = {}
    for name, buf in s.read.items():
        s.grid.download_ptr(name, buf.data_ptr())
        out[name] = buf if s.case["precision"] == "fp64" else buf.to(DEV).float()
    return out


def run(s):
    case = s.case
    kind = case["kind"]
    if kind == "path":
        for name, buf in s.reset.items():
            s.grid.upload_ptr(name, buf.data_ptr())
        for name in ("latch", "previous_component", "frontier_reached"):
            s.grid.upload(name, s.zero_i32)
        if s.seeds is not None:
            s.path.frontier.seed_cells(s.seeds)
        for idx, tgt in s.cuts:
            st = s.path.step(DT, idx, tgt)
        return {"fields": _read_out(s), "labels": s.path.avalanche.labels(),
                "record": [st.substeps, st.unstable_cells, st.regions, st.largest]}
    if kind == "mobile":
        for name, buf in s.reset.items():
            s.grid.upload_ptr(name, buf.data_ptr())
        for _ in range(case["steps"]):
            rec = s.solver.step_resident(DT)
        out = _read_out(s)
        del out["b_eff"]  # the operator does not move the support
        return {"fields": out, "substeps": rec.substeps}
    if kind == "solver":
        st = s.solver.step(s.state, DT, external_acceleration_m_s2=s.external)
        h, q = st.state.h_m, st.state.q_m2_s
        if case["precision"] == "fx32":
            h, q = h.astype(np.float32), q.astype(np.float32)
        return {"h": h, "q": q, "substeps": st.substeps}
    if kind == "batch":
        for i, h in enumerate(s.start):
            s.batch.upload(i, "mobile", h)
            s.batch.upload(i, "momentum_x", s.zero[i])
            s.batch.upload(i, "momentum_y", s.zero[i])
        for _ in range(case["steps"]):
            stats = s.batch.step_stats(DT)
        out = {"substeps": np.array([st.substeps for st in stats])}
        for name, buf in s.read.items():
            at = 0
            for i in range(s.batch.n_patches):
                field = s.batch.download(i, name).ravel()
                buf[at:at + field.size] = field
                at += field.size
        out.update(s.read)
        return out
    if kind == "relax":
        h, st = soilb200.relax_critical_slope(s.height, (DX, DX), 35.0,
                                              tolerance=case["tolerance"],
                                              precision=case["precision"])
        return {"height": h, "iterations": st.iterations}
    if kind == "settle":
        s.grid.upload_ptr("b_eff", s.start.data_ptr())
        st = s.relaxation.relax_scheduled(
            1e-4 * DX, learned.SCHEDULE if case["schedule"] == "learned" else learned.PLAIN)
        s.grid.download_ptr("b_eff", s.read.data_ptr())
        return {"height": s.read, "sweeps": st.iterations}
    tan = REPOSE
    n, b = case["n"], case["batch"]
    feat = learned.features_f64(s.pre, DX, DX, tan)
    loss, grads, flux = learned.loss_and_grads(s.net, feat, s.target, DX, DX, tan,
                                               1.0 / ((tan * DX) ** 2 * b * n * n))
    return {"loss": loss, "grads": grads, "flux": flux}


def work(case):
    kind = case["kind"]
    if kind == "batch":  # the sides' mean product under their aspect rule; 3 fields in and out
        cells = 46000 * case["patches"]
        return {"bytes": cells * (3 * 16 + 28 * 4 * case["steps"]),
                "flops": cells * 200 * 4 * case["steps"]}
    if kind == "train":
        px = case["batch"] * case["n"] ** 2
        macs = 9 * sum(ci * co for ci, co in learned.REAL)
        first = 9 * learned.REAL[0][0] * learned.REAL[0][1]
        return {"bytes": px * (8 + 4 + 2 * 4 + 2 * 3 * 32 * 2 * 2),
                "flops": px * 2 * (3 * macs - first)}
    cells = case["ny"] * case["nx"]
    if kind == "path":  # each step reads the surface (3 fields) and writes the labels
        e = 4 if case["precision"] == "fx32" else 8
        return {"bytes": cells * (8 * 8 + case["steps"] * (3 * e + 4)),
                "flops": cells * 40 * case["steps"]}
    if kind == "mobile":  # about three CFL substeps a step, each reads 4 and writes 3 fields
        e = 4 if case["precision"] == "fx32" else 8
        return {"bytes": cells * (6 * 8 + case["steps"] * 3 * 7 * e),
                "flops": cells * 200 * 3 * case["steps"]}
    if kind == "solver":
        return {"bytes": cells * 8 * 7, "flops": cells * 200 * 3}
    # relaxation: the heights in and out; some hundred sweeps of four directions
    return {"bytes": cells * 16, "flops": cells * 4 * 6 * 200}


# ---------------------------------------------------------------------------
# 64-bit values in plain torch
# ---------------------------------------------------------------------------
def _div(a, b, where):
    return torch.where(where, a / torch.where(where, b, torch.ones_like(b)), torch.zeros_like(a))


def _faces(b, h, qn, qt, lam, dry, K=0.45, g=9.81):
    """Rusanov face fluxes along the last axis with hydrostatic reconstruction;
    returns the changes of (h, normal, tangential momentum)."""
    lo, hi = (Ellipsis, slice(None, -1)), (Ellipsis, slice(1, None))
    top = torch.maximum(b[lo], b[hi])
    side = []
    for k in (lo, hi):
        hs = ((b[k] + K * h[k] - top) / K).clamp_min(0.0)
        f = _div(hs, h[k], h[k] > dry)
        n, t = qn[k] * f, qt[k] * f
        wet = hs > dry
        u, v = _div(n, hs, wet), _div(t, hs, wet)
        side.append((hs, n, t, n * u + 0.5 * K * g * hs * hs, n * v,
                     u.abs() + torch.sqrt(K * g * hs), 0.5 * K * g * (h[k] ** 2 - hs * hs)))
    (hl, nl, tl, fl, gl, sl, cl), (hr, nr, tr, fr, gr, sr, cr) = side
    half = 0.5 * torch.maximum(sl, sr)
    fh = 0.5 * (nl + nr) - half * (hr - hl)
    fn = 0.5 * (fl + fr) - half * (nr - nl)
    ft = 0.5 * (gl + gr) - half * (tr - tl)
    dh, dn, dt = torch.zeros_like(h), torch.zeros_like(h), torch.zeros_like(h)
    dh[lo] -= lam * fh
    dh[hi] += lam * fh
    dn[lo] -= lam * (fn + cl)
    dn[hi] += lam * (fn + cr)
    dt[lo] -= lam * ft
    dt[hi] += lam * ft
    return dh, dn, dt


def _steepest(H):
    """Largest |gradient| of each patch (central differences, one-sided edges)."""
    gy, gx = torch.gradient(H, spacing=DX, dim=(-2, -1), edge_order=1)
    return torch.hypot(gx, gy).amax((-2, -1))


def _flow(b, h, qx, qy, *, dt, cfl, mu, start_deg, ext=(0.0, 0.0), dry=1e-10, g=9.81, K=0.45):
    """One physics step of patches [P, ny, nx]; returns (h, qx, qy, substeps [P])."""
    P = h.shape[0]
    moving = torch.maximum(qx.abs().amax((-2, -1)), qy.abs().amax((-2, -1))) > 1e-14
    live = moving | (_steepest(b + h) > math.tan(math.radians(start_deg)) + 1e-14)
    if ext != (0.0, 0.0):
        live = torch.ones_like(live)
    rem = torch.where(live, dt, 0.0)
    subs = torch.zeros(P, dtype=torch.int64, device=h.device)
    while True:
        run = rem > 1e-14
        if not bool(run.any()):
            return h, qx, qy, subs
        wet = h > dry
        w = (torch.sqrt(_div(qx, h, wet) ** 2 + _div(qy, h, wet) ** 2)
             + torch.sqrt(K * g * h.clamp_min(0.0))).amax((-2, -1))
        sub = torch.where(run, torch.minimum(rem, torch.where(w > 1e-14, cfl * DX / w, rem)), 0.0)
        k = sub[:, None, None]
        lam = k / DX
        dh, dx_, dy_ = _faces(b, h, qx, qy, lam, dry)
        th, ty, tx = _faces(b.transpose(1, 2), h.transpose(1, 2), qy.transpose(1, 2),
                            qx.transpose(1, 2), lam, dry)
        hn = (h + dh + th.transpose(1, 2)).clamp_min(0.0)
        wet = hn > dry
        nx = torch.where(wet, qx + dx_ + tx.transpose(1, 2), 0.0) + hn * ext[0] * k
        ny = torch.where(wet, qy + dy_ + ty.transpose(1, 2), 0.0) + hn * ext[1] * k
        u, v = _div(nx, hn, wet), _div(ny, hn, wet)
        spd = torch.sqrt(u * u + v * v)
        f = (1.0 - mu * g * k / spd.clamp_min(1e-15)).clamp_min(0.0)
        go = run[:, None, None]
        h, qx, qy = (torch.where(go, hn, h), torch.where(go, hn * u * f, qx),
                     torch.where(go, hn * v * f, qy))
        rem = rem - sub
        subs += run


def _repose(h, crit, tol, limit):
    """Eight-phase coloured relaxation of one height map; returns (heights, sweeps)."""
    ny, nx = h.shape
    row = torch.arange(ny, device=h.device)[:, None].expand(ny, nx)
    col = torch.arange(nx, device=h.device)[None, :].expand(ny, nx)
    phases = []
    for dr, dc in ((1, 0), (0, 1), (1, 1), (1, -1)):
        c0, c1 = max(0, -dc), nx - max(0, dc)
        a = (slice(0, ny - dr), slice(c0, c1))
        b = (slice(dr, ny), slice(c0 + dc, c1 + dc))
        limit_h = crit * math.hypot(dr * DX, dc * DX)
        line = row[a] if dr else col[a]
        for par in (0, 1):
            phases.append((a, b, limit_h, (line % 2 == par).to(h.dtype)))
    h = h.clone()
    for it in range(1, limit + 1):
        worst = torch.zeros((), device=h.device, dtype=h.dtype)
        for a, b, limit_h, on in phases:
            d = h[a] - h[b]
            ex = (d.abs() - limit_h).clamp_min(0.0)
            worst = torch.maximum(worst, ex.max())
            t = 0.5 * ex * torch.sign(d) * on
            h[a] -= t
            h[b] += t
        if float(worst) <= tol:
            break
    return h, it


def exact(case, seed):
    kind = case["kind"]
    if kind == "path":
        if case["residual"] == "always":
            return None  # the frontier's own schedule of whole tiles has no closed form
        b = _pile(case["ny"], case["nx"], seed)
        sched = _cut_schedule(case, seed, b.cpu().numpy())
        h = torch.zeros_like(b)
        b, h, qx, qy = b[None], h[None], h[None], h[None]
        for idx, tgt in sched:
            at = torch.from_numpy(idx).long().to(DEV)
            fb, fh = b.reshape(-1), h.reshape(-1)
            d = torch.minimum((fb[at] - torch.from_numpy(tgt).to(DEV)).clamp_min(0.0),
                              fb[at].clamp_min(0.0))
            fb[at] -= d
            h = h.clone()
            h.reshape(-1)[at] += d
            h, qx, qy, _ = _flow(b, h, qx, qy, dt=DT, cfl=0.18, mu=FRICTION, start_deg=START_DEG)
        return {"fields": {"b_eff": b[0], "mobile": h[0], "momentum_x": qx[0],
                           "momentum_y": qy[0]}, "labels": None, "record": None}
    if kind == "mobile":
        b, h, qx, qy = (t[None] for t in _moving_layer(case["ny"], case["nx"], seed))
        for _ in range(case["steps"]):
            h, qx, qy, _ = _flow(b, h, qx, qy, dt=DT, cfl=0.18, mu=0.15, start_deg=34.0)
        return {"fields": {"mobile": h[0], "momentum_x": qx[0], "momentum_y": qy[0]},
                "substeps": None}
    if kind == "solver":
        z, h = _mound(case["ny"], case["nx"], np.random.default_rng([seed, 13]))
        h, qx, qy, _ = _flow(z[None], h[None], 0.3 * h[None], -0.2 * h[None], dt=DT, cfl=0.4,
                             mu=REPOSE, start_deg=34.0,
                             ext=(0.4, -0.3) if case["external"] else (0.0, 0.0))
        return {"h": h[0], "q": torch.stack((qx[0], qy[0]), dim=-1), "substeps": None}
    if kind == "batch":
        parts = _patches(case, seed)
        groups = {}
        for i, (z, h) in enumerate(parts):
            groups.setdefault(tuple(h.shape), []).append(i)
        done = [None] * len(parts)
        for at in groups.values():
            b = torch.stack([parts[i][0] for i in at])
            h = torch.stack([parts[i][1] for i in at])
            qx, qy = torch.zeros_like(h), torch.zeros_like(h)
            for _ in range(case["steps"]):
                h, qx, qy, _ = _flow(b, h, qx, qy, dt=DT, cfl=case["cfl"], mu=REPOSE,
                                     start_deg=34.0)
            for j, i in enumerate(at):
                done[i] = (h[j].reshape(-1), qx[j].reshape(-1), qy[j].reshape(-1))
        return {"substeps": None, "mobile": torch.cat([d[0] for d in done]),
                "momentum_x": torch.cat([d[1] for d in done]),
                "momentum_y": torch.cat([d[2] for d in done])}
    if kind == "relax":
        h, _ = _repose(_cut_pile(case["ny"], case["nx"], seed), REPOSE,
                       case["tolerance"], 20000)
        return {"height": h, "iterations": None}
    if kind == "settle":
        if case["schedule"] == "learned":
            return None  # the network's proposals decide the path to repose
        h, _ = _repose(_cut_pile(case["ny"], case["nx"], seed), REPOSE,
                       1e-4 * DX, 20000)
        return {"height": h, "sweeps": None}
    weights, pre, target = _train_inputs(case, seed)
    tan = REPOSE
    n, b = case["n"], case["batch"]
    edges = ((0, 1), (1, 0), (1, 1), (1, -1))
    feat = torch.zeros(b, 4, n, n, device=DEV, dtype=torch.float64)
    for k, (dr, dc) in enumerate(edges):
        c0, c1 = max(0, -dc), n - max(0, dc)
        feat[:, k, :n - dr, c0:c1] = ((pre[:, :n - dr, c0:c1] - pre[:, dr:, c0 + dc:c1 + dc])
                                      / (math.hypot(dr * DX, dc * DX) * tan))
    params, x = [], feat
    for li, ((ci, co), (ri, ro)) in enumerate(zip(learned.LAYERS, learned.REAL)):
        w = weights[li][:, :, :ri, :ro].to(DEV).double().requires_grad_()
        params.append(w)
        x = torch.nn.functional.conv2d(x, w.permute(3, 2, 0, 1), padding=1)
        if li < 3:
            x = torch.relu(x)
    dh = torch.zeros(b, n, n, device=DEV, dtype=torch.float64)
    for k, (dr, dc) in enumerate(edges):
        c0, c1 = max(0, -dc), n - max(0, dc)
        t = x[:, k, :n - dr, c0:c1] * (tan * DX)
        dh = dh - torch.nn.functional.pad(t, (c0, n - c1, 0, dr))
        dh = dh + torch.nn.functional.pad(t, (c0 + dc, n - c1 - dc, dr, 0))
    loss = ((dh - target.double()) ** 2).sum() / ((tan * DX) ** 2 * b * n * n)
    found = torch.autograd.grad(loss, params)
    grads = []
    for (ci, co), (ri, ro), gr in zip(learned.LAYERS, learned.REAL, found):
        full = torch.zeros(3, 3, ci, co, device=DEV, dtype=torch.float64)
        full[:, :, :ri, :ro] = gr
        grads.append(full)
    return {"loss": float(loss), "grads": grads,
            "flux": x.permute(0, 2, 3, 1).contiguous().detach()}
