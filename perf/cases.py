"""The work that a user of this framework has it do, as cases that can be timed and compared.

Three kinds, each through the public Python entry points:

frame   one steady frame of one map (`DOM.updatePose` + `DOM.updateGrid` / `updateGridAsync`), for
        both variants, scans on the host or in device memory, and the map read back the way the
        program reads it: as a registered occupancy output or as the node's GridCell array.
batch   one steady frame of many independent maps (`BatchDOM`).
calib   the differentiable update: a gradient step on the kernel-inference parameters
        (`calibration_loss` + backward + the parameter step), or the occupancy at candidate
        parameters (`Calibration.occupancy`).

Sizes are those of the repository's configurations (scene.config0 .. config4, scene.small and the
YAML files of the tests), and `draw` spreads others over the same ranges.
"""
from __future__ import annotations

import math

import numpy as np
import torch

import k3dom_b200 as K
from k3dom_b200 import calib as KC

DEV = "cuda:0"
SCANS = 6  # scans of a state's sequence, replayed to and fro


# ------------------------------------------------------------------ cases
def _frame(name, variant, G, Gz, res, P, B, points, beams=64, step=0.0, ls=0.3, scans="device", read="occupancy",
           tuned=False, off_x=0.0, off_y=0.0, off_z=0.0):
    return dict(name=name, kind="frame", variant=variant, G=G, Gz=Gz, res=res, P=P, B=B, points=points, beams=beams,
                step=step, ls=ls, scans=scans, read=read, tuned=tuned, off_x=off_x, off_y=off_y, off_z=off_z)


def _batch(name, scenes, g_lo, g_hi, gz_lo, gz_hi, res, p_lo, p_hi, n_lo, n_hi, sizes, variant="k3dom",
           scans="device", read="one", tuned=True):
    return dict(name=name, kind="batch", variant=variant, scenes=scenes, g_lo=g_lo, g_hi=g_hi, gz_lo=gz_lo,
                gz_hi=gz_hi, res=res, p_lo=p_lo, p_hi=p_hi, n_lo=n_lo, n_hi=n_hi, sizes=sizes, scans=scans,
                read=read, tuned=tuned)


def _calib(name, G, Gz, res, points, frames=2, heldout=10, heldout_points=30000, read="grad", ls=0.3):
    return dict(name=name, kind="calib", G=G, Gz=Gz, res=res, points=points, frames=frames, heldout=heldout,
                heldout_points=heldout_points, read=read, ls=ls)


def listed():
    return [
        # scene.small: a close-range map of a small robot, 16 beams; the smallest call, all latency
        _frame("frame_small", "k3dom", 32, 8, 0.2, 16384, 4096, 2000, beams=16),
        # scene.config0: a 12.8 m map from a 32-beam scanner, scans produced on the GPU
        _frame("frame_config0", "k3dom", 64, 16, 0.2, 262144, 65536, 30000, beams=32, step=0.05),
        # k3dom.yaml + kitti.yaml through the node's own cycle: cloud in host memory, a synchronous
        # update, the whole GridCell array read back
        _frame("frame_kitti_cells", "k3dom", 100, 12, 0.4, 1000000, 100000, 60000, step=0.21, ls=0.5, scans="host",
               read="cells", off_z=1.0),
        # k3dom.yaml + complex.yaml: 0.2 m voxels and a kernel of 0.5 m, off-centre sensor, host
        # clouds, the occupancy registered as the frame's output; tiling left at its default
        _frame("frame_complex_host", "k3dom", 200, 25, 0.2, 1000000, 100000, 60000, step=0.21, ls=0.5, scans="host",
               off_x=5.0, off_y=-4.7),
        # scene.config1: 2.1 M voxels, 4.2 M particles, 120,000 returns, moving sensor (map shifts),
        # tiling autotuned on live frames as a long-running program has it
        _frame("frame_config1", "k3dom", 256, 32, 0.1, 4194304, 1048576, 120000, step=0.21, tuned=True),
        # scene.config2: the same map under the DS-PHD/MIB variant
        _frame("ds_config2", "dsphdmib", 256, 32, 0.1, 4194304, 1048576, 120000, step=0.21, tuned=True),
        # dsphdmib.yaml + complex.yaml: the DS node's parameters, host clouds
        _frame("ds_complex_host", "dsphdmib", 200, 25, 0.2, 1000000, 100000, 60000, step=0.21, scans="host",
               off_x=5.0, off_y=-4.7),
        # scene.config3: sixteen uneven maps stepped together (a fleet's replay), the largest call
        _batch("batch_config3", 16, 64, 256, 16, 32, 0.1, 18, 22, 10000, 200000, 3),
        # many small maps stepped together, every map read each frame: parameter sweeps, simulated robots
        _batch("batch_small", 24, 32, 64, 8, 16, 0.2, 14, 18, 2000, 30000, 5, read="all", tuned=False),
        # scene.config4: a gradient step of the calibration on config0's grid
        _calib("calib_config0", 64, 16, 0.2, 30000),
        # the same on config1's grid, held-out scans of 120,000 returns
        _calib("calib_config1", 256, 32, 0.1, 120000, heldout_points=120000),
        # the map at candidate parameters, three training frames on a ragged grid
        _calib("calib_occupancy", 90, 13, 0.2, 25001, frames=3, heldout=3, heldout_points=10007, read="occupancy"),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["frame", "frame", "frame", "frame", "batch", "calib"])
    if kind == "frame":
        res = rng.choice([0.1, 0.2, 0.4])
        G, Gz = _log(rng, 24, 256), rng.randint(6, 32)
        P = _log(rng, 10000, 4194304)
        variant = rng.choice(["k3dom", "k3dom", "dsphdmib"])
        c = _frame("", variant, G, Gz, res, P, max(1, P // rng.choice([4, 10])), _log(rng, 1500, 120000),
                   beams=rng.choice([16, 32, 64]), step=rng.choice([0.0, 0.05, 0.21]),
                   ls=0.3 if res == 0.1 else rng.choice([0.3, 0.5]), scans=rng.choice(["device", "host"]),
                   read=rng.choice(["occupancy", "occupancy", "cells"]), tuned=rng.random() < 0.3)
        if c["read"] == "cells" and G * G * Gz <= 300000:
            c["scans"] = "host"
        else:  # the whole array of a large map takes longer to copy than the frame: not read each frame
            c["read"] = "occupancy"
    elif kind == "batch":
        res = rng.choice([0.1, 0.2])
        hi = _log(rng, 48, 200)
        p_hi = rng.randint(15, 20)
        n_hi = _log(rng, 5000, 90000)
        c = _batch("", rng.randint(2, 16), max(24, hi // 3), hi, 8, rng.randint(12, 32), res, 14, p_hi,
                   max(1000, n_hi // 10), n_hi, rng.randint(0, 1 << 20),
                   variant=rng.choice(["k3dom", "k3dom", "dsphdmib"]), scans=rng.choice(["device", "host"]),
                   read="all" if hi <= 80 else "one", tuned=rng.random() < 0.5)
    else:
        res = rng.choice([0.1, 0.2])
        c = _calib("", _log(rng, 32, 200), rng.randint(8, 32), res, _log(rng, 3000, 100000),
                   frames=rng.choice([1, 2, 2, 3, 5]), heldout=rng.randint(1, 8),
                   heldout_points=_log(rng, 2000, 40000), read=rng.choice(["grad", "grad", "occupancy"]))
    del c["name"]
    return c


# ------------------------------------------------------------------ scenes, made on the GPU
class _World:
    """Ground, cuboids (half of them moving) and an enclosing wall, as k3dom_b200.scene lays them
    out; scans are ray cast on the GPU. Every number comes from the seed."""

    def __init__(self, seed, G, Gz, res, beams, step, n_boxes=20):
        self.g = torch.Generator(device=DEV).manual_seed(int(seed))
        size = G * res
        self.max_range = size
        self.ground = -min(1.5, 0.45 * Gz * res)
        extent = max(1.2, size / 2 - 0.5)
        side = self._u(n_boxes, 3) * min(1.0, size / 8) + min(1.0, size / 16)
        ang = self._u(n_boxes) * 2 * math.pi
        r = 1.2 + side.max() + self._u(n_boxes) * extent
        self.half = side / 2
        self.centre = torch.stack([r * torch.cos(ang), r * torch.sin(ang), self.ground + self.half[:, 2]], 1)
        sp, hd = self._u(n_boxes) * 3.0 * (torch.arange(n_boxes, device=DEV) % 2), self._u(n_boxes) * 2 * math.pi
        self.vel = torch.stack([sp * torch.cos(hd), sp * torch.sin(hd), torch.zeros_like(sp)], 1)
        hd = float(self._u(1)[0]) * 2 * math.pi
        self.ego = np.array([step * math.cos(hd), step * math.sin(hd), 0.0])  # per frame
        self.beams = beams

    def _u(self, *shape):
        return torch.rand(*shape, generator=self.g, device=DEV, dtype=torch.float64)

    def scan(self, k, n, offset=(0.0, 0.0, 0.0), turn=0.0):
        """(sensor position, (n, 3) float32 CUDA tensor of sensor-relative points) of frame k."""
        s = self.ego * k + np.asarray(offset, np.float64)
        st = torch.tensor(s, device=DEV)
        n_az = -(-n // self.beams)
        az = torch.arange(n_az, device=DEV, dtype=torch.float64) * (2 * math.pi / n_az) + turn
        el = torch.deg2rad(torch.linspace(-25.0, 15.0, self.beams, device=DEV, dtype=torch.float64))
        d = torch.stack([torch.cos(el)[:, None] * torch.cos(az), torch.cos(el)[:, None] * torch.sin(az),
                         torch.sin(el)[:, None].expand(self.beams, n_az)], -1).reshape(-1, 3)[:n]
        t = self.max_range / torch.hypot(d[:, 0], d[:, 1]).clamp_min(1e-9)
        tg = (self.ground - s[2]) / d[:, 2]
        t = torch.where((d[:, 2] < 0) & (tg > 0), torch.minimum(t, tg), t)
        c = self.centre + self.vel * (0.1 * k) - st
        t0, t1 = (c - self.half)[None] / d[:, None], (c + self.half)[None] / d[:, None]
        near, far = torch.minimum(t0, t1).amax(-1), torch.maximum(t0, t1).amin(-1)
        hit = torch.where((far >= near) & (near > 0), near, math.inf)
        t = torch.minimum(t, hit.amin(1))
        t = t + 0.02 * torch.randn(n, generator=self.g, device=DEV, dtype=torch.float64)
        return s, (d * t[:, None]).to(torch.float32)


def _params(variant, G, Gz, res, P, B, points, ls, seed, off=(0.0, 0.0, 0.0)):
    """The reference YAML files' values in index units, as the node converts them."""
    size, size_z = (G + 0.5) * res, (Gz + 0.5) * res  # the grid is the integer part of size / resolution
    ds = variant == "dsphdmib"
    prior = 0.0 if ds else 0.001
    return K.make_params(variant, size=size, size_z=size_z, resolution=res, particle_count=P,
                         new_born_particle_count=B, mass_scale=2.5, persistence_prob=0.99,
                         stddev_process_noise_position=0.01 / res, stddev_process_noise_velocity=0.1 / res,
                         birth_prob=0.02, stddev_velocity=4.0 / res, init_max_velocity=5.0 / res,
                         particle_min_vel=0.0 if ds else 0.1 / res, sensor_off_x=off[0], sensor_off_y=off[1],
                         sensor_off_z=off[2], map_shift_thresh=int(1.0 / res), prior_free=prior, prior_static=prior,
                         prior_dynamic=prior, prior_occ=0.0, sigma=0.1, ls=ls, gamma=0.99, max_range=50.0,
                         meas_occ_stddev=0.1, seed=seed, max_points=points)


def _scans(world, n, host):
    out = []
    for k in range(SCANS):
        s, p = world.scan(k, n)
        out.append((s, p.cpu().numpy() if host else p))
    return out


def _at(k):
    """Scan of pass k: 0 1 2 3 4 5 4 3 2 1 0 ... (the sensor drives to and fro)."""
    k %= 2 * (SCANS - 1)
    return k if k < SCANS else 2 * (SCANS - 1) - k


def _field(variant):
    return "occ_mean" if variant == "k3dom" else "occ_prob"


def _prepare_frame(c, seed):
    world = _World(seed, c["G"], c["Gz"], c["res"], c["beams"], c["step"])
    scans = _scans(world, c["points"], c["scans"] == "host")
    dom = K.DOM(_params(c["variant"], c["G"], c["Gz"], c["res"], c["P"], c["B"], c["points"], c["ls"], seed + 1,
                        (c["off_x"], c["off_y"], c["off_z"])), c["variant"])
    out = None
    if c["read"] == "occupancy":
        n = dom.grid_cell_count
        out = torch.zeros(n, device=DEV) if c["scans"] == "device" else torch.zeros(n).pin_memory()
        torch.cuda.synchronize()
        dom.set_output(_field(c["variant"]), out)
    st = dict(kind="frame", dom=dom, scans=scans, k=0, out=out, device=c["scans"] == "device")
    warm = 3
    if c["tuned"]:
        dom.autotune(True)
        warm += dom.tuning()["candidates"]
    for _ in range(warm):  # the first frame, the tuning's frames, and the frame program's capture
        _step_frame(st)
    dom.synchronize()
    return st


def _step_frame(st):
    dom, k = st["dom"], st["k"]
    st["k"] = k + 1
    s, pts = st["scans"][_at(k)]
    dom.updatePose(*s)
    if st["device"]:
        dom.updateGridAsync(0.1 * (k + 1), pts)
    else:
        dom.updateGrid(0.1 * (k + 1), pts)


def _run_frame(st):
    _step_frame(st)
    if st["out"] is not None:
        return st["out"]
    cells = st["dom"].get_gridcells()
    words = cells.view(np.int32).reshape(-1, 17)
    return {"ranges": words[:, :2], "values": words[:, 2:].view(np.float32)}


def _batch_sizes(c):
    """The scenes' sizes: part of the case (they follow from its "sizes" number, not the seed)."""
    rng = np.random.Generator(np.random.PCG64(c["sizes"]))
    out = []
    for _ in range(c["scenes"]):
        out.append((int(rng.integers(c["g_lo"], c["g_hi"] + 1)), int(rng.integers(c["gz_lo"], c["gz_hi"] + 1)),
                    int(round(2.0 ** rng.uniform(c["p_lo"], c["p_hi"]))), int(rng.integers(c["n_lo"], c["n_hi"] + 1))))
    return out


def _prepare_batch(c, seed):
    host = c["scans"] == "host"
    params, scans = [], []
    for s, (G, Gz, P, n) in enumerate(_batch_sizes(c)):
        world = _World(seed * 1000 + s, G, Gz, c["res"], 64, 0.1)
        scans.append(_scans(world, n, host))
        params.append(_params(c["variant"], G, Gz, c["res"], P, max(1, P // 4), n, 0.3, seed * 64 + s + 1))
    b = K.BatchDOM(params, c["variant"])
    out = None
    if c["read"] == "one":  # one map followed each frame, the others read when they are asked for
        out = torch.zeros(b.scene(0).grid_cell_count, device=DEV)
        torch.cuda.synchronize()
        b.scene(0).set_output(_field(c["variant"]), out)
    st = dict(kind="batch", dom=b, scans=scans, k=0, out=out, host=host, field=_field(c["variant"]))
    warm = 3
    if c["tuned"]:
        b.autotune(True)
        warm += b.tuning()["candidates"]
    for _ in range(warm):
        _step_batch(st)
    b.synchronize()
    return st


def _step_batch(st):
    b, k = st["dom"], st["k"]
    st["k"] = k + 1
    j = _at(k)
    for s in range(len(b)):
        b.updatePose(s, *st["scans"][s][j][0])
    t = [0.1 * (k + 1)] * len(b)
    (b.update if st["host"] else b.update_async)(t, [v[j][1] for v in st["scans"]])


def _run_batch(st):
    _step_batch(st)
    if st["out"] is not None:
        return st["out"]
    return [st["dom"].scene(s).get_cell_field(st["field"]) for s in range(len(st["dom"]))]


THETA0 = (0.3, 1.0, 0.1, 0.01, 0.01)
RATE, FLOOR = 1e-3, 1e-3  # the calibration loop's step and the projection that keeps theta positive


def _calib_inputs(c, seed):
    """Training frames [(dt, sensor, points, particle weight sums)] and held-out scans."""
    world = _World(seed, c["G"], c["Gz"], c["res"], 32 if c["points"] < 60000 else 64, 0.05)
    C = c["G"] * c["G"] * c["Gz"]
    rng = np.random.Generator(np.random.PCG64(seed))
    frames = []
    for k in range(c["frames"]):
        s, p = world.scan(k, c["points"])
        dyn = None
        if k > 0:  # the particle filter's weight sums: a few occupied cells
            u = world._u(C)
            dyn = torch.where(u > 0.9, (u - 0.9) * 5.0, 0.0).to(torch.float32).cpu().numpy()
        frames.append((0.1 if k else 0.0, s.astype(np.float32), p.cpu().numpy(), dyn))
    held = []
    for _ in range(c["heldout"]):
        off = rng.uniform(-0.5, 0.5, 3) * np.array([1.0, 1.0, 0.2])
        s, p = world.scan(c["frames"] - 1, c["heldout_points"], off, float(rng.uniform(0, 2 * math.pi)))
        held.append((s.astype(np.float32), p.cpu().numpy()))
    return frames, held


def _prepare_calib(c, seed):
    frames, held = _calib_inputs(c, seed)
    prob = KC.Calibration(_params("k3dom", c["G"], c["Gz"], c["res"], 1024, 256, c["points"], c["ls"], 1))
    for dt, s, p, dyn in frames:
        prob.add_frame(dt, s, p, dyn)
    for s, p in held:
        prob.add_heldout(s, p)
    return dict(kind="calib", calib=prob, k=0, read=c["read"],
                theta=torch.tensor((c["ls"],) + THETA0[1:], dtype=torch.float32))


def _run_calib(st):
    k = st["k"]
    st["k"] = k + 1
    if st["read"] == "occupancy":  # a sweep over candidate length-scales
        th = st["theta"].clone()
        th[0] *= 1.0 + 2e-3 * (k % 16)
        return st["calib"].occupancy(th.numpy())
    theta = st["theta"].clone().requires_grad_(True)
    loss = KC.calibration_loss(theta, st["calib"])
    loss.backward()
    with torch.no_grad():
        st["theta"] = (theta - RATE * theta.grad).clamp_min(FLOOR)
    return {"loss": loss.detach(), "grad": theta.grad, "theta": st["theta"]}


# ------------------------------------------------------------------ what is measured
def prepare(case, seed):
    return {"frame": _prepare_frame, "batch": _prepare_batch, "calib": _prepare_calib}[case["kind"]](case, int(seed))


def run(state):
    return {"frame": _run_frame, "batch": _run_batch, "calib": _run_calib}[state["kind"]](state)


def _evals(G, Gz, res, n, ls):
    """In-support (cell, ray) evaluations of a scan: rays of about a third of the grid's width in
    length, with ls around them."""
    return n * (0.33 * G) * math.pi * (ls / res) ** 2


def _frame_work(variant, G, Gz, res, P, B, n, ls, read):
    C = G * G * Gz
    ds = variant == "dsphdmib"
    # particles read once and written once (33 B each way), births written, the cells' state
    # (10 floats) read and written, the scan, and what is read back
    b = 66 * P + 33 * B + 80 * C + 12 * n + (68 if read == "cells" else 4) * C
    # K3DOM: 20 FLOP per in-support evaluation; DS: 25 per neighbour within the 0.866-voxel window
    e = n * (0.5 * G) * math.pi * 0.75 * 25 if ds else _evals(G, Gz, res, n, ls) * 20
    return b, e + 150.0 * P + 60.0 * C


def work(case):
    c = case
    if c["kind"] == "frame":
        b, f = _frame_work(c["variant"], c["G"], c["Gz"], c["res"], c["P"], c["B"], c["points"], c["ls"], c["read"])
    elif c["kind"] == "batch":
        b = f = 0.0
        for G, Gz, P, n in _batch_sizes(c):
            x, y = _frame_work(c["variant"], G, Gz, c["res"], P, P // 4, n, 0.3, "occupancy")
            b, f = b + x, f + y
    else:
        C = c["G"] * c["G"] * c["Gz"]
        # per frame the scan and the weight sums; the labels once; 30 FLOP per evaluation (value and
        # derivative), 200 per cell and frame for the recursion and its adjoint
        b = c["frames"] * (12 * c["points"] + 4 * C) + 8 * C + (4 * C if c["read"] == "occupancy" else 0)
        f = c["frames"] * (_evals(c["G"], c["Gz"], c["res"], c["points"], c["ls"]) * 30 + 200.0 * C)
    return {"bytes": float(b), "flops": float(f)}


# ------------------------------------------------------------------ 64-bit values
def exact(case, seed):
    """The calibration's outputs in FP64. A map's frame has no such value: it depends on the
    particles' random draws and on the discrete choices (voxels, slots, ancestors) made in FP32."""
    c = case
    if c["kind"] != "calib":
        return None
    C = c["G"] * c["G"] * c["Gz"]
    if float(C) * c["points"] * c["frames"] > 2.5e10:  # more than about 20 s of pairs
        return None
    frames, held = _calib_inputs(c, int(seed))
    f64 = dict(device=DEV, dtype=torch.float64)
    res = float(np.float32(c["res"]))
    th = np.array((c["ls"],) + THETA0[1:], np.float32).astype(np.float64)
    ix = torch.arange(C, device=DEV)
    half = torch.tensor([c["G"] / 2.0, c["G"] / 2.0, c["Gz"] / 2.0], **f64)
    idx = torch.stack([ix % c["G"], ix // c["G"] % c["G"], ix // (c["G"] * c["G"])], 1).to(torch.float64)
    sums = []
    for _, s, p, _ in frames:
        x = (idx + 0.5 - half) * res - torch.tensor(s, **f64)
        sums.append(_pair_sums(x, torch.tensor(p, **f64), float(th[0]), res))
    labels = None
    if c["read"] == "grad":
        labels = _labels(c, held, res)
    t = torch.tensor(th, **f64).requires_grad_(True)
    p = _recursion(t, frames, sums, C)
    if c["read"] == "occupancy":
        return p.detach().cpu().numpy()
    n0, n1 = labels
    q = p.clamp(1e-7, 1 - 1e-7)
    loss = -(n1 * torch.log(q) + n0 * torch.log(1 - q)).sum() / (n0.sum() + n1.sum())
    loss.backward()
    g = t.grad.cpu()
    return {"loss": loss.detach().cpu(), "grad": g, "theta": (t.detach().cpu() - RATE * g).clamp_min(FLOOR)}


def _pair_sums(x, m, ls, res):
    """Per cell: sums of f(d / ls) over the occupied and the free pairs, and of -x f'(x)."""
    out = torch.zeros(4, x.shape[0], device=DEV, dtype=torch.float64)
    dm = m.norm(dim=1)
    u = m / dm.clamp_min(1e-300)[:, None]
    margin = torch.maximum(0.9 * dm, dm - 2.0 * res)
    x2 = (x * x).sum(1)
    step = max(1, 150_000_000 // x.shape[0])
    for a in range(0, m.shape[0], step):
        d, mg = dm[a:a + step], margin[a:a + step]
        proj = x @ u[a:a + step].T
        along = proj.clamp_max(0.0) + (proj - mg).clamp_min(0.0)
        # |x|^2 - proj^2 in 64 bits: 1e-14 of squares of some tens of metres
        df = (x2[:, None] - proj * proj).clamp_min(0.0) + along * along
        df = torch.where(proj < d, df, math.inf)
        do = x2[:, None] - 2.0 * proj * d + (d * d)
        for row, d2 in ((0, do), (1, df)):
            near = (d2 < ls * ls).nonzero(as_tuple=True)
            r = d2[near].clamp_min(0.0).sqrt() / ls
            w = 2 * math.pi
            f = (2 + torch.cos(w * r)) * (1 - r) / 3 + torch.sin(w * r) / (2 * 3.141592)
            fp = (-w * torch.sin(w * r) * (1 - r) - (2 + torch.cos(w * r))) / 3 + w * torch.cos(w * r) / (2 * 3.141592)
            on = f > 0
            out[row].index_add_(0, near[0], torch.where(on, f, 0.0))
            out[row + 2].index_add_(0, near[0], torch.where(on, -r * fp, 0.0))
    return out


def _recursion(t, frames, sums, C):
    """Occupancy of every cell after the frames, at theta = t (differentiable at its value)."""
    ls, sigma, gamma, po, pf = t
    one = torch.ones(C, device=DEV, dtype=torch.float64)
    mf, ms, md = pf * one, po / 2 * one, po / 2 * one

    def credit(v):
        return torch.tanh(v / 2.5)  # 1 - 2 / (1 + exp(2 v / mass_scale))

    def pos(v):
        return v.clamp_min(0.0)

    for (dt, _, _, dyn), s in zip(frames, sums):
        lin = (ls - ls.detach()) / ls.detach()  # zero; carries dE / dls = sigma H / ls
        eo, ef = sigma * (s[0] + lin * s[2]), sigma * (s[1] + lin * s[3])
        g = gamma ** float(np.float32(dt)) if dt else torch.ones((), device=DEV, dtype=torch.float64)
        w = torch.zeros_like(one) if dyn is None else torch.tensor(dyn, device=DEV, dtype=torch.float64)
        total = (mf + md) * g
        s1 = ms * g
        d1 = torch.minimum(w, pos(total - s1))
        f1 = total - d1
        on = (eo.detach() > 0) | (ef.detach() > 0)
        a, b = torch.where(on, eo, 1.0), torch.where(on, ef, 1.0)
        z = (a + b) * (f1 + s1 + d1)
        k = credit(z.sqrt()) / z
        dtf, stf, ftd = k * pos(b - a) * d1, k * pos(b - a) * pos(s1 + d1 - f1), k * pos(a - b) * pos(f1 - s1 - d1)
        f2 = f1 + stf / 2 * s1 + dtf * d1 - ftd * f1
        s2 = s1 - stf * s1
        d2 = d1 + ftd * f1 + stf / 2 * s1 - dtf * d1
        cr = credit(s2 + d2)
        ok = (s2.detach() > 0) & (d2.detach() >= 0)
        ratio = torch.where(ok, s2 / torch.where(ok, s2 + d2, 1.0), 0.0)
        beta = (1 - cr) + cr * ratio
        mf = torch.where(on, f2 + b, f1)
        ms = torch.where(on, s2 + beta * a, s1)
        md = torch.where(on, d2 + (1 - beta) * a, d1)
    return (ms + md) / (mf + ms + md)


def _labels(c, held, res):
    """Held-out label counts by 3-D traversal: 1 for the voxel of a hit, 0 for those before it."""
    dims = torch.tensor([c["G"], c["G"], c["Gz"]], device=DEV)
    C = c["G"] * c["G"] * c["Gz"]
    stride = torch.tensor([1, c["G"], c["G"] * c["G"]], device=DEV)
    n0 = torch.zeros(C, device=DEV, dtype=torch.float64)
    n1 = torch.zeros_like(n0)
    for s, p in held:
        a = torch.tensor(s, device=DEV, dtype=torch.float64) / res + dims / 2.0
        m = torch.tensor(p, device=DEV, dtype=torch.float64)
        b = (torch.tensor(s, device=DEV, dtype=torch.float64) + m) / res + dims / 2.0
        d = b - a
        v, e = torch.floor(a).expand_as(b).clone().long(), torch.floor(b).long()
        step = torch.sign(d).long()
        tdel = torch.where(d != 0, 1.0 / d.abs(), math.inf)
        edge = torch.where(d > 0, v + 1 - a, a - v)
        tmax = torch.where(d != 0, edge * tdel, math.inf)
        left = (e - v).abs().sum(1) + 1
        live = torch.arange(m.shape[0], device=DEV)
        while live.numel():
            go = ((v[live] != e[live]).any(1)) & (left[live] > 0)
            live = live[go]
            vl = v[live]
            inside = ((vl >= 0) & (vl < dims)).all(1)
            n0.index_add_(0, (vl[inside] * stride).sum(1), torch.ones(int(inside.sum()), device=DEV, dtype=n0.dtype))
            k = torch.argmin(tmax[live], dim=1)
            v[live, k] += step[live, k]
            tmax[live, k] += tdel[live, k]
            left[live] -= 1
        inside = ((e >= 0) & (e < dims)).all(1)
        n1.index_add_(0, (e[inside] * stride).sum(1), torch.ones(int(inside.sum()), device=DEV, dtype=n0.dtype))
    return n0, n1
