"""The work that users of this framework have it do, as cases that can be timed.

A streamline study traces a DTM (fields in both directions, recorded
trajectories), conditions it first (preprocess), maps channels and segments
from the fields, and estimates densities of the log lengths (KDE); many small
tiles go through one batched launch; the learned scheduler is trained and
asked for predictions.  Each case is one of these calls through its public
entry point: tensor-level where the caller's arrays live on the GPU, the stage
classes where they live on the host.

Terrain is made on the GPU from the seed alone, after the recipes of
``slm_b200.synth``: fBm hills on a tilt ("hills"), fBm with incised valleys
("incised"), and mountains over an alluvial fan with unfilled pits ("fan").
"""
from __future__ import annotations

import math
import types

import numpy as np
import torch

from slm_b200 import kernels
from slm_b200.analysis import Bivariate_distribution, Univariate_distribution
from slm_b200.batch import Tile, TileBatch
from slm_b200.fields import Fields
from slm_b200.mapping_device import DeviceMapping
from slm_b200.params import kernel_params
from slm_b200.preprocess import conditioned_gradient_vector_field
from slm_b200.scheduler import LengthModel, bf16_round, init_params, spatial_order
from slm_b200.trajectories import Trajectories
from slm_b200.useful import Data, Info, compute_stats, create_seeds, default_parameters

PAD = 2


def listed():
    return [
        # the smallest trace: one 256 px tile, where launch latency and the
        # longest trajectory decide
        {"name": "fields_tile256_rk2", "kind": "fields", "terrain": "hills", "nx": 256, "ny": 256, "density": 2,
         "jitter": 1.0, "rk": 2, "step": 0.1, "max_steps": 2000, "pixel": 1.0},
        # an ordinary study area of no round size: incised relief at 2 m, RK4
        {"name": "fields_incised_odd_rk4", "kind": "fields", "terrain": "incised", "nx": 1531, "ny": 2039,
         "density": 2, "jitter": 1.0, "rk": 4, "step": 0.1, "max_steps": 10000, "pixel": 2.0},
        # the large divergent terrain: mountains, fan and pits, RK4
        {"name": "fields_fan4096_rk4", "kind": "fields", "terrain": "fan", "nx": 4096, "ny": 4096, "density": 2,
         "jitter": 1.0, "rk": 4, "step": 0.1, "max_steps": 20000, "pixel": 1.0},
        # the Fields stage on host arrays with the default job parameters
        # (3x3 seeds, step 0.5 px, RK2), seed list and finished arrays included
        {"name": "fields_stage_defaults", "kind": "stage", "terrain": "incised", "nx": 701, "ny": 1113, "density": 3,
         "jitter": 1.0, "rk": 2, "step": 0.5, "max_steps": 2000, "pixel": 1.0},
        # many tiles of uneven sizes in one batched launch per direction
        {"name": "batch_tiles_rk2", "kind": "batch", "terrain": "hills", "tiles": 24, "lo": 96, "hi": 512,
         "density": 2, "jitter": 1.0, "rk": 2, "step": 0.1, "max_steps": 2000, "pixel": 1.0},
        # the Trajectories stage on host arrays: 1000 recorded streamlines
        # each way, for the statistics and the plots
        {"name": "trajectories_stage", "kind": "traj", "terrain": "incised", "nx": 1024, "ny": 900, "seeds": 1000,
         "rk": 2, "step": 0.1, "max_steps": 2000, "pixel": 2.0},
        # conditioning a lidar DTM that already lies on the GPU
        {"name": "preprocess_f32", "kind": "preprocess", "terrain": "incised", "nx": 4096, "ny": 3001, "f64": False,
         "normalize": True, "pixel": 1.0},
        # the marginal density of log lengths, which sets the channel threshold
        {"name": "kde_univariate", "kind": "kde1", "n": 2000003, "bins": 2048, "points": 256,
         "kernel": "epanechnikov", "bandwidth": 10.0},
        # the joint density of two log quantities
        {"name": "kde_bivariate", "kind": "kde2", "n": 1000003, "bins": 1024, "points": 256, "kernel": "gaussian",
         "bandwidth": 5.0},
        # the scheduler's predictions for every seed of a grid
        {"name": "scheduler_predict", "kind": "predict", "terrain": "fan", "nx": 1500, "ny": 2048},
        # one training step of the scheduler's network
        {"name": "scheduler_train_step", "kind": "train", "terrain": "fan", "nx": 1024, "ny": 1024, "batch": 4096},
        # channels, segments and flanks of an area whose fields are on the GPU
        {"name": "mapping_incised1024", "kind": "mapping", "terrain": "incised", "nx": 1024, "ny": 1024,
         "step": 0.1, "max_steps": 10000, "pixel": 2.0},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["fields", "fields", "fields", "stage", "batch", "traj", "preprocess", "kde1", "kde2",
                       "predict", "train", "mapping"])
    terrain = rng.choice(["hills", "incised", "fan"])
    if kind == "fields":
        # at most 24 M trajectories a direction; long steps and 3x3 seeds are
        # the defaults of a job, the plain form has no jitter
        d = rng.choice([1, 2, 2, 3])
        hi = {1: 3000, 2: 2000, 3: 1300}[d] if terrain != "hills" else 600
        return {"kind": kind, "terrain": terrain, "nx": _log(rng, 64, hi), "ny": _log(rng, 64, hi), "density": d,
                "jitter": rng.choice([1.0, 1.0, 0.0, 0.7]), "rk": rng.choice([2, 4]),
                "step": rng.choice([0.1, 0.1, 0.5]), "max_steps": rng.choice([2000, 10000]),
                "pixel": rng.choice([1.0, 2.0])}
    if kind == "stage":
        return {"kind": kind, "terrain": terrain, "nx": _log(rng, 64, 1000), "ny": _log(rng, 64, 1000),
                "density": rng.choice([1, 2, 3]), "jitter": 1.0, "rk": rng.choice([2, 4]), "step": 0.5,
                "max_steps": 2000, "pixel": rng.choice([1.0, 2.0])}
    if kind == "batch":
        return {"kind": kind, "terrain": terrain, "tiles": rng.randint(2, 24), "lo": 64, "hi": _log(rng, 100, 512),
                "density": rng.choice([1, 2]), "jitter": 1.0, "rk": rng.choice([2, 4]), "step": 0.1,
                "max_steps": 2000, "pixel": 1.0}
    if kind == "traj":
        return {"kind": kind, "terrain": terrain, "nx": _log(rng, 64, 1024), "ny": _log(rng, 64, 1024),
                "seeds": rng.choice([100, 1000, 2000]), "rk": rng.choice([2, 4]), "step": rng.choice([0.1, 0.5]),
                "max_steps": 2000, "pixel": rng.choice([1.0, 2.0])}
    if kind == "preprocess":
        return {"kind": kind, "terrain": terrain, "nx": _log(rng, 100, 4000), "ny": _log(rng, 100, 3000),
                "f64": rng.random() < 0.5, "normalize": rng.random() < 0.8, "pixel": rng.choice([0.5, 1.0, 2.0])}
    if kind == "kde1":
        points = rng.choice([128, 256, 1024])
        return {"kind": kind, "n": _log(rng, 1000, 2000000), "bins": points * rng.choice([2, 8]), "points": points,
                "kernel": rng.choice(["epanechnikov", "gaussian", "triangle"]), "bandwidth": rng.choice([2.0, 10.0])}
    if kind == "kde2":
        return {"kind": kind, "n": _log(rng, 1000, 1000000), "bins": rng.choice([256, 512, 1024]),
                "points": rng.choice([64, 128, 256]), "kernel": rng.choice(["epanechnikov", "gaussian"]),
                "bandwidth": rng.choice([2.0, 5.0])}
    if kind == "predict":
        return {"kind": kind, "terrain": terrain, "nx": _log(rng, 64, 1500), "ny": _log(rng, 64, 2048)}
    if kind == "train":
        return {"kind": kind, "terrain": terrain, "nx": _log(rng, 128, 1024), "ny": _log(rng, 128, 1024),
                "batch": _log(rng, 100, 4096)}
    return {"kind": "mapping", "terrain": "incised", "nx": _log(rng, 128, 1024), "ny": _log(rng, 128, 1024),
            "step": 0.1, "max_steps": 10000, "pixel": 2.0}


# ---------------------------------------------------------------- terrain
def _gen(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(int(seed))
    return g


def _fbm(nx, ny, hurst, rms, g):
    """Isotropic fractional Brownian surface by spectral synthesis."""
    kx = torch.fft.fftfreq(nx, device="cuda", dtype=torch.float64)[:, None]
    ky = torch.fft.rfftfreq(ny, device="cuda", dtype=torch.float64)[None, :]
    k = torch.sqrt(kx * kx + ky * ky)
    k[0, 0] = 1.0
    amp = k ** (-(hurst + 1.0))
    amp[0, 0] = 0.0
    phase = torch.rand(amp.shape, generator=g, device="cuda", dtype=torch.float64) * (2.0 * math.pi)
    z = torch.fft.irfft2(torch.polar(amp, phase), s=(nx, ny))
    z -= z.mean()
    return z * (rms / z.std())


def _dtm(case, seed, nx=None, ny=None):
    """A DTM [nx, ny] float32 on the GPU."""
    nx, ny = nx or case["nx"], ny or case["ny"]
    g = _gen(seed)
    rng = np.random.default_rng(int(seed))
    x = torch.arange(nx, device="cuda", dtype=torch.float64)[:, None]
    y = torch.arange(ny, device="cuda", dtype=torch.float64)[None, :]
    if case["terrain"] == "hills":
        z = 0.05 * x + _fbm(nx, ny, 0.7, 0.5, g)
        for _ in range(max(1, round(12 * nx * ny / 512.0 ** 2))):
            a, s = rng.uniform(5.0, 40.0), rng.uniform(20.0, 80.0)
            cx, cy = rng.uniform(0, nx), rng.uniform(0, ny)
            z += a * torch.exp(-((x - cx) ** 2) / (2.0 * s * s)) * torch.exp(-((y - cy) ** 2) / (2.0 * s * s))
        return z.to(torch.float32)
    if case["terrain"] == "incised":
        z = _fbm(nx, ny, 0.75, 30.0, g)
        m = max(8, round(400 * nx * ny / 2048.0 ** 2))
        steps = max(64, min(nx, ny) // 8)
        px, py = rng.uniform(0, nx, m), rng.uniform(0, ny, m)
        ang = rng.uniform(0, 2 * np.pi, m)
        xs, ys = np.empty((m, steps)), np.empty((m, steps))
        for s in range(steps):
            ang += rng.normal(0.0, 0.3, m)
            px = np.clip(px + np.cos(ang), 0.0, nx - 1.0)
            py = np.clip(py + np.sin(ang), 0.0, ny - 1.0)
            xs[:, s], ys[:, s] = px, py
        depth = torch.from_numpy(np.repeat(rng.uniform(1.0, 8.0, m), steps)).cuda()
        ix = torch.from_numpy(np.round(xs).astype(np.int64).reshape(-1)).cuda()
        iy = torch.from_numpy(np.round(ys).astype(np.int64).reshape(-1)).cuda()
        cut = torch.zeros(nx * ny, device="cuda", dtype=torch.float64)
        for ox in (-1, 0, 1):
            for oy in (-1, 0, 1):
                at = (ix + ox).clamp(0, nx - 1) * ny + (iy + oy).clamp(0, ny - 1)
                cut.scatter_reduce_(0, at, depth * (1.0 if ox == 0 and oy == 0 else 0.5), "amax")
        return (z - cut.view(nx, ny)).to(torch.float32)
    z = _fbm(nx, ny, 0.8, 40.0, g)
    n = max(nx, ny)
    r = torch.sqrt((x - 0.5 * nx) ** 2 + y ** 2)
    theta = torch.atan2(y.expand(nx, ny), (x - 0.5 * nx).expand(nx, ny))
    w = torch.clamp(1.0 - r / (0.6 * n), 0.0, 1.0)
    z = (1.0 - w) * z + w * (-0.03 * r + 0.3 * torch.sin(24.0 * theta)) + 0.03 * (n * 0.6)
    pits = max(8, round(5000 * nx * ny / 8192.0 ** 2))
    qx = torch.from_numpy(rng.integers(2, nx - 2, size=pits)).cuda()
    qy = torch.from_numpy(rng.integers(2, ny - 2, size=pits)).cuda()
    d = torch.from_numpy(rng.uniform(0.05, 0.5, size=pits)).cuda()
    for ox in (-1, 0, 1):
        for oy in (-1, 0, 1):
            at, f = (qx + ox) * ny + qy + oy, 1.0 if ox == 0 and oy == 0 else 0.5
            low = torch.zeros(nx * ny, device="cuda", dtype=torch.float64)
            low.scatter_reduce_(0, at, f * d, "amax")
            z -= low.view(nx, ny)
    return z.to(torch.float32)


def _gradient(z, pixel):
    """np.gradient / pixel of a 2-D tensor, in its own type."""
    gx, gy = torch.empty_like(z), torch.empty_like(z)
    gx[1:-1] = (z[2:] - z[:-2]) / 2.0
    gx[0], gx[-1] = z[1] - z[0], z[-1] - z[-2]
    gy[:, 1:-1] = (z[:, 2:] - z[:, :-2]) / 2.0
    gy[:, 0], gy[:, -1] = z[:, 1] - z[:, 0], z[:, -1] - z[:, -2]
    return gx / pixel, gy / pixel


def _edge_pad(a):
    return torch.nn.functional.pad(a[None, None], (PAD, PAD, PAD, PAD), mode="replicate")[0, 0]


def _flow(z, pixel):
    """(uv [nxp, nyp, 2] float32, mask [nxp, nyp] bool) of a DTM, on the GPU."""
    gx, gy = _gradient(z, pixel)
    speed = torch.hypot(gx, gy)
    speed = torch.where(torch.isfinite(speed) & (speed != 0.0), speed, torch.ones_like(speed))
    uv = torch.stack((_edge_pad(-gx / speed), _edge_pad(-gy / speed)), dim=2).contiguous()
    mask = torch.ones(uv.shape[:2], dtype=torch.bool, device="cuda")
    mask[PAD:-PAD, PAD:-PAD] = False
    return uv, mask


def _info(case, nx, ny, density=None, jitter=None, n_traj=1000):
    d = default_parameters()
    d.trace.subpixel_seed_point_density = density or case.get("density", 1)
    d.trace.jitter_magnitude = case.get("jitter", 0.0) if jitter is None else jitter
    d.trace.integrator_step_factor = case["step"]
    d.trace.max_length = case["max_steps"] * case["step"]
    d.trace.n_trajectory_seed_points = n_traj
    info = Info(d.state, d.trace, case["pixel"])
    info.set_xy(nx, ny, PAD)
    return info


def _seeds(nx, ny, seed):
    """Every pixel once, shuffled, as (x, y) rows."""
    p = torch.randperm(nx * ny, generator=_gen(seed + 1), device="cuda")
    return torch.stack((p // ny, p % ny), dim=1).to(torch.float32).contiguous()


def _stats(info):
    """Statistics of a recorded trace, as the Trajectories stage leaves them."""
    n = np.full((4, 2), 200, np.uint16)
    return compute_stats(np.full((4, 2), 18.0, np.float32), n, info.pixel_size)


# ---------------------------------------------------------------- cases
def prepare(case, seed):
    kind = case["kind"]
    s = types.SimpleNamespace(case=case)
    if kind in ("fields", "mapping"):
        nx, ny = case["nx"], case["ny"]
        uv, mask = _flow(_dtm(case, seed), case["pixel"])
        s.nx, s.ny, s.uv, s.mask = nx, ny, uv, mask.view(torch.uint8)
        s.seeds = _seeds(nx, ny, seed)
        s.info = _info(case, nx, ny)
        s.info.n_seed_points = nx * ny
        s.prm = [kernel_params(s.info, "INTEGRATE_FIELDS", sign) for sign in (1.0, -1.0)]
        s.nxy = uv.shape[0] * uv.shape[1]
        s.acc = torch.zeros((2, 2, s.nxy), dtype=torch.uint64, device="cuda")
        s.work = kernels.workspace("cuda")
        if kind == "mapping":
            kernels.integrate_fields_pair(s.prm[0], s.prm[1], s.seeds, s.mask, s.uv, s.acc[:, 0], s.acc[:, 1],
                                          s.work, integrator=2)
            shape = tuple(uv.shape[:2])
            slc = math.sqrt(2.0) * s.acc[:, 0].view(torch.int64).to(torch.float64) ** (2.0 / 3.0)
            slt = torch.sqrt(s.acc[:, 1].view(torch.int64).to(torch.float32) * 0.1)
            fields = [f.view(2, *shape).permute(1, 2, 0).contiguous() for f in (slt, slc)]
            inside = fields[0][:, :, 0][~mask]
            top = torch.sort(inside).values[int(0.94 * inside.numel())]
            s.info.set_thresholds(segmentation_threshold=np.uint32(10), channel_threshold=np.float32(top.item()))
            s.data = types.SimpleNamespace(mask_array=mask, uv_array=uv, slt_array=fields[0], slc_array=fields[1],
                                           mapping_array=torch.zeros(shape, dtype=torch.uint32, device="cuda"))
            del s.acc
    elif kind in ("stage", "traj"):
        uv, mask = _flow(_dtm(case, seed), case["pixel"])
        s.info = _info(case, case["nx"], case["ny"], n_traj=case.get("seeds", 1000))
        s.data = Data(info=s.info, mask_array=mask.cpu().numpy(), uv_array=uv.cpu().numpy(),
                      mapping_array=np.zeros(tuple(mask.shape), np.uint32), traj_stats_df=_stats(s.info))
    elif kind == "batch":
        rng = np.random.default_rng(case["tiles"] * 10007 + case["hi"])  # the sizes belong to the case
        tiles = []
        for k in range(case["tiles"]):
            nx, ny = (int(round(math.exp(rng.uniform(math.log(case["lo"]), math.log(case["hi"]))))) for _ in "xy")
            uv, mask = _flow(_dtm(case, seed + 7 * k, nx, ny), case["pixel"])
            info = _info(case, nx, ny)
            host = mask.cpu().numpy()
            rows, info.n_seed_points, info.n_padded_seed_points = create_seeds(host, PAD, info.n_work_items,
                                                                               rng_seed=int(seed) % 1000)
            tiles.append(Tile(uv.cpu().numpy(), host, info, rows))
        s.batch = TileBatch(tiles, integrator=case["rk"])
    elif kind == "preprocess":
        z = _dtm(case, seed)
        g = _gen(seed + 1)
        at = torch.rand((3, 2), generator=g, device="cuda")  # three patches without data
        for px, py in ((at * 0.9).cpu() * torch.tensor([case["nx"], case["ny"]])).to(torch.int64).tolist():
            z[px:px + 9, py:py + 13] = float("nan")
        s.roi = z.to(torch.float64) if case["f64"] else z
    elif kind == "kde1":
        rng = np.random.default_rng(int(seed))
        v = np.log(rng.lognormal(3.0, 0.8, size=case["n"])).astype(np.float32)
        s.d = Univariate_distribution(logx_array=v, logy_array=v, n_hist_bins=case["bins"],
                                      n_pdf_points=case["points"], cl_device=0)
    elif kind == "kde2":
        rng = np.random.default_rng(int(seed))
        v = np.log(rng.lognormal(2.0, 0.6, size=case["n"])).astype(np.float32)
        w = (0.5 * v + np.log(rng.lognormal(1.0, 0.4, size=case["n"]))).astype(np.float32)
        s.d = Bivariate_distribution(logx_array=v, logy_array=w, n_hist_bins=case["bins"],
                                     n_pdf_points=case["points"], cl_device=0)
    else:
        nx, ny = case["nx"], case["ny"]
        s.uv, _ = _flow(_dtm(case, seed), 1.0)
        s.seeds = _seeds(nx, ny, seed)
        s.model = LengthModel("cuda", init_params(int(seed) % 1000))
        s.n, s.nx, s.ny = nx * ny, nx, ny
        if kind == "train":
            n = case["batch"]
            g = _gen(seed + 2)
            s.index = torch.randint(0, s.n, (n,), generator=g, device="cuda").to(torch.int32)
            s.target = 4.0 + torch.randn((n, 2), generator=g, device="cuda")
    return s


def run(s):
    case = s.case
    kind = case["kind"]
    if kind == "fields":
        order = spatial_order(s.seeds, s.nx * s.ny, s.nx, s.ny)
        s.acc.zero_()
        kernels.integrate_fields_pair(s.prm[0], s.prm[1], s.seeds, s.mask, s.uv, s.acc[:, 0], s.acc[:, 1], s.work,
                                      integrator=case["rk"], order=order)
        return s.acc.view(torch.int64)
    if kind == "stage":
        Fields(0, 0, info=s.info, data=s.data, integrator=case["rk"]).integrate()
        d = s.data
        return {"slc": d.slc_array, "slt": d.slt_array, "sla": d.sla_array, "seeds": d.seed_point_array}
    if kind == "batch":
        s.batch.trace()
        return s.batch.acc.view(torch.int64)
    if kind == "traj":
        Trajectories(0, 0, info=s.info, data=s.data, integrator=case["rk"]).integrate()
        d = s.data
        steps = []
        for a in d.streamline_arrays_list:  # the streamlines of a direction end to end, then nothing
            flat = np.zeros((len(a) * int(s.info.max_n_steps), 2), np.int8)
            np.concatenate(list(a), out=flat[:sum(len(t) for t in a)])
            steps.append(flat)
        return {"steps": steps, "n": d.traj_nsteps_array, "length": d.traj_length_array}
    if kind == "preprocess":
        r = conditioned_gradient_vector_field(s.roi, case["pixel"], PAD, do_normalize_speed=case["normalize"],
                                              download=False)
        return {"uv": r.uv_array, "slope": r.slope_array, "uv_mask": r.uv_mask_array, "mask": r.mask_array,
                "blockages": r.blockages_array, "blocked": r.blocked_neighbors_array, "loops": r.loop_cells,
                "n_loops": r.n_loop_cells, "gradx": r.roi_gradx_array, "grady": r.roi_grady_array}
    if kind in ("kde1", "kde2"):
        s.d.compute_kde_opencl(kernel=case["kernel"], bandwidth=case["bandwidth"])
        return {"pdf": s.d.pdf, "histogram": s.d.histogram, "cdf": s.d.cdf}
    if kind == "predict":
        visit = spatial_order(s.seeds, s.n, s.nx, s.ny)
        return s.model.predict(s.uv, s.nx + 2 * PAD, s.ny + 2 * PAD, PAD, s.seeds, s.n, visit=visit)
    if kind == "train":
        m, n = s.model, case["batch"]
        x1 = m.gather(s.uv, s.nx + 2 * PAD, s.ny + 2 * PAD, PAD, s.seeds, s.index, n)
        loss = m.loss_and_grad(x1, s.target, n)
        m.adam(1e-3)
        return {"loss": loss, "grad": m.grad, "weights": m.master}
    s.data.mapping_array.zero_()
    dm = DeviceMapping(s.info, s.data, torch.device("cuda", 0))
    dm.map_channels_segments()
    return {"mapping": dm.mapping, "label": dm.label, "count": dm.count, "link": dm.link,
            "channel_label": dm.channel_label}


# ---------------------------------------------------------------- work
# mean RK steps of a trajectory on each terrain at step 0.1 px (shorter steps
# per trajectory where the step is longer), and the arithmetic of one step:
# per stage a bilinear sample, two normalisations and the products, and the
# step's own sums and length
_MEAN_STEPS = {"hills": 700.0, "incised": 80.0, "fan": 110.0}


def _step_flops(rk, jitter):
    return rk * (30 + 6 + (10 if jitter else 0) + 4) + 30


def _traj_steps(case):
    mean = _MEAN_STEPS[case["terrain"]] * 0.1 / case["step"]
    return min(mean, 1.0 * case["max_steps"], 0.5 * case.get("nx", case.get("hi", 256)) / case["step"])


def work(case):
    kind = case["kind"]
    if kind in ("fields", "stage", "batch"):
        if kind == "batch":  # the mean of a log-uniform edge, squared
            lo, hi = case["lo"], case["hi"]
            mean = (hi - lo) / math.log(hi / lo) if hi > lo else hi
            px = case["tiles"] * mean * mean
        else:
            px = case["nx"] * case["ny"]
        traj = 2 * px * case["density"] ** 2
        out = 2 * 16 if kind != "stage" else 2 * 16 + 8  # sums, or the finished arrays and the seed rows
        return {"bytes": px * (8 + 1 + 8 + out),
                "flops": traj * _traj_steps(case) * _step_flops(case["rk"], case["jitter"])}
    if kind == "traj":
        steps = 2 * case["seeds"] * _traj_steps(case)
        return {"bytes": case["nx"] * case["ny"] * 9 + steps * 2 + case["seeds"] * 12,
                "flops": steps * _step_flops(case["rk"], 0.0)}
    px = case.get("nx", 0) * case.get("ny", 0)
    if kind == "preprocess":
        return {"bytes": px * ((8 if case["f64"] else 4) + 8 + 4 + 1 + 1 + 3 + 8), "flops": px * 120}
    if kind == "kde1":
        reach = min(case["points"], 16)
        return {"bytes": case["n"] * 4 + case["bins"] * 12 + case["points"] * 12,
                "flops": case["n"] * 3 + case["bins"] * reach * 4}
    if kind == "kde2":
        b2, p2 = case["bins"] ** 2, case["points"] ** 2
        return {"bytes": case["n"] * 8 + b2 * 16 + p2 * 12, "flops": case["n"] * 6 + b2 * 20 * 4 + b2 * 20 * 4}
    macs = 16 * 32 * 32 + 4 * 128 * 64 + 256 * 2
    if kind == "predict":
        return {"bytes": px * (8 + 8 + 8), "flops": 2.0 * px * macs}
    if kind == "train":
        n = case["batch"]
        return {"bytes": n * (256 * 8 + 8 + 12) + 9762 * 7 * 4, "flops": 2.0 * n * macs * 3}
    return {"bytes": px * (1 + 8 + 4 + 8 + 5 * 4), "flops": px * 400.0}


# ---------------------------------------------------------------- 64 bits
def _weight(kernel, x, w):
    if kernel == "triangle":
        return np.maximum(1.0 - np.abs(x / w), 0.0)
    if kernel == "epanechnikov":
        return np.maximum(1.0 - (x / w) ** 2, 0.0)
    sd = w * float(np.float32(0.4))
    return np.exp(-0.5 * (x / sd) ** 2)


def _f32(*v):
    return [float(np.float32(x)) for x in v]


def _exact_kde1(s):
    """Histogram in float32 bins (its definition), the half-kernel sums in 64 bits."""
    d, case = s.d, s.case
    nb, n_pdf = case["bins"], case["points"]
    x = d.logx_data.reshape(-1)
    lo, span = np.float32(d.logx_min), np.float32(d.logx_range)
    bins = np.minimum(((x - lo) / span * np.float32(nb)).astype(np.int64), nb - 1)
    hist = np.bincount(bins, minlength=nb).astype(np.float64)
    bandwidth = case["bandwidth"] / (2.0 if case["kernel"] == "gaussian" else 1.0)
    width = 1.06 * np.std(d.logx_data) * np.power(d.n_data, -0.2) * bandwidth
    part = int(np.floor(width / d.pdf_dx)) // 2
    w, pdf_dx, bin_dx = _f32(width, d.pdf_dx, d.bin_dx)
    per = nb // n_pdf
    acc, norm = np.zeros(n_pdf), np.zeros(n_pdf)
    at = np.arange(n_pdf)
    for k in range(part + 1):
        for h in range(per):
            kv = _weight(case["kernel"], k * pdf_dx - pdf_dx / 2.0 + bin_dx * (h + 0.5), w)
            right = at + k < n_pdf
            acc[right] += kv * hist[(at[right] + k) * per + h]
            norm[right] += kv
            left = (at - k + 1 > 0) & (k != 0)
            acc[left] += kv * hist[(at[left] - k + 1) * per - h - 1]
            norm[left] += kv
    pdf = acc / norm
    pdf /= pdf.sum() * float(d.bin_dx)
    cdf = np.cumsum(pdf) * float(d.bin_dx)
    return {"pdf": pdf.reshape(-1, 1), "histogram": (hist / (hist.sum() * float(d.bin_dx))).reshape(-1, 1), "cdf": cdf}


def _exact_kde2(s):
    d, case = s.d, s.case
    nb, n_pdf = case["bins"], case["points"]
    nbm = np.float32(nb - 1)
    idx = []
    for v, lo, span in ((d.logxy_data[:, 0], d.logx_min, d.logx_range), (d.logxy_data[:, 1], d.logy_min, d.logy_range)):
        idx.append(np.minimum(((v - np.float32(lo)) / np.float32(span) * nbm).astype(np.int64), nb - 1))
    hist = np.bincount(idx[0] * nb + idx[1], minlength=nb * nb).reshape(nb, nb).astype(np.float64)
    parts = []
    for c, dx in ((0, d.bin_dx), (1, d.bin_dy)):
        width = 1.06 * np.std(d.logxy_data[:, c]) * np.power(d.n_data, -0.2) * case["bandwidth"]
        parts.append(int(np.floor(width / dx)) // 2)
    acc, norm = np.zeros((nb, nb)), np.ones(nb)
    for k in range(parts[1] + 1):  # along y, one row of x at a time
        kv = _weight(case["kernel"], float(k), parts[1] + 0.5)
        acc[:, :nb - k] += kv * hist[:, k:]
        norm[:nb - k] += kv
        if k:
            acc[:, k - 1:] += kv * hist[:, :nb - k + 1]
            norm[k - 1:] += kv
    partial = acc / norm
    per = nb // n_pdf
    cols = partial.reshape(nb, n_pdf, per).sum(2)  # each pdf column's bins
    acc, norm = np.zeros((n_pdf, n_pdf)), np.ones((n_pdf, n_pdf))
    rows = np.arange(n_pdf)
    for k in range(parts[0] + 1):
        for h in range(per):
            kv = _weight(case["kernel"], h + float(k) * per, parts[0] + 0.5)
            ok = rows + k < n_pdf
            acc[ok] += kv * cols[(rows[ok] + k) * per + h]
            norm[ok] += kv * per
            ok = (rows - k >= 0) & (k != 0)
            acc[ok] += kv * cols[(rows[ok] - k) * per + per - 1 - h]
            norm[ok] += kv * per
    pdf = acc / norm
    dxy = float(d.bin_dx) * float(d.bin_dy)
    pdf /= pdf.sum() * dxy
    return {"pdf": pdf, "histogram": hist / (hist.sum() * dxy), "cdf": np.cumsum(pdf) * float(d.bin_dx)}


def _patches(s, index):
    """conv1 input rows [n, 16, 32] of the seeds, bfloat16-rounded, in 64 bits."""
    at = s.seeds[index].to(torch.int64) + PAD
    t, m = torch.arange(16, device="cuda")[:, None], torch.arange(16, device="cuda")[None, :]
    x = (at[:, 0, None, None] - 8 + 4 * (t // 4) + m // 4).clamp(0, s.nx + 2 * PAD - 1)
    y = (at[:, 1, None, None] - 8 + 4 * (t % 4) + m % 4).clamp(0, s.ny + 2 * PAD - 1)
    return bf16_round(s.uv[x, y]).to(torch.float64).reshape(-1, 16, 32)


def _network(s, x1, p):
    """Predictions in 64 bits with the activations rounded to bfloat16, as the network is defined."""
    def rounded(a):  # the gradient passes the rounding by
        return a + (a.to(torch.float32).to(torch.bfloat16).to(torch.float64) - a).detach()
    n = x1.shape[0]
    a1 = rounded(torch.relu(x1 @ p["w1"] + p["b1"]))  # [n, 16, 32]
    x2 = a1.view(n, 2, 2, 2, 2, 32).permute(0, 1, 3, 2, 4, 5).reshape(n, 4, 128)
    a2 = rounded(torch.relu(x2 @ p["w2"] + p["b2"]))
    return a2.reshape(n, 256) @ p["w3"] + p["b3"]


def _exact_network(s):
    p = {k: v.to(torch.float64) for k, v in s.model.W.items()}
    if s.case["kind"] == "predict":
        out = torch.empty((s.n, 2), dtype=torch.float64, device="cuda")
        for a in range(0, s.n, 1 << 17):
            i = torch.arange(a, min(s.n, a + (1 << 17)), device="cuda")
            out[i] = _network(s, _patches(s, i), p)
        return out
    for v in p.values():
        v.requires_grad_(True)
    y = _network(s, _patches(s, s.index.to(torch.int64)), p)
    loss = ((y - s.target.to(torch.float64)) ** 2).mean()
    loss.backward()
    return {"loss": loss.detach().reshape(1), "grad": torch.cat([v.grad.reshape(-1) for v in p.values()]),
            "weights": None}


def exact(case, seed):
    kind = case["kind"]
    if kind in ("fields", "batch", "traj", "stage", "mapping"):
        # whole numbers, and floats that follow from quantised steps and
        # running sums whose 32-bit rounding is their definition
        return None
    s = prepare(case, seed)
    if kind == "preprocess":
        gx, gy = _gradient(s.roi.to(torch.float32).to(torch.float64), float(np.float32(case["pixel"])))
        speed = torch.hypot(gx, gy)
        speed = torch.where(torch.isfinite(speed) & (speed != 0.0), speed, torch.ones_like(speed))
        return {"slope": _edge_pad(torch.rad2deg(torch.atan(speed))), "gradx": gx, "grady": gy}
    if kind == "kde1":
        return _exact_kde1(s)
    if kind == "kde2":
        return _exact_kde2(s)
    return _exact_network(s)
