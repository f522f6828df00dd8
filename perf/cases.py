"""Performance cases: the calls a localisation program makes, over the sizes it makes them at.

listed() names the cases, draw() gives more of the same ranges, prepare() makes
what a program has in hand before the call, run() is one pass through the public
entry points (the C ABI's device forms, the Python host forms), work() the bytes
and operations a pass cannot do without, exact() the outputs in 64 bits.

The maps are the framework's seeded synthetic ones (a room at 0.064 m in the
reference's chunks, the 100 x 100 x 10 m building at 0.05 m, a warehouse and a
tunnel at 0.1 m); the seed moves the robot, redraws the scan's noise and the
particles.  One context (one stream) and one device map per layout serve a
process, as they serve a running filter.
"""
from __future__ import annotations

import ctypes as C
import math

import numpy as np
import torch

from tsdf_localization_gb300 import (Context, DeviceMap, FilterBatch, MotionModel, ResidualSystematicResampler,
                                     SystematicResampler, TSDFEvaluator, build_map_codes, pack_cloud, synth)
from tsdf_localization_gb300 import _native as N

MODEL = (0.9, 0.1, 0.0, 100.0)   # a_hit, a_range, a_max, max_range
SIGMA = 0.1                      # metres, of the likelihood
HEIGHT = 0.0                     # metres, of the scanner above the base frame

# name -> (world kind, world seed, voxel mm, chunk edge, largest scan rings x columns, reduction cell)
MAPS = {
    "room": (synth.ROOM, 1, 64, 64, 16, 1024, 0.064),
    "building": (synth.BUILDING, 2, 50, 8, 64, 2048, 0.05),
    "warehouse": (synth.WAREHOUSE, 23, 100, 16, 64, 2048, 0.1),
    "tunnel": (synth.TUNNEL, 24, 100, 16, 64, 2048, 0.1),
}


def listed() -> list[dict]:
    return [
        # a small robot: one update and resampling of 1,000 particles; launches and latency are all there is
        {"name": "room 1k x 2k", "kind": "step", "map": "room", "layout": "compact", "cloud": "tracking", "P": 1000,
         "N": 2048, "resampler": "systematic"},
        # the headline: tracking with 100,000 particles and a dense scan in the building
        {"name": "building 100k x 8k", "kind": "step", "map": "building", "layout": "compact", "cloud": "tracking",
         "P": 100_000, "N": 8192, "resampler": "systematic"},
        # global localisation: a million particles over the whole lower storey, any yaw
        {"name": "global 1M x 2k", "kind": "step", "map": "building", "layout": "compact", "cloud": "global",
         "P": 1_000_000, "N": 2048, "resampler": "systematic"},
        # a mid-size filter of odd size on the plain brick table (the C++ plug-in's map), mcl_3d's default resampler
        {"name": "warehouse 23k x 5k brick", "kind": "step", "map": "warehouse", "layout": "brick",
         "cloud": "tracking", "P": 23_457, "N": 5003, "resampler": "residual_systematic"},
        # the drop-in call: host particles and points in, weights and resampled particles out
        {"name": "host 5k x 4k", "kind": "host", "map": "room", "layout": "brick", "P": 5000, "N": 4000,
         "resampler": "systematic"},
        # the drop-in call on the raw point cloud: reduction and update in one
        {"name": "cloud 2k x 16x1024", "kind": "cloud", "map": "room", "layout": "compact", "P": 2000, "rings": 16,
         "columns": 1024},
        # one whole filter step on the device: motion, update, best particle, resampling
        {"name": "filter 20k x 4k", "kind": "filter", "map": "tunnel", "layout": "compact", "P": 20_000, "N": 4099,
         "resampler": "systematic"},
        # scan pre-processing of a 64-ring scanner's cloud
        {"name": "scan 64x2048", "kind": "scan", "map": "building", "rings": 64, "columns": 2048},
        # odometry motion update
        {"name": "motion 100k", "kind": "motion", "P": 100_000, "motion": "odom"},
        # mcl_3d's default resampler alone
        {"name": "residual systematic 100k", "kind": "resample", "P": 100_000, "resampler": "residual_systematic"},
        # a fleet of small robots in one process, replayed from a captured graph
        {"name": "batch 24 x 1k-10k", "kind": "batch", "filters": 24, "Pmin": 1000, "Pmax": 10_000, "Nmin": 1000,
         "Nmax": 8000},
        # global localisation with every particle on its own 256 of the points
        {"name": "subsampled 300k x 256", "kind": "subsampled", "map": "building", "layout": "compact", "P": 300_000,
         "N": 2048, "K": 256},
    ]


def _log_int(rng, lo: int, hi: int) -> int:
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng) -> dict:
    kind = rng.choice(["step", "step", "step", "host", "cloud", "filter", "scan", "motion", "resample", "resample",
                       "batch", "subsampled"])
    if kind == "step":
        cloud = rng.choice(["tracking", "tracking", "global"])
        name = rng.choice(["building", "warehouse"] if cloud == "global" else list(MAPS))
        P = _log_int(rng, 20_000, 1_000_000) if cloud == "global" else _log_int(rng, 300, 200_000)
        most = 8000 if name == "room" else 16_000
        n = min(_log_int(rng, 200, most), 2_000_000_000 // P)
        return {"kind": kind, "map": name, "layout": rng.choice(["compact", "compact", "brick"]), "cloud": cloud,
                "P": P, "N": n, "resampler": rng.choice(["systematic", "residual_systematic"])}
    if kind == "host":
        return {"kind": kind, "map": rng.choice(["room", "warehouse", "tunnel"]),
                "layout": rng.choice(["compact", "brick"]), "P": _log_int(rng, 300, 50_000),
                "N": _log_int(rng, 300, 8000), "resampler": rng.choice(["systematic", "residual_systematic"])}
    if kind == "cloud":
        return {"kind": kind, "map": rng.choice(["room", "tunnel"]), "layout": rng.choice(["compact", "brick"]),
                "P": _log_int(rng, 300, 20_000), "rings": rng.choice([16, 32]),
                "columns": _log_int(rng, 400, 2048)}
    if kind == "filter":
        return {"kind": kind, "map": rng.choice(["room", "warehouse", "tunnel"]),
                "layout": rng.choice(["compact", "compact", "brick"]), "P": _log_int(rng, 500, 100_000),
                "N": _log_int(rng, 300, 8000), "resampler": rng.choice(["systematic", "residual_systematic"])}
    if kind == "scan":
        return {"kind": kind, "map": rng.choice(["room", "warehouse", "tunnel"]),
                "rings": rng.choice([16, 32, 64]), "columns": _log_int(rng, 400, 4096)}
    if kind == "motion":
        return {"kind": kind, "P": _log_int(rng, 500, 1_000_000), "motion": rng.choice(["odom", "scale", "delta"])}
    if kind == "resample":
        return {"kind": kind, "P": _log_int(rng, 500, 1_000_000),
                "resampler": rng.choice(["systematic", "residual_systematic", "residual_systematic", "wheel",
                                         "residual", "metropolis", "rejection"])}
    if kind == "batch":
        lo = _log_int(rng, 300, 5000)
        return {"kind": kind, "filters": rng.randint(6, 32), "Pmin": lo, "Pmax": lo * rng.randint(2, 8),
                "Nmin": 500, "Nmax": _log_int(rng, 1000, 8000)}
    n = _log_int(rng, 500, 8000)
    return {"kind": kind, "map": rng.choice(["building", "warehouse"]), "layout": rng.choice(["compact", "brick"]),
            "P": _log_int(rng, 10_000, 1_000_000), "N": n, "K": min(n, rng.randint(100, 400))}


# ---------------------------------------------------------------- what a program keeps

_kept: dict = {}


def _keep(key, make):
    if key not in _kept:
        _kept[key] = make()
    return _kept[key]


def _ctx() -> Context:
    return _keep("ctx", lambda: Context(0))


def _world(name: str) -> synth.World:
    kind, seed = MAPS[name][:2]
    return _keep(("world", name), lambda: synth.World(kind, seed))


def _map_arrays(name: str):
    """(coef, brick table, slot codes) of a map."""
    def make():
        _, _, voxel_mm, edge = MAPS[name][:4]
        pos, raw = _world(name).tsdf_chunks(voxel_mm, edge)
        return build_map_codes(pos, raw, edge, voxel_mm, SIGMA, want_free=False)[:3]
    return _keep(("map", name), make)


def _device_map(name: str, layout: str) -> DeviceMap:
    def make():
        coef, occ, codes = _map_arrays(name)
        return DeviceMap(_ctx(), coef, occ, codes=codes, sigma=SIGMA, dense=layout == "compact")
    return _keep(("device", name, layout), make)


# ---------------------------------------------------------------- inputs

def _pose(name: str, seed: int) -> np.ndarray:
    """The robot's true pose: the world's, moved by up to 0.2 m and turned."""
    rng = np.random.default_rng([seed, 1])
    p = _world(name).pose.copy()
    p[:2] += rng.uniform(-0.2, 0.2, 2).astype(np.float32)
    p[5] = np.float32(rng.uniform(-np.pi, np.pi))
    return p


def _cloud(name: str, seed: int, rings: int, columns: int):
    """The scanner's raw cloud at the robot's pose: (xyz, ring)."""
    return _world(name).scan(_pose(name, seed), rings, columns, dropout=0.01, seed=seed * 7 + 1)


def _points(name: str, seed: int, n: int) -> np.ndarray:
    rings, columns, cell = MAPS[name][4:]
    return synth.subsample(synth.reduce_scan(*_cloud(name, seed, rings, columns), cell), n, seed * 7 + 2)


def _particles(name: str, cloud: str, seed: int, n: int) -> np.ndarray:
    p = _pose(name, seed)
    if cloud == "global":
        z = float(p[2])
        return _world(name).particles_free_space(n, 0.3, z - 0.3, z + 0.3, math.radians(3.0), seed * 7 + 3)
    return synth.particles_gaussian(p, 0.3, math.radians(5.0), n, seed * 7 + 3)


def _u0(resampler: str, seed: int, n: int) -> float:
    """The resampler's draw: [0, 1/n) for the systematic one, [0, 1) else."""
    u = np.random.default_rng([seed, 2]).random()
    return float(np.float32(u / n if resampler == "systematic" else u))


def _weighted(seed: int, n: int) -> np.ndarray:
    """Particles after an update: poses and normalised, uneven weights."""
    rng = np.random.default_rng([seed, 3])
    p = np.empty((n, 7), np.float32)
    p[:, :3] = rng.normal(0, 0.3, (n, 3)) + (10, 12, 1)
    p[:, 3:6] = rng.normal(0, math.radians(5.0), (n, 3)) + (0, 0, 0.7)
    w = 0.02 + rng.gamma(0.8, size=n)
    p[:, 6] = w / w.sum()
    return p


def _motion_inputs(case: dict):
    """(inputs, time difference) of the motion-model overloads."""
    return {"odom": ([0.8, 0.2], 0.1), "scale": ([0.5, 0.2], 0.1),
            "delta": ([0.04, 0.01, 0.0, 0.002, -0.001, 0.02, 0.005, 0.002], 0.0)}[case.get("motion", "scale")]


def _points_drawn(case: dict, seed: int) -> list[tuple[str, int, int]]:
    """A batch's filters: (map, particles, points)."""
    rng = np.random.default_rng([seed, 4])
    out = []
    for i in range(case["filters"]):
        P = int(round(math.exp(rng.uniform(math.log(case["Pmin"]), math.log(case["Pmax"])))))
        out.append((("room", "warehouse", "tunnel")[i % 3], P, int(rng.integers(case["Nmin"], case["Nmax"] + 1))))
    return out


def _batch_specs(case: dict, seed: int):
    """The sizes are the fleet's (they belong to the case); the seed redraws clouds and scans."""
    scans = {}
    for i, (name, P, n) in enumerate(_points_drawn(case, case["filters"])):
        if name not in scans:
            scans[name] = _points(name, seed, 1 << 30)
        pts = synth.subsample(scans[name], n, seed * 100 + i)
        yield name, synth.particles_gaussian(_pose(name, seed), 0.3, math.radians(5.0), P, seed * 100 + i), pts


def _cuda(a: np.ndarray) -> torch.Tensor:
    return torch.from_numpy(a).cuda()


def prepare(case: dict, seed: int) -> dict:
    kind, ctx = case["kind"], _ctx()
    s = dict(case, ctx=ctx, seed=seed, model=N.Model(*MODEL), tf=synth.sensor_tf(HEIGHT))
    if kind == "scan":
        xyz, ring = _cloud(case["map"], seed, case["rings"], case["columns"])
        s["records"] = xyz.shape[0]
        s["d_cloud"] = _cuda(pack_cloud(xyz, ring))
        s["d_out"] = torch.zeros((case["rings"] * case["columns"], 3), device="cuda")
        s["d_count"] = torch.zeros(1, dtype=torch.int32, device="cuda")
        torch.cuda.synchronize()
        return s
    if kind == "batch":
        specs = list(_batch_specs(case, seed))
        rng = np.random.default_rng([seed, 5])
        total = sum(p.shape[0] for _, p, _ in specs)
        s["d_particles"] = _cuda(np.concatenate([p for _, p, _ in specs]))
        s["d_points"] = _cuda(np.concatenate([q for _, _, q in specs]))
        s["d_pose"] = torch.zeros((len(specs), 6), device="cuda")
        s["d_u0"] = _cuda(np.array([rng.random() / p.shape[0] for _, p, _ in specs], np.float32))
        s["d_out"] = torch.zeros((2 * total + 16 * len(specs), 7), device="cuda")
        s["d_count"] = torch.zeros(len(specs), dtype=torch.int32, device="cuda")
        filters, p0, q0, o0 = [], 0, 0, 0
        for i, (name, p, q) in enumerate(specs):
            P, n = p.shape[0], q.shape[0]
            filters.append({"map": _device_map(name, "compact"), "P": P, "N": n, "tf": s["tf"], "model": MODEL,
                            "particles": s["d_particles"].data_ptr() + 28 * p0,
                            "points": s["d_points"].data_ptr() + 12 * q0, "pose_out": s["d_pose"].data_ptr() + 24 * i,
                            "u0": s["d_u0"].data_ptr() + 4 * i, "resampled": s["d_out"].data_ptr() + 28 * o0,
                            "cap": 2 * P + 16, "count": s["d_count"].data_ptr() + 4 * i})
            p0, q0, o0 = p0 + P, q0 + n, o0 + 2 * P + 16
        torch.cuda.synchronize()
        s["batch"] = FilterBatch(ctx, filters)
        s["batch"].capture()
        return s

    P = case["P"]
    cap = 2 * P + 16
    if kind in ("resample", "motion"):
        s["d_particles"] = _cuda(_weighted(seed, P))
    if kind in ("step", "host", "cloud", "filter", "subsampled"):
        s["dmap"] = _device_map(case["map"], case["layout"])
        cloud = "global" if kind == "subsampled" else case.get("cloud", "tracking")
        particles = _particles(case["map"], cloud, seed, P)
        if kind in ("host", "cloud"):
            s["particles"] = particles
            s["evaluator"] = TSDFEvaluator(s["dmap"], False, *MODEL)
        else:
            s["d_particles"] = _cuda(particles)
        if kind == "cloud":
            xyz, ring = _cloud(case["map"], seed, case["rings"], case["columns"])
            s["records"], s["cloud"] = xyz.shape[0], pack_cloud(xyz, ring)
        else:
            pts = _points(case["map"], seed, case["N"])
            s["N"] = pts.shape[0]
            s["points" if kind == "host" else "d_points"] = pts if kind == "host" else _cuda(pts)
    if "resampler" in case:
        s["u0"] = _u0(case["resampler"], seed, P)
        if kind == "host":
            make = SystematicResampler if case["resampler"] == "systematic" else ResidualSystematicResampler
            s["host_resampler"] = make(ctx, 0)
            s["next"] = np.zeros((cap, 7), np.float32)   # the filter's other particle buffer
        else:
            s["d_out"] = torch.zeros((cap, 7), device="cuda")
            s["d_count"] = torch.zeros(1, dtype=torch.int32, device="cuda")
    if kind in ("step", "filter", "subsampled"):
        s["d_pose"] = torch.zeros(6, device="cuda")
        ctx.reserve(cap if kind == "filter" else P, s["N"])
    if kind in ("motion", "filter"):
        inputs, dt = _motion_inputs(case)
        s["motion"] = MotionModel(ctx).distributions(case.get("motion", "scale"), inputs, dt)
        s["d_best"] = torch.zeros(1, dtype=torch.int32, device="cuda")
    torch.cuda.synchronize()
    return s


# ---------------------------------------------------------------- one pass

def _p(t):
    return C.c_void_p(t.data_ptr())


def _evaluate(s: dict) -> None:
    N.check(N.lib().tsdfl_evaluate_device(s["ctx"].handle, s["dmap"].handle, C.byref(s["model"]),
                                          _p(s["d_particles"]), s["P"], _p(s["d_points"]), s["N"],
                                          s["tf"].ctypes.data_as(C.c_void_p), 0, _p(s["d_pose"])))


def _resample(s: dict) -> None:
    lib, h, src, P, out = N.lib(), s["ctx"].handle, _p(s["d_particles"]), s["P"], _p(s["d_out"])
    cap, cnt, which = s["d_out"].shape[0], _p(s["d_count"]), s["resampler"]
    if which == "systematic":
        N.check(lib.tsdfl_resample_systematic_device(h, src, P, s["u0"], out, cap, cnt))
    elif which == "residual_systematic":
        N.check(lib.tsdfl_resample_residual_systematic_device(h, src, P, s["u0"], out, cap, cnt))
    elif which == "wheel":
        N.check(lib.tsdfl_resample_wheel_device(h, src, P, None, s["seed"], out))
    elif which == "residual":
        N.check(lib.tsdfl_resample_residual_device(h, src, P, None, 0, s["seed"], out))
    elif which == "metropolis":
        N.check(lib.tsdfl_resample_metropolis_device(h, src, P, 50, None, None, s["seed"], out))
    else:
        N.check(lib.tsdfl_resample_rejection_device(h, src, P, s["seed"], out))


def _move(s: dict) -> None:
    N.check(N.lib().tsdfl_motion_update_device(s["ctx"].handle, _p(s["d_particles"]), s["P"], C.byref(s["motion"]),
                                               s["seed"], 0, None))


def run(s: dict) -> dict:
    kind = s["kind"]
    if kind == "step":
        _evaluate(s)
        _resample(s)
        return {"weights": s["d_particles"][:, 6], "pose": s["d_pose"], "resampled": s["d_out"],
                "count": s["d_count"]}
    if kind == "host":
        pose = s["evaluator"].evaluate(s["particles"], s["points"], s["tf"])
        resampled = s["host_resampler"].resample(s["particles"], s["u0"])
        count = resampled.shape[0]
        s["next"][:count] = resampled
        return {"weights": s["particles"][:, 6], "pose": pose.as_array(), "resampled": s["next"], "count": count}
    if kind == "cloud":
        cell = MAPS[s["map"]][6]
        pose, n = s["evaluator"].evaluate_cloud(s["particles"], s["cloud"], s["records"], 16, s["tf"],
                                                reduction_cell_size=cell)
        return {"weights": s["particles"][:, 6], "pose": pose.as_array(), "points": n}
    if kind == "filter":
        _move(s)
        _evaluate(s)
        N.check(N.lib().tsdfl_best_particle_device(s["ctx"].handle, _p(s["d_particles"]), s["P"], _p(s["d_best"])))
        _resample(s)
        return {"poses": s["d_particles"][:, :6], "weights": s["d_particles"][:, 6], "pose": s["d_pose"],
                "best": s["d_best"], "resampled": s["d_out"], "count": s["d_count"]}
    if kind == "scan":
        N.check(N.lib().tsdfl_reduce_scan_device(s["ctx"].handle, _p(s["d_cloud"]), s["records"], 16, 0, 12,
                                                 MAPS[s["map"]][6], 0, _p(s["d_out"]),
                                                 s["d_out"].shape[0], _p(s["d_count"])))
        return {"points": s["d_out"], "count": s["d_count"]}
    if kind == "motion":
        _move(s)
        return {"poses": s["d_particles"][:, :6]}
    if kind == "resample":
        _resample(s)
        return {"resampled": s["d_out"], "count": s["d_count"]}
    if kind == "batch":
        s["batch"].run()
        return {"weights": s["d_particles"][:, 6], "pose": s["d_pose"], "resampled": s["d_out"],
                "count": s["d_count"]}
    N.check(N.lib().tsdfl_evaluate_subsampled_device(s["ctx"].handle, s["dmap"].handle, C.byref(s["model"]),
                                                     _p(s["d_particles"]), s["P"], _p(s["d_points"]), s["N"],
                                                     s["tf"].ctypes.data_as(C.c_void_p), s["K"], s["seed"],
                                                     _p(s["d_pose"])))
    return {"weights": s["d_particles"][:, 6], "pose": s["d_pose"]}


# ---------------------------------------------------------------- what a pass cannot do without

MAP_BYTES = {"room": 20e6, "building": 1.359e9, "warehouse": 269e6, "tunnel": 59e6}   # 2 bytes a slot


def _update_work(name: str, P: float, n: float) -> tuple[float, float]:
    """One sensor update: poses in, weights out, the scan once, of the map the
    slots looked up (at most all of it); per lookup the transform, the scaling
    to a slot and the sum, per particle the pose and the normalisation."""
    return 28.0 * P + 12.0 * n + min(2.0 * P * n, MAP_BYTES[name]), 22.0 * P * n + 120.0 * P


def work(case: dict) -> dict:
    kind = case["kind"]
    P = float(case.get("P", 0))
    if kind == "scan":
        n = float(case["rings"] * case["columns"])
        return {"bytes": (16.0 + 12.0) * n, "flops": 20.0 * n}
    if kind == "motion":
        return {"bytes": 48.0 * P, "flops": 400.0 * P}
    if kind == "resample":
        return {"bytes": 56.0 * P, "flops": 8.0 * P}
    if kind == "batch":
        parts = [_update_work(*f) for f in _points_drawn(case, case["filters"])]
        total = float(sum(f[1] for f in _points_drawn(case, case["filters"])))
        return {"bytes": sum(b for b, _ in parts) + 56.0 * total, "flops": sum(f for _, f in parts) + 8.0 * total}
    if kind == "cloud":
        raw = float(case["rings"] * case["columns"])
        b, f = _update_work(case["map"], P, 0.85 * raw)
        return {"bytes": b + 16.0 * raw, "flops": f + 20.0 * raw}
    b, f = _update_work(case["map"], P, float(case["K"] if kind == "subsampled" else case["N"]))
    if kind == "filter":
        b, f = b + 48.0 * P, f + 400.0 * P
    if "resampler" in case:
        b, f = b + 56.0 * P, f + 8.0 * P
    return {"bytes": b, "flops": f}


# ---------------------------------------------------------------- the outputs in 64 bits

def _likelihoods() -> torch.Tensor:
    """Likelihood of every slot code: |tsdf| in mm below 600, then the init value and a miss."""
    mm = torch.arange(600, dtype=torch.float64, device="cuda") * 1e-3
    peak = 1.0 / math.sqrt(2.0 * math.pi * SIGMA * SIGMA)
    v = (torch.exp(-mm * mm / (2.0 * SIGMA * SIGMA)) * peak) ** 3
    return torch.cat([v, torch.zeros(2, dtype=torch.float64, device="cuda")])   # exp(-5000) is 0 in float


class _Lookup:
    """The map as the reference indexes it: float offsets, 1 m bricks, sub-voxels
    by float division, and its conversions of negative floats to size_t."""

    def __init__(self, name: str):
        coef, occ, codes = _map_arrays(name)
        self.c = coef
        self.occ = torch.from_numpy(np.ascontiguousarray(occ, np.int32)).cuda()
        self.codes = torch.from_numpy(codes.view(np.int16)).cuda()
        self.values = _likelihoods()
        # a tensor: torch multiplies by the reciprocal of a number
        self.resolution = torch.tensor(coef.resolution, dtype=torch.float32, device="cuda")
        # largest brick coordinate that passes the check against the map's size in voxels
        whole = torch.arange(8192, dtype=torch.float32, device="cuda")
        self.last = [int((torch.floor(whole / self.resolution) < d).sum()) - 1
                     for d in (coef.dim_x, coef.dim_y, coef.dim_z)]

    def __call__(self, x, y, z):
        c = self.c
        up = idx = odd = 0
        ok = torch.ones_like(x, dtype=torch.bool)
        for v, lo, last, brick, sub in ((x, c.min_x, self.last[0], 1, 1),
                                        (y, c.min_y, self.last[1], c.up_dim_x, c.sub_dim),
                                        (z, c.min_z, self.last[2], c.up_dim_2, c.sub_dim_2)):
            o = v - torch.tensor(lo, dtype=torch.float32, device="cuda")
            t = torch.trunc(o)
            far = o <= -1.0
            ok &= t <= last
            q = torch.trunc((o - t) / self.resolution)
            up = up + t.long() * brick
            idx = idx + torch.where(far, torch.zeros_like(q), q).long() * sub
            odd = odd + far.long() * sub
        ok &= (up >= 0) & (up < c.grid_occ_size) & (odd % 2 == 0)
        base = self.occ[torch.where(ok, up, torch.zeros_like(up))].long()
        idx = idx + base
        ok &= (base >= 0) & (idx >= 0) & (idx < c.data_size)
        code = self.codes[torch.where(ok, idx, torch.zeros_like(idx))].long()
        return self.values[torch.where(ok, code, torch.full_like(code, 601))]


def _laser_poses(particles: torch.Tensor) -> torch.Tensor:
    """3 x 4 transforms: sines and cosines rounded to float, float products and sums."""
    a = particles[:, 3:6].double()
    (sa, sb, sg), (ca, cb, cg) = a.sin().float().unbind(1), a.cos().float().unbind(1)
    x, y, z = particles[:, 0], particles[:, 1], particles[:, 2] + HEIGHT
    return torch.stack([cb * cg, sa * sb * cg - ca * sg, ca * sb * cg + sa * sg, x,
                        cb * sg, sa * sb * sg + ca * cg, ca * sb * sg - sa * cg, y,
                        -sb, sa * cb, ca * cb, z], 1)


def _kept_points(seed: int, P: int, n: int, K: int) -> torch.Tensor:
    """Scan index of each particle's K points: one per stratum of consecutive
    points, by SplitMix64 (Steele, Lea and Flood 2014) per particle."""
    def signed(v):
        return v - (1 << 64) if v >= 1 << 63 else v

    def mix(v):
        for shift, factor in ((30, 0xBF58476D1CE4E5B9), (27, 0x94D049BB133111EB)):
            v = (v ^ ((v >> shift) & ((1 << (64 - shift)) - 1))) * signed(factor)
        return v ^ ((v >> 31) & ((1 << 33) - 1))

    k = torch.arange(K, device="cuda")
    start = mix(seed ^ mix(torch.arange(P, device="cuda")))
    u = (mix(start[:, None] + (k + 1) * signed(0x9E3779B97F4A7C15)) >> 32) & 0xFFFFFFFF
    b0, b1 = k * n // K, (k + 1) * n // K
    return b0 + ((u * (b1 - b0)) >> 32)


def _update64(name: str, particles: np.ndarray, points: np.ndarray, K: int = 0, seed: int = 0):
    """(weights, mean pose) of a sensor update: likelihoods, sums, normalisation
    and means in 64 bits, of the slots the float transform falls in."""
    a_hit, a_range, a_max, max_range = MODEL
    look = _Lookup(name)
    p, q = _cuda(particles), _cuda(points)
    T = _laser_poses(p)
    inside = q.double().square().sum(1) < max_range ** 2
    term = torch.where(inside, a_range / max_range, a_max).double()
    raw = torch.empty(p.shape[0], dtype=torch.float64, device="cuda")
    step = max(1, (1 << 23) // (K or q.shape[0]))
    chosen = _kept_points(seed, p.shape[0], q.shape[0], K) if K else None
    for i in range(0, p.shape[0], step):
        t = T[i:i + step, :, None]
        pts = q[chosen[i:i + step]] if K else q[None]
        x, y, z = pts.unbind(2)
        v = look(((t[:, 0] * x + t[:, 1] * y) + t[:, 2] * z) + t[:, 3],
                 ((t[:, 4] * x + t[:, 5] * y) + t[:, 6] * z) + t[:, 7],
                 ((t[:, 8] * x + t[:, 9] * y) + t[:, 10] * z) + t[:, 11])
        raw[i:i + step] = a_hit * v.sum(1) + (term[chosen[i:i + step]].sum(1) if K else term.sum())
    w = raw / raw.sum()
    d = p.double()
    angles = [torch.atan2((d[:, k].sin() * w).sum(), (d[:, k].cos() * w).sum()) for k in (3, 4, 5)]
    return w, torch.stack([*(d[:, :3] * w[:, None]).sum(0), *angles])


def _philox(counters: np.ndarray, key: tuple[int, int]) -> np.ndarray:
    """Philox4x64 with 10 rounds (Salmon et al., SC 2011) of (n, 4) counters."""
    def mul(a, b):
        low, half = np.uint64(0xFFFFFFFF), np.uint64(32)
        b = np.uint64(b)
        al, ah, bl, bh = a & low, a >> half, b & low, b >> half
        mid = ah * bl + ((al * bl) >> half)
        mid2 = al * bh + (mid & low)
        return ah * bh + (mid >> half) + (mid2 >> half), a * b

    c = [counters[:, k].copy() for k in range(4)]
    k0, k1 = key
    with np.errstate(over="ignore"):
        for _ in range(10):
            h0, l0 = mul(c[0], 0xD2E7470EE14C6C93)
            h1, l1 = mul(c[2], 0xCA5A826395121157)
            c = [h1 ^ c[1] ^ np.uint64(k0), l1, h0 ^ c[3] ^ np.uint64(k1), l0]
            k0, k1 = (k0 + 0x9E3779B97F4A7C15) % (1 << 64), (k1 + 0xBB67AE8584CAA73B) % (1 << 64)
    return np.stack(c, 1)


def _rotation(r, p, y) -> np.ndarray:
    """Rz Ry Rx of angle arrays, (n, 3, 3)."""
    cr, sr, cp, sp, cy, sy = np.cos(r), np.sin(r), np.cos(p), np.sin(p), np.cos(y), np.sin(y)
    return np.stack([cp * cy, sr * sp * cy - cr * sy, cr * sp * cy + sr * sy,
                     cp * sy, sr * sp * sy + cr * cy, cr * sp * sy - sr * cy,
                     -sp, sr * cp, cr * cp], 1).reshape(-1, 3, 3)


def _motion64(case: dict, particles: np.ndarray, seed: int) -> np.ndarray:
    """Poses after the motion update: six Box-Muller normals a particle, composed with its pose."""
    inputs, dt = _motion_inputs(case)
    m = MotionModel(_ctx()).distributions(case.get("motion", "scale"), inputs, dt)
    n = particles.shape[0]
    words = []
    for block in (0, 1):
        c = np.zeros((n, 4), np.uint64)
        c[:, 0], c[:, 1] = np.arange(n), block
        words.append(_philox(c, (seed, 0x6D6F74696F6E0001)))
    words = np.concatenate(words, 1)[:, :6] >> np.uint64(11)
    r = np.sqrt(-2.0 * np.log((words[:, ::2] + 1.0) * 2.0 ** -53))
    angle = 2.0 * np.pi * (words[:, 1::2] * 2.0 ** -53)
    z = np.stack([r * np.cos(angle), r * np.sin(angle)], 2).reshape(n, 6)
    d = z * np.array(m.stddev[:]) + np.array(m.mean[:])
    p = particles.astype(np.float64)
    R = _rotation(p[:, 3], p[:, 4], p[:, 5])
    M = R @ _rotation(d[:, 3], d[:, 4], d[:, 5])
    return np.concatenate([p[:, :3] + (R @ d[:, :3, None])[..., 0],
                           np.stack([np.arctan2(M[:, 2, 1], M[:, 2, 2]), -np.arcsin(M[:, 2, 0]),
                                     np.arctan2(M[:, 1, 0], M[:, 0, 0])], 1)], 1)


def exact(case: dict, seed: int):
    kind = case["kind"]
    if kind in ("scan", "resample", "filter"):
        # points and particles passed on as they are; a filter step's update
        # scores the float poses its motion update left
        return None
    if kind == "motion":
        return {"poses": _motion64(case, _weighted(seed, case["P"]), seed)}
    if kind == "batch":
        parts = [_update64(*spec) for spec in _batch_specs(case, seed)]
        return {"weights": torch.cat([w for w, _ in parts]), "pose": torch.stack([q for _, q in parts]),
                "resampled": None, "count": None}
    if kind == "cloud":
        return None   # the reduced points are not among the outputs
    cloud = "global" if kind == "subsampled" else case.get("cloud", "tracking")
    points = _points(case["map"], seed, case["N"])
    w, pose = _update64(case["map"], _particles(case["map"], cloud, seed, case["P"]), points, case.get("K", 0), seed)
    if kind == "subsampled":
        return {"weights": w, "pose": pose}
    return {"weights": w, "pose": pose, "resampled": None, "count": None}
