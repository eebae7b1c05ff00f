"""Timed cases of the photon engine, through the calls a user's program makes.

A program either calls ``run`` once per optical set (inputs on the host, tallies
back on the host: upload, cell maps, seeding, photon loop, read-back), or keeps a
``Plan`` and executes it (photon loop and read-back).  Every case returns all the
tallies of the call: reflected weight and its square per bin, transmitted weight
per bin, the fourteen totals of each job, and the absorption map where asked for.
They are 64-bit integer sums, the same for the same inputs.

Sizes are those of the five workloads of ``ymc3d_b200.workloads`` and of its skin
model, at photon counts from a quick look to a full simulation.
"""
from __future__ import annotations

import math

import numpy as np

import ymc3d_b200 as ymc
from ymc3d_b200 import workloads


def listed():
    return [
        # a quick look at one medium: a call of few photons, ruled by set-up and by the
        # longest path
        _case("pencil_64_1e4", "pencil", 64, 64, 64, 0.1, 10_000, beam="pencil"),
        # the plain method's own size: one tissue, pencil beam, 1e6 photons
        _case("pencil_64_1e6", "pencil", 64, 64, 64, 0.1, 1_000_000, beam="pencil"),
        # the skin model with its vessel (50 x 50 x 85 voxels), one wavelength
        _case("skin_2e5", "skin", 50, 50, 85, 0.02, 200_000),
        # one wavelength on the layered model with a vessel, whole call
        _case("layered_1e6", "layered", 256, 256, 128, 0.02, 1_000_000),
        # the same model as a long simulation on a kept plan: the photon loop itself
        _case("layered_plan_4e7", "layered", 256, 256, 128, 0.02, 40_000_000, plan=True),
        # the reference's one step per voxel face, on a kept plan
        _case("layered_voxel_2e6", "layered", 256, 256, 128, 0.02, 2_000_000, plan=True,
              steps="voxel"),
        # absorbed weight per voxel beside the reflectance (fluence maps)
        _case("layered_absorption_5e5", "layered", 256, 256, 128, 0.02, 500_000,
              absorption=True),
        # hyperspectral sweep: 128 optical sets on one geometry in one launch, replayed
        # from a CUDA graph
        _case("sweep_128", "sweep", 64, 64, 64, 0.1, 10_000_000, jobs=128, plan=True,
              graph=True),
        # geometries of different sizes with ellipsoid inclusions in one launch
        _case("uneven_12", "uneven", 160, 160, 80, 0.02, 1_200_000, jobs=12),
        # a grid far beyond the L2 cache, high albedo, long paths
        _case("deep_1e5", "deep", 1024, 1024, 256, 0.01, 100_000),
        # FP64 stepping, the precision study's other arm
        _case("layered_f64_2e5", "layered", 256, 256, 128, 0.02, 200_000, math="f64"),
        # reproducible math, photon by photon comparable with the CPU transcription
        _case("layered_exact_1e5", "layered", 128, 128, 64, 0.04, 100_000, math="exact"),
    ]


def _case(name, model, nx, ny, nz, voxel, photons, jobs=1, beam="uniform", math="fast",
          steps="merged", absorption=False, plan=False, graph=False):
    c = dict(model=model, nx=nx, ny=ny, nz=nz, voxel=voxel, photons=photons, jobs=jobs,
             beam=beam, math=math, steps=steps, absorption=absorption, plan=plan, graph=graph)
    if name:
        c["name"] = name
    return c


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    """Another case of the same kinds: grids from 32 voxels an axis up, odd sizes among
    them, photon counts over the logarithm of their range."""
    kind = rng.choice(["pencil", "skin", "layered", "layered", "voxel", "absorption", "sweep",
                       "uneven", "deep", "f64", "exact"])
    beam = rng.choice(["uniform", "pencil"])
    if kind == "pencil":
        n = _log(rng, 32, 160)
        return _case("", kind, n, n, n, rng.choice([0.05, 0.1]), _log(rng, 1e4, 5e6), beam=beam,
                     plan=rng.random() < 0.3)
    if kind == "skin":
        n = _log(rng, 40, 120)
        return _case("", kind, n, n, int(round(1.7 * n)), 1.0 / n, _log(rng, 1e4, 2e6), beam=beam)
    if kind == "sweep":
        jobs = _log(rng, 4, 128)
        return _case("", kind, 64, 64, 64, 0.1, jobs * _log(rng, 5e3, 1e5), jobs=jobs, beam=beam,
                     plan=rng.random() < 0.5, graph=rng.random() < 0.5)
    if kind == "uneven":
        jobs = rng.randint(2, 12)
        n = _log(rng, 64, 160)
        return _case("", kind, n, n, max(64, n // 2), 0.02, jobs * _log(rng, 1e4, 2e5), jobs=jobs)
    if kind == "deep":
        n = _log(rng, 192, 640)
        return _case("", kind, n, n - rng.randint(0, 31), _log(rng, 64, 256), 0.01,
                     _log(rng, 1e4, 2e5))
    nx, ny, nz = _log(rng, 48, 320), _log(rng, 48, 320), _log(rng, 32, 160)
    voxel = rng.choice([0.02, 0.03, 0.04])
    if kind == "layered":
        return _case("", kind, nx, ny, nz, voxel, _log(rng, 1e4, 2e7), beam=beam,
                     plan=rng.random() < 0.5)
    if kind == "voxel":
        return _case("", "layered", nx, ny, nz, voxel, _log(rng, 1e4, 2e6), beam=beam,
                     steps="voxel", plan=rng.random() < 0.5)
    if kind == "absorption":
        return _case("", "layered", nx, ny, nz, voxel, _log(rng, 1e4, 1e6), beam=beam,
                     absorption=True)
    return _case("", "layered", nx, ny, nz, voxel, _log(rng, 1e4, 2e5), beam=beam, math=kind)


def _workload(case, seed):
    rng = np.random.Generator(np.random.PCG64(seed))
    nx, ny, nz, d, photons = (case[k] for k in ("nx", "ny", "nz", "voxel", "photons"))
    job_seed = int(rng.integers(1, 1 << 31))
    model, jobs = case["model"], case["jobs"]
    if model == "sweep":
        w = workloads.sweep(jobs, rng_seed=seed, seed_base=job_seed, beam=case["beam"])
        total = w.photons
        for j in w.jobs:
            j.photons = max(1, int(j.photons * photons / total))
        return w.geoms, w.props, w.jobs
    if model == "uneven":
        # the grids' sizes are the case's; the inclusions' place and the tissues are the seed's
        w = workloads.uneven(jobs, photons // jobs, rng_seed=nx + 1000 * jobs, d=d,
                             seed_base=job_seed, max_dim=nx)
        for g, p in zip(w.geoms, w.props):
            g.tissue = np.ascontiguousarray(np.roll(g.tissue, int(rng.integers(64)), 2))
            p.mua[1:] *= rng.uniform(0.9, 1.1, len(p.mua) - 1).astype(np.float32)
            p.mus[1:] *= rng.uniform(0.9, 1.1, len(p.mus) - 1).astype(np.float32)
        return w.geoms, w.props, w.jobs
    if model == "deep":
        w = workloads.deep_grid(photons, rng_seed=seed, nx=nx, ny=ny, nz=nz, d=d, seed=job_seed)
        return w.geoms, w.props, w.jobs
    # one geometry and one optical set, its absorption and scattering up to 10 % off
    # the model's as another wavelength's are
    if model == "pencil":
        geom = ymc.Geometry(np.ones((nz, ny, nx), np.uint8), d, d, d)
        rows = [workloads.HOMOGENEOUS_ROW]
    elif model == "skin":
        geom = workloads.skin_geometry(dx=d, length_xy=nx * d, length_z=nz * d)
        props = workloads.skin_optprops(float(rng.uniform(500, 800)),
                                        lambda oxygenation, lam: 500.0 + 300.0 * oxygenation)
        rows = list(zip(props.mua, props.mus, props.g, props.n))[1:]
    else:
        geom = workloads.layered_vessel_geometry(nx, ny, nz, d)
        rows = workloads.LAYER_ROWS
    rows = [(a * rng.uniform(0.9, 1.1), s * rng.uniform(0.9, 1.1), g, n) for a, s, g, n in rows]
    return ([geom], [ymc.OpticalProps.from_tissues(rows)],
            [ymc.Job(0, 0, photons, job_seed, case["beam"])])


def prepare(case, seed):
    """Geometry, optical sets, jobs and the safe-prime table, and the plan where the
    program keeps one."""
    geoms, props, jobs = _workload(case, seed)
    table = ymc.default_table()
    how = dict(math=case["math"], steps=case["steps"])
    if case["plan"]:
        return {"plan": ymc.Plan(geoms, props, jobs, table, use_graph=case["graph"], **how)}
    return {"args": (geoms, props, jobs, table),
            "how": dict(how, absorption_map=case["absorption"])}


def run(state):
    if "plan" in state:
        state["plan"].execute()
        results = state["plan"].read()
    else:
        results = ymc.run(*state["args"], **state["how"])
    if len(results) == 1:
        r = results[0]
        out = {"drs": r.drs.view(np.int64), "drs_sq": r.drs_sq.view(np.int64),
               "trans": r.trans.view(np.int64)}
        if r.absorption is not None:
            out["absorption"] = r.absorption.view(np.int64)
    else:
        out = {k: np.concatenate([getattr(r, k).reshape(-1) for r in results]).view(np.int64)
               for k in ("drs", "drs_sq", "trans")}
    out["totals"] = np.array([[r.totals[k] for k in ymc.TOTAL_FIELDS] for r in results], np.int64)
    return out


def exact(case, seed):
    """None: the outputs are integer tallies of a seeded simulation."""
    return None


# Steps of one photon, the mean the engine's totals report: with the face crossings
# inside uniform tissue merged (160 elementary operations a step), and with one step
# per face (152) on the layered grid of 0.02 mm, where their number goes with 1 / voxel.
_MERGED = {"pencil": 1850, "skin": 750, "layered": 1950, "sweep": 1800, "uneven": 640,
           "deep": 20000}
_FACES_LAYERED = 10600


def work(case):
    voxels = case["nx"] * case["ny"] * case["nz"]
    bins = case["nx"] * case["ny"]
    geoms = case["jobs"] if case["model"] == "uneven" else 1
    if case["model"] == "uneven":  # sizes are uniform from 64 up to the largest
        mean = (64 + case["nx"]) / 2
        voxels, bins = mean * mean * (64 + case["nz"]) / 2, mean * mean
    nbytes = voxels * geoms + 24 * bins * case["jobs"] + 4 * min(case["photons"], 1 << 20)
    if case["absorption"]:
        nbytes += 8 * voxels
    ops = 160.0 * _MERGED[case["model"]]
    if case["steps"] == "voxel" or case["math"] == "exact":
        ops = 152.0 * _FACES_LAYERED * 0.02 / case["voxel"]
    return {"bytes": nbytes, "flops": ops * case["photons"]}
