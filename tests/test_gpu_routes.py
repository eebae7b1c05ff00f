"""Routes that a launch takes by size or by inputs give the same photons.

A photon's trajectory depends on the table, the seed, the stream and the math and
step mode only.  These tests compare, bit for bit, runs that reach the same photons
by different code: maps from the tiled passes against closed forms, blocks of one
warp (which never hand photons over) against larger ones, jobs in one launch against
jobs alone, and fast-math tallies against recorded ones.
"""
from __future__ import annotations

import hashlib
import json
from pathlib import Path

import numpy as np
import pytest

import ymc3d_b200 as m
from helpers import oracle_job, residual, safe_distance_bruteforce
from ymc3d_b200 import workloads

pytestmark = pytest.mark.gpu

GOLDEN = Path(__file__).parent / "golden" / "fast_tallies.json"


def _log(r):
    return r.photon_log.view(np.uint8).reshape(len(r.photon_log), -1)


# tiles are 64 lines of 64 voxels with a halo of 63, rows whole words, bits 32 to a word
@pytest.mark.parametrize("shape", [(1, 1, 1), (2, 5, 67), (65, 63, 4), (66, 129, 31),
                                   (3, 64, 65), (130, 3, 33), (70, 66, 130)])
@pytest.mark.parametrize("kind", ["blocks", "specks", "one"])
def test_safe_distance_tile_edges(shape, kind):
    rng = np.random.default_rng(sum(shape))
    if kind == "one":
        t = np.full(shape, 2, np.uint8)
    elif kind == "blocks":
        c = rng.integers(0, 4, [s // 37 + 1 for s in shape]).astype(np.uint8)
        t = np.kron(c, np.ones((37, 37, 37), np.uint8))[:shape[0], :shape[1], :shape[2]]
    else:
        t = np.ones(shape, np.uint8)
        for _ in range(3):
            t[tuple(rng.integers(0, s) for s in shape)] = 3
    t = np.ascontiguousarray(t)
    assert np.array_equal(m.safe_distance(t), safe_distance_bruteforce(t))


# A voxel more than 63 below everything the photons reach changes the route of the whole
# map (one tissue -> passes, one index -> classes' map) and none of the cells they read.
@pytest.mark.parametrize("extra", ["same tissue", "other index"])
@pytest.mark.parametrize("nx,ny", [(33, 66), (70, 31)])
def test_map_routes_agree(table, extra, nx, ny):
    t = np.ones((190, ny, nx), np.uint8)
    if extra == "other index":
        t[:, ny // 2:] = 2
    far = t.copy()
    far[-1, 0, 0] = 2 if extra == "same tissue" else 3
    rows = [(8.0, 40.0, 0.9, 1.4), (8.0, 30.0, 0.8, 1.4),
            (8.0, 30.0, 0.8, 1.4 if extra == "same tissue" else 1.37)]
    p = m.OpticalProps.from_tissues(rows)
    job = m.Job(0, 0, 20_000, 4711, "uniform")
    a, b = (m.run([m.Geometry(g, 0.05, 0.05, 0.05)], [p], [job], table=table,
                  photon_log=True)[0] for g in (t, far))
    assert a.photon_log["z"].max() < 100 * 0.05
    assert np.array_equal(_log(a), _log(b)) and a.totals == b.totals


# Streams of several photons, jobs whose paths differ by 100 times, the step cap and the
# absorption map: a block of one warp keeps every photon where it started, larger blocks
# hand them over while the launch drains.
@pytest.mark.parametrize("math,steps,photons", [("fast", "merged", 4000), ("fast", "voxel", 1500),
                                                ("exact", "merged", 700), ("f64", "merged", 700)])
@pytest.mark.parametrize("absorption", [False, True])
def test_drain_keeps_photons(table, math, steps, photons, absorption):
    g = workloads.layered_vessel_geometry(40, 33, 20, 0.1)
    props = [m.OpticalProps.from_tissues(workloads.LAYER_ROWS),
             m.OpticalProps.from_tissues([(0.02 * a, s, gg, n)
                                          for a, s, gg, n in workloads.LAYER_ROWS])]
    jobs = [m.Job(0, 0, photons, 11, "uniform", streams=67),
            m.Job(0, 1, photons // 4, 12, "pencil"),
            m.Job(0, 0, 65, 13, "uniform")]
    kw = dict(table=table, math=math, steps=steps, photon_log=True, max_steps=60_000,
              absorption_map=absorption)
    base = m.run([g], props, jobs, block=32, **kw)
    for block in (64, 96, 128, 256):
        for x, y in zip(base, m.run([g], props, jobs, block=block, **kw)):
            assert x.totals == y.totals and residual(y.totals) == 0
            assert np.array_equal(_log(x), _log(y))
            assert np.array_equal(x.drs, y.drs) and np.array_equal(x.trans, y.trans)
            if absorption:
                assert np.array_equal(x.absorption, y.absorption)


def test_job_order_is_the_callers(table):
    """Eight jobs, the least absorbing last: their streams start in another order, their
    tallies come back in the caller's (read at once, more than four jobs)."""
    g = workloads.homogeneous(n=24).geoms[0]
    props = [m.OpticalProps.from_tissues([(0.5 / 2 ** k, 10.0, 0.9, 1.4)]) for k in range(8)]
    jobs = [m.Job(0, k, 2000 + 300 * k, 21 + k, "uniform") for k in range(8)]
    plan = m.Plan([g], props, jobs, table=table)
    plan.execute()
    for k, r in enumerate(plan.read()):
        alone = m.run([g], [props[k]], [m.Job(0, 0, jobs[k].photons, 21 + k, "uniform")],
                      table=table)[0]
        assert r.totals == alone.totals
        assert np.array_equal(r.drs, alone.drs) and np.array_equal(r.drs_sq, alone.drs_sq)
    plan.close()


def fast_cases():
    """name -> (geometries, sets, jobs, options) of the recorded tallies"""
    rng = np.random.default_rng(3)
    blocks = np.kron(rng.integers(0, 5, (5, 6, 7)), np.ones((4, 4, 4))).astype(np.uint8)
    blocks[:4] = np.maximum(blocks[:4], 1)
    airy = m.Geometry(blocks, 0.05, 0.07, 0.04)
    rows = m.OpticalProps.from_tissues([(0.3, 10, 0.8, 1.4), (0.05, 15, 0.9, 1.37),
                                        (1.0, 20, 0.7, 1.5), (0.01, 5, 0.6, 1.33)])
    lay = workloads.layered_vessel(60_000, seed=777)
    un = workloads.uneven(3, 10_000, max_dim=80)
    sw = workloads.sweep(6, photon_scale=2e-4)
    lv = (lay.geoms, lay.props, lay.jobs)
    return {
        "layered_merged": (*lv, {}),
        "layered_voxel": (lay.geoms, lay.props, [m.Job(0, 0, 10_000, 777)], {"steps": "voxel"}),
        "layered_absorption": (*lv, {"absorption_map": True}),
        "uneven_merged": (un.geoms, un.props, un.jobs, {}),
        "uneven_absorption": (un.geoms, un.props, un.jobs, {"absorption_map": True}),
        "uneven_voxel": (un.geoms, un.props, [m.Job(k, k, 2000, 5 + k) for k in range(3)],
                         {"steps": "voxel"}),
        "air_blocks": ([airy], [rows], [m.Job(0, 0, 40_000, 123, "uniform", 1000)], {}),
        "sweep": (sw.geoms, sw.props, sw.jobs, {}),
    }


def tallies(results):
    out = []
    for r in results:
        h = hashlib.sha256(r.drs.tobytes() + r.drs_sq.tobytes() + r.trans.tobytes())
        if r.absorption is not None:
            h.update(r.absorption.tobytes())
        out.append({"totals": {k: int(v) for k, v in r.totals.items()}, "sha256": h.hexdigest()})
    return out


@pytest.mark.parametrize("name", ["layered_merged", "layered_voxel", "layered_absorption",
                                  "uneven_merged", "uneven_absorption", "uneven_voxel",
                                  "air_blocks", "sweep"])
def test_fast_tallies_are_the_recorded_ones(table, name):
    """Fast math writes down which products it fuses, so its tallies are a property of the
    inputs; the recorded ones are of the last build that left the choice to the compiler."""
    geoms, props, jobs, how = fast_cases()[name]
    want = json.loads(GOLDEN.read_text())[name]
    assert tallies(m.run(geoms, props, jobs, table=table, **how)) == want


@pytest.mark.parametrize("scale", [1.0, 2.0 ** -58, 2.0 ** -66, 2.0 ** 64])
@pytest.mark.parametrize("absorption", [False, True])
def test_exact_divisions_at_the_range_ends(table, scale, absorption):
    """Exact math divides by voxel sizes and mu_t through their reciprocals within
    [2^-60, 2^60] and by IEEE division beyond: photon by photon the CPU transcription's
    states on both sides (a layered medium scaled in length, and so in 1/mm)."""
    g = workloads.layered_vessel_geometry(31, 28, 17, 0.11)
    g = m.Geometry(g.tissue, 0.11 * scale, 0.13 * scale, 0.07 * scale)
    p = m.OpticalProps.from_tissues([(a / scale, s / scale, gg, n)
                                     for a, s, gg, n in workloads.LAYER_ROWS])
    job = m.Job(0, 0, 600, 271828, "uniform")
    r = m.run([g], [p], [job], table=table, math="exact", photon_log=True, max_steps=20_000,
              absorption_map=absorption)[0]
    o = oracle_job(g, p, job, table, photon_log=True, max_steps=20_000)
    assert np.array_equal(_log(r), o["photon_log"].view(np.uint8).reshape(600, -1))
    assert r.totals == o["totals"] and np.array_equal(r.drs, o["drs"])


# A grid with more than 2^21 voxels along an axis takes the kernels without the short
# index arithmetic, and takes the launch's other jobs with it.
@pytest.mark.parametrize("steps,absorption", [("merged", False), ("merged", True),
                                              ("voxel", False), ("voxel", True)])
def test_long_axis_kernels_agree(table, steps, absorption):
    rng = np.random.default_rng(5)
    geo = lambda t: m.Geometry(np.ascontiguousarray(t), 0.05, 0.04, 0.06)
    t = np.kron(rng.integers(1, 4, (3, 4, 5)), np.ones((9, 7, 8), int)).astype(np.uint8)
    t[:2, :3, :3] = 0
    p = m.OpticalProps.from_tissues([(0.3, 9.0, 0.9, 1.4), (2.0, 20.0, 0.7, 1.33),
                                     (0.1, 4.0, 0.0, 1.5)])
    job = m.Job(0, 0, 30_000, 99, "uniform")
    long = np.ones((1, 1, (1 << 21) + 1), np.uint8)
    runs = []
    for last in (long[:, :, :-1], long):
        runs.append(m.run([geo(t), geo(last)], [p], [job, m.Job(1, 0, 2_000, 7, "pencil")],
                          table=table, steps=steps, absorption_map=absorption, photon_log=True))
    (a, _), (b, w) = runs
    assert np.array_equal(_log(a), _log(b)) and a.totals == b.totals
    assert np.array_equal(a.drs, b.drs) and np.array_equal(a.trans, b.trans)
    alone = m.run([geo(long)], [p], [m.Job(0, 0, 2_000, 7, "pencil")], table=table, steps=steps,
                  absorption_map=absorption, photon_log=True)[0]
    assert residual(w.totals) == 0 and residual(alone.totals) == 0
    if absorption:
        assert np.array_equal(a.absorption, b.absorption)
        assert int(alone.absorption.sum()) == alone.totals["absorbed"]
    else:
        assert np.array_equal(_log(w), _log(alone)) and w.totals == alone.totals


def test_long_axis_noalloc(table):
    """the allocation-free entry's kernel for such a grid against mc3d_run's"""
    import ctypes as C

    import torch

    t = np.ones((1, 1, (1 << 21) + 1), np.uint8)
    g, p = m.Geometry(t, 0.05, 0.04, 0.06), m.OpticalProps.from_tissues([(0.3, 9.0, 0.9, 1.4)])
    job = m.Job(0, 0, 2_000, 7, "uniform")
    tab = np.ascontiguousarray(table[:100_001])
    ref = m.run([g], [p], [job], table=tab, steps="voxel")[0]
    dev = torch.device("cuda", 0)
    tissue = torch.from_numpy(t.reshape(-1).copy()).to(dev)
    outs = [torch.zeros(t.size, dtype=torch.int64, device=dev) for _ in range(3)]
    totals = torch.zeros(14, dtype=torch.int64, device=dev)
    cg, cp, cj = m.CGeom(t.size, 1, 1, 0, g.dx, g.dy, g.dz, tissue.data_ptr()), p.c(), job.c()
    assert m.lib().mc3d_run_noalloc(C.byref(cg), C.byref(cp), C.byref(cj), tab.ctypes.data,
                                    len(tab), 0, None, *[o.data_ptr() for o in outs],
                                    totals.data_ptr()) == 0
    torch.cuda.synchronize(dev)
    assert list(ref.totals.values()) == totals.tolist()
    assert np.array_equal(outs[0].cpu().numpy().view(np.uint64), ref.drs.reshape(-1))
