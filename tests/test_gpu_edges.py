"""Inputs and launches at the edges of what a call accepts: lanes without a stream,
coefficients below the normal range, photons without a position, memory and tables at
their limits."""
from __future__ import annotations

import subprocess
import sys

import numpy as np
import pytest
import torch

import ymc3d_b200 as m
from conftest import ROOT
from helpers import oracle_job, residual, safe_distance_bruteforce, total_z
from ymc3d_b200 import autotune, workloads

pytestmark = pytest.mark.gpu

MODES = [("fast", "merged"), ("fast", "voxel"), ("exact", "merged"), ("f64", "merged"),
         ("f64", "voxel")]


def _log(r):
    return r.photon_log.view(np.uint8).reshape(len(r.photon_log), -1)


def _same(a, b):
    assert a.totals == b.totals and residual(a.totals) == 0
    assert np.array_equal(a.drs, b.drs) and np.array_equal(a.drs_sq, b.drs_sq)
    assert np.array_equal(a.trans, b.trans)
    if a.photon_log is not None and b.photon_log is not None:
        assert np.array_equal(_log(a), _log(b))


def _blocks(seed, shape, tissues):
    t = np.random.default_rng(seed).integers(1, tissues + 1, shape)
    return np.kron(t, np.ones((5, 4, 6), int)).astype(np.uint8)


# Most lanes of these launches never get a stream, in blocks that have photons and in
# blocks that have none; they pass the chunk loop all the same, which names a geometry.
@pytest.mark.parametrize("math,steps", MODES)
@pytest.mark.parametrize("streams", [1, 33])
def test_fewer_streams_than_threads(table, math, steps, streams):
    geoms = [m.Geometry(_blocks(1, (3, 4, 4), 2), 0.1, 0.08, 0.12),
             m.Geometry(_blocks(2, (5, 3, 2), 2), 0.06, 0.1, 0.05)]
    props = [m.OpticalProps.from_tissues([(0.5, 10, 0.8, 1.4), (2.0, 15, 0.9, 1.33)]),
             m.OpticalProps.from_tissues([(1.0, 20, 0.7, 1.5), (0.8, 12, 0.6, 1.4)])]
    jobs = [m.Job(k, k, 3 * streams, 41 + k, "uniform", streams=streams) for k in range(2)]
    kw = dict(table=table, math=math, steps=steps, photon_log=True)
    together = m.run(geoms, props, jobs, **kw)
    for k, r in enumerate(together):
        alone = m.run([geoms[k]], [props[k]], [m.Job(0, 0, 3 * streams, 41 + k, "uniform",
                                                     streams=streams)], **kw)[0]
        assert r.totals["photons"] == 3 * streams
        _same(r, alone)


# Voxel sizes so small that the residuals of a quotient by them, and then their
# reciprocals, leave the normal range: the kernels for such sizes divide along every axis.
@pytest.mark.parametrize("voxel,optical", [(-112, -112), (-126, -118), (-130, -118)])
@pytest.mark.parametrize("absorption", [False, True])
def test_exact_divides_by_tiny_voxels(table, voxel, optical, absorption):
    g = workloads.layered_vessel_geometry(31, 28, 17, 0.11)
    g = m.Geometry(g.tissue, *(d * 2.0 ** voxel for d in (0.11, 0.13, 0.07)))
    p = m.OpticalProps.from_tissues([(a / 2.0 ** optical, s / 2.0 ** optical, gg, n)
                                     for a, s, gg, n in workloads.LAYER_ROWS])
    job = m.Job(0, 0, 300, 271828, "uniform")
    r = m.run([g], [p], [job], table=table, math="exact", photon_log=True, max_steps=5_000,
              absorption_map=absorption)[0]
    o = oracle_job(g, p, job, table, photon_log=True, max_steps=5_000,
                   absorption_map=absorption)
    assert np.array_equal(_log(r), o["photon_log"].view(np.uint8).reshape(300, -1))
    assert r.totals == o["totals"] and np.array_equal(r.drs, o["drs"])
    if absorption:
        assert np.array_equal(r.absorption, o["absorption"])


# With g = 0 the scattering cosine is 0/0, so a photon has no position after its first
# scattering.  Until the quickfix removes it, its absorbed weight goes to the voxel its
# tissue is looked up in: the first one in FP32, the last one in FP64.
@pytest.mark.parametrize("math,steps", MODES)
def test_absorption_without_a_position(table, math, steps):
    t = np.ones((9, 7, 11), np.uint8)
    p = m.OpticalProps.from_tissues([(1.0, 5.0, 0.0, 1.4)])
    r = m.run([m.Geometry(t, 0.1, 0.1, 0.1)], [p], [m.Job(0, 0, 500, 77, "pencil")],
              table=table, math=math, steps=steps, absorption_map=True)[0]
    a = r.absorption.copy()
    assert int(a.sum()) == r.totals["absorbed"] and r.totals["quickfix"] > 0
    corners = [(0, 0, 0), (8, 6, 10)]
    lost, none = corners[::-1] if math == "f64" else corners
    assert a[lost] > 0 and a[none] == 0
    a[lost] = 0
    a[:, 3, 5] = 0  # the beam's column
    assert not a.any()


# Fast math flushes denormals, so a tissue whose mu_t is one stops a photon as air does and
# absorbs nothing of one that has no position (of a tissue with g = 0; it is looked up in the
# first voxel).  FP64 and exact math do not flush.
@pytest.mark.parametrize("steps", ["merged", "voxel"])
@pytest.mark.parametrize("mua,mus", [(1e-42, 0.0), (0.0, 1e-40), (3e-39, 4e-39)])
@pytest.mark.parametrize("g,n", [(0.8, 1.4), (0.8, 1.33), (0.0, 1.33)])
def test_denormal_mu_t_is_zero(table, steps, mua, mus, g, n):
    t = np.ones((12, 10, 14), np.uint8)
    t[7:] = 2
    t[:4, 2:5, 3:6] = 2
    t[0, 0, 0] = 2
    runs = []
    for a, s in ((0.0, 0.0), (mua, mus)):
        p = m.OpticalProps.from_tissues([(0.2, 8.0, g, 1.4), (a, s, 0.8, n)])
        runs.append(m.run([m.Geometry(t, 0.1, 0.1, 0.1)], [p], [m.Job(0, 0, 3000, 5, "uniform")],
                          table=table, steps=steps, photon_log=True, max_steps=20_000)[0])
    assert runs[0].totals["t_in"] > 0 and runs[0].totals["capped"] == 0
    _same(*runs)


@pytest.mark.parametrize("mua,mus", [(-50.0, 60.0), (-120.0, 150.0)])
def test_exact_follows_a_gain_medium(table, mua, mus):
    """A weight that grows beyond FP32's range: still the CPU transcription's photons."""
    t = np.ones((12, 10, 14), np.uint8)
    t[6:] = 2
    g = m.Geometry(t, 0.1, 0.1, 0.1)
    p = m.OpticalProps.from_tissues([(mua, mus, 0.8, 1.4), (0.5, 5.0, 0.6, 1.33)])
    job = m.Job(0, 0, 300, 99, "uniform")
    r = m.run([g], [p], [job], table=table, math="exact", photon_log=True, max_steps=3_000)[0]
    o = oracle_job(g, p, job, table, photon_log=True, max_steps=3_000)
    assert np.isnan(o["photon_log"]["W"]).any()
    for k in r.photon_log.dtype.names:
        assert np.array_equal(r.photon_log[k], o["photon_log"][k], equal_nan=True), k


def _in_fresh_process(code):
    """the process's last line of output; its library starts with an empty memory pool"""
    run = subprocess.run([sys.executable, "-c", code], cwd=ROOT, capture_output=True, text=True,
                         timeout=300)
    assert run.returncode == 0, run.stdout + run.stderr
    return run.stdout.splitlines()[-1]


_PLAN = """
import sys
sys.path.insert(0, ".")
import numpy as np, torch
import ymc3d_b200 as m
MiB = 1 << 20
free = lambda: torch.cuda.mem_get_info()[0]
dev = torch.device("cuda", 0)
torch.zeros(1, device=dev)
def fill(leave):
    torch.cuda.synchronize()
    return torch.empty(free() - leave, dtype=torch.uint8, device=dev)
"""


def test_optional_states_leave_room_for_the_rest():
    """A plan keeps its streams' states (8 bytes each, 512 MiB here) only beside what it
    cannot do without: an absorption map (512 MiB) that fits without them still fits, and
    the photons are the same either way."""
    out = _in_fresh_process(_PLAN + """
g = m.Geometry(np.ones((256, 512, 512), np.uint8), 0.05, 0.05, 0.05)
p = m.OpticalProps.from_tissues([(50.0, 5.0, 0.5, 1.4)])
job = m.Job(0, 0, 1 << 26, 7, "uniform")
m.run([m.Geometry(np.ones((2, 2, 2), np.uint8), 1, 1, 1)], [p], [m.Job(0, 0, 10, 7)])
hold = fill(64 * MiB + 2 * 512 * 512 * 319 + 512 * MiB + 200 * MiB)
a = m.run([g], [p], [job], absorption_map=True)[0]
del hold
torch.cuda.empty_cache()
b = m.run([g], [p], [job], absorption_map=True)[0]
assert a.totals == b.totals and a.totals["photons"] == 1 << 26
assert np.array_equal(a.drs, b.drs) and np.array_equal(a.absorption, b.absorption)
print("same")
""")
    assert out == "same"


def test_states_are_given_back_after_a_rejection():
    """A rejected seeding attempt makes the kept states useless: their memory (128 MiB) serves
    the next plan."""
    out = _in_fresh_process(_PLAN + """
table = m.default_table().copy()
table[1 + 12345] = 3
g = m.Geometry(np.ones((4, 4, 4), np.uint8), 0.1, 0.1, 0.1)
p = m.OpticalProps.from_tissues([(5.0, 5.0, 0.5, 1.4)])
plans = [m.Plan([g], [p], [m.Job(0, 0, 1 << 24, 7, "uniform")], table)]
before = free()
plans.append(m.Plan([g], [p], [m.Job(0, 0, 1 << 24, 8, "uniform")], table))
print((before - free()) // MiB)
""")
    assert int(out) < 64


def _many_sets(n):
    """n optical sets of five tissues, 240 bytes each in a block's shared memory"""
    return [m.OpticalProps.from_tissues([(a * (0.5 + k / n), s, g, i)
                                         for a, s, g, i in workloads.LAYER_ROWS])
            for k in range(n)]


# An SM has 228 KB for each block's tables, 136 bytes a thread and 1 KB a block, and registers
# for 20 warps in FP32: the most warps that fit in blocks of 128 to 256 threads.
@pytest.mark.parametrize("math", ["fast", "exact"])
@pytest.mark.parametrize("sets,warps", [(20, 20), (120, 20), (180, 18), (340, 14), (360, 12)])
def test_large_tables_keep_warps(table, math, sets, warps):
    g = m.Geometry(_blocks(7, (4, 5, 4), 4), 0.05, 0.05, 0.05)
    props = _many_sets(sets)
    jobs = [m.Job(0, k, 40, 100 + k, "uniform") for k in range(sets)]
    plan = m.Plan([g], props, jobs, table=table, math=math)
    block, grid, smem = plan.shape()
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    assert grid % sms == 0 and block * grid // sms == 32 * warps
    plan.execute()
    for a, b in zip(plan.read(), m.run([g], props, jobs, table=table, math=math, block=64)):
        _same(a, b)
    plan.close()


def test_fp64_tables_take_no_shared_memory(table):
    """FP64 stepping reads its tables from global memory: their size leaves its 16 warps an SM
    and the L1 cache alone."""
    g = m.Geometry(_blocks(7, (4, 5, 4), 4), 0.05, 0.05, 0.05)
    shapes = []
    for sets in (1, 340, 800):
        props = _many_sets(sets)
        jobs = [m.Job(0, k, 20, 100 + k, "uniform") for k in range(sets)]
        plan = m.Plan([g], props, jobs, table=table, math="f64")
        shapes.append(plan.shape())
        plan.execute()
        last = plan.read()[-1]
        plan.close()
        _same(last, m.run([g], props[-1:], [m.Job(0, 0, 20, 99 + sets, "uniform")], table=table,
                          math="f64")[0])
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    assert shapes[0] == shapes[1] == shapes[2]
    assert shapes[0][0] * shapes[0][1] // sms == 512


# Without a block size, a limit on the blocks leaves an SM as many threads as it can: blocks
# of 256 for one or two (16 warps is what fits of them), then what gives more.
@pytest.mark.parametrize("math", ["fast", "exact", "f64"])
@pytest.mark.parametrize("limit,warps", [(1, 8), (2, 16), (3, 18), (4, 20), (5, 20), (9, 20)])
def test_block_limit_counts_the_largest_blocks(table, math, limit, warps):
    g = m.Geometry(np.ones((8, 8, 8), np.uint8), 0.1, 0.1, 0.1)
    p = m.OpticalProps.from_tissues([(1.0, 10.0, 0.9, 1.4)])
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    job = m.Job(0, 0, 500, 3, "uniform")
    plan = m.Plan([g], [p], [job], table=table, math=math, blocks_per_sm=limit)
    block, grid, _ = plan.shape()
    assert grid // sms <= limit
    assert block * grid // sms == 32 * min(warps, 16 if math == "f64" else 20)
    plan.execute()
    _same(plan.read()[0], m.run([g], [p], [job], table=table, math=math)[0])
    plan.close()
    plan = m.Plan([g], [p], [job], table=table, math=math, block=64, blocks_per_sm=limit)
    assert plan.shape()[:2] == (64, sms * min(limit, 8 if math == "f64" else 9))
    plan.close()


def test_autotuner_starts_from_the_plans_shape(table):
    """42 KB of tables: a plan takes 3 blocks of 192, which the tuner times first"""
    g = m.Geometry(_blocks(7, (4, 5, 4), 4), 0.05, 0.05, 0.05)
    props = _many_sets(180)
    jobs = [m.Job(0, k, 40, 100 + k, "uniform") for k in range(180)]
    plan = m.Plan([g], props, jobs, table=table)
    block, grid, _ = plan.shape()
    plan.close()
    first = autotune.tune([g], props, jobs, table=table, use_cache=False)["table"][0]
    assert (first["block"], first["grid"]) == (block, grid) and block == 192


@pytest.mark.parametrize("shape", [(5, 7, 1), (5, 1, 7), (9, 6, 2), (9, 2, 6), (4, 5, 3), (1, 2, 1),
                                   (66, 3, 3)])
def test_narrow_grids(table, shape):
    """Grids whose voxels all lie on a lateral face, and the narrowest others: maps by
    definition, and merged steps as steps at every face (the tissues differ in index)."""
    t = np.random.default_rng(sum(shape)).integers(1, 4, shape).astype(np.uint8)
    t[shape[0] // 2:] = 1
    assert np.array_equal(m.safe_distance(t), safe_distance_bruteforce(t))
    p = m.OpticalProps.from_tissues([(0.5, 9.0, 0.9, 1.4), (1.0, 5.0, 0.7, 1.33),
                                     (0.8, 20.0, 0.8, 1.5)])
    a, b = (m.run([m.Geometry(t, 0.1, 0.12, 0.09)], [p], [m.Job(0, 0, 400, 3, "uniform")],
                  table=table, photon_log=True, steps=steps)[0] for steps in ("merged", "voxel"))
    if min(shape[1:]) <= 2:
        _same(a, b)
    assert residual(a.totals) == 0


def test_narrow_grid_needs_no_padded_maps():
    """One voxel wide, three tissues of two indices: cells and grid fit where maps of four
    bytes a voxel would not."""
    out = _in_fresh_process(_PLAN + """
n = 16384
t = np.ones((n - 63, n, 1), np.uint8)
t[100:200] = 2
t[200:300] = 3
g = m.Geometry(t, 0.1, 0.1, 0.1)
p = m.OpticalProps.from_tissues([(1.0, 9.0, 0.9, 1.4), (1.0, 5.0, 0.7, 1.4), (1.0, 5.0, 0.7, 1.3)])
m.run([m.Geometry(t[:2, :2], 1, 1, 1)], [p], [m.Job(0, 0, 10, 7)])
hold = fill(7 * n * n + 200 * MiB)
plan = m.Plan([g], [p], [m.Job(0, 0, 1000, 7, "uniform")])
plan.execute()
print(plan.read()[0].photons)
""")
    assert int(out) == 1000


# The absorption map changes no photon, nor does a second geometry in the launch: with one
# exception.  The fast merged kernel that maps one geometry's absorption rounds the square
# of the scattering cosine by itself, so a seeded run has tallies of its own there.
@pytest.mark.parametrize("math,steps", MODES)
def test_photons_with_and_without_the_map(table, math, steps):
    g = m.Geometry(_blocks(11, (4, 5, 4), 3), 0.07, 0.07, 0.07)
    other = m.Geometry(_blocks(12, (3, 3, 3), 3), 0.05, 0.06, 0.07)
    p = m.OpticalProps.from_tissues([(0.3, 9.0, 0.9, 1.4), (0.5, 15.0, 0.7, 1.33),
                                     (0.1, 6.0, 0.8, 1.4)])
    job = m.Job(0, 0, 4000, 17, "uniform")
    beside = m.Job(1, 0, 500, 18, "pencil")
    kw = dict(table=table, math=math, steps=steps, photon_log=True)
    off = m.run([g], [p], [job], **kw)[0]
    on = m.run([g], [p], [job], absorption_map=True, **kw)[0]
    _same(off, m.run([g, other], [p], [job, beside], **kw)[0])
    batched = m.run([g, other], [p], [job, beside], absorption_map=True, **kw)[0]
    _same(off, batched)
    assert int(on.absorption.sum()) == on.totals["absorbed"] and residual(on.totals) == 0
    if (math, steps) == ("fast", "merged"):
        assert on.totals["steps"] != off.totals["steps"]
        assert abs(total_z(on.totals, off.totals)) < 5
        _same(on, m.run([g], [p], [job], absorption_map=True, block=64, **kw)[0])
    else:
        _same(on, off)
        assert np.array_equal(on.absorption, batched.absorption)
