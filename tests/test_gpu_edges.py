"""Inputs and launches at the edges of what a call accepts: lanes without a stream,
coefficients below the normal range, photons without a position, memory and tables at
their limits."""
from __future__ import annotations

import numpy as np
import pytest

import ymc3d_b200 as m
from helpers import residual

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
