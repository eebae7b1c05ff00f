"""The autotuner's cache key and its choice, without a GPU."""
from __future__ import annotations

from ymc3d_b200 import autotune


def _result(block, blocks, ms):
    return {"block": block, "blocks_per_sm": 0, "grid": 148 * blocks, "ms": ms}


def test_key_knows_the_build_and_the_candidates(engine, tmp_path, monkeypatch):
    key = autotune.cache_key("B200", "sig")
    assert key == autotune.cache_key("B200", "sig", list(autotune.CANDIDATES))
    assert key != autotune.cache_key("B200", "sig", autotune.CANDIDATES[:-1])
    assert key != autotune.cache_key("B200", "other")
    other = tmp_path / "libmc3d.so"
    other.write_bytes(engine.LIB_PATH.read_bytes()[:-1] + b"x")
    assert autotune._build_id(other) != autotune._build_id(engine.LIB_PATH)
    monkeypatch.setattr(autotune, "_build_id", lambda: "another build")
    assert key != autotune.cache_key("B200", "sig")


def test_fewer_threads_win_by_more_than_two_per_cent():
    first = _result(128, 5, 100.0)
    assert autotune.choose([first, _result(128, 4, 98.5)]) is first
    fewer = _result(128, 3, 97.0)
    assert autotune.choose([first, fewer]) is fewer
    assert autotune.choose([first, _result(256, 2, 98.5)]) is first


def test_more_threads_win_by_any_margin():
    """large optical tables: 128 threads hold 12 warps an SM, 256 hold 16"""
    few, many = _result(128, 3, 100.0), _result(256, 2, 99.5)
    assert autotune.choose([few, many]) is many
