"""Shared fixtures.  GPU tests carry @pytest.mark.gpu; everything else runs on CPU."""
from __future__ import annotations

import sys
from pathlib import Path

import pytest

ROOT = Path(__file__).resolve().parents[1]
if str(ROOT) not in sys.path:
    sys.path.insert(0, str(ROOT))


def pytest_configure(config):
    config.addinivalue_line("markers", "gpu: needs a CUDA GPU (B200)")


@pytest.fixture(scope="session")
def engine():
    import ymc3d_b200
    from ymc3d_b200 import build
    build.build()
    ymc3d_b200.lib()
    return ymc3d_b200


@pytest.fixture(scope="session")
def orc():
    import oracle
    from oracle import build
    build.build()
    oracle.lib()
    return oracle


@pytest.fixture(scope="session")
def table(engine):
    return engine.default_table()


def has_gpu() -> bool:
    try:
        import torch
        return torch.cuda.is_available()
    except Exception:
        return False


def pytest_collection_modifyitems(items):
    """The tests against the reference's own build (oracle/_ref, which needs its checkout)
    fail where there is none.  They run last then, so that a run stopping at its first
    failure has run every other test."""
    if not (ROOT / "oracle" / "_ref").exists():
        needs = {"run_reference", "ref_rng"}
        items.sort(key=lambda item: not needs.isdisjoint(item.function.__code__.co_names))
