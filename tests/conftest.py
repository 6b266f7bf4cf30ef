"""Shared test setup: import paths, the `gpu` marker, common helpers."""
from __future__ import annotations

import os
import sys
from pathlib import Path

import numpy as np
import pytest

ROOT = Path(__file__).resolve().parents[1]
sys.path.insert(0, str(ROOT / "edegpredict-engine-rotary_b200"))
sys.path.insert(0, str(ROOT))


def pytest_configure(config):
    config.addinivalue_line("markers", "gpu: needs a CUDA GPU (B200) and runs the CUDA path")


def _skip_without_reference(e: Exception) -> None:
    from oracle.oracle import ReferenceMissing

    if isinstance(e, ReferenceMissing) and not os.environ.get("MPM_REFERENCE_SRC"):
        pytest.skip(str(e))


# A test that runs the reference's own kernels is skipped where neither they
# nor the sources to build them from are present (MPM_REFERENCE_SRC); with the
# sources named, a missing build is a failure.
@pytest.hookimpl(wrapper=True)
def pytest_runtest_setup(item):
    try:
        return (yield)
    except Exception as e:
        _skip_without_reference(e)
        raise


@pytest.hookimpl(wrapper=True)
def pytest_runtest_call(item):
    try:
        return (yield)
    except Exception as e:
        _skip_without_reference(e)
        raise


def has_gpu() -> bool:
    try:
        import torch

        return torch.cuda.is_available()
    except Exception:
        return False


def max_rel(a, b, scale=None) -> float:
    """max |a - b| / scale, scale = max |b| unless given."""
    a = np.asarray(a, dtype=np.float64)
    b = np.asarray(b, dtype=np.float64)
    if a.size == 0:
        return 0.0
    s = float(np.abs(b).max()) if scale is None else float(scale)
    return float(np.abs(a - b).max() / max(s, 1e-300))


@pytest.fixture(scope="session")
def oracle():
    from oracle.oracle import Oracle

    return Oracle()
