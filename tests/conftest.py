"""Test configuration: import paths, the `gpu` marker and fixture helpers.

CPU tests (``-m "not gpu"``) check the oracle against the golden fixtures,
the host-side geometry front-end of the C-ABI library and the Python
wrappers' argument handling; GPU tests (``-m gpu``) check the CUDA path
against the oracle and the fixtures.
"""
import os
import sys

import numpy as np
import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
PKG = os.path.join(ROOT, "ccpi-reconstruction_b200")
for p in (PKG, os.path.join(ROOT, "oracle"), ROOT):
    if p not in sys.path:
        sys.path.insert(0, p)

GOLDEN = os.path.join(ROOT, "tests", "golden")


def pytest_configure(config):
    config.addinivalue_line("markers", "gpu: needs a CUDA GPU (B200)")


@pytest.hookimpl(hookwrapper=True)
def pytest_runtest_call(item):
    """A test that comes to a call of the reference's own build where that
    build is absent is skipped, not failed."""
    outcome = yield
    from oracle import ReferenceMissing
    if outcome.excinfo is not None and issubclass(outcome.excinfo[0], ReferenceMissing):
        outcome.force_exception(pytest.skip.Exception("the reference library is not built"))


def golden(name):
    with np.load(os.path.join(GOLDEN, name + ".npz")) as z:
        return {k: z[k] for k in z.files}


def golden_names(prefix):
    return sorted(f[:-4] for f in os.listdir(GOLDEN) if f.startswith(prefix) and f.endswith(".npz"))


def have_gpu():
    try:
        import torch
        return torch.cuda.is_available()
    except Exception:
        return False


@pytest.fixture(scope="session")
def cuda():
    if not have_gpu():
        pytest.skip("no CUDA device")
    import torch
    return torch.device("cuda:0")


def max_rel(a, b):
    a = np.asarray(a, np.float64)
    b = np.asarray(b, np.float64)
    m = np.abs(b).max()
    return float(np.abs(a - b).max() / (m if m > 0 else 1.0))


def rel_l2(a, b):
    a = np.asarray(a, np.float64)
    b = np.asarray(b, np.float64)
    n = np.linalg.norm(b)
    return float(np.linalg.norm(a - b) / (n if n > 0 else 1.0))
