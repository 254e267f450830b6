"""Shared test fixtures.  GPU tests are marked ``gpu``; everything else runs on CPU."""
import glob
import os
import sys

import numpy as np
import pytest

REPO = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
PKG_ROOT = os.path.join(REPO, "ptatin-gene_b200")
for p in (REPO, PKG_ROOT):
    if p not in sys.path:
        sys.path.insert(0, p)

GOLDEN_DIR = os.path.join(REPO, "tests", "golden")


def pytest_configure(config):
    config.addinivalue_line("markers", "gpu: needs a CUDA device (B200, sm_100a)")


def pytest_runtest_setup(item):
    """Tests against the reference's own operators are skipped, not errors, where
    neither its compiled library nor its sources are at hand."""
    import oracle
    for fixture, lib in (("ref", "libptref.so"), ("shim", "libshimtest.so")):
        if fixture in getattr(item, "fixturenames", ()) and not oracle.reference_tree() \
                and not os.path.exists(os.path.join(REPO, "oracle", "_ref", lib)):
            pytest.skip(f"oracle/_ref/{lib} is not built and the reference's sources are absent")


def golden_names():
    """Operator fixtures (inputs and the reference's A11/diag/B/B^T/A outputs)."""
    return sorted(os.path.basename(p)[:-4] for p in glob.glob(os.path.join(GOLDEN_DIR, "*.npz"))
                  if not os.path.basename(p).startswith(("markers_", "residual_")))


def residual_golden_names():
    """Momentum residual fixtures (FormFunctionLocal_U inputs and output)."""
    return sorted(os.path.basename(p)[:-4] for p in glob.glob(os.path.join(GOLDEN_DIR, "residual_*.npz")))


def marker_golden_names():
    """Marker -> Gauss-point projection fixtures."""
    return sorted(os.path.basename(p)[:-4] for p in glob.glob(os.path.join(GOLDEN_DIR, "markers_*.npz")))


def load_golden(name):
    with np.load(os.path.join(GOLDEN_DIR, name + ".npz")) as z:
        return {k: z[k] for k in z.files}


def relerr(a, b):
    """||a - b||_inf / ||b||_inf, the parity metric of this project."""
    a = np.asarray(a, dtype=np.float64)
    b = np.asarray(b, dtype=np.float64)
    return float(np.abs(a - b).max() / max(np.abs(b).max(), 1e-300))


@pytest.fixture(scope="session")
def ora():
    import oracle
    return oracle.Oracle()
