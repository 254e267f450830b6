"""Where the reference is absent its tests skip, so that a run with -x goes on."""
import os
import subprocess
import sys

import pytest

from conftest import REPO


@pytest.mark.parametrize("path", ["tests/test_gpu_residual.py::test_residual_at_64cubed", "tests/test_gpu_scale_parity.py::test_c1_a11_matmult",
                                  "tests/test_gpu_shim.py::test_plugin_matches_reference"])
def test_reference_tests_skip_without_the_reference(path):
    import oracle
    if oracle.reference_tree() or os.path.exists(os.path.join(REPO, "oracle", "_ref")):
        pytest.skip("the reference is at hand")
    r = subprocess.run([sys.executable, "-m", "pytest", path, "-q", "-x", "-m", "gpu", "-p", "no:cacheprovider"],
                       cwd=REPO, capture_output=True, text=True, timeout=600)
    last = r.stdout.strip().splitlines()[-1]
    assert r.returncode == 0 and "skipped" in last and "error" not in last, r.stdout[-2000:]
