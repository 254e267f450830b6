"""Marker projection with elements that hold very many markers (they are summed eight
at a time by their lanes): counts at both sides of the lines of that route and at the
remainders of eight, in a small box and in one that fills the device."""
import numpy as np
import pytest

from conftest import relerr

pytestmark = pytest.mark.gpu

TOL64 = 1e-12  # the project's parity bar for FP64 operators


@pytest.mark.parametrize("dims,counts", [((3, 2, 4), [256, 257, 263, 264, 265, 1024, 2003, 255]),
                                         ((26, 26, 26), [257, 1023, 1024, 1025, 1031, 1032, 1033, 5000])])
def test_crowded_elements_match_oracle(ora, dims, counts):
    import torch

    from pt_b200 import MatStokesMF
    nel = dims[0] * dims[1] * dims[2]
    rng = np.random.default_rng(11)
    per = rng.integers(1, 6, size=nel)
    per[rng.permutation(nel)[:len(counts)]] = counts
    wil = rng.permutation(np.repeat(np.arange(nel), per)).astype(np.int32)
    n = wil.size
    xi, eta, rho = rng.uniform(-1, 1, size=3 * n), 10.0 ** rng.uniform(0, 4, size=n), rng.uniform(1, 2, size=n)
    want = ora.marker_project(dims, wil, xi, eta, rho)
    dev = [torch.from_numpy(a).cuda() for a in (wil, xi, eta, rho)]
    with MatStokesMF(*dims) as op:
        got = [g.cpu().numpy() for g in op.ProjectMarkers(*dev, install=False)]
    for g, w in zip(got, want):
        assert relerr(g, w) < TOL64
