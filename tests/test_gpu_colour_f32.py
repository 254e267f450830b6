"""The FP32 apply of the 8-colour kernel: its copies of coordinates and viscosity are
made when those are set, not in the apply, and follow them."""
import numpy as np
import pytest

from conftest import relerr
from pt_b200 import mesh as M

pytestmark = pytest.mark.gpu

TOL32 = 5e-5  # the project's bar for the FP32 apply


def _problem(seed):
    m, eta, mask = M.problem("box:7,6,5", seed=seed)
    return m, eta, mask


@pytest.mark.parametrize("route", ["by name", "late", "not positive"])
def test_fp32_colour_apply_converts_nothing(ora, route):
    import torch

    from pt_b200 import MatStokesMF
    m, eta, mask = _problem(3)
    m2, eta2, _ = _problem(4)
    if route == "not positive":  # the tile kernels do not take it
        eta[40] = eta2[41] = 0.0
    x = M.uniform_vec(m.nvel, 5)
    x32 = torch.from_numpy(x).cuda().float()
    with MatStokesMF(*m.dims, a11_op="b200_colour" if route == "by name" else "b200_layer") as op:
        op.SetUp(m.coords, eta, mask)
        if route == "late":
            op.MatMult_MFStokes_A11(x32)
            op.set_a11_op("b200_colour")
        y = torch.empty_like(x32)
        for c, e in ((m.coords, eta), (m.coords, eta2), (m2.coords, eta2)):
            op.set_coords(c)
            op.set_eta(e)
            op.MatMult_MFStokes_A11(x32, y)
            assert relerr(y.double().cpu(), ora.matmult_a11(m.dims, c, e, mask, x)) < TOL32
            n = op.launch_count()
            op.MatMult_MFStokes_A11(x32, y)
            n32, n = op.launch_count() - n, op.launch_count()
            op.MatMult_MFStokes_A11(x32.double())
            assert n32 == op.launch_count() - n  # as many launches as in FP64: no conversions
