"""Calls that run without the memory of the faster routes: with the device nearly full
the operator falls back on kernels that need no more than K."""
import numpy as np
import pytest

from conftest import relerr
from pt_b200 import mesh as M

pytestmark = pytest.mark.gpu

TOL64 = 1e-12  # the project's parity bar for FP64 operators
TOL32 = 5e-5   # and for the FP32 apply
MB = 1 << 20


def _calls(op, u, p):
    import torch
    out = [op.MatMult_MFStokes_A11(u), op.MFStokesWrapper_A11(u), op.MatMult_MFStokes_A11(u.float()).double(),
           op.MatGetDiagonal_MFStokes_A11(torch.empty_like(u)), op.MatMult_MFStokes_A12(p), op.MatMult_MFStokes_A21(u),
           *op.MatMult_MFStokes_A(u, p), op.FormFunctionLocal_U(u, p)]
    return [o.cpu().numpy() for o in out]


def _load_colour_kernels(m, eta, u, p):
    """The colour kernels' local memory (1.4 GB for the whole device) is the driver's
    and is taken at their first launch: here, in the forms that run without factors."""
    import torch

    from pt_b200 import MatStokesMF
    with MatStokesMF(*m.dims, a11_op="b200_colour") as op:
        op.SetUp(m.coords, eta, None)
        op.MatMult_MFStokes_A11(u)
        op.MatGetDiagonal_MFStokes_A11(torch.empty_like(u))
        yu, yp = torch.empty_like(u), torch.empty_like(p)
        st = torch.cuda.Stream()
        op.set_stream(st)
        g = torch.cuda.CUDAGraph()
        with torch.cuda.graph(g, stream=st):
            op.MFStokesWrapper_A12(p, yu)
            op.MFStokesWrapper_A21(u, yp)
        g.replay()
        torch.cuda.synchronize()


# room beside K: none for B's factors; none for the tiles' sums either
@pytest.mark.parametrize("beside_k", [130 * MB, 22 * MB])
def test_calls_with_the_device_nearly_full(beside_k):
    import torch

    from pt_b200 import MatStokesMF
    dims = (40, 40, 40)
    k_bytes, b_bytes, sums = 64000 * 243 * 12, 64000 * 324 * 8, 500 * 57 * 1024
    assert beside_k < b_bytes and (beside_k < sums or beside_k > sums + 64000 * 108 * 8)
    m, eta, mask = M.problem("box:%d,%d,%d" % dims, seed=4)
    u, p = (torch.from_numpy(M.uniform_vec(n, 3)).cuda() for n in (m.nvel, m.npres))
    fu = torch.from_numpy(M.uniform_vec(81 * m.nel, 7)).cuda()
    with MatStokesMF(*dims) as op:
        op.SetUp(m.coords, eta, mask)
        op.set_body_force(fu)
        want = _calls(op, u, p)
    _load_colour_kernels(m, eta, u, p)
    torch.empty(1600 * MB, dtype=torch.uint8, device="cuda")  # stays in torch's cache, for the calls' outputs
    with MatStokesMF(*dims) as op:
        op.SetUp(m.coords, eta, mask)
        op.set_body_force(fu)
        torch.cuda.synchronize()
        free, _ = torch.cuda.mem_get_info()
        hog = torch.empty(free - k_bytes - beside_k, dtype=torch.uint8, device="cuda")
        try:
            got = _calls(op, u, p)
        finally:
            del hog
            torch.cuda.empty_cache()
    for i, (g, w) in enumerate(zip(got, want)):
        assert relerr(g, w) < (TOL32 if i == 2 else TOL64), i



@pytest.mark.parametrize("fp32", [False, True])
def test_batch_with_no_room_for_the_sums(fp32):
    import torch

    from pt_b200 import MatStokesMF
    from pt_b200.batch import BatchA11
    m, eta, mask = M.problem("box:40,40,40", seed=4)
    u = torch.from_numpy(M.uniform_vec(m.nvel, 3)).cuda()
    u = u.float() if fp32 else u
    torch.empty(600 * MB, dtype=torch.uint8, device="cuda")  # stays in torch's cache
    with MatStokesMF(40, 40, 40) as op, MatStokesMF(9, 8, 7) as small:
        s, eta_s, _ = M.problem("box:9,8,7", seed=5)
        small.SetUp(s.coords, eta_s, None)
        small.MatMult_MFStokes_A11(M.uniform_vec(s.nvel, 6))
        with BatchA11([small], lz=2) as b:  # the streaming batch kernels are loaded
            v = torch.ones(s.nvel, dtype=u.dtype, device="cuda")
            b.apply([v], [torch.empty_like(v)])
        op.SetUp(m.coords, eta, mask)
        want = op.MatMult_MFStokes_A11(u)
        torch.cuda.synchronize()
        free, _ = torch.cuda.mem_get_info()
        hog = torch.empty(free - 18 * MB, dtype=torch.uint8, device="cuda")  # the sums take 29 MB
        try:
            y = torch.empty_like(u)
            with BatchA11([op]) as b:
                b.apply([u], [y])
                torch.cuda.synchronize()
        finally:
            del hog
            torch.cuda.empty_cache()
    assert relerr(y.double().cpu(), want.double().cpu()) < (TOL32 if fp32 else TOL64)


def test_a_failed_call_does_not_fail_the_next_one(ora):
    from pt_b200 import MatStokesMF, _capi
    m, eta, mask = M.problem("box:5,4,3", seed=5)
    x = M.uniform_vec(m.nvel, 6)
    with MatStokesMF(*m.dims) as op:
        with pytest.raises(_capi.PtError):
            MatStokesMF(2, 2, 2, node_box=(8000, 8000, 8000, 0, 0, 0))  # 12 TB of coordinates
        op.SetUp(m.coords, eta, mask)
        assert relerr(op.MatMult_MFStokes_A11(x), ora.matmult_a11(m.dims, m.coords, eta, mask, x)) < TOL64
