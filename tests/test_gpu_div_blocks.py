"""B u and B^T p from stored element blocks (small one-rank boxes): every entry point
against the oracle where the set-up's element groups and the blocks of the factors
end, and the last box of that route and the first of the next."""
import numpy as np
import pytest

from conftest import relerr
from pt_b200 import mesh as M

pytestmark = pytest.mark.gpu

TOL64 = 1e-12  # the project's parity bar for FP64 operators


@pytest.mark.parametrize("workload", ["box:1,1,1", "box:2,1,1", "box:3,1,1", "box:5,1,1", "box:31,1,1", "box:2,16,1",
                                      "box:3,11,1", "box:7,5,3", "box:8,8,8", "box:50,50,50", "box:51,50,50"])
def test_b_and_bt_match_oracle(ora, workload):
    import torch

    from pt_b200 import MatStokesMF
    m, eta, mask = M.problem(workload, seed=3)
    u, p = M.uniform_vec(m.nvel, 4), M.uniform_vec(m.npres, 5)
    ud, pd = torch.from_numpy(u).cuda(), torch.from_numpy(p).cuda()
    with MatStokesMF(*m.dims) as op:
        op.SetUp(np.roll(m.coords, 3), eta, mask)  # other coordinates first: the blocks follow them
        op.MFStokesWrapper_A21(ud)
        op.set_coords(m.coords)
        assert relerr(op.MFStokesWrapper_A21(ud).cpu(), ora.a21(m.dims, m.coords, u)) < TOL64
        assert relerr(op.MatMult_MFStokes_A21(ud).cpu(), ora.matmult_a21(m.dims, m.coords, mask, u)) < TOL64
        assert relerr(op.MFStokesWrapper_A12(pd).cpu(), ora.a12(m.dims, m.coords, p)) < TOL64
        y = op.MatMult_MFStokes_A12(pd).cpu().numpy()
        assert relerr(y, ora.matmult_a12(m.dims, m.coords, mask, p)) < TOL64
        assert not y[mask.astype(bool)].any()
        op.set_a11_op("b200_colour")  # the whole operator block by block: B^T p added to A11 u
        yu, yp = op.MFStokesWrapper_A(ud, pd)
        assert relerr(yu.cpu(), ora.a11(m.dims, m.coords, eta, u) + ora.a12(m.dims, m.coords, p)) < TOL64
        assert relerr(yp.cpu(), ora.a21(m.dims, m.coords, u)) < TOL64


@pytest.mark.parametrize("workload", ["box:1,1,1", "box:8,8,8", "box:9,8,8", "box:13,13,12"])
def test_whole_operator_matches_oracle(ora, workload):
    """Block by block up to 512 elements, in one pass above."""
    import torch

    from pt_b200 import MatStokesMF
    m, eta, mask = M.problem(workload, seed=3)
    u, p = M.uniform_vec(m.nvel, 4), M.uniform_vec(m.npres, 5)
    ud, pd = torch.from_numpy(u).cuda(), torch.from_numpy(p).cuda()
    bc = mask.astype(bool)
    with MatStokesMF(*m.dims) as op:
        op.SetUp(m.coords, eta, mask)
        yu, yp = (y.cpu().numpy() for y in op.MFStokesWrapper_A(ud, pd))
        assert relerr(yu, ora.a11(m.dims, m.coords, eta, u) + ora.a12(m.dims, m.coords, p)) < TOL64
        assert relerr(yp, ora.a21(m.dims, m.coords, u)) < TOL64
        yu, yp = (y.cpu().numpy() for y in op.MatMult_MFStokes_A(ud, pd))
        ref = ora.matmult_a11(m.dims, m.coords, eta, mask, u) + ora.matmult_a12(m.dims, m.coords, mask, p)
        assert relerr(yu, ref) < TOL64 and np.array_equal(yu[bc], u[bc])
        assert relerr(yp, ora.matmult_a21(m.dims, m.coords, mask, u)) < TOL64
        pa = pd.clone()  # one vector as xp and yp
        yb, ya = op.MatMult_MFStokes_A(ud, pa, None, pa)
        assert np.array_equal(yb.cpu(), yu) and np.array_equal(ya.cpu(), yp)
