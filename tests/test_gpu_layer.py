"""Layer tiles ("b200_layer"): the A11 apply and the diagonal on single-layer
tiles with a gather, against the oracle at the shapes where a tile can go
wrong (rows that do not divide a tile, tiles that cross layers, one and
several x-tiles, single rows), in both precisions, with and without Dirichlet
dofs, on ghosted boxes, batched, and through the pinned-host pipeline."""
import numpy as np
import pytest

from conftest import relerr
from pt_b200 import mesh as M

pytestmark = pytest.mark.gpu

TOL64 = 1e-12  # the project's parity bar for FP64 operators
TOL32 = 5e-5   # and for the FP32 apply

SHAPES = ["box:1,1,1", "box:2,1,3", "box:3,2,4", "box:8,8,8", "box:31,3,5", "box:32,4,2", "box:33,5,2", "box:41,7,5",
          "box:64,3,3", "box:97,3,2", "box:128,2,3", "box:129,3,2", "box:257,1,2", "box:2,40,3"]


def _op(m, eta, mask, a11_op="b200_layer"):
    from pt_b200 import MatStokesMF
    return MatStokesMF(*m.dims, a11_op=a11_op).SetUp(m.coords, eta, mask)


@pytest.mark.parametrize("workload", SHAPES)
def test_layer_tiles_match_oracle(ora, workload):
    import torch
    m, eta, mask = M.problem(workload, seed=15)
    x = M.uniform_vec(m.nvel, 16)
    xd = torch.from_numpy(x).cuda()
    with _op(m, eta, mask) as op:
        assert op.a11_op == "b200_layer"
        y = op.MatMult_MFStokes_A11(xd).cpu().numpy()
        assert relerr(y, ora.matmult_a11(m.dims, m.coords, eta, mask, x)) < TOL64
        assert np.array_equal(y[mask.astype(bool)], x[mask.astype(bool)])
        assert np.array_equal(op.MatMult_MFStokes_A11(xd).cpu().numpy(), y)
        assert relerr(op.MFStokesWrapper_A11(x), ora.a11(m.dims, m.coords, eta, x)) < TOL64
        assert relerr(op.MatGetDiagonal_MFStokes_A11(), ora.getdiag_a11(m.dims, m.coords, eta, mask)) < TOL64
        assert relerr(op.MFStokesWrapper_diagA11(), ora.diag(m.dims, m.coords, eta)) < TOL64
        y32 = op.MatMult_MFStokes_A11(xd.float()).double().cpu().numpy()
        assert relerr(y32, ora.matmult_a11(m.dims, m.coords, eta, mask, x)) < TOL32


def test_layer_tiles_on_a_ghosted_box(ora):
    """Nodes outside the element box are written as zeros, Dirichlet dofs there are copied."""
    import torch

    from pt_b200 import MatStokesMF
    sub, off, nb = (37, 4, 3), (2, 0, 1), (37 * 2 + 1 + 4, 4 * 2 + 1 + 2, 3 * 2 + 1 + 3)
    rng = np.random.default_rng(5)
    sl = tuple(slice(o, o + 2 * n + 1) for o, n in zip(off[::-1], sub[::-1]))
    m, eta, _ = M.problem("box:%d,%d,%d" % sub, seed=6)
    cg = rng.uniform(size=(nb[2], nb[1], nb[0], 3))
    cg[sl] = m.coords.reshape(cg[sl].shape)
    u = rng.uniform(-1, 1, size=cg.shape)
    mask = rng.uniform(size=cg.shape) < 0.1
    uz = np.where(mask, 0.0, u)
    ref = np.zeros_like(u)
    ref[sl] = ora.a11(sub, m.coords, eta, np.ascontiguousarray(uz[sl].reshape(-1))).reshape(ref[sl].shape)
    ref[mask] = u[mask]
    dref = np.zeros_like(u)
    dref[sl] = ora.diag(sub, m.coords, eta).reshape(dref[sl].shape)
    dref[mask] = 1.0
    with MatStokesMF(*sub, a11_op="b200_layer", node_box=(*nb, *off)) as op:
        op.SetUp(np.ascontiguousarray(cg.reshape(-1)), eta, mask.astype(np.uint8).reshape(-1))
        y = op.MatMult_MFStokes_A11(torch.from_numpy(u.reshape(-1)).cuda()).cpu().numpy()
        assert relerr(y, ref.reshape(-1)) < TOL64
        assert np.array_equal(y[mask.reshape(-1)], u[mask])
        assert relerr(op.MatGetDiagonal_MFStokes_A11(), dref.reshape(-1)) < TOL64


@pytest.mark.parametrize("fp32", [False, True])
def test_batch_of_layer_boxes_is_bitwise_each_boxs_own_apply(fp32):
    """Boxes on layer tiles, one without a mask, next to a box on coloured tiles."""
    import torch

    from pt_b200.batch import BatchA11
    ops, us = [], []
    for i, (dims, kind) in enumerate([((12, 11, 10), "b200_layer"), ((41, 5, 6), "b200_layer"), ((9, 4, 3), "b200_layer"),
                                      ((40, 5, 7), "b200_stream")]):
        m = M.make_mesh(*dims, perturb=0.05, seed=i)
        ops.append(_op(m, M.eta_per_element(m, 1e4, seed=i), None if i == 2 else M.bc_mask_freeslip(*dims), kind))
        u = torch.from_numpy(M.uniform_vec(m.nvel, 70 + i)).cuda()
        us.append(u.float() if fp32 else u)
    for masked in (True, False):
        ys = [torch.full_like(u, float("nan")) for u in us]
        with BatchA11(ops) as b:
            b.apply(us, ys, masked=masked)
            torch.cuda.synchronize()
        for op, u, y in zip(ops, us, ys):
            assert torch.equal(y, op.MatMult_MFStokes_A11(u) if masked else op.MFStokesWrapper_A11(u))
    for op in ops:
        op.Destroy()


@pytest.mark.parametrize("workload", ["box:24,10,30", "box:5,3,41", "box:50,2,13"])
def test_pinned_host_apply_of_layer_tiles_is_bitwise_the_device_apply(workload):
    import torch
    m, eta, mask = M.problem(workload, seed=23)
    x = torch.from_numpy(M.uniform_vec(m.nvel, 24))
    xp, yp = x.pin_memory(), torch.empty(m.nvel, dtype=torch.float64).pin_memory()
    with _op(m, eta, mask) as op:
        op.MatMult_MFStokes_A11(xp.numpy(), yp.numpy())
        assert np.array_equal(yp.numpy(), op.MatMult_MFStokes_A11(x.cuda()).cpu().numpy())
        op.MFStokesWrapper_A11(xp.numpy(), yp.numpy())
        assert np.array_equal(yp.numpy(), op.MFStokesWrapper_A11(x.cuda()).cpu().numpy())


@pytest.mark.parametrize("workload", SHAPES)
def test_divergence_and_gradient_match_oracle(ora, workload):
    """B u and B^T p from the Gauss-point factors, MatShell and SpMVOp level,
    before any viscosity is set, into a pressure vector of odd alignment too."""
    import torch

    from pt_b200 import MatStokesMF
    m, _, mask = M.problem(workload, seed=17)
    u, p = M.uniform_vec(m.nvel, 18), M.uniform_vec(m.npres, 19)
    with MatStokesMF(*m.dims) as op:
        op.set_coords(m.coords)
        op.set_bc_mask(mask)
        ud, buf = torch.from_numpy(u).cuda(), torch.empty(m.npres + 1, dtype=torch.float64, device="cuda")
        for yp in (buf[:-1], buf[1:]):
            assert relerr(op.MatMult_MFStokes_A21(ud, yp).cpu().numpy(), ora.matmult_a21(m.dims, m.coords, mask, u)) < TOL64
        assert relerr(op.MFStokesWrapper_A21(u), ora.a21(m.dims, m.coords, u)) < TOL64
        assert relerr(op.MatMult_MFStokes_A12(p), ora.matmult_a12(m.dims, m.coords, mask, p)) < TOL64
        assert relerr(op.MFStokesWrapper_A12(p), ora.a12(m.dims, m.coords, p)) < TOL64


@pytest.mark.parametrize("workload", SHAPES)
def test_whole_operator_matches_oracle_and_follows_its_coefficients(ora, workload):
    """A11 and the pressure blocks in one pass, MatShell and SpMVOp level and
    the residual; new viscosity and new coordinates reach its factors."""
    import torch

    from pt_b200 import MatStokesMF
    m, eta, mask = M.problem(workload, seed=27)
    m2 = M.make_mesh(*m.dims, perturb=0.05, seed=28)
    eta2 = 1.0 + eta[::-1].copy()
    u, p, fu = M.uniform_vec(m.nvel, 29), M.uniform_vec(m.npres, 30), M.uniform_vec(81 * m.nel, 31)
    ud, pd = torch.from_numpy(u).cuda(), torch.from_numpy(p).cuda()
    with MatStokesMF(*m.dims) as op:
        op.SetUp(m.coords, eta, mask)
        op.set_body_force(fu)
        for c, e in ((m.coords, eta), (m.coords, eta2), (m2.coords, eta2)):
            op.set_coords(c)
            op.set_eta(e)
            yu, yp = op.MatMult_MFStokes_A(ud, pd)
            ru, rp = ora.matmult_a(m.dims, c, e, mask, u, p)
            assert relerr(yu.cpu().numpy(), ru) < TOL64 and relerr(yp.cpu().numpy(), rp) < TOL64
            yu, yp = op.MFStokesWrapper_A(ud, pd)
            a = ora.a11(m.dims, c, e, u) + ora.a12(m.dims, c, p)
            assert relerr(yu.cpu().numpy(), a) < TOL64 and relerr(yp.cpu().numpy(), ora.a21(m.dims, c, u)) < TOL64
            assert relerr(op.FormFunctionLocal_U(ud, pd).cpu().numpy(), ora.residual_u(m.dims, c, e, fu, u, p)) < TOL64


def test_whole_operator_on_a_ghosted_box_is_the_sum_of_its_blocks():
    import torch

    from pt_b200 import MatStokesMF
    sub, off, nb = (37, 4, 3), (2, 0, 1), (37 * 2 + 1 + 4, 4 * 2 + 1 + 2, 3 * 2 + 1 + 3)
    rng = np.random.default_rng(7)
    m, eta, _ = M.problem("box:%d,%d,%d" % sub, seed=8)
    sl = tuple(slice(o, o + 2 * n + 1) for o, n in zip(off[::-1], sub[::-1]))
    cg = rng.uniform(size=(nb[2], nb[1], nb[0], 3))
    cg[sl] = m.coords.reshape(cg[sl].shape)
    mask = (rng.uniform(size=cg.size) < 0.1).astype(np.uint8)
    u = torch.from_numpy(rng.uniform(-1, 1, size=cg.size)).cuda()
    p = torch.from_numpy(rng.uniform(-1, 1, size=4 * m.nel)).cuda()
    with MatStokesMF(*sub, node_box=(*nb, *off)) as op:
        op.SetUp(np.ascontiguousarray(cg.reshape(-1)), eta, mask)
        yu, yp = op.MFStokesWrapper_A(u, p)
        ref = op.MFStokesWrapper_A11(u) + op.MFStokesWrapper_A12(p)
        assert float((yu - ref).abs().max()) < 1e-13 * float(ref.abs().max())
        rp = op.MFStokesWrapper_A21(u)
        assert float((yp - rp).abs().max()) < 1e-13 * float(rp.abs().max())
        yu, yp = op.MatMult_MFStokes_A(u, p)
        bc = torch.from_numpy(mask != 0).cuda()
        ref = torch.where(bc, u, op.MatMult_MFStokes_A11(u) + op.MFStokesWrapper_A12(p))
        assert float((yu - ref).abs().max()) < 1e-13 * float(ref.abs().max())
        assert torch.equal(yu[bc], u[bc])


@pytest.mark.parametrize("dims,counts", [((1, 1, 1), (3, 3)), ((2, 1, 3), (1, 1)), ((33, 5, 2), (1, 9)), ((129, 1, 2), (2, 5))])
def test_marker_projection_with_uneven_counts_matches_oracle(ora, dims, counts):
    """Elements of different marker counts (around the loop's load-ahead), a last
    block that is not full, viscosity only or density too, installed or not."""
    import torch

    from pt_b200 import MatStokesMF
    m, eta, _ = M.problem("box:%d,%d,%d" % dims, seed=3)
    rng = np.random.default_rng(4)
    wil = np.repeat(np.arange(m.nel, dtype=np.int32), rng.integers(counts[0], counts[1] + 1, size=m.nel))
    wil = rng.permutation(wil).astype(np.int32)
    xi = rng.uniform(-1, 1, size=(len(wil), 3))
    e, r = 10.0 ** rng.uniform(-3, 3, size=len(wil)), rng.uniform(1, 2, size=len(wil))
    ref_e, ref_r = ora.marker_project(m.dims, wil, xi, e, r)
    t = lambda a: torch.from_numpy(np.ascontiguousarray(a)).cuda()
    u = M.uniform_vec(m.nvel, 5)
    with MatStokesMF(*m.dims) as op:
        op.SetUp(m.coords, eta)
        before = op.MFStokesWrapper_A11(u)
        for install in (False, True):
            eq, rq = op.ProjectMarkers(t(wil), t(xi), t(e), t(r), install=install)
            assert relerr(eq.cpu().numpy(), ref_e) < TOL64 and relerr(rq.cpu().numpy(), ref_r) < TOL64
            y = op.MFStokesWrapper_A11(u)
            if not install:
                assert np.array_equal(y, before)
            else:
                assert relerr(y, ora.a11(m.dims, m.coords, ref_e, u)) < TOL64
