"""The default kernel ("b200") in each precision: every route of the rule is bitwise
the kernel of that name, alone and in a batch, and a kernel chosen by name is used in
both precisions."""
import numpy as np
import pytest

from conftest import relerr
from pt_b200 import mesh as M

pytestmark = pytest.mark.gpu

TOL32 = 5e-5  # the project's bar for the FP32 apply

# box, kernel of the FP64 and of the FP32 apply
ROUTES = [((60, 60, 60), "b200_layer", "b200_layer"), ((64, 64, 64), "b200_stream", "b200_layer"),
          ((122, 60, 60), "b200_layer", "b200_stream"), ((128, 64, 48), "b200_stream", "b200_stream")]


@pytest.fixture(scope="module", params=ROUTES, ids=lambda r: "x".join(map(str, r[0])))
def box(request):
    import torch

    from pt_b200 import MatStokesMF
    dims, k64, k32 = request.param
    m = M.make_mesh(*dims, perturb=0.05, seed=1)
    eta, mask = M.eta_per_element(m, contrast=1e4, seed=2), M.bc_mask_freeslip(*dims)
    with MatStokesMF(*dims) as op:
        op.SetUp(m.coords, eta, mask)
        yield m, eta, mask, torch.from_numpy(M.uniform_vec(m.nvel, 3)).cuda(), op, k64, k32


def _applies(op, u):
    import torch
    return [op.MatMult_MFStokes_A11(u, torch.empty_like(u)), op.MFStokesWrapper_A11(u, torch.empty_like(u))]


def test_default_route_is_the_named_kernel(box):
    import torch
    m, eta, mask, u, op, k64, k32 = box
    op.set_a11_op("b200")
    assert op.a11_op == k64
    got = [*_applies(op, u), *_applies(op, u.float())]
    for name in (k64, k32):
        op.set_a11_op(name)
        want = [*_applies(op, u), *_applies(op, u.float())]
        for i, (g, w) in enumerate(zip(got, want)):
            if name == (k64 if i < 2 else k32):
                assert torch.equal(g, w), (name, i)
    op.set_a11_op("b200")


def test_default_fp32_apply_matches_oracle(box, ora):
    m, eta, mask, u, op, k64, k32 = box
    op.set_a11_op("b200")
    y = op.MatMult_MFStokes_A11(u.float()).double().cpu().numpy()
    assert relerr(y, ora.matmult_a11(m.dims, m.coords, eta, mask, u.cpu().numpy())) < TOL32


@pytest.mark.parametrize("fp32", [False, True])
def test_batch_of_default_ops_is_bitwise_their_own_applies(box, fp32):
    import torch

    from pt_b200 import MatStokesMF
    from pt_b200.batch import BatchA11
    m, eta, mask, u, op, k64, k32 = box
    op.set_a11_op("b200")
    small = M.make_mesh(17, 17, 15, perturb=0.05, seed=4)
    with MatStokesMF(17, 17, 15) as other:
        other.SetUp(small.coords, M.eta_per_element(small, contrast=1e2, seed=5), M.bc_mask_freeslip(17, 17, 15))
        us = [u, torch.from_numpy(M.uniform_vec(small.nvel, 6)).cuda()]
        us = [v.float() for v in us] if fp32 else us
        for masked in (True, False):
            ys = [torch.full_like(v, float("nan")) for v in us]
            with BatchA11([op, other]) as b:
                b.apply(us, ys, masked=masked)
                torch.cuda.synchronize()
            for o, v, y in zip((op, other), us, ys):
                assert torch.equal(y, _applies(o, v)[0 if masked else 1])


def test_default_fp32_apply_on_a_ghosted_box(ora):
    """FP32 of a ghosted streaming box: zeros outside the element box, Dirichlet dofs
    there copied, the inside the oracle's."""
    import torch

    from pt_b200 import MatStokesMF
    dims, g = (64, 56, 60), 1
    m = M.make_mesh(*dims, perturb=0.05, seed=1)
    eta = M.eta_per_element(m, contrast=1e4, seed=2)
    nb = tuple(2 * d + 1 + 2 * g for d in dims)
    rng = np.random.default_rng(3)
    sl = tuple(slice(g, g + 2 * d + 1) for d in dims[::-1])
    c = rng.uniform(size=(nb[2], nb[1], nb[0], 3))
    c[sl] = m.coords.reshape(c[sl].shape)
    u = rng.uniform(-1, 1, size=c.shape)
    mask = rng.uniform(size=c.shape) < 0.05
    uz = np.where(mask, 0.0, u)
    ref = np.zeros_like(u)
    ref[sl] = ora.a11(dims, m.coords, eta, np.ascontiguousarray(uz[sl].reshape(-1))).reshape(ref[sl].shape)
    ref[mask] = u[mask]
    with MatStokesMF(*dims, node_box=(*nb, g, g, g)) as op:
        op.SetUp(np.ascontiguousarray(c.reshape(-1)), eta, np.ascontiguousarray(mask.reshape(-1)).astype(np.uint8))
        assert op.a11_op == "b200_stream"
        ud = torch.from_numpy(np.ascontiguousarray(u.reshape(-1))).cuda().float()
        y = op.MatMult_MFStokes_A11(ud).double().cpu().numpy()
        assert relerr(y, ref.reshape(-1)) < TOL32
        inside = np.zeros(c.shape, dtype=bool)
        inside[sl] = True
        assert not y.reshape(c.shape)[~inside & ~mask].any()


def test_fp32_alone_from_element_matrices(ora):
    """Between the two lines of the stored matrices FP32 applies use them, FP64 ones the
    layer tiles; graphs record the tiles, and both follow the viscosity."""
    import torch

    from pt_b200 import MatStokesMF
    dims = (16, 16, 16)
    m = M.make_mesh(*dims, perturb=0.05, seed=1)
    etas = [M.eta_per_element(m, contrast=1e3, seed=s) for s in (2, 3)]
    mask = M.bc_mask_freeslip(*dims)
    u = torch.from_numpy(M.uniform_vec(m.nvel, 3)).cuda()
    u32, y = u.float(), torch.empty(m.nvel, dtype=torch.float32, device="cuda")
    want = [ora.matmult_a11(m.dims, m.coords, e, mask, u.cpu().numpy()) for e in etas]

    def record(op):
        st = torch.cuda.Stream()
        op.set_stream(st)
        g = torch.cuda.CUDAGraph()
        with torch.cuda.graph(g, stream=st):
            op.MatMult_MFStokes_A11(u32, y)
        return g

    with MatStokesMF(*dims) as op, MatStokesMF(*dims) as named:
        op.SetUp(m.coords, etas[0], mask)
        assert op.a11_op == "b200_layer"
        op.MatMult_MFStokes_A11(u)
        graphs = [record(op)]  # FP32 has not run yet
        torch.cuda.synchronize()
        for name, dtype in (("b200_layer", torch.float64), ("b200_ebe", torch.float32)):
            named.set_a11_op(name)
            named.SetUp(m.coords, etas[0], mask)
            assert torch.equal(op.MatMult_MFStokes_A11(u.to(dtype)), named.MatMult_MFStokes_A11(u.to(dtype)))
        torch.cuda.synchronize()
        graphs.append(record(op))
        for e, w in zip(etas, want):
            op.set_eta(e)
            op.MatMult_MFStokes_A11(u)  # an FP64 apply renews what the graphs read
            for g in graphs:
                y.fill_(float("nan"))
                torch.cuda.synchronize()
                g.replay()
                torch.cuda.synchronize()
                assert relerr(y.double().cpu(), w) < TOL32
            y32 = op.MatMult_MFStokes_A11(u32)
            torch.cuda.synchronize()
            assert relerr(y32.double().cpu(), w) < TOL32
        op.set_a11_op("b200_ebe")  # FP64 from matrices too, from here on
        y64 = op.MatMult_MFStokes_A11(u)
        torch.cuda.synchronize()  # the op is on the capture's stream
        assert relerr(y64.cpu(), want[1]) < 1e-12
        assert relerr(op.MatGetDiagonal_MFStokes_A11(), ora.getdiag_a11(m.dims, m.coords, etas[1], mask)) < 1e-12
