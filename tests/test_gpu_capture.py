"""Applies recorded in CUDA graphs: first uses inside a capture, inputs that change
between replays, several graphs of one op."""
import numpy as np
import pytest

from conftest import relerr
from pt_b200 import mesh as M

pytestmark = pytest.mark.gpu

TOL64 = 1e-12  # the project's parity bar for FP64 operators
SUB, OFF, NB = (37, 4, 3), (2, 0, 1), (37 * 2 + 1 + 4, 4 * 2 + 1 + 2, 3 * 2 + 1 + 3)


def _ghosted(seed):
    """Coordinates of a ghosted box (a rank's node box around SUB elements)."""
    rng = np.random.default_rng(seed)
    m, eta, _ = M.problem("box:%d,%d,%d" % SUB, seed=seed)
    c = rng.uniform(size=(NB[2], NB[1], NB[0], 3))
    sl = tuple(slice(o, o + 2 * n + 1) for o, n in zip(OFF[::-1], SUB[::-1]))
    c[sl] = m.coords.reshape(c[sl].shape)
    return np.ascontiguousarray(c.reshape(-1)), eta, rng.uniform(-1, 1, size=c.size)


def _record(op, call):
    import torch
    st = torch.cuda.Stream()
    op.set_stream(st)
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g, stream=st):
        call()
    return g, st


def test_ghosted_b_and_bt_recorded_before_their_first_use(ora):
    """No warm-up is needed, and replays follow the coordinates."""
    import torch

    from pt_b200 import MatStokesMF
    c, eta, u = _ghosted(3)
    p = np.random.default_rng(4).uniform(-1, 1, size=4 * eta.size // 27)
    ud, pd = torch.from_numpy(u).cuda(), torch.from_numpy(p).cuda()
    yp, yu = torch.empty_like(pd), torch.empty_like(ud)

    def calls(op):
        op.MFStokesWrapper_A21(ud, yp)
        op.MFStokesWrapper_A12(pd, yu)

    for warm in (False, True):
        with MatStokesMF(*SUB, node_box=(*NB, *OFF)) as op, MatStokesMF(*SUB, node_box=(*NB, *OFF)) as own:
            op.set_coords(c)
            if warm:
                calls(op)
            g, st = _record(op, lambda: calls(op))
            for seed in (3, 8):
                cs = _ghosted(seed)[0]
                op.set_coords(cs)
                own.set_coords(cs)
                yp.fill_(np.nan)
                yu.fill_(np.nan)
                torch.cuda.synchronize()
                g.replay()
                torch.cuda.synchronize()
                assert relerr(yp.cpu(), own.MFStokesWrapper_A21(u)) < TOL64, (warm, seed)
                assert relerr(yu.cpu(), own.MFStokesWrapper_A12(p)) < TOL64, (warm, seed)


@pytest.mark.parametrize("workload", ["box:8,8,8", "box:21,13,17"])
def test_whole_operator_recorded_after_its_blocks(ora, workload):
    import torch

    from pt_b200 import MatStokesMF
    m, eta, mask = M.problem(workload, seed=7)
    u, p = M.uniform_vec(m.nvel, 8), M.uniform_vec(m.npres, 9)
    ud, pd = torch.from_numpy(u).cuda(), torch.from_numpy(p).cuda()
    yu, yp = torch.empty_like(ud), torch.empty_like(pd)
    with MatStokesMF(*m.dims) as op:
        op.SetUp(m.coords, eta, mask)
        op.MatMult_MFStokes_A11(ud, yu)
        op.MatMult_MFStokes_A12(pd, yu)
        op.MatMult_MFStokes_A21(ud, yp)
        g, st = _record(op, lambda: op.MatMult_MFStokes_A(ud, pd, yu, yp))
        yu.fill_(np.nan)
        yp.fill_(np.nan)
        torch.cuda.synchronize()
        g.replay()
        torch.cuda.synchronize()
        wu, wp = op.MatMult_MFStokes_A(u, p)
        assert relerr(yu.cpu(), wu) < TOL64 and relerr(yp.cpu(), wp) < TOL64


def test_graphs_of_one_op_on_two_streams():
    """Replayed at the same time, each gives what its call gives alone."""
    import torch

    from pt_b200 import MatStokesMF
    m, eta, mask = M.problem("box:33,30,28", seed=5)
    xs = [torch.from_numpy(M.uniform_vec(m.nvel, 6 + i)).cuda() for i in range(3)]
    pd = torch.from_numpy(M.uniform_vec(m.npres, 9)).cuda()
    with MatStokesMF(*m.dims) as op:
        op.SetUp(m.coords, eta, mask)
        assert op.a11_op == "b200_layer"
        calls = [lambda y: op.MatMult_MFStokes_A11(xs[0], y), lambda y: op.MFStokesWrapper_A11(xs[1], y),
                 lambda y: op.MatMult_MFStokes_A(xs[2], pd, y, yp), lambda y: op.MatMult_MFStokes_A12(pd, y),
                 lambda y: op.MatGetDiagonal_MFStokes_A11(y)]
        yp = torch.empty_like(pd)
        want = []
        for c in calls:
            y = torch.empty_like(xs[0])
            c(y)
            torch.cuda.synchronize()
            want.append(y)
        got = [torch.empty_like(xs[0]) for _ in calls]
        graphs = [_record(op, lambda: c(y))[0] for c, y in zip(calls, got)]
        streams = [torch.cuda.Stream() for _ in calls]
        for _ in range(20):
            for y in got:
                y.fill_(np.nan)
            torch.cuda.synchronize()
            for g, st in zip(graphs, streams):
                with torch.cuda.stream(st):
                    for _ in range(3):
                        g.replay()
            torch.cuda.synchronize()
            for k, (y, w) in enumerate(zip(got, want)):
                assert torch.equal(y, w), k


def test_graphs_follow_the_mask():
    """Recorded with one mask, replayed with another and with none."""
    import torch

    from pt_b200 import MatStokesMF
    m, eta, mask = M.problem("box:13,15,12", seed=5)
    u, p = (torch.from_numpy(M.uniform_vec(n, 3)).cuda() for n in (m.nvel, m.npres))
    yp, ya, yb, yu, yq = (torch.empty_like(v) for v in (p, u, u, u, p))

    def calls(op):
        op.MatMult_MFStokes_A21(u, yp)
        op.MatMult_MFStokes_A12(p, ya)
        op.MatMult_MFStokes_A11(u, yb)
        op.MatMult_MFStokes_A(u, p, yu, yq)

    with MatStokesMF(*m.dims) as op, MatStokesMF(*m.dims) as own:
        op.SetUp(m.coords, eta, mask)
        own.SetUp(m.coords, eta, mask)
        calls(op)
        g, st = _record(op, lambda: calls(op))
        for mk in (mask, np.roll(mask, 3), None):
            op.set_bc_mask(mk)
            own.set_bc_mask(mk)
            for y in (yp, ya, yb, yu, yq):
                y.fill_(np.nan)
            torch.cuda.synchronize()
            g.replay()
            torch.cuda.synchronize()
            got = [y.clone() for y in (yp, ya, yb, yu, yq)]
            calls(own)
            torch.cuda.synchronize()
            for k, (a, b) in enumerate(zip(got, (yp, ya, yb, yu, yq))):
                assert torch.equal(a, b), (k, mk is None)
