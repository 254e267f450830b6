"""One op or one batch used from several host threads, streams or captured graphs:
every result is bitwise that of the same call alone."""
import threading

import numpy as np
import pytest

from pt_b200 import mesh as M

pytestmark = pytest.mark.gpu


def _op(m, eta, mask, a11_op="b200_layer"):
    from pt_b200 import MatStokesMF
    return MatStokesMF(*m.dims, a11_op=a11_op).SetUp(m.coords, eta, mask)


def test_pinned_host_applies_beside_device_applies_of_another_thread():
    """The pipelined host apply is enqueued in groups whose gathers read sums of the
    groups before; another thread's applies use the same scratch."""
    import torch
    m, eta, mask = M.problem("box:14,15,40", seed=2)
    hx = torch.from_numpy(M.uniform_vec(m.nvel, 3)).pin_memory().numpy()
    hy = torch.empty(m.nvel, dtype=torch.float64).pin_memory().numpy()
    xd = torch.from_numpy(M.uniform_vec(m.nvel, 4)).cuda()
    pd = torch.from_numpy(M.uniform_vec(m.npres, 5)).cuda()
    with _op(m, eta, mask) as op:
        want_h = op.MatMult_MFStokes_A11(hx).copy()
        want = [op.MatMult_MFStokes_A11(xd), op.MFStokesWrapper_A12(pd)]
        got = [torch.empty_like(xd), torch.empty_like(xd)]
        torch.cuda.synchronize()
        stop, bad, seen = threading.Event(), [], []

        def other():
            try:
                while not stop.is_set():
                    op.MatMult_MFStokes_A11(xd, got[0])
                    op.MFStokesWrapper_A12(pd, got[1])
                    torch.cuda.synchronize()
                    seen.append(all(torch.equal(a, b) for a, b in zip(got, want)))
            except Exception as e:  # pragma: no cover
                bad.append(e)

        t = threading.Thread(target=other)
        t.start()
        ok = []
        for _ in range(150):
            hy[:] = np.nan
            ok.append(np.array_equal(op.MatMult_MFStokes_A11(hx, hy), want_h))
        stop.set()
        t.join()
        assert not bad and seen and all(seen) and all(ok), (bad, len(seen), sum(seen), sum(ok))


@pytest.mark.parametrize("fp32", [False, True])
def test_one_batch_on_two_streams_and_in_a_graph(fp32):
    """Each apply of a batch has scratch of its own: applies that overlap on two
    streams, and a recorded one replayed beside them, are bitwise the apply alone."""
    import torch

    from pt_b200.batch import BatchA11
    ops, us = [], []
    try:
        for i, dims in enumerate([(17, 13, 11), (33, 20, 9), (8, 8, 8), (41, 7, 5)]):
            m = M.make_mesh(*dims, perturb=0.05, seed=i)
            ops.append(_op(m, M.eta_per_element(m, contrast=1e3, seed=i), M.bc_mask_freeslip(*dims)))
            us.append([torch.from_numpy(M.uniform_vec(m.nvel, 9 * i + k)).cuda() for k in range(3)])
        us = [[v.float() if fp32 else v for v in row] for row in us]
        xs = [[row[k] for row in us] for k in range(3)]  # three input sets
        with BatchA11(ops) as b:
            want = [[torch.empty_like(v) for v in x] for x in xs]
            got = [[torch.empty_like(v) for v in x] for x in xs]
            for x, w, g in zip(xs, want, got):
                b.apply(x, w)
                b.tables(x, g)  # pointer tables exist before the capture
            torch.cuda.synchronize()
            st = [torch.cuda.Stream() for _ in range(3)]
            graph = torch.cuda.CUDAGraph()
            with torch.cuda.graph(graph, stream=st[2]):
                b.apply(xs[2], got[2], stream=st[2])
            for _ in range(20):
                for g in got:
                    for y in g:
                        y.fill_(np.nan)
                torch.cuda.synchronize()
                for _ in range(3):
                    b.apply(xs[0], got[0], stream=st[0])
                    b.apply(xs[1], got[1], stream=st[1])
                    with torch.cuda.stream(st[2]):
                        graph.replay()
                torch.cuda.synchronize()
                for k in range(3):
                    assert all(torch.equal(a, w) for a, w in zip(got[k], want[k])), k
    finally:
        for op in ops:
            op.Destroy()


@pytest.mark.parametrize("dims", [(9, 8, 7), (52, 50, 50)])
def test_first_calls_of_two_threads(dims):
    """B u, B^T p and the tiles' sums are set up by whichever thread comes first."""
    import torch

    from pt_b200 import MatStokesMF
    m = M.make_mesh(*dims, perturb=0.05, seed=1)
    u, p = (torch.from_numpy(M.uniform_vec(n, 3)).cuda() for n in (m.nvel, m.npres))
    calls = [lambda op: op.MFStokesWrapper_A12(p), lambda op: op.MFStokesWrapper_A21(u)]
    want = None
    for _ in range(6):
        with MatStokesMF(*dims) as op:
            op.set_coords(m.coords)
            op.set_stream(torch.cuda.Stream())
            got, start = {}, threading.Barrier(4)

            def run(k):
                start.wait()
                got[k] = calls[k % 2](op)

            ts = [threading.Thread(target=run, args=(k,)) for k in range(4)]
            for t in ts:
                t.start()
            for t in ts:
                t.join()
            torch.cuda.synchronize()
            want = want or [c(op) for c in calls]
            torch.cuda.synchronize()
            assert all(torch.equal(got[k], want[k % 2]) for k in range(4))


@pytest.mark.parametrize("dims", [(8, 8, 8), (16, 16, 16), (20, 18, 16)])
def test_applies_of_two_threads(dims):
    """Both precisions of the default op from two host threads: the launches of an apply
    stay together whatever kernel serves it."""
    import torch
    m = M.make_mesh(*dims, perturb=0.05, seed=1)
    u = torch.from_numpy(M.uniform_vec(m.nvel, 3)).cuda()
    us = [u, -2.0 * u, u.float(), (-2.0 * u).float()]
    with _op(m, M.eta_per_element(m, contrast=1e3, seed=2), M.bc_mask_freeslip(*dims), "b200") as op:
        want = [op.MatMult_MFStokes_A11(v) for v in us]
        got = [[torch.empty_like(v) for _ in range(50)] for v in us]
        torch.cuda.synchronize()
        ts = [threading.Thread(target=lambda k=k: [op.MatMult_MFStokes_A11(us[k], y) for y in got[k]])
              for k in range(len(us))]
        for t in ts:
            t.start()
        for t in ts:
            t.join()
        torch.cuda.synchronize()
        for k, w in enumerate(want):
            assert all(torch.equal(y, w) for y in got[k]), k
