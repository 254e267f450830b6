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
