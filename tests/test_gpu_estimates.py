"""Two parts of the preconditioner on their own, which a solve would survive if they
were poor: the Lanczos estimate of lambda_max(D^-1 A) (solver and request server) and
the dense inverse of a small level (blocked Gauss-Jordan), against dense FP64 algebra
on the oracle's operator."""
import numpy as np
import pytest

from pt_b200 import mesh as M

pytestmark = pytest.mark.gpu


def _dense(ora, m, eta, mask):
    A = np.empty((m.nvel, m.nvel))
    for j in range(m.nvel):
        e = np.zeros(m.nvel)
        e[j] = 1.0
        A[:, j] = ora.matmult_a11(m.dims, m.coords, eta, mask, e)
    return A


def _hash(n, seed=12345):
    """The estimate's start vector (splitmix64 of the index)."""
    with np.errstate(over="ignore"):
        z = np.arange(n, dtype=np.uint64) + np.uint64(seed) * np.uint64(0x9E3779B97F4A7C15)
        z = (z ^ (z >> np.uint64(30))) * np.uint64(0xBF58476D1CE4E5B9)
        z = (z ^ (z >> np.uint64(27))) * np.uint64(0x94D049BB133111EB)
        z ^= z >> np.uint64(31)
    return (z >> np.uint64(11)).astype(np.float64) * (2.0 / 9007199254740992.0) - 1.0


def _lanczos(A, its):
    """Largest eigenvalue of the tridiagonal matrix of `its` Jacobi-PCG steps."""
    d = np.diag(A)
    r = _hash(len(d))
    z = r / d
    p, rz, al, be = z.copy(), r @ z, [], []
    for _ in range(its):
        q = A @ p
        al.append(rz / (p @ q))
        r = r - al[-1] * q
        z = r / d
        be.append((r @ z) / rz)
        rz = r @ z
        p = z + be[-1] * p
    t = [1.0 / al[k] + (be[k - 1] / al[k - 1] if k else 0.0) for k in range(its)]
    o = [np.sqrt(be[k]) / al[k] for k in range(its - 1)]
    return np.linalg.eigvalsh(np.diag(t) + np.diag(o, 1) + np.diag(o, -1))[-1]


# Rounding differs (order of the sums), the recurrence does not; up to 20 steps its
# growth stays far below 1e-9.  From 40 steps on the estimate is the eigenvalue
# itself to 1e-14 for boxes of this size.
@pytest.mark.parametrize("its", [1, 2, 7, 20, 40])
@pytest.mark.parametrize("workload", ["box:2,2,2", "box:3,2,2"])
def test_lambda_max(ora, workload, its):
    import torch

    from pt_b200 import MatStokesMF
    from pt_b200.serve import Server
    from pt_b200.solver import KSPSolveA11
    m, eta, mask = M.problem(workload, seed=4)
    A = _dense(ora, m, eta, mask)
    want = _lanczos(A, its)
    if its >= 40:
        d = np.sqrt(np.diag(A))
        exact = np.linalg.eigvalsh(A / d[:, None] / d[None, :])[-1]
        assert abs(want / exact - 1) < 1e-12
    f = M.uniform_vec(m.nvel, 5) * (mask == 0)
    fd = torch.from_numpy(f).cuda()
    with MatStokesMF(*m.dims) as op:
        op.SetUp(m.coords, eta, mask)
        with KSPSolveA11(op, pc="cheby_jacobi", eig_its=its, max_it=2) as k:
            got = k.solve(fd, torch.zeros_like(fd))["lambda_max"]
    assert abs(got / want - 1) < 1e-9
    with Server(eig_its=its, max_it=2, memory_budget_bytes=1 << 30) as s:
        s.submit(0, m.dims, m.coords, eta, mask, f)
        out = []
        while not out:
            s.step(2)
            out = s.done()
    assert abs(out[0]["lambda_max"] / want - 1) < 1e-9


# Sizes: one block of 32 rows and less, exact and ragged multiples, the largest
# level that is inverted.  Condition numbers are below 1e4, so FP64 elimination
# leaves less than 1e4 * 1029 * 1.1e-16 = 1.2e-9 of the solution.  An FP32 inverse of
# these boxes applied in FP32 by numpy leaves 1e-7; another order of the sums may add
# sqrt(n) roundings of the largest term, within 1e-5.
@pytest.mark.parametrize("fp32", [0, 1])
@pytest.mark.parametrize("workload", ["box:1,1,1", "box:2,1,1", "box:2,2,2", "box:3,2,2", "box:3,3,3"])
def test_dense_coarse_inverse(ora, workload, fp32):
    import torch

    from pt_b200 import MatStokesMF
    from pt_b200.solver import KSPSolveA11
    m, eta, mask = M.problem(workload, seed=6)
    A = _dense(ora, m, eta, mask)
    assert np.linalg.cond(A) < 1e4
    r = M.uniform_vec(m.nvel, 7)
    rd = torch.from_numpy(r).cuda()
    z = torch.empty_like(rd)
    with MatStokesMF(*m.dims) as op:
        op.SetUp(m.coords, eta, mask)
        with KSPSolveA11(op, pc="mg", mg_levels=1, mg_assembled=1, cheby_fp32=fp32) as k:
            k.apply_pc(rd, z)
            torch.cuda.synchronize()
    want = np.linalg.solve(A, r)
    err = np.linalg.norm(z.cpu().numpy() - want) / np.linalg.norm(want)
    assert err < (1e-5 if fp32 else 1.2e-9), err
