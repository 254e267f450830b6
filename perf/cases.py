"""The work that a user of the framework has it do, as cases that can be timed and checked.

Each kind of case goes through the public Python entry points (``pt_b200``):

``a11``      MatMult_MFStokes_A11, the viscous block inside every Krylov iteration (FP64) and smoother sweep (FP32).
``divgrad``  MatMult_MFStokes_A21 and MatMult_MFStokes_A12, the two off-diagonal blocks of a Schur-complement step.
``stokes``   MatMult_MFStokes_A, one apply of the whole operator on a one-rank box.
``rank``     MFStokesWrapper_A and MFStokesWrapper_diagA11 on the ghosted box of one rank of a multi-rank run.
``step``     a nonlinear iteration of a time step with a moved mesh: coordinates, viscosity and body force are
             new, then the momentum residual and the Jacobi diagonal.
``markers``  material points to Gauss-point viscosity and density, installed for the next apply.
``batch``    one apply over many independent boxes.
``solve``    a Picard step: new viscosity, then the multigrid-preconditioned viscous solve (its set-up included).
``serve``    a handful of solve requests through the request server, until the last one is done.

Sizes: 8^3, 64^3 and 128^3 are the boxes that the repository's tests and benchmark use; the others are ragged boxes
in between.  Solves run to a tight tolerance, so the solution does not depend on the rounding inside the
preconditioner.  Everything is made on the GPU from the seed alone.
"""
import math
import os
import sys

import numpy as np
import torch

_PKG = os.path.join(os.getcwd(), "ptatin-gene_b200")
if _PKG not in sys.path:
    sys.path.insert(1, _PKG)

from pt_b200 import MatStokesMF  # noqa: E402
from pt_b200.batch import BatchA11  # noqa: E402
from pt_b200.serve import Server  # noqa: E402
from pt_b200.solver import KSPSolveA11  # noqa: E402

F64 = torch.float64


def listed():
    return [
        # the smallest call: a coarse level or a unit-test box, where launches and host work count
        {"name": "a11_8", "kind": "a11", "mx": 8, "my": 8, "mz": 8, "f32": False},
        # an ordinary ragged box of one rank, odd in every axis
        {"name": "a11_41x37x29", "kind": "a11", "mx": 41, "my": 37, "mz": 29, "f32": False},
        # the benchmark's box: 50.9 M velocity dofs
        {"name": "a11_128", "kind": "a11", "mx": 128, "my": 128, "mz": 128, "f32": False},
        # a smoother's single-precision apply on a ragged box
        {"name": "a11_f32_97x70x81", "kind": "a11", "mx": 97, "my": 70, "mz": 81, "f32": True},
        # a nonlinear iteration after the mesh moved
        {"name": "step_64x48x40", "kind": "step", "mx": 64, "my": 48, "mz": 40},
        # divergence and gradient, ragged
        {"name": "divgrad_61x50x77", "kind": "divgrad", "mx": 61, "my": 50, "mz": 77},
        # the whole operator on a large one-rank box
        {"name": "stokes_96x96x64", "kind": "stokes", "mx": 96, "my": 96, "mz": 64},
        # one rank of a multi-rank run (two ghost nodes on each side)
        {"name": "rank_48x40x36", "kind": "rank", "mx": 48, "my": 40, "mz": 36},
        # 2.1 M material points on the 64^3 box
        {"name": "markers_64", "kind": "markers", "mx": 64, "my": 64, "mz": 64, "per_element": 8},
        # many small boxes in one apply
        {"name": "batch_96", "kind": "batch", "boxes": 96, "lo": 8, "hi": 32, "f32": False},
        # a Picard step of the precision form
        {"name": "solve_40", "kind": "solve", "mx": 40, "my": 40, "mz": 40},
        # a few requests of different sizes through the server
        {"name": "serve_12", "kind": "serve", "requests": 12, "lo": 8, "hi": 20},
    ]


def _log_uniform(rng, lo, hi):
    return math.exp(rng.uniform(math.log(lo), math.log(hi)))


def _dims(rng, lo, hi):
    """An element box of lo..hi elements in all, its axes within a factor of about two of each other."""
    n = _log_uniform(rng, lo, hi) ** (1.0 / 3.0)
    ax, ay = _log_uniform(rng, 0.7, 1.5), _log_uniform(rng, 0.7, 1.5)
    mx, my = max(2, round(n * ax)), max(2, round(n * ay))
    return {"mx": mx, "my": my, "mz": max(2, min(round(n / (ax * ay)), int(hi / (mx * my))))}


def draw(rng):
    kind = rng.choice(["a11", "a11", "a11", "divgrad", "stokes", "rank", "step", "markers", "batch", "solve", "serve"])
    if kind == "a11":
        return {"kind": kind, **_dims(rng, 64, 128 ** 3), "f32": rng.random() < 0.4}
    if kind in ("divgrad", "stokes"):
        return {"kind": kind, **_dims(rng, 512, 96 * 96 * 64)}
    if kind in ("rank", "step"):
        return {"kind": kind, **_dims(rng, 512, 72 ** 3)}
    if kind == "markers":
        return {"kind": kind, **_dims(rng, 512, 64 ** 3), "per_element": rng.randint(4, 8)}
    if kind == "batch":
        lo = rng.randint(4, 12)
        return {"kind": kind, "boxes": rng.randint(4, 96), "lo": lo, "hi": lo + rng.randint(4, 20), "f32": rng.random() < 0.4}
    if kind == "solve":
        return {"kind": kind, "mx": 8 * rng.randint(1, 5), "my": 8 * rng.randint(2, 5), "mz": 8 * rng.randint(2, 5)}
    lo = rng.randint(4, 10)
    return {"kind": kind, "requests": rng.randint(1, 12), "lo": lo, "hi": lo + rng.randint(2, 10)}


# ---- inputs, from the seed alone ------------------------------------------------------------------------------------

class _Box:
    """A perturbed unit box: coordinates, node box, and how elements find their nodes."""

    def __init__(self, mx, my, mz, gen, ghost=0, perturb=0.05):
        self.m, self.ghost = (mx, my, mz), ghost
        self.nel = mx * my * mz
        self.n = tuple(2 * m + 1 + 2 * ghost for m in (mx, my, mz))  # node box
        self.nnodes = self.n[0] * self.n[1] * self.n[2]
        h = [1.0 / m for m in (mx, my, mz)]
        ax = [(torch.arange(n, dtype=F64, device="cuda") - ghost) * (0.5 * hh) for n, hh in zip(self.n, h)]
        c = torch.empty(self.n[2], self.n[1], self.n[0], 3, dtype=F64, device="cuda")
        c[..., 0], c[..., 1], c[..., 2] = ax[0][None, None, :], ax[1][None, :, None], ax[2][:, None, None]
        for d in range(3):
            r = (2.0 * torch.rand(c.shape[:3], dtype=F64, device="cuda", generator=gen) - 1.0) * (perturb * h[d])
            for face in (0, -1):  # nodes keep to the face that they lie on
                r.select(2 - d, face).zero_()
            c[..., d] += r
        self.coords = c.reshape(-1)

    def node_box(self):
        return None if not self.ghost else (*self.n, self.ghost, self.ghost, self.ghost)

    def nodes(self, lo, hi):
        """(hi-lo, 27) node numbers of elements lo..hi."""
        e = torch.arange(lo, hi, device="cuda")
        ei, ej, ek = e % self.m[0], (e // self.m[0]) % self.m[1], e // (self.m[0] * self.m[1])
        X, XY, g = self.n[0], self.n[0] * self.n[1], self.ghost
        base = (2 * ei + g) + (2 * ej + g) * X + (2 * ek + g) * XY
        o = torch.arange(3, device="cuda")
        off = (o[None, None, :] + o[None, :, None] * X + o[:, None, None] * XY).reshape(-1)
        return base[:, None] + off[None, :]

    def mask(self):
        """Dirichlet on the x-faces, the normal component on the others (free slip)."""
        m = torch.zeros(self.n[2], self.n[1], self.n[0], 3, dtype=torch.uint8, device="cuda")
        m[:, :, 0, :] = 1
        m[:, :, -1, :] = 1
        for k in (0, -1):
            m[:, k, :, 1] = 1
            m[k, :, :, 2] = 1
        return m.reshape(-1)


_G1 = torch.tensor([-math.sqrt(0.6), 0.0, math.sqrt(0.6)], dtype=F64)
_W1 = torch.tensor([5.0 / 9.0, 8.0 / 9.0, 5.0 / 9.0], dtype=F64)


def _basis():
    """Q2 basis (27 points, 27 nodes), its gradient (27, 27, 3) and the weights at the 3x3x3 Gauss points."""
    b = torch.stack([0.5 * _G1 * (_G1 - 1), (1 + _G1) * (1 - _G1), 0.5 * (1 + _G1) * _G1], 1)
    d = torch.stack([_G1 - 0.5, -2 * _G1, _G1 + 0.5], 1)
    prod = lambda z, y, x: torch.einsum("ak,bj,ci->abckji", z, y, x).reshape(27, 27)  # noqa: E731
    w = torch.einsum("a,b,c->abc", _W1, _W1, _W1).reshape(27)
    return prod(b, b, b).cuda(), torch.stack([prod(b, b, d), prod(b, d, b), prod(d, b, b)], 2).cuda(), w.cuda()


def _chunks(n, size=1 << 16):
    return [(s, min(s + size, n)) for s in range(0, n, size)]


def _viscosity(box, gen, contrast, spheres=16, radius=0.1):
    """Layers along y and spherical inclusions, at the physical Gauss points: [27 nel]."""
    N, _, _ = _basis()
    centre = torch.rand(spheres, 3, dtype=F64, device="cuda", generator=gen)
    half = 0.5 * math.log10(contrast)
    value = 10.0 ** ((2.0 * torch.rand(spheres, dtype=F64, device="cuda", generator=gen) - 1.0) * half)
    out = torch.empty(box.nel, 27, dtype=F64, device="cuda")
    c = box.coords.view(-1, 3)
    for lo, hi in _chunks(box.nel):
        x = torch.einsum("qn,end->eqd", N, c[box.nodes(lo, hi)])
        e = torch.where(x[..., 1] < 0.4, 10.0 ** (0.5 * half), torch.ones_like(x[..., 1]))
        for s in range(spheres):
            e = torch.where(((x - centre[s]) ** 2).sum(-1) < radius * radius, value[s], e)
        out[lo:hi] = e
    return out.reshape(-1)


def _uniform(n, gen, dtype=F64):
    return (2.0 * torch.rand(n, dtype=F64, device="cuda", generator=gen) - 1.0).to(dtype)


def _inputs(case, seed):
    gen = torch.Generator(device="cuda")
    gen.manual_seed(int(seed))
    kind = case["kind"]
    if kind in ("batch", "serve"):
        # the sizes belong to the case, not to the seed: a side's work is the same for every seed
        sizes = torch.Generator()
        sizes.manual_seed(977 * case["lo"] + case["hi"])
        count = case["boxes"] if kind == "batch" else case["requests"]
        items = []
        for _ in range(count):
            m = torch.randint(case["lo"], case["hi"] + 1, (3,), generator=sizes).tolist()
            box = _Box(*m, gen)
            eta = torch.repeat_interleave(10.0 ** (2.0 * torch.rand(box.nel, dtype=F64, device="cuda", generator=gen)), 27)
            u = _uniform(3 * box.nnodes, gen, torch.float32 if case.get("f32") else F64)
            items.append({"box": box, "eta": eta, "mask": box.mask(), "u": u})
        return {"items": items}
    box = _Box(case["mx"], case["my"], case["mz"], gen, ghost=2 if kind == "rank" else 0)
    s = {"box": box, "eta": _viscosity(box, gen, 1e4 if kind == "solve" else 1e6)}
    s["mask"] = None if kind == "rank" else box.mask()
    s["u"] = _uniform(3 * box.nnodes, gen, torch.float32 if case.get("f32") else F64)
    if kind in ("divgrad", "stokes", "rank", "step"):
        s["p"] = _uniform(4 * box.nel, gen)
    if kind == "step":
        s["fu"] = _uniform(81 * box.nel, gen)
    if kind == "markers":
        k = case["per_element"]
        n = k * box.nel
        perm = torch.randperm(n, device="cuda", generator=gen)
        s["wil"] = torch.arange(n, device="cuda", dtype=torch.int32).div(k, rounding_mode="floor")[perm].contiguous()
        s["xi"] = _uniform(3 * n, gen)
        s["meta"] = 1.0 + 9999.0 * (torch.rand(n, dtype=F64, device="cuda", generator=gen) < 0.1).to(F64)
        s["mrho"] = 1.0 + 0.1 * torch.rand(n, device="cuda", generator=gen, dtype=F64)
    return s


def prepare(case, seed):
    s = _inputs(case, seed)
    kind = case["kind"]
    s["kind"] = kind
    if kind == "batch":
        s["ops"] = [MatStokesMF(*it["box"].m).SetUp(it["box"].coords, it["eta"], it["mask"].cpu().numpy()) for it in s["items"]]
        s["us"] = [it["u"] for it in s["items"]]
        # the results of all boxes in one buffer, box after box
        s["y"] = torch.empty(sum(u.numel() for u in s["us"]), dtype=s["us"][0].dtype, device="cuda")
        s["ys"] = list(s["y"].split([u.numel() for u in s["us"]]))
        s["batch"] = BatchA11(s["ops"], tile_x=64)
        del s["items"]
        return s
    if kind == "serve":
        host = lambda t: t.cpu().numpy()  # noqa: E731
        s["server"] = Server(rtol=1e-12, cheby_emin=0.03, memory_budget_bytes=8 << 30)
        s["requests"] = [(it["box"].m, host(it["box"].coords), host(it["eta"]), host(it["mask"]),
                          host(it["u"] * (it["mask"] == 0))) for it in s["items"]]
        del s["items"]
        return s
    box = s["box"]
    op = MatStokesMF(*box.m, node_box=box.node_box())
    op.SetUp(box.coords, s["eta"], None if s["mask"] is None else s["mask"].cpu().numpy())
    s["op"] = op
    if kind == "step":
        op.set_body_force(s["fu"])
    if kind in ("a11", "step", "stokes", "rank", "divgrad"):
        s["y"] = torch.empty_like(s["u"])
    if kind in ("divgrad", "stokes", "rank"):
        s["yp"] = torch.empty(4 * box.nel, dtype=F64, device="cuda")
    if kind in ("rank", "step"):
        s["d"] = torch.empty_like(s["u"])
    if kind == "solve":
        s["f"] = s["u"] * (s["mask"] == 0)
        s["x"] = torch.zeros_like(s["f"])
        s["ksp"] = KSPSolveA11(op, ksp="fcg", pc="mg", rtol=1e-12, cheby_emin=0.03, pc_graph=1)
    return s


def run(s):
    kind = s["kind"]
    if kind == "batch":
        s["batch"].apply(s["us"], s["ys"])
        return s["y"]
    if kind == "serve":
        server = s["server"]
        xs = [server.submit(i, *r) for i, r in enumerate(s["requests"])]
        done = 0
        while done < len(xs):
            server.step(8)
            done += len(server.done())
        return xs
    op = s["op"]
    if kind == "a11":
        return op.MatMult_MFStokes_A11(s["u"], s["y"])
    if kind == "divgrad":
        return [op.MatMult_MFStokes_A21(s["u"], s["yp"]), op.MatMult_MFStokes_A12(s["p"], s["y"])]
    if kind == "stokes":
        return list(op.MatMult_MFStokes_A(s["u"], s["p"], s["y"], s["yp"]))
    if kind == "rank":
        return [*op.MFStokesWrapper_A(s["u"], s["p"], s["y"], s["yp"]), op.MFStokesWrapper_diagA11(s["d"])]
    if kind == "step":
        op.set_coords(s["box"].coords)
        op.set_eta(s["eta"])
        op.set_body_force(s["fu"])
        return [op.FormFunctionLocal_U(s["u"], s["p"], s["y"]), op.MatGetDiagonal_MFStokes_A11(s["d"])]
    if kind == "markers":
        return list(op.ProjectMarkers(s["wil"], s["xi"], s["meta"], s["mrho"], install=True))
    op.set_eta(s["eta"])
    s["x"].zero_()
    s["ksp"].solve(s["f"], s["x"])
    return s["x"]


# ---- what a pass cannot do without -----------------------------------------------------------------------------------

# Sum-factorised operations of one element: gradient of a 3-component Q2 field at the 27 Gauss points (or its
# transpose), Jacobian and adjugate at the points, the viscous action.
_GRAD, _GEOM, _VISC = 2200, 2700, 2600


def work(case):
    kind = case["kind"]
    if kind in ("batch", "serve"):
        sizes = torch.Generator()
        sizes.manual_seed(977 * case["lo"] + case["hi"])
        nel = nvel = 0
        for _ in range(case["boxes"] if kind == "batch" else case["requests"]):
            m = torch.randint(case["lo"], case["hi"] + 1, (3,), generator=sizes).tolist()
            nel += m[0] * m[1] * m[2]
            nvel += 3 * (2 * m[0] + 1) * (2 * m[1] + 1) * (2 * m[2] + 1)
    else:
        m = (case["mx"], case["my"], case["mz"])
        nel = m[0] * m[1] * m[2]
        nvel = 3 * (2 * m[0] + 1) * (2 * m[1] + 1) * (2 * m[2] + 1)
    a11 = 2 * _GRAD + _GEOM + _VISC
    if kind in ("a11", "batch"):
        return {"bytes": (3 * nvel + 27 * nel) * (4 if case["f32"] else 8), "flops": a11 * nel}
    if kind == "divgrad":
        return {"bytes": 8 * 2 * (2 * nvel + 4 * nel), "flops": 2 * (_GRAD + _GEOM + 300) * nel}
    if kind == "stokes":
        return {"bytes": 8 * (3 * nvel + 35 * nel), "flops": (a11 + 800) * nel}
    if kind == "rank":
        return {"bytes": 8 * (4 * nvel + 35 * nel), "flops": (a11 + 800 + 6000) * nel}
    if kind == "step":
        return {"bytes": 8 * (4 * nvel + (27 + 81 + 4) * nel), "flops": (a11 + 1500 + 6000) * nel}
    if kind == "markers":
        return {"bytes": nel * (case["per_element"] * 44 + 8 * 54), "flops": nel * (case["per_element"] * 80 + 27 * 40)}
    # a solve: the least is one apply of the operator and its diagonal, whatever the number of iterations
    return {"bytes": 8 * (4 * nvel + 27 * nel), "flops": (a11 + 6000) * nel}


# ---- the same in 64 bits, by plain torch -----------------------------------------------------------------------------

def _operator(box, eta, u=None, p=None, fu=None, mask=None, diag=False, a11=True):
    """Dense element arithmetic in FP64 chunk by chunk: A11 u (+ B^T p - F), B u and the diagonal, no Dirichlet rows."""
    N, dN, w = _basis()
    c = box.coords.view(-1, 3)
    n3 = 3 * box.nnodes
    y = torch.zeros(box.nnodes, 3, dtype=F64, device="cuda")
    d = torch.zeros(box.nnodes, 3, dtype=F64, device="cuda") if diag else None
    yp = torch.empty(box.nel, 4, dtype=F64, device="cuda") if u is not None else None
    if u is not None:
        uu = u.to(F64)
        if mask is not None:
            uu = torch.where(mask != 0, 0.0, uu)
        uu = uu.view(-1, 3)
    for lo, hi in _chunks(box.nel, 1 << 15):
        nid = box.nodes(lo, hi)
        x = c[nid]
        J = torch.einsum("qnd,enl->eqdl", dN, x)          # d x_l / d xi_d
        c0, c1, c2 = (torch.cross(J[..., a, :], J[..., b, :], dim=-1) for a, b in ((1, 2), (2, 0), (0, 1)))
        det = (J[..., 0, :] * c0).sum(-1)
        inv = torch.stack([c0, c1, c2], -1) / det[..., None, None]   # d xi_d / d x_l at [l, d]
        wd = w * det
        gN = torch.einsum("qnd,eqld->eqnl", dN, inv)      # physical basis gradients
        xq = torch.einsum("qn,enl->eql", N, x)
        L = torch.stack([x[:, 14, 0] - x[:, 12, 0], x[:, 16, 1] - x[:, 10, 1], x[:, 22, 2] - x[:, 4, 2]], -1)
        Np = torch.cat([torch.ones_like(xq[..., :1]), (xq - x.mean(1)[:, None]) / L[:, None]], -1)
        we = wd * eta.view(-1, 27)[lo:hi] if eta is not None else None
        out = torch.zeros(hi - lo, 27, 3, dtype=F64, device="cuda")
        if u is not None:
            g = torch.einsum("eqnk,enl->eqkl", gN, uu[nid])  # d u_l / d x_k
            if a11:
                out += torch.einsum("eqnk,eqkl->enl", gN, we[..., None, None] * (g + g.transpose(-1, -2)))
            div = g[..., 0, 0] + g[..., 1, 1] + g[..., 2, 2]
            yp[lo:hi] = -torch.einsum("eq,eqi->ei", wd * div, Np)
        if p is not None:
            pq = torch.einsum("eqi,ei->eq", Np, p.view(-1, 4)[lo:hi])
            out -= torch.einsum("eq,eqnl->enl", wd * pq, gN)
        if fu is not None:
            out -= torch.einsum("eq,qn,eql->enl", wd, N, fu.view(-1, 27, 3)[lo:hi])
        y.index_add_(0, nid.reshape(-1), out.reshape(-1, 3))
        if diag:
            g2 = gN ** 2
            dd = torch.einsum("eq,eqnl->enl", we, g2 + g2.sum(-1, keepdim=True))
            d.index_add_(0, nid.reshape(-1), dd.reshape(-1, 3))
    return y.view(n3), None if yp is None else yp.view(-1), None if d is None else d.view(n3)


def _projection(s):
    """Nodal sums over the markers (Q1 weights at the vertices, 1 at the other nodes), divided, then the Q1 interpolant
    of the vertex values at the Gauss points within the range of the element's nodes."""
    box = s["box"]
    vert = torch.tensor([0, 2, 6, 8, 18, 20, 24, 26], device="cuda")
    sign = torch.tensor([[2.0 * (v & 1) - 1, 2.0 * (v >> 1 & 1) - 1, 2.0 * (v >> 2) - 1] for v in range(8)], dtype=F64, device="cuda")
    el, xi = s["wil"].long(), s["xi"].view(-1, 3)
    part = torch.zeros(box.nel, 27, 3, dtype=F64, device="cuda")
    val = torch.stack([s["meta"], s["mrho"], torch.ones_like(s["meta"])], -1)
    for n in range(27):
        v = (vert == n).nonzero()
        wt = torch.prod(1.0 + xi * sign[int(v)], -1) / 8.0 if len(v) else torch.ones_like(s["meta"])
        acc = torch.zeros(box.nel, 3, dtype=F64, device="cuda")
        acc.index_add_(0, el, wt[:, None] * val)
        part[:, n] = acc
    nid = box.nodes(0, box.nel)
    node = torch.zeros(box.nnodes, 3, dtype=F64, device="cuda")
    node.index_add_(0, nid.reshape(-1), part.reshape(-1, 3))
    f = (node[:, :2] / node[:, 2:])[nid]                   # (nel, 27, 2)
    g = torch.stack(torch.meshgrid(_G1, _G1, _G1, indexing="ij"), -1).reshape(27, 3).flip(-1).cuda()
    N1 = torch.prod(1.0 + g[:, None] * sign[None], -1) / 8.0
    q = torch.einsum("qv,evf->eqf", N1, f[:, vert])
    q = torch.minimum(torch.maximum(q, f.amin(1, keepdim=True)), f.amax(1, keepdim=True))
    return [q[..., 0].reshape(-1).contiguous(), q[..., 1].reshape(-1).contiguous()]


def _rows(y, x, mask):
    return torch.where(mask != 0, x.to(F64), y)


def exact(case, seed):
    kind = case["kind"]
    if kind in ("solve", "serve"):
        return None
    s = _inputs(case, seed)
    if kind == "batch":
        return torch.cat([_rows(_operator(it["box"], it["eta"], it["u"], mask=it["mask"])[0], it["u"], it["mask"])
                          for it in s["items"]])
    if kind == "markers":
        return _projection(s)
    box = s["box"]
    if kind == "a11":
        return _rows(_operator(box, s["eta"], s["u"], mask=s["mask"])[0], s["u"], s["mask"])
    if kind == "divgrad":
        _, yp, _ = _operator(box, None, s["u"], mask=s["mask"], a11=False)
        yu, _, _ = _operator(box, None, p=s["p"])
        return [yp, torch.where(s["mask"] != 0, 0.0, yu)]
    if kind == "stokes":
        yu, yp, _ = _operator(box, s["eta"], s["u"], s["p"], mask=s["mask"])
        return [_rows(yu, s["u"], s["mask"]), yp]
    if kind == "rank":
        return list(_operator(box, s["eta"], s["u"], s["p"], diag=True))
    yu, _, d = _operator(box, s["eta"], s["u"], s["p"], s["fu"], diag=True)
    return [yu, torch.where(s["mask"] != 0, 1.0, d)]
