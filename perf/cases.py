"""The work that programs have this library do, as measured cases.

One Newton step of a ChiDG run makes these calls: the Jacobian and residual are
written (by the host code, or by the Euler assembly here), the preconditioner
is updated on the new Jacobian, and FGMRES applies it and the matrix some
twenty to forty times.  The cases are those calls, alone and as whole solves:
from boxes of a few elements, where the latency of a call is all there is, to
the 24^3 box of order 2 whose Jacobian holds 13.6 GB.  Block sizes are those of
five fields on tensor Legendre bases of orders 1, 2 and 3 (40, 135 and 320
rows).  Values follow the seeded synthetic Jacobians of the tests: a shifted
diagonal, dense random blocks and the face couplings of an upwinded flux.
"""
import math
import random

import numpy as np
import torch

from chidg_b200 import api, euler, mesh

NFIELDS = 5
# diagonal shift, spread of the diagonal block, scales of the face blocks
# XI_MIN..ZETA_MAX, scale of the time-coupling blocks
SHIFT, SPREAD, FACES, COUPLING = 1.0, 0.6, (1.0, 0.4, 0.7, 0.4, 0.7, 0.4), 0.1
RTOL = 1e-8


def listed():
    return [
        # products of a coarse box: what one call costs
        _mv("mv_p1_small", 4, 3, 2, "1"),
        # products with an order per element (adapted meshes): ragged blocks
        _mv("mv_orders", 11, 13, 12, "123"),
        # a new Jacobian: update the block ILU0, apply it once (the smoother's use)
        _precon("precon_p1", 10, 9, 8, 1),
        _precon("precon_p2", 13, 14, 12, 2),
        _precon("precon_p3", 9, 8, 10, 3),
        # whole linear solves of a Newton step, the update included
        _solve("solve_p1", 8, 8, 8, 1, 30),
        _solve("solve_p2", 24, 24, 24, 2, 50),
        # the same with FP32 inner solves
        _solve("solve_mixed_p2", 14, 15, 13, 2, 30, precision="mixed_fp32"),
        # an adjoint solve: A^T throughout, transposed anew
        _solve("solve_adjoint_p2", 9, 11, 10, 2, 30, adjoint=True),
        # harmonic balance: time levels coupled in the matrix, precon_HB
        _solve("solve_hb", 6, 7, 5, 1, 30, ntime=7, precon="hb"),
        # many small systems in one call
        {"name": "solve_batched", "kind": "batched", "systems": 24, "lo": 4, "hi": 8, "orders": "12", "nkrylov": 30},
        # the caller side: residual and Jacobian of the Euler equations, then
        # one product with that Jacobian
        {"name": "euler_p2", "kind": "euler", "nx": 12, "ny": 11, "nz": 13, "order": 2},
    ]


def _mv(name, nx, ny, nz, orders):
    return {"name": name, "kind": "mv", "nx": nx, "ny": ny, "nz": nz, "orders": orders}


def _precon(name, nx, ny, nz, order):
    return {"name": name, "kind": "precon", "nx": nx, "ny": ny, "nz": nz, "order": order}


def _solve(name, nx, ny, nz, order, nkrylov, precision="fp64", adjoint=False, ntime=1, precon="ilu0"):
    return {"name": name, "kind": "solve", "nx": nx, "ny": ny, "nz": nz, "order": order, "nkrylov": nkrylov,
            "precision": precision, "adjoint": adjoint, "ntime": ntime, "precon": precon}


# elements of the largest drawn box of an order
_MOST = {1: 6000, 2: 4000, 3: 700}


def _draw_box(rng, order, least=8, share=1.0):
    """Sides of a box of least..most elements, log-uniform, sides within a factor of two."""
    target = math.exp(rng.uniform(math.log(least), math.log(_MOST[order] * share)))
    side = target ** (1.0 / 3.0)
    return [max(1, int(round(side * rng.uniform(0.75, 1.25)))) for _ in range(3)]


def draw(rng):
    kind = rng.choice(["mv", "precon", "precon", "solve", "solve", "solve", "batched", "euler"])
    if kind == "mv":
        orders = rng.choice(["1", "2", "3", "12", "123"])
        nx, ny, nz = _draw_box(rng, int(orders[-1]))
        c = _mv("", nx, ny, nz, orders)
    elif kind == "precon":
        order = rng.choice([1, 2, 3])
        nx, ny, nz = _draw_box(rng, order)
        c = _precon("", nx, ny, nz, order)
    elif kind == "solve":
        form = rng.choice(["plain", "plain", "mixed", "adjoint", "hb"])
        order = 1 if form == "hb" else rng.choice([1, 2, 3])
        nx, ny, nz = _draw_box(rng, order, share=0.05 if form == "hb" else 0.5)
        c = _solve("", nx, ny, nz, order, rng.choice([30, 50]), precision="mixed_fp32" if form == "mixed" else "fp64",
                   adjoint=form == "adjoint", ntime=rng.choice([3, 5, 7]) if form == "hb" else 1,
                   precon=rng.choice(["ilu0", "hb"]) if form == "hb" else "ilu0")
    elif kind == "batched":
        c = {"kind": "batched", "systems": rng.randint(3, 40), "lo": rng.randint(2, 5), "hi": rng.randint(5, 8),
             "orders": rng.choice(["1", "2", "12"]), "nkrylov": 30}
    else:
        order = rng.choice([1, 2, 3])
        nx, ny, nz = _draw_box(rng, order, share=0.5)
        c = {"kind": "euler", "nx": nx, "ny": ny, "nz": nz, "order": order}
    c.pop("name", None)
    return c


# ---- inputs --------------------------------------------------------------------

def _pattern(nx, ny, nz, order, ntime=1):
    return mesh.box_pattern(nx, ny, nz, NFIELDS, mesh.nterms_of_order(order), ntime=ntime)


def _ragged_pattern(case):
    orders = [int(o) for o in case["orders"]]
    if len(orders) == 1:
        return _pattern(case["nx"], case["ny"], case["nz"], orders[0])
    pat = _pattern(case["nx"], case["ny"], case["nz"], 1)
    rng = random.Random("%(nx)d %(ny)d %(nz)d" % case)
    return mesh.with_element_orders(pat, [rng.choice(orders) for _ in range(pat.nelem)])


def _batch_patterns(case):
    rng = random.Random("%(systems)d %(lo)d %(hi)d" % case)
    return [_pattern(*(rng.randint(case["lo"], case["hi"]) for _ in range(3)), int(rng.choice(case["orders"])))
            for _ in range(case["systems"])]


def _uniform(n, gen):
    return torch.rand(n, dtype=torch.float64, device="cuda", generator=gen).mul_(2.0).sub_(1.0)


def _values(pat, gen):
    """Packed column-major block values of a pattern."""
    nr, nc = (torch.as_tensor(d, device="cuda") for d in pat.block_dims())
    face = torch.as_tensor(np.asarray(pat.blk_face, dtype=np.int64), device="cuda")
    scale = torch.tensor(FACES + (SPREAD, COUPLING), dtype=torch.float64, device="cuda")[face] / nc.double().sqrt()
    sizes = nr * nc
    vals = _uniform(int(sizes.sum()), gen)
    if int(sizes.min()) == int(sizes.max()):
        vals.view(len(sizes), -1).mul_(scale[:, None])
    else:
        vals.mul_(torch.repeat_interleave(scale, sizes))
    first = torch.cumsum(sizes, 0) - sizes
    diag = face == mesh.DIAG
    b = nr[diag]
    start = torch.repeat_interleave(first[diag], b)
    within = torch.arange(int(b.sum()), device="cuda") - torch.repeat_interleave(torch.cumsum(b, 0) - b, b)
    vals[start + within * (torch.repeat_interleave(b, b) + 1)] += SHIFT
    return vals


class _DeviceArray:
    """FP64 device memory of the library, seen by torch without a copy."""

    def __init__(self, owner, ptr, n):
        self.owner = owner
        self.__cuda_array_interface__ = {"shape": (n,), "typestr": "<f8", "data": (ptr, False), "version": 3,
                                         "strides": None}


def _view(v):
    return torch.as_tensor(_DeviceArray(v, v.device_ptr(), v.n), device="cuda")


def _matrix(pat, vals):
    A = api.ChidgMatrix(pat)
    torch.cuda.synchronize()
    A.upload_device(vals.data_ptr())
    A.ctx.sync()
    return A


def _vector(A, vals=None):
    v = api.ChidgVector(A)
    if vals is not None:
        _view(v).copy_(vals)
        torch.cuda.synchronize()
    return v


def _inputs(case, seed):
    """The pattern (of the packed systems for a batch), its block values and a vector."""
    gen = torch.Generator(device="cuda").manual_seed(1000003 * int(seed) + 17)
    if case["kind"] == "mv":
        pat = _ragged_pattern(case)
    elif case["kind"] == "batched":
        pat = mesh.concat_patterns(_batch_patterns(case))[0]
    else:
        pat = _pattern(case["nx"], case["ny"], case["nz"], case["order"], case.get("ntime", 1))
    return pat, _values(pat, gen), _uniform(pat.vector_size(), gen)


def _euler_inputs(case, seed):
    """Box, state (an oblique freestream with a few per cent of disturbance in
    every mode) and a direction."""
    gen = torch.Generator(device="cuda").manual_seed(1000003 * int(seed) + 29)
    box = euler.EulerBox(case["nx"], case["ny"], case["nz"], case["order"], vel_inf=(0.3, 0.1, -0.05))
    u = torch.tensor(box.vel_inf, dtype=torch.float64, device="cuda")
    energy = box.p_inf / (euler.GAMMA - 1.0) + 0.5 * box.rho_inf * (u * u).sum()
    free = torch.cat([torch.tensor([box.rho_inf], dtype=torch.float64, device="cuda"), box.rho_inf * u, energy[None]])
    degree = torch.as_tensor(euler.MODE_ORDER[:box.nterms].sum(axis=1), device="cuda")
    q = 0.02 * _uniform(box.nelem * NFIELDS * box.nterms, gen).view(box.nelem, NFIELDS, -1) / (1 + degree) ** 2
    q[:, :, 0] += free
    return box, q.reshape(-1), _uniform(q.numel(), gen)


def _options(case):
    o = dict(tol=0.0, rtol=RTOL, nkrylov=case["nkrylov"], nmax=300, inner_fgmres=0)
    if case.get("precision", "fp64") != "fp64":
        o["precision"] = case["precision"]
    return o


def prepare(case, seed):
    s = {"kind": case["kind"]}
    if case["kind"] == "euler":
        box, q, v = _euler_inputs(case, seed)
        s["A"] = A = api.ChidgMatrix(box.pattern)
        s["device"] = euler.EulerDevice(box)
        s["q"], s["v"], s["r"], s["y"] = _vector(A, q), _vector(A, v), _vector(A), _vector(A)
        s["out"] = {"r": _view(s["r"]), "jv": _view(s["y"])}
        return s
    pat, vals, v = _inputs(case, seed)
    s["A"] = A = _matrix(pat, vals)
    s["v"], s["y"] = _vector(A, v), _vector(A)
    s["out"] = _view(s["y"])
    if case["kind"] == "precon":
        s["M"] = api.create_preconditioner("ilu0").init(A)
    elif case["kind"] in ("solve", "batched"):
        if case.get("adjoint"):
            A.transposed = True
            s["values"] = vals
        s["M"] = api.create_preconditioner(case.get("precon", "ilu0")).init(A)
        s["solver"] = api.create_linear_solver("fgmres", **_options(case))
        if case["kind"] == "batched":
            s["sys_elem"] = mesh.concat_patterns(_batch_patterns(case))[1]
    return s


def run(s):
    kind = s["kind"]
    if kind == "mv":
        api.chidg_mv(s["A"], s["v"], s["y"])
        return s["out"]
    if kind == "precon":
        s["M"].update(s["A"])
        s["M"].apply(s["A"], s["v"], s["y"])
        return s["out"]
    if kind == "euler":
        s["device"].assemble(s["q"], s["r"], s["A"])
        api.chidg_mv(s["A"], s["v"], s["y"])
        return s["out"]
    if kind == "batched":
        s["solver"].solve_batched(s["A"], s["y"], s["v"], s["M"], s["sys_elem"])
        return s["out"]
    if "values" in s:                       # each Newton step's adjoint has a new matrix
        s["A"].upload_device(s["values"].data_ptr())
    s["solver"].solve(s["A"], s["y"], s["v"], s["M"])
    return s["out"]


# ---- what a pass cannot do without ------------------------------------------------

def _counts(pat):
    """Block entries (all, diagonal, lower local) and the work of the factorisation."""
    nr, nc = pat.block_dims()
    re, ce = np.asarray(pat.blk_row_elem), np.asarray(pat.blk_col_elem)
    local = np.asarray(pat.blk_face) != mesh.OTHER
    diag, low = np.asarray(pat.blk_face) == mesh.DIAG, local & (ce < re)
    size = nr * nc
    # L = A inv(D), D -= L U and the inverses
    flops = float((4.0 * nr[low] * nc[low] * nc[low]).sum() + (2.0 * nr[diag] ** 3).sum())
    return float(size.sum()), float(size[diag].sum()), float(size[low].sum()), float(size[local & ~diag & ~low].sum()), flops


def _iterations(case, box):
    """About the number of Arnoldi steps these systems take (counted on boxes of 6^3 to 24^3)."""
    if case.get("precon") == "hb":
        return 100
    return int(round(18 + 0.85 * sum(box) / 3.0))


def _solve_work(pat, case, box):
    every, diag, low, up, flops = _counts(pat)
    n, it = pat.vector_size(), _iterations(case, box)
    if case.get("precon") == "hb":
        flops, stored = 2.0 * pat.nelem * float(pat.bsize()[0] * pat.ntime) ** 3, pat.nelem * float(pat.bsize()[0] * pat.ntime) ** 2
        step, width = stored + every, 8
    else:
        # an Arnoldi step reads the factors and the matrix; U serves the sweep and the product
        step, width = diag + low + every, 4 if case.get("precision", "fp64") != "fp64" else 8
    return {"bytes": 8.0 * (every + diag + low) + it * (width * step + 8.0 * (it + 8) * n),
            "flops": flops + it * (2.0 * step + 4.0 * it * n)}


def work(case):
    if case["kind"] == "mv":
        pat = _ragged_pattern(case)
        every = _counts(pat)[0]
        return {"bytes": 8.0 * (every + 2 * pat.vector_size()), "flops": 2.0 * every}
    if case["kind"] == "batched":
        works = [_solve_work(p, case, p.shape) for p in _batch_patterns(case)]
        return {k: sum(w[k] for w in works) for k in ("bytes", "flops")}
    box = (case["nx"], case["ny"], case["nz"])
    if case["kind"] == "solve":
        return _solve_work(_pattern(*box, case["order"], case["ntime"]), case, box)
    pat = _pattern(*box, case["order"])
    every, diag, low, up, flops = _counts(pat)
    n = pat.vector_size()
    if case["kind"] == "precon":
        # the matrix in, the factors out; then the factors and U for the apply
        return {"bytes": 8.0 * (every + 2 * (diag + low) + up + 3 * n), "flops": flops + 2.0 * (diag + low + up)}
    # nodes of the quadrature: (3/2 (P+1))^3 in the volume, squared on a face;
    # the tensor-product basis is not exploited in this count
    nt = mesh.nterms_of_order(case["order"])
    nq = math.ceil(1.5 * (case["order"] + 1))
    faces = float(pat.nblocks - pat.nelem)
    flops = 2.0 * 25 * nt * (pat.nelem * (nq ** 3 * (3 + nt) + 6 * nq ** 2 * (1 + nt)) + faces * nq ** 2 * (1 + nt))
    return {"bytes": 8.0 * (2 * every + 4 * n), "flops": flops + 2.0 * every}


def tolerance(case):
    if case["kind"] in ("mv", "euler"):
        # FP64 sums in another order: 2e-16 to 1.2e-15 against `exact`, 1.8e-14
        # for the Euler residual, whose terms cancel
        return {"rel": 1e-14} if case["kind"] == "mv" else {"rel": 1e-13}
    if case["kind"] == "precon":
        return {"rel": 2e-14}                         # through block inverses: 0.8e-15 to 2.4e-15
    if case.get("precision", "fp64") != "fp64":
        return {"rel": 2e-8}                          # stopped at a residual of 1e-8, FP32 inside: 1.4e-9 to 2.4e-9
    return {"rel": 2e-14}                             # the same Arnoldi process, rounded otherwise: 0.9e-15 to 2.4e-15


# ---- the same results in plain torch ----------------------------------------------

class _BlockMatrix:
    """Equal square blocks; rows are (element, time level), element-major."""

    def __init__(self, pat, vals, transposed=False):
        self.b = b = int(pat.bsize()[0])
        self.nt, self.shape = pat.ntime, pat.shape
        dev = lambda a: torch.as_tensor(np.asarray(a, dtype=np.int64), device="cuda")
        self.row = dev(pat.blk_row_elem) * self.nt + dev(pat.blk_row_time)
        self.col = dev(pat.blk_col_elem) * self.nt + dev(pat.blk_col_time)
        self.local = dev(pat.blk_face) != mesh.OTHER
        self.V = vals.view(-1, b, b)                                   # column-major blocks
        if transposed:
            self.row, self.col = self.col, self.row
        else:
            self.V = self.V.transpose(1, 2)
        self.n = pat.nelem * self.nt

    def mv(self, x):
        y = torch.zeros(self.n, self.b, dtype=torch.float64, device="cuda")
        x = x.view(self.n, self.b)
        for k in range(0, len(self.row), 20000):
            s = slice(k, k + 20000)
            y.index_add_(0, self.row[s], torch.bmm(self.V[s], x[self.col[s], :, None])[:, :, 0])
        return y.view(-1)


class _ILU0:
    """Block ILU0: L = A_lower inv(D), D -= L A_upper, wavefront by wavefront."""

    def __init__(self, A):
        self.A, dev = A, "cuda"
        e = torch.arange(A.n, device=dev) // A.nt
        nx, ny, _ = A.shape
        front = e % nx + (e // nx) % ny + e // (nx * ny)
        key = A.row * A.n + A.col
        order = torch.argsort(key)
        lower = torch.nonzero(A.local & (A.col < A.row)).view(-1)
        upper = torch.nonzero(A.local & (A.col > A.row)).view(-1)
        mirror = order[torch.searchsorted(key[order], A.col[lower] * A.n + A.row[lower])]
        diag = torch.nonzero(A.row == A.col).view(-1)
        D = torch.empty(A.n, A.b, A.b, dtype=torch.float64, device=dev)
        D[A.row[diag]] = A.V[diag]
        self.L = torch.empty(len(lower), A.b, A.b, dtype=torch.float64, device=dev)
        self.D, self.levels = D, []
        for f in range(int(front.max()) + 1):
            rows = torch.nonzero(front == f).view(-1)
            lo = torch.nonzero(front[A.row[lower]] == f).view(-1)
            up = torch.nonzero(front[A.row[upper]] == f).view(-1)
            if len(lo):
                self.L[lo] = torch.bmm(A.V[lower[lo]], D[A.col[lower[lo]]])
                D.index_add_(0, A.row[lower[lo]], torch.bmm(self.L[lo], A.V[mirror[lo]]), alpha=-1.0)
            D[rows] = torch.linalg.inv(D[rows])
            self.levels.append((rows, lo, A.row[lower[lo]], A.col[lower[lo]], upper[up]))

    def apply(self, v):
        A = self.A
        z = v.view(A.n, A.b).clone()
        for rows, lo, r, c, up in self.levels:
            if len(lo):
                z.index_add_(0, r, torch.bmm(self.L[lo], z[c, :, None])[:, :, 0], alpha=-1.0)
        for rows, lo, r, c, up in reversed(self.levels):
            if len(up):
                z.index_add_(0, A.row[up], torch.bmm(A.V[up], z[A.col[up], :, None])[:, :, 0], alpha=-1.0)
            z[rows] = torch.bmm(self.D[rows], z[rows, :, None])[:, :, 0]
        return z.view(-1)


class _ElementInverse:
    """precon_HB: the inverse of each element's blocks over all its time levels."""

    def __init__(self, A):
        ne, w = A.n // A.nt, A.nt * A.b
        D = torch.zeros(ne, A.nt, A.nt, A.b, A.b, dtype=torch.float64, device="cuda")
        own = torch.nonzero(A.row // A.nt == A.col // A.nt).view(-1)
        D[A.row[own] // A.nt, A.row[own] % A.nt, A.col[own] % A.nt] = A.V[own]
        self.D = torch.linalg.inv(D.permute(0, 1, 3, 2, 4).reshape(ne, w, w))

    def apply(self, v):
        return torch.bmm(self.D, v.view(self.D.shape[0], -1, 1)).view(-1)


def _fgmres(A, M, b, nkrylov, rtol, nmax=300):
    """Restarted right-preconditioned FGMRES, classical Gram-Schmidt with one
    selective second pass."""
    x, steps, first = torch.zeros_like(b), 0, None
    while True:
        r = b - A.mv(x)
        beta = float(r.norm())
        first = beta if first is None else first
        V, Z = torch.empty(nkrylov + 1, b.numel(), dtype=b.dtype, device=b.device), []
        V[0] = r / beta
        H, g, rot, done = np.zeros((nkrylov + 1, nkrylov)), np.zeros(nkrylov + 1), [], False
        g[0] = beta
        for j in range(nkrylov):
            Z.append(M.apply(V[j]))
            w = A.mv(Z[j])
            before, h = float(w.norm()), np.zeros(j + 1)
            for _ in range(2):
                c = V[:j + 1] @ w
                w = w - c @ V[:j + 1]
                h += c.cpu().numpy()
                if np.abs(h).sum() / before < 1.0:
                    break
            H[:j + 1, j], H[j + 1, j] = h, float(w.norm())
            V[j + 1] = w / H[j + 1, j]
            for i, (cs, sn) in enumerate(rot):
                H[i, j], H[i + 1, j] = cs * H[i, j] + sn * H[i + 1, j], -sn * H[i, j] + cs * H[i + 1, j]
            d = math.hypot(H[j, j], H[j + 1, j])
            rot.append((H[j, j] / d, H[j + 1, j] / d))
            H[j, j], H[j + 1, j] = d, 0.0
            g[j], g[j + 1] = rot[j][0] * g[j], -rot[j][1] * g[j]
            steps += 1
            done = abs(g[j + 1]) / first < rtol or steps >= nmax
            if done:
                break
        y = np.linalg.solve(H[:j + 1, :j + 1], g[:j + 1])
        for yi, z in zip(y, Z):
            x = x + float(yi) * z
        if done:
            return x


def _euler_residual(box, q):
    """R(q) of the Euler equations on the box, q real or complex (for the
    derivative in a direction by the complex step)."""
    gam, t = euler.GAMMA, lambda a: torch.as_tensor(np.ascontiguousarray(a), dtype=torch.float64, device="cuda")
    nt, nx, ny, nz = box.nterms, *box.shape
    h = [1.0 / s for s in box.shape]
    xg, wg = np.polynomial.legendre.leggauss(math.ceil(1.5 * (box.order + 1)))
    basis = [np.polynomial.legendre.Legendre.basis(k) for k in range(box.order + 1)]
    val, der, end = (np.array([f(p) for p in basis]) for f in (
        lambda p: p(xg), lambda p: p.deriv()(xg), lambda p: p(np.array([-1.0, 1.0]))))
    a, b, c = euler.MODE_ORDER[:nt].T
    U = q.view(-1, NFIELDS, nt)
    mix = lambda P, W: torch.einsum("qm,efm->eqf", t(P).to(W.dtype), W)
    grid = lambda A, B, C: np.einsum("mi,mj,mk->ijkm", A, B, C).reshape(-1, nt)
    wv = np.einsum("i,j,k->ijk", wg, wg, wg).reshape(-1)
    wf = np.einsum("i,j->ij", wg, wg).reshape(-1)

    def state(Q):
        rho, m, E = Q[..., 0], [Q[..., i] for i in (1, 2, 3)], Q[..., 4]
        p = (gam - 1.0) * (E - 0.5 * (m[0] ** 2 + m[1] ** 2 + m[2] ** 2) / rho)
        return rho, m, E, p

    def flux(Q, d):
        rho, m, E, p = state(Q)
        u = m[d] / rho
        f = [m[d]] + [mi * u for mi in m] + [(E + p) * u]
        f[1 + d] = f[1 + d] + p
        return torch.stack(f, -1)

    def absval(z):
        return z * torch.sign(z.real)

    def roe(QL, QR, d):
        (rl, ml, El, pl), (rr, mr, Er, pr) = state(QL), state(QR)
        sl, sr = torch.sqrt(rl), torch.sqrt(rr)
        mean = lambda p, s: (sl * p + sr * s) / (sl + sr)
        ul, ur = [m / rl for m in ml], [m / rr for m in mr]
        u, H, rho = [mean(p, s) for p, s in zip(ul, ur)], mean((El + pl) / rl, (Er + pr) / rr), torch.sqrt(rl * rr)
        k2 = u[0] ** 2 + u[1] ** 2 + u[2] ** 2
        cc = torch.sqrt((gam - 1.0) * (H - 0.5 * k2))
        du, dp, eps = [p - s for p, s in zip(ul, ur)], pl - pr, 0.01 * cc

        def speed(l):
            l = absval(l)
            return torch.where(l.real < eps.real, 0.5 * (eps + l * l / eps), l)

        k1 = speed(u[d] - cc) * (dp - rho * cc * du[d]) / (2.0 * cc * cc)
        k3 = speed(u[d] + cc) * (dp + rho * cc * du[d]) / (2.0 * cc * cc)
        ke, ks = speed(u[d]) * ((rl - rr) - dp / (cc * cc)), speed(u[d]) * rho
        out = [k1 + ke + k3]
        for i in range(3):
            n = 1.0 if i == d else 0.0
            out.append(k1 * (u[i] - cc * n) + ke * u[i] + ks * (du[i] - du[d] * n) + k3 * (u[i] + cc * n))
        turn = u[0] * du[0] + u[1] * du[1] + u[2] * du[2] - u[d] * du[d]
        out.append(k1 * (H - cc * u[d]) + ke * 0.5 * k2 + ks * turn + k3 * (H + cc * u[d]))
        return 0.5 * torch.stack(out, -1)

    def farfield(Q, d, sign):
        rho, m, E, p = state(Q)
        ui, ri, pi = box.vel_inf, box.rho_inf, box.p_inf
        inflow = (m[d] * sign).real <= euler.RKTOL
        um = [x / rho for x in m]
        minus = ui[d] * sign - 2.0 * math.sqrt(gam * pi / ri) / (gam - 1.0)
        plus = um[d] * sign + 2.0 * torch.sqrt(gam * p / rho) / (gam - 1.0)
        cb, un = (gam - 1.0) / 4.0 * (plus - minus), 0.5 * (plus + minus)
        pick = lambda i, o: torch.where(inflow, torch.full_like(o, i), o)
        entropy = pick(pi / ri ** gam, p / rho ** gam)
        rb = (cb * cb / (entropy * gam)) ** (1.0 / (gam - 1.0))
        ub = [un * sign if i == d else pick(ui[i], um[i]) for i in range(3)]
        return torch.stack([rb] + [rb * x for x in ub] +
                           [entropy * rb ** gam / (gam - 1.0) + 0.5 * rb * (ub[0] ** 2 + ub[1] ** 2 + ub[2] ** 2)], -1)

    R = torch.zeros_like(U)
    put = lambda P, w, F: torch.einsum("qm,eqf->efm", t(P * w[:, None]).to(F.dtype), F)
    jac = h[0] * h[1] * h[2] / 8.0
    Q = mix(grid(val[a], val[b], val[c]), U)
    for d in range(3):
        G = grid(*(der[s] if i == d else val[s] for i, s in enumerate((a, b, c)))) * (2.0 / h[d])
        R -= jac * put(G, wv, flux(Q, d))
    e = torch.arange(nx * ny * nz, device="cuda")
    pos = (e % nx, (e // nx) % ny, e // (nx * ny))
    for d, (count, stride) in enumerate(zip(box.shape, (1, nx, nx * ny))):
        area = jac * 2.0 / h[d]
        face = []
        for side in range(2):
            s = [val[a], val[b], val[c]]
            s[d] = end[(a, b, c)[d], side][:, None]
            face.append(np.einsum("mi,mj,mk->ijkm", *s).reshape(-1, nt))
        L = e[pos[d] < count - 1]
        if len(L):
            QL, QR = mix(face[1], U[L]), mix(face[0], U[L + stride])
            I = area * (0.5 * (flux(QL, d) + flux(QR, d)) + roe(QL, QR, d))
            R[L] += put(face[1], wf, I)
            R[L + stride] -= put(face[0], wf, I)
        for side, sign in ((0, -1.0), (1, 1.0)):
            B = e[pos[d] == (0 if side == 0 else count - 1)]
            R[B] += put(face[side], wf, area * sign * flux(farfield(mix(face[side], U[B]), d, sign), d))
    return R.reshape(-1)


def exact(case, seed):
    if case["kind"] == "euler":
        box, q, v = _euler_inputs(case, seed)
        step = 1e-30
        out = _euler_residual(box, torch.complex(q, step * v))
        return {"r": out.real.clone(), "jv": out.imag / step}
    pat, vals, v = _inputs(case, seed)
    if case["kind"] == "mv":
        (nr, nc), (first, _) = pat.block_dims(), pat.value_offsets()
        off = pat.elem_offsets()
        y = torch.zeros_like(v)
        for m, n in sorted(set(zip(nr.tolist(), nc.tolist()))):
            k = np.nonzero((nr == m) & (nc == n))[0]
            at = lambda o, count: torch.as_tensor(o, device="cuda")[:, None] + torch.arange(count, device="cuda")
            blocks = vals[at(first[k], m * n)].view(-1, n, m).transpose(1, 2)
            prod = torch.bmm(blocks, v[at(off[np.asarray(pat.blk_col_elem)[k]], n)][:, :, None])[:, :, 0]
            y.index_add_(0, at(off[np.asarray(pat.blk_row_elem)[k]], m).reshape(-1), prod.reshape(-1))
        return y
    if case["kind"] == "precon":
        return _ILU0(_BlockMatrix(pat, vals)).apply(v)
    if case["kind"] == "batched":
        xs, iv, ix = [], 0, 0
        for p in _batch_patterns(case):
            nv, n = p.value_offsets()[1], p.vector_size()
            A = _BlockMatrix(p, vals[iv:iv + nv])
            xs.append(_fgmres(A, _ILU0(A), v[ix:ix + n], case["nkrylov"], RTOL))
            iv, ix = iv + nv, ix + n
        return torch.cat(xs)
    A = _BlockMatrix(pat, vals, case["adjoint"])
    M = _ElementInverse(A) if case["precon"] == "hb" else _ILU0(A)
    if case["precision"] != "fp64":
        return _fgmres(A, M, v, 100, 1e-12)
    return _fgmres(A, M, v, case["nkrylov"], RTOL)
