"""What a program that uses this framework has it do: factor and solve hybridized quad-mesh
block systems, through the handle (``native.NativeSystem``), the batch of independent
systems (``batch.BatchedSystem``) and the drop-in class (``hybsol.BlockSystem``).

Every case is a mesh of ``n x n`` elements: an element carries one block of ``p*p`` unknowns,
an edge one block of ``max(p)`` over its elements, with N(0,1)/sqrt(columns) couplings and
diagonal blocks shifted by ``shift`` times (the Frobenius norms of the row's couplings + 1).
``p`` is one order, or drawn per element from ``p .. pmax``. Kinds of pass:

* ``step``  -- one step of a time-stepping or Newton loop on a kept handle: new values from
  device memory, a factorization, a solve;
* ``solve`` -- the same with the factors kept: a solve for new right-hand sides only;
* ``many``  -- independent systems stacked on one handle, factored and solved together with
  right-hand sides and solutions in host memory;
* ``once``  -- the drop-in class on host data, from the assembled blocks to the solution: the
  whole life of a system that is solved once.
"""

import random
import sys
from pathlib import Path

import numpy as np
import torch

sys.path.insert(0, str(Path(__file__).resolve().parents[1] / "hybridized-solver_b200"))

DEV = "cuda"
F64 = torch.float64


def listed():
    return [
        # the smallest system in earnest: every stage is launch latency
        _case("tiny_fp64", "step", n=8, p=3),
        # the reference's own benchmark mesh (16x16, p=4) on a kept handle
        _case("mesh16_p4_fp64", "step", n=16, p=4),
        # an odd mesh of middling blocks (36 and 6 rows): padded 64-row pivots
        _case("mesh25_p6_fp64", "step", n=25, p=6),
        # an ordinary p=8 mesh in the plain form: one element per stage, too little work to fill the chip
        _case("mesh24_p8_fp64", "step", n=24, p=8),
        # a large p=8 mesh in the plain form: bound by the FP64 updates
        _case("mesh64_p8_fp64", "step", n=64, p=8),
        # the mixed form on an odd, ordinary p=8 mesh
        _case("mesh31_p8_mixed", "step", n=31, p=8, precision="mixed"),
        # the mixed form on the largest mesh whose state fits the card three times over
        _case("mesh96_p8_mixed", "step", n=96, p=8, precision="mixed"),
        # an ill-conditioned value set (condition number about 1e6): several refinement steps
        _case("reduced32_p8_mixed", "step", n=32, p=8, precision="mixed", shift=0.2013112914936568),
        # uneven orders 2..10 (blocks of 4 to 100 rows), four right-hand sides
        _case("uneven32_fp64", "step", n=32, p=2, pmax=10, nrhs=4),
        # many independent systems in one handle, four right-hand sides each
        _case("many24_mixed", "many", n=8, nmax=24, count=24, p=3, pmax=6, nrhs=4, precision="mixed"),
        # a time step with the factors kept
        _case("solve40_p8_fp64", "solve", n=40, p=8),
        # build, factor and solve once with the drop-in class
        _case("once12_p5_fp64", "once", n=12, p=5),
    ]


def _case(name, kind, n, p, pmax=0, nmax=0, count=1, nrhs=1, precision="fp64", shift=1.0):
    c = dict(kind=kind, n=n, p=p, pmax=pmax, nmax=nmax, count=count, nrhs=nrhs, precision=precision, shift=shift)
    return dict(name=name, **c) if name else c


def _log(rng, lo, hi):
    return int(round(lo * (hi / lo) ** rng.random()))


def draw(rng: random.Random):
    kind = rng.choice(["step", "step", "step", "step", "uneven", "solve", "many", "once"])
    precision = rng.choice(["fp64", "mixed"])
    if kind == "step":
        # whole range of orders; the plain form and orders without 64-row blocks cost more per element
        p = rng.choice([8, 8, 8, 8, 3, 4, 5, 6, 7, 10])
        top = 64 if p < 8 else 90 if (p == 8 and precision == "mixed") else 60 if p == 8 else 40
        return _case(None, "step", n=_log(rng, 8, top), p=p, nrhs=rng.choice([1, 1, 2]), precision=precision)
    if kind == "uneven":
        lo = rng.choice([2, 3])
        return _case(None, "step", n=_log(rng, 8, 40), p=lo, pmax=rng.choice([6, 8, 9, 10]), nrhs=rng.randint(1, 5),
                     precision=precision)
    if kind == "solve":
        return _case(None, "solve", n=_log(rng, 12, 56), p=rng.choice([4, 6, 8, 8]), nrhs=rng.choice([1, 2, 3, 8]),
                     precision=precision)
    if kind == "many":
        n = rng.randint(6, 12)
        return _case(None, "many", n=n, nmax=n + rng.randint(4, 14), count=rng.randint(8, 30), p=3, pmax=rng.randint(4, 6),
                     nrhs=rng.randint(1, 4), precision=precision)
    return _case(None, "once", n=_log(rng, 6, 24), p=rng.choice([3, 4, 5, 6, 8]), nrhs=rng.choice([1, 3]), precision=precision)


# ---------------------------------------------------------------------------------------
# The meshes of a case, their patterns and their values.


def _meshes(case):
    """Per system: (elements per side, orders of the elements)."""
    rng = np.random.default_rng(case["n"] * 1000 + case["count"])
    out = []
    for _ in range(case["count"]):
        n = int(rng.integers(case["n"], case["nmax"] + 1)) if case["nmax"] else case["n"]
        if case["kind"] == "many":  # one order per system
            out.append((n, np.full(n * n, rng.integers(case["p"], case["pmax"] + 1))))
        elif case["pmax"]:
            out.append((n, rng.integers(case["p"], case["pmax"] + 1, n * n)))
        else:
            out.append((n, np.full(n * n, case["p"])))
    return out


class _Mesh:
    """Sizes and couplings in the natural numbering: elements, horizontal edges, vertical edges."""

    def __init__(self, n, orders):
        ne, x, y = n * n, np.arange(n * n) % n, np.arange(n * n) // n
        h, v = ne, ne + n * (n + 1)
        self.ne, self.nf = ne, 2 * n * (n + 1)
        self.edges = np.stack([h + y * n + x, h + (y + 1) * n + x, v + y * (n + 1) + x, v + y * (n + 1) + x + 1], 1)
        order = np.zeros(ne + self.nf, np.int64)
        for k in range(4):
            np.maximum.at(order, self.edges[:, k], orders)
        order[:ne] = orders * orders
        self.sizes = order
        # blocks by where their values lie: (E) element diagonals, (U) element x edge, (L) edge x element, (F) edge diagonals
        e, k = np.repeat(np.arange(ne), 4), np.tile(np.arange(4), ne)
        f = self.edges.ravel()
        rows = np.concatenate([np.arange(ne), e, f, np.arange(ne, ne + self.nf)])
        cols = np.concatenate([np.arange(ne), f, e, np.arange(ne, ne + self.nf)])
        self.P, self.Q = int(self.sizes[:ne].max()), int(self.sizes[ne:].max())
        P, Q = self.P, self.Q
        at = [np.arange(ne) * P * P, ne * P * P + (e * 4 + k) * P * Q, ne * P * P + 4 * ne * P * Q + (e * 4 + k) * P * Q,
              ne * P * P + 8 * ne * P * Q + np.arange(self.nf) * Q * Q]
        stride = np.concatenate([np.full(ne, P), np.full(4 * ne, Q), np.full(4 * ne, P), np.full(self.nf, Q)])
        self.rows, self.cols, self.at, self.stride = rows, cols, np.concatenate(at), stride

    def pattern(self, order):
        """(sizes, row_ptr, cols, which block comes at each place) with block i renumbered order[i]."""
        r, c = order[self.rows], order[self.cols]
        which = np.lexsort((c, r))
        sizes = np.empty_like(self.sizes)
        sizes[order] = self.sizes
        return sizes, np.concatenate([[0], np.cumsum(np.bincount(r, minlength=len(sizes)))]), c[which], which


def _padded(mesh, seed, shift, nrhs):
    """Values on the device, padded to the largest block: E, U, L, F (diagonal padding one, the rest zero) and b."""
    g = torch.Generator(DEV).manual_seed(int(seed))
    P, Q = mesh.P, mesh.Q
    se = torch.from_numpy(mesh.sizes[: mesh.ne]).to(DEV)
    sf = torch.from_numpy(mesh.sizes[mesh.ne :]).to(DEV)
    f = torch.from_numpy(mesh.edges - mesh.ne).to(DEV)
    ie = (torch.arange(P, device=DEV) < se[:, None]).to(F64)
    jf = (torch.arange(Q, device=DEV) < sf[:, None]).to(F64)
    draw_ = lambda *s: torch.randn(*s, generator=g, device=DEV, dtype=F64)  # noqa: E731
    U = draw_(mesh.ne, 4, P, Q) / sf[f][..., None, None].sqrt() * ie[:, None, :, None] * jf[f][:, :, None, :]
    L = draw_(mesh.ne, 4, Q, P) / se[:, None, None, None].sqrt() * ie[:, None, None, :] * jf[f][:, :, :, None]
    norm_e = U.square().sum((2, 3)).sqrt().sum(1)
    norm_f = torch.zeros(mesh.nf, device=DEV, dtype=F64)
    for k in range(4):  # an edge is each side's at most once: no order to depend on
        norm_f[f[:, k]] += L[:, k].square().sum((1, 2)).sqrt()
    E = draw_(mesh.ne, P, P) / se[:, None, None].sqrt() * ie[:, :, None] * ie[:, None, :]
    F = draw_(mesh.nf, Q, Q) / sf[:, None, None].sqrt() * jf[:, :, None] * jf[:, None, :]
    E.diagonal(dim1=1, dim2=2).add_(ie * (shift * (norm_e + 1))[:, None] + (1 - ie))
    F.diagonal(dim1=1, dim2=2).add_(jf * (shift * (norm_f + 1))[:, None] + (1 - jf))
    be = (2 * torch.rand(mesh.ne, P, nrhs, generator=g, device=DEV, dtype=F64) - 1) * ie[..., None]
    bf = (2 * torch.rand(mesh.nf, Q, nrhs, generator=g, device=DEV, dtype=F64) - 1) * jf[..., None]
    return E, U, L, F, be, bf, ie, jf, f


def _values(mesh, pad, which):
    """The blocks `which`, row-major one after the other."""
    src = torch.cat([t.reshape(-1) for t in pad[:4]])
    nr, nc = mesh.sizes[mesh.rows[which]], mesh.sizes[mesh.cols[which]]
    count = torch.from_numpy(nr * nc).to(DEV)
    start = torch.cumsum(count, 0) - count
    put = lambda a: torch.repeat_interleave(torch.from_numpy(a).to(DEV) if isinstance(a, np.ndarray) else a, count)  # noqa: E731
    t = torch.arange(int(count.sum()), device=DEV) - put(start)
    w = put(nc.astype(np.int64))
    i = torch.div(t, w, rounding_mode="floor")
    t -= i * w
    return src[put(mesh.at[which]) + i * put(mesh.stride[which]) + t]


def _vector(e, f, ie, jf, edges_first, nrhs):
    """Padded element and edge vectors as one (dof,) or (dof, nrhs) vector."""
    parts = [e[ie > 0], f[jf > 0]]
    v = torch.cat(parts[::-1] if edges_first else parts)
    return v[:, 0].contiguous() if nrhs == 1 else v.contiguous()


# ---------------------------------------------------------------------------------------


def prepare(case, seed):
    from hybsol.b200 import batch, meshgen, native

    precision = native.MIXED if case["precision"] == "mixed" else native.FP64
    state = dict(kind=case["kind"], precision=precision, nrhs=case["nrhs"])
    meshes = [_Mesh(n, orders) for n, orders in _meshes(case)]
    if case["kind"] in ("step", "solve"):
        mesh = meshes[0]
        pad = _padded(mesh, seed, case["shift"], case["nrhs"])
        _, row_ptr, cols, _ = mesh.pattern(np.arange(len(mesh.sizes)))
        order = native.compute_ordering(row_ptr, cols, "first").astype(np.int64)
        sizes, row_ptr, cols, which = mesh.pattern(order)
        state["system"] = native.NativeSystem(sizes, row_ptr, cols)
        state["values"] = _values(mesh, pad, which)
        # the ordering places every edge before every element and keeps their order
        state["b"] = _vector(pad[4], pad[5], pad[6], pad[7], True, case["nrhs"])
        state["x"] = torch.empty_like(state["b"])
        torch.cuda.synchronize()
        if case["kind"] == "solve":
            state["system"].set_values(state["values"], device=True)
            state["system"].decompose(precision)
        return state
    mats, rhs = [], []
    for s, mesh in enumerate(meshes):
        pad = _padded(mesh, seed * 1000 + s, case["shift"], case["nrhs"])
        sizes, row_ptr, cols, which = mesh.pattern(np.arange(len(mesh.sizes)))
        nval = sizes[mesh.rows[which]] * sizes[cols]
        vals = _values(mesh, pad, which).cpu().numpy()
        mats.append(meshgen.BlockMatrix(sizes, row_ptr, cols, np.concatenate([[0], np.cumsum(nval)]), vals))
        rhs.append(_vector(pad[4], pad[5], pad[6], pad[7], False, case["nrhs"]).cpu().numpy())
    if case["kind"] == "many":
        state["system"], state["b"] = batch.BatchedSystem(mats), rhs
        return state
    import hybsol

    state["precision"] = case["precision"]
    m = mats[0]
    system = hybsol.BlockSystem(*(int(s) for s in m.sizes))
    system.add_blocks(np.repeat(np.arange(len(m.sizes)), np.diff(m.row_ptr)), m.cols, m.vals)
    state["order"] = system.compute_reordering("first")
    system.reorder_blocks(state["order"])
    state["system"], state["b"] = system, rhs[0]
    return state


def run(state):
    system = state["system"]
    if state["kind"] == "step":
        system.set_values(state["values"], device=True)
        system.decompose(state["precision"])
    if state["kind"] in ("step", "solve"):
        system.solve_device(state["b"], state["x"], state["nrhs"])
        return state["x"]
    if state["kind"] == "many":
        system.decompose(state["precision"])
        return system.solve(state["b"])[0]
    new = system.copy()  # decompose() consumes the assembled blocks
    new.decompose(precision=state["precision"])
    order, b = state["order"], state["b"]
    if b.ndim == 1:  # unorder_vector maps to the reordered layout, reorder_vector back
        return new.reorder_vector(order, new.solve(new.unorder_vector(order, b)))
    # both take one vector at a time
    x = new.solve(np.stack([new.unorder_vector(order, c) for c in np.ascontiguousarray(b.T)], 1))
    return np.stack([new.reorder_vector(order, c) for c in np.ascontiguousarray(x.T)], 1)


def work(case):
    """Each input and output once: the values (a step), the factors written (a step) or read (a solve), b and x."""
    from hybsol.b200 import native

    total = dict(bytes=0.0, flops=0.0)
    word = 4 if case["precision"] == "mixed" else 8
    for n, orders in _meshes(case):
        mesh = _Mesh(n, orders)
        order = np.concatenate([mesh.nf + np.arange(mesh.ne), np.arange(mesh.nf)])
        sizes, row_ptr, cols, which = mesh.pattern(order)
        a = native.analyze(sizes, row_ptr, cols)
        values = float((mesh.sizes[mesh.rows] * mesh.sizes[mesh.cols]).sum())
        total["bytes"] += word * a["factor_values"] + 16.0 * sizes.sum() * case["nrhs"]
        total["flops"] += 2.0 * a["factor_values"] * case["nrhs"]
        if case["kind"] != "solve":
            total["bytes"] += 8 * values
            total["flops"] += a["factor_flops"]
    return {k: float(v) for k, v in total.items()}


# ---------------------------------------------------------------------------------------


def _solve64(mesh, pad, shift):
    """The solution by eliminating the elements first, in batched torch; None where that is too large."""
    E, U, L, F, be, bf, _, _, f = pad
    nrhs, ne, nf, Q = be.shape[2], mesh.ne, mesh.nf, mesh.Q
    U4, L4 = U.permute(0, 2, 1, 3).reshape(ne, mesh.P, 4 * Q), L.reshape(ne, 4 * Q, mesh.P)
    lu = torch.linalg.lu_factor(E)
    EU = torch.linalg.lu_solve(*lu, U4)
    place = (f[:, :, None] * Q + torch.arange(Q, device=DEV)).reshape(ne, 4 * Q)
    S = L4 @ EU
    if nf * Q <= 20000:
        A = torch.zeros(nf, Q, nf, Q, device=DEV, dtype=F64)
        A[torch.arange(nf), :, torch.arange(nf), :] = F
        A = A.view(nf * Q, nf * Q)
        A.index_put_((place[:, :, None].expand(-1, -1, 4 * Q), place[:, None, :].expand(-1, 4 * Q, -1)), -S, accumulate=True)
        A = torch.linalg.lu_factor(A)
        inner = lambda g: torch.linalg.lu_solve(*A, g.reshape(nf * Q, nrhs)).view(nf, Q, nrhs)  # noqa: E731
        steps = 3
    elif shift >= 1:  # diagonally dominant: block Jacobi contracts fast
        Flu = torch.linalg.lu_factor(F)
        inner = lambda g: torch.linalg.lu_solve(*Flu, g)  # noqa: E731
        steps = 60
    else:
        return None
    xe, xf = torch.zeros_like(be), torch.zeros_like(bf)
    for _ in range(steps):
        re = be - E @ xe - U4 @ xf.reshape(nf * Q, nrhs)[place]
        rf = bf.reshape(nf * Q, nrhs) - (F @ xf).reshape(nf * Q, nrhs)
        rf = rf.index_add(0, place.reshape(-1), (L4 @ (xe + torch.linalg.lu_solve(*lu, re))).reshape(-1, nrhs), alpha=-1)
        df = inner(rf.view(nf, Q, nrhs))
        xe = xe + torch.linalg.lu_solve(*lu, re) - EU @ df.reshape(nf * Q, nrhs)[place]
        xf = xf + df
    return xe, xf


def exact(case, seed):
    many, out = case["kind"] in ("many", "once"), []
    for s, (n, orders) in enumerate(_meshes(case)):
        mesh = _Mesh(n, orders)
        pad = _padded(mesh, seed * 1000 + s if many else seed, case["shift"], case["nrhs"])
        x = _solve64(mesh, pad, case["shift"])
        if x is None:
            return None
        out.append(_vector(x[0], x[1], pad[6], pad[7], not many, case["nrhs"]))
    return out if case["kind"] == "many" else out[0]
