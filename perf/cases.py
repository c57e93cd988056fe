"""The calls whose speed counts: what programs do with the solver, over the sizes they do it at.

Kinds of case, all through the package's public entry points:

* ``hsolve``  -- fastSolver2's own call ``hsolve(nrow, nrhs, rank, nPart, LD, K, U, V)`` on the reference's inputs
  (uniform U and V shared by all levels, D + 1000 on the diagonal), in place, from device or host buffers.
* ``system``  -- a kept handle takes a new matrix of its shape (leaf blocks, bases of every level), factors it and
  solves for its right-hand sides.
* ``resolve`` -- a kept factorisation solves for new right-hand sides, with A and with A^T.
* ``adjoint`` -- a training step: new matrix, factor, solve, and the gradients of L = ||x||^2 / 2 with respect to
  b, D, U, V and s.
* ``batch``   -- many independent systems of different shapes: new matrices, one factorisation, one solve.
"""
import math
import random

import numpy as np
import torch

import fastsolver2_gb300 as fs

F64 = torch.float64


def listed():
    return [
        # the reference's smallest test problem through its own entry point: launches and host work are the time
        {"name": "hsolve_n512", "kind": "hsolve", "leaf": 64, "levels": 3, "rank": 8, "nrhs": 1, "host": False},
        # the reference's default leaf size and rank, called as its host code calls it: numpy buffers in place
        {"name": "hsolve_host_n1600", "kind": "hsolve", "leaf": 400, "levels": 2, "rank": 10, "nrhs": 1, "host": True},
        # the reference's CPU-size problem: one small matrix after another in a host loop
        {"name": "fp64_n4096", "kind": "system", "leaf": 256, "levels": 4, "rank": 16, "nrhs": 1, "mixed": False,
         "shift": 4.0, "decay": 0.0},
        # an ordinary FP64 system with a block of right-hand sides
        {"name": "fp64_n64k", "kind": "system", "leaf": 128, "levels": 9, "rank": 32, "nrhs": 8, "mixed": False,
         "shift": 4.0, "decay": 0.0},
        # the largest: FP64 at N = 2^20 with 64 right-hand sides
        {"name": "fp64_n1m", "kind": "system", "leaf": 128, "levels": 13, "rank": 32, "nrhs": 64, "mixed": False,
         "shift": 4.0, "decay": 0.0},
        # ordinary mixed-precision system
        {"name": "mixed_n128k", "kind": "system", "leaf": 128, "levels": 10, "rank": 24, "nrhs": 16, "mixed": True,
         "shift": 4.0, "decay": 0.0},
        # the benchmark workload: decaying singular values, weaker diagonal, mixed precision
        {"name": "mixed_n1m", "kind": "system", "leaf": 128, "levels": 13, "rank": 32, "nrhs": 64, "mixed": True,
         "shift": 1.5, "decay": 6.0},
        # leaf size, rank and column count that no tile divides
        {"name": "fp64_odd", "kind": "system", "leaf": 100, "levels": 8, "rank": 13, "nrhs": 5, "mixed": False,
         "shift": 4.0, "decay": 0.0},
        # time stepping or Krylov use: the factors are kept, single vectors come one after another, both directions
        {"name": "resolve_n256k", "kind": "resolve", "leaf": 128, "levels": 11, "rank": 16, "nrhs": 1, "mixed": False,
         "shift": 4.0, "decay": 0.0},
        # a training step at the size of the adjoint benchmark
        {"name": "adjoint_n256k", "kind": "adjoint", "leaf": 128, "levels": 11, "rank": 24, "nrhs": 1, "mixed": False,
         "shift": 4.0, "decay": 0.0},
        # ragged batches, N log-uniform in 2^10 .. 2^16
        {"name": "batch_fp64", "kind": "batch", "count": 64, "shapes": 11, "mixed": False, "shift": 4.0},
        {"name": "batch_mixed", "kind": "batch", "count": 64, "shapes": 12, "mixed": True, "shift": 4.0},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["hsolve", "system", "system", "system", "resolve", "adjoint", "batch"])
    if kind == "batch":
        return {"kind": "batch", "count": _log_int(rng, 4, 64), "shapes": rng.randrange(1 << 20),
                "mixed": rng.random() < 0.5, "shift": 4.0}
    # tuned leaf sizes as often as others; the row count log-uniform
    leaf = rng.choice([64, 128, 256]) if rng.random() < 0.5 else _log_int(rng, 48, 300)
    if kind == "hsolve":
        levels = rng.randint(1, 5)
        return {"kind": "hsolve", "leaf": leaf, "levels": levels, "rank": rng.randint(1, min(32, leaf // 4)),
                "nrhs": rng.randint(1, 8), "host": rng.random() < 0.5}
    levels = max(2, int(round(math.log2(rng.uniform(1.0, 2.0) * 2 ** rng.uniform(11, 17.5) / leaf))))
    rank = rng.choice([8, 16, 24, 32, 48, 64]) if rng.random() < 0.5 else rng.randint(4, 64)
    case = {"kind": kind, "leaf": leaf, "levels": levels, "rank": min(rank, leaf // 2),
            "nrhs": _log_int(rng, 1, 64) if kind != "adjoint" else _log_int(rng, 1, 8),
            "mixed": kind != "adjoint" and rng.random() < 0.5, "shift": 4.0, "decay": 0.0}
    if rng.random() < 0.3:
        case.update(shift=2.0, decay=6.0)
    return case


# ------------------------------------------------------------------ inputs
def _gen(seed, device="cuda"):
    g = torch.Generator(device=device)
    g.manual_seed(seed)
    return g


def _normal(g, rows, cols, scale=1.0):
    """N(0, scale^2), rows x cols, column-major."""
    return torch.randn((cols, rows), generator=g, dtype=F64, device="cuda").mul_(scale).t()


def _leaf_blocks(g, nleaf, m, shift):
    """[leaf][column][row]: G / sqrt(m) + shift I."""
    D = torch.randn((nleaf, m, m), generator=g, dtype=F64, device="cuda").mul_(1.0 / math.sqrt(m))
    D.diagonal(dim1=1, dim2=2).add_(shift)
    return D


def _matrix(g, leaf, levels, rank, shift, decay):
    n = leaf << levels
    D = _leaf_blocks(g, 1 << levels, leaf, shift)
    U, V, s = [], [], []
    for l in range(levels):
        c = 1.0 / math.sqrt(n >> (l + 1))
        U.append(_normal(g, n, rank, c))
        V.append(_normal(g, n, rank, c))
        s.append(torch.tensor([10.0 ** (-decay * i / rank) for i in range(rank)], dtype=F64, device="cuda"))
    return D, U, V, s


def _batch_shapes(case):
    """(n, leaf, levels, rank, nrhs) of every system of a batch."""
    r = random.Random(case["shapes"])
    out = []
    for _ in range(case["count"]):
        leaf = r.choice([64, 128, 256])
        levels = max(1, int(round(r.uniform(10.0, 16.0) - math.log2(leaf))))
        rank = r.choice([x for x in (8, 16, 32, 64) if x < leaf])
        out.append((leaf << levels, leaf, levels, rank, r.randint(1, 8)))
    return out


def _hsolve_inputs(case, seed):
    m, L, r, k = case["leaf"], case["levels"], case["rank"], case["nrhs"]
    n = m << L
    g = _gen(seed, "cpu")
    rand = lambda rows, cols: torch.rand((cols, rows), generator=g, dtype=F64).t()  # noqa: E731
    u, v, b, d = rand(n, r), rand(n, r), rand(n, k), rand(n, 1)[:, 0] + 1000.0
    blocks = torch.bmm(u.reshape(-1, m, r), v.reshape(-1, m, r).transpose(1, 2)) + torch.diag_embed(d.reshape(-1, m))
    col = lambda t: t.t().contiguous().t()  # noqa: E731
    return col(blocks.reshape(n, m)), col(torch.cat([b] + [u] * L, dim=1)), col(v)


def _systems(case, seed):
    """The matrices and right-hand sides of a case: (shape, (D, U, V, s), B) per system."""
    if case["kind"] == "batch":
        shapes = _batch_shapes(case)
        decay = 0.0
    else:
        m, L = case["leaf"], case["levels"]
        shapes, decay = [(m << L, m, L, case["rank"], case["nrhs"])], case["decay"]
    g = _gen(seed)
    out = []
    for n, m, L, r, k in shapes:
        A = _matrix(g, m, L, r, case["shift"], decay)
        out.append(((n, m, L, r, k), A, _normal(g, n, k)))
    return out


# ------------------------------------------------------------------- calls
def _set(solver, shape, A):
    m = shape[1]
    D, U, V, s = A
    solver.set_leaf_blocks(D.reshape(-1), ld=m, leaf_stride=m * m)
    for l in range(shape[2]):
        solver.set_lowrank(l, U[l], V[l], s[l])


def _copy(B):
    """A column-major copy (the solves are in place)."""
    return B.t().clone().t()


def prepare(case, seed):
    if case["kind"] == "hsolve":
        K, U, V = _hsolve_inputs(case, seed)
        st = {"case": case}
        if case["host"]:
            st.update(K=K.numpy(), U=U.numpy(), V=V.numpy())
        else:
            dev = lambda t: t.t().cuda().t()  # noqa: E731
            st.update(K=dev(K), U=dev(U), V=dev(V), stream=torch.cuda.Stream())
            torch.cuda.synchronize()
        return st
    systems = _systems(case, seed)
    prec = fs.PREC_MIXED if case["mixed"] else fs.PREC_FP64
    stream = torch.cuda.Stream()
    st = {"case": case, "systems": systems, "stream": stream}
    if case["kind"] == "batch":
        st["batch"] = fs.Batch([x[0] for x in systems], precision=prec, stream=stream.cuda_stream)
    else:
        (n, m, L, r, k), A, B = systems[0]
        st["solver"] = fs.Solver(n, m, L, r, nrhs_max=k, precision=prec, stream=stream.cuda_stream)
        if case["kind"] == "adjoint":
            e = lambda c: torch.empty(c, dtype=F64, device="cuda")  # noqa: E731
            st["grads"] = {"db": e(n * k).reshape(k, n).t(), "dD": e(n * m), "dU": e(L * n * r), "dV": e(L * n * r),
                           "ds": e(L * r)}
    torch.cuda.synchronize()
    if case["kind"] == "resolve":
        _set(st["solver"], systems[0][0], systems[0][1])
        st["solver"].factor()
    return st


def run(st):
    case = st["case"]
    kind = case["kind"]
    if kind == "hsolve":
        m, L, r, k = case["leaf"], case["levels"], case["rank"], case["nrhs"]
        n = m << L
        if case["host"]:
            K, U = st["K"].copy(order="F"), st["U"].copy(order="F")
            fs.hsolve(n, k, r, 1 << L, n, K, U, st["V"])
            return {"K": K, "U": U}
        with torch.cuda.stream(st["stream"]):
            K, U = _copy(st["K"]), _copy(st["U"])
            fs.hsolve(n, k, r, 1 << L, n, K, U, st["V"], stream=st["stream"].cuda_stream)
        return {"K": K, "U": U}
    systems = st["systems"]
    with torch.cuda.stream(st["stream"]):
        if kind == "batch":
            b = st["batch"]
            for i, (shape, (D, U, V, s), B) in enumerate(systems):
                m = shape[1]
                b.set_leaf_blocks(i, D.reshape(-1), ld=m, leaf_stride=m * m)
                for l in range(shape[2]):
                    b.set_lowrank(i, l, U[l], V[l])
            b.factor()
            Xs = [_copy(x[2]) for x in systems]
            b.solve(Xs)
            return torch.cat([X.t().reshape(-1) for X in Xs])
        solver, (shape, A, B) = st["solver"], systems[0]
        if kind == "resolve":
            X, Y = _copy(B), _copy(B)
            solver.solve(X)
            solver.solve(Y, transpose=True)
            return {"x": X, "y": Y}
        _set(solver, shape, A)
        solver.factor()
        X = _copy(B)
        solver.solve(X)
        if kind == "system":
            return X
        gr = st["grads"]
        solver.adjoint(X, X, **gr)
        return {"x": X, **gr}


# -------------------------------------------------------------------- work
def _factor_flops(n, m, L, r):
    f = 2.0 / 3.0 * n * m * m + 2.0 * n * m * L * r
    for l in range(L):
        f += 2.0 * n * r * r + 4.0 * n * r * r * l + 2.0 ** l * (16.0 / 3.0 * r ** 3 + 8.0 * r ** 3 * l)
    return f


def _solve_flops(n, m, L, r, k):
    return 2.0 * n * m * k + sum(4.0 * n * r * k + 8.0 * 2 ** l * r * r * k for l in range(L))


def work(case):
    kind = case["kind"]
    if kind == "hsolve":
        m, L, r, k = case["leaf"], case["levels"], case["rank"], case["nrhs"]
        n = m << L
        # K, [b | U ...] read and written, V read
        return {"bytes": 8.0 * n * (2 * m + 2 * (k + L * r) + r), "flops": _factor_flops(n, m, L, r)
                + _solve_flops(n, m, L, r, k)}
    shapes = _batch_shapes(case) if kind == "batch" else [
        (case["leaf"] << case["levels"], case["leaf"], case["levels"], case["rank"], case["nrhs"])]
    nbytes = flops = 0.0
    for n, m, L, r, k in shapes:
        inputs, vec = 8.0 * n * (m + 2 * L * r), 8.0 * n * k
        F, S = _factor_flops(n, m, L, r), _solve_flops(n, m, L, r, k)
        if kind == "resolve":
            nbytes += 2 * (inputs + 2 * vec)
            flops += 2 * S
        elif kind == "adjoint":  # the gradients are as large as the inputs
            nbytes += 2 * inputs + 3 * vec
            flops += F + 2 * S + 2.0 * n * m * k + 8.0 * n * r * k * L
        else:
            nbytes += inputs + 2 * vec
            flops += F + S
    return {"bytes": nbytes, "flops": flops}


# ------------------------------------------------------------------- exact
def _recursion(D, U, V, s, B):
    """x = A^{-1} B and Utilde^(l) = A_c^{-1} U^(l)_c; D [leaf][row][column], U and V per level, in 64 bits."""
    L, nleaf, m = len(U), D.shape[0], D.shape[1]
    n, k = B.shape
    Y = torch.cat([B] + list(U), dim=1)
    Y = torch.linalg.solve(D, Y.reshape(nleaf, m, -1)).reshape(n, -1)
    for l in range(L - 1, -1, -1):
        r, nb = U[l].shape[1], 2 << l
        c = Y.shape[1]
        u0 = k + sum(x.shape[1] for x in U[:l])
        Yb = Y.reshape(nb, n // nb, c)
        T = torch.bmm(V[l].reshape(nb, n // nb, r).transpose(1, 2), Yb) * s[l][None, :, None]
        T = T.reshape(nb // 2, 2, r, c)
        S = torch.eye(2 * r, dtype=F64, device=Y.device).repeat(nb // 2, 1, 1)
        S[:, :r, r:] = T[:, 1, :, u0:u0 + r]
        S[:, r:, :r] = T[:, 0, :, u0:u0 + r]
        E = torch.linalg.solve(S, torch.cat([T[:, 1, :, :u0], T[:, 0, :, :u0]], dim=1)).reshape(nb, r, u0)
        Yb[:, :, :u0] -= torch.bmm(Yb[:, :, u0:u0 + r], E)
    return Y[:, :k], Y[:, k:]


def exact(case, seed):
    kind = case["kind"]
    if kind == "hsolve":
        K, U, V = _hsolve_inputs(case, seed)
        m, L, r, k = case["leaf"], case["levels"], case["rank"], case["nrhs"]
        D, u = K.reshape(1 << L, m, m), U[:, k:k + r]
        x, ut = _recursion(D, [u] * L, [V] * L, [torch.ones(r, dtype=F64)] * L, U[:, :k])
        lu = torch.linalg.lu_factor(D)[0].reshape(m << L, m)
        out = {"K": lu, "U": torch.cat([x, ut], dim=1)}
        return {key: v.numpy() for key, v in out.items()} if case["host"] else out
    xs = []
    for (n, m, L, r, k), (D, U, V, s), B in _systems(case, seed):
        D = D.transpose(1, 2)
        x = _recursion(D, U, V, s, B)[0]
        if kind in ("resolve", "adjoint"):
            y = _recursion(D.transpose(1, 2), V, U, s, B if kind == "resolve" else x)[0]
        if kind == "resolve":
            return {"x": x, "y": y}
        if kind == "adjoint":
            return {"x": x, **_gradients(x, y, U, V, s, m)}
        if kind == "system":
            return x
        xs.append(x.t().reshape(-1))
    return torch.cat(xs)


def _gradients(x, lam, U, V, s, m):
    """The gradients of L = ||x||^2 / 2 from x and lam = A^{-T} x, laid out as the library writes them."""
    n, k = x.shape
    blocks = lambda t, nb: t.reshape(nb, n // nb, t.shape[1])  # noqa: E731
    dD = -torch.bmm(blocks(x, n // m), blocks(lam, n // m).transpose(1, 2))  # [leaf][column][row]
    dU, dV, ds = [], [], []
    for l in range(len(U)):
        nb, r = 2 << l, U[l].shape[1]
        sib = [c ^ 1 for c in range(nb)]
        T = torch.bmm(blocks(V[l], nb).transpose(1, 2), blocks(x, nb))[sib]   # r x k: V^T x of the sibling
        W = torch.bmm(blocks(U[l], nb).transpose(1, 2), blocks(lam, nb))      # U^T lambda of the child
        ds.append(-(W * T).sum(dim=(0, 2)))
        dU.append((-torch.bmm(blocks(lam, nb), T.transpose(1, 2)) * s[l]).reshape(n, r).t().reshape(-1))
        dV.append((-torch.bmm(blocks(x, nb), W[sib].transpose(1, 2)) * s[l]).reshape(n, r).t().reshape(-1))
    return {"db": lam, "dD": dD.reshape(-1), "dU": torch.cat(dU), "dV": torch.cat(dV), "ds": torch.cat(ds)}
