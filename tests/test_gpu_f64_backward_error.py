"""FP64 solves with ill-conditioned leaves and capacitance systems: the backward error
||A x - b|| / (||A|| ||x||) stays that of an LU factorisation, in both directions.

Bound: that of the FP64 FMA kernels on the same data, or sqrt(n) 2^-53 where that is
more (n roundings of random sign), four times.  (An inverse formed by eliminating above
and below the pivots at once solves A x = b with an error that grows with the condition
number, and A^T x = b without.)"""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

U53 = 2.0 ** -53


def col(a):
    return torch.from_numpy(np.ascontiguousarray(np.asarray(a).T)).cuda().t()


def two_paths(f, monkeypatch):
    out = []
    for off in ("0", "1"):
        monkeypatch.setenv("HODLR_NO_TCGEN05", off)
        out.append(f())
    return out


def backward_error(A, x, b):
    r = (A.astype(np.longdouble) @ x.astype(np.longdouble) - b).astype(np.float64)
    return np.linalg.norm(r) / (np.linalg.norm(A, 2) * np.linalg.norm(x))


def leaf(kind, m, rng):
    if kind.startswith("svd"):
        Q, P = (np.linalg.qr(rng.standard_normal((m, m)))[0] for _ in range(2))
        return Q @ np.diag(np.logspace(0, -float(kind[4:]), m)) @ P.T
    x = np.sort(rng.random(m))  # a Gaussian kernel with a nugget
    return np.exp(-(x[:, None] - x[None, :]) ** 2 / 0.1) + 10.0 ** -float(kind[7:]) * np.eye(m)


@pytest.mark.parametrize("m", [64, 128, 256])
@pytest.mark.parametrize("kind", ["svd 4", "svd 7", "svd 10", "kernel 2", "kernel 4", "kernel 6"])
@pytest.mark.parametrize("k", [1, 16])
def test_ill_conditioned_leaves(hodlr, m, kind, k, monkeypatch):
    rng = np.random.default_rng(m + len(kind))
    nl = 2
    D = np.stack([leaf(kind, m, rng) for _ in range(nl)])
    B = rng.standard_normal((nl * m, k))
    d, zero = torch.from_numpy(np.ascontiguousarray(D.transpose(0, 2, 1))).cuda(), col(np.zeros((nl * m, 1)))

    def solve():
        s = hodlr.Solver(nl * m, m, 1, 1, nrhs_max=k)
        torch.cuda.synchronize()
        s.set_leaf_blocks(d.reshape(-1), ld=m, leaf_stride=m * m)
        s.set_lowrank(0, zero, zero)
        s.factor()
        errors = []
        for transpose in (False, True):
            x = col(B)
            torch.cuda.synchronize()
            s.solve(x, transpose=transpose)
            x = x.cpu().numpy()
            errors.append(max(backward_error(D[i].T if transpose else D[i], x[i * m:(i + 1) * m], B[i * m:(i + 1) * m])
                              for i in range(nl)))
        s.close()
        return errors

    for tc, fma in zip(*two_paths(solve, monkeypatch)):
        assert tc <= 4 * max(fma, m ** 0.5 * U53)


@pytest.mark.parametrize("r", [8, 20, 40, 64])
@pytest.mark.parametrize("delta", [1e-2, 1e-5, 1e-8])
def test_ill_conditioned_capacitance(hodlr, r, delta, monkeypatch):
    """S = [I, X; (1 - delta) X^-1, I] on identity leaves: nearly singular, X of condition 100."""
    rng = np.random.default_rng(r)
    m, k = 128, 12
    Q, P = (np.linalg.qr(rng.standard_normal((r, r)))[0] for _ in range(2))
    X = Q @ np.diag(np.logspace(1, -1, r)) @ P.T
    W = [np.linalg.qr(rng.standard_normal((m, r)))[0] for _ in range(2)]
    U = np.concatenate([W[0] @ ((1 - delta) * np.linalg.inv(X)), W[1] @ X])  # V0^T U0, V1^T U1
    V = np.concatenate(W)
    A = np.eye(2 * m)
    A[:m, m:], A[m:, :m] = U[:m] @ V[m:].T, U[m:] @ V[:m].T
    B = rng.standard_normal((2 * m, k))
    d, u, v = torch.eye(m, dtype=torch.float64, device="cuda").repeat(2, 1, 1), col(U), col(V)

    def solve():
        s = hodlr.Solver(2 * m, m, 1, r, nrhs_max=k)
        torch.cuda.synchronize()
        s.set_leaf_blocks(d.reshape(-1), ld=m, leaf_stride=m * m)
        s.set_lowrank(0, u, v)
        s.factor()
        errors = []
        for transpose in (False, True):
            x = col(B)
            torch.cuda.synchronize()
            s.solve(x, transpose=transpose)
            errors.append(backward_error(A.T if transpose else A, x.cpu().numpy(), B))
        s.close()
        return errors

    for tc, fma in zip(*two_paths(solve, monkeypatch)):
        assert tc <= 4 * max(fma, (2 * m) ** 0.5 * U53)
