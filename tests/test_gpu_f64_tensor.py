"""FP64 products on the tensor cores (exact digit products, csrc/f64_tc.cuh)
against quadruple precision, at the edges of their tiles.

Bound: the digit products are exact and the operands rounded below FP64's own
rounding, so the result may be no further off (relative 2-norm) than the FP64
FMA path on the same data, or than one correct rounding (2^-53) where that is
more."""
import os

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

HALF_ULP = 2.0 ** -53


@pytest.fixture()
def lib():
    import fastsolver2_gb300 as fs
    return fs


def col(a):
    return torch.from_numpy(np.ascontiguousarray(np.asarray(a).T)).cuda().t()


def both_paths(f):
    """f() with the tensor cores and with the FP64 FMA kernels."""
    old = os.environ.get("HODLR_NO_TCGEN05")
    out = []
    try:
        for off in ("0", "1"):
            os.environ["HODLR_NO_TCGEN05"] = off
            out.append(f())
    finally:
        if old is None:
            del os.environ["HODLR_NO_TCGEN05"]
        else:
            os.environ["HODLR_NO_TCGEN05"] = old
    return out


def rel_err(x, exact):
    d = (x.astype(np.longdouble) - exact).astype(np.float64)
    return np.linalg.norm(d) / np.linalg.norm(exact.astype(np.float64))


def broadcast(fs, npart, nblock, alpha, U, B, W):
    """hodlr_gemm_broadcast: W + alpha U B."""
    u, b, w = col(U), col(B), col(W)
    n, K = U.shape
    fs.check(fs.lib().hodlr_gemm_broadcast(n, npart, nblock, K, W.shape[1], alpha, u.data_ptr(), n, b.data_ptr(),
                                           B.shape[0], 1.0, w.data_ptr(), n))
    return w.cpu().numpy()


def exact_broadcast(nblock, alpha, U, B, W):
    out, per, K = W.astype(np.longdouble), U.shape[0] // nblock, U.shape[1]
    for i in range(nblock):
        out[i * per:(i + 1) * per] += np.longdouble(alpha) * (
            U[i * per:(i + 1) * per].astype(np.longdouble) @ B[i * K:(i + 1) * K].astype(np.longdouble))
    return out


# (rows, partitions, blocks, inner, columns): one tile, tails of 128 rows, 32 columns and
# 16 / 32 inner values, both inner chunks, blocks that end inside a tile
@pytest.mark.parametrize("n,npart,nblock,K,N", [(128, 1, 1, 32, 32), (129, 1, 1, 33, 33), (127, 1, 1, 31, 9),
                                                (300, 3, 3, 17, 64), (640, 5, 1, 1, 65), (4096, 8, 4, 64, 96),
                                                (64, 1, 1, 48, 63)])
@pytest.mark.parametrize("kind", ["normal", "uniform"])
def test_update_no_less_exact_than_fma(lib, n, npart, nblock, K, N, kind):
    rng = np.random.default_rng(n + K + N)
    draw = rng.standard_normal if kind == "normal" else rng.random
    U, B, W = draw((n, K)), draw((nblock * K, N)), draw((n, N))
    tc, fma = both_paths(lambda: broadcast(lib, npart, nblock, -1.0, U, B, W))
    exact = exact_broadcast(nblock, -1.0, U, B, W)
    assert rel_err(tc, exact) <= max(rel_err(fma, exact), HALF_ULP)


def test_update_alpha_units_and_zeros(lib):
    """alpha, an exact factor on the inner index with its inverse on the other
    operand (other units), zero rows and columns."""
    rng = np.random.default_rng(5)
    U, B, W = rng.standard_normal((300, 40)), rng.standard_normal((40, 50)), rng.standard_normal((300, 50))
    U[7], U[:, 3], B[:, 11] = 0.0, 0.0, 0.0
    tc, fma = both_paths(lambda: broadcast(lib, 1, 1, 0.375, U, B, W))
    exact = exact_broadcast(1, 0.375, U, B, W)
    assert rel_err(tc, exact) <= max(rel_err(fma, exact), HALF_ULP)
    p = 2.0 ** rng.integers(-60, 60, 40)
    assert np.array_equal(tc, broadcast(lib, 1, 1, 0.375, U * p, B / p[:, None], W))
    assert np.array_equal(tc[7], W[7]) and np.array_equal(tc[:, 11], W[:, 11])


def test_update_non_finite_stays_in_its_row_and_column(lib):
    rng = np.random.default_rng(6)
    U, B, W = rng.standard_normal((200, 20)), rng.standard_normal((20, 40)), rng.standard_normal((200, 40))
    U[3, 4], B[2, 7] = np.nan, np.inf
    tc, fma = both_paths(lambda: broadcast(lib, 1, 1, -1.0, U, B, W))
    ok = np.isfinite(fma)
    assert np.array_equal(ok, np.isfinite(tc))
    # entries of size 1 .. 20, sums of 21 terms: 2^-53 x 21 x 20 each way
    assert np.abs(tc[ok] - fma[ok]).max() <= 2 * 21 * 20 * HALF_ULP


def test_update_extreme_scales(lib):
    """Products far outside the unit range: scaled by exact powers of two."""
    rng = np.random.default_rng(7)
    U, B = rng.standard_normal((128, 16)), rng.standard_normal((16, 32))
    W = np.zeros((128, 32))
    base = broadcast(lib, 1, 1, 1.0, U, B, W)
    for ea, eb in ((-500, -400), (500, 400), (-900, 900)):
        got = broadcast(lib, 1, 1, 1.0, np.ldexp(U, ea), np.ldexp(B, eb), W)
        assert np.array_equal(got, np.ldexp(base, ea + eb))


def reduce(fs, npart, V, X):
    """hodlr_gemm_reduce: the partitions' V^T X stacked."""
    v, x = col(V), col(X)
    n, r = V.shape
    w = torch.zeros((X.shape[1], npart * r), dtype=torch.float64, device="cuda").t()
    fs.check(fs.lib().hodlr_gemm_reduce(n, npart, r, X.shape[1], v.data_ptr(), n, x.data_ptr(), n, w.data_ptr(),
                                        npart * r))
    return w.cpu().numpy()


def exact_reduce(npart, V, X):
    per, q = V.shape[0] // npart, np.longdouble
    return np.concatenate([V[i * per:(i + 1) * per].astype(q).T @ X[i * per:(i + 1) * per].astype(q)
                           for i in range(npart)])


# (rows, partitions, rank, columns): groups of 64 rows and their halves, 32 ranks, 128 columns, row chunks
@pytest.mark.parametrize("n,npart,r,C", [(64, 1, 32, 128), (65, 1, 33, 129), (63, 1, 31, 9), (96, 3, 1, 65),
                                         (2000, 2, 16, 40), (5120, 1, 64, 200), (40, 1, 8, 17)])
@pytest.mark.parametrize("kind", ["normal", "uniform"])
def test_reduce_no_less_exact_than_fma(lib, n, npart, r, C, kind):
    rng = np.random.default_rng(n + r + C)
    draw = rng.standard_normal if kind == "normal" else rng.random
    V, X = draw((n, r)), draw((n, C))
    tc, fma = both_paths(lambda: reduce(lib, npart, V, X))
    exact = exact_reduce(npart, V, X)
    assert rel_err(tc, exact) <= max(rel_err(fma, exact), HALF_ULP)


def test_reduce_units_zeros_and_non_finite(lib):
    rng = np.random.default_rng(8)
    V, X = rng.standard_normal((300, 20)), rng.standard_normal((300, 40))
    V[5], X[9], V[:, 3], X[:, 7] = 0.0, 0.0, 0.0, 0.0
    tc = reduce(lib, 1, V, X)
    assert not tc[3].any() and not tc[:, 7].any()
    p = 2.0 ** rng.integers(-60, 60, 300)
    assert np.array_equal(tc, reduce(lib, 1, V * p[:, None], X / p[:, None]))
    V[70, 4], X[200, 11] = np.inf, np.nan
    bad, fma = both_paths(lambda: reduce(lib, 1, V, X))
    ok = np.ones_like(bad, dtype=bool)
    ok[4], ok[:, 11] = False, False
    assert np.isfinite(bad[ok]).all() and not np.isfinite(bad[~ok]).any()
    V[70, 4], X[200, 11] = 0.0, 0.0  # in rank 4 and column 11 only: out of the compared entries
    exact = exact_reduce(1, V, X)
    assert rel_err(bad[ok], exact[ok]) <= max(rel_err(fma[ok], exact[ok]), HALF_ULP)


# column counts around the 32-column tiles and the pairs of them; two leaves at least
@pytest.mark.parametrize("m", [64, 128, 256])
@pytest.mark.parametrize("k", [9, 32, 65])
def test_leaf_application_no_less_exact_than_fma(lib, m, k):
    """Leaf solves alone (zero coupling): X = blockdiag(D)^-1 B, in place."""
    rng = np.random.default_rng(m + k)
    nl = 4
    D = rng.standard_normal((nl, m, m)) / np.sqrt(m) + 4.0 * np.eye(m)
    B = rng.standard_normal((nl * m, k))
    zero = torch.zeros((1, nl * m), dtype=torch.float64, device="cuda").t()

    def solve():
        s = lib.Solver(nl * m, m, 2, 1, nrhs_max=k)
        d = torch.from_numpy(np.ascontiguousarray(D.transpose(0, 2, 1))).cuda()
        s.set_leaf_blocks(d.reshape(-1), ld=m, leaf_stride=m * m)
        for l in range(2):
            s.set_lowrank(l, zero, zero)
        s.factor()
        b = col(B)
        s.solve(b)
        out = b.cpu().numpy()
        s.close()
        return out

    tc, fma = both_paths(solve)
    q = np.longdouble
    x = np.concatenate([np.linalg.solve(D[i], B[i * m:(i + 1) * m]) for i in range(nl)]).astype(q)
    for _ in range(2):  # refined in quadruple precision
        r = [B[i * m:(i + 1) * m].astype(q) - D[i].astype(q) @ x[i * m:(i + 1) * m] for i in range(nl)]
        x = x + np.concatenate([np.linalg.solve(D[i], r[i].astype(np.float64)) for i in range(nl)])
    assert rel_err(tc, x) <= max(rel_err(fma, x), HALF_ULP)


def factored_leaves(lib, D, B):
    """X of blockdiag(D) X = B through a solver, and the handle."""
    nl, m = D.shape[:2]
    s = lib.Solver(nl * m, m, int(np.log2(nl)), 1, nrhs_max=B.shape[1])
    d = torch.from_numpy(np.ascontiguousarray(D.transpose(0, 2, 1))).cuda()
    s.set_leaf_blocks(d.reshape(-1), ld=m, leaf_stride=m * m)
    zero = torch.zeros((1, nl * m), dtype=torch.float64, device="cuda").t()
    for l in range(int(np.log2(nl))):
        s.set_lowrank(l, zero, zero)
    s.factor()
    b = col(B)
    s.solve(b)
    return b.cpu().numpy(), s


@pytest.mark.parametrize("m", [64, 128, 256])
def test_leaf_inverse_that_pivots(lib, m):
    """Blocks whose pivots lie far from the diagonal, in every panel: a
    permutation of rows moves the large entries away.  Bound: an inverse formed
    by elimination with pivoting and applied, 4 m 2^-53 cond^2."""
    rng = np.random.default_rng(m)
    D = np.stack([(rng.standard_normal((m, m)) / np.sqrt(m) + 4.0 * np.eye(m))[rng.permutation(m)] for _ in range(2)])
    B = rng.standard_normal((2 * m, 3))
    x, s = factored_leaves(lib, D, B)
    for i in range(2):
        exact = np.linalg.solve(D[i], B[i * m:(i + 1) * m])
        err = np.linalg.norm(x[i * m:(i + 1) * m] - exact) / np.linalg.norm(exact)
        assert err <= 4 * m * HALF_ULP * np.linalg.cond(D[i]) ** 2
    # the LU factors and pivots, formed on request: P D = L U
    lu = torch.zeros(2 * m * m, dtype=torch.float64, device="cuda")
    piv = torch.zeros(2 * m, dtype=torch.int32, device="cuda")
    s.get_factors(leaf_lu=lu, leaf_ipiv=piv)
    lu, piv = lu.cpu().numpy().reshape(2, m, m).transpose(0, 2, 1), piv.cpu().numpy().reshape(2, m)
    for i in range(2):
        P = D[i].copy()
        for k, p in enumerate(piv[i]):
            P[[k, p - 1]] = P[[p - 1, k]]
        L, R = np.tril(lu[i], -1) + np.eye(m), np.triu(lu[i])
        assert (np.abs(P - L @ R) <= 2 * m * HALF_ULP * (np.abs(L) @ np.abs(R))).all()


@pytest.mark.parametrize("m", [64, 128, 256])
@pytest.mark.parametrize("kind", ["equal rows", "zero row", "zero column", "rank one"])
def test_singular_leaf_is_refused(lib, m, kind):
    rng = np.random.default_rng(m)
    D = np.stack([rng.standard_normal((m, m)) for _ in range(2)])
    if kind == "equal rows":
        D[1] = np.where(np.arange(m)[:, None] == m - 3, D[1, 2], D[1]) if m != 256 else np.ones((m, m))
    elif kind == "zero row":
        D[1, m // 2] = 0.0
    elif kind == "zero column":
        D[1, :, m - 1] = 0.0
    else:
        D[1] = 1.0
    with pytest.raises(lib.HodlrError) as e:
        factored_leaves(lib, D, np.ones((2 * m, 1)))
    assert e.value.code == lib.HODLR_ERR_SINGULAR_LEAF and "index 1" in str(e.value)


# padded sizes 32, 64 and 128 and their edges: 2r at, below and above a panel
@pytest.mark.parametrize("r", [1, 8, 15, 16, 17, 31, 32, 33, 48, 64])
def test_capacitance_factors_of_a_solver(lib, r):
    """The LU factors, pivots and solutions of the capacitance systems of a
    two-level solver with identity leaves: S = [I, s V1^T U1; s V0^T U0, I] of the
    bottom nodes, P S = L U, and x against a dense solve.  Bounds: the standard
    componentwise bound of a factorisation of order n, 2 n 2^-53 |L| |U|, and 4 n
    2^-53 cond^2 for the inverses, on the whole matrix."""
    rng = np.random.default_rng(r)
    m, L = 128, 2
    n = m << L
    D = np.stack([np.eye(m)] * (1 << L))
    Us, Vs = ([rng.standard_normal((n, r)) / np.sqrt(m) for _ in range(L)] for _ in range(2))
    s = lib.Solver(n, m, L, r, nrhs_max=12)
    s.set_leaf_blocks(torch.from_numpy(D).cuda().reshape(-1), ld=m, leaf_stride=m * m)
    for l in range(L):
        s.set_lowrank(l, col(Us[l]), col(Vs[l]))
    s.factor()
    n2 = 2 * r
    lu = torch.zeros(3 * n2 * n2, dtype=torch.float64, device="cuda")
    piv = torch.zeros(3 * n2, dtype=torch.int32, device="cuda")
    s.get_factors(cap_lu=lu, cap_ipiv=piv)
    lu, piv = lu.cpu().numpy().reshape(3, n2, n2).transpose(0, 2, 1), piv.cpu().numpy().reshape(3, n2)
    # one level of the recursion by node numbering: the two nodes of either end of the list
    found = 0
    for q in range(2):
        c0, c1 = slice(2 * q * m, (2 * q + 1) * m), slice((2 * q + 1) * m, (2 * q + 2) * m)
        S = np.eye(n2)
        S[:r, r:], S[r:, :r] = Vs[L - 1][c1].T @ Us[L - 1][c1], Vs[L - 1][c0].T @ Us[L - 1][c0]
        for k in range(3):
            P, Lf, R = S.copy(), np.tril(lu[k], -1) + np.eye(n2), np.triu(lu[k])
            for i, p in enumerate(piv[k]):
                P[[i, p - 1]] = P[[p - 1, i]]
            # S itself is formed from sums of m products: m 2^-53 |V|^T |U| more
            slack = np.pad(np.zeros((r, r)), (0, r))
            slack[:r, r:], slack[r:, :r] = (np.abs(Vs[L - 1][c]).T @ np.abs(Us[L - 1][c]) for c in (c1, c0))
            bound = 2 * n2 * HALF_ULP * (np.abs(Lf) @ np.abs(R)) + m * HALF_ULP * slack.max()
            found += (np.abs(P - Lf @ R) <= bound).all()
    assert found == 2
    A = np.eye(n)
    for l in range(L):
        h = n >> (l + 1)
        for p in range(1 << l):
            c0, c1 = slice(2 * p * h, (2 * p + 1) * h), slice((2 * p + 1) * h, (2 * p + 2) * h)
            A[c0, c1], A[c1, c0] = Us[l][c0] @ Vs[l][c1].T, Us[l][c1] @ Vs[l][c0].T
    B = rng.standard_normal((n, 12))
    b = col(B)
    s.solve(b)
    exact = np.linalg.solve(A, B)
    err = np.linalg.norm(b.cpu().numpy() - exact) / np.linalg.norm(exact)
    assert err <= 4 * n * HALF_ULP * np.linalg.cond(A) ** 2


def test_singular_capacitance_is_refused(lib):
    """A = [I, e e^T; e e^T, I] on one node: S is exactly singular."""
    m, r = 128, 20
    s = lib.Solver(2 * m, m, 1, r)
    D = np.stack([np.eye(m)] * 2)
    U = np.zeros((2 * m, r))
    for q in range(r):
        U[q, q] = U[m + q, q] = 1.0
    s.set_leaf_blocks(torch.from_numpy(D).cuda().reshape(-1), ld=m, leaf_stride=m * m)
    s.set_lowrank(0, col(U), col(U))
    with pytest.raises(lib.HodlrError) as e:
        s.factor()
    assert e.value.code == lib.HODLR_ERR_SINGULAR_CAPACITANCE
