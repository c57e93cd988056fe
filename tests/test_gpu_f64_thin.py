"""The FP64 kernels for few columns (csrc/f64_thin.cu) at the edges of their
cases: column templates 1, 2, 4, 8, ranks per warp, row tails, the lanes' sums,
inner dimensions past one staged chunk, both directions of the leaf and
capacitance applications.

Bounds.  A sum of K products in FP64, in any order, is off by at most
(K + 2) 2^-53 times the sum of the products' magnitudes (the two are the
scaling and the addition to C).  An explicit inverse of an n x n block formed
by LU and applied is off by at most 4 n 2^-53 cond^2 in the relative 2-norm
(inverse: 2 n cond^2, its application: n cond, for the well-conditioned blocks
used here)."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

U = 2.0 ** -53
Q = np.longdouble


@pytest.fixture()
def lib():
    import fastsolver2_gb300 as fs
    return fs


def col(a):
    return torch.from_numpy(np.ascontiguousarray(np.asarray(a).T)).cuda().t()


@pytest.mark.parametrize("n,npart,K,N", [(1, 1, 1, 1), (33, 1, 5, 1), (257, 1, 8, 2), (96, 3, 17, 3), (100, 1, 65, 4),
                                         (512, 2, 130, 1), (31, 1, 64, 4), (300, 1, 9, 5), (129, 1, 33, 8)])
def test_update_few_columns(lib, n, npart, K, N):
    rng = np.random.default_rng(n + K + N)
    A, B, W = rng.standard_normal((n, K)), rng.standard_normal((K, N)), rng.standard_normal((n, N))
    a, b, w = col(A), col(B), col(W)
    lib.check(lib.lib().hodlr_gemm_broadcast(n, npart, 1, K, N, -0.75, a.data_ptr(), n, b.data_ptr(), K, 1.0,
                                             w.data_ptr(), n))
    exact = W.astype(Q) - Q(0.75) * (A.astype(Q) @ B.astype(Q))
    bound = (K + 2) * U * (np.abs(W) + np.abs(A) @ np.abs(B))
    assert (np.abs((w.cpu().numpy() - exact).astype(np.float64)) <= bound).all()


@pytest.mark.parametrize("n,K,N", [(1, 1, 33), (257, 1, 31), (70, 2, 32), (128, 3, 100), (300, 4, 65), (64, 4, 1)])
def test_update_small_inner_dimension(lib, n, K, N):
    rng = np.random.default_rng(n + K + N)
    A, B, W = rng.standard_normal((n, K)), rng.standard_normal((K, N)), rng.standard_normal((n, N))
    a, b, w = col(A), col(B), col(W)
    lib.check(lib.lib().hodlr_gemm_broadcast(n, 1, 1, K, N, 1.5, a.data_ptr(), n, b.data_ptr(), K, 1.0, w.data_ptr(),
                                             n))
    exact = W.astype(Q) + Q(1.5) * (A.astype(Q) @ B.astype(Q))
    bound = (K + 2) * U * (np.abs(W) + 1.5 * np.abs(A) @ np.abs(B))
    assert (np.abs((w.cpu().numpy() - exact).astype(np.float64)) <= bound).all()


@pytest.mark.parametrize("n,npart,r,C", [(1, 1, 1, 1), (31, 1, 8, 8), (33, 1, 9, 3), (1000, 2, 16, 2), (513, 1, 17, 1),
                                         (4000, 1, 32, 5), (384, 3, 33, 4), (777, 1, 64, 8), (129, 1, 64, 1)])
def test_reduce_few_columns(lib, n, npart, r, C):
    rng = np.random.default_rng(n + r + C)
    V, X = rng.standard_normal((n, r)), rng.standard_normal((n, C))
    v, x = col(V), col(X)
    w = torch.zeros((C, npart * r), dtype=torch.float64, device="cuda").t()
    lib.check(lib.lib().hodlr_gemm_reduce(n, npart, r, C, v.data_ptr(), n, x.data_ptr(), n, w.data_ptr(), npart * r))
    per = n // npart
    parts = [slice(i * per, (i + 1) * per) for i in range(npart)]
    exact = np.concatenate([V[p].astype(Q).T @ X[p].astype(Q) for p in parts])
    bound = (per + 2) * U * np.concatenate([np.abs(V[p]).T @ np.abs(X[p]) for p in parts])
    assert (np.abs((w.cpu().numpy() - exact).astype(np.float64)) <= bound).all()


@pytest.mark.parametrize("m", [64, 128, 256])
@pytest.mark.parametrize("k", [1, 2, 3, 8])
@pytest.mark.parametrize("transpose", [False, True])
def test_leaf_application_few_columns(lib, m, k, transpose):
    rng = np.random.default_rng(m + k)
    nl = 2
    D = rng.standard_normal((nl, m, m)) / np.sqrt(m) + 4.0 * np.eye(m)
    B = rng.standard_normal((nl * m, k))
    zero = torch.zeros((1, nl * m), dtype=torch.float64, device="cuda").t()
    s = lib.Solver(nl * m, m, 1, 1, nrhs_max=k)
    d = torch.from_numpy(np.ascontiguousarray(D.transpose(0, 2, 1))).cuda()
    s.set_leaf_blocks(d.reshape(-1), ld=m, leaf_stride=m * m)
    s.set_lowrank(0, zero, zero)
    s.factor()
    b = col(B)
    s.solve(b, transpose=transpose)
    x = b.cpu().numpy()
    for i in range(nl):
        A = D[i].T if transpose else D[i]
        exact = np.linalg.solve(A, B[i * m:(i + 1) * m])
        err = np.linalg.norm(x[i * m:(i + 1) * m] - exact) / np.linalg.norm(exact)
        assert err <= 4 * m * U * np.linalg.cond(A) ** 2


@pytest.mark.parametrize("r", [1, 13, 16, 17, 32, 48, 64])
@pytest.mark.parametrize("k", [1, 2, 4, 7])
def test_capacitance_application_few_columns(lib, r, k):
    """hodlr_node_solve against a dense solve of S = [I, T1; T0, I]."""
    rng = np.random.default_rng(r + k)
    nn = 3
    VTu = 0.3 * rng.standard_normal((2 * r * nn, r)) / np.sqrt(r)
    VTd = rng.standard_normal((2 * r * nn, k))
    u, d = col(VTu), col(VTd)
    lib.check(lib.lib().hodlr_node_solve(nn, r, k, u.data_ptr(), 2 * r * nn, d.data_ptr(), 2 * r * nn))
    got = d.cpu().numpy()
    for p in range(nn):
        T0, T1 = VTu[2 * r * p:2 * r * p + r], VTu[2 * r * p + r:2 * r * (p + 1)]
        S = np.block([[np.eye(r), T1], [T0, np.eye(r)]])
        rhs = np.concatenate([VTd[2 * r * p + r:2 * r * (p + 1)], VTd[2 * r * p:2 * r * p + r]])
        exact = np.linalg.solve(S, rhs)
        err = np.linalg.norm(got[2 * r * p:2 * r * (p + 1)] - exact) / np.linalg.norm(exact)
        assert err <= 4 * 2 * r * U * np.linalg.cond(S) ** 2
