"""Infinities and NaNs in FP64 updates and reductions on the tensor
cores: the results of the FP64 FMA kernels."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

U53 = 2.0 ** -53


@pytest.fixture()
def lib():
    import fastsolver2_gb300 as fs
    return fs


def col(a):
    return torch.from_numpy(np.ascontiguousarray(np.asarray(a).T)).cuda().t()


def two_paths(f, monkeypatch):
    out = []
    for off in ("0", "1"):
        monkeypatch.setenv("HODLR_NO_TCGEN05", off)
        out.append(f())
    return out


def update(fs, U, B, W):
    """W - U B by hodlr_gemm_broadcast."""
    u, b, w = col(U), col(B), col(W)
    n, K = U.shape
    fs.check(fs.lib().hodlr_gemm_broadcast(n, 1, 1, K, W.shape[1], -1.0, u.data_ptr(), n, b.data_ptr(), K, 1.0,
                                           w.data_ptr(), n))
    return w.cpu().numpy()


def reduce(fs, V, X):
    """V^T X by hodlr_gemm_reduce."""
    v, x = col(V), col(X)
    n, r = V.shape
    w = torch.zeros((X.shape[1], r), dtype=torch.float64, device="cuda").t()
    fs.check(fs.lib().hodlr_gemm_reduce(n, 1, r, X.shape[1], v.data_ptr(), n, x.data_ptr(), n, w.data_ptr(), r))
    return w.cpu().numpy()


def same(tc, fma, terms):
    """The same infinities and NaNs; finite values to `terms` roundings of the largest."""
    assert np.array_equal(np.isnan(tc), np.isnan(fma))
    inf = np.isinf(fma)
    assert np.array_equal(np.isinf(tc), inf) and np.array_equal(tc[inf], fma[inf])
    ok = np.isfinite(fma)
    assert np.abs(tc[ok] - fma[ok]).max() <= 2 * terms * U53 * np.abs(fma[ok]).max()


# one tile, tails of every kind, both inner chunks, several row tiles a CTA
@pytest.mark.parametrize("n,K,N", [(128, 20, 40), (300, 33, 70), (128 * 400 + 7, 64, 9)])
def test_update_with_infinities_and_nans(lib, n, K, N, monkeypatch):
    rng = np.random.default_rng(n + K)
    U, B, W = rng.standard_normal((n, K)), rng.standard_normal((K, N)), rng.standard_normal((n, N))
    U[3, 4], U[n // 2, 1], U[n - 1, K - 1] = np.inf, np.nan, -np.inf
    B[2, 7], B[K - 1, N - 1], B[0, 2] = -np.inf, np.inf, np.nan
    U[n // 2 + 1, 2] = 0.0                      # 0 times an infinity
    U[9, 4], U[9, 5], B[4, 3], B[5, 3] = np.inf, np.inf, 1.0, -1.0   # infinities that cancel
    W[5, 6], W[11, 7] = np.inf, -np.inf
    tc, fma = two_paths(lambda: update(lib, U, B, W), monkeypatch)
    same(tc, fma, K + 1)
    assert np.isinf(fma).sum() > 50 and np.isnan(fma).sum() > 5


@pytest.mark.parametrize("n,r,C", [(64, 20, 40), (300, 33, 130), (9001, 64, 9)])
def test_reduction_with_infinities_and_nans(lib, n, r, C, monkeypatch):
    rng = np.random.default_rng(n + r)
    V, X = rng.standard_normal((n, r)), rng.standard_normal((n, C))
    V[3, 4], V[n // 2, 1], V[n - 1, r - 1] = np.inf, np.nan, -np.inf
    X[2, 7], X[n - 1, C - 1], X[0, 2] = -np.inf, np.inf, np.nan
    V[2, 5] = 0.0
    V[10, 6], V[11, 6], X[10, 5], X[11, 5] = np.inf, np.inf, 1.0, -1.0
    tc, fma = two_paths(lambda: reduce(lib, V, X), monkeypatch)
    same(tc, fma, n)
    assert np.isinf(fma).sum() > 20 and np.isnan(fma).sum() > 5
