"""FP64 low-rank updates on the tensor cores (csrc/f64_update_tc.cu) over many
tiles: every CTA passes several row tiles of a block."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

SMS, TILE = 152, 128


@pytest.fixture()
def lib():
    import fastsolver2_gb300 as fs
    return fs


def col(a):
    return torch.from_numpy(np.ascontiguousarray(np.asarray(a).T)).cuda().t()


def broadcast(fs, alpha, U, B, W):
    """hodlr_gemm_broadcast of one block: W + alpha U B (W is left as it is)."""
    n, K = U.shape
    w = W.t().clone().t()
    fs.check(fs.lib().hodlr_gemm_broadcast(n, 1, 1, K, W.shape[1], alpha, U.data_ptr(), n, B.data_ptr(), K, 1.0,
                                           w.data_ptr(), n))
    return w


@pytest.mark.parametrize("K,N", [(8, 9), (32, 32), (33, 32), (32, 33)])
def test_row_scales_of_many_row_tiles(lib, K, N):
    """One tile of rows over and over, each time in other units (a power of two):
    every tile's result is the first one's in its units, bit for bit.  At one
    column tile the scales of a row tile are replaced soonest."""
    rng = np.random.default_rng(K + N)
    tiles = SMS * 12
    p = 2.0 ** rng.integers(-200, 200, tiles)
    p[0] = 1.0
    p = torch.from_numpy(p).cuda()
    base = torch.from_numpy(rng.standard_normal((K, TILE))).cuda()
    U = (base[:, None, :] * p[None, :, None]).reshape(K, tiles * TILE).t()
    B = col(rng.standard_normal((K, N)))
    W = torch.zeros((N, tiles * TILE), dtype=torch.float64, device="cuda").t()
    for _ in range(5):
        got = broadcast(lib, 1.0, U, B, W).t().reshape(N, tiles, TILE)
        assert torch.equal(got, got[:, :1] * p[None, :, None])
    assert got[:, 0].abs().max() > 0
