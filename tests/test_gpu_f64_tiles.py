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


# ------------------------------------------------- bases that change from tile to tile
U53 = 2.0 ** -53


def bases(kind, n, K, rng):
    """n x K factors whose columns change size along the rows."""
    i = np.arange(n)
    t, x = i // TILE, (i + 0.5) / n
    G = rng.standard_normal((n, K))
    k = np.arange(K)
    if kind == "zero in every other tile":
        G[(t % 2 == 0)[:, None] & (k % 2 == 1)] = 0.0
    elif kind == "small in every other tile":
        G[t % 2 == 0, 1] *= 1e-6
    elif kind == "units of the tile":
        G *= 2.0 ** rng.integers(-60, 60, (t[-1] + 1, K))[t]
    elif kind == "unit vectors":
        G = (t[:, None] % K == k).astype(float)
    elif kind == "bumps":
        G = np.exp(-((x[:, None] - (k + 0.5) / K) * 20.0) ** 2)
    elif kind == "monomials":
        G = x[:, None] ** (k % 24)
    elif kind == "decay from both ends":
        G *= np.exp(-40.0 * np.where(k % 2 == 0, x[:, None], 1.0 - x[:, None]))
    return G


KINDS = ["zero in every other tile", "small in every other tile", "units of the tile", "unit vectors", "bumps",
         "monomials", "decay from both ends"]


@pytest.mark.parametrize("K,N", [(17, 9), (32, 40), (64, 96)])
@pytest.mark.parametrize("kind", KINDS)
def test_update_of_bases_that_change_along_the_rows(lib, kind, K, N):
    """Every element within the bound of the digit products, and the same bits
    as its row tile alone.

    The bound: with c_k the power of two of the largest |U(., k)| of the row tile,
    alpha the largest |U(i, k)| / c_k of the row and beta the largest |B(k, j)| c_k
    of the column, both operands are rounded to 2^-55 of a bound of at most twice
    alpha or beta, K products: K 2^-53 alpha beta; the digits left out less than
    half of that; the result and its sum with W one rounding each."""
    rng = np.random.default_rng(K + len(kind))
    n = TILE * SMS * 3 + 50
    U, B = bases(kind, n, K, rng), rng.standard_normal((K, N))
    u, b = col(U), col(B)
    w = torch.zeros((N, n), dtype=torch.float64, device="cuda").t()
    got = broadcast(lib, 1.0, u, b, w).cpu().numpy()
    for t in list(range(0, 12)) + list(range(13, n // TILE, 17)) + [n // TILE]:
        rows = slice(t * TILE, min(n, (t + 1) * TILE))
        A, g = U[rows], got[rows]
        top = np.abs(A).max(axis=0)
        c = 2.0 ** np.floor(np.log2(np.where(top > 0, top, 1.0)))
        alpha = (np.abs(A) / c).max(axis=1)[:, None]
        beta = (np.abs(B) * np.where(top > 0, c, 0.0)[:, None]).max(axis=0)[None, :]
        exact = A.astype(np.longdouble) @ B.astype(np.longdouble)
        err = np.abs(g - exact).astype(np.float64)
        assert (err <= U53 * (1.5 * K * alpha * beta + 2 * np.abs(g))).all(), (t, err.max())
        alone = broadcast(lib, 1.0, col(A), b, w[rows].t().contiguous().t()).cpu().numpy()
        assert np.array_equal(alone, g), t


def two_paths(f, monkeypatch):
    """f() with the tensor cores and with the FP64 FMA kernels."""
    out = []
    for off in ("0", "1"):
        monkeypatch.setenv("HODLR_NO_TCGEN05", off)
        out.append(f())
    return out


def tile_diff(a, b):
    """Largest difference of a 128-row tile, relative to the tile (2-norms)."""
    n = a.shape[0] // TILE * TILE
    a, b = (x[:n].reshape(-1, TILE * x.shape[1]) for x in (a, b))
    scale = torch.maximum(b.norm(dim=1), 1e-30 * b.norm())
    return float(((a - b).norm(dim=1) / scale).max())


M, L, R, COLS = 128, 9, 16, 16


def hodlr_inputs(kind, seed):
    rng = np.random.default_rng(seed)
    n = M << L
    g = torch.Generator(device="cuda").manual_seed(seed)
    D = torch.randn((n // M, M, M), generator=g, dtype=torch.float64, device="cuda") / M ** 0.5
    D.diagonal(dim1=1, dim2=2).add_(4.0)
    U, V = [], []
    for l in range(L):
        for out in (U, V):
            # orthonormal columns a block at most: the couplings stay below the leaves
            X = bases(kind, n, R, rng)
            q = np.linalg.norm(X.reshape(2 << l, -1, R), axis=1).max(axis=0)
            out.append(col(X / np.where(q > 0, q, 1.0)))
    B = torch.randn((COLS, n), generator=g, dtype=torch.float64, device="cuda").t()
    return n, D, U, V, B


def set_up(lib, n, D, U, V, m):
    s = lib.Solver(n, m, len(U), U[0].shape[1], nrhs_max=COLS)
    s.set_leaf_blocks(D.reshape(-1), ld=m, leaf_stride=m * m)
    for l in range(len(U)):
        s.set_lowrank(l, U[l], V[l])
    return s


SOLVER_KINDS = ["zero in every other tile", "small in every other tile", "unit vectors", "bumps"]


@pytest.mark.parametrize("kind", SOLVER_KINDS)
@pytest.mark.parametrize("transpose", [False, True])
def test_matvec_of_bases_that_change_along_the_rows(lib, kind, transpose, monkeypatch):
    """The two paths agree in every 128-row tile.  Sums of up to n / 2 products,
    in groups of 64 at least, a level: n / 128 + 64 + M + L R roundings of terms as
    large as the tile."""
    n, D, U, V, B = hodlr_inputs(kind, 5)

    def product():
        s = set_up(lib, n, D, U, V, M)
        Y = torch.empty((COLS, n), dtype=torch.float64, device="cuda").t()
        s.matvec(B, Y, transpose=transpose)
        s.close()
        return Y

    tc, fma = two_paths(product, monkeypatch)
    assert tile_diff(tc, fma) <= 2 * U53 * (n // 128 + 64 + M + L * R)


@pytest.mark.parametrize("kind", SOLVER_KINDS)
def test_solve_and_gradients_of_bases_that_change_along_the_rows(lib, kind, monkeypatch):
    """Factor, solve and gradients (8 columns) on both paths.  The leaves dominate
    (singular values 2 .. 6, couplings of norm 1 at most a level): the solutions and
    the gradients of the levels agree to 2^-53 times the roundings above and a
    condition number of (6 + L) / 1."""
    n, D, U, V, B = hodlr_inputs(kind, 7)
    k = 8

    def step():
        s = set_up(lib, n, D, U, V, M)
        s.factor()
        X = B.t().clone().t()
        s.solve(X)
        x = X[:, :k].t().clone().t()
        e = lambda c: torch.empty(c, dtype=torch.float64, device="cuda")  # noqa: E731
        g = {"db": e(n * k).reshape(k, n).t(), "dD": e(n * M), "dU": e(L * n * R), "dV": e(L * n * R), "ds": e(L * R)}
        s.adjoint(x, x, **g)
        s.close()
        return X, g

    (x, g), (xf, gf) = two_paths(step, monkeypatch)
    tol = 2 * U53 * (n // 128 + 64 + M + L * R) * (6 + L)
    assert tile_diff(x, xf) <= tol
    for name, shape in (("db", None), ("dU", (L * R, n)), ("dV", (L * R, n)), ("dD", (n // M, M * M))):
        a, b = g[name], gf[name]
        if shape is None:
            assert tile_diff(a, b) <= tol
        else:  # a column of a level's gradient, a leaf's block
            a, b = a.reshape(shape), b.reshape(shape)
            scale = torch.maximum(b.norm(dim=1), 1e-3 * b.norm() / shape[0] ** 0.5)
            assert float(((a - b).norm(dim=1) / scale).max()) <= tol, name


@pytest.mark.parametrize("m", [256, 300])
@pytest.mark.parametrize("kind", ["banded", "blocks", "arrow"])
def test_sparse_leaves_of_several_row_tiles(lib, m, kind):
    """Leaves with zero blocks, 64 of them: every CTA of the products of their
    factorisation and of their substitutions passes several row tiles of a leaf.  The
    residual of every leaf against the bound 4 m 2^-53 cond."""
    rng = np.random.default_rng(m)
    nl = 64
    i = np.arange(m)
    D = rng.standard_normal((nl, m, m)) / np.sqrt(m)
    far = np.abs(i[:, None] - i[None, :])
    if kind == "banded":
        D = np.where(far <= 5, rng.standard_normal((nl, m, m)) / 4.0, 0.0)
    elif kind == "blocks":
        D *= (i[:, None] // 64 + i[None, :] // 64) % 2 == 0
    else:
        D = np.where((i[:, None] < 8) | (i[None, :] < 8), D, 0.0)
    D = D + 4.0 * np.eye(m)
    D[1::2] = D[1::2, rng.permutation(m)]  # pivots far from the diagonal
    Bm = rng.standard_normal((nl, m, COLS))
    n = nl * m
    zero = torch.zeros((1, n), dtype=torch.float64, device="cuda").t()
    d = torch.from_numpy(np.ascontiguousarray(D.transpose(0, 2, 1))).cuda()
    s = set_up(lib, n, d, [zero] * 6, [zero] * 6, m)
    s.factor()
    X = col(Bm.reshape(n, COLS))
    s.solve(X)
    x = X.cpu().numpy().reshape(nl, m, COLS)
    exact = np.linalg.solve(D, Bm)
    err = np.linalg.norm(x - exact, axis=(1, 2)) / np.linalg.norm(exact, axis=(1, 2))
    assert (err <= 4 * m * U53 * np.linalg.cond(D)).all(), err.max()
