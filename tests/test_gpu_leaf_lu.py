"""LU of leaves without an explicit inverse by panels (csrc/leaf_blocked.cu) and
the substitutions with many and few right-hand sides (csrc/leaf_kernels.cu)."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.fixture()
def lib():
    import fastsolver2_gb300 as fs
    return fs


def col(a):
    return torch.from_numpy(np.ascontiguousarray(np.asarray(a).T)).cuda().t()


def factored_leaves(lib, D, B, mixed=False):
    """X of blockdiag(D) X = B through a solver, and the handle."""
    nl, m = D.shape[:2]
    levels = int(np.log2(nl))
    s = lib.Solver(nl * m, m, levels, 1, nrhs_max=B.shape[1],
                   precision=lib.PREC_MIXED if mixed else lib.PREC_FP64)
    d = torch.from_numpy(np.ascontiguousarray(D.transpose(0, 2, 1))).cuda()
    s.set_leaf_blocks(d.reshape(-1), ld=m, leaf_stride=m * m)
    zero = torch.zeros((1, nl * m), dtype=torch.float64, device="cuda").t()
    for l in range(levels):
        s.set_lowrank(l, zero, zero)
    s.factor()
    b = col(B)
    s.solve(b)
    return b.cpu().numpy(), s


def pivoting_blocks(rng, nl, m):
    """Well-conditioned blocks whose pivots lie far from the diagonal."""
    return np.stack([(rng.standard_normal((m, m)) / np.sqrt(m) + 4.0 * np.eye(m))[rng.permutation(m)]
                     for _ in range(nl)])


# one row, panels and diagonal blocks of 32 rows and their edges, the one-CTA kernel's largest
# leaf and the next in either precision, more rows than threads of a panel or of a substitution
@pytest.mark.parametrize("mixed,eps", [(False, 2.0 ** -53), (True, 2.0 ** -24)])
@pytest.mark.parametrize("m", [1, 31, 33, 63, 65, 96, 97, 100, 167, 168, 236, 239, 257, 320, 321, 400, 641, 700])
def test_factors_and_solution(lib, m, mixed, eps):
    """P D = L U within the standard componentwise bound of a factorisation of
    order m (and of D's own rounding to the working precision), and the solutions
    within that of the substitutions, 4 m 2^-53 cond^2 (refined in the mixed
    precision); 2 leaves, so that few columns leave SMs idle."""
    rng = np.random.default_rng(m)
    D = pivoting_blocks(rng, 2, m)
    B = rng.standard_normal((2 * m, 5))
    x, s = factored_leaves(lib, D, B, mixed)
    lu = torch.zeros(2 * m * m, dtype=torch.float64, device="cuda")
    piv = torch.zeros(2 * m, dtype=torch.int32, device="cuda")
    s.get_factors(leaf_lu=lu, leaf_ipiv=piv)
    lu, piv = lu.cpu().numpy().reshape(2, m, m).transpose(0, 2, 1), piv.cpu().numpy().reshape(2, m)
    for i in range(2):
        P = D[i].copy()
        for k, p in enumerate(piv[i]):
            P[[k, p - 1]] = P[[p - 1, k]]
        L, R = np.tril(lu[i], -1) + np.eye(m), np.triu(lu[i])
        assert (np.abs(L) <= 1.0 + 4 * eps).all()
        assert (np.abs(P - L @ R) <= 2 * (m + 1) * eps * (np.abs(L) @ np.abs(R)) + eps * np.abs(P)).all()
        exact = np.linalg.solve(D[i], B[i * m:(i + 1) * m])
        err = np.linalg.norm(x[i * m:(i + 1) * m] - exact) / np.linalg.norm(exact)
        assert err <= max(4 * m * 2.0 ** -53 * np.linalg.cond(D[i]) ** 2, 1e-12 if mixed else 0)


# 1, 2, 4 and 8 columns a CTA, full and ragged tiles
@pytest.mark.parametrize("k", [1, 2, 3, 7, 8, 9, 17, 33])
@pytest.mark.parametrize("nl,m", [(4, 100), (64, 50), (128, 33)])
def test_substitution_column_tiles(lib, nl, m, k):
    rng = np.random.default_rng(nl + k)
    D = pivoting_blocks(rng, nl, m)
    B = rng.standard_normal((nl * m, k))
    x, _ = factored_leaves(lib, D, B)
    exact = np.linalg.solve(D, B.reshape(nl, m, k)).reshape(-1, k)
    assert np.linalg.norm(x - exact) / np.linalg.norm(exact) <= 4 * m * 2.0 ** -53 * max(map(np.linalg.cond, D)) ** 2


@pytest.mark.parametrize("m", [100, 170, 400])
@pytest.mark.parametrize("kind", ["zero row", "zero column", "rank one"])
def test_singular_leaf_is_refused(lib, m, kind):
    rng = np.random.default_rng(m)
    D = np.stack([rng.standard_normal((m, m)) for _ in range(2)])
    if kind == "zero row":
        D[1, m // 2] = 0.0
    elif kind == "zero column":
        D[1, :, m - 1] = 0.0
    else:
        D[1] = 1.0
    with pytest.raises(lib.HodlrError) as e:
        factored_leaves(lib, D, np.ones((2 * m, 1)))
    assert e.value.code == lib.HODLR_ERR_SINGULAR_LEAF and "index 1" in str(e.value)


@pytest.mark.parametrize("m", [100, 200])
def test_pivots_of_any_magnitude(lib, m):
    """Rows scaled by powers of two from 2^-300 to 2^300, right-hand sides
    alike: the solution is that of the unscaled system bit for bit but for the
    choice of pivots, so within its bound."""
    rng = np.random.default_rng(m)
    D = np.stack([rng.standard_normal((m, m)) / np.sqrt(m) + 4.0 * np.eye(m) for _ in range(2)])
    B = rng.standard_normal((2 * m, 2))
    sc = 2.0 ** rng.integers(-300, 301)
    x, _ = factored_leaves(lib, D * sc, B * sc)
    exact = np.linalg.solve(D, B.reshape(2, m, 2)).reshape(-1, 2)
    assert np.linalg.norm(x - exact) / np.linalg.norm(exact) <= 4 * m * 2.0 ** -53 * max(map(np.linalg.cond, D)) ** 2


@pytest.mark.parametrize("m", [64, 128])
@pytest.mark.parametrize("npart", [1, 4, 8])
def test_hsolve_writes_back_the_factors(lib, m, npart):
    """K's leaves become their LU factors while the inverses are formed: L U has the
    rows of D in some order, within the componentwise bound of a factorisation of
    order m, |L| <= 1, and X solves the system."""
    rng = np.random.default_rng(m + npart)
    n, r, levels = npart * m, 3, npart.bit_length() - 1
    D = pivoting_blocks(rng, npart, m)
    B = rng.standard_normal((n, 2))
    K = np.asfortranarray(D.reshape(n, m))
    U = np.asfortranarray(np.hstack([B] + [rng.standard_normal((n, r)) for _ in range(levels)]))
    V = np.asfortranarray(rng.standard_normal((n, r)) / n)
    A = np.zeros((n, n))
    for i in range(npart):
        A[i * m:(i + 1) * m, i * m:(i + 1) * m] = D[i]
    for l in range(levels):
        h = n >> (l + 1)
        Ul = U[:, 2 + l * r:2 + (l + 1) * r]
        for q in range(1 << l):
            c0, c1 = slice(2 * q * h, (2 * q + 1) * h), slice((2 * q + 1) * h, (2 * q + 2) * h)
            A[c0, c1], A[c1, c0] = Ul[c0] @ V[c1].T, Ul[c1] @ V[c0].T
    lib.hsolve(n, 2, r, npart, n, K, U, V)
    assert np.linalg.norm(A @ U[:, :2] - B) <= 8 * n * 2.0 ** -53 * np.linalg.cond(A) ** 2 * np.linalg.norm(B)
    for i in range(npart):
        lu = K[i * m:(i + 1) * m]
        L, R = np.tril(lu, -1) + np.eye(m), np.triu(lu)
        assert (np.abs(L) <= 1.0 + 2.0 ** -50).all()
        P = L @ R
        order = [int(np.argmin(np.abs(D[i] - P[k]).max(axis=1))) for k in range(m)]
        assert sorted(order) == list(range(m))
        assert (np.abs(P - D[i][order]) <= 2 * m * 2.0 ** -53 * (np.abs(L) @ np.abs(R))).all()


@pytest.mark.parametrize("nl,m,k", [(1024, 33, 32), (512, 65, 33), (128, 100, 90), (64, 260, 65)])
def test_mixed_substitutions_by_blocks(lib, nl, m, k):
    """FP32 substitutions for many columns: the refined solution within the
    refinement's tolerance, 1e-12 of the residual, times the condition number."""
    rng = np.random.default_rng(m)
    D = pivoting_blocks(rng, nl, m)
    B = rng.standard_normal((nl * m, k))
    x, _ = factored_leaves(lib, D, B, mixed=True)
    exact = np.linalg.solve(D, B.reshape(nl, m, k)).reshape(-1, k)
    assert np.linalg.norm(x - exact) / np.linalg.norm(exact) <= 2e-12 * max(map(np.linalg.cond, D[:64]))


# factors staged in shared memory or not, by leaf size and number, both ways
@pytest.mark.parametrize("nl,m", [(512, 64), (512, 63), (256, 100), (32, 129), (64, 129), (2, 165)])
@pytest.mark.parametrize("k", [1, 8])
@pytest.mark.parametrize("transpose", [False, True])
def test_few_columns_staged_or_not(lib, nl, m, k, transpose):
    rng = np.random.default_rng(nl + m)
    D = pivoting_blocks(rng, nl, m)
    B = rng.standard_normal((nl * m, k))
    _, s = factored_leaves(lib, D, np.ones((nl * m, 8)))
    b = col(B)
    s.solve(b, transpose=transpose)
    A = D.transpose(0, 2, 1) if transpose else D
    exact = np.linalg.solve(A, B.reshape(nl, m, k)).reshape(-1, k)
    err = np.linalg.norm(b.cpu().numpy() - exact) / np.linalg.norm(exact)
    assert err <= 4 * m * 2.0 ** -53 * max(map(np.linalg.cond, D[:64])) ** 2
