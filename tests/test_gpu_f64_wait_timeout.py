"""Bounded waits of the FP64 tensor-core kernels that run out (no GPU fault, no
hang), through every call that launches one.

The test hook hodlr_debug_wait_fault makes one CTA withhold the announcement of one
tile's, row group's or chunk's digits, so nothing completes the wait for them: it
ends by its short clock budget, the CTA's roles stop, and the call has to report
HODLR_ERR_TIMEOUT with the CTA's index.  With the hook off the same call then gives
the bits it gave before."""
import threading

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

F64 = torch.float64


def rand(rows, cols, seed):
    g = torch.Generator(device="cuda").manual_seed(seed)
    return torch.randn((cols, rows), dtype=F64, device="cuda", generator=g).t()


def zeros(rows, cols):
    return torch.zeros((cols, rows), dtype=F64, device="cuda").t()


def times_out(fs, cta, stage, call):
    """call() before, with the hook on and after it: the status between, the same result around it."""
    before = call()
    fs.debug_wait_fault(cta, stage, budget_cycles=200000)
    try:
        with pytest.raises(fs.HodlrError) as e:
            call()
    finally:
        fs.debug_wait_fault(-1)
    assert e.value.code == fs.HODLR_ERR_TIMEOUT
    assert "(index %d)" % cta in str(e.value)
    for a, b in zip(before, call()):
        assert torch.equal(a, b)


@pytest.mark.parametrize("cta,stage", [(0, 0), (3, 5)])
def test_gemm_broadcast(hodlr, cta, stage):
    n, K, N = 128 * 608, 32, 64
    U, B = rand(n, K, 1), rand(K, N, 2)

    def call():
        W = zeros(n, N)
        hodlr.check(hodlr.lib().hodlr_gemm_broadcast(n, 1, 1, K, N, 1.0, U.data_ptr(), n, B.data_ptr(), K, 1.0,
                                                     W.data_ptr(), n))
        return [W]

    times_out(hodlr, cta, stage, call)


@pytest.mark.parametrize("name", ["hodlr_gemm_reduce", "hodlr_gemm_reduce_noalloc"])
@pytest.mark.parametrize("cta,stage", [(1, 0), (0, 2)])
def test_gemm_reduce(hodlr, name, cta, stage):
    n, r, C = 1 << 16, 32, 64
    V, X = rand(n, r, 3), rand(n, C, 4)

    def call():
        W = zeros(r, C)
        hodlr.check(getattr(hodlr.lib(), name)(n, 1, r, C, V.data_ptr(), n, X.data_ptr(), n, W.data_ptr(), r))
        return [W]

    times_out(hodlr, cta, stage, call)


@pytest.mark.parametrize("m", [128, 256])
@pytest.mark.parametrize("stage", [0, 1])
def test_leaf_application(hodlr, m, stage):
    """One leaf and no level: the solve is its application."""
    s = hodlr.Solver(m, m, 0, 1, nrhs_max=16)
    s.set_leaf_blocks((rand(m, m, 5) / m ** 0.5 + 4.0 * torch.eye(m, dtype=F64, device="cuda")).t().contiguous().t())
    s.factor()
    B = rand(m, 16, 6)

    def call():
        X = B.t().clone().t()
        s.solve(X)
        return [X]

    times_out(hodlr, 0, stage, call)
    s.close()


def test_node_solve(hodlr):
    nn, r, k = 200, 16, 32
    Tu, Td = rand(2 * r * nn, r, 7) / 8.0, rand(2 * r * nn, k, 8)

    def call():
        X = Td.t().clone().t()
        hodlr.check(hodlr.lib().hodlr_node_solve(nn, r, k, Tu.data_ptr(), 2 * r * nn, X.data_ptr(), 2 * r * nn))
        return [X]

    times_out(hodlr, 0, 0, call)


M, L, R, K = 128, 4, 16, 16
N = M << L


def handle(fs):
    s = fs.Solver(N, M, L, R, nrhs_max=K)
    B = zeros(N, K)
    s.generate(31, shift=4.0, B=B)
    return s, B


@pytest.mark.parametrize("what", ["factor", "solve", "matvec", "matvec transposed", "adjoint", "set_uvd", "generate"])
def test_calls_of_a_handle(hodlr, what):
    s, B = handle(hodlr)
    s.factor()
    X = B.t().clone().t()
    s.solve(X)
    e = lambda c: torch.zeros(c, dtype=F64, device="cuda")  # noqa: E731

    def call():
        if what == "factor":
            s.factor()
            ut = zeros(N, L * R)
            s.get_factors(utilde=ut)
            return [ut]
        Y = B.t().clone().t()
        if what == "solve":
            s.solve(Y)
            return [Y]
        if what.startswith("matvec"):
            s.matvec(X, Y, transpose="transposed" in what)
            return [Y]
        if what == "adjoint":
            g = {"db": zeros(N, K), "dD": e(N * M), "dU": e(L * N * R), "dV": e(L * N * R), "ds": e(L * R)}
            s.adjoint(X, B, **g)
            return list(g.values())
        D = e(N * M)
        if what == "generate":
            s.generate(31, shift=4.0, orthonormal=True)
            U = e(L * N * R)
            s.get_inputs(U=U)
            return [U]
        U, V = rand(N, R, 9), rand(N, R, 10)
        d = torch.ones(N, dtype=F64, device="cuda")
        hodlr.check(hodlr.lib().hodlr_set_uvd(s.h, U.data_ptr(), N, V.data_ptr(), N, d.data_ptr()))
        s.get_inputs(D=D)
        return [D]

    times_out(hodlr, 0, 0, call)
    s.close()


def test_calls_without_a_handle_from_many_threads(hodlr):
    """More callers than status words are not needed to wait for each other's results."""
    n, K, C = 128 * 20, 16, 40
    U, B, V = rand(n, K, 11), rand(K, C, 12), rand(n, C, 13)
    torch.cuda.synchronize()
    want = (U @ B).cpu().numpy(), (U.t() @ V).cpu().numpy()
    bad = []

    def work():
        for _ in range(4):
            W, T = zeros(n, C), zeros(K, C)
            torch.cuda.synchronize()
            for rc in (hodlr.lib().hodlr_gemm_broadcast(n, 1, 1, K, C, 1.0, U.data_ptr(), n, B.data_ptr(), K, 1.0,
                                                        W.data_ptr(), n),
                       hodlr.lib().hodlr_gemm_reduce(n, 1, K, C, U.data_ptr(), n, V.data_ptr(), n, T.data_ptr(), K)):
                if rc != hodlr.HODLR_OK:
                    bad.append(rc)
            for got, w in zip((W, T), want):
                if not np.allclose(got.cpu().numpy(), w, rtol=0, atol=1e-10):
                    bad.append("values")

    threads = [threading.Thread(target=work) for _ in range(80)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not bad
