"""HODLR_RESID_FP64 is the residual in native FP64: a caller who asks for it gets FMAs.

The shape (leaf 100, rank 16, mixed) puts no other kernel of a solve under the test
hook of the bounded waits, which stops the FP64 tensor-core kernels."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("transpose", [False, True])
@pytest.mark.parametrize("k", [9, 16])
def test_native_residual_takes_no_tensor_core_kernel(hodlr, transpose, k):
    m, L, r = 100, 3, 16  # 400, 200 and 100 rows a block
    n = m << L
    s = hodlr.Solver(n, m, L, r, nrhs_max=k, precision=hodlr.PREC_MIXED, residual=hodlr.RESID_FP64)
    B = torch.empty((k, n), dtype=torch.float64, device="cuda").t()
    s.generate(5, shift=4.0, B=B)
    s.factor()
    hodlr.debug_wait_fault(0, 0, budget_cycles=200000)
    try:
        for _ in range(3):  # eager, captured, replayed
            X = B.t().clone().t()
            info = s.solve(X, transpose=transpose)
            assert info.status == hodlr.HODLR_OK and info.rel_residual <= 1e-12
    finally:
        hodlr.debug_wait_fault(-1)
    s.close()
