"""FP64 handles without digit images and without the workspace of the blocked
capacitance factorisation: what a handle is that was created where these would have
taken more than a quarter of the free memory.  HODLR_NO_TCGEN05=1 during the creation
gives the same handle; afterwards it is unset, so that updates and reductions run as
in any other.  Factors, solutions in both directions and saved state agree with those of a
handle that has both."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

U53 = 2.0 ** -53


def col(rows, cols):
    return torch.empty((cols, rows), dtype=torch.float64, device="cuda").t()


def copy(B):
    return B.t().clone().t()


@pytest.mark.parametrize("m,L,r,k", [(64, 4, 16, 20), (128, 3, 40, 3), (256, 2, 16, 20), (256, 3, 64, 9), (100, 3, 20, 20)])
def test_handle_without_images(hodlr, m, L, r, k, monkeypatch):
    n = m << L

    def results(low):
        if low:
            monkeypatch.setenv("HODLR_NO_TCGEN05", "1")
        s = hodlr.Solver(n, m, L, r, nrhs_max=k)
        monkeypatch.setenv("HODLR_NO_TCGEN05", "0")
        B = col(n, k)
        s.generate(3, shift=4.0, B=B)
        out = []
        for _ in range(3):  # eager, captured, replayed
            s.factor()
            x, y = copy(B), copy(B)
            s.solve(x)
            s.solve(y, transpose=True)
            out.append((x, y))
        for x, y in out[1:]:
            assert torch.equal(x, out[0][0]) and torch.equal(y, out[0][1])
        lu = torch.empty(n * m, dtype=torch.float64, device="cuda")
        piv = torch.empty(n, dtype=torch.int32, device="cuda")
        ut, cap = col(n, L * r), torch.empty(((1 << L) - 1) * 4 * r * r, dtype=torch.float64, device="cuda")
        s.get_factors(leaf_lu=lu, leaf_ipiv=piv, utilde=ut, cap_lu=cap)
        A = col(n, k)
        s.matvec(x, A)
        assert float((A - B).norm() / B.norm()) <= 1e-13
        data = s.checkpoint()
        s.close()
        t = hodlr.Solver.from_checkpoint(data)
        z = copy(B)
        t.solve(z)
        t.close()
        return x, y, lu, piv, ut, cap, z

    low, full = results(True), results(False)
    # leaves of condition (4 + 2) / (4 - 2), sums of at most n products
    tol = 4 * m * U53 * 9 * np.sqrt(n / m)
    for i, (a, b) in enumerate(zip(low, full)):
        if a.dtype == torch.int32:
            assert torch.equal(a, b)
        else:
            assert float((a - b).norm() / b.norm()) <= tol, i
    # the loaded handle's solution: of a handle that may have the images by then
    for x, z in ((low[0], low[6]), (full[0], full[6])):
        assert float((x - z).norm() / x.norm()) <= tol
