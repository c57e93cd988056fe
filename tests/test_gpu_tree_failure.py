"""What a failed hodlr_tree_factor leaves behind: the subtrees before the one that
failed are factored, those after it are as they were."""
import pytest
import torch

from oracle import problems as P
from tests.test_gpu_solver import to_dev
from tests.test_gpu_tree import make_tree

pytestmark = pytest.mark.gpu


def factored(hodlr, t, j, n):
    """Whether subtree j answers a request for its factors."""
    ipiv = torch.zeros(n, dtype=torch.int32, device="cuda")
    rc = hodlr.lib().hodlr_get_factors(t.subtree(j).h, None, ipiv.data_ptr(), None, None, None)
    assert rc in (hodlr.HODLR_OK, hodlr.HODLR_ERR_NOT_FACTORED)
    return rc == hodlr.HODLR_OK


@pytest.mark.parametrize("top,bad", [(2, 0), (2, 1), (4, 5), (4, 15)])
def test_subtrees_after_the_failing_one_are_as_they_were(hodlr, top, bad):
    nsub = 1 << top
    tp = P.tree_problem(top, [(64 if j % 3 else 40, 1, 4) for j in range(nsub)], [3] * (2 * (nsub - 1)), nrhs=2, seed=top)
    t = make_tree(hodlr, tp, nrhs=2)
    sub = tp.subs[bad]
    zero = torch.zeros(sub.n * sub.leaf, dtype=torch.float64, device="cuda")
    t.subtree(bad).set_leaf_blocks(zero, ld=sub.leaf, leaf_stride=sub.leaf ** 2)
    with pytest.raises(hodlr.HodlrError):
        t.factor()
    assert [factored(hodlr, t, j, tp.subs[j].n) for j in range(nsub)] == [j < bad for j in range(nsub)]
    # once factored, they stay so
    t.subtree(bad).set_leaf_blocks(to_dev(sub.K))
    t.factor()
    t.subtree(bad).set_leaf_blocks(zero, ld=sub.leaf, leaf_stride=sub.leaf ** 2)
    last = nsub - 1
    t.subtree(last).set_leaf_blocks(to_dev(tp.subs[last].K)) if last != bad else None
    with pytest.raises(hodlr.HodlrError):
        t.factor()
    assert [factored(hodlr, t, j, tp.subs[j].n) for j in range(nsub)] == [j != bad and (j < bad or j != last)
                                                                         for j in range(nsub)]
