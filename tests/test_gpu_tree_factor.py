"""Subtrees factored side by side (hodlr_tree_factor): the first failure by index
is reported, and the tree factors and solves once its leaves are repaired."""
import numpy as np
import pytest
import torch

from oracle import problems as P
from tests.test_gpu_solver import to_dev, to_host
from tests.test_gpu_tree import make_tree

pytestmark = pytest.mark.gpu


# more subtrees than side streams, too
@pytest.mark.parametrize("top,bad", [(2, [1, 2]), (2, [3]), (4, [5, 13]), (4, [0])])
def test_first_failing_subtree_is_reported(hodlr, top, bad):
    shapes = [(64 if j % 3 else 40, 1 + j % 2, 4) for j in range(1 << top)]
    tp = P.tree_problem(top, shapes, [3] * (2 * ((1 << top) - 1)), nrhs=2, seed=top)
    t = make_tree(hodlr, tp, nrhs=2)
    for _ in range(3):  # eager, captured, replayed
        for j in bad:
            t.subtree(j).set_leaf_blocks(torch.zeros(tp.subs[j].n * tp.subs[j].leaf, dtype=torch.float64, device="cuda"),
                                         ld=tp.subs[j].leaf, leaf_stride=tp.subs[j].leaf ** 2)
        with pytest.raises(hodlr.HodlrError) as e:
            t.factor()
        assert e.value.code == hodlr.HODLR_ERR_SINGULAR_LEAF and "subtree %d:" % bad[0] in str(e.value)
        for j in bad:
            t.subtree(j).set_leaf_blocks(to_dev(tp.subs[j].K))
        t.factor()
        B = to_dev(tp.B)
        t.solve(B)
        R = tp.B - tp.matvec(to_host(B))
        # backward stable in FP64 on a well-conditioned tree of a few thousand rows
        assert np.linalg.norm(R) / np.linalg.norm(tp.B) < 1e-12


def test_subtrees_keep_their_streams(hodlr):
    """A subtree moved to a stream of the caller's: its inputs set there are seen by
    the next factorisation, which leaves it on that stream."""
    shapes = [(64, 2, 4)] * 4
    tp = P.tree_problem(2, shapes, [3] * 6, nrhs=2, seed=1)
    t = make_tree(hodlr, tp, nrhs=2)
    side = torch.cuda.Stream()
    hodlr.check(hodlr.lib().hodlr_set_stream(t.subtree(1).h, side.cuda_stream))
    for _ in range(3):
        with torch.cuda.stream(side):
            D = to_dev(tp.subs[1].K)
            t.subtree(1).set_leaf_blocks(D)
        t.factor()
        B = to_dev(tp.B)
        torch.cuda.synchronize()
        t.solve(B)
        R = tp.B - tp.matvec(to_host(B))
        assert np.linalg.norm(R) / np.linalg.norm(tp.B) < 1e-12
