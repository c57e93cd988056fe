"""Inputs set from device memory (csrc/set_inputs.cu: one pass for the copy and
everything derived from it) against the same inputs set from host memory, bit
for bit: layouts whose alignment or leading dimension the wide accesses do not
take, odd sizes, the stacked column-major leaf layout, a batch's row offsets."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.fixture()
def lib():
    import fastsolver2_gb300 as fs
    return fs


def placed(a, ld, offset):
    """Column-major copy of a on the device: leading dimension ld, `offset` doubles into its allocation."""
    rows, cols = a.shape
    buf = torch.zeros(offset + ld * cols, dtype=torch.float64, device="cuda")
    view = torch.as_strided(buf, (rows, cols), (1, ld), offset)
    view.copy_(torch.from_numpy(a))
    return view


# sizes with and without the tensor-core residual, odd row counts; leading dimension and base offset
@pytest.mark.parametrize("leaf,levels,rank", [(64, 2, 8), (128, 1, 32), (256, 1, 40), (100, 2, 13), (33, 1, 5)])
@pytest.mark.parametrize("pad,offset", [(0, 0), (2, 0), (1, 1), (0, 1), (8, 2)])
@pytest.mark.parametrize("mixed", [False, True])
def test_device_and_host_inputs_give_the_same_bits(lib, leaf, levels, rank, pad, offset, mixed):
    rng = np.random.default_rng(leaf + pad)
    n, nl = leaf << levels, 1 << levels
    K = rng.standard_normal((n, leaf)) / np.sqrt(leaf)
    for i in range(nl):
        K[i * leaf:(i + 1) * leaf] += 4.0 * np.eye(leaf)
    Us, Vs = ([rng.standard_normal((n, rank)) / np.sqrt(n) for _ in range(levels)] for _ in range(2))
    B = np.asfortranarray(rng.standard_normal((n, 3)))
    out = []
    for device in (False, True):
        s = lib.Solver(n, leaf, levels, rank, nrhs_max=3, precision=lib.PREC_MIXED if mixed else lib.PREC_FP64)
        put = (lambda a: placed(a, n + pad, offset)) if device else (lambda a: torch.from_numpy(np.asfortranarray(a)))
        keep = [put(K)]
        s.set_leaf_blocks(keep[0], ld=n + pad if device else n)
        for l in range(levels):
            keep += [put(Us[l]), put(Vs[l])]
            s.set_lowrank(l, keep[-2], keep[-1])
        torch.cuda.synchronize()
        s.factor()
        b = torch.from_numpy(B.T.copy()).cuda().t()
        s.solve(b)
        D = torch.zeros(nl * leaf * leaf, dtype=torch.float64)
        U, V = (torch.zeros(levels * n * rank, dtype=torch.float64) for _ in range(2))
        s.get_inputs(D=D, U=U, V=V)
        out.append([x.cpu().numpy() for x in (b, D, U, V)])
        s.close()
    for host, dev in zip(*out):
        assert np.array_equal(host, dev)


@pytest.mark.parametrize("mixed", [False, True])
def test_batch_device_and_host_inputs_give_the_same_bits(lib, mixed):
    rng = np.random.default_rng(3)
    systems = [(512, 128, 2, 16, 2), (256, 128, 1, 16, 1), (256, 64, 2, 8, 3), (128, 64, 1, 8, 1)]
    data = []
    for n, m, L, r, k in systems:
        D = rng.standard_normal((n // m, m, m)) / np.sqrt(m) + 4.0 * np.eye(m)
        data.append((D, [[rng.standard_normal((n, r)) / np.sqrt(n) for _ in range(2)] for _ in range(L)],
                     rng.standard_normal((n, k))))
    out = []
    for device in (False, True):
        b = lib.Batch(systems, precision=lib.PREC_MIXED if mixed else lib.PREC_FP64)
        for i, ((n, m, L, r, k), (D, UV, _)) in enumerate(zip(systems, data)):
            d = torch.from_numpy(np.ascontiguousarray(D.transpose(0, 2, 1)))
            b.set_leaf_blocks(i, d.cuda() if device else d, ld=m, leaf_stride=m * m)
            for l, (U, V) in enumerate(UV):
                u, v = (torch.from_numpy(np.asfortranarray(x)) for x in (U, V))
                sv = torch.linspace(1.0, 0.5, r, dtype=torch.float64) if l else None
                if device:
                    u, v = u.t().cuda().t(), v.t().cuda().t()
                b.set_lowrank(i, l, u, v, sv.cuda() if device and sv is not None else sv)
        b.factor()
        Xs = [torch.from_numpy(B.T.copy()).cuda().t() for _, _, B in data]
        torch.cuda.synchronize()
        b.solve(Xs)
        out.append([x.cpu().numpy() for x in Xs])
        b.close()
    for host, dev in zip(*out):
        assert np.array_equal(host, dev)
