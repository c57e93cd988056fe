"""The reciprocal and the quotients of the FP64 panels (csrc/dense_ops.cuh) against
exact rational arithmetic and against the GPU's own division.

Bounds, from their derivation beside the code: newton_rcp 0.52 ulp; Quotient
0.5 + 2^-40 ulp where neither the quotient nor its second part (2^-53 of it) is
subnormal, 1 ulp below that."""
import ctypes
import math
import os
import subprocess
from fractions import Fraction

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


@pytest.fixture(scope="module")
def helpers(tmp_path_factory):
    so = str(tmp_path_factory.mktemp("reciprocals") / "reciprocals.so")
    subprocess.check_call(["nvcc", "-gencode", "arch=compute_103a,code=sm_103a", "-O3", "-std=c++17", "-shared",
                           "-Xcompiler", "-fPIC", "-I" + os.path.join(ROOT, "fastsolver2_gb300", "csrc"),
                           "-I" + os.path.join(ROOT, "include"), os.path.join(ROOT, "tests", "cpp", "reciprocals.cu"),
                           "-o", so])
    lib = ctypes.CDLL(so)
    for f in (lib.reciprocals, lib.quotients):
        f.restype = ctypes.c_char_p
    return lib


def mantissas(rng, n):
    """1 <= m < 2: random ones, and those next to powers of two, to 3/2 and to sqrt(2)."""
    edge = [1.0, math.nextafter(1.0, 2.0), 1.0 + 2.0 ** -26, 1.5, math.nextafter(1.5, 2.0), math.sqrt(2.0),
            2.0 - 2.0 ** -52, 2.0 - 2.0 ** -51, 2.0 - 2.0 ** -26]
    return np.concatenate([edge, rng.uniform(1.0, 2.0, n - len(edge))])


def dev(a):
    return torch.from_numpy(np.ascontiguousarray(a)).cuda()


def p(t):
    return ctypes.c_void_p(t.data_ptr())


def ulps(got, exact):
    """|got - exact| in units of the last place of got's binade (2^-1074 at least)."""
    return abs(Fraction(got) - exact) / Fraction(math.ulp(got))


@pytest.mark.parametrize("exponent", [-960, -959, -700, -53, -1, 0, 1, 52, 700, 959, 960])
def test_reciprocal(helpers, exponent):
    rng = np.random.default_rng(exponent + 1000)
    x = np.ldexp(mantissas(rng, 3000), exponent) * rng.choice([-1.0, 1.0], 3000)
    y, div = (torch.zeros(x.size, dtype=torch.float64, device="cuda") for _ in range(2))
    usual = torch.zeros(x.size, dtype=torch.int32, device="cuda")
    assert helpers.reciprocals(p(dev(x)), x.size, p(y), p(usual), p(div)) is None
    assert usual.all()
    y, div = y.cpu().numpy(), div.cpu().numpy()
    worst = max(ulps(float(b), 1 / Fraction(float(a))) for a, b in zip(x, y))
    assert worst <= 0.52, float(worst)
    assert np.abs((y - div) / np.spacing(np.abs(div))).max() <= 1.0


def test_reciprocal_range(helpers):
    """What rcp_usual leaves to the division."""
    x = np.array([0.0, -0.0, 5e-324, 1e-310, 2.0 ** -961, 2.0 ** 961, 1e300, np.inf, -np.inf, np.nan])
    y, div = (torch.zeros(x.size, dtype=torch.float64, device="cuda") for _ in range(2))
    usual = torch.ones(x.size, dtype=torch.int32, device="cuda")
    assert helpers.reciprocals(p(dev(x)), x.size, p(y), p(usual), p(div)) is None
    assert not usual.any()


@pytest.mark.parametrize("eu", [-929, -500, -1, 0, 1, 500, 929])
@pytest.mark.parametrize("ex", [-1060, -1022, -600, 0, 600, 1023])
def test_quotients(helpers, eu, ex):
    rng = np.random.default_rng([eu + 2000, ex + 2000])
    n = 1200
    u = np.ldexp(mantissas(rng, n), eu) * rng.choice([-1.0, 1.0], n)
    x = np.ldexp(rng.permutation(mantissas(rng, n)), ex) * rng.choice([-1.0, 1.0], n)
    x[:3] = u[:3] * 3.0  # exact quotients
    q, div = (torch.zeros(n, dtype=torch.float64, device="cuda") for _ in range(2))
    assert helpers.quotients(p(dev(u)), p(dev(x)), n, p(q), p(div)) is None
    q, div = q.cpu().numpy(), div.cpu().numpy()
    finite = np.isfinite(div)
    assert np.array_equal(q[~finite], div[~finite])
    for a, b, c, d in zip(u[finite], x[finite], q[finite], div[finite]):
        exact = Fraction(float(b)) / Fraction(float(a))
        normal = abs(exact) >= Fraction(2) ** -960
        assert ulps(float(c), exact) <= (Fraction(1, 2) + Fraction(1, 2 ** 40) if normal else 1), (a, b, c)
        assert abs(c - d) <= math.ulp(d)


def test_quotients_of_extremes(helpers):
    """Divisors and dividends that are left to the division, and their signs."""
    e = np.array([0.0, -0.0, 5e-324, -1e-310, 1e-281, 1.0, -3.0, 1e281, 1e308, np.inf, -np.inf, np.nan])
    u, x = (a.ravel() for a in np.meshgrid(e, e))
    q, div = (torch.zeros(u.size, dtype=torch.float64, device="cuda") for _ in range(2))
    assert helpers.quotients(p(dev(u)), p(dev(x)), u.size, p(q), p(div)) is None
    q, div = q.cpu().numpy(), div.cpu().numpy()
    assert np.array_equal(np.isnan(q), np.isnan(div))
    some = ~np.isnan(div)
    assert np.array_equal(np.signbit(q[some]), np.signbit(div[some]))
    usual = np.isin(np.abs(u), (1.0, 3.0))
    assert np.array_equal(q[some & ~usual], div[some & ~usual])
    with np.errstate(invalid="ignore"):
        d = np.abs(q[some & usual] - div[some & usual])
    assert (d[np.isfinite(d)] <= np.spacing(np.abs(div[some & usual][np.isfinite(d)]))).all()
