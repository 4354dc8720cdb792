"""The branch-free rotation chain and the one-warp Cholesky factor where their
fast paths end: operands whose products leave the range the relative test is
decided in (tiny, huge: every rotation takes the IEEE operations), equal column
norms (a quotient of zero), nearly orthogonal columns (angles at the relative
test and at the large-cotangent limit), strongly graded hyperbolic columns
(reciprocal roots of 1 - t^2 next to 1).  Bits against the CPU oracle."""

import numpy as np
import pytest

from gpujachx_b200 import synth

pytestmark = pytest.mark.gpu

M, N = 128, 64


def _hadamard(n):
    h = np.ones((1, 1))
    while h.shape[0] < n:
        h = np.block([[h, h], [h, -h]])
    return h


def _input(kind):
    r = np.random.default_rng(17)
    g = r.standard_normal((M, N))
    if kind == "tiny":
        return g * 2.0 ** -300
    if kind == "huge":
        return g * 2.0 ** 300
    if kind == "equal_norms":  # exact +-1 columns, some pairs far from orthogonal
        h = _hadamard(M)[:, :N].copy()
        h[:, 1::2] = np.where(r.random((M, N // 2)) < 0.1, -h[:, 1::2], h[:, 1::2])
        return h
    if kind == "nearly_orthogonal":
        q = np.linalg.qr(g)[0]
        return q + q @ np.triu(10.0 ** r.uniform(-17.0, -5.0, (N, N)), 1)
    return synth.graded(M, N, 5, lo=-12.0)  # "graded"


@pytest.mark.parametrize("alg,nplus", [(3, N), (11, N), (11, 23), (8, 40), (3, 23)])
@pytest.mark.parametrize("kind", ["tiny", "huge", "equal_norms", "nearly_orthogonal", "graded"])
def test_same_bits_as_the_oracle(kind, alg, nplus, built, oracle):
    import gpujachx_b200 as g
    G = _input(kind)
    g.init_strats(built["strat"], "cycwor", 32, "cycwor", N // 16)
    r = g.hypJacL2(alg, G, nplus)
    o = oracle.hypjac_l2(alg, G, nplus, oracle.load_strat(built["strat"], "cycwor", 32),
                         oracle.load_strat(built["strat"], "cycwor", N // 16))
    assert (r.sweeps, r.rot_s, r.rot_b) == (o["sweeps"], o["rot_s"], o["rot_b"])
    for a, b in ((r.U, o["G"]), (r.V, o["V"]), (r.D, o["D"])):
        if a is not None:
            assert np.array_equal(a.view(np.uint64), b.view(np.uint64))


@pytest.mark.parametrize("exponents", [(-1070, 1020), (-2, 2), (-1, 0)])
def test_reciprocal_square_root_is_correctly_rounded(exponents, built, oracle):
    """rsqrt_rn on random significands, all-zero and all-one tails among them,
    over the whole range and next to 1 and 4."""
    import ctypes

    import torch

    import gpujachx_b200 as g
    r = np.random.default_rng(3)
    n = 20000
    m = r.integers(0, 1 << 52, n, dtype=np.uint64)
    m[::5] &= np.uint64(0xF)
    m[1::5] |= np.uint64((1 << 52) - 16)
    x = np.ldexp(1.0 + m.astype(np.float64) * 2.0 ** -52, r.integers(exponents[0], exponents[1], n))
    t = torch.from_numpy(x).cuda()
    out = torch.empty_like(t)
    assert g.lib().gjx_rsqrt_rn_dev(ctypes.c_void_p(t.data_ptr()), ctypes.c_void_p(out.data_ptr()), n) == 0
    torch.cuda.synchronize()
    want = np.array([oracle.rsqrt_rn(v) for v in x])
    assert np.array_equal(out.cpu().numpy().view(np.uint64), want.view(np.uint64))


def _significands(r, n):
    """Random ones, few leading or trailing bits set, next to 1 and 2."""
    m = r.integers(0, 1 << 52, n, dtype=np.uint64)
    m[::7] &= np.uint64(0xF)
    m[1::7] |= np.uint64((1 << 52) - 16)
    m[2::7] &= ~np.uint64((1 << 40) - 1)
    return 1.0 + m.astype(np.float64) * 2.0 ** -52


def _midpoint(q):
    """q + ulp(q) / 2, a float between two neighbours: as an exact fraction."""
    from fractions import Fraction
    return (Fraction(float(q)) + Fraction(float(np.nextafter(q, np.inf)))) / 2


@pytest.mark.parametrize("op", [0, 1, 2, 3, 4])
def test_proved_operations(op, built, oracle):
    """What the branch-free quotient, reciprocal, roots and the series next to 1
    declare proved is the IEEE operation's result (the correctly rounded
    reciprocal root for the last two), on random operands and on operands whose
    result lies as near to a midpoint of two floats as one operand can put it; and
    they prove all but a few of the random ones."""
    import torch

    import gpujachx_b200 as g
    r = np.random.default_rng(11 + op)
    n, hard = 200000, 20000
    e = r.integers(-300, 300, n) if op < 2 else 2 * r.integers(-300, 300, n) + r.integers(0, 2, n)
    a = np.ldexp(_significands(r, n), e)
    h = np.ldexp(_significands(r, n), r.integers(-300, 300, n)) * r.choice([-1.0, 1.0], n)
    if op < 2:
        a *= r.choice([-1.0, 1.0], n)
    if op == 4:  # 1 +- t^2, t from 2^-60 to 2^-10 (proved below 2^-15)
        t = np.ldexp(_significands(r, n), r.integers(-60, -10, n))
        a = 1.0 + np.where(r.random(n) < 0.5, 1.0, -1.0) * t * t
    else:
        q = 1.0 + r.random(hard)
        for i in range(hard):
            m = _midpoint(q[i])
            if op == 0:
                h[i] = float(m * abs(_frac(a[i])))
            elif op == 1:
                a[i] = float(1 / m)
            elif op == 2:
                a[i] = float(m * m)
            else:
                a[i] = float(1 / (m * m))
    dh, da = torch.from_numpy(h).cuda(), torch.from_numpy(a).cuda()
    out, ok = torch.empty_like(da), torch.zeros(n, dtype=torch.int32, device="cuda")
    assert g.lib().gjx_exact_ops_dev(op, dh.data_ptr(), da.data_ptr(), out.data_ptr(), ok.data_ptr(), n) == 0
    out, ok = out.cpu().numpy(), ok.cpu().numpy() != 0
    want = (h / a if op == 0 else 1.0 / a if op == 1 else np.sqrt(a) if op == 2 else
            np.array([oracle.rsqrt_rn(v) for v in a]))
    assert np.array_equal(out[ok].view(np.uint64), want[ok].view(np.uint64))
    plain = np.arange(n) >= hard
    if op == 4:
        plain &= np.abs(1.0 - a) < 2.0 ** -30
        assert ok[plain].all() and plain.sum() > n // 2
        assert not ok[np.abs(1.0 - a) >= 2.0 ** -30].any()
    else:
        plain &= np.arange(n) % 7 > 2
        assert ok[plain].mean() > 0.99
    assert g.lib().gjx_exact_ops_dev(5, 0, 0, 0, 0, 0) == -1


def _frac(x):
    from fractions import Fraction
    return Fraction(float(x))
