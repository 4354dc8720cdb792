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
