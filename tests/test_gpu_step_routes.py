"""The routes of a single decomposition's outer steps against the fused step
kernel with one CTA per block pair, which the other tests hold against the
oracle: clusters of 8 CTAs per pair; the update as a launch of its own, its
stages dealt out to all SMs, with 1 to 8 CTAs per pair before it, with more
pairs than SMs, with partial stages and with pairs that do not change; and the
split form with V updated beside the next step's pair kernel.  The same bits."""

import numpy as np
import pytest

from gpujachx_b200 import synth

pytestmark = pytest.mark.gpu


def _same(a, b, full):
    assert (a.sweeps, a.rot_s, a.rot_b) == (b.sweeps, b.rot_s, b.rot_b)
    for x, y in ((a.U, b.U), (a.D, b.D)) + (((a.V, b.V),) if full else ()):
        assert np.array_equal(x.view(np.uint64), y.view(np.uint64))


def _fused(g, alg, G, nplus):
    """One CTA per block pair, one pair at a time, the update by the step kernel."""
    g.lib().gjx_set_sweep_mode(0)
    g.lib().gjx_set_split(1)
    g.lib().gjx_set_pairs_per_cta(1)
    try:
        return g.hypJacL2(alg, G, nplus)
    finally:
        g.lib().gjx_set_split(0)
        g.lib().gjx_set_pairs_per_cta(0)


@pytest.mark.parametrize("m,n,nplus,alg", [(64, 32, 32, 11), (1088, 64, 20, 11), (4096, 192, 192, 10), (2112, 256, 100, 3),
                                           (1024, 512, 512, 9)])
@pytest.mark.parametrize("split", [0, 2, 4, 8])
def test_clusters(m, n, nplus, alg, split, built):
    import gpujachx_b200 as g
    G = synth.make("graded", m, n, 5)
    g.init_strats(None, "cycwor", 32, "cycwor", n // 16)
    ref = _fused(g, alg, G, nplus)
    g.lib().gjx_set_split(split)
    try:
        _same(g.hypJacL2(alg, G, nplus), ref, alg & 2)
    finally:
        g.lib().gjx_set_split(0)
        g.lib().gjx_set_sweep_mode(-1)


@pytest.mark.parametrize("m,n,nplus,alg", [(6016, 640, 640, 11), (8256, 896, 300, 10), (3072, 2560, 2560, 9),
                                           (3136, 3072, 1000, 11), (5120, 5120, 5120, 9)])
def test_update_launch(m, n, nplus, alg, built):
    import gpujachx_b200 as g
    G = synth.make("gaussian", m, n, 6)
    g.init_strats(None, "cycwor", 32, "cycwor", n // 16)
    ref = _fused(g, alg, G, nplus)
    g.lib().gjx_set_sweep_mode(-1)
    g.profile(False)
    r = g.hypJacL2(alg, G, nplus)
    assert g.profile_read()["launches"] > 2 * (n // 16 - 1) * r.sweeps  # two launches a step
    _same(r, ref, alg & 2)


def test_update_launch_with_unchanged_pairs(built):
    """Blocks orthogonal to each other (ALG 10 does not sort).  In some each column
    has one entry, in a row of its own: their Gram matrices are diagonal, so a
    pair of two of them rotates nothing and its flag is clear."""
    import gpujachx_b200 as g
    m, n = 8192, 640
    r = np.random.default_rng(4)
    G = np.zeros((m, n), order="F")
    for b in range(n // 16):
        blk = r.standard_normal((m // 64, 16))
        G[b * (m // 64):(b + 1) * (m // 64), 16 * b:16 * b + 16] = blk if b % 5 == 0 else np.linalg.qr(blk)[0] * 2.0 ** (b % 7)
        if b % 5 > 2:
            G[:, 16 * b:16 * b + 16] = 0.0
            G[b * (m // 64) + np.arange(16), 16 * b + np.arange(16)] = 3.0 * 2.0 ** (np.arange(16) % 3)
    g.init_strats(None, "cycwor", 32, "cycwor", n // 16)
    ref = _fused(g, 10, G, n)
    g.lib().gjx_set_sweep_mode(-1)
    g.profile(False)
    r = g.hypJacL2(10, G, n)
    assert g.profile_read()["launches"] > 2 * (n // 16 - 1) * r.sweeps  # two launches a step
    _same(r, ref, True)
    keep = np.flatnonzero(np.arange(n) // 16 % 5 > 2)  # the columns of those blocks
    assert np.array_equal(r.U[:, keep], (G[:, keep] != 0.0).astype(float))
    assert np.array_equal(r.V[:, keep], np.eye(n)[:, keep])


@pytest.mark.parametrize("m,n,nplus,alg,beside", [(64, 64, 64, 11, False), (1088, 320, 100, 11, True), (2112, 2048, 2048, 3, True),
                                                  (512, 512, 512, 10, True), (192, 128, 60, 11, True),
                                                  (5120, 5120, 5120, 10, False)])
def test_split_form_with_v_beside(m, n, nplus, alg, beside, built):
    """Timed (gjx_profile) launches keep V's update on the main stream: two
    launches a step, with V beside four (and initV, the maxima of V and of G,
    initD).  Not beside: one step a sweep, and too little room beside 80 pairs."""
    import torch

    import gpujachx_b200 as g
    G = synth.make("graded" if nplus < n else "gaussian", m, n, 8) if n < 5120 else np.diag(np.logspace(0.0, -4.0, n))
    g.init_strats(None, "cycwor", 32, "cycwor", n // 16)
    runs = []
    for timed in (True, False):
        dG = torch.tensor(np.ascontiguousarray(G.T), device="cuda")
        dV = torch.zeros((n, n), dtype=torch.float64, device="cuda")
        dD = torch.zeros(n, dtype=torch.float64, device="cuda")
        g.profile(timed)
        counts = g.hypJacL2_split(alg, dG, nplus, dV, dD)
        per_step = 4 if beside and not timed else 2
        assert g.profile_read()["launches"] == 4 + per_step * (n // 32 - 1) * counts[1]
        g.profile(False)
        runs.append((counts, dG.cpu().numpy(), dV.cpu().numpy(), dD.cpu().numpy()))
    a, b = runs
    assert a[0] == b[0]
    for x, y in zip(a[1:], b[1:]):
        assert np.array_equal(x.view(np.uint64), y.view(np.uint64))
