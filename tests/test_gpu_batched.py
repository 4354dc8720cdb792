"""The batched form (gjx_hypJacL2_batched): every matrix of a batch gets
exactly what the single-matrix device call gives it -- U, V, D bit for bit,
sweeps and rotation counts -- for mixed sizes (64..512 columns, square and
tall), mixed signatures (J = I, J = -I, mixed), all four kernel variants
(ALG 3, 9, 11, 1), one and two block pairs per CTA of 8 warps and of 4 warps (two CTAs per SM), and a
matrix with invalid arguments that is reported and left alone while the others run."""

import numpy as np
import pytest

from gpujachx_b200 import synth


def _dev(G, full):
    import torch
    m, n = G.shape
    dG = torch.tensor(np.ascontiguousarray(G.T), dtype=torch.float64, device="cuda")
    dV = torch.zeros((n, n), dtype=torch.float64, device="cuda") if full else None
    dD = torch.zeros(n, dtype=torch.float64, device="cuda")
    return dG, dV, dD


def _bits(t):
    return t.cpu().numpy().view(np.uint64)


CASES = [(64, 64, 64), (128, 128, 64), (192, 192, 0), (256, 256, 256), (320, 320, 160), (384, 384, 384),
         (448, 448, 224), (512, 512, 512), (256, 128, 128), (512, 256, 100), (128, 64, 32), (640, 320, 320)]


@pytest.mark.gpu
@pytest.mark.parametrize("mode", [0, 1])
@pytest.mark.parametrize("width", [2, 1, 3, 4])
@pytest.mark.parametrize("alg", [11, 9, 3, 1])
def test_batched_equals_single(built, alg, width, mode):
    import torch
    import gpujachx_b200 as g
    g.lib().gjx_set_pairs_per_cta(width)   # 2 (4): two block pairs per CTA (of 4 warps), from different matrices too
    g.lib().gjx_set_batch_mode(mode)       # 0: one launch per step index, 1: one launch per sweep
    g.init_strats(None, "cycwor", 32, "cycwor", 4)   # the family; each matrix takes its own n1 table
    full = bool(alg & 2)
    mats = []
    for k, (m, n, p) in enumerate(CASES):
        gen = "svd_synth" if m == n else "graded"
        G = synth.make(gen, m, n, 5000 + k, **({"smin": 1e-6} if gen == "svd_synth" else {}))
        mats.append((G, p))
    batch = [_dev(G, full) for G, _ in mats]
    res = g.hypJacL2_batched(alg, [b[0] for b in batch], [p for _, p in mats], Vs=[b[1] for b in batch] if full else None,
                             Ds=[b[2] for b in batch])
    g.lib().gjx_set_pairs_per_cta(0)
    g.lib().gjx_set_batch_mode(-1)
    assert res.info == [0] * len(mats)
    for k, (G, p) in enumerate(mats):
        n = G.shape[1]
        g.init_strats(None, "cycwor", 32, "cycwor", n // 16)
        dG, dV, dD = _dev(G, full)
        ret, sw, rs, rb = g.hypJacL2_dev(alg, dG, p, dV, dD)
        torch.cuda.synchronize()
        assert (res.sweeps[k], res.rot_s[k], res.rot_b[k]) == (sw, rs, rb), (k, CASES[k])
        assert np.array_equal(_bits(batch[k][0]), _bits(dG)), k
        assert np.array_equal(_bits(batch[k][2]), _bits(dD)), k
        if full:
            assert np.array_equal(_bits(batch[k][1]), _bits(dV)), k


@pytest.mark.gpu
def test_batched_bad_matrix_is_reported(built):
    import torch
    import gpujachx_b200 as g
    g.init_strats(None, "cycwor", 32, "cycwor", 4)
    G1 = synth.gaussian(128, 64, 1)
    good = _dev(G1, True)
    bad = _dev(synth.gaussian(96, 48, 2), True)          # 96 rows: not a multiple of 64
    keep = bad[0].clone()
    res = g.hypJacL2_batched(11, [good[0], bad[0]], [64, 48], Vs=[good[1], bad[1]], Ds=[good[2], bad[2]])
    assert res.info[0] == 0 and res.info[1] == -2
    assert res.sweeps[1] == 0 and torch.equal(bad[0], keep)
    g.init_strats(None, "cycwor", 32, "cycwor", 4)
    ref = _dev(G1, True)
    r = g.hypJacL2_dev(11, ref[0], 64, ref[1], ref[2])
    assert res.sweeps[0] == r[1] and np.array_equal(_bits(good[0]), _bits(ref[0]))


@pytest.mark.gpu
def test_batch_autotuner_picks_and_keeps_bits(built):
    """gjx_autotune_batched times (pairs per CTA) x (per-step / per-sweep
    launches) on random matrices of the batch's shapes; the batch run after it
    (with the tuned choice) still gives every matrix the single call's bits."""
    import torch
    import gpujachx_b200 as g
    shapes = [(128, 128, 128), (256, 256, 128), (192, 192, 0), (320, 320, 320), (128, 64, 64)]
    g.init_strats(None, "cycwor", 32, "cycwor", 4)
    pick = g.autotune_batched(11, [m for m, _, _ in shapes], [n for _, n, _ in shapes], [p for _, _, p in shapes])
    assert pick["pairs_per_cta"] in (1, 2, 3, 4) and pick["mode"] in (0, 1)
    mats = [synth.make("svd_synth", m, n, 7000 + k, smin=1e-6) if m == n else synth.make("graded", m, n, 7000 + k)
            for k, (m, n, _) in enumerate(shapes)]
    batch = [_dev(G, True) for G in mats]
    res = g.hypJacL2_batched(11, [b[0] for b in batch], [p for _, _, p in shapes], Vs=[b[1] for b in batch],
                             Ds=[b[2] for b in batch])
    g.lib().gjx_autotune_clear()
    for k, (G, (m, n, p)) in enumerate(zip(mats, shapes)):
        g.init_strats(None, "cycwor", 32, "cycwor", n // 16)
        dG, dV, dD = _dev(G, True)
        ret, sw, rs, rb = g.hypJacL2_dev(11, dG, p, dV, dD)
        torch.cuda.synchronize()
        assert (res.sweeps[k], res.rot_s[k], res.rot_b[k]) == (sw, rs, rb)
        assert np.array_equal(_bits(batch[k][0]), _bits(dG)) and np.array_equal(_bits(batch[k][1]), _bits(dV))


def _orthogonal(n, m):
    """Column j of an m x n matrix: one entry, 2^-(j // 8)."""
    import torch
    G = torch.zeros((n, m), dtype=torch.float64, device="cuda")
    s = torch.tensor([2.0 ** -(j // 8) for j in range(n)], dtype=torch.float64, device="cuda")
    j = torch.arange(n, device="cuda")
    G[j, j * (m // n)] = s
    return G, s


@pytest.mark.gpu
@pytest.mark.parametrize("m,launches", [(1 << 17, 2 * 4 + 1), ((1 << 17) + 64, 2 * 8 + 1)])
def test_untuned_launches_by_rows(m, launches, built):
    """One graph of 4 sweeps up to 2^17 rows, above it one of 8 steps (and initD)."""
    import torch
    import gpujachx_b200 as g
    g.init_strats(None, "cycwor", 32, "cycwor", 4)
    G, s = _orthogonal(64, m)
    g.profile(False)
    r = g.hypJacL2_batched(9, [G], [64], Ds=[torch.empty_like(s)])
    torch.cuda.synchronize()
    assert r.info == [0] and r.sweeps[0] == 1
    assert g.profile_read()["launches"] == launches


@pytest.mark.gpu
def test_very_tall_matrix(built):
    """8 block pairs of 4 M rows, 15 steps of about 0.1 s: in one launch per sweep
    the last step's items would wait for the 14 before them, longer than a wait
    may take."""
    import torch
    import gpujachx_b200 as g
    g.init_strats(None, "cycwor", 32, "cycwor", 16)
    G, s = _orthogonal(256, 1 << 22)
    D = torch.zeros(256, dtype=torch.float64, device="cuda")
    r = g.hypJacL2_batched(9, [G], [256], Ds=[D])
    torch.cuda.synchronize()
    assert r.info == [0] and r.sweeps[0] == 1 and r.rot_b[0] == 0
    assert torch.equal(D, s * s)
    assert torch.equal(G.amax(dim=1), torch.ones_like(s))
    del G
    torch.cuda.empty_cache()


@pytest.mark.gpu
@pytest.mark.parametrize("m,n,count", [(64, 64, 148), (128, 128, 65), (256, 256, 20), (256, 256, 37), (512, 512, 18),
                                       (4096, 128, 72)])
def test_untuned_is_not_slower_than_two_pairs_per_cta(m, n, count, built):
    """One to two block pairs per SM: a second wave of one-pair CTAs was up to 17 %
    slower than two pairs per CTA, one launch per step.  (Measured 8 to 33 %
    faster; the best of five runs of each.)"""
    import time

    import torch
    import gpujachx_b200 as g
    g.init_strats(None, "cycwor", 32, "cycwor", 4)
    torch.manual_seed(6)
    G = torch.randn((count, n, m), dtype=torch.float64, device="cuda")
    W, D = torch.empty_like(G), torch.zeros((count, n), dtype=torch.float64, device="cuda")
    best = {}
    for _ in range(5):
        for form in ((0, -1), (2, 0)):
            g.lib().gjx_set_pairs_per_cta(form[0])
            g.lib().gjx_set_batch_mode(form[1])
            W.copy_(G)
            torch.cuda.synchronize()
            t = time.perf_counter()
            g.hypJacL2_batched(9, list(W), n, Ds=list(D))
            best[form] = min(best.get(form, 1e9), time.perf_counter() - t)
    g.lib().gjx_set_pairs_per_cta(0)
    g.lib().gjx_set_batch_mode(-1)
    assert best[0, -1] < best[2, 0]
