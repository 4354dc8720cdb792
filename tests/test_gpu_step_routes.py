"""The routes of a single decomposition's outer steps against the fused step
kernel with one CTA per block pair, which the other tests hold against the
oracle: clusters of 2, 4 and 8 CTAs per pair.  The same bits."""

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
