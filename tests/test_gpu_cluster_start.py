"""The CTAs of a cluster write their Gram shares into one another's shared
memory, which is defined only once every CTA of the cluster has started.  The
shortest way from launch to that store (one 64-row tile), with other work on the
GPU while the clusters are placed: the bits of one CTA per block pair."""

import numpy as np
import pytest

from gpujachx_b200 import synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [32, 64])
@pytest.mark.parametrize("mode", [0, 1])
@pytest.mark.parametrize("split", [2, 4, 8])
def test_one_tile_beside_other_work(n, mode, split, built):
    import torch

    import gpujachx_b200 as g
    G = synth.make("graded", 64, n, 12)
    g.init_strats(None, "cycwor", 32, "cycwor", n // 16)
    busy, a = torch.cuda.Stream(), torch.randn(2048, 2048, device="cuda")

    def run(s):
        g.lib().gjx_set_split(s)
        g.lib().gjx_set_sweep_mode(mode)
        try:
            with torch.cuda.stream(busy):
                for _ in range(20):
                    a @ a
            return g.hypJacL2(11, G, n // 2)
        finally:
            g.lib().gjx_set_split(0)
            g.lib().gjx_set_sweep_mode(-1)

    ref = run(1)
    for _ in range(5):
        r = run(split)
        assert (r.sweeps, r.rot_s, r.rot_b) == (ref.sweeps, ref.rot_s, ref.rot_b)
        for x, y in ((r.U, ref.U), (r.V, ref.V), (r.D, ref.D)):
            assert np.array_equal(x.view(np.uint64), y.view(np.uint64))
    torch.cuda.synchronize()
