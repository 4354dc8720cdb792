"""Calls with no device memory left: what a faster route would take beside the
caller's own buffers is not a condition of the call, which takes the route
without it and gives the same bits."""

import contextlib
import ctypes

import numpy as np
import pytest

from gpujachx_b200 import synth

pytestmark = pytest.mark.gpu


class Full:
    """The device's memory taken down to pieces of 64 KB, but for `hole` bytes."""

    def __init__(self, hole=0):
        import torch  # loads the CUDA runtime
        torch.cuda.synchronize()
        torch.cuda.empty_cache()
        self.rt, self.hole, self.held = ctypes.CDLL("libcudart.so.12"), hole, []

    def take(self, size):
        p = ctypes.c_void_p()
        if self.rt.cudaMalloc(ctypes.byref(p), ctypes.c_size_t(size)):
            self.rt.cudaGetLastError()
            return False
        self.held.append(p)
        return True

    def __enter__(self):
        if self.hole:
            assert self.take(self.hole)
        for k in range(37, 15, -1):
            while self.take(1 << k):
                pass
        if self.hole:
            self.rt.cudaFree(self.held.pop(0))
        return self

    def __exit__(self, *a):
        for p in self.held:
            self.rt.cudaFree(p)


def _dev(G, full):
    import torch
    n = G.shape[1]
    dG = torch.tensor(np.ascontiguousarray(G.T), device="cuda")
    dV = torch.zeros((n, n), dtype=torch.float64, device="cuda") if full else None
    return dG, dV, torch.zeros(n, dtype=torch.float64, device="cuda")


def _bits(t):
    return None if t is None else t.cpu().numpy().view(np.uint64)


@pytest.mark.parametrize("m,n,apart", [(2048, 1024, False), (6016, 640, True)])
def test_update_launch(m, n, apart, built):
    """The transforms of the separate update launch: not allocated by a call that
    does not use them, and done without by one that would."""
    import torch

    import gpujachx_b200 as g
    G = synth.make("gaussian", m, n, 9)
    g.init_strats(None, "cycwor", 32, "cycwor", n // 16)
    runs = []

    def run(bufs):
        g.profile(False)
        r = g.hypJacL2_dev(11, bufs[0], n, bufs[1], bufs[2])
        torch.cuda.synchronize()
        runs.append((r, g.profile_read()["launches"] > 2 * (n // 16 - 1) * r[1], bufs))

    run(_dev(G, True))
    g.lib().gjx_set_pairs_per_cta(1)  # the step kernels update
    run(_dev(G, True))
    g.lib().gjx_set_pairs_per_cta(0)
    bufs = _dev(G, True)
    g.lib().gjx_release_cache()
    with Full():
        run(bufs)
    run(_dev(G, True))
    assert [a for _, a, _ in runs] == [apart, False, False, apart]
    for r, _, b in runs[1:]:
        assert r == runs[0][0]
        assert all(np.array_equal(_bits(x), _bits(y)) for x, y in zip(b, runs[0][2]))


def test_split_form_v_beside(built):
    """The two steps' V_loc of V's update on its own stream.  (A timed call
    allocates the rest of the split form's memory for this order.)"""
    import torch

    import gpujachx_b200 as g
    n = 4608  # 72 block pairs: more than any other call of the suite with V beside
    G = np.asfortranarray(np.diag(np.logspace(0.0, -3.0, n)))
    G[:2, :2] = [[1.0, 0.5], [0.25, 0.75]]
    g.init_strats(None, "cycwor", 32, "cycwor", 64)
    runs = []

    def run(bufs):
        r = g.hypJacL2_split(11, bufs[0], n, bufs[1], bufs[2])
        torch.cuda.synchronize()
        runs.append((r, g.profile_read()["launches"], bufs))

    steps = n // 32 - 1
    g.profile(True)
    run(_dev(G, True))
    g.profile(False)
    bufs = _dev(G, True)
    with Full():
        run(bufs)
    g.profile(False)
    run(_dev(G, True))
    assert [k for _, k, _ in runs] == [4 + c * steps * runs[0][0][1] for c in (2, 2, 4)]
    for r, _, b in runs[1:]:
        assert r == runs[0][0]
        assert all(np.array_equal(_bits(x), _bits(y)) for x, y in zip(b, runs[0][2]))


def test_batched_form(built):
    """The items of a launch per sweep: 6 bytes per block pair and step."""
    import torch

    import gpujachx_b200 as g
    n, k = 4096, 24  # 128 pairs, 255 steps: 4.7 MB
    g.init_strats(None, "cycwor", 32, "cycwor", n // 16)
    s = torch.tensor([2.0 ** -(j // 64) for j in range(n)], dtype=torch.float64, device="cuda")
    Gs = [torch.empty((n, n), dtype=torch.float64, device="cuda") for _ in range(k)]
    Ds = [torch.zeros(n, dtype=torch.float64, device="cuda") for _ in range(k)]
    launches = []
    for full in (False, True):
        for G, D in zip(Gs, Ds):
            G.zero_().diagonal().copy_(s)
            D.zero_()
        g.profile(False)
        with Full(hole=4 << 20) if full else contextlib.nullcontext():
            r = g.hypJacL2_batched(9, Gs, n, Ds=Ds)
            torch.cuda.synchronize()
        launches.append(g.profile_read()["launches"])
        assert r.info == [0] * k and r.sweeps == [1] * k
        assert all(torch.equal(d, s * s) for d in Ds)
    assert launches[0] == 2 * 4 + 1 and launches[1] == 2 * 256 + 1  # 4 sweeps a graph; 255 steps, 8 a graph
