"""The measured cases: the decompositions that a program has this framework do.

Every public form is here: the drop-in call on host arrays (``hypJacL2``), the
call on device-resident matrices (``hypJacL2_dev``), the batch
(``hypJacL2_batched``) and the split-precision form (``hypJacL2_split``); the
ordinary SVD (J = I) and the hyperbolic one; with and without V; one inner
sweep per block pair and the full inner iteration (ALG bit 8 clear); from one
outer step per sweep to 304 column blocks; square, tall and odd block counts.

The strategy tables are the program's own file (the ``sdy`` argument of
``init_strats``).  The one used here is written by this file: parallel
orderings of any even order, by doubling and step reversal, which for the
powers of two are the reference's ``cycwor`` tables.
"""

from __future__ import annotations

import atexit
import math
import os
import shutil
import subprocess
import tempfile

import numpy as np
import torch

import gpujachx_b200 as gjx

FAMILY = "cycwor"

# ---------------------------------------------------------------------------
# the cases
# ---------------------------------------------------------------------------
_LISTED = [
    # the smallest call: one decomposition of a few blocks on the device, the inner solver of another algorithm
    dict(name="dev_128x64", form="dev", m=128, n=64, nplus=64, alg=11, gen="gaussian"),
    # the drop-in call on host arrays, singular values over eight decades, no V
    dict(name="host_256_alg9", form="host", m=256, n=256, nplus=256, alg=9, gen="geometric", smin=1e-8),
    # an odd number of block pairs, the full inner iteration of every block pair (ALG 3)
    dict(name="dev_704x672_alg3", form="dev", m=704, n=672, nplus=672, alg=3, gen="gaussian"),
    # the hyperbolic SVD of graded columns: an indefinite eigenvalue problem in factored form
    dict(name="dev_hsvd_2048x1024", form="dev", m=2048, n=1024, nplus=512, alg=11, gen="graded"),
    # a tall matrix: a least-squares or principal-component problem, without sorting
    dict(name="dev_16384x256_alg10", form="dev", m=16384, n=256, nplus=256, alg=10, gen="gaussian"),
    # the headline size
    dict(name="dev_4096x2048", form="dev", m=4096, n=2048, nplus=2048, alg=11, gen="gaussian"),
    # square, more block pairs than half the SMs
    dict(name="dev_3072", form="dev", m=3072, n=3072, nplus=3072, alg=11, gen="gaussian"),
    # the largest plain call: more block pairs than SMs, values and left vectors only
    dict(name="dev_4864_alg9", form="dev", m=4864, n=4864, nplus=4864, alg=9, gen="gaussian"),
    # a few small matrices at once: the blocks of one larger problem
    dict(name="batch_24", form="batch", count=24, lo=64, hi=256, alg=11, pick=3),
    # a throughput batch of uneven sizes, half SVD and half HSVD
    dict(name="batch_320", form="batch", count=320, lo=64, hi=512, alg=11, pick=7),
    # split precision, hyperbolic, an odd number of 64-column pairs
    dict(name="split_hsvd_1600x1344", form="split", m=1600, n=1344, nplus=640, alg=11, gen="graded"),
    # split precision at a large square size
    dict(name="split_4096", form="split", m=4096, n=4096, nplus=4096, alg=11, gen="gaussian"),
]


def listed():
    return [dict(c) for c in _LISTED]


def _log_multiple(rng, lo, hi, step):
    """A multiple of step in [lo, hi], spread over its logarithm."""
    x = math.exp(rng.uniform(math.log(lo), math.log(hi)))
    return int(min(hi, max(lo, step * round(x / step))))


def draw(rng):
    form = rng.choice(("dev", "dev", "dev", "host", "batch", "split"))
    if form == "batch":
        lo = 64 * rng.randint(1, 4)
        hi = rng.choice((256, 384, 512))
        count = _log_multiple(rng, 3, 320, 1)
        return dict(form=form, count=count, lo=lo, hi=max(lo, hi), alg=rng.choice((9, 11, 11)), pick=rng.randrange(1000))
    if form == "host":
        n = _log_multiple(rng, 32, 1024, 32)
        m = 64 * rng.randint((n + 63) // 64, 2048 // 64)
        gen = rng.choice(("gaussian", "geometric", "graded"))
    elif form == "dev":
        n = _log_multiple(rng, 32, 3072, 32)
        m = _log_multiple(rng, 64 * ((n + 63) // 64), max(4096, 64 * ((n + 63) // 64)) if n > 512 else 16384, 64)
        gen = rng.choice(("gaussian", "gaussian", "geometric", "graded"))
    else:
        n = _log_multiple(rng, 256, 3072, 64)
        m = _log_multiple(rng, n, 4096, 64)
        gen = rng.choice(("gaussian", "graded"))
    nplus = n
    if gen == "graded":
        nplus = rng.choice((n // 2, n // 3, n))
    # (without sorting the split form's columns come in an order that rounding decides)
    c = dict(form=form, m=m, n=n, nplus=nplus, alg=rng.choice((9, 11) if form == "split" else (9, 10, 11, 11, 11)), gen=gen)
    if gen == "geometric":
        c["smin"] = rng.choice((1e-4, 1e-6, 1e-8))
    if form == "dev" and n <= 704 and gen == "gaussian":
        c["alg"] = rng.choice((1, 3, 11))
    return c


# ---------------------------------------------------------------------------
# strategy tables: parallel orderings of the blocks (and of the columns of a
# block pair), every pair once a sweep
# ---------------------------------------------------------------------------
_tables: dict = {}
_libraries: dict = {}
_loaded = None


def _doubled(n):
    """[n - 1][n / 2][2]: from a round robin of order 2 * odd (or 2), each step
    of order k gives two of order 2k, after one step inside the halves."""
    if n in _tables:
        return _tables[n]
    if n == 2 or n % 4:
        s, k = np.arange(n - 1)[:, None], np.arange(1, n // 2)[None, :]
        t = np.empty((n - 1, n // 2, 2), dtype=np.int64)
        t[:, :1, 0], t[:, :1, 1] = s, n - 1
        t[:, 1:, 0], t[:, 1:, 1] = (s + k) % (n - 1), (s - k) % (n - 1)
        t.sort(axis=2)
    else:
        h = _doubled(n // 2)
        t = np.empty((n - 1, n // 2, 2), dtype=np.int64)
        t[0, :, 0] = 2 * np.arange(n // 2)
        t[0, :, 1] = t[0, :, 0] + 1
        t[1::2, 0::2] = 2 * h
        t[1::2, 1::2] = 2 * h + 1
        t[2::2, 0::2] = 2 * h + (0, 1)
        t[2::2, 1::2] = 2 * h + (1, 0)
    _tables[n] = t
    return t


def _library(orders):
    """A shared library with the tables "<family>%05u" of these orders."""
    key = tuple(sorted(set(orders)))
    if key not in _libraries:
        tmp = tempfile.mkdtemp(prefix="strat_")
        atexit.register(shutil.rmtree, tmp, True)
        lines = ["\t.data"]
        for n in key:
            name = "%s%05d" % (FAMILY, n)
            t = _doubled(n)[::-1]
            path = os.path.join(tmp, name + ".bin")
            np.ascontiguousarray(t, dtype=np.uint8 if n <= 256 else np.uint16).tofile(path)
            lines += ["\t.globl " + name, "\t.type %s, @object" % name, "\t.balign 16", name + ":",
                      '\t.incbin "%s"' % path, "\t.size %s, .-%s" % (name, name)]
        lines.append('\t.section .note.GNU-stack,"",@progbits')
        src, out = os.path.join(tmp, "strat.s"), os.path.join(tmp, "strat.so")
        with open(src, "w") as f:
            f.write("\n".join(lines) + "\n")
        subprocess.check_call(["gcc", "-shared", "-nostdlib", "-o", out, src])
        _libraries[key] = out
    return _libraries[key]


def _load(tables):
    """init_strats, as a program does once for the matrices that it works on."""
    global _loaded
    if _loaded != tables:
        gjx.init_strats(tables[0], FAMILY, 32, FAMILY, tables[1])
        _loaded = tables


# ---------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------
def _generator(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    return g


def _randn(g, *shape):
    return torch.randn(shape, dtype=torch.float64, device="cuda", generator=g)


def _haar(g, n):
    q, r = torch.linalg.qr(_randn(g, n, n))
    return q * torch.sign(torch.diagonal(r))


def _columns(case, seed):
    """The matrix column by column: row j of the (n, m) tensor is column j."""
    g, m, n = _generator(seed), case["m"], case["n"]
    if case["gen"] == "gaussian":
        return _randn(g, n, m)
    if case["gen"] == "graded":  # B diag(d), d over six decades
        d = 10.0 ** (-6.0 * torch.rand((n, 1), dtype=torch.float64, device="cuda", generator=g))
        return _randn(g, n, m) * d
    sv = torch.logspace(0.0, math.log10(case["smin"]), n, dtype=torch.float64, device="cuda")
    q1 = torch.linalg.qr(_randn(g, m, n))[0]
    return ((q1 * sv) @ _haar(g, n).T).T.contiguous()


def _sizes(case):
    """(n, nplus) of each matrix of a batch: n uniform over multiples of 64, half SVD, half HSVD."""
    r = np.random.default_rng(case["pick"])
    n = 64 * r.integers(case["lo"] // 64, case["hi"] // 64 + 1, size=case["count"])
    return [(int(k), int(k) if b % 2 == 0 else int(k) // 2) for b, k in enumerate(n)]


def _matrices(flat, sizes):
    """The n x n matrices of a batch that lie back to back in one buffer."""
    out, at = [], 0
    for n, _ in sizes:
        out.append(flat[at:at + n * n].view(n, n))
        at += n * n
    return out


def _batch(case, seed):
    """Q1 diag(s) Q2^T of each size, s geometric from 1 to 1e-6: dense
    orthogonal factors of each n, moved by reflections of each matrix's own."""
    g, fixed, sizes = _generator(seed), {}, _sizes(case)
    flat = torch.empty(sum(n * n for n, _ in sizes), dtype=torch.float64, device="cuda")
    for (n, _), to in zip(sizes, _matrices(flat, sizes)):
        if n not in fixed:
            sv = torch.logspace(0.0, -6.0, n, dtype=torch.float64, device="cuda")
            fixed[n] = (_haar(g, n) * sv) @ _haar(g, n).T
        a = fixed[n]
        u, v = _randn(g, n, 1), _randn(g, n, 1)
        a = a - (2.0 / (u * u).sum()) * u @ (u.T @ a)
        a = a - (2.0 / (v * v).sum()) * (a @ v) @ v.T
        to.copy_(a.T)
    return flat


def _orders(case):
    if case["form"] == "batch":
        ns = {n for n, _ in _sizes(case)}
        return [32] + [n // 16 for n in ns], max(ns) // 16
    n1 = case["n"] // 16
    return [32, 64, n1] + ([n1 // 2] if case["form"] == "split" else []), n1


def prepare(case, seed):
    orders, n1 = _orders(case)
    s = dict(case=case, tables=(_library(orders), n1))
    _load(s["tables"])
    full = bool(case["alg"] & 2)
    new = dict(dtype=torch.float64, device="cuda")
    if case["form"] == "batch":
        sizes = _sizes(case)
        s["G"] = _batch(case, seed)
        s["work"] = torch.empty_like(s["G"])
        s["V"] = torch.empty_like(s["G"]) if full else None
        s["D"] = torch.empty(sum(n for n, _ in sizes), **new)
        s["nplus"] = [p for _, p in sizes]
        s["Gs"] = _matrices(s["work"], sizes)
        s["Vs"] = _matrices(s["V"], sizes) if full else None
        s["Ds"] = list(s["D"].split([n for n, _ in sizes]))
    elif case["form"] == "host":
        s["G"] = _columns(case, seed).cpu().numpy().T  # column major, as the C interface has it
    else:
        n = case["n"]
        s["G"] = _columns(case, seed)
        s["work"] = torch.empty_like(s["G"])
        s["V"] = torch.empty((n, n), **new) if full else None
        s["D"] = torch.empty(n, **new)
    return s


def run(s):
    """One decomposition (or batch) from the untouched input: the calls work in place, on a fresh copy."""
    c = s["case"]
    _load(s["tables"])
    if c["form"] == "host":
        r = gjx.hypJacL2(c["alg"], s["G"], c["nplus"])
        return dict(U=r.U, V=r.V, D=r.D, counts=np.array([r.sweeps, r.rot_s, r.rot_b]))
    s["work"].copy_(s["G"])
    if c["form"] == "batch":
        r = gjx.hypJacL2_batched(c["alg"], s["Gs"], s["nplus"], Vs=s["Vs"], Ds=s["Ds"])
        return dict(U=s["work"], V=s["V"], D=s["D"], counts=np.array([r.sweeps, r.rot_s, r.rot_b]))
    call = gjx.hypJacL2_split if c["form"] == "split" else gjx.hypJacL2_dev
    _, sweeps, rot_s, rot_b = call(c["alg"], s["work"], c["nplus"], V=s["V"], D=s["D"])
    if c["form"] == "dev":
        return dict(U=s["work"], V=s["V"], D=s["D"], counts=np.array([sweeps, rot_s, rot_b]))
    # the plain forms promise the reference's bits, the split form does not: a
    # program fixes the signs of its singular vectors, by each one's largest entry
    sign = torch.sign(s["work"].gather(1, s["work"].abs().argmax(1, keepdim=True)))
    s["work"].mul_(sign)
    if s["V"] is not None:
        s["V"].mul_(sign)
    return dict(U=s["work"], V=s["V"], D=s["D"])


# ---------------------------------------------------------------------------
# what a pass cannot do without, and how far a right answer may be off
# ---------------------------------------------------------------------------
def _cost(m, n, full, sweeps):
    """G in, U, D and V out; a sweep of block pairs of 32 columns forms their
    Gram matrices (2 M 32^2 each), and updates G (2 M 32^2) and V (2 N 32^2)."""
    pairs = (n // 16) * (n // 16 - 1) // 2
    return (8 * (2 * m * n + n + (n * n if full else 0)),
            sweeps * pairs * 1024 * (4 * m + (2 * n if full else 0)))


def work(case):
    full = bool(case["alg"] & 2)
    if case["form"] == "batch":
        each = [_cost(n, n, full, 15) for n, _ in _sizes(case)]
    else:
        sweeps = {"gaussian": 9, "graded": 6, "geometric": 15}[case["gen"]]
        each = [_cost(case["m"], case["n"], full, sweeps)]
    return {"bytes": sum(b for b, _ in each), "flops": sum(f for _, f in each)}


def tolerance(case):
    # The plain forms promise the reference's bits; the split form FP64 accuracy:
    # inputs moved by 2^-52 of each entry move its vectors by up to 1.9e-11 (the
    # largest entry by 1.5e-9; close singular values), measured over the ranges.
    if case["form"] == "split":
        return {"rel": 1e-10, "max": 1e-8}
    return "exact"


def _values(a, nplus):
    """D in 64 bits, each sign's values from the largest down."""
    n = a.shape[0]
    if nplus in (0, n):
        d = torch.linalg.svdvals(a) ** 2
        return d if nplus else -d
    j = torch.ones(n, dtype=torch.float64, device=a.device)
    j[nplus:] = -1.0
    r = torch.linalg.qr(a.T)[1]
    d = torch.linalg.eigvalsh((r * j) @ r.T)
    return torch.cat([d[d > 0].flip(0), d[d <= 0].flip(0)])


def exact(case, seed):
    """D in the order that sorting leaves it in; the vectors are determined up
    to their signs only, and the counts belong to the algorithm."""
    if not case["alg"] & 1:
        return None
    none = dict(U=None, V=None)
    if case["form"] == "batch":
        sizes = _sizes(case)
        gs = _matrices(_batch(case, seed), sizes)
        return dict(none, D=torch.cat([_values(a, p) for a, (_, p) in zip(gs, sizes)]), counts=None)
    d = _values(_columns(case, seed), case["nplus"])
    if case["form"] == "split":
        return dict(none, D=d)
    return dict(none, D=d.cpu().numpy() if case["form"] == "host" else d, counts=None)
