"""Strategy tables that a construction gives.

Outer tables beyond the reference's largest order (896 blocks, N = 14336
columns): the rowcyc and colcyc tables of orders 960 and 1024 (N = 15360 and
16384), built by the reference's own doubling construction
(strat/n2n/n2n.sh.cpp:41-129) from its tables of orders 480 and 512.

The construction, for an order-n table T of n-1 parallel steps of n/2
disjoint pairs, gives the order-2n table:
  * step 0: the pairs (2k, 2k+1), k < n;
  * each step s of T becomes steps 2s+1 and 2s+2; its a-th pair (i, j) gives
    pairs 2a and 2a+1 of them: (2i, 2j), (2i+1, 2j+1) in the first;
    (2i, 2j+1), (2i+1, 2j) (rowcyc) or (2i+1, 2j), (2i, 2j+1) (colcyc) in
    the second.
Every pair of blocks meets once per sweep and each step is a perfect
matching, as in T.  The reference's tables of every order 2n <= 896 whose
half it also ships are this doubling of it (all 112 of them;
tests/test_strat_doubling.py checks it against the tables in strat.so).

Where the reference tree is not at hand, the families are built whole
(family_sources).  The cyclic ones for the orders 2^k, 3 2^k, 5 2^k, 7 2^k and
9 2^k: a base of order 2, 6, 10, 14 or 18, doubled; the rowcyc (colcyc) base is the first
complete set of perfect matchings that a backtracking search finds when it
takes the pairs in row-cyclic (column-cyclic) order, and cycwor (cycloc) is
rowcyc (colcyc) with its steps reversed.  BrentL is the ordering of R. P. Brent
and F. T. Luk (1985), mmstep the modulus ordering with the two indices that
meet themselves paired (n steps).  The recorded outputs of the reference pin
these tables: rowcyc, colcyc and cycloc of orders 12 and 32, cycwor of orders 2
to 512 among them 12, 20, 24 and 28, BrentL and mmstep of orders 16 and 32 give
its bits (tests/test_oracle_golden.py).

Used by build.build_strat; the generated tables get the reference's symbol
names (rowcyc00960, ...) and element type (unsigned short above 256).
"""

from __future__ import annotations

import re

import numpy as np

FAMILIES = ("rowcyc", "colcyc")
ORDERS = (960, 1024)


def parse_header(text: str, n: int) -> np.ndarray:
    """The table of a reference header (``... name[S][n/2][2] = {{{i, j}, ...}, ...};``)."""
    body = text[text.index("=") + 1:]
    v = np.array([int(x) for x in re.findall(r"\d+", body)], dtype=np.int64)
    if v.size % n:
        raise ValueError(f"table of order {n}: {v.size} entries")
    return v.reshape(v.size // n, n // 2, 2)


def double_table(t: np.ndarray, family: str) -> np.ndarray:
    """The order-2n table of the doubling construction from the order-n table t."""
    if family not in FAMILIES:
        raise ValueError(f"no doubling rule for {family}")
    steps, half, _ = t.shape
    n = 2 * half
    out = np.zeros((2 * steps + 1, n, 2), dtype=np.int64)
    out[0, :, 0] = 2 * np.arange(n)
    out[0, :, 1] = 2 * np.arange(n) + 1
    i, j = t[:, :, 0], t[:, :, 1]
    first, second = out[1::2], out[2::2]
    first[:, 0::2, 0], first[:, 0::2, 1] = 2 * i, 2 * j
    first[:, 1::2, 0], first[:, 1::2, 1] = 2 * i + 1, 2 * j + 1
    if family == "rowcyc":
        second[:, 0::2, 0], second[:, 0::2, 1] = 2 * i, 2 * j + 1
        second[:, 1::2, 0], second[:, 1::2, 1] = 2 * i + 1, 2 * j
    else:
        second[:, 0::2, 0], second[:, 0::2, 1] = 2 * i + 1, 2 * j
        second[:, 1::2, 0], second[:, 1::2, 1] = 2 * i, 2 * j + 1
    return out


def base_table(n: int, family: str) -> np.ndarray:
    """The order-n table (n = 2 odd) that a backtracking search finds first,
    its steps filled with the pairs in row-cyclic (rowcyc: 01 02 .. 12 ..) or
    column-cyclic (colcyc: 01 02 12 03 ..) order."""
    if family == "rowcyc":
        order = [(i, j) for i in range(n) for j in range(i + 1, n)]
    else:
        order = [(i, j) for j in range(n) for i in range(j)]
    used: set = set()
    steps: list = []

    def matchings(start, busy, m):
        if len(m) == n // 2:
            yield list(m)
            return
        for k in range(start, len(order)):
            i, j = order[k]
            if order[k] in used or i in busy or j in busy:
                continue
            yield from matchings(k + 1, busy | {i, j}, m + [order[k]])

    def search():
        if len(steps) == n - 1:
            return True
        for m in matchings(0, frozenset(), []):
            steps.append(m)
            used.update(m)
            if search():
                return True
            steps.pop()
            used.difference_update(m)
        return False

    if not search():
        raise ValueError(f"no table of order {n}")
    return np.array(steps, dtype=np.int64)


def cyclic_table(family: str, n: int) -> np.ndarray:
    """The order-n table of a cyclic family (rowcyc, colcyc, cycwor, cycloc)."""
    fwd = {"cycwor": "rowcyc", "cycloc": "colcyc"}.get(family, family)
    b = n
    while b % 4 == 0:
        b //= 2
    t = base_table(b, fwd)
    while 2 * t.shape[1] < n:
        t = double_table(t, fwd)
    return t if fwd == family else t[::-1]


def brent_luk_table(n: int) -> np.ndarray:
    """n - 1 steps: two rows of n/2 indices, paired by column; from step to
    step the first index stays and the others move one place around."""
    top, bottom = list(range(0, n, 2)), list(range(1, n, 2))
    steps = []
    for _ in range(n - 1):
        steps.append([(min(p), max(p)) for p in zip(top, bottom)])
        top, bottom = [top[0], bottom[0]] + top[1:-1], bottom[1:] + top[-1:]
    return np.array(steps, dtype=np.int64)


def modulus_table(n: int) -> np.ndarray:
    """n steps, s = n - 1, 0, 1, ..., n - 2: the pairs i + j = s (mod n), and for
    even s the two i with 2 i = s (mod n) paired with each other."""
    steps = []
    for t in range(n):
        s = (n - 1 + t) % n
        pairs = [(i, (s - i) % n) for i in range(n) if i < (s - i) % n]
        if s % 2 == 0:
            pairs.append((s // 2, s // 2 + n // 2))
        steps.append(pairs)
    return np.array(steps, dtype=np.int64)


# what family_tables gives, for messages
CONSTRUCTED = ("mmstep and BrentL of orders 16, 32, ..., 896; rowcyc, colcyc, cycwor and cycloc of orders 2^k b, "
               "b = 2, 6, 10, 14, 18, up to 896 (rowcyc and colcyc also 1024)")


def family_tables():
    """(family, n, table) of every table that is built without a reference tree."""
    orders = sorted(b << k for b in (2, 6, 10, 14, 18) for k in range(10) if b << k <= 1024)
    for fam in ("rowcyc", "colcyc", "cycwor", "cycloc"):
        for n in orders:
            if n <= 896 or fam in FAMILIES:
                yield fam, n, cyclic_table(fam, n)
    for n in range(16, 897, 16):
        yield "BrentL", n, brent_luk_table(n)
        yield "mmstep", n, modulus_table(n)


def family_sources() -> dict[str, str]:
    """{file name: assembler source} of every table of family_tables."""
    out: dict[str, str] = {}
    for fam, n, t in family_tables():
        name, t = "%s%05u" % (fam, n), t.ravel()
        word = ".byte" if n <= 256 else ".short"
        data = "\n".join("\t%s %s" % (word, ",".join(map(str, t[i:i + 64]))) for i in range(0, t.size, 64))
        out[fam + ".s"] = out.get(fam + ".s", "\t.data\n") + (
            "\t.globl %s\n\t.type %s, @object\n\t.balign 16\n%s:\n%s\n\t.size %s, .-%s\n"
            % (name, name, name, data, name, name))
    return {k: v + '\t.section .note.GNU-stack,"",@progbits\n' for k, v in out.items()}


def c_source(family: str, n: int, t: np.ndarray) -> str:
    """A C definition of the table with the reference's symbol name and type."""
    typ = "unsigned char" if n <= 256 else "unsigned short"
    rows = []
    for step in t:
        rows.append("{" + ",".join("{%d,%d}" % (int(a), int(b)) for a, b in step) + "}")
    return ('__attribute__((visibility("default"))) %s %s%05u[%u][%u][2] = {\n%s\n};\n'
            % (typ, family, n, t.shape[0], t.shape[1], ",\n".join(rows)))


def extension_sources(strat_dir: str) -> dict[str, str]:
    """{file name: C source} of the tables to add to strat.so: each family's
    orders in ORDERS that strat_dir lacks and whose half it has."""
    import os
    out = {}
    for fam in FAMILIES:
        for n in ORDERS:
            full = os.path.join(strat_dir, fam, "%05u.h" % n)
            half = os.path.join(strat_dir, fam, "%05u.h" % (n // 2))
            if os.path.exists(full) or not os.path.exists(half):
                continue
            with open(half) as f:
                t = parse_header(f.read(), n // 2)
            out["%s%05u.c" % (fam, n)] = c_source(fam, n, double_table(t, fam))
    return out
