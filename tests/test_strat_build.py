"""build_strat without the reference tree: it says what it leaves out, marks the
library, and builds it again from the reference's headers once a tree is given;
the tables that it makes are parallel orderings."""

import numpy as np
import pytest

from gpujachx_b200 import build as B
from gpujachx_b200 import strat_gen


@pytest.fixture
def tree(tmp_path, monkeypatch):
    """A reference tree of one table per family, and an empty library folder."""
    for fam in B.STRAT_FAMILIES:
        d = tmp_path / "ref" / "strat" / fam
        d.mkdir(parents=True)
        (d / "00002.h").write_text("unsigned char %s00002[1][1][2]\n#ifdef USE_STRAT_ARRAY_DECLARATOR\n= {{{0,1}}}\n"
                                   "#endif\n;\n" % fam)
    monkeypatch.setattr(B, "LIBDIR", str(tmp_path / "lib"))
    monkeypatch.setattr(B, "STRAT", str(tmp_path / "lib" / "strat.so"))
    monkeypatch.setattr(strat_gen, "family_tables", lambda: iter([("rowcyc", 6, strat_gen.cyclic_table("rowcyc", 6))]))
    monkeypatch.delenv("GJX_REF_ROOT", raising=False)
    return str(tmp_path / "ref")


def test_constructed_library_is_reported_and_built_again(tree, capfd):
    B.build_strat(verbose=False)
    err = capfd.readouterr().err
    assert "GJX_REF_ROOT" in err and "left out" in err and "1024" in err
    assert B.strat_constructed() and "rowcyc00006" in B.strat_symbols()
    B.build_strat(ref_root=tree, verbose=False)
    assert not B.strat_constructed()
    assert "mmstep00002" in B.strat_symbols() and "rowcyc00006" not in B.strat_symbols()


def test_reference_tables_stay(tree, capfd):
    B.build_strat(ref_root=tree, verbose=False)
    for force in (False, True):
        B.build_strat(force=force, verbose=False)
        assert not B.strat_constructed()
    assert not capfd.readouterr().err


def test_constructed_tables_are_parallel_orderings(built):
    import gpujachx_b200 as g
    seen = set()
    for fam, n, t in strat_gen.family_tables():
        seen.add((fam, n))
        r = g.validate_pairs(np.ascontiguousarray(t, dtype=np.uint16))
        assert r["code"] == 0 and r["missing"] == 0, (fam, n)
        assert r["repeats"] == (n // 2 if fam == "mmstep" else 0), (fam, n)
    assert len(seen) == 262
    assert {n for f, n in seen if f == "rowcyc" and n > 896} == {1024} == {n for f, n in seen if f == "colcyc" and n > 896}
