"""Targets that are not in lowest terms: the same matrix with every entry times a power of sqrt2 and the exponent raised
to match. The spec format takes them, the residuals of the search are always in lowest terms, and the answers are those
of the C restatement on the same text (plain search, batch) or of the target in lowest terms (state targets, table, meet
in the middle). Product and entangled targets and the identity; 1, 2, 5 and 8 factors of sqrt2."""
import pytest

import cheese_b200 as cz
from conftest import run_oracle, spec_text

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def engine():
    e = cz.Engine(0)
    yield e
    e.close()


def times_sqrt2(row):
    v = [int(x) for x in row.split()]
    out = []
    for i in range(0, len(v), 4):
        a, b, c, d = v[i:i + 4]
        out += [b - d, a + c, b + d, c - a]           # times w - w^3
    return " ".join(map(str, out))


def scaled(text, j):
    """the spec with its searched matrix (the start rows of a state target, else the target) over sqrt2^(k + j)"""
    key = "start" if "\nstart " in text else "target"
    head, rest = text.split(f"\n{key} ", 1)
    k, rows = rest.split("\n", 1)
    rows = rows.split("\n")
    n = int(text.split("\nn ", 1)[1].split()[0])
    for r in range(1 << n):
        for _ in range(j):
            rows[r] = times_sqrt2(rows[r])
    return f"{head}\n{key} {int(k) + j}\n" + "\n".join(rows)


def identity_text():
    text = spec_text("rand-22")
    head, rest = text.split("\ntarget ", 1)
    rows = rest.split("\n")
    for r in range(8):
        rows[1 + r] = " ".join("1 0 0 0" if c == r else "0 0 0 0" for c in range(8))
    rows[0] = "0"
    return f"{head}\ntarget " + "\n".join(rows)


CASES = [("rand-22", None), ("rand-00", 6), ("toffoli", 8), ("relative-phase-toffoli", 8), ("cs", None), ("qft_2", 8),
         ("rand-05", 6), ("identity", 3)]


@pytest.mark.parametrize("j", [1, 2, 5, 8])
@pytest.mark.parametrize("name,depth", CASES)
def test_matches_restatement(engine, oracle_bin, tmp_path, name, depth, j):
    text = scaled(identity_text() if name == "identity" else spec_text(name), j)
    p = tmp_path / "t.spec"
    p.write_text(text)
    rc, lines = run_oracle(oracle_bin, p, ["--depth", str(depth)] if depth else [])
    for store64 in (False, True):
        out = engine.search(text, depth=depth or -1, store64=store64)
        assert (out.rc, out.lines()) == (rc, lines)


@pytest.mark.parametrize("name,depth", [("states-rand-1", 6), ("states-rand-4", 5), ("rus2-states", 7)])
@pytest.mark.parametrize("j", [1, 2, 5])
def test_state_targets_as_in_lowest_terms(engine, name, depth, j):
    want = engine.search(spec_text(name), depth=depth)
    out = engine.search(scaled(spec_text(name), j), depth=depth)
    assert (out.rc, out.lines(), out.circuit) == (want.rc, want.lines(), want.circuit)


@pytest.mark.parametrize("j", [2, 3])
def test_batch(engine, j):
    texts = [scaled(spec_text(s), j) for s in ("rand-22", "toffoli", "peres", "rand-05")]
    b = cz.Batch(engine, 3)
    ids = [b.submit(t, depth=7) for t in texts]
    b.run()
    for t, i in zip(texts, ids):
        plain, got = engine.search(t, depth=7), b.result(i)
        assert (got.rc, got.lines(), got.circuit) == (plain.rc, plain.lines(), plain.circuit)
    b.close()


@pytest.mark.parametrize("name,depth", [("rand-22", -1), ("toffoli", 9), ("peres", 9), ("rand-05", -1), ("identity", 3)])
@pytest.mark.parametrize("j", [1, 2])
def test_table_and_mitm_as_in_lowest_terms(engine, name, depth, j):
    text = identity_text() if name == "identity" else spec_text(name)
    want = engine.search(text, depth=depth)
    for kw in ({"table_k": 2}, {"table_k": 5}, {"mitm": True}):
        if "mitm" in kw and name == "identity":
            continue                                   # its two sides start equal; the table answers at once
        engine.search(text, depth=depth, cache_dir=None, **kw)     # (the first call prints the table's levels too)
        low = engine.search(text, depth=depth, cache_dir=None, **kw)
        out = engine.search(scaled(text, j), depth=depth, cache_dir=None, **kw)
        assert out.rc == low.rc == want.rc
        if name != "identity":
            assert (out.lines(), out.circuit) == (low.lines(), low.circuit)
