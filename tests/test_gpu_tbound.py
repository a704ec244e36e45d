"""The T bound's packed form (unitary residuals with qubits + exponent up to 7: four components to a register, the
entries that are already dead left early) and the general form beside it, through whole searches against the C
restatement: targets whose residuals lie on both sides of the limit, and a target that is not unitary (general form
throughout). Counts are whole numbers and must be equal."""
import random

import pytest

import cheese_b200 as cz
from cheese_b200 import workloads
from conftest import run_oracle, spec_text

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def engine():
    e = cz.Engine(0)
    yield e
    e.close()


def target(seed):
    """a circuit rich in H and T gates: residual exponents 4 (2 qubits) and 5 (3 qubits) at the root"""
    rng = random.Random(seed)
    n = 3 if seed % 3 else 2
    circ = []
    for _ in range(rng.randint(10, 16)):
        g = rng.choice(["h", "h", "h", "h", "cx", "cx", "t", "t"])
        circ.append((g, tuple(rng.sample(range(n), 2)) if g == "cx" else (rng.randrange(n),)))
    return n, circ


@pytest.mark.parametrize("seed,exponent,budget", [(85, 5, 10), (509, 5, 12), (581, 5, 12), (2740, 5, 12),
                                                  (303, 4, 10), (2046, 4, 10)])
def test_exponents_around_the_packed_limit(engine, oracle_bin, tmp_path, seed, exponent, budget):
    n, circ = target(seed)
    assert workloads.unitary(n, circ)[0] == exponent
    text = workloads.make_spec(n, circ, budget)
    p = tmp_path / "t.spec"
    p.write_text(text)
    rc, lines = run_oracle(oracle_bin, p, [])
    out = engine.search(text)
    assert (out.rc, out.lines()) == (rc, lines)
    assert out.raw.t_evals > 0


def test_target_that_is_not_unitary(engine, oracle_bin, tmp_path):
    text = spec_text("toffoli")
    head, rest = text.split("\ntarget ", 1)
    rows = rest.split("\n")
    for r in range(1, 9):                       # the rows of the target, every entry times 3
        rows[r] = " ".join(str(3 * int(v)) for v in rows[r].split())
    text = head + "\ntarget " + "\n".join(rows)
    p = tmp_path / "t.spec"
    p.write_text(text)
    rc, lines = run_oracle(oracle_bin, p, ["--depth", "9"])
    out = engine.search(text, depth=9)
    assert (out.rc, out.lines()) == (rc, lines)
    assert out.raw.t_evals > 0


@pytest.mark.parametrize("sym", [True, False])
@pytest.mark.parametrize("seed,n,length", [(1, 3, 6), (2, 3, 7), (3, 3, 5), (4, 2, 7), (5, 2, 6), (6, 3, 6), (7, 1, 5)])
def test_children_decided_from_their_parent(engine, oracle_bin, tmp_path, seed, n, length, sym):
    """every kind of candidate the level kernel tells apart: unit monomials with phases (y), two-qubit diagonals (cz),
    non-affine permutations (ccx), Hadamards and cx, on targets that are products and entangled ones"""
    rng = random.Random(seed)
    gates = ["y", "t", "h", "s"] + (["cz", "cx"] if n > 1 else []) + (["ccx"] if n > 2 else [])
    circ = [(g, tuple(rng.sample(range(n), {"cz": 2, "cx": 2, "ccx": 3}.get(g, 1)))) for g in
            gates[:length] + [rng.choice(gates) for _ in range(max(0, length - len(gates)))]]
    rng.shuffle(circ)
    text = workloads.make_spec(n, circ, length)
    p = tmp_path / "t.spec"
    p.write_text(text)
    rc, lines = run_oracle(oracle_bin, p, ["--depth", "5"] + ([] if sym else ["--no-sym"]))
    out = engine.search(text, depth=5, sym=sym)
    assert (out.rc, out.lines()) == (rc, lines), circ


def times3(text):
    """the spec with its target's entries times 3: not unitary, the general form takes its whole queue"""
    head, rest = text.split("\ntarget ", 1)
    rows = rest.split("\n")
    for r in range(1, 9):
        rows[r] = " ".join(str(3 * int(v)) for v in rows[r].split())
    return head + "\ntarget " + "\n".join(rows)


def test_both_forms_in_one_batch(engine):
    """jobs for the packed form alone, for both (residuals past the limit, non-monomial candidates) and for the general
    one alone, advanced together: the same as each on its own"""
    low = [workloads.make_spec(3, [("h", (0,)), ("t", (0,)), ("cx", (0, 1)), ("t", (1,)), ("h", (2,)), ("cx", (1, 2))], 6)]
    high = [workloads.make_spec(3, target(s)[1], 10) for s in (85, 509, 581, 2740)]
    texts = low + [spec_text("toffoli"), spec_text("ccx-lite")] + high + [times3(spec_text("toffoli")), times3(high[0])]
    specs = [cz.Spec(t) for t in texts]
    assert {s.n for s in specs} == {3}
    for group in (specs, specs[:1], specs[2:3], specs[-1:], specs[1:4]):
        b = cz.Batch(engine, 3)
        ids = [b.submit(s, depth=8) for s in group]
        b.run()
        for s, i in zip(group, ids):
            plain, got = engine.search(s, depth=8), b.result(i)
            assert (got.rc, got.lines(), got.circuit) == (plain.rc, plain.lines(), plain.circuit)
        b.close()


@pytest.mark.parametrize("n,length,budget", [(1, 12, 12), (2, 14, 9), (3, 18, 9)])
@pytest.mark.parametrize("seed", range(6))
def test_root_exponents(engine, oracle_bin, tmp_path, n, length, budget, seed):
    """roots of every small exponent at budgets where it bounds the residuals' exponents, and where the level does"""
    rng = random.Random(100 * n + seed)
    circ = []
    for _ in range(length):
        g = rng.choice(["h", "h", "t", "cx"] if n > 1 else ["h", "t", "t"])
        circ.append((g, tuple(rng.sample(range(n), 2)) if g == "cx" else (rng.randrange(n),)))
    text = workloads.make_spec(n, circ, budget)
    p = tmp_path / "t.spec"
    p.write_text(text)
    rc, lines = run_oracle(oracle_bin, p, [])
    out = engine.search(text)
    assert (out.rc, out.lines()) == (rc, lines)
