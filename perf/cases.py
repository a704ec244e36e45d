"""The workloads that the performance of this library is measured on, each through its public Python entry points.

listed() names the cases, draw() gives further ones of the same ranges, prepare() makes a case's inputs from a seed,
run() is one pass, work() the bytes and integer operations a pass cannot do without, and exact() the result of the
cases that plain torch can compute. Every path is exact integer work, so outputs are whole numbers: exit codes, the
per-level counts that the search programs print, found circuits, sorted pairs.

Like a program that serves synthesis requests, a process here keeps one engine (device buffers grown, tables
resident) and one batch session per qubit count for all its calls; what a call's own inputs need (their specs parsed)
is made by prepare(). The one case about start-up makes an engine of its own in every pass.
"""
import random

import numpy as np
import torch

import cheese_b200 as cz
from cheese_b200 import tcwork, workloads

# a Toffoli with controls 0, 1 and target 2 over Clifford+T (15 gates, the optimum)
TOFFOLI = [("h", (2,)), ("cx", (1, 2)), ("tdg", (2,)), ("cx", (0, 2)), ("t", (2,)), ("cx", (1, 2)), ("tdg", (2,)),
           ("cx", (0, 2)), ("t", (1,)), ("t", (2,)), ("h", (2,)), ("cx", (0, 1)), ("t", (0,)), ("tdg", (1,)),
           ("cx", (0, 1))]
# a repeat-until-success circuit with 12 T gates on two qubits (qubit 0 measured, outcome 1 the success)
RUS = ("h z t h t h s cz s h t h sdg t h s y t sdg h t h t sdg h s t h s y t sdg h s t h s h cz s h t h t s h").split()

# mean "prefixes" of one search of a Toffoli between local gates, per budget: with symmetry classes, without
PROOF_PREFIXES = {6: (1e3, 2e3), 7: (3e3, 6e3), 8: (1.2e4, 2.5e4), 9: (7e4, 1.7e5), 10: (4e5, 1e6),
                  11: (1.8e6, 4.7e6), 12: (9.1e6, 2.5e7)}
# per prefix: the residual update and tests of a child, and its share of the exact T bounds (110,656 operations each)
OPS_PER_PREFIX = 16000
OPS_PEEL = {3: 64 * 64 * 9, 2: 16 * 4 * 9}   # one rotation peeled off a channel matrix and its coset key, per qubits


def listed():
    return [
        # the smallest searches: a few 2-qubit circuits re-synthesised one by one, as a peephole optimiser does
        {"name": "small_2q", "path": "search", "n": 2, "gates": 6, "targets": 8},
        # budgets 1, 2, .. 9 in turn on one target: how an optimum is looked for, launch latency counts
        {"name": "ladder_9", "path": "ladder", "budget": 9, "targets": 1},
        # impossibility proofs of 3-qubit targets: ordinary size, and the deepest of the benchmark
        {"name": "proof_11", "path": "proof", "budget": 11, "targets": 4, "sym": True},
        {"name": "proof_12", "path": "proof", "budget": 12, "targets": 2, "sym": True},
        # the largest frontiers: symmetry classes off (--no-sym), tens of millions of prefixes
        {"name": "proof_12_nosym", "path": "proof", "budget": 12, "targets": 2, "sym": False},
        # batched search: uneven 2- and 3-qubit targets of 6 to 10 gates advanced together
        {"name": "batch_96", "path": "batch", "jobs": 96, "shortest": 6, "longest": 10},
        # searches that meet a resident distance table of the last 7 gates (--table 7)
        {"name": "table_13", "path": "table", "table_k": 7, "budget": 13, "targets": 2},
        # T-count queries against the resident 3-qubit coset table, 1 to 7 T gates
        {"name": "tcount_14", "path": "tcount", "table_k": 4, "tgates": 7, "queries": 14},
        # a process that starts up: Clifford group table and coset table built, first query and lookups answered
        {"name": "tables_cold", "path": "tables", "table_k": 3, "lookups": 4096},
        # Clifford gates around a circuit's T gates minimised (cliffopt, table resident)
        {"name": "cliffopt_3t", "path": "cliffopt", "tgates": 3, "beam": 16, "jobs": 2},
        # T-count of repeat-until-success circuits against the resident coset table
        {"name": "rus_6", "path": "rus", "table_k": 6, "maxt": 11, "targets": 2},
        # the stable sort of (64-bit key, 32-bit value) pairs that dedupes a frontier, at the largest frontiers' size
        {"name": "sort_30m", "path": "sort", "pairs": 30000000, "lo": 32, "hi": 64},
    ]


def draw(rng):
    path = rng.choice(["search", "ladder", "proof", "proof", "batch", "table", "tcount", "tables", "cliffopt", "rus",
                       "sort", "sort"])
    if path == "search":
        n = rng.choice([2, 3])
        return {"path": path, "n": n, "gates": rng.randint(4, 9 if n == 2 else 7), "targets": rng.randint(1, 24)}
    if path == "ladder":
        return {"path": path, "budget": rng.randint(5, 10), "targets": rng.randint(2, 8)}
    if path == "proof":
        sym = rng.random() < 0.6
        b = rng.randint(7, 12)
        return {"path": path, "budget": b, "sym": sym, "targets": rng.randint(1, {11: 3, 12: 1}.get(b, 12))}
    if path == "batch":
        lo = rng.randint(4, 6)
        return {"path": path, "jobs": rng.randint(8, 96), "shortest": lo, "longest": rng.randint(lo + 2, 10)}
    if path == "table":
        return {"path": path, "table_k": rng.randint(4, 7), "budget": rng.randint(9, 13), "targets": rng.randint(1, 4)}
    if path == "tcount":
        return {"path": path, "table_k": rng.randint(3, 4), "tgates": rng.randint(1, 6), "queries": rng.randint(1, 16)}
    if path == "tables":
        return {"path": path, "table_k": rng.randint(1, 3), "lookups": int(2 ** rng.uniform(0, 12))}
    if path == "cliffopt":
        return {"path": path, "tgates": rng.randint(0, 3), "beam": rng.randint(1, 16), "jobs": rng.randint(1, 2)}
    if path == "rus":
        return {"path": path, "table_k": rng.randint(5, 7), "maxt": rng.randint(10, 12), "targets": rng.randint(1, 4)}
    lo = rng.choice([0, 32, 32, 40])
    return {"path": path, "pairs": int(10 ** rng.uniform(3, 7.47)), "lo": lo, "hi": 64}


# ---------------- inputs ----------------
_kept = {}


def engine():
    """the process's engine"""
    if "engine" not in _kept:
        _kept["engine"] = cz.Engine(0)
    return _kept["engine"]


def session(n):
    """the process's batch session of n qubits"""
    if n not in _kept:
        _kept[n] = cz.Batch(engine(), n, memory_gb=40.0)
    return _kept[n]


def local_layer(rng):
    gates = [(rng.choice([None, "x", "z", "s", "sdg"]), (q,)) for q in range(3)]
    return [(g, q) for g, q in gates if g]


def dressed_toffoli(rng):
    """a Toffoli on shuffled qubits between two layers of one-qubit Cliffords: needs more gates than the budgets"""
    p = [0, 1, 2]
    rng.shuffle(p)
    core = [(g, tuple(p[q] for q in qs)) for g, qs in TOFFOLI]
    return local_layer(rng) + core + local_layer(rng)


def rus_circuit(rng):
    """the repeat-until-success circuit with random Cliffords on its data qubit before and after"""
    def word():
        return [(rng.choice(["h", "s", "sdg", "x", "y", "z"]), (1,)) for _ in range(rng.randint(1, 4))]
    return word() + [(g, (0, 1) if g == "cz" else (0,)) for g in RUS] + word()


def prepare(case, seed):
    rng = random.Random(seed)
    path = case["path"]
    if path == "search":
        circs = [workloads.random_circuit(rng, case["n"], case["gates"])[1] for _ in range(case["targets"])]
        return dict(case, specs=[cz.Spec(workloads.make_spec(case["n"], c, len(c))) for c in circs])
    if path in ("ladder", "proof", "table"):
        specs = [cz.Spec(workloads.make_spec(3, dressed_toffoli(rng), case["budget"])) for _ in range(case["targets"])]
        if path == "table":             # the distance table, built by the process's first search that needs it
            engine().search(specs[0], depth=1, table_k=case["table_k"], cache_dir=None)
        return dict(case, specs=specs)
    if path == "batch":
        jobs = [workloads.random_circuit(rng, None, rng.randint(case["shortest"], case["longest"]))
                for _ in range(case["jobs"])]
        return dict(case, specs=[cz.Spec(workloads.make_spec(n, c, len(c))) for n, c in jobs])
    if path in ("tcount", "tables"):
        texts = []
        for i in range(case.get("queries", 1)):
            circ = tcwork.random_clifford_word(rng, 3)
            for _ in range(1 + i % case.get("tgates", case["table_k"])):
                circ += [("t", (rng.randrange(3),))] + tcwork.random_clifford_word(rng, 3)
            texts.append(cz.tspec_generate(3, circ))
        if path == "tcount":            # the coset table, built by the process's first query
            engine().tcount(texts[0], table_k=case["table_k"], cache_dir=None)
            return dict(case, texts=texts)
        index = [rng.randrange(tcwork.CLIFFORD_ORDER[3]) for _ in range(case["lookups"])]
        return dict(case, texts=texts, index=index)
    if path == "cliffopt":
        engine().clifford_table(3)
        return dict(case, texts=[tcwork.random_clifford_job(rng, 3, 40, case["tgates"]) for _ in range(case["jobs"])])
    if path == "rus":
        texts = [cz.rspec_generate(2, rus_circuit(rng), outcome=1)[0] for _ in range(case["targets"])]
        engine().rus(texts[0], table_k=case["table_k"], maxt=1, cache_dir=None)
        return dict(case, texts=texts)
    engine()
    keys, vals = pairs(case, seed)
    return dict(case, keys=keys, vals=vals, sorted_keys=torch.empty_like(keys), sorted_vals=torch.empty_like(vals))


def pairs(case, seed):
    """class keys as a level leaves them: 64-bit hashes, about a third of them seen before, values 0, 1, 2, .."""
    n = case["pairs"]
    g = torch.Generator(device="cuda").manual_seed(seed)
    keys = torch.randint(-(1 << 62), 1 << 62, (n,), dtype=torch.int64, device="cuda", generator=g)
    again = torch.randint(0, n, (n // 3,), device="cuda", generator=g)
    keys[n - n // 3:] = keys[again]
    return keys, torch.arange(n, dtype=torch.int32, device="cuda")


# ---------------- one pass ----------------
COUNTS = ("t", "parents", "prefixes", "cut_w3", "cut_lb", "survivors", "distinct")
COSETS = ("table", "t", "parents", "children", "cosets", "fresh")


def padded(values, length):
    """a result of varying length in a place of fixed length (-1 behind its end)"""
    return (list(values) + [-1] * length)[:length]


def search_numbers(r):
    """what the search program prints of an outcome: exit code, circuit, every level's counts (at most 16 levels)"""
    return ([r.rc, r.n_found, len(r.levels)] + padded(r.raw.found[:r.raw.found_len], 16) +
            padded([l[k] for l in r.levels for k in COUNTS], 16 * len(COUNTS)))


def coset_numbers(rc, levels, sequence):
    """what the T-count programs print: exit code, every level's counts (at most 16 levels), the decomposition"""
    return ([rc, len(levels)] + padded([l[k] for l in levels for k in COSETS], 16 * len(COSETS)) +
            padded(sequence, 64))


def run(state):
    path = state["path"]
    out = []
    if path == "search":
        for s in state["specs"]:
            out += search_numbers(engine().search(s))
    elif path == "ladder":
        for s in state["specs"]:
            for budget in range(1, state["budget"] + 1):
                out += search_numbers(engine().search(s, depth=budget))
    elif path == "proof":
        for s in state["specs"]:
            out += search_numbers(engine().search(s, sym=state["sym"]))
    elif path == "table":
        for s in state["specs"]:
            out += search_numbers(engine().search(s, table_k=state["table_k"], cache_dir=None))
    elif path == "batch":
        ids = [(s.n, session(s.n).submit(s)) for s in state["specs"]]
        for n in sorted({n for n, _ in ids}):
            session(n).run()
        for n, i in ids:
            out += search_numbers(session(n).result(i))
    elif path == "tcount":
        for t in state["texts"]:
            rc, levels, r = engine().tcount(t, table_k=state["table_k"], cache_dir=None)
            out += coset_numbers(rc, levels, [r["tcount"]] + [v for rot in r["rotations"] for v in rot])
    elif path == "tables":
        eng = cz.Engine(0)
        table = eng.clifford_table(3)
        elements = eng.clifford_element(3, state["index"])
        dist = eng.clifford_dist(3, elements)
        rc, levels, r = eng.tcount(state["texts"][0], table_k=state["table_k"], cache_dir=None)
        eng.close()
        out = (table["per_distance"] + elements + dist +
               coset_numbers(rc, levels, [r["tcount"]] + [v for rot in r["rotations"] for v in rot]))
    elif path == "cliffopt":
        for t in state["texts"]:
            rc, r, lines, steps = engine().cliffopt(t, beam=state["beam"])
            out += [rc, r["clifford_gates"], r["clifford_gates_before"]] + [v for s in steps for v in s]
            out += padded("\n".join(lines).encode(), 4096)
    elif path == "rus":
        for t in state["texts"]:
            rc, levels, r = engine().rus(t, table_k=state["table_k"], maxt=state["maxt"], cache_dir=None)
            out += coset_numbers(rc, levels, [r["tcount"], r["root"], r["cliff"]] + r["fw"] + r["tb"])
    else:
        keys, vals = state["sorted_keys"], state["sorted_vals"]
        keys.copy_(state["keys"])
        vals.copy_(state["vals"])
        torch.cuda.current_stream().synchronize()    # the sort runs on the engine's stream
        engine().sort_pairs(keys.data_ptr(), vals.data_ptr(), state["pairs"], state["lo"], state["hi"])
        return keys, vals
    return np.array(out, dtype=np.int64)


# ---------------- what a pass cannot do without ----------------
def work(case):
    path = case["path"]
    if path == "search":
        # a random circuit's optimum is often below its length
        prefixes = case["targets"] * (3.7 if case["n"] == 2 else 5.0) ** case["gates"]
        return {"bytes": case["targets"] * 4e4, "flops": prefixes * OPS_PER_PREFIX}
    if path in ("ladder", "proof"):
        col = 0 if case.get("sym", True) else 1
        budgets = range(1, case["budget"] + 1) if path == "ladder" else [case["budget"]]
        prefixes = case["targets"] * sum(PROOF_PREFIXES.get(b, (500, 500))[col] for b in budgets)
        return {"bytes": case["targets"] * 4e4, "flops": prefixes * OPS_PER_PREFIX}
    if path == "table":
        prefixes = case["targets"] * 13.4 ** (case["budget"] - case["table_k"])
        return {"bytes": case["targets"] * 4e4, "flops": prefixes * OPS_PER_PREFIX}
    if path == "batch":
        span = range(case["shortest"], case["longest"] + 1)
        prefixes = case["jobs"] * sum(4.4 ** g for g in span) / len(span)
        return {"bytes": case["jobs"] * 4e4, "flops": prefixes * OPS_PER_PREFIX}
    if path == "tcount":
        levels = [max(0, 1 + i % case["tgates"] - case["table_k"]) for i in range(case["queries"])]
        peels = sum(1 + sum(63.0 ** l for l in range(1, j + 1)) for j in levels)
        return {"bytes": case["queries"] * 5e4, "flops": peels * OPS_PEEL[3]}
    if path == "tables":
        # every group element claimed once and its distance written; the coset table's peels
        peels = sum(63.0 ** l for l in range(1, case["table_k"] + 1))
        return {"bytes": 92897280.0, "flops": 92897280.0 * 21 * 10 + peels * OPS_PEEL[3]}
    if path == "cliffopt":
        # per T gate: every beam state x two sides x the placements (4.4 million), a composed tableau and its rank
        evals = case["jobs"] * (1 + case["tgates"] * case["beam"] * 2 * 4.4e6)
        return {"bytes": case["jobs"] * 2e3, "flops": evals * 60}
    if path == "rus":
        # 12 roots, 15 rotations, the children of a level about 10 times those of the one before; optimum 10
        levels = max(0, min(case["maxt"], 10) - case["table_k"])
        peels = case["targets"] * (1 + sum(180.0 * 10.0 ** l for l in range(levels)))
        return {"bytes": case["targets"] * 1.5e6, "flops": peels * OPS_PEEL[2]}
    return {"bytes": 24.0 * case["pairs"], "flops": 0}


def exact(case, seed):
    """the sorted pairs by torch's own stable sort; the search paths have no such plain form"""
    if case["path"] != "sort":
        return None
    keys, vals = pairs(case, seed)
    digits = keys ^ torch.iinfo(torch.int64).min if case["lo"] == 0 else (keys >> case["lo"]) & ((1 << (64 - case["lo"])) - 1)
    _, order = torch.sort(digits, stable=True)
    return keys[order], vals[order]
