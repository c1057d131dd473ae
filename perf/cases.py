"""Timed cases of the engine: the calls that a program makes, over the sizes it makes them at.

A case is a dict of plain values. ``listed()`` are the named ones; ``draw(rng)`` gives one
more of the same ranges; ``prepare(case, seed)`` builds what a program has in hand before
the call (automata, inputs, an engine or a captured step), from the seed alone;
``run(state)`` makes one pass through the package's public entry points and returns its
verdicts; ``work(case)`` is what a pass cannot do without.

The automata and length distributions are those of ``abstraction_regret_gb300.workloads``
(seeded differently per state). The inputs of a random NFA are random walks of it, so its
active set stays alive; those of a DFA are uniform bytes. ``accept`` is the share of
accepting states. Beside them each automaton carries a signature, a short chain of states
to an accepting one that matches near the end of one of its inputs (and hardly anywhere
else): a scan that looks at nearly every byte and finds something now and then.

The ``call`` of a case says which entry point it uses:

* ``run`` / ``run_batch``: the drop-in call on host ``bytes`` with its default technique;
* ``engine``: ``PersistentEngine.run_requests``, host requests over a pool of automata;
* ``step``: ``GraphRunner.kernel_only``, the engine's step on inputs resident in HBM;
* ``replay``: ``GraphRunner.replay`` and ``verdicts``, the captured end-to-end step from
  pinned host memory;
* ``launch``: an executor's ``launch``, one plain launch on resident inputs.
"""

from __future__ import annotations

import math

import numpy as np
import torch

from abstraction_regret_gb300 import anml, api
from abstraction_regret_gb300 import workloads as W
from abstraction_regret_gb300.automata import DFA, nfa_from_edges, random_dfa
from abstraction_regret_gb300.engine import GraphRunner, PersistentEngine
from abstraction_regret_gb300.executors import CudaDFAExecutor

KIB = 1 << 10
MIB = 1 << 20


def listed() -> list[dict]:
    return [
        # one short string against a small pattern automaton: an interactive check, where
        # the call's own overhead is the time
        dict(name="run-one-256", call="run", kind="nfa", states=1024, degree=2.0, accept=0.0,
             inputs=1, lo=256, hi=256),
        # a small batch of equal records (log lines grouped into pages) with 1% accepting
        # states, most of which latch early
        dict(name="batch-64x4k", call="run_batch", kind="nfa", states=1024, degree=2.0,
             accept=0.01, inputs=64, lo=4 * KIB, hi=4 * KIB),
        # an ordinary batch of files of very uneven length, scanned to the end
        dict(name="batch-uneven-8m", call="run_batch", kind="nfa", states=16384, degree=4.0,
             accept=0.0, inputs=64, lo=256, hi=MIB),
        # the largest batch of host bytes: the benchmark's uneven batch through the drop-in call
        dict(name="batch-uneven-260m", call="run_batch", kind="nfa", states=16384, degree=4.0,
             accept=0.0, inputs=2048, lo=256, hi=MIB),
        # the benchmark's step: the same batch resident in HBM, planning included
        dict(name="step-uneven-260m", call="step", kind="nfa", states=16384, degree=4.0,
             accept=0.0, inputs=2048, lo=256, hi=MIB),
        # the benchmark's end-to-end step: pinned host inputs in, verdicts out, one graph
        dict(name="replay-uneven-260m", call="replay", kind="nfa", states=16384, degree=4.0,
             accept=0.0, inputs=2048, lo=256, hi=MIB),
        # a rule set of many automata over resident traffic, 16 inputs each
        dict(name="step-pool-64", call="step", kind="pool", nfas=64, dfas=0, accept=0.0,
             inputs=1024, lo=KIB, hi=256 * KIB),
        # one batch of a service: requests over a mixed pool of NFAs and DFAs, some matching
        dict(name="engine-mixed", call="engine", kind="pool", nfas=16, dfas=16, accept=0.0005,
             inputs=500, lo=64, hi=MIB),
        # short records through a small compiled DFA
        dict(name="dfa-records", call="run_batch", kind="dfa", states=512, accept=0.0,
             inputs=2000, lo=64, hi=4 * KIB),
        # a compiled DFA over many equal resident blocks: one plain launch
        dict(name="dfa-blocks", call="launch", kind="dfa", states=4096, accept=0.0,
             inputs=4096, lo=64 * KIB, hi=64 * KIB),
        # a few long files through a large compiled DFA
        dict(name="dfa-long", call="step", kind="dfa", states=8192, accept=0.0, inputs=8,
             lo=2 * MIB, hi=2 * MIB),
        # signature patterns loaded from ANML (epsilon edges, wildcards) over documents
        dict(name="anml-documents", call="run_batch", kind="anml", patterns=100, inputs=64,
             lo=4 * KIB, hi=32 * KIB),
    ]


def _log_int(rng, lo: int, hi: int) -> int:
    return int(min(hi, max(lo, math.exp(rng.uniform(math.log(lo), math.log(hi))))))


def draw(rng) -> dict:
    """One more case: a call and a kind of automaton as listed, its sizes drawn over the
    listed range (over their logarithm), odd ones among them; the offered bytes stay below
    the largest listed case's."""
    pick = rng.randrange(8)
    if pick == 0:  # one input, from a few bytes to a page or two
        n = _log_int(rng, 16, 16 * KIB)
        return dict(call="run", kind="nfa", states=_log_int(rng, 200, 16384),
                    degree=rng.choice([2.0, 3.0, 4.0]), accept=rng.choice([0.0, 0.01]), inputs=1,
                    lo=n, hi=n)
    if pick in (1, 2, 3):  # an uneven batch of one NFA, host bytes or resident
        hi = _log_int(rng, 2 * KIB, MIB)
        # mean of a log-uniform length is (hi - lo) / ln(hi / lo): at most about 200 MB
        most = int(min(4096, 200 * MIB * math.log(hi / 256) / (hi - 256)))
        return dict(call=("run_batch", "step", "replay")[pick - 1], kind="nfa",
                    states=_log_int(rng, 256, 65536), degree=rng.choice([2.0, 3.0, 4.0, 4.5]),
                    accept=rng.choice([0.0, 0.0, 0.001]), inputs=_log_int(rng, 8, most), lo=256,
                    hi=hi)
    if pick == 4:  # a pool: NFAs alone over resident inputs, or a mixed batch of requests
        mixed = rng.random() < 0.5
        return dict(call="engine" if mixed else "step", kind="pool", nfas=rng.randint(3, 24),
                    dfas=rng.randint(3, 16) if mixed else 0, accept=rng.choice([0.0, 0.0005]),
                    inputs=_log_int(rng, 50, 800), lo=64, hi=_log_int(rng, 8 * KIB, 512 * KIB))
    if pick == 5:  # short or ordinary records through a DFA
        call = rng.choice(["run_batch", "launch"])
        hi = _log_int(rng, KIB, 32 * KIB)
        return dict(call=call, kind="dfa", states=_log_int(rng, 64, 16384),
                    accept=rng.choice([0.0, 0.0005]), inputs=_log_int(rng, 100, 6000), lo=64,
                    hi=hi)
    if pick == 6:  # long inputs through a DFA
        return dict(call="step", kind="dfa", states=_log_int(rng, 256, 16384),
                    accept=rng.choice([0.0, 0.0, 0.00001]), inputs=rng.randint(1, 24),
                    lo=512 * KIB, hi=_log_int(rng, MIB, 4 * MIB))
    return dict(call="run_batch", kind="anml", patterns=_log_int(rng, 10, 200),
                inputs=_log_int(rng, 8, 128), lo=KIB, hi=_log_int(rng, 4 * KIB, 32 * KIB))


# ---- inputs and automata of a case -------------------------------------------------------------


def _nfa(states: int, seed: int, degree: float, accept: float):
    states -= SIGNATURE
    if degree == int(degree) and degree < 4:
        return W.random_nfa(states, seed=seed, degree=int(degree), accept_prob=accept)
    if degree == 4.5:  # uniform 1..8, as the pools of the configurations
        return W.random_nfa(states, seed=seed, degree=(1, 8), accept_prob=accept)
    return W.random_nfa(states, seed=seed, poisson=degree, accept_prob=accept)


def _dfa(states: int, seed: int, accept: float):
    return random_dfa(states - DFA_SIGNATURE, accept_prob=accept, seed=seed)


SIGNATURE = 4        # states of an NFA's signature chain
DFA_SIGNATURE = 2    # ... of a DFA's
SIGNATURE_REACH = 100_000  # the signature lies within the first so many bytes of its input


def _signed_input(lens: np.ndarray, rng, chain: int) -> tuple[int, int]:
    """The input that carries the signature (one of the shorter ones that hold it) and the
    position at which the signature starts, near that input's end."""
    fit = np.flatnonzero(lens > chain)
    if not fit.size:
        return -1, 0
    fit = fit[np.argsort(lens[fit], kind="stable")]
    i = int(fit[int(rng.integers(0, max(1, fit.size // 4)))])
    last = int(min(lens[i], SIGNATURE_REACH)) - chain
    return i, max(0, last - int(rng.integers(0, max(1, last // 8))))


def _sign_nfa(a, data: np.ndarray, off: np.ndarray, rng):
    """``a`` plus a chain of states that reads the bytes of one of its inputs from one of
    the states active there, its last state accepting."""
    i, at = _signed_input(np.diff(off), rng, SIGNATURE)
    if i < 0:
        return a
    x = data[off[i]:off[i] + at + SIGNATURE].tolist()
    rows = [(a.sym_symbols[b:e].tolist(), a.sym_targets[b:e].tolist())
            for b, e in zip(a.sym_row_ptr[:-1].tolist(), a.sym_row_ptr[1:].tolist())]
    active = {int(a.start_state)}
    for c in x[:at]:
        step = {t for s in active for y, t in zip(*rows[s]) if y == c}
        if not step:
            return a
        active = step
    n = int(a.num_states)
    src = np.repeat(np.arange(n, dtype=np.int64), np.diff(a.sym_row_ptr))
    chain = np.arange(n, n + SIGNATURE)
    accept = np.concatenate([a.accept, np.arange(SIGNATURE) == SIGNATURE - 1])
    return nfa_from_edges(n + SIGNATURE, a.start_state, accept,
                          np.concatenate([src, [min(active)], chain[:-1]]),
                          np.concatenate([a.sym_symbols, x[at:]]),
                          np.concatenate([a.sym_targets, chain]))


def _sign_dfa(a, data: np.ndarray, off: np.ndarray, rng):
    """``a`` plus states that follow its walk over a few bytes of one of its inputs, the
    last one accepting; on other bytes they go on as the states they stand for."""
    i, at = _signed_input(np.diff(off), rng, DFA_SIGNATURE)
    if i < 0:
        return a
    x = data[off[i]:off[i] + at + DFA_SIGNATURE].tolist()
    s = int(a.start_state)
    flat = a.trans.tolist()
    for c in x[:at]:
        s = flat[s * 256 + c]
    n = int(a.num_states)
    trans = a.trans.reshape(n, 256)
    follow = []  # the states that the chain stands for
    t = s
    for c in x[at:]:
        t = int(trans[t, c])
        follow.append(t)
    trans = np.concatenate([trans, trans[follow]])
    at_state = s
    for k, c in enumerate(x[at:]):
        trans[at_state, c] = n + k
        at_state = n + k
    accept = np.concatenate([a.accept, np.arange(DFA_SIGNATURE) == DFA_SIGNATURE - 1])
    return DFA(num_states=n + DFA_SIGNATURE, start_state=a.start_state, accept=accept,
               trans=trans.reshape(-1))


def _lengths(case: dict) -> np.ndarray:
    # lengths belong to the case (the same for every seed), so that every state of a case
    # is the same amount of work
    rng = np.random.default_rng([case["inputs"], case["lo"], case["hi"]])
    return W.log_uniform_lengths(rng, case["inputs"], case["lo"], case["hi"])


def _uniform(total: int, seed: int) -> np.ndarray:
    gen = torch.Generator(device="cuda").manual_seed(seed)
    return torch.randint(0, 256, (max(total, 1),), dtype=torch.uint8, device="cuda",
                         generator=gen)[:total].cpu().numpy()


def _pool_states(case: dict) -> tuple[list[int], list[int]]:
    rng = np.random.default_rng([case["nfas"], case["dfas"], 9])
    nfas = [int(math.exp(x)) for x in rng.uniform(math.log(256), math.log(65536), case["nfas"])]
    dfas = [int(math.exp(x)) for x in rng.uniform(math.log(1024), math.log(16384), case["dfas"])]
    return nfas, dfas


def _pool(case: dict, seed: int):
    """The pool, each input's automaton, the flat inputs and their offsets. Resident rule
    sets group the inputs by automaton; requests name automata at random."""
    ns, ds = _pool_states(case)
    automata = [_nfa(s, seed * 1000 + k, 4.5, case["accept"]) for k, s in enumerate(ns)]
    automata += [_dfa(s, seed * 1000 + 500 + k, case["accept"]) for k, s in enumerate(ds)]
    n = case["inputs"]
    if case["call"] == "step":
        aut = np.arange(n, dtype=np.int64) * len(automata) // n
    else:
        aut = np.random.default_rng([n, 3]).integers(0, len(automata), n)
    off = W.offsets_of(_lengths(case))
    data = _uniform(int(off[-1]), seed)
    for k in range(len(automata)):
        ids = np.flatnonzero(aut == k)
        sub = W.offsets_of(off[ids + 1] - off[ids])
        rng = np.random.default_rng([seed, k])
        if k < len(ns):
            own = W.walk_bytes(automata[k], sub, seed=seed * 1000 + k)
            for j, i in enumerate(ids):
                data[off[i]:off[i + 1]] = own[sub[j]:sub[j + 1]]
            automata[k] = _sign_nfa(automata[k], own, sub, rng)
        elif k < len(ns) + 2:  # two of the DFAs (walking the inputs of each takes long)
            own = np.concatenate([data[off[i]:off[i + 1]] for i in ids] + [data[:0]])
            automata[k] = _sign_dfa(automata[k], own, sub, rng)
    return automata, aut, data, off


def _batch(case: dict, seed: int):
    """One automaton (in a list), automaton ids, the flat inputs and their offsets."""
    if case["kind"] == "pool":
        return _pool(case, seed)
    off = W.offsets_of(_lengths(case))
    rng = np.random.default_rng([seed, 77])
    if case["kind"] == "nfa":
        a = _nfa(case["states"], seed, case["degree"], case["accept"])
        data = W.walk_bytes(a, off, seed=seed + 1)
        a = _sign_nfa(a, data, off, rng)
    elif case["kind"] == "dfa":
        a = _dfa(case["states"], seed, case["accept"])
        data = _uniform(int(off[-1]), seed + 1)
        a = _sign_dfa(a, data, off, rng)
    else:
        a = anml.load_anml_string(W.anml_patterns(case["patterns"], seed=seed, min_len=8))
        lens = np.diff(off)
        data = np.concatenate([np.frombuffer(W.anml_inputs(a, 1, int(m), seed * 1000 + i,
                                                           plant=0.3)[0], dtype=np.uint8)
                               for i, m in enumerate(lens)])
    return [a], np.zeros(case["inputs"], dtype=np.int64), data, off


def prepare(case: dict, seed: int):
    automata, aut, data, off = _batch(case, seed)
    call = case["call"]
    inputs = [data[off[i]:off[i + 1]].tobytes() for i in range(len(off) - 1)] \
        if call in ("run", "run_batch", "engine") else None
    if call in ("run", "run_batch"):
        # the executor (the automaton's device layout) is kept per automaton by the package;
        # a program that scans with an automaton has it from its first call
        api.run_batch(automata[0], [b""])
        return call, automata[0], inputs
    if call == "engine":
        return call, PersistentEngine(automata), (aut, inputs)
    if call in ("step", "replay"):
        engine = PersistentEngine(automata)
        runner = GraphRunner(engine, aut, data, off, with_examined=True,
                             ingest="pipelined" if call == "replay" else "copy")
        return call, runner, None
    n = len(off) - 1
    d_data = torch.zeros(max(16, -(-int(off[-1]) // 16) * 16), dtype=torch.uint8, device="cuda")
    d_data[: int(off[-1])].copy_(torch.from_numpy(data))
    d_off = torch.from_numpy(off).cuda()
    out = torch.zeros((3, n), dtype=torch.int32, device="cuda")
    return call, CudaDFAExecutor(automata[0]), (d_data, d_off, n, out)


def run(state):
    call, what, more = state
    if call == "run":
        r = api.run(what, more[0])
        return [r.accepted, r.match_len]
    if call == "run_batch":
        res = api.run_batch(what, more)
        return [np.array([r.accepted for r in res]), np.array([r.match_len for r in res])]
    if call == "engine":
        flags, lens, examined, _, _ = what.run_requests(more[0], more[1], with_examined=True)
        return [flags, lens, examined]
    if call == "step":
        what.kernel_only()
        return [what.d_out]
    if call == "replay":
        what.replay()
        return list(what.verdicts())
    d_data, d_off, n, out = more
    what.launch(d_data, d_off, n, out[0], out[1], out[2])
    return [out]


def work(case: dict) -> dict:
    """Bytes: each input byte that a run has to look at read once (inputs that accept stop
    early: on average after 1 / accept bytes), the automaton's edges (three bytes: label
    and target) or table (two bytes an entry) read once, the verdicts written. There are no
    floating-point operations; one lookup per byte is counted as an operation."""
    lens = _lengths(case).astype(np.float64)
    p = case.get("accept", 0.0)
    looked = float(np.minimum(lens, 1.0 / p).sum()) if p else float(lens.sum())
    if case["kind"] == "pool":
        ns, ds = _pool_states(case)
        table = 3 * 4.5 * sum(ns) + 512 * sum(ds)
    elif case["kind"] == "nfa":
        table = 3 * case["degree"] * case["states"]
    elif case["kind"] == "dfa":
        table = 512 * case["states"]
    else:
        table = 3 * 16 * 20 * case["patterns"]
    return {"bytes": looked + table + 12.0 * case["inputs"], "flops": looked}


def exact(case: dict, seed: int):
    """Verdicts are whole numbers: there is no rounding to compare, so no 64-bit value."""
    return None
