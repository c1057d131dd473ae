"""Slot tables (csrc/slots.cu): the packed transition function of an epsilon-free NFA that
lane chunks walk (csrc/lane_slots.cuh).

CPU: every slot of a state or coded set leads where the automaton's edges lead, codes lie
in the ranges that the kernels test, and empty slots never hit. GPU: the three places a
table is read from (shared memory at 4 or at 3 bytes a slot, global memory) and the edges
between them, against the oracle.
"""

from __future__ import annotations

import numpy as np
import pytest

import abstraction_regret_gb300 as G
from abstraction_regret_gb300 import build, device, native
from abstraction_regret_gb300 import workloads as W
from abstraction_regret_gb300.engine import GraphRunner, PersistentEngine
from oracle import oracle as O


def _letters(n: int, letters: int, degree: int, accept: float, seed: int):
    """Edges labelled from a small alphabet: most states step to sets."""
    rng = np.random.default_rng(seed)
    acc = rng.random(n) < accept
    acc[0] = False
    return G.nfa_from_edges(n, 0, acc, np.repeat(np.arange(n), degree),
                            rng.integers(65, 65 + letters, n * degree),
                            rng.integers(0, n, n * degree))


def _wild(n: int, share: float, seed: int):
    rng = np.random.default_rng(seed)
    syms = np.where(rng.random(3 * n) < share, G.ANY_SYMBOL, rng.integers(0, 256, 3 * n))
    return G.nfa_from_edges(n, 0, np.arange(n) % 50 == 3, np.repeat(np.arange(n), 3), syms,
                            rng.integers(0, n, 3 * n))


AUTOMATA = {
    "one state": lambda: W.random_nfa(1, seed=1, degree=0),
    "degree 1, half accepting": lambda: W.random_nfa(300, seed=5, degree=1, accept_prob=0.5),
    "degree 200": lambda: W.random_nfa(50, seed=1, degree=200, accept_prob=0.1),
    "1024 states": lambda: W.random_nfa(1024, seed=0, degree=2, accept_prob=0.01),
    "16384 states": lambda: W.random_nfa(16384, seed=2, poisson=4.0, accept_prob=0.001),
    "32768 states": lambda: W.random_nfa(32768, seed=3, degree=(1, 8), accept_prob=0.01),
    "six letters": lambda: _letters(400, 6, 3, 0.02, 7),
    "two letters": lambda: _letters(300, 2, 9, 0.0, 8),  # sets of more than 8 states
    "a few wildcards": lambda: _wild(400, 0.01, 9),
}


@pytest.mark.parametrize("name", AUTOMATA)
def test_slots_hold_the_transition_function(name):
    build.build()
    a = AUTOMATA[name]()
    t = device.slot_table(a)
    slots, pairs, multi = t["slots"], t["pairs"], t["multi_code"]
    state = {int(c): s for s, c in enumerate(t["state_code"])}
    coded = {int(c): (int(ls), int(k)) for c, ls, k in t["sets"]}
    assert len(set(state) | set(coded)) == a.num_states + len(t["sets"])
    assert slots.size == 2 * multi + 256

    def members(code):
        code = int(code)
        if code in coded:
            out = members(coded[code][0])
            assert len(out) == coded[code][1] <= 8
            return out
        out = set()
        while code > multi:
            out.add(state[int(pairs[2 * (code - multi - 1)])])
            code = int(pairs[2 * (code - multi - 1) + 1])
        return out | {state[code]}

    rp, sy, tg = a.sym_row_ptr, a.sym_symbols, a.sym_targets
    rng = np.random.default_rng(0)
    for code in list(rng.permutation(list(state))[:60]) + list(coded)[:40]:
        mem = members(code)
        accepting = any(bool(a.accept[s]) for s in mem)
        assert (code >= t["accept_code"]) == accepting and code < multi
        assert (code < t["set_code"]) == (len(mem) == 1 and not accepting)
        for c in range(256):
            want = {int(y) for s in mem for x, y in zip(sy[rp[s]:rp[s + 1]], tg[rp[s]:rp[s + 1]])
                    if x in (c, G.ANY_SYMBOL)}
            e = int(slots[2 * int(code) + c])
            assert (members(e >> 8) if e & 0xFF == c else set()) == want
    none = slots[2 * multi:2 * multi + 256]
    assert ((none & 0xFF) != np.arange(256)).all()
    narrow = device.narrow_slots(t)
    if narrow is not None:
        n16 = -(-slots.size // 16) * 16
        assert np.array_equal(narrow[:slots.size], slots & 0xFF)
        assert np.array_equal(narrow[n16:n16 + 2 * slots.size].view(np.uint16), slots >> 8)


def test_wildcard_heavy_automata_have_no_slot_table():
    build.build()
    assert device.slot_table(_wild(400, 0.15, 11)) is None


@pytest.mark.gpu
@pytest.mark.parametrize("name", [k for k in AUTOMATA if k != "one state"])
@pytest.mark.parametrize("chunk", [0, 64, 333])
def test_lane_chunks_over_slots(name, chunk):
    """Short chunks (below the checkpoints and the overlap), unaligned ones, and the
    planner's own, by the one-automaton launch and by the pool's."""
    a = AUTOMATA[name]()
    lengths = np.concatenate([np.arange(0, 70), W.log_uniform_lengths(
        np.random.default_rng(3), 120, 60, 9000)])
    off = W.offsets_of(lengths)
    data = W.walk_bytes(a, off, seed=4)
    eng = PersistentEngine([a], chunk_bytes=chunk, lane_pair_mean=float("inf"))
    other = PersistentEngine([a, W.random_nfa(64, seed=1, degree=2)], chunk_bytes=chunk,
                             lane_pair_mean=float("inf"))
    want = O.nfa_batch(a, data, off)[:3]
    for e in (eng, other):
        g = GraphRunner(e, np.zeros(lengths.size), data, off, with_examined=True)
        g.replay()
        for got, w in zip(g.verdicts(), want):
            assert np.array_equal(got, w)


@pytest.mark.gpu
def test_where_the_lane_launch_keeps_a_table():
    stage = {k: PersistentEngine([AUTOMATA[k]()]).lane_stage[0]
             for k in ("1024 states", "16384 states", "32768 states")}
    assert stage == {"1024 states": native.LANE_STAGE_WIDE,
                     "16384 states": native.LANE_STAGE_NARROW,
                     "32768 states": native.LANE_STAGE_NONE}
