"""Symbol lists (device.symbol_lists) and the steppers that use them (csrc/sym_device.cuh,
csrc/sym_fixup.cu): automata with epsilon edges or many wildcards.

CPU: the lists hold the edges of every byte, closed under epsilon edges. GPU: chunks, whole
inputs and the serial fix-up against the oracle, with lists shorter and longer than what is
loaded ahead, sets that die, accept at any byte or never link, and inputs of every length
around a chunk.
"""

from __future__ import annotations

import numpy as np
import pytest

import abstraction_regret_gb300 as G
from abstraction_regret_gb300 import device
from abstraction_regret_gb300 import workloads as W
from abstraction_regret_gb300.engine import PersistentEngine
from oracle import oracle as O


def _nfa(n, seed, letters=3, degree=2, eps=0.3, wild=0.0, accepts=1, stay=False):
    """Random edges on a few letters, some epsilon edges, the last states accepting; with
    ``stay`` state 0 keeps itself active on every byte."""
    rng = np.random.default_rng(seed)
    src = np.repeat(np.arange(n), degree)
    sym = np.where(rng.random(src.size) < wild, G.ANY_SYMBOL,
                   rng.integers(97, 97 + letters, src.size))
    dst = rng.integers(0, max(1, n - accepts), src.size)
    if stay:
        src, sym, dst = np.r_[src, 0], np.r_[sym, G.ANY_SYMBOL], np.r_[dst, 0]
    # one edge on a byte of its own into each accepting state
    src = np.r_[src, rng.integers(0, n - accepts, accepts)]
    sym = np.r_[sym, np.full(accepts, 120)]
    dst = np.r_[dst, np.arange(n - accepts, n)]
    esrc = np.flatnonzero(rng.random(n - accepts) < eps)
    edst = rng.integers(0, n - accepts, esrc.size)
    return G.nfa_from_edges(n, 0, np.arange(n) >= n - accepts, src, sym, dst, esrc, edst)


def _closure(nfa, states):
    erp, etg = np.asarray(nfa.eps_row_ptr), np.asarray(nfa.eps_targets)
    out, todo = set(states), list(states)
    while todo:
        s = todo.pop()
        for t in etg[erp[s]:erp[s + 1]].tolist():
            if t not in out:
                out.add(t)
                todo.append(t)
    return out


@pytest.mark.parametrize("kw", [dict(n=1, seed=1, accepts=0, degree=1), dict(n=40, seed=2),
                                dict(n=40, seed=3, eps=0.0, wild=0.2),
                                dict(n=300, seed=4, wild=0.05, accepts=3, stay=True)])
def test_lists_hold_the_closed_edges_of_every_byte(kw):
    a = _nfa(**kw)
    row, pairs = device.symbol_lists(a)
    assert row.size == 258 and row[-1] == pairs.size
    rp, sy, tg = a.sym_row_ptr, a.sym_symbols, a.sym_targets
    src = np.repeat(np.arange(a.num_states), np.diff(rp))
    for c in list(range(95, 125)) + [0, 255]:
        want = {(int(s), t) for s, y, x in zip(src, sy, tg) if y in (c, G.ANY_SYMBOL)
                for t in _closure(a, [int(x)])}
        got = [(int(p) & 0x7FFF, (int(p) >> 15) & 0x7FFF) for p in pairs[row[c]:row[c + 1]]]
        assert len(got) == len(set(got)) and set(got) == want
        assert all(bool(int(p) >> 30) == bool(a.accept[(int(p) >> 15) & 0x7FFF])
                   for p in pairs[row[c]:row[c + 1]])
    start = {(int(p) >> 15) & 0x7FFF for p in pairs[row[256]:row[257]]}
    assert start == _closure(a, [a.start_state])


def test_no_lists_beyond_their_limits():
    assert device.symbol_lists(W.random_nfa(32769, seed=1, degree=1)) is None
    assert device.symbol_lists(_nfa(2000, seed=5, wild=1.0, degree=3)) is None


def _inputs(seed, letters, lengths, mark=0.5):
    rng = np.random.default_rng(seed)
    out = []
    for n in lengths:
        x = rng.integers(97, 97 + letters, int(n), dtype=np.uint8)
        if n and rng.random() < mark:
            x[rng.integers(0, n, 3)] = 120
        out.append(x.tobytes())
    return out


@pytest.mark.gpu
@pytest.mark.parametrize("kw", [
    dict(n=40, seed=11), dict(n=64, seed=12, stay=True), dict(n=65, seed=13, stay=True, wild=0.05),
    dict(n=300, seed=14, letters=2, degree=3, stay=True),   # lists of 256..512 pairs
    dict(n=1500, seed=15, letters=2, degree=2, eps=0.1),    # longer than the pairs ahead
    dict(n=9000, seed=16, letters=40, degree=2, eps=0.1, stay=True),  # 3 clears a thread
    dict(n=30, seed=17, letters=6, degree=1, eps=0.1),      # sets that die
])
def test_chunks_whole_inputs_and_serial_fixups(kw):
    a = _nfa(**kw)
    assert device.symbol_lists(a) is not None
    lengths = np.r_[np.arange(0, 20), np.arange(250, 262), np.arange(508, 520),
                    np.random.default_rng(1).integers(600, 6000, 60)]
    inputs = _inputs(kw["seed"], kw.get("letters", 3), lengths)
    data, off = O.flatten(inputs)
    of, ol, oe, _ = O.nfa_batch(a, data, off)
    for chunk in (0, 256, None):
        eng = PersistentEngine([a], chunk_bytes=chunk)
        f, l, e, _, _ = eng.run_requests([0] * len(inputs), inputs, with_examined=True)
        assert np.array_equal(f, of) and np.array_equal(l, ol) and np.array_equal(e, oe), chunk


@pytest.mark.gpu
def test_pool_of_automata_with_and_without_lists():
    pool = [_nfa(64, 21, stay=True), W.random_nfa(1024, seed=0, degree=2, accept_prob=0.01),
            _nfa(40, 22), _nfa(40000, 23, letters=100)]
    assert device.symbol_lists(pool[3]) is None
    rng = np.random.default_rng(2)
    aut = rng.integers(0, len(pool), 160)
    inputs = [_inputs(i, 3 if a < 3 else 100, [int(rng.integers(0, 4000))])[0]
              for i, a in enumerate(aut)]
    eng = PersistentEngine(pool, chunk_bytes=256)
    f, l, _, _, _ = eng.run_requests(aut, inputs)
    want = [O.verdicts(pool[a], [x])[0] for a, x in zip(aut, inputs)]
    assert [(bool(x), int(y)) for x, y in zip(f, l)] == [(bool(x), int(y)) for x, y in want]
