"""How much work symbol lists may be (device.symbol_lists, csrc/closures.cu), on the CPU."""

from __future__ import annotations

import time

import numpy as np
import pytest

import abstraction_regret_gb300 as G
from abstraction_regret_gb300 import device, native


def _chain(n, targets, seed=1, dense=0):
    """Epsilon edges from every state to the next (dense: among the first `dense` states), and
    an edge on a byte to each of `targets`."""
    src = np.arange(len(targets))
    sym = np.random.default_rng(seed).integers(97, 123, len(targets))
    if dense:
        es, et = np.repeat(np.arange(dense), dense), np.tile(np.arange(dense), dense)
    else:
        es, et = np.arange(n - 1), np.arange(1, n)
    return G.nfa_from_edges(n, 0, np.arange(n) == n - 1, src, sym, np.asarray(targets), es, et)


@pytest.mark.parametrize("states", [2000, 16000, 32768])
def test_a_long_chain_is_given_up_at_once(states):
    t0 = time.perf_counter()
    assert device.symbol_lists(_chain(states, np.arange(states))) is None
    assert time.perf_counter() - t0 < 1.0


def test_many_epsilon_edges_among_few_states_end_the_search():
    a = _chain(3000, np.arange(3000) % 2500, dense=2500)
    t0 = time.perf_counter()
    assert device.symbol_lists(a) is None
    assert time.perf_counter() - t0 < 2.0


@pytest.mark.parametrize("targets", [[31999], [31990, 31995, 5], [], [31000] * 200])
def test_closures_that_fit_are_found(targets):
    n = 32000
    a = _chain(n, targets)
    got = device.symbol_lists(a)
    pairs = sum(n - t for t in targets)
    if pairs > device.SYMBOL_LIST_LIMIT:
        assert got is None
        return
    row, p = got
    assert row[257] - row[256] == n  # the start's closure is the chain
    sym = np.asarray(a.sym_symbols)
    want = {(s << 0 | t << 15, int(sym[s])) for s, x in enumerate(targets) for t in range(x, n)}
    have = {(int(v) & 0x3FFFFFFF, c) for c in range(256) for v in p[row[c]:row[c + 1]]}
    assert have == want


def test_the_limit_is_exact():
    n, targets = 100, [90, 95, 99]
    pairs = sum(n - t for t in targets)
    a = _chain(n, targets)
    assert device.symbol_lists(a, limit=pairs) is not None
    assert device.symbol_lists(a, limit=pairs - 1) is None


def test_bad_arguments_are_refused():
    lib = native.lib()
    row, states, w = np.zeros(3, np.int64), np.zeros(9, np.int32), np.ones(2, np.int64)
    for erp, etg in (([0, 1, 2], [0, 2]), ([0, 2, 1], [0, 1]), ([1, 1, 1], [0])):
        erp, etg = np.array(erp, np.int32), np.array(etg, np.int32)
        assert lib.gbfsm_eps_closures(2, erp.ctypes.data, etg.ctypes.data, w.ctypes.data, 0, 7,
                                      row.ctypes.data, states.ctypes.data) == native.INVALID_ARG


def _looping(n, degree, loops, seed=1):
    """Random edges, one epsilon edge, and states that keep themselves active, entered with
    the start state."""
    rng = np.random.default_rng(seed)
    src, own = np.repeat(np.arange(n), degree), np.arange(n, n + loops)
    return G.nfa_from_edges(n + loops, 0, np.zeros(n + loops, bool), np.r_[src, own],
                            np.r_[rng.integers(0, 256, src.size), np.full(loops, G.ANY_SYMBOL)],
                            np.r_[rng.integers(0, n, src.size), own],
                            np.r_[1, np.zeros(loops, int)], np.r_[2, own])


@pytest.mark.parametrize("n,degree,loops,pays", [
    (18000, 4, 0, True),     # 281 pairs a byte
    (20000, 8, 0, False),    # 625, sets that die
    (20000, 8, 20, False),   # 646, 20 edges to step over
    (20000, 8, 80, True),    # 706, 80
    (4000, 63, 0, False),    # 984, sets that die
    (1000, 63, 40, True),    # 286
])
def test_long_lists_are_for_large_sets(n, degree, loops, pays):
    a = _looping(n, degree, loops)
    assert device.symbol_lists_pay(a, *device.symbol_lists(a)) == pays


@pytest.mark.parametrize("patterns", [20, 160, 200, 320])
def test_pattern_sets_step_by_their_lists(patterns):
    from abstraction_regret_gb300 import anml
    from abstraction_regret_gb300 import workloads as W

    a = anml.load_anml_string(W.anml_patterns(patterns, seed=patterns, min_len=8))
    assert device.symbol_lists_pay(a, *device.symbol_lists(a))


@pytest.mark.gpu
@pytest.mark.parametrize("degree,states", [(7, 32766), (16, 16000)])
def test_small_sets_on_long_lists_take_no_longer_than_member_by_member(degree, states,
                                                                       monkeypatch):
    """The engine's choice against the same step without lists, 64 inputs that keep one or two
    states active."""
    import torch

    from abstraction_regret_gb300 import workloads as W
    from abstraction_regret_gb300.engine import GraphRunner, PersistentEngine
    from oracle import oracle as O

    a = _looping(states, degree, 0)
    off = W.offsets_of(np.full(64, 16384, dtype=np.int64))
    data = W.walk_bytes(a, off, seed=2)
    want = O.nfa_batch(a, data, off)

    def best():
        r = GraphRunner(PersistentEngine([a]), np.zeros(64, np.int64), data, off,
                        with_examined=True)
        times = []
        for _ in range(6):
            t = [torch.cuda.Event(enable_timing=True) for _ in range(2)]
            t[0].record()
            r.kernel_only()
            t[1].record()
            t[1].synchronize()
            times.append(t[0].elapsed_time(t[1]))
        got = r.d_out.cpu().numpy()
        assert all(np.array_equal(got[k], want[k]) for k in range(3))
        return min(times)

    chosen = best()
    monkeypatch.setattr(device, "symbol_lists", lambda nfa: None)
    assert chosen <= 1.25 * best()
