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
