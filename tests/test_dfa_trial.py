"""Trials of how a DFA's set of all states shrinks (csrc/dfa_trial.cu), on the CPU, against
the set walk written out."""

from __future__ import annotations

import numpy as np
import pytest

from abstraction_regret_gb300 import device as D
from abstraction_regret_gb300 import engine as E
from abstraction_regret_gb300 import native
from abstraction_regret_gb300.automata import DFA, random_dfa


def _dfa(trans):
    n = trans.shape[0]
    return DFA(num_states=n, start_state=0, accept=np.zeros(n, bool),
               trans=trans.reshape(-1).astype(np.int32))


def _permuting(n, seed=1, alphabet=range(256)):
    """Bytes of the alphabet permute the states, the others lead to state 0."""
    rng = np.random.default_rng(seed)
    trans = np.zeros((n, 256), dtype=np.int32)
    for c in alphabet:
        trans[:, c] = rng.permutation(n)
    return _dfa(trans)


@pytest.mark.parametrize("states", [1, 2, 16, 17, 33, 300, 2500])
def test_trial_is_the_set_walk(states):
    dfa = random_dfa(states, accept_prob=0.0, seed=states)
    trans = dfa.trans.reshape(states, 256)
    for name, text in D._trial_texts().items():
        members, lookups, pos = np.arange(states), 0, 0
        while members.size > D.DFA_ENTRY_STATES:
            lookups += members.size
            members = np.unique(trans[members, text[pos]])
            pos += 1
        got = D.collapse_trial(dfa)[name]
        assert (got[0], got[2]) == (pos, lookups)


@pytest.mark.parametrize("states", [300, 4096, 32768])
def test_random_dfas_shrink_on_schedule(states):
    for t, x, _ in D.collapse_trial(random_dfa(states, accept_prob=0.0, seed=3)).values():
        assert states / 16 < t < states / 4 and 0.5 < x < 1.5


def test_permuted_states_never_shrink():
    trial = D.collapse_trial(_permuting(4096))
    # given up after the lookups allowed and at most one step more
    assert list(trial) == ["bytes"] and trial["bytes"][0] == -1
    assert trial["bytes"][1] <= D.COLLAPSE_SCHEDULES + 1
    digits = D.collapse_trial(_permuting(4096, alphabet=range(48, 58)))
    assert digits["bytes"][0] <= 3 and digits["lines"][0] <= 16 and digits["digits"][0] == -1


def test_a_set_that_stops_above_the_entry_states():
    trans = np.random.default_rng(4).integers(0, 17, size=(200, 256))
    for c in range(256):
        trans[:17, c] = np.random.default_rng(c).permutation(17)
    assert all(t == -1 for t, _, _ in D.collapse_trial(_dfa(trans)).values())
    trans = trans % 16
    for c in range(256):
        trans[:16, c] = np.random.default_rng(c).permutation(16)
    assert all(t == 1 for t, _, _ in D.collapse_trial(_dfa(trans)).values())


def test_bad_tables_are_refused():
    dfa = _permuting(20)
    dfa.trans[:] = 20
    with pytest.raises(ValueError):
        D.collapse_trial(dfa)
    lib, out, one = native.lib(), np.zeros(3, np.int64), np.ones(1, np.int32)
    text = np.zeros(16, np.uint8)
    for states, texts in ((0, 1), (20, 0), (20, 9)):
        assert lib.gbfsm_dfa_collapse_trial(
            states, dfa.trans.ctypes.data, text.ctypes.data, texts, 1, 16, one.ctypes.data,
            out.ctypes.data) == native.INVALID_ARG


def _lazy(n, share, seed=1):
    """Every byte permutes the states but for a share of them, which it sends anywhere: the
    set of all states shrinks more slowly than a random DFA's the smaller the share."""
    rng = np.random.default_rng(seed)
    trans = np.empty((n, 256), dtype=np.int32)
    for c in range(256):
        p = rng.permutation(n)
        anywhere = rng.random(n) < share
        p[anywhere] = rng.integers(0, n, int(anywhere.sum()))
        trans[:, c] = p
    return _dfa(trans)


@pytest.mark.parametrize("states,share,seed", [(4096, 1.0, 1), (16384, 1.0, 2), (16384, 0.3, 3),
                                               (4096, 0.15, 4), (2000, 0.0, 5)])
def test_shortest_chunk_holds_the_collapse(states, share, seed):
    """The shortest chunk is a random DFA's, or half as long again as the collapse where that
    takes longer, or the long length where the set does not shrink."""
    dfa = _lazy(states, share, seed)
    trial = D.collapse_trial(dfa)
    texts = [trial[k] for k in ("bytes", "lines") if k in trial]
    ends = all(t >= 0 for t, _, _ in texts)
    length, cost = E.dfa_chunk_plan(states, max(t for t, _, _ in texts) if ends else None,
                                    max(k for _, _, k in texts))
    assert length % 64 == 0 and 1.3 * cost >= max(k for _, _, k in texts)
    assert ends == (share > 0.1)
    if share == 1.0:
        assert length == E.dfa_chunk_length(states)
    elif ends:
        assert E.dfa_chunk_length(states) < length < 8 * states
        # the collapse of other texts ends within the chunk
        rng = np.random.default_rng(6)
        trans = dfa.trans.reshape(states, 256)
        for _ in range(4):
            members, pos = np.arange(states), 0
            while members.size > D.DFA_ENTRY_STATES:
                members = np.unique(trans[members, int(rng.integers(0, 256))])
                pos += 1
            assert pos < length
    else:
        assert length == max(16 << 10, 8 * states)


@pytest.mark.parametrize("states", [300, 1024, 16384])
def test_dfas_that_accept_often_get_long_chunks(states):
    """Where the inputs hardly ever reach a second chunk, none are cut that are shorter than
    two long ones."""
    args = (states, states // 8, 13 * states)
    for share in (0.0, 1e-5, 0.001):
        assert E.dfa_chunk_plan(*args, share)[0] == E.dfa_chunk_length(states)
    for share in (0.0015, 0.005, 0.5):
        length, cost = E.dfa_chunk_plan(*args, share)
        assert length == max(16 << 10, 8 * states)
        assert cost == E.dfa_chunk_plan(*args)[1]
