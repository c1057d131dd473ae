"""Engines whose launches need different amounts of shared memory, used in turn (GPU): the
limit that a kernel is opted in to is the kernel's, not the layout's, so a smaller layout
must not lower it under a larger one that was sized before."""

from __future__ import annotations

import numpy as np
import pytest

from abstraction_regret_gb300 import workloads as W
from abstraction_regret_gb300.automata import random_dfa
from abstraction_regret_gb300.engine import PersistentEngine
from oracle import oracle as O

pytestmark = pytest.mark.gpu


def _check(automaton, inputs):
    eng = PersistentEngine([automaton])
    f, l, _, _, _ = eng.run_requests([0] * len(inputs), inputs)
    want = O.verdicts(automaton, inputs)
    assert [(bool(a), int(b)) for a, b in zip(f, l)] == [(bool(a), int(b)) for a, b in want]


def test_persistent_launches_of_two_sizes_in_turn():
    large = W.random_nfa(65536, seed=1, degree=2, accept_prob=0.01)  # 96 KiB a CTA
    small = W.random_nfa(32768, seed=2, degree=2, accept_prob=0.01)  # 64 KiB
    rng = np.random.default_rng(3)
    inputs = [rng.integers(0, 256, int(n), dtype=np.uint8).tobytes() for n in (0, 5, 700, 4000)]
    for a in (large, small, large):
        _check(a, inputs)


def test_dfa_collapses_of_two_sizes_in_turn():
    large = random_dfa(32768, accept_prob=0.0, seed=1)
    small = random_dfa(24000, accept_prob=0.0, seed=2)
    rng = np.random.default_rng(4)
    inputs = [rng.integers(0, 256, n, dtype=np.uint8).tobytes() for n in (40000, 17000)]
    for a in (large, small, large):
        _check(a, inputs)
