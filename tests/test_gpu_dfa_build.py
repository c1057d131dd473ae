"""What building a DFA's device table takes and finds out (GPU)."""

from __future__ import annotations

import numpy as np
import pytest
import torch

from abstraction_regret_gb300 import native
from abstraction_regret_gb300.automata import DFA, random_dfa
from abstraction_regret_gb300.device import DeviceDFA

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("states", [32768, 50000])
def test_build_needs_little_beside_the_table(states):
    """The table and the caller's 4-byte entries, and at most a byte an entry more."""
    trans = np.random.default_rng(1).integers(0, states, states * 256, dtype=np.int32)
    dfa = DFA(num_states=states, start_state=0, accept=np.arange(states) < 3, trans=trans)
    DeviceDFA(random_dfa(64, accept_prob=0.0, seed=1))  # the library is loaded
    torch.cuda.synchronize()
    before = torch.cuda.memory_allocated()
    torch.cuda.reset_peak_memory_stats()
    dev = DeviceDFA(dfa)
    torch.cuda.synchronize()
    peak = torch.cuda.max_memory_allocated() - before
    assert peak <= dev.table_bytes + 5 * trans.size + (4 << 20)


@pytest.mark.parametrize("states,accepting,rare", [(50, 0, True), (4096, 1, False),
                                                   (32768, 0, True)])
def test_accept_share(states, accepting, rare):
    rng = np.random.default_rng(states)
    trans = rng.integers(accepting, states, states * 256, dtype=np.int32)
    trans[rng.permutation(trans.size)[:100 * accepting]] = 0  # 100 entries to accepting ones
    dfa = DFA(num_states=states, start_state=1, accept=np.arange(states) < accepting, trans=trans)
    dev = DeviceDFA(dfa)
    assert dev.accept_share == float((trans < accepting).sum()) / trans.size
    assert bool(dev.desc.flags & native.DFA_RARE_ACCEPT) == rare
