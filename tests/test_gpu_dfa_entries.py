"""Chunked DFA walks by entry states (csrc/dfa_chunks.cuh) against the oracle (GPU), where
the collapse changes form: DFAs of as many states as a chunk has entry states, a warp has
lanes or the member list has places, and one more; sets that stay too large; accepts so
frequent that some entry states' walks accept and others do not (a warp walks two chunks,
which stop at different bytes)."""

from __future__ import annotations

import numpy as np
import pytest

from abstraction_regret_gb300.automata import DFA, random_dfa
from abstraction_regret_gb300.engine import PersistentEngine
from oracle import oracle as O

pytestmark = pytest.mark.gpu


def _check(dfa, inputs, **kw):
    eng = PersistentEngine([dfa], **kw)
    f, l, e, _, _ = eng.run_requests([0] * len(inputs), inputs, with_examined=True)
    data, off = O.flatten(inputs)
    of, ol, oe = O.dfa_batch(dfa, data, off)
    assert np.array_equal(f, of) and np.array_equal(l, ol) and np.array_equal(e, oe)
    return of


@pytest.mark.parametrize("states", [1, 2, 16, 17, 32, 33, 1024, 1025, 1500, 4097])
@pytest.mark.parametrize("accept", [0.0, 0.0002, 0.002])
def test_random_dfas_of_every_form(states, accept):
    dfa = random_dfa(states, accept_prob=accept, seed=states)
    if accept and states > 16:  # at least one accepting state, never the start
        acc = dfa.accept.copy()
        acc[0], acc[-1] = False, True
        dfa = DFA(num_states=states, start_state=0, accept=acc, trans=dfa.trans)
    rng = np.random.default_rng(states)
    lengths = np.concatenate([rng.integers(0, 2048, 20), rng.integers(2048, 40000, 40),
                              [1023, 1024, 1025, 2047, 2048, 2049, 4095, 4096, 4097]])
    inputs = [rng.integers(0, 256, int(n), dtype=np.uint8).tobytes() for n in lengths]
    _check(dfa, inputs)


@pytest.mark.parametrize("group", [8, 16, 17, 40])
def test_sets_that_stop_shrinking(group):
    """States of a ``group`` are permuted by every byte: the set of all states shrinks to
    the group and no further (up to 16: entry states that never meet; above: no entry
    states, every chunk walked through by the first one)."""
    rng = np.random.default_rng(group)
    n = 200
    trans = rng.integers(0, group, size=(n, 256))
    for c in range(256):
        trans[:group, c] = rng.permutation(group)
    trans[0, 7] = n - 1  # a rare way to the accepting state
    accept = np.arange(n) == n - 1
    dfa = DFA(num_states=n, start_state=1, accept=accept, trans=trans.reshape(-1).astype(np.int32))
    inputs = []
    for k in range(12):
        x = rng.integers(8, 256, 9000 + 777 * k, dtype=np.uint8)
        if k % 3:
            x[rng.integers(0, x.size, k)] = 7
        inputs.append(x.tobytes())
    flags = _check(dfa, inputs)
    assert 0 < int(flags.sum()) < len(inputs)


def test_few_and_many_short_inputs():
    """DFA groups of one input and of several (more inputs than resident warps)."""
    dfa = random_dfa(300, accept_prob=0.004, seed=5)
    rng = np.random.default_rng(6)
    for n in (3, 6000):
        _check(dfa, [rng.integers(0, 256, int(k), dtype=np.uint8).tobytes()
                     for k in rng.integers(0, 400, n)])


def _plain(dfa, inputs):
    """One plain launch (the default technique) against the oracle, examined bytes too."""
    from abstraction_regret_gb300.executors import CudaDFAExecutor

    f, l, e, _, _ = CudaDFAExecutor(dfa).run_arrays(inputs, with_examined=True)
    data, off = O.flatten(inputs)
    of, ol, oe = O.dfa_batch(dfa, data, off)
    assert np.array_equal(f, of) and np.array_equal(l, ol) and np.array_equal(e, oe)
    return of


@pytest.mark.parametrize("states,n_inputs", [(500, 3), (500, 700), (1000, 1500), (1000, 4500),
                                             (600, 2500), (5000, 40)])
def test_plain_launch_cuts_inputs(states, n_inputs):
    """4, 2 or 1 warps per input by their number, and more inputs than one wave (no cut);
    lengths around one, two and eight chunks; an alarm byte at the cuts and elsewhere."""
    rng = np.random.default_rng(states + n_inputs)
    trans = rng.integers(0, states - 2, size=(states, 256), dtype=np.int32)
    trans[7, 255] = states - 2   # two steps to the accepting state: few entries lead there
    trans[:, 254] = 7
    trans[states - 2, 253] = states - 1
    accept = np.arange(states) == states - 1
    dfa = DFA(num_states=states, start_state=0, accept=accept, trans=trans.reshape(-1))
    chunk = max(256, 2 * states)
    lengths = np.r_[0, 1, 15, 16, chunk, 2 * chunk - 1, 2 * chunk, 2 * chunk + 1, 8 * chunk,
                    9 * chunk + 5, rng.integers(0, 5 * chunk, 60)]
    inputs = []
    for i in range(n_inputs):
        n = int(lengths[i % lengths.size]) if n_inputs < 3000 else int(rng.integers(0, 600))
        x = rng.integers(0, 250, n, dtype=np.uint8)
        if n > 8 and i % 2:
            prefix = min(1024, n // 16)
            at = [prefix, prefix + (n - prefix) // 2, int(rng.integers(0, n - 3)), n - 3]
            k = min(max(at[i // 2 % 4] - int(rng.integers(0, 4)), 0), n - 3)
            x[k:k + 3] = (254, 255, 253)
        inputs.append(x.tobytes())
    flags = _plain(dfa, inputs)
    if n_inputs > 10:  # (the first three are too short for the alarm)
        assert 0 < int(flags.sum()) < len(inputs)


@pytest.mark.parametrize("states", [500, 3000])
def test_plain_launch_of_a_dfa_that_accepts_at_once(states):
    """The start state accepts: an empty walk, whatever the length."""
    dfa = random_dfa(states, accept_prob=0.0, seed=states)
    acc = dfa.accept.copy()
    acc[0] = True
    dfa = DFA(num_states=states, start_state=0, accept=acc,
              trans=np.where(dfa.trans == 0, 1, dfa.trans).astype(np.int32))
    _plain(dfa, [bytes(n) for n in (0, 1, 100, 30000)])


@pytest.mark.parametrize("states", [64, 3000])
def test_every_alignment_and_tail(states):
    """Inputs of 0 to 70 bytes packed behind one another, so that a warp's lanes start at
    every offset of a 16-byte block and end at every other; one accept at a random byte."""
    rng = np.random.default_rng(states)
    trans = rng.integers(0, states - 1, size=(states, 256), dtype=np.int32)
    trans[:, 255] = states - 1
    dfa = DFA(num_states=states, start_state=0, accept=np.arange(states) == states - 1,
              trans=trans.reshape(-1))
    inputs = []
    for k in range(71 * 17):
        x = rng.integers(0, 255, k % 71, dtype=np.uint8)
        if x.size and k % 3 == 0:
            x[int(rng.integers(0, x.size))] = 255
        inputs.append(x.tobytes())
    flags = _plain(dfa, inputs)
    assert 0 < int(flags.sum()) < len(inputs)
    _check(dfa, inputs)


def _permuting(n, seed, alphabet):
    """Bytes of the alphabet permute the states, the others lead to state 0; state n - 1
    accepts and is entered from state 1 by byte 48 alone."""
    rng = np.random.default_rng(seed)
    trans = np.zeros((n, 256), dtype=np.int32)
    for c in alphabet:
        trans[:n - 1, c] = rng.permutation(n - 1)
    trans[1, 48] = n - 1
    return DFA(num_states=n, start_state=0, accept=np.arange(n) == n - 1,
               trans=trans.reshape(-1))


def _ms(call, repeats=3):
    import torch

    best = float("inf")
    for _ in range(1 + repeats):
        a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        a.record()
        call()
        b.record()
        b.synchronize()
        best = min(best, a.elapsed_time(b))
    return best


@pytest.mark.parametrize("alphabet", [range(256), range(48, 58)])
def test_plain_launch_of_permuted_states(alphabet):
    """A cut would follow all states through every chunk: the launch takes no longer than
    the serial walk of its longest input (under 0.3 us a byte) allows."""
    import torch

    from abstraction_regret_gb300.executors import CudaDFAExecutor

    dfa = _permuting(4096, 7, alphabet)
    rng = np.random.default_rng(8)
    inputs = [rng.integers(48, 58, n, dtype=np.uint8).tobytes()
              for n in [16384] * 60 + [0, 100, 5000, 9999]]
    _plain(dfa, inputs)
    ex = CudaDFAExecutor(dfa)
    data, off = O.flatten(inputs)
    d = torch.from_numpy(np.concatenate([data, np.zeros(16, np.uint8)])).cuda()
    o = torch.from_numpy(off).cuda()
    out = torch.zeros((3, len(inputs)), dtype=torch.int32, device="cuda")
    ms = _ms(lambda: ex.launch(d, o, len(inputs), out[0], out[1], out[2]))
    assert ms < 16384 * 0.3e-3 * 2


@pytest.mark.parametrize("alphabet", [range(256), range(48, 58)])
def test_chunks_of_permuted_states(alphabet):
    """Chunks give up on a set that does not shrink: verdicts are exact and the step takes no
    longer than the serial walk of its longest input allows."""
    from abstraction_regret_gb300.engine import GraphRunner

    dfa = _permuting(4096, 9, alphabet)
    rng = np.random.default_rng(10)
    inputs = [rng.integers(48, 58, n, dtype=np.uint8).tobytes()
              for n in [16384] * 60 + [0, 100, 5000, 9999]]
    _check(dfa, inputs, dfa_chunk_bytes=4096)
    eng = PersistentEngine([dfa], dfa_chunk_bytes=4096)
    data, off = O.flatten(inputs)
    runner = GraphRunner(eng, [0] * len(inputs), data, off)
    assert _ms(runner.kernel_only) < 16384 * 0.3e-3 * 2


def test_inputs_of_permuted_states_run_whole():
    """Inputs shorter than two long chunks are not cut: the step takes no longer than the
    serial walk of its longest input allows."""
    from abstraction_regret_gb300.engine import GraphRunner

    dfa = _permuting(4096, 11, range(256))
    rng = np.random.default_rng(12)
    inputs = [rng.integers(0, 256, n, dtype=np.uint8).tobytes()
              for n in [16384] * 60 + [0, 100, 5000, 9999]]
    _check(dfa, inputs)
    data, off = O.flatten(inputs)
    runner = GraphRunner(PersistentEngine([dfa]), [0] * len(inputs), data, off)
    assert _ms(runner.kernel_only) < 16384 * 0.3e-3 * 2


@pytest.mark.parametrize("states,share", [(8192, 0.15), (16384, 0.3), (16384, 1.0)])
def test_slow_collapses_end_in_their_chunks(states, share):
    """Bytes permute all states but a share, which they send anywhere: chunks are long enough
    for the set to shrink, so nearly all of them have entry states."""
    from abstraction_regret_gb300 import native

    rng = np.random.default_rng(states)
    trans = np.empty((states, 256), dtype=np.int32)
    for c in range(256):
        p = rng.permutation(states)
        anywhere = rng.random(states) < share
        p[anywhere] = rng.integers(0, states, int(anywhere.sum()))
        trans[:, c] = p
    dfa = DFA(num_states=states, start_state=0, accept=np.zeros(states, bool),
              trans=trans.reshape(-1))
    eng = PersistentEngine([dfa])
    inputs = [rng.integers(0, 256, n, dtype=np.uint8).tobytes() for n in (1 << 20, 300_000)]
    f, l, e, _, _ = eng.run_requests([0, 0], inputs, with_examined=True)
    assert not f.any() and e.tolist() == [len(x) for x in inputs]
    n = int(eng._dplan.h_header.numpy()[native.PLAN_CHUNKS])
    p = eng._dplan.records[: n * native.CHUNK_RECORD_BYTES].cpu().numpy().view(np.int32) \
        .reshape(n, -1)[:, 0]
    assert n >= 8 and (p >= 0).mean() > 0.95


def test_texts_that_the_trial_did_not_foresee():
    """Bytes 0 and 1 permute the states and every other byte leads to state 0, so the set falls
    together on every trial text but never on these inputs: collapses run out of budget, the
    plain launch's (which cuts the inputs) and the engine's."""
    import torch

    from abstraction_regret_gb300 import native
    from abstraction_regret_gb300.engine import GraphRunner
    from abstraction_regret_gb300.executors import CudaDFAExecutor

    dfa = _permuting(4096, 13, (0, 1))
    rng = np.random.default_rng(14)
    inputs = []
    for k in range(64):
        x = rng.integers(0, 2, (16384, 16384, 16383, 9000)[k % 4], dtype=np.uint8)
        if k % 3 == 0:
            x[int(rng.integers(0, x.size))] = 48
        inputs.append(x.tobytes())
    _plain(dfa, inputs)
    _check(dfa, inputs)
    ex = CudaDFAExecutor(dfa)
    assert ex.dev.desc.flags == native.DFA_RARE_ACCEPT | native.DFA_COLLAPSES
    data, off = O.flatten(inputs)
    d = torch.from_numpy(np.concatenate([data, np.zeros(16, np.uint8)])).cuda()
    o = torch.from_numpy(off).cuda()
    out = torch.zeros((3, len(inputs)), dtype=torch.int32, device="cuda")
    assert _ms(lambda: ex.launch(d, o, len(inputs), out[0], out[1], out[2])) < 16384 * 0.3e-3 * 2
    runner = GraphRunner(PersistentEngine([dfa]), [0] * len(inputs), data, off)
    assert _ms(runner.kernel_only) < 16384 * 0.3e-3 * 2
