"""Plain compact launches whose sets outgrow a lane in the middle of an input (GPU): the warp
goes on from the byte on which they do (csrc/nfa_kernels.cu), with the verdicts and examined
bytes of the oracle."""

from __future__ import annotations

import numpy as np
import pytest
import torch

from abstraction_regret_gb300 import native
from abstraction_regret_gb300 import workloads as W
from abstraction_regret_gb300.automata import ANY_SYMBOL, nfa_from_edges
from abstraction_regret_gb300.executors import CudaNFAExecutor
from oracle import oracle as O

pytestmark = pytest.mark.gpu

STATES = 300


def _fan(fan: int, stay: bool, seed: int = 1):
    """A random NFA on bytes below 250; byte 255 leads every state to `fan` states, which stay
    active on the bytes below 250 ("any": on every byte, by one wildcard edge; or die), and
    byte 254 from one of those to an accepting one. Returns it and the NFA without the fan,
    whose walks keep one state active."""
    rng = np.random.default_rng(seed)
    src = np.repeat(np.arange(STATES), 3)
    sym, dst = rng.integers(0, 250, src.size), rng.integers(0, STATES, src.size)
    plain = nfa_from_edges(STATES, 0, np.zeros(STATES, bool), src, sym, dst)
    f = np.arange(STATES, STATES + fan)
    last = STATES + fan
    own = np.array([ANY_SYMBOL]) if stay == "any" else np.arange(250 if stay else 0)
    loops = np.repeat(f, own.size)
    a = nfa_from_edges(
        last + 1, 0, np.arange(last + 1) == last,
        np.concatenate([src, np.repeat(np.arange(STATES), fan), loops, [f[-1]]]),
        np.concatenate([sym, np.full(STATES * fan, 255), np.tile(own, fan), [254]]),
        np.concatenate([dst, np.tile(f, STATES), loops, [last]]))
    return a, plain


def _inputs(plain, lengths, fans, accepts, seed=3):
    """Walks of the plain automaton with byte 255 at `fans` and byte 254 at `accepts` (-1:
    none)."""
    off = W.offsets_of(np.asarray(lengths, dtype=np.int64))
    data = W.walk_bytes(plain, off, seed=seed).copy()
    for at, byte in ((fans, 255), (accepts, 254)):
        for i, p in enumerate(at):
            if 0 <= p < lengths[i]:
                data[off[i] + p] = byte
    return data, off


@pytest.mark.parametrize("fan", [8, 9, 40])
@pytest.mark.parametrize("stay", [True, "any", False])
@pytest.mark.parametrize("stage", [0, 1])
def test_verdicts_of_inputs_that_fall_back(fan, stay, stage):
    a, plain = _fan(fan, stay)
    lengths, fans, accepts = [], [], []
    for n in (1, 2, 7, 40, 333):
        for at in (0, 1, 3, 4, 5, 15, 16, 17, n - 2, n - 1, -1):
            for accept in (-1, at + 1, at + 9):
                lengths.append(n)
                fans.append(at)
                accepts.append(accept if at >= 0 else -1)
    data, off = _inputs(plain, lengths, fans, accepts)
    of, ol, oe, _ = O.nfa_batch(a, data, off)
    ex = CudaNFAExecutor(a, plan=native.make_plan(native.TECH_COMPACT, stage=stage))
    assert ex.dev.desc.slots
    inputs = [data[off[i]:off[i + 1]].tobytes() for i in range(len(lengths))]
    f, l, e, _, _ = ex.run_arrays(inputs, with_examined=True)
    assert np.array_equal(f, of) and np.array_equal(l, ol) and np.array_equal(e, oe)
    assert 0 < int(f.sum()) < len(inputs)


def _ms(ex, data, off):
    n = off.size - 1
    d = torch.from_numpy(np.concatenate([data, np.zeros(16, np.uint8)])).cuda()
    o = torch.from_numpy(off).cuda()
    out = torch.zeros((3, n), dtype=torch.int32, device="cuda")
    best = float("inf")
    for _ in range(4):
        t = [torch.cuda.Event(enable_timing=True) for _ in range(2)]
        t[0].record()
        ex.launch(d, o, n, out[0], out[1], out[2])
        t[1].record()
        t[1].synchronize()
        best = min(best, t[0].elapsed_time(t[1]))
    return best


@pytest.mark.parametrize("stage", [0, 1])
def test_a_late_fall_back_costs_the_bytes_that_are_left(stage):
    """One input whose set outgrows the lane near its end, against one that leaves it at once:
    the bytes before are the lane's alone, a tenth of the warp's time."""
    a, plain = _fan(12, "any")
    n = 16384
    ex = CudaNFAExecutor(a, plan=native.make_plan(native.TECH_COMPACT, stage=stage))
    late = _ms(ex, *_inputs(plain, [n], [n - 64], [-1]))
    at_once = _ms(ex, *_inputs(plain, [n], [5], [-1]))
    assert late < 0.25 * at_once
