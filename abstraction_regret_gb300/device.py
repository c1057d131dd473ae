"""Device-resident automata: the engine's GPU layouts, built once per automaton.

The reference re-uploads the CSR and re-packs the accept words on every call
(src/gpufsm/backends/cuda/nfa.py:44-52 and :105-121, ``dev_copy`` in
native/include/common.cuh:150-159). Here an automaton is uploaded once, converted on the
device by the layout kernels of ``libgbfsm`` (which also validate every index), and kept
resident as PyTorch tensors for as long as its executor lives.

NFA layout (``gbfsm_nfa_dev``): uint32 row arrays, 16-byte edge records
``{target, symbol | accept/eps flags of target, target's edge-row begin, end}`` and the
packed accept words (pack_accept layout). DFA layout (``gbfsm_dfa_dev``): 2-byte entries
(up to 32768 states) or 4-byte entries holding the successor with ``accept[successor]``
in the top bit, plus packed accept bits.
"""

from __future__ import annotations

from functools import lru_cache

import numpy as np
import torch

from . import native
from .automata import ALPHABET, ANY_SYMBOL
from .packing import words_for


def _stream_handle(device: torch.device) -> int:
    return torch.cuda.current_stream(device).cuda_stream


def _padded(n_elems: int, elem_bytes: int, device, dtype=torch.uint8) -> torch.Tensor:
    """A zero-filled device buffer of at least ``n_elems * elem_bytes`` bytes, padded to 16."""
    nbytes = max(16, -(-(n_elems * elem_bytes) // 16) * 16)
    itemsize = torch.empty((), dtype=dtype).element_size()
    return torch.zeros(nbytes // itemsize, dtype=dtype, device=device)


def _records(recs: np.ndarray, device) -> torch.Tensor:
    """uint32[k, 4] records as a 16-byte-aligned device buffer (at least one record)."""
    buf = _padded(max(1, recs.shape[0]), 16, device)
    if recs.size:
        buf[: recs.nbytes].copy_(torch.from_numpy(np.ascontiguousarray(recs, dtype=np.uint32)
                                                  .view(np.uint8).ravel()))
    return buf


def _to_dev(a: np.ndarray, dtype, device) -> torch.Tensor:
    arr = np.ascontiguousarray(a, dtype=dtype)
    if arr.size == 0:
        arr = np.zeros(4, dtype=dtype)
    return torch.from_numpy(arr).to(device)


def resolve_device(device=None) -> torch.device:
    if not torch.cuda.is_available():
        raise RuntimeError("the CUDA backend needs a CUDA device (torch.cuda.is_available() is False)")
    if device is None:
        return torch.device("cuda", torch.cuda.current_device())
    d = torch.device(device)
    if d.type != "cuda":
        raise ValueError(f"device must be a CUDA device, got {d}")
    return torch.device("cuda", d.index if d.index is not None else torch.cuda.current_device())


SUPERSET_LIMIT = 1 << 25  # records; above this an automaton is not chunked speculatively


def first_lists(nfa, limit: int = SUPERSET_LIMIT):
    """Per byte c, the distinct targets of edges labelled c or ANY, as engine state records.

    Returns ``(row int32[257], records uint32[k, 4])`` or ``None`` when the lists would
    exceed ``limit`` records (many wildcard targets). After consuming byte c an NFA's
    active set is contained in the epsilon closure of these targets, whatever the set
    before it: the starting superset of a speculative chunk.
    """
    n = int(nfa.num_states)
    syms = np.asarray(nfa.sym_symbols, dtype=np.int64)
    tgts = np.asarray(nfa.sym_targets, dtype=np.int64)
    any_t = np.unique(tgts[syms == ANY_SYMBOL])
    plain = syms != ANY_SYMBOL
    if int(plain.sum()) + 256 * any_t.size > limit:
        return None
    keys = syms[plain] * n + tgts[plain]
    if any_t.size:
        keys = np.concatenate([keys, (np.arange(256)[:, None] * n + any_t[None, :]).ravel()])
    keys = np.unique(keys)
    c, t = keys // n, keys % n
    row = np.zeros(257, dtype=np.int64)
    np.cumsum(np.bincount(c, minlength=256), out=row[1:])
    srp = np.asarray(nfa.sym_row_ptr, dtype=np.int64)
    recs = np.stack([t, _info(nfa, t), srp[t], srp[t + 1]], axis=1).astype(np.uint32)
    return row.astype(np.int32), recs


PAIR_LIMIT = 1 << 24  # records; above this an automaton gets no two-byte superset table


def _info(nfa, t: np.ndarray) -> np.ndarray:
    acc = np.asarray(nfa.accept, dtype=bool)
    erp = np.asarray(nfa.eps_row_ptr, dtype=np.int64)
    return (acc[t].astype(np.int64) << 9) | ((erp[t + 1] > erp[t]).astype(np.int64) << 10)


def pair_lists(nfa, first, limit: int = PAIR_LIMIT):
    """Two-byte supersets for an automaton without epsilon edges.

    For bytes c1, c2: the distinct targets, reachable by a c2 (or ANY) edge, of the states
    in ``first`` for c1 -- i.e. every state the automaton can occupy after reading c1 c2,
    from any set. Returns ``(row int32[65537], records uint32[k, 4])`` or ``None`` (epsilon
    edges, no first lists, or more than ``limit`` records).
    """
    if first is None or int(np.asarray(nfa.eps_targets).size):
        return None
    row1, recs1 = first
    n = int(nfa.num_states)
    srp = np.asarray(nfa.sym_row_ptr, dtype=np.int64)
    syms = np.asarray(nfa.sym_symbols, dtype=np.int64)
    tgts = np.asarray(nfa.sym_targets, dtype=np.int64)
    states = recs1[:, 0].astype(np.int64)
    c1_of = np.repeat(np.arange(256, dtype=np.int64), np.diff(row1.astype(np.int64)))
    deg = srp[states + 1] - srp[states]
    total = int(deg.sum())
    if total > 4 * limit:
        return None
    offs = np.cumsum(deg) - deg
    edge = np.arange(total, dtype=np.int64) - np.repeat(offs, deg) + np.repeat(srp[states], deg)
    c1_e = np.repeat(c1_of, deg)
    e_sym, e_tgt = syms[edge], tgts[edge]
    plain = e_sym != ANY_SYMBOL
    keys = (c1_e[plain] * 256 + e_sym[plain]) * n + e_tgt[plain]
    if (~plain).any():
        c1_a, t_a = c1_e[~plain], e_tgt[~plain]
        if c1_a.size * 256 > 4 * limit:
            return None
        keys = np.concatenate([keys, ((c1_a[:, None] * 256 + np.arange(256)[None, :]) * n
                                      + t_a[:, None]).ravel()])
    keys = np.unique(keys)
    if keys.size > limit:
        return None
    pair, t = keys // n, keys % n
    row = np.zeros(65537, dtype=np.int64)
    np.cumsum(np.bincount(pair, minlength=65536), out=row[1:])
    recs = np.stack([t, _info(nfa, t), srp[t], srp[t + 1]], axis=1).astype(np.uint32)
    return row.astype(np.int32), recs


def lane_state_records(nfa):
    """Lane record (gbfsm_lane_rec) of every state, uint32[n, 4], and the packed symbols
    of its edges 8..15, uint32[n, 2]; None when the automaton has 2^25 states or more."""
    n = int(nfa.num_states)
    if n >= 1 << native.LANE_STATE_BITS:
        return None
    srp = np.asarray(nfa.sym_row_ptr, dtype=np.int64)
    syms = np.asarray(nfa.sym_symbols, dtype=np.int64)
    nnz = int(srp[-1])
    deg = srp[1:] - srp[:-1]
    src = np.repeat(np.arange(n, dtype=np.int64), deg)
    has_any = np.bincount(src[syms == ANY_SYMBOL], minlength=n)[:n] > 0
    slow = (deg > native.LANE_FAST_DEGREE) | has_any
    j = np.arange(native.LANE_FAST_DEGREE, dtype=np.int64)
    idx = np.minimum(srp[:-1, None] + j[None, :], max(nnz - 1, 0))
    lab = np.where(j[None, :] < deg[:, None], syms[idx] if nnz else 0, 0) & 0xFF
    words = [lab[:, 4 * k] | (lab[:, 4 * k + 1] << 8) | (lab[:, 4 * k + 2] << 16)
             | (lab[:, 4 * k + 3] << 24) for k in range(4)]
    lo, hi = words[0], words[1]
    ext = np.stack([np.where(slow, 0, words[2]), np.where(slow, 0, words[3])], axis=1)
    acc = np.asarray(nfa.accept, dtype=bool)
    x = (np.arange(n, dtype=np.int64) | (np.where(slow, 0, deg) << native.LANE_DEG_SHIFT)
         | (slow.astype(np.int64) << 30) | (acc.astype(np.int64) << 31))
    recs = np.stack([x, srp[:-1], np.where(slow, srp[1:], lo), np.where(slow, 0, hi)], axis=1)
    return recs.astype(np.uint32), ext.astype(np.uint32)


SYMBOL_LIST_LIMIT = 256 * 1024  # pairs; 1024 to a byte on average
SYMBOL_STATES = 1 << 15
# automata that lanes run (two-byte supersets this small, engine.LANE_PAIR_MEAN) need none
SYMBOL_PAIR_MEAN = 32.0
# A step by the lists costs their length, one member by member the active states' edges. Up to
# about SYMBOL_SHORT pairs a byte the lists are never slower; above, an edge to step over is
# worth SYMBOL_EDGE pairs. Chunks of 64 inputs of 16 KiB, lists / member by member: 20000
# states, 312 pairs a byte, one active state of 4 edges 0.89 / 0.88 ms; 328 pairs, 20 edges
# 0.94 / 1.1; 875 pairs, 7 edges 2.9 / 1.1; 940 pairs, 30 edges 3.0 / 1.8; 60 edges 3.0 / 3.0.
SYMBOL_SHORT = 300
SYMBOL_EDGE = 14


def _closures(nfa, weight: np.ndarray, limit: int):
    """``(row int64[n + 1], states int32[])``: the epsilon closures of the start state and of
    the states of positive ``weight`` that have epsilon edges; None when the sum of weight x
    closure size passes ``limit``."""
    n = int(nfa.num_states)
    erp, etg = (np.ascontiguousarray(x, dtype=np.int32) for x in (nfa.eps_row_ptr,
                                                                  nfa.eps_targets))
    weight = np.ascontiguousarray(weight, dtype=np.int64)
    row = np.zeros(n + 1, dtype=np.int64)
    states = np.empty(limit + n, dtype=np.int32)
    st = native.lib().gbfsm_eps_closures(
        n, erp.ctypes.data, etg.ctypes.data if etg.size else None, weight.ctypes.data,
        int(nfa.start_state), limit, row.ctypes.data, states.ctypes.data)
    if st == native.UNSUPPORTED:
        return None
    native.check(st, "gbfsm_eps_closures")
    return row, states


def symbol_lists(nfa, limit: int = SYMBOL_LIST_LIMIT):
    """``(row uint32[258], pairs uint32[k])``: for every byte, the (from, to) pairs of its
    edges, targets closed under epsilon edges (csrc/sym_device.cuh); list 256 is the start
    closure. None for automata of more than 32768 states or ``limit`` pairs."""
    n = int(nfa.num_states)
    if n > SYMBOL_STATES:
        return None
    srp = np.asarray(nfa.sym_row_ptr, dtype=np.int64)
    sym = np.asarray(nfa.sym_symbols, dtype=np.int64)
    to = np.asarray(nfa.sym_targets, dtype=np.int64)
    src = np.repeat(np.arange(n, dtype=np.int64), np.diff(srp))
    wild = sym == ANY_SYMBOL
    # pairs that a state's closure is multiplied by: one for an edge to it, 256 for a wildcard
    weight = np.bincount(to, np.where(wild, 256, 1), n).astype(np.int64)
    if int(weight.sum()) > limit:
        return None
    start = int(nfa.start_state)
    first = np.array([start], dtype=np.int64)
    if int(nfa.eps_row_ptr[-1]):  # edges to a state with epsilon edges lead to its closure
        has_eps = np.diff(np.asarray(nfa.eps_row_ptr, dtype=np.int64)) > 0
        found = _closures(nfa, weight, limit - int(weight[~has_eps].sum()))
        if found is None:
            return None
        row, states = found
        size = np.diff(row)
        if size[start]:
            first = states[row[start]:row[start + 1]].astype(np.int64)
        more = np.flatnonzero(has_eps[to])
        if more.size:  # (these edges alone: an automaton has few of them)
            one = ~has_eps[to]
            count = size[to[more]]
            at = np.repeat(row[to[more]] - np.cumsum(count) + count, count) + \
                np.arange(int(count.sum()))
            src = np.concatenate([src[one], np.repeat(src[more], count)])
            sym = np.concatenate([sym[one], np.repeat(sym[more], count)])
            to = np.concatenate([to[one], states[at].astype(np.int64)])
            wild = sym == ANY_SYMBOL
    c = np.concatenate([sym[~wild], np.repeat(np.arange(256), int(wild.sum()))])
    src = np.concatenate([src[~wild], np.tile(src[wild], 256)])
    to = np.concatenate([to[~wild], np.tile(to[wild], 256)])
    key = np.unique(np.concatenate([(c << 30) | (src << 15) | to, (256 << 30) | first]))
    row = np.searchsorted(key, np.arange(258, dtype=np.int64) << 30)
    acc = np.asarray(nfa.accept, dtype=bool)
    src, to = (key >> 15) & 0x7FFF, key & 0x7FFF
    pairs = src | (to << 15) | (acc[to].astype(np.int64) << 30)
    return row.astype(np.uint32), pairs.astype(np.uint32)


def symbol_lists_pay(nfa, row: np.ndarray, pairs: np.ndarray) -> bool:
    """Whether warps should step by the symbol lists: short lists, or sets whose members have
    many edges on trial texts (from all targets of a byte, as a chunk starts)."""
    if int(row[256]) <= 256 * SYMBOL_SHORT:
        return True
    degree = np.diff(np.asarray(nfa.sym_row_ptr, dtype=np.int64))
    enough = (int(row[256]) / 256 - SYMBOL_SHORT) / SYMBOL_EDGE + 12
    src, to = pairs & 0x7FFF, (pairs >> 15) & 0x7FFF
    start, steps = 8, 32  # bytes that a chunk's superset is given to shrink; bytes counted
    for name in ("bytes", "lines"):
        total, active = 0, None
        for i, c in enumerate(_trial_texts()[name][: start + steps].tolist()):
            a, b = int(row[c]), int(row[c + 1])
            hit = to[a:b] if active is None else to[a:b][active[src[a:b]]]
            active = np.zeros(degree.size, dtype=bool)
            active[hit] = True
            total += int(degree[active].sum()) if i >= start else 0
        if total > enough * steps:
            return True
    return False


def slot_table(nfa):
    """The slot table of an epsilon-free NFA (csrc/slots.cu): a dict of ``slots``, ``pairs``
    (uint32), ``state_code`` (uint32 [n]), ``sets`` (uint32 [k, 3]: code, list, size),
    ``set_code``, ``accept_code`` and ``multi_code``; None when the automaton's wildcard
    edges (256 entries each) make it far larger than its edges."""
    n = int(nfa.num_states)
    srp, tgt, sym = (np.ascontiguousarray(x, dtype=np.int32) for x in
                     (nfa.sym_row_ptr, nfa.sym_targets, nfa.sym_symbols))
    acc = np.ascontiguousarray(nfa.accept, dtype=np.uint8)
    nnz = int(srp[-1])
    cap = 4 * nnz + 4 * n + 4096
    cap_pairs = 4 * nnz + 1024
    slots = np.empty(cap, dtype=np.uint32)
    pairs = np.empty(2 * cap_pairs, dtype=np.uint32)
    codes = np.empty(n + 3 * (n // 4 + 64), dtype=np.uint32)
    info = np.zeros(8, dtype=np.int64)
    st = native.lib().gbfsm_slots_build(
        n, srp.ctypes.data, tgt.ctypes.data if nnz else None, sym.ctypes.data if nnz else None,
        acc.ctypes.data, cap, slots.ctypes.data, cap_pairs, pairs.ctypes.data, codes.size,
        codes.ctypes.data, info.ctypes.data)
    if st == native.UNSUPPORTED:
        return None
    native.check(st, "gbfsm_slots_build")
    n_slots, n_pairs, set_code, accept_code, multi_code, n_sets = (int(x) for x in info[:6])
    return {"slots": slots[:n_slots], "pairs": pairs[:2 * n_pairs], "state_code": codes[:n],
            "sets": codes[n:n + 3 * n_sets].reshape(n_sets, 3), "set_code": set_code,
            "accept_code": accept_code, "multi_code": multi_code}


def narrow_slots(table) -> np.ndarray | None:
    """A slot table's 3-byte form (uint8 bytes: labels, then 16-bit codes, then pairs, each
    padded to 16 bytes); None when a code needs more than 16 bits."""
    slots, pairs = table["slots"], table["pairs"]
    if table["multi_code"] + 1 + pairs.size // 2 > 1 << 16:
        return None
    parts = [(slots & 0xFF).astype(np.uint8), (slots >> 8).astype(np.uint16),
             pairs.astype(np.uint16)]
    return np.concatenate([np.concatenate([p.view(np.uint8),
                                           np.zeros(-p.nbytes % 16, np.uint8)]) for p in parts])


class DeviceNFA:
    """An NFA (ours or gpufsm's, duck-typed on the CSR fields) resident on a GPU."""

    def __init__(self, nfa, device=None) -> None:
        dev = resolve_device(device)
        lib = native.lib()
        n = int(nfa.num_states)
        if n < 1:
            raise ValueError("cannot simulate an NFA with zero states")
        start = int(nfa.start_state)
        if not 0 <= start < n:
            raise ValueError(f"start_state {start} out of range (0..{n - 1})")
        srp = np.asarray(nfa.sym_row_ptr)
        erp = np.asarray(nfa.eps_row_ptr)
        if srp.shape != (n + 1,) or erp.shape != (n + 1,):
            raise ValueError("row pointer arrays must have num_states + 1 entries")
        ssy = np.asarray(nfa.sym_symbols)
        nnz, nne = int(srp[-1]), int(erp[-1])
        if nnz != np.asarray(nfa.sym_targets).size or nne != np.asarray(nfa.eps_targets).size:
            raise ValueError("row pointers disagree with the edge array lengths")
        self.device = dev
        self.num_states = n
        self.start_state = start
        self.num_words = words_for(n)
        self.num_sym_edges = nnz
        self.num_eps_edges = nne
        self.has_eps = nne > 0
        self.uses_any = bool(np.any(ssy == ANY_SYMBOL)) if nnz else False
        with torch.cuda.device(dev):
            src = [_to_dev(nfa.sym_row_ptr, np.int32, dev), _to_dev(nfa.sym_targets, np.int32, dev),
                   _to_dev(nfa.sym_symbols, np.int32, dev), _to_dev(nfa.eps_row_ptr, np.int32, dev),
                   _to_dev(nfa.eps_targets, np.int32, dev), _to_dev(nfa.accept, np.uint8, dev)]
            self.sym_row = _padded(n + 1, 4, dev)
            self.eps_row = _padded(n + 1, 4, dev)
            self.sym_edges = _padded(max(nnz, 1), 16, dev)
            self.eps_edges = _padded(max(nne, 1), 16, dev)
            self.accept_words = _padded(self.num_words, 8, dev)
            err = torch.zeros(4, dtype=torch.int32, device=dev)
            status = lib.gbfsm_nfa_layout(
                n, src[0].data_ptr(), src[1].data_ptr(), src[2].data_ptr(), src[3].data_ptr(),
                src[4].data_ptr(), src[5].data_ptr(), nnz, nne, self.sym_row.data_ptr(),
                self.sym_edges.data_ptr(), self.eps_row.data_ptr(), self.eps_edges.data_ptr(),
                self.accept_words.data_ptr(), err.data_ptr(), _stream_handle(dev))
            native.check(status, "gbfsm_nfa_layout")
            code = int(err[0].item())  # synchronises: the layout is checked before any use
            if code:
                raise ValueError(f"invalid NFA: layout check failed with code {code} "
                                 f"(1 row pointers, 2 target, 3 symbol, 4 epsilon target)")
        d = native.NfaDev()
        d.num_states = n
        d.start_state = start
        d.num_words = self.num_words
        d.flags = (native.NFA_HAS_EPS if self.has_eps else 0) | (
            native.NFA_HAS_ANY if self.uses_any else 0)
        d.sym_row = self.sym_row.data_ptr()
        d.sym_edges = self.sym_edges.data_ptr()
        d.eps_row = self.eps_row.data_ptr()
        d.eps_edges = self.eps_edges.data_ptr()
        d.accept_words = self.accept_words.data_ptr()
        d.num_sym_edges = nnz
        d.num_eps_edges = nne
        lists = first_lists(nfa)
        self.speculative = lists is not None
        if lists is not None:
            row, recs = lists
            with torch.cuda.device(dev):
                self.first_row = torch.from_numpy(np.ascontiguousarray(row)).to(dev)
                self.first_edges = _padded(max(1, recs.shape[0]), 16, dev)
                if recs.size:
                    self.first_edges[: recs.nbytes].copy_(
                        torch.from_numpy(np.ascontiguousarray(recs).view(np.uint8).ravel()))
            d.first_row = self.first_row.data_ptr()
            d.first_edges = self.first_edges.data_ptr()
        pairs = pair_lists(nfa, lists)
        self.lanes = pairs is not None
        self.pair_sizes = np.diff(pairs[0]).astype(np.int32) if pairs is not None else None
        self.pair_mean = float(self.pair_sizes.mean()) if pairs is not None else float("inf")
        table = slot_table(nfa) if pairs is not None else None
        lane = lane_state_records(nfa) if pairs is not None and table is None else None
        self.stage, self.stage_bytes = native.LANE_STAGE_NONE, 0
        if lane is None and table is None:
            pairs = None
            self.lanes = False
            self.pair_sizes, self.pair_mean = None, float("inf")
        if pairs is not None:
            prow, precs = pairs
            with torch.cuda.device(dev):
                self.pair_row = torch.from_numpy(np.ascontiguousarray(prow)).to(dev)
                if table is not None:
                    self._upload_slots(d, table, precs[:, 0], srp, nfa, dev)
                else:
                    self._upload_lane_records(d, lane, precs[:, 0], ssy, nfa, dev)
            d.pair_row = self.pair_row.data_ptr()
        lists = symbol_lists(nfa) if self.pair_mean > SYMBOL_PAIR_MEAN else None
        if lists is not None and not symbol_lists_pay(nfa, *lists):
            lists = None
        self.sym_pairs = 0 if lists is None else int(lists[1].size)
        if lists is not None:
            with torch.cuda.device(dev):
                self.sym_list_row = torch.from_numpy(lists[0].view(np.int32)).to(dev)
                self.sym_lists = _padded(max(1, lists[1].size), 4, dev)
                if lists[1].size:
                    self.sym_lists[: lists[1].nbytes].copy_(
                        torch.from_numpy(lists[1].view(np.uint8)))
            d.sym_lists = self.sym_lists.data_ptr()
            d.sym_list_row = self.sym_list_row.data_ptr()
        self.desc = d

    def _upload_slots(self, d, table, pair_states, srp, nfa, dev) -> None:
        """The slot table, the codes of the two-byte supersets and the state record of
        every code; how the lane launch of a pool of this automaton alone may stage it."""
        code, multi = table["state_code"], table["multi_code"]
        n = self.num_states
        ids = np.arange(n, dtype=np.int64)
        row = np.asarray(srp, dtype=np.int64)
        recs = np.zeros((multi, 4), dtype=np.uint32)
        recs[code] = np.stack([ids, _info(nfa, ids), row[:-1], row[1:]], axis=1)
        sets = table["sets"]
        recs[sets[:, 0], 0] = sets[:, 1]
        recs[sets[:, 0], 1] = native.CODE_SET
        recs[sets[:, 0], 2] = sets[:, 2]

        def put(a):
            raw = np.ascontiguousarray(a).view(np.uint8).ravel()
            buf = _padded(max(1, raw.size), 1, dev)
            if raw.size:
                buf[: raw.size].copy_(torch.from_numpy(raw))
            return buf

        self.slots = put(table["slots"])
        self.slot_pairs = put(table["pairs"])
        self.pair_codes = put(code[pair_states.astype(np.int64)])
        self.code_recs = put(recs)
        narrow = narrow_slots(table)
        self.slot_narrow = put(narrow) if narrow is not None else None
        d.slots = self.slots.data_ptr()
        d.slot_pairs = self.slot_pairs.data_ptr()
        d.slot_narrow = self.slot_narrow.data_ptr() if narrow is not None else None
        self.pair_size = put(np.minimum(self.pair_sizes, 255).astype(np.uint8))
        d.pair_codes = self.pair_codes.data_ptr()
        d.pair_size = self.pair_size.data_ptr()
        d.code_recs = self.code_recs.data_ptr()
        d.num_slots = table["slots"].size
        d.num_pairs = table["pairs"].size // 2
        d.set_code, d.accept_code, d.multi_code = table["set_code"], table["accept_code"], multi
        d.start_code = int(code[self.start_state])
        limit = int(native.lib().gbfsm_lanes_stage_limit())
        wide = -(-table["slots"].nbytes // 16) * 16 + -(-table["pairs"].nbytes // 16) * 16
        if wide <= limit:
            self.stage, self.stage_bytes = native.LANE_STAGE_WIDE, wide
        elif narrow is not None and narrow.size <= limit:
            self.stage, self.stage_bytes = native.LANE_STAGE_NARROW, int(narrow.size)

    def _upload_lane_records(self, d, lane, pair_states, ssy, nfa, dev) -> None:
        """Lane records of every edge's target and of the two-byte supersets' states."""
        tg = np.asarray(nfa.sym_targets, dtype=np.int64)
        nnz = self.num_sym_edges
        self.edge_sym = _padded(max(1, nnz), 2, dev, torch.int16)
        if nnz:
            self.edge_sym[:nnz].copy_(torch.from_numpy(np.ascontiguousarray(ssy, dtype=np.int16)))
        lane_states, lane_ext = lane
        self.pair_lanes = _records(lane_states[pair_states.astype(np.int64)], dev)
        self.lane_edges = _records(lane_states[tg] if nnz else lane_states[:0], dev)
        self.lane_labels_ext = torch.from_numpy(
            np.ascontiguousarray(lane_ext).view(np.int32).ravel()).to(dev)
        d.edge_sym = self.edge_sym.data_ptr()
        d.pair_lanes = self.pair_lanes.data_ptr()
        d.lane_edges = self.lane_edges.data_ptr()
        d.lane_labels_ext = self.lane_labels_ext.data_ptr()

    @property
    def edge_bytes(self) -> int:
        """Bytes of the resident layout (rows + edge records + accept words)."""
        return (self.sym_row.numel() + self.eps_row.numel() + self.sym_edges.numel()
                + self.eps_edges.numel() + self.accept_words.numel())


# the chunked walks of a DFA follow its set of all states until it has this many members
DFA_ENTRY_STATES = 16  # kEntries (csrc/dfa_chunks.cuh)
# a set that has not shrunk so far after this many times a random DFA's lookups does not
COLLAPSE_SCHEDULES = 32
# how much slower than a random DFA's it may shrink for a plain launch to cut its inputs:
# 4096 inputs of 64 KiB on 4096 random states spend 3 of 7.4 ms on it, and whole take 12.6
SPLIT_SCHEDULES = 2


TRIAL_TEXTS = ("bytes", "lines", "digits")


@lru_cache(maxsize=1)
def _trial_texts() -> dict[str, np.ndarray]:
    """Texts on which a DFA's set of all states is tried: any bytes, lines of printable
    ones, and digits (a counter over digits leaves every other byte to a sink, so that on
    any other text its states fall together at once). Rows of one array."""
    # (SplitMix64 counters; numpy's own generator takes 8 ms to come up)
    z = np.arange(1, (3 << 15) // 8 + 1, dtype=np.uint64) * np.uint64(0x9E3779B97F4A7C15)
    z = (z ^ (z >> np.uint64(30))) * np.uint64(0xBF58476D1CE4E5B9)
    z = (z ^ (z >> np.uint64(27))) * np.uint64(0x94D049BB133111EB)
    out = (z ^ (z >> np.uint64(31))).view(np.uint8).reshape(3, -1).copy()
    line = np.concatenate([32 + np.arange(252) % 95, [10] * 4]).astype(np.uint8)
    out[1] = line[out[1]]
    out[2] = 48 + out[2] % 10
    return dict(zip(TRIAL_TEXTS, out))


def collapse_trial(dfa) -> dict[str, tuple[int, float, int]]:
    """For each trial text, the bytes after which ``dfa``'s set of all states has at most
    DFA_ENTRY_STATES members (-1: not within the text or COLLAPSE_SCHEDULES times the lookups
    that a random DFA's takes, SPLIT_SCHEDULES times for digits), the lookups as a multiple of
    a random DFA's, and the lookups. Up to the first text on which it has not."""
    trans = np.ascontiguousarray(dfa.trans, dtype=np.int32)
    texts = _trial_texts()
    schedules = np.array([SPLIT_SCHEDULES if name == "digits" else COLLAPSE_SCHEDULES
                          for name in TRIAL_TEXTS], dtype=np.int32)
    out = np.zeros((3, 3), dtype=np.int64)
    st = native.lib().gbfsm_dfa_collapse_trial(
        int(dfa.num_states), trans.ctypes.data, texts["bytes"].ctypes.data, len(TRIAL_TEXTS),
        texts["bytes"].size, DFA_ENTRY_STATES, schedules.ctypes.data, out.ctypes.data)
    native.check(st, "gbfsm_dfa_collapse_trial")
    found = {}
    for name, (end, lookups, random) in zip(TRIAL_TEXTS, out.tolist()):
        found[name] = (end, lookups / random, lookups)
        if end < 0:
            break
    return found


class DeviceDFA:
    """A DFA (ours or gpufsm's) resident on a GPU as a packed transition table."""

    def __init__(self, dfa, device=None, entry_bytes: int | None = None) -> None:
        dev = resolve_device(device)
        lib = native.lib()
        n = int(dfa.num_states)
        if n < 1:
            raise ValueError("cannot simulate a DFA with zero states")
        start = int(dfa.start_state)
        if not 0 <= start < n:
            raise ValueError(f"start_state {start} out of range (0..{n - 1})")
        trans = np.asarray(dfa.trans)
        if trans.size != n * ALPHABET:
            raise ValueError(f"trans must have num_states * 256 = {n * ALPHABET} entries")
        if entry_bytes is None:
            entry_bytes = 2 if n <= 32768 else 4
        self.device = dev
        self.num_states = n
        self.start_state = start
        self.entry_bytes = entry_bytes
        self.table_bytes = n * ALPHABET * entry_bytes
        with torch.cuda.device(dev):
            t_dev = _to_dev(trans, np.int32, dev)
            a_dev = _to_dev(dfa.accept, np.uint8, dev)
            self.table = _padded(n * ALPHABET, entry_bytes, dev)
            self.accept_bits = _padded(-(-n // 32), 4, dev)
            err = torch.zeros(4, dtype=torch.int32, device=dev)
            status = lib.gbfsm_dfa_layout(n, t_dev.data_ptr(), a_dev.data_ptr(), entry_bytes,
                                          self.table.data_ptr(), self.accept_bits.data_ptr(),
                                          err.data_ptr(), _stream_handle(dev))
            native.check(status, "gbfsm_dfa_layout")
            code = int(err[0].item())
            if code:
                raise ValueError(f"invalid DFA: a successor is outside [0, {n}) (code {code})")
            # the share of entries that lead to an accepting state (their top bits), for the
            # paths over 2-byte tables; counted a slice at a time, as a sum over booleans
            # takes 9 bytes an entry
            self.accept_share = None
            if entry_bytes == 2:
                top = self.table[: 2 * n * ALPHABET].view(torch.int16)
                accepting = sum((part < 0).sum() for part in top.split(1 << 20))
                self.accept_share = int(accepting.item()) / (n * ALPHABET)
        d = native.DfaDev()
        d.num_states = n
        d.start_state = start
        d.entry_bytes = entry_bytes
        rare = self.accept_share is not None and self.accept_share * 50000 <= 1.0
        d.flags = native.DFA_RARE_ACCEPT if rare else 0
        # how its set of all states shrinks, for the same paths. Digits decide about the plain
        # launch's cut alone: it gains a factor of two at most and has no longer chunks to
        # fall back on
        trial = collapse_trial(dfa) if entry_bytes == 2 else {}
        if len(trial) == 3 and all(t >= 0 and x <= SPLIT_SCHEDULES
                                   for t, x, _ in trial.values()):
            d.flags |= native.DFA_COLLAPSES
        texts = [trial[k] for k in ("bytes", "lines") if k in trial]
        # bytes and lookups of a chunk's collapse (no bytes: it does not end)
        self.collapse_bytes, self.collapse_lookups = None, max([k for _, _, k in texts] or [0])
        if texts and all(t >= 0 for t, _, _ in texts):
            self.collapse_bytes = max(t for t, _, _ in texts)
            d.collapse_lookups = max(1, self.collapse_lookups)
        d.table = self.table.data_ptr()
        d.accept_bits = self.accept_bits.data_ptr()
        d.table_bytes = self.table_bytes
        self.desc = d
