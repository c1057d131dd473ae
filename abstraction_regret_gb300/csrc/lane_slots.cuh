// One speculative chunk per lane over an automaton's slot table (slots.cu): the lane
// launch's path for automata that have one.
//
// A set of states is kept as the codes of its members in registers. While it holds one
// member -- nearly always: a speculative superset shrinks to the true set within a few
// bytes, and true sets of sparse automata hold one or two states -- a byte costs one slot
// lookup: position 2 * code + byte, hit when the slot's label is the byte, and the slot's
// code is the next state. Death, an accepting state and several successors all fail the
// one test `hit && code < accept_begin` and are handled out of line (about 1% of bytes), as
// is every byte while the set holds more than one member (the lane then carries the code
// multi_begin, whose lookups never hit, so the common path needs no size test).
// Sets that a single state steps to have codes of their own and count as one member here.
//
// What bounds it. With the table in shared memory, the bank conflicts of the lookups: 32
// lanes read 32 unrelated words, so a load takes about 3.5 passes where one would do, and
// the 3-byte form needs two loads. 16384 states, 65689 edges, 260.7 MB in chunks of 1728
// bytes (one per resident lane): 0.381 ms, against 1.85 ms with the label compares of
// lane_chunk() (165 warp instructions a byte, 22 of 32 lanes active, one dependent 16-byte
// gather a byte; here 18 and 30, LSU data pipe 69% busy, ncu). From global memory, the
// latency of the dependent load: 64 automata, 45 MB in chunks of 320 bytes 0.27 ms against
// 0.59 ms. On the way: handling sets out of line without codes of their own 0.72 ms;
// branching at every byte instead of every fourth 0.62 ms.
//
// Tables. WideSlots reads the 4-byte slots, from global memory through L1 or from a copy in
// shared memory; NarrowSlots reads 1-byte labels and 2-byte codes from shared memory (3
// bytes per edge), which holds automata of up to about 76000 edges.
#pragma once

#include <stddef.h>

#include "chunks.cuh"
#include "common.cuh"

namespace gbfsm {

constexpr int kSlotMembers = 8;  // members a lane holds
static_assert(kSlotMembers <= kEndCap, "a chunk's final set fits its record");
// the record is written as 16-byte groups: counts and accepts, then from dead_at on
static_assert(kCheckpoints == 6 && offsetof(ChunkRecord, dead_at) == 48 &&
                  offsetof(ChunkRecord, ov_counts) == 64 && offsetof(ChunkRecord, begin) == 88 &&
                  offsetof(ChunkRecord, end) == 96,
              "chunk record layout");

// An automaton's code ranges (slots.cu) and the records of its codes.
struct SlotCodes {
    uint32_t set_begin, accept_begin, multi_begin;
    const uint4 *__restrict__ recs;

    // The list of a code that may stand for several states: a list or a coded set.
    __device__ __forceinline__ uint32_t list_of(uint32_t code) const {
        if (code < set_begin || code > multi_begin) return code;
        const uint4 r = __ldg(recs + code);
        return (r.y & GBFSM_CODE_SET) ? r.x : code;
    }

    __device__ __forceinline__ int size_of(uint32_t code) const {
        if (code < set_begin) return 1;
        const uint4 r = __ldg(recs + code);
        return (r.y & GBFSM_CODE_SET) ? (int)r.z : 1;
    }
};

struct GlobalSlots {
    const uint32_t *__restrict__ slots;
    const uint32_t *__restrict__ pairs;
    __device__ __forceinline__ bool look(uint32_t code, uint32_t c, uint32_t &next) const {
        const uint32_t e = __ldg(slots + 2u * code + c);
        next = e >> 8;
        return (e & 0xffu) == c;
    }
    __device__ __forceinline__ uint2 pair(uint32_t i) const {
        return __ldg(reinterpret_cast<const uint2 *>(pairs) + i);
    }
};

// The same arrays in shared memory (byte addresses in the shared window).
struct WideSlots {
    uint32_t slots;
    uint32_t pairs;
    __device__ __forceinline__ bool look(uint32_t code, uint32_t c, uint32_t &next) const {
        uint32_t e;
        asm volatile("ld.shared.u32 %0, [%1];" : "=r"(e) : "r"(slots + 8u * code + 4u * c));
        next = e >> 8;
        return (e & 0xffu) == c;
    }
    __device__ __forceinline__ uint2 pair(uint32_t i) const {
        uint2 v;
        asm volatile("ld.shared.v2.u32 {%0, %1}, [%2];" : "=r"(v.x), "=r"(v.y) : "r"(pairs + 8u * i));
        return v;
    }
};

struct NarrowSlots {
    uint32_t labels;  // 1 byte per slot
    uint32_t codes;   // 2 bytes per slot
    uint32_t pairs;   // two 16-bit codes
    __device__ __forceinline__ bool look(uint32_t code, uint32_t c, uint32_t &next) const {
        const uint32_t p = 2u * code + c;
        uint32_t label;
        unsigned short n;
        asm volatile("ld.shared.u8 %0, [%1];" : "=r"(label) : "r"(labels + p));
        asm volatile("ld.shared.u16 %0, [%1];" : "=h"(n) : "r"(codes + 2u * p));
        next = n;
        return label == c;
    }
    __device__ __forceinline__ uint2 pair(uint32_t i) const {
        uint32_t v;
        asm volatile("ld.shared.u32 %0, [%1];" : "=r"(v) : "r"(pairs + 4u * i));
        return make_uint2(v & 0xffffu, v >> 16);
    }
};

// Adds a state's code to the distinct members set[0 .. m); m goes past kSlotMembers when
// there is no room.
__device__ __forceinline__ void slot_add(uint32_t *set, int &m, uint32_t code) {
    for (int q = 0; q < m && q < kSlotMembers; ++q)
        if (set[q] == code) return;
    if (m < kSlotMembers) set[m] = code;
    ++m;
}

// Adds the states that a slot's code stands for.
template <typename Table>
__device__ __forceinline__ void slot_add_code(const Table &T, const SlotCodes &K, uint32_t *set,
                                              int &m, uint32_t code) {
    code = K.list_of(code);
    while (code > K.multi_begin && m <= kSlotMembers) {
        const uint2 p = T.pair(code - K.multi_begin - 1u);
        slot_add(set, m, p.x);
        code = p.y;
    }
    if (code < K.multi_begin) slot_add(set, m, code);
}

// A running set. It is `one` code (a state or a coded set), or, when `one` is multi_begin
// (whose lookups never hit), the m states set[0 .. m).
struct SlotRun {
    uint32_t one;
    int m;
    uint32_t *set;  // kSlotMembers codes, in local memory
};

enum SlotEvent { kSlotAlive = 0, kSlotDead = 1, kSlotAccept = 2, kSlotFull = 3 };

// One byte from any set: {one, m, event} of the next (kSlotFull: more members than a lane
// holds; set[0 .. m) is then still the set before the byte when it was that). Out of line: a few bytes per chunk come here, and the loops that inline the
// common case stay small.
template <typename Table>
__device__ __noinline__ int3 slot_step_any(Table T, SlotCodes K, uint32_t one, int m,
                                           uint32_t *set, uint32_t c) {
    uint32_t next;
    if (one != K.multi_begin) {
        if (!T.look(one, c, next)) return make_int3((int)K.multi_begin, 0, kSlotDead);
        if (next < K.multi_begin)
            return make_int3((int)next, 1, next < K.accept_begin ? kSlotAlive : kSlotAccept);
        m = 0;
        slot_add_code(T, K, set, m, next);
    } else {
        uint32_t out[kSlotMembers];
        int n = 0;
        for (int q = 0; q < m; ++q)
            if (T.look(set[q], c, next)) slot_add_code(T, K, out, n, next);
        m = n;
        if (n <= kSlotMembers)
            for (int q = 0; q < n; ++q) set[q] = out[q];
    }
    if (m == 0) return make_int3((int)K.multi_begin, 0, kSlotDead);
    if (m > kSlotMembers) return make_int3((int)K.multi_begin, 0, kSlotFull);
    bool acc = false;
    for (int q = 0; q < m; ++q) acc = acc || set[q] >= K.accept_begin;
    return make_int3((int)(m == 1 ? set[0] : K.multi_begin), m, acc ? kSlotAccept : kSlotAlive);
}

template <typename Table>
__device__ __forceinline__ int slot_step(const Table &T, const SlotCodes &K, SlotRun &r,
                                         uint32_t c) {
    uint32_t next;
    if (T.look(r.one, c, next) && next < K.accept_begin) {
        r.one = next;
        return kSlotAlive;
    }
    const int3 v = slot_step_any(T, K, r.one, r.m, r.set, c);
    r.one = (uint32_t)v.x;
    r.m = v.y;
    return v.z;
}

// Four bytes at once, without a branch: a lookup that is not a hit on a plain code leads to
// multi_begin, which no later lookup leaves. Returns whether all four were plain; if not,
// the run is unchanged and the bytes are stepped one by one.
template <typename Table>
__device__ __forceinline__ bool slot_word(const Table &T, const SlotCodes &K, SlotRun &r,
                                          uint32_t w) {
    uint32_t s = r.one;
#pragma unroll
    for (int t = 0; t < 4; ++t) {
        const uint32_t c = (w >> (8 * t)) & 0xffu;
        uint32_t next;
        const bool hit = T.look(s, c, next);
        s = hit && next < K.accept_begin ? next : K.multi_begin;
    }
    if (s == K.multi_begin) return false;
    r.one = s;
    return true;
}

__device__ __forceinline__ int slot_size(const SlotCodes &K, const SlotRun &r) {
    return r.one == K.multi_begin ? r.m : K.size_of(r.one);
}

// Start set of a later chunk at b when the two-byte superset there holds more states than
// a lane: the two-byte superset at b - 2 (at most kWideStart members) stepped over x[b-2]
// and x[b-1], as widened_start does; false when either is too large.
template <typename Table>
__device__ __forceinline__ bool slot_widened_start(const gbfsm_nfa_dev &A, const Table &T,
                                                   const SlotCodes &K, const uint8_t *base,
                                                   int64_t b, uint32_t *set, int &m) {
    if (b < 4) return false;
    const uint32_t key = byte_at(base + b - 4) * 256u + byte_at(base + b - 3);
    const uint32_t pr = __ldg(A.pair_row + key);
    const uint32_t cnt = __ldg(A.pair_row + key + 1) - pr;
    if (cnt > kWideStart) return false;
    const uint32_t s1 = byte_at(base + b - 2), s2 = byte_at(base + b - 1);
    m = 0;
    for (uint32_t q = 0; q < cnt && m <= kSlotMembers; ++q) {
        uint32_t c1;
        if (!T.look(__ldg(A.pair_codes + pr + q), s1, c1)) continue;
        c1 = K.list_of(c1);
        for (;;) {  // every successor on s1, then its successors on s2
            uint32_t t = c1;
            bool more = false;
            if (c1 > K.multi_begin) {
                const uint2 p = T.pair(c1 - K.multi_begin - 1u);
                t = p.x;
                c1 = p.y;
                more = true;
            }
            uint32_t c2;
            if (T.look(t, s2, c2)) slot_add_code(T, K, set, m, c2);
            if (!more) break;
        }
    }
    return m <= kSlotMembers;
}

// lane_chunk() (chunks.cuh) over a slot table: the same record, false (nothing usable
// written) when the chunk outgrows the lane. `mask`: the lanes of the warp that call it;
// they meet again between its parts, so that a lane that took longer in one part does not
// run the next by itself.
template <typename Table>
__device__ __forceinline__ bool slot_chunk(const gbfsm_nfa_dev &A, const Table &T,
                                           const uint8_t *base, int64_t b, int64_t e,
                                           int64_t ov_end, int index, ChunkRecord *rec,
                                           uint32_t mask) {
    const SlotCodes K{A.set_code, A.accept_code, A.multi_code,
                      reinterpret_cast<const uint4 *>(A.code_recs)};
    uint32_t set[kSlotMembers];
    SlotRun run{K.multi_begin, 0, set};
    // counts[4..5] and every accept position; accepts are written over them as found
    int4 *out = reinterpret_cast<int4 *>(rec);
    out[1] = make_int4(0, 0, -1, -1);
    out[2] = make_int4(-1, -1, -1, -1);
    int32_t dead_at = -1;
    bool stopped = false, fits = true;
    if (index == 0) {
        set[0] = A.start_code;
        run.m = 1;
        if (A.start_code >= K.accept_begin) {
            rec->acc_after[0] = 0;
            stopped = true;
        }
    } else {
        const uint32_t key = byte_at(base + b - 2) * 256u + byte_at(base + b - 1);
        const uint32_t pr = __ldg(A.pair_row + key);
        const uint32_t cnt = __ldg(A.pair_row + key + 1) - pr;
        if (cnt <= (uint32_t)kSlotMembers) {
            for (uint32_t q = 0; q < cnt; ++q) set[q] = __ldg(A.pair_codes + pr + q);
            run.m = (int)cnt;
        } else {
            fits = slot_widened_start(A, T, K, base, b, set, run.m);
        }
        if (run.m == 0) dead_at = (int32_t)b;
        stopped = !fits || run.m == 0;
    }
    if (run.m == 1) run.one = set[0];
    const int32_t len = (int32_t)(e - b);
    const int32_t b32 = (int32_t)b;
    const uint8_t *p = base + b;
    int32_t j = 0;
    uint32_t sizes = 0;  // set sizes at the checkpoints, four bits each
    // the checkpoints that no accept lies after yet (a first chunk records its own first
    // accept only, in acc_after[0])
    uint32_t open_acc = index > 0 ? (1u << kCheckpoints) - 1u : 1u;
    // One byte. An accept closes the checkpoints it is the first one after; a death, a
    // first chunk's accept and one past the checkpoints end the run.
    auto byte = [&](uint32_t c) {
        const int ev = slot_step(T, K, run, c);
        ++j;
        if (ev == kSlotAlive) return;
        stopped = true;
        if (ev == kSlotFull) {
            fits = false;
        } else if (ev == kSlotDead) {  // reference.py:59-60
            dead_at = b32 + j;
        } else {
            for (int c2 = 0; c2 < kCheckpoints; ++c2)
                if (((open_acc >> c2) & 1u) && (index == 0 || j > (1 << c2))) {
                    rec->acc_after[c2] = b32 + j;
                    open_acc &= ~(1u << c2);
                }
            stopped = index == 0 || j > kOverlap;
        }
    };
    auto word = [&](uint32_t w) {
        if (slot_word(T, K, run, w)) {
            j += 4;
            return;
        }
        for (int t = 0; t < 4 && !stopped; ++t, w >>= 8) byte(w & 0xffu);
    };
    auto note_size = [&](uint32_t &to, int32_t at) {
        const int cp = checkpoint_of(at);
        if (cp >= 0 && !stopped) to |= (uint32_t)slot_size(K, run) << (4 * cp);
    };
    __syncwarp(mask);
    // The head: kOverlap bytes with their checkpoints, and on to a 16-byte block. The first
    // four bytes, where the set is still large, go one by one.
    const int32_t lead =
        min(len, kOverlap + (int32_t)((16u - ((uint32_t)reinterpret_cast<uint64_t>(p) & 15u)) &
                                      15u));
    if (!stopped && len > 0) {
        WordStream words;
        words.init(p, base + e);
        uint32_t w = words.next_word();
        for (int t = 0; t < 4 && j < lead && !stopped; ++t, w >>= 8) {
            byte(w & 0xffu);
            note_size(sizes, j);
        }
        while (!stopped && lead - j >= 4) {
            word(words.next_word());
            note_size(sizes, j);
        }
        if (!stopped && j < lead) {
            w = words.next_word();
            for (; j < lead && !stopped; w >>= 8) byte(w & 0xffu);
        }
    }
    __syncwarp(mask);
    out[0] = make_int4((int)(sizes & 15u), (int)((sizes >> 4) & 15u), (int)((sizes >> 8) & 15u),
                       (int)((sizes >> 12) & 15u));
    *reinterpret_cast<int2 *>(&rec->counts[4]) =
        make_int2((int)((sizes >> 16) & 15u), (int)(sizes >> 20));
    // whole blocks, one block ahead in flight
    if (!stopped && len - j >= 16) {
        uint4 ahead = ld_stream16(p + j);
        while (!stopped && len - j >= 16) {
            uint4 v = ahead;
            if (len - j >= 32) ahead = ld_stream16(p + j + 16);
#pragma unroll 1
            for (int i = 0; i < 4 && !stopped; ++i) {
                word(v.x);
                v.x = v.y;
                v.y = v.z;
                v.z = v.w;
            }
        }
    }
    __syncwarp(mask);
    if (!stopped && j < len) {
        WordStream words;
        words.init(p + j, base + e);
        while (!stopped && len - j >= 4) word(words.next_word());
        if (!stopped && j < len) {
            uint32_t w = words.next_word();
            for (; j < len && !stopped; w >>= 8) byte(w & 0xffu);
        }
    }
    __syncwarp(mask);
    int32_t end_count = -1, ov_len = 0, ov_event = 0;
    uint32_t ov_sizes = 0;
    if (!stopped) {
        end_count = run.m;
        if (run.one != K.multi_begin) {
            end_count = 0;
            slot_add_code(T, K, set, end_count, run.one);
        }
        for (int q = 0; q < end_count; ++q) rec->end_recs[q] = __ldg(K.recs + set[q]);
        // the overlap: its first event ends it, as does a set that outgrows the lane
        const int32_t ov = (int32_t)(ov_end - e);
        auto over = [&](uint32_t c) {
            const int ev = slot_step(T, K, run, c);
            stopped = ev != kSlotAlive;
            if (ev == kSlotFull) return;
            ++ov_len;
            if (stopped) ov_event = ev == kSlotDead ? -ov_len : ov_len;
        };
        if (ov > 0) {
            WordStream words;
            words.init(base + e, base + e + ov);
            while (!stopped && ov_len < ov) {
                uint32_t w = words.next_word();
                if (ov_len >= 4 && ov - ov_len >= 4 && slot_word(T, K, run, w)) {
                    ov_len += 4;
                    note_size(ov_sizes, ov_len);
                } else {
                    for (int t = 0; t < 4 && ov_len < ov && !stopped; ++t, w >>= 8) {
                        over(w & 0xffu);
                        note_size(ov_sizes, ov_len);
                    }
                }
            }
        }
    }
    out[3] = make_int4(dead_at, end_count, ov_len, ov_event);
    out[4] = make_int4((int)(ov_sizes & 15u), (int)((ov_sizes >> 4) & 15u),
                       (int)((ov_sizes >> 8) & 15u), (int)((ov_sizes >> 12) & 15u));
    out[5] = make_int4((int)((ov_sizes >> 16) & 15u), (int)(ov_sizes >> 20), (int)b32,
                       (int)(b >> 32));
    rec->end = e;
    return fits;
}

// One lane: a whole input from the start state. False (no verdict) when a set outgrows the
// lane: `at` is then the position before the byte that it does so on, and set[0 .. m) the set
// there (m <= kSlotMembers codes of states).
template <typename Table>
__device__ __forceinline__ bool slot_whole(const gbfsm_nfa_dev &A, const Table &T,
                                           const uint8_t *in, int64_t len, Verdict &v,
                                           int64_t &at, uint32_t *set, int &m) {
    const SlotCodes K{A.set_code, A.accept_code, A.multi_code,
                      reinterpret_cast<const uint4 *>(A.code_recs)};
    SlotRun run{A.start_code, 1, set};
    v = Verdict{0, 0, len};
    if (A.start_code >= K.accept_begin) {
        v = Verdict{1, 0, 0};
        return true;
    }
    if (len <= 0) return true;
    WordStream words;
    words.init(in, in + len);
    for (int64_t pos = 0; pos < len; pos += 4) {
        uint32_t w = words.next_word();
        if (len - pos >= 4 && slot_word(T, K, run, w)) continue;
        for (int t = 0; t < 4 && pos + t < len; ++t, w >>= 8) {
            const uint32_t one = run.one;
            m = run.m;
            const int ev = slot_step(T, K, run, w & 0xffu);
            if (ev == kSlotAlive) continue;
            if (ev == kSlotFull) {
                at = pos + t;
                if (one != K.multi_begin) {
                    m = 0;
                    slot_add_code(T, K, set, m, one);
                }
                return false;
            }
            const int64_t end = pos + t + 1;
            v = ev == kSlotAccept ? Verdict{1, (int32_t)end, end} : Verdict{0, 0, end};
            return true;
        }
    }
    return true;
}

}  // namespace gbfsm
