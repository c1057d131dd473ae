// Chunked walks of long DFA inputs: one input's chunks run in parallel, with exact
// verdicts (dfa_chunks.cu, tasks GBFSM_TASK_DFA_CHUNK and GBFSM_TASK_DFA_FIXUP).
//
// A DFA walk is one dependent table lookup per byte, so a long input is a long chain. Cut
// it into chunks and follow every state a chunk might start in. For a random DFA the set
// of all n states shrinks like 2n/t after t bytes, so it is down to 16 members after about
// n/8 bytes, where it takes 2n bytes to reach a single one. So:
//
// 1. Collapse (a warp per chunk): from the chunk's start b the set of all states is walked
//    until it has at most kEntries members; its position p and the members, the chunk's
//    entry states, go to its record. The first chunk instead walks its first bytes exactly
//    from the start state: one entry state.
// 2. Walk (kEntries lanes per chunk, a lane per entry state): from p through the chunk and
//    on to the next chunk's p. Each lane records its state there and its first accept.
//    Lanes whose states have met read the same table entries, which costs nothing more.
// 3. Fix-up (a warp per input): the true state at the first chunk's p is known; it is one
//    of the entry states of its chunk, whose record gives the state at the next chunk's p,
//    and so on. The first accept on that path is the input's verdict.
//
// A chunk whose set does not shrink to kEntries members within its bytes and its budget of
// lookups has no entry states: the chunk before walks on through it (up to the automaton's
// dfa_overlap bytes past its own end). Where a walk ends before the next entry position, the
// fix-up walks the gap. The budget (collapse_budget) is what keeps a DFA whose states are
// permuted by every byte from spending n lookups a byte to its chunks' ends.
//
// Early stop: an accept of the first chunk, or one found by every lane of a chunk, is in
// the input's true walk whatever came before, so the input's verdict lies at or before it.
// The chunk lowers the input's latch to its index, and chunks of a higher index, polling
// the latch, stop (p = -2). The fix-up returns before it reads a stopped chunk.
//
// What bounds it. The walk: the latency of a dependent lookup through L2, 0.2 us a byte,
// along a chunk. The collapse: about 2n ln(n/8) lookups a chunk, gathers of one table
// column (2-byte entries 512 bytes apart) that the LSU takes one sector at a time. The
// planner's chunk length balances the two. 8 inputs of 2 MiB on 8192 states: 3.1 ms
// (collapse 1.5, walk 1.6, fix-up 0.06) against 29.7 ms when a chunk had to collapse to a
// single state before its walk counted; 24 inputs of 0.5..4 MB on 16384 states 8.8 against
// 71 ms; one of 1 MiB on 256 states 0.33 against 1.46 ms.
//
// Positions count the bytes consumed from the start of the input.
#pragma once

#include "common.cuh"
#include "dfa_device.cuh"
#include "nfa_device.cuh"

namespace gbfsm {

constexpr int kEntries = 16;  // entry states of a chunk: two chunks walk in a warp

// Record of a DFA chunk, in its GBFSM_CHUNK_RECORD_BYTES record slot.
struct DfaChunkRecord {
    int32_t p;      // entry position; -1: the set stayed larger, -2: stopped
    int32_t at;     // the same, but never -2 (the chunk before reads it while this one walks)
    int32_t count;  // entry states
    int32_t done;   // position the lanes walked to
    uint16_t entry[kEntries];
    uint16_t exit[kEntries];  // each lane's state at `done`, when it has not accepted
    int32_t acc[kEntries];    // first accept in (p, done], -1: none (first chunk: in [0, p] too)
};
static_assert(sizeof(DfaChunkRecord) <= GBFSM_CHUNK_RECORD_BYTES, "DFA chunk record slot");

__device__ __forceinline__ DfaChunkRecord *dfa_record(void *records, int32_t chunk) {
    return reinterpret_cast<DfaChunkRecord *>(static_cast<uint8_t *>(records) +
                                              (size_t)chunk * GBFSM_CHUNK_RECORD_BYTES);
}

__device__ __forceinline__ const DfaChunkRecord *dfa_record(const void *records,
                                                            int32_t chunk) {
    return dfa_record(const_cast<void *>(records), chunk);
}

template <typename Entry>
__device__ __forceinline__ uint32_t dfa_entry(const Entry *T, uint32_t s, uint32_t c) {
    return __ldg(T + (typename RowIndex<Entry>::type)s * (uint32_t)kAlphabet + c);
}

constexpr int kLatchPollBytes = 256;  // serial steps between two polls of the latch
constexpr int kLatchPollSets = 16;    // light bitmap steps between two polls
constexpr int kPollEveryStep = 512;   // set size above which every bitmap step polls
constexpr int kMeetBytes = 4;  // bytes between two removals of members that have met
constexpr int kListMembers = 1024;    // members from which a set is kept as a list

// (the latch lies in global memory, or in shared memory for a CTA's own input)
__device__ __forceinline__ int32_t read_latch(const int32_t *latch) {
    return *static_cast<const volatile int32_t *>(latch);
}

// True when a chunk of index below `index` has latched the input (latch may be NULL).
__device__ __forceinline__ bool latched_below(const int32_t *latch, int32_t index) {
    return latch && read_latch(latch) < index;
}

// The same for the whole warp (latch and index warp-uniform): lane 0 reads the latch and
// every lane gets its answer, so the warp leaves a collective walk together.
__device__ __forceinline__ bool warp_latched_below(const int32_t *latch, int32_t index) {
    if (!latch) return false;
    int32_t v = lane_id() == 0 ? read_latch(latch) : 0;
    v = __shfl_sync(GBFSM_FULL_MASK, v, 0);
    return v < index;
}

template <typename Entry>
struct GlobalEntries {
    const Entry *T;
    __device__ __forceinline__ uint32_t operator()(uint32_t s, uint32_t c) const {
        return dfa_entry(T, s, c);
    }
};

__device__ __forceinline__ int32_t warp_sum_i32(int32_t v) {
#pragma unroll
    for (int d = 16; d > 0; d >>= 1) v += __shfl_xor_sync(GBFSM_FULL_MASK, v, d);
    return v;
}

// Lookups that the collapse of a chunk of `len` bytes may take, `per_byte` of them for each
// byte: twice what a trial of the automaton took (where nothing is known, as if that had been
// twice a random DFA's), and a share of what the chunk's own walk costs, for texts on which the set
// shrinks later than on the trial's. One warp makes about 57 set lookups in the time of one
// step of a walk, and the whole device 30 lookups for every byte that 5000 warps walk.
__device__ __forceinline__ int32_t collapse_budget(const gbfsm_dfa_dev &d, int64_t len,
                                                    uint32_t per_byte) {
    const int64_t known = d.collapse_lookups ? (int64_t)d.collapse_lookups
                                             : 2 * collapse_schedule((uint32_t)d.num_states);
    return (int32_t)min(2 * known + (int64_t)per_byte * len, (int64_t)1 << 30);
}

// The whole warp: walk the set of all n states from position b over bytes [b, e) until it
// has at most `want` (<= 32) members. Returns that position (lane l < count holds a member
// in `member`), -1 when the set is still larger at e or after `budget` lookups (steps of at
// most 32 members cost no more than a walk's and are not counted), or -2 when a chunk below `index` has
// latched the input (latch may be NULL). bm0 / bm1: shared bitmaps of at least ceil(n / 32)
// words; list: 2 * kListMembers shared 16-bit words. The set is a bitmap while it is large,
// then a list (a step then costs a lookup, an atomic and a ballot per 32 members, whatever
// n; scanning the bitmap for 64 members of 8192 states took 10 times the instructions),
// then a member per lane.
template <typename Entry>
__device__ int64_t dfa_collapse(const Entry *T, uint32_t n, const uint8_t *base, int64_t b,
                                int64_t e, int want, uint32_t *bm0, uint32_t *bm1,
                                uint16_t *list, uint32_t &member, int32_t &count,
                                const int32_t *latch, int32_t index, int32_t budget) {
    constexpr uint32_t ACC = EntryTraits<Entry>::kAccept;
    const uint32_t lane = lane_id();
    const uint32_t nw = (n + 31u) >> 5;
    count = 0;
    member = 0;
    if (e <= b) return -1;
    if (warp_latched_below(latch, index)) return -2;
    int64_t pos = b;
    uint32_t polls = 0;
    ByteStream bytes;
    if (n <= 32u) {  // every state, one per lane
        count = (int32_t)n;
        member = lane < n ? lane : 0xffffffffu;
    } else {
        // first byte: the successors of every state
        for (uint32_t w = lane; w < nw; w += 32) bm1[w] = 0u;
        __syncwarp();
        {
            const uint32_t c = __ldg(base + b);
            for (uint32_t s0 = lane; s0 < n; s0 += 32 * 8) {  // eight lookups in flight
                uint32_t t[8];
#pragma unroll
                for (int u = 0; u < 8; ++u)
                    if (s0 + 32u * u < n) t[u] = dfa_entry(T, s0 + 32u * u, c) & ~ACC;
#pragma unroll
                for (int u = 0; u < 8; ++u)
                    if (s0 + 32u * u < n) atomicOr(bm1 + (t[u] >> 5), 1u << (t[u] & 31u));
            }
        }
        __syncwarp();
        pos = b + 1;
        budget -= (int32_t)n;
        uint32_t *cur = bm1, *nxt = bm0;
        for (uint32_t w = lane; w < nw; w += 32) count += __popc(cur[w]);
        count = warp_sum_i32(count);
        // many members: bitmaps
        while (count > kListMembers && pos < e) {
            if ((count > kPollEveryStep || (pos - b) % kLatchPollSets == 0) &&
                warp_latched_below(latch, index))
                return -2;
            if (budget < 0) return -1;
            budget -= count;
            const uint32_t c = __ldg(base + pos);
            for (uint32_t w = lane; w < nw; w += 32) nxt[w] = 0u;
            __syncwarp();
            for (uint32_t w = lane; w < nw; w += 32) {
                uint32_t bits = cur[w];
                while (bits) {  // up to four lookups in flight per lane
                    uint32_t s4[4];
                    int k = 0;
#pragma unroll
                    for (int u = 0; u < 4; ++u) {
                        if (bits) {
                            s4[u] = (w << 5) + (uint32_t)(__ffs(bits) - 1);
                            bits &= bits - 1u;
                            k = u + 1;
                        }
                    }
                    uint32_t t4[4];
#pragma unroll
                    for (int u = 0; u < 4; ++u)
                        if (u < k) t4[u] = dfa_entry(T, s4[u], c) & ~ACC;
#pragma unroll
                    for (int u = 0; u < 4; ++u)
                        if (u < k) atomicOr(nxt + (t4[u] >> 5), 1u << (t4[u] & 31u));
                }
            }
            __syncwarp();
            count = 0;
            for (uint32_t w = lane; w < nw; w += 32) count += __popc(nxt[w]);
            count = warp_sum_i32(count);
            uint32_t *tmp = cur;
            cur = nxt;
            nxt = tmp;
            ++pos;
        }
        if (count > kListMembers) return -1;
        // members to the list (bitmap bits in word order)
        uint16_t *from = list, *to = list + kListMembers;
        int32_t mine = 0;
        for (uint32_t w = lane; w < nw; w += 32) mine += __popc(cur[w]);
        int32_t before = mine;
#pragma unroll
        for (int d = 1; d < 32; d <<= 1) {
            const int32_t y = __shfl_up_sync(GBFSM_FULL_MASK, before, d);
            if ((int)lane >= d) before += y;
        }
        before -= mine;
        for (uint32_t w = lane; w < nw; w += 32) {
            uint32_t bits = cur[w];
            while (bits) {
                from[before++] = (uint16_t)((w << 5) + (uint32_t)(__ffs(bits) - 1));
                bits &= bits - 1u;
            }
            nxt[w] = 0u;  // the members seen in a step; all zero between steps
        }
        __syncwarp();
        bytes.init(base + pos, e - pos);
        while (count > 32 && pos < e) {
            if (++polls % 4 == 0 && warp_latched_below(latch, index)) return -2;
            if (budget < 0) return -1;
            // up to kMeetBytes bytes, then the members that met are dropped
            const int k = (int)min((int64_t)kMeetBytes, e - pos);
            budget -= count * k;
            uint32_t c[kMeetBytes];
#pragma unroll
            for (int j = 0; j < kMeetBytes; ++j) c[j] = j < k ? bytes.next() : 0u;
            int32_t n_to = 0;
            for (int32_t i0 = 0; i0 < count; i0 += 32 * 8) {  // eight lookups in flight
                uint32_t t[8];
#pragma unroll
                for (int u = 0; u < 8; ++u) {
                    const int32_t i = i0 + 32 * u + (int32_t)lane;
                    t[u] = i < count ? from[i] : 0xffffffffu;
                }
#pragma unroll
                for (int j = 0; j < kMeetBytes; ++j)
                    if (j < k)
#pragma unroll
                        for (int u = 0; u < 8; ++u)
                            if (t[u] != 0xffffffffu) t[u] = dfa_entry(T, t[u], c[j]) & ~ACC;
                uint32_t seen[8];
#pragma unroll
                for (int u = 0; u < 8; ++u)
                    seen[u] = t[u] != 0xffffffffu ? atomicOr(nxt + (t[u] >> 5), 1u << (t[u] & 31u))
                                                  : 0xffffffffu;
#pragma unroll
                for (int u = 0; u < 8; ++u) {
                    if (i0 + 32 * u >= count) break;
                    const bool fresh = !((seen[u] >> (t[u] & 31u)) & 1u);
                    const uint32_t ball = __ballot_sync(GBFSM_FULL_MASK, fresh);
                    if (fresh) to[n_to + __popc(ball & lanemask_lt())] = (uint16_t)t[u];
                    n_to += __popc(ball);
                }
            }
            __syncwarp();
            for (int32_t i = (int32_t)lane; i < n_to; i += 32) nxt[to[i] >> 5] = 0u;
            __syncwarp();
            uint16_t *tmp = from;
            from = to;
            to = tmp;
            count = n_to;
            pos += k;
        }
        if (count > 32) return -1;
        member = (int32_t)lane < count ? from[lane] : 0xffffffffu;
        __syncwarp();
    }
    // one member per lane (lanes without one hold 0xffffffff); of several that met, the
    // first lane's stays
    uint32_t alive = __ballot_sync(GBFSM_FULL_MASK, member != 0xffffffffu);
    if (pos == b) bytes.init(base + pos, e - pos);  // (every state had a lane from the start)
    while (__popc(alive) > want && pos < e) {
        if (++polls % 64 == 0 && warp_latched_below(latch, index)) return -2;
        const int k = (int)min((int64_t)kMeetBytes, e - pos);
        if ((alive >> lane) & 1u) {
#pragma unroll
            for (int j = 0; j < kMeetBytes; ++j)
                if (j < k) member = dfa_entry(T, member, bytes.next()) & ~ACC;
        } else {
            for (int j = 0; j < k; ++j) bytes.next();
            member = 0xffffffffu;
        }
        __syncwarp();
        const uint32_t same = __match_any_sync(GBFSM_FULL_MASK, member);
        alive = __ballot_sync(GBFSM_FULL_MASK, ((alive >> lane) & 1u) &&
                                                   (uint32_t)(__ffs(same) - 1) == lane);
        pos += k;
    }
    count = __popc(alive);
    if (count > want) return -1;
    // members to lanes 0 .. count - 1
    const uint32_t src = lane < (uint32_t)count ? select_bit(alive, lane) : 0u;
    member = __shfl_sync(GBFSM_FULL_MASK, member, src);
    return pos;
}

// Collapse of chunk `index` of an input, spanning positions [b, e) of `base` (the input's
// first byte): its entry position and states, to rec. per_byte: see collapse_budget.
template <typename Entry>
__device__ void dfa_chunk_collapse(const gbfsm_dfa_dev &d, const uint8_t *base, int64_t b,
                                   int64_t e, int index, uint32_t *bm0, uint32_t *bm1,
                                   uint16_t *list, DfaChunkRecord *rec, int32_t *latch,
                                   uint32_t per_byte) {
    const Entry *T = static_cast<const Entry *>(d.table);
    const uint32_t lane = lane_id();
    int64_t p;
    int32_t count = 1, acc = -1;
    uint32_t member = (uint32_t)d.start_state;
    if (index == 0) {
        // about as many steps as the other chunks' collapses take: an input that accepts
        // early is then latched before most of its chunks' work is done (and up to 4096 bytes
        // where accepts are not rare: an input that is not latched here has all its chunks
        // collapse; 300 inputs of up to 4 MiB, 0.5% of the entries accepting, 0.93 ms with
        // 1024 bytes and 0.74 with 4096)
        p = max((int64_t)1024, (int64_t)d.num_states / 4);
        if (!(d.flags & GBFSM_DFA_RARE_ACCEPT)) p = max(p, min((e - b) / 4, (int64_t)4096));
        p = min(e, p);
        if (lane == 0) {
            if ((__ldg(d.accept_bits + (member >> 5)) >> (member & 31u)) & 1u)
                acc = 0;
            else
                member = dfa_walk_span(GlobalEntries<Entry>{T}, EntryTraits<Entry>::kAccept,
                                       member, base, 0, (int32_t)p, acc);
            if (latch && acc >= 0) atomicMin(latch, 0);
        }
    } else {
        p = dfa_collapse<Entry>(T, (uint32_t)d.num_states, base, b, e, kEntries, bm0, bm1, list,
                                member, count, latch, index, collapse_budget(d, e - b, per_byte));
    }
    if (lane == 0) {
        rec->p = (int32_t)p;
        rec->at = p == -2 ? -1 : (int32_t)p;
        rec->count = p >= 0 ? count : 0;
        rec->done = p >= 0 ? (int32_t)p : 0;
    }
    if (lane < (uint32_t)kEntries) {
        rec->entry[lane] = rec->exit[lane] = (uint16_t)member;
        rec->acc[lane] = lane == 0 ? acc : -1;
    }
    __syncwarp();
}

// The whole warp, a chunk per half (kEntries lanes, one per entry state): walk the chunk of
// record `rec` from its entry position to `target`; valid = false: this half has none.
// latch: the input's latch word, or NULL. The halves stay in step, 256 bytes at a time, so
// that their loads are in flight together.
template <typename Entry>
__device__ __forceinline__ void dfa_chunk_walk(bool valid, const Entry *table,
                                               const uint8_t *base, int32_t target, int index,
                                               DfaChunkRecord *rec, int32_t *latch) {
    constexpr uint32_t ACC = EntryTraits<Entry>::kAccept;
    const GlobalEntries<Entry> look{table};
    const uint32_t lane = lane_id();
    const int g = (int)(lane % kEntries);
    const uint32_t half = ((1u << kEntries) - 1u) << (lane - (uint32_t)g);
    int count = 0;
    uint32_t s = 0;
    int32_t acc = -1, q = 0;
    if (valid) {
        count = rec->count;
        const int k = g < count ? g : 0;  // lanes past the entry states repeat the first's walk
        s = rec->entry[k];
        acc = rec->acc[k];
        q = rec->p;
    }
    bool stopped = false, all = false;
    for (;;) {
        all = (__ballot_sync(GBFSM_FULL_MASK, acc >= 0) & half) == half;
        bool more = valid && !all && !stopped && q < target;
        const bool below = more && latched_below(latch, index);
        const uint32_t stops = __ballot_sync(GBFSM_FULL_MASK, below);
        stopped = stopped || (stops & half) != 0u;
        more = more && !stopped;
        if (!__any_sync(GBFSM_FULL_MASK, more)) break;
        if (more) {
            const int32_t to = target - q > kLatchPollBytes ? q + kLatchPollBytes : target;
            if (acc < 0) s = dfa_walk_span(look, ACC, s, base, q, to, acc);
            q = to;
        }
        __syncwarp();
    }
    if (!valid) return;
    if (g < count) {
        rec->exit[g] = (uint16_t)s;
        rec->acc[g] = acc;
    }
    if (g == 0) {
        if (all && latch) atomicMin(latch, index);
        rec->done = q;
        if (stopped) rec->p = -2;  // the verdict lies in an earlier chunk
    }
}

// Where the walk of a chunk ending at e ends: at the next entry position of its input, or
// the input's end, but at most `overlap` bytes past e.
__device__ __forceinline__ int32_t dfa_walk_target(const gbfsm_chunk *chunks, int32_t n_chunks,
                                                   const void *records, int32_t chunk,
                                                   int64_t e, int64_t len, int32_t overlap) {
    const int64_t cap = min(len, e + (int64_t)max(overlap, 0));
    const int32_t input = chunks[chunk].input;
    for (int32_t j = chunk + 1; j < n_chunks; ++j) {
        if (chunks[j].input != input || chunks[j].index != chunks[j - 1].index + 1) break;
        const int32_t at = dfa_record(records, j)->at;
        if (at >= 0) return (int32_t)min(cap, (int64_t)at);
    }
    return (int32_t)cap;
}

// A DFA_FIXUP task (the whole warp): the verdict of an input from its chunks' records
// (chunks first .. first + count).
template <typename Entry>
__device__ Verdict dfa_fixup(const gbfsm_dfa_dev &d, const uint8_t *base, int64_t len,
                             const void *records, int32_t first, int32_t count) {
    const GlobalEntries<Entry> look{static_cast<const Entry *>(d.table)};
    constexpr uint32_t ACC = EntryTraits<Entry>::kAccept;
    const uint32_t lane = lane_id();
    uint32_t s = 0;
    int32_t pos = 0, acc = -1;
    bool known = false;
    // the records do not depend on the state, so the next ones load while one is looked up
    constexpr int kAhead = 8;
    for (int32_t k0 = 0; k0 < count; k0 += kAhead) {
        int32_t p[kAhead], n[kAhead], done[kAhead], a[kAhead];
        uint32_t entry[kAhead], exit[kAhead];
#pragma unroll
        for (int u = 0; u < kAhead; ++u) {
            p[u] = -1;
            if (k0 + u < count) {
                const DfaChunkRecord *r = dfa_record(records, first + k0 + u);
                p[u] = r->p;
                n[u] = r->count;
                done[u] = r->done;
                const uint32_t g = lane < (uint32_t)kEntries ? lane : 0u;
                entry[u] = r->entry[g];
                exit[u] = r->exit[g];
                a[u] = r->acc[g];
            }
        }
#pragma unroll
        for (int u = 0; u < kAhead; ++u) {
            if (p[u] < 0) continue;
            if (!known) {  // the first chunk's entry state is the true one
                known = true;
                s = __shfl_sync(GBFSM_FULL_MASK, entry[u], 0);
            } else if (pos < p[u]) {
                s = dfa_walk_span(look, ACC, s, base, pos, p[u], acc);  // every lane alike
                if (acc >= 0) return Verdict{1, acc, acc};
            } else if (pos > p[u]) {
                continue;
            }
            const uint32_t hit = __ballot_sync(
                GBFSM_FULL_MASK, (int32_t)lane < n[u] && lane < (uint32_t)kEntries && entry[u] == s);
            pos = p[u];
            if (hit == 0u) continue;
            const int src = __ffs(hit) - 1;
            const int32_t at = __shfl_sync(GBFSM_FULL_MASK, a[u], src);
            if (at >= 0) return Verdict{1, at, at};
            s = __shfl_sync(GBFSM_FULL_MASK, exit[u], src);
            pos = done[u];
        }
    }
    if (pos < len) {
        s = dfa_walk_span(look, ACC, s, base, pos, (int32_t)len, acc);
        if (acc >= 0) return Verdict{1, acc, acc};
    }
    return Verdict{0, 0, len};
}

}  // namespace gbfsm
