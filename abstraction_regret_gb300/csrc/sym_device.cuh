// Warp simulation of an NFA by symbol lists: for every byte, the pairs (from, to) of all its
// edges on that byte (wildcards included, targets closed under epsilon edges). A step reads
// the byte's list, 32 pairs at a time, and for every pair whose source is in the set puts
// the target in the next set; both sets are bitmaps in shared memory. Its cost is the
// length of the list, however many states are active, and the lists do not depend on the
// set, so the next byte's pairs are loaded while this byte's are tested.
//
// It serves the automata that lanes cannot run -- epsilon edges, or so many wildcards that
// the sets stay large: patterns loaded from ANML hold one state active for good and others
// (`[...]+` loops) for long, about 100 of 1400, and the member-by-member steps of WarpNfa
// took 12-20 us a byte on them (chunks of 64 documents of 4..32 KiB: 4.5 ms, 0.33 ms by the
// lists). The bound here is the latency of a step: bitmap tests, one shared atomic, a warp
// reduction and the clearing of the old set.
//
// The same interface as WarpNfa (nfa_device.cuh), for the chunk runners of chunks.cuh.
#pragma once

#include "common.cuh"
#include "nfa_device.cuh"

namespace gbfsm {

constexpr uint32_t kSymStateBits = 15;  // a pair: from | to << 15 | accept(to) << 30
constexpr uint32_t kSymStateMask = (1u << kSymStateBits) - 1u;
constexpr uint32_t kSymAccept = 1u << 30;
constexpr int kSymAhead = 8;  // pairs per lane loaded a byte ahead

// Whether the lists can be used with this scratch: the second bitmap lies in the member
// lists' space.
__device__ __forceinline__ bool sym_usable(const gbfsm_nfa_dev &A, int list_capacity) {
    return A.sym_lists != nullptr && A.num_states <= (int32_t)kSymStateMask + 1 &&
           A.num_words * 8 <= 32 * max(list_capacity, 32);
}

// A byte stream with the two bytes after the current one (-1 past the end).
struct BytesAhead {
    ByteStream bytes;
    int64_t left;  // bytes not yet taken from the stream
    int next, next2;

    __device__ __forceinline__ int take() { return left > 0 ? (--left, (int)bytes.next()) : -1; }

    __device__ __forceinline__ void init(const uint8_t *in, int64_t len) {
        bytes.init(in, len);
        left = len;
        next = take();
        next2 = take();
    }

    __device__ __forceinline__ int advance() {
        const int now = next;
        next = next2;
        next2 = take();
        return now;
    }
};

struct SymNfa {
    const gbfsm_nfa_dev &A;
    uint32_t *cur;  // the set; the other bitmap is all zero between steps
    uint32_t *nxt;
    int words;      // 32-bit words of a bitmap
    // two bytes in the pipeline: the pairs of the byte `sym1` and the list bounds of `sym2`
    uint32_t ahead[kSymAhead];
    uint32_t row1, end1, row2, end2;
    int sym1, sym2;  // -1: nothing loaded

    __device__ __forceinline__ SymNfa(const gbfsm_nfa_dev &a, const Rows &, const WarpScratch &S)
        : A(a), cur(reinterpret_cast<uint32_t *>(S.V)), nxt(reinterpret_cast<uint32_t *>(S.LA)),
          words(2 * a.num_words), row1(0), end1(0), row2(0), end2(0), sym1(-1), sym2(-1) {
        for (int w = (int)lane_id(); w < words; w += 32) nxt[w] = 0u;
        __syncwarp();
    }

    __device__ __forceinline__ void load_bounds(int sym) {
        sym2 = sym;
        if (sym < 0) return;
        row2 = __ldg(A.sym_list_row + sym);
        end2 = __ldg(A.sym_list_row + sym + 1);
    }

    __device__ __forceinline__ void load_pairs(int sym) {
        if (sym2 != sym) load_bounds(sym);
        sym1 = sym;
        row1 = row2;
        end1 = end2;
#pragma unroll
        for (int u = 0; u < kSymAhead; ++u) {
            const uint32_t i = row1 + 32u * u + lane_id();
            ahead[u] = i < end1 ? __ldg(A.sym_lists + i) : 0u;
        }
    }

    // The targets of the pairs of list `sym` (every pair, or those whose source is in the
    // set) become the set. next, next2 >= 0: the bytes after, whose pairs and list bounds
    // are loaded meanwhile.
    __device__ __forceinline__ int advance(int sym, bool every, int next, int next2) {
        if (sym1 != sym) load_pairs(sym);
        const uint32_t row = row1, end = end1;
        uint32_t e[kSymAhead], in[kSymAhead];
#pragma unroll
        for (int u = 0; u < kSymAhead; ++u) e[u] = ahead[u];
        if (next >= 0) {
            load_pairs(next);
            load_bounds(next2);
        }
        uint32_t seen = 0;  // bit 0: a member, kSymAccept: an accepting one
        auto put = [&](uint32_t p) {
            const uint32_t t = (p >> kSymStateBits) & kSymStateMask;
            atomicOr(nxt + (t >> 5), 1u << (t & 31u));
            seen |= (p & kSymAccept) | 1u;
        };
#pragma unroll
        for (int u = 0; u < kSymAhead; ++u) {  // the tests of a list's part together
            in[u] = 0u;
            if (row + 32u * u + lane_id() < end) {
                const uint32_t s = e[u] & kSymStateMask;
                in[u] = every ? 1u : (cur[s >> 5] >> (s & 31u)) & 1u;
            }
        }
#pragma unroll
        for (int u = 0; u < kSymAhead; ++u)
            if (in[u]) put(e[u]);
        for (uint32_t i = row + 32u * kSymAhead + lane_id(); i < end; i += 32) {
            const uint32_t p = __ldg(A.sym_lists + i), s = p & kSymStateMask;
            if (every || ((cur[s >> 5] >> (s & 31u)) & 1u)) put(p);
        }
        seen = __reduce_or_sync(GBFSM_FULL_MASK, seen);
        for (int w = (int)lane_id(); w < words; w += 32) cur[w] = 0u;
        uint32_t *t = cur;
        cur = nxt;
        nxt = t;
        __syncwarp();
        return (seen & kSymAccept) ? kAccept : (seen ? kAlive : kDead);
    }

    __device__ __forceinline__ int init_start() { return advance(kAlphabet, true, -1, -1); }

    // The superset of a chunk start: whatever the set was before byte c.
    __device__ __forceinline__ int init_after(uint32_t c) { return advance((int)c, true, -1, -1); }

    __device__ __forceinline__ int step(uint32_t sym) { return advance((int)sym, false, -1, -1); }

    using Bytes = BytesAhead;  // what next_step() reads

    __device__ __forceinline__ int next_step(Bytes &bytes) {
        const int sym = bytes.advance();
        return advance(sym, false, bytes.next, bytes.next2);
    }

    __device__ __forceinline__ int count() const {
        int c = 0;
        for (int w = (int)lane_id(); w < words; w += 32) c += __popc(cur[w]);
#pragma unroll
        for (int d = 16; d > 0; d >>= 1) c += __shfl_xor_sync(GBFSM_FULL_MASK, c, d);
        return c;
    }

    // The members' records to out[0 .. m) when there are at most `cap`; m, or -1.
    __device__ __forceinline__ int export_recs(uint4 *out, int cap) const {
        const int m = count();
        if (m > cap) return -1;
        int base = 0;
        for (int w0 = 0; w0 < words; w0 += 32) {
            const int w = w0 + (int)lane_id();
            uint32_t bits = w < words ? cur[w] : 0u;
            const uint32_t c = __popc(bits);
            const uint32_t incl = warp_inclusive_scan(c);
            int at = base + (int)(incl - c);
            while (bits) {
                const uint32_t s = ((uint32_t)w << 5) + (uint32_t)(__ffs(bits) - 1);
                bits &= bits - 1u;
                uint32_t info = 0;
                if ((A.accept_words[s >> 6] >> (s & 63u)) & 1ull) info |= GBFSM_EDGE_ACCEPT;
                if (__ldg(A.eps_row + s + 1) > __ldg(A.eps_row + s)) info |= GBFSM_EDGE_HAS_EPS;
                out[at++] = make_uint4(s, info, __ldg(A.sym_row + s), __ldg(A.sym_row + s + 1));
            }
            base += (int)__shfl_sync(GBFSM_FULL_MASK, incl, 31);
        }
        return m;
    }

    __device__ __forceinline__ void cleanup() {
        __syncwarp();
        for (int w = (int)lane_id(); w < words; w += 32) cur[w] = nxt[w] = 0u;
        __syncwarp();
    }
};

}  // namespace gbfsm
