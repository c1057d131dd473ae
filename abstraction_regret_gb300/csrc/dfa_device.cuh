// Device-side DFA table walk (latch-first-match), shared by the plain DFA kernel
// (dfa_kernels.cu) and the persistent engine (persistent.cu).
//
// Semantics: src/gpufsm/reference.py:68-81 (simulate_dfa): accept[start] gives (1, 0);
// then cur = trans[cur * 256 + byte] per byte and the first accepting cur gives
// (1, pos + 1); running off the end gives (0, 0). The device table folds accept[next]
// into the top bit of each entry, so one load per byte yields both the successor and
// the latch test (the reference reads trans and then accept, dfa.cu:21-22).
//
// Input bytes are streamed with 16-byte loads (L1::no_allocate) one block ahead of use, four
// at a time whatever their alignment, so that lanes on inputs of different alignments stay
// together.
#pragma once

#include "common.cuh"

namespace gbfsm {

template <typename Entry>
struct EntryTraits;
template <>
struct EntryTraits<uint16_t> {
    static constexpr uint32_t kAccept = 0x8000u;
};
template <>
struct EntryTraits<uint32_t> {
    static constexpr uint32_t kAccept = 0x80000000u;
};

// Table lookups that walking the set of all n states of a random DFA takes until it has 16
// members: the set holds about 2n/t states after t bytes, so n + the sum of 2n/t up to n/8.
__host__ __device__ inline int64_t collapse_schedule(uint32_t n) {
    const float m = n > 16u ? (float)n : 16.0f;
    return (int64_t)(2.0f * m * (1.0f + logf(m / 16.0f)));
}

// Row index type: 32-bit for 2-byte tables (at most 32768 states), 64-bit otherwise.
template <typename Entry>
struct RowIndex {
    using type = uint64_t;
};
template <>
struct RowIndex<uint16_t> {
    using type = uint32_t;
};

// Table entry lookup from one array: shared memory of this CTA (kStaged) or global
// memory read through L2.
template <typename Entry, bool kStaged>
struct ArrayTable {
    const Entry *t;
    __device__ __forceinline__ uint32_t operator()(uint32_t state, uint32_t byte) const {
        const typename RowIndex<Entry>::type idx =
            (typename RowIndex<Entry>::type)state * (uint32_t)kAlphabet + byte;
        if (kStaged) return t[idx];
        return __ldg(t + idx);
    }
};

// One lane: consume bytes [a, b) of `base` from state s. Returns the state at b, or at the
// first accepting position q in (a, b], which goes to `acc` (-1 when none). Four lookups
// are made before their accept flags are looked at, so that the chain of dependent loads
// has no branch in it.
template <typename Lookup>
__device__ __forceinline__ uint32_t dfa_walk_span(const Lookup &look, uint32_t accept, uint32_t s,
                                                  const uint8_t *base, int32_t a, int32_t b,
                                                  int32_t &acc) {
    acc = -1;
    if (b <= a) return s;
    WordStream words;
    words.init(base + a, base + b);
    for (int32_t q = a; q < b; q += 4) {
        uint32_t w = words.next_word();
        if (b - q >= 4) {
            const uint32_t e0 = look(s, w & 0xffu);
            const uint32_t e1 = look(e0 & ~accept, (w >> 8) & 0xffu);
            const uint32_t e2 = look(e1 & ~accept, (w >> 16) & 0xffu);
            const uint32_t e3 = look(e2 & ~accept, w >> 24);
            if ((e0 | e1 | e2 | e3) & accept) {
                const int t = (e0 & accept) ? 0 : (e1 & accept) ? 1 : (e2 & accept) ? 2 : 3;
                acc = q + t + 1;
                return (t == 0 ? e0 : t == 1 ? e1 : t == 2 ? e2 : e3) & ~accept;
            }
            s = e3;
        } else {
            for (int t = 0; t < b - q; ++t, w >>= 8) {
                const uint32_t e = look(s, w & 0xffu);
                s = e & ~accept;
                if (e & accept) {
                    acc = q + t + 1;
                    return s;
                }
            }
        }
    }
    return s;
}

// One input, one thread, table entries through `lookup(state, byte)`. Returns (flag,
// len, examined) through references.
template <typename Entry, typename Lookup>
__device__ __forceinline__ void dfa_walk_with(const Lookup &table_at, const uint32_t *accept_bits,
                                              uint32_t start, const uint8_t *in, int64_t len,
                                              int32_t &flag, int32_t &mlen, int64_t &examined) {
    flag = 0;
    mlen = 0;
    examined = len;
    if ((__ldg(accept_bits + (start >> 5)) >> (start & 31u)) & 1u) {
        flag = 1;
        examined = 0;
        return;
    }
    for (int64_t pos = 0; pos < len; pos += 1 << 30) {
        int32_t acc;
        start = dfa_walk_span(table_at, EntryTraits<Entry>::kAccept, start, in + pos, 0,
                              (int32_t)min(len - pos, (int64_t)1 << 30), acc);
        if (acc >= 0) {
            flag = 1;
            mlen = (int32_t)(pos + acc);
            examined = pos + acc;
            return;
        }
    }
}

template <typename Entry, bool kStaged>
__device__ __forceinline__ void dfa_walk(const Entry *table, const uint32_t *accept_bits,
                                         uint32_t start, const uint8_t *in, int64_t len,
                                         int32_t &flag, int32_t &mlen, int64_t &examined) {
    dfa_walk_with<Entry>(ArrayTable<Entry, kStaged>{table}, accept_bits, start, in, len, flag,
                         mlen, examined);
}

}  // namespace gbfsm
