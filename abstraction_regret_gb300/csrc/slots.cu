// Builder of an automaton's slot table (host code): the transition function of an
// epsilon-free NFA as one displaced array, so that a lane finds a state's successor on a
// byte with a single load.
//
// Every state owns a distinct even position, its base, and is named by its code, base / 2.
// The entry of state s for byte c lies in slot base(s) + c and carries the label c and the
// successor's code. Because bases are distinct, a slot holding label c at position p
// belongs to the one state whose base is p - c, so comparing the label with the byte tells
// a hit from another state's entry; an empty slot carries the label 0 or 1 that would put
// its base at an odd position, so it never hits. Rows of different states interleave:
// positions are given out first fit, longest rows first, 64 candidate bases at a time (the
// AND of the rows' shifted occupancy words), which fills about 93% of the slots of a random
// automaton of 16384 states and 4 edges a state.
//
// States with several edges on one byte step to a set. The sets that arise this way are
// given positions and codes of their own, as the states of a subset construction, as far
// as a budget of sets and slots goes: a walk then passes through a set of two or three
// states and back at the price of any other byte, which matters because a warp pays for
// the one lane of 32 that leaves the common path (16384 states, 4 edges a state: 1.6% of
// the bytes of a walk enter or leave a set, a third of a warp's steps).
//
// Codes are ordered so that one compare finds everything out of the ordinary: states that
// do not accept lie below set_begin, sets without an accepting member below accept_begin,
// then accepting states and sets up to multi_begin, then multi_begin itself (no state: its
// slots never hit), then the lists: code multi_begin + 1 + i stands for pairs[2i] (a
// state's code) and the rest of the list pairs[2i + 1] (a state's code or a list again).
#include <algorithm>
#include <map>
#include <new>
#include <utility>
#include <vector>

#include "common.cuh"

namespace gbfsm {
namespace {

// labels of a table that the lane launch can hold in shared memory at 3 bytes each
constexpr int64_t kSharedLabels = 75500;
constexpr uint64_t kEvenBits = 0x5555555555555555ull;

// Occupied slots and taken bases, grown as positions are given out.
struct Positions {
    std::vector<uint64_t> occ, base;

    void reach(size_t words) {
        if (occ.size() < words + 8) {
            occ.resize(words + words / 2 + 64, 0);
            base.resize(occ.size(), 0);
        }
    }

    // Occupancy of the 64 slots from 64 * w + shift.
    uint64_t window(size_t w, uint32_t shift) const {
        const size_t q = w + (shift >> 6);
        const uint32_t r = shift & 63u;
        return r ? (occ[q] >> r) | (occ[q + 1] << (64u - r)) : occ[q];
    }

    uint64_t candidates(size_t w, const uint8_t *labels, int n) {
        reach(w + 8);
        uint64_t c = kEvenBits & ~base[w];
        for (int k = 0; k < n && c; ++k) c &= ~window(w, labels[k]);
        return c;
    }

    void take(uint64_t b, const uint8_t *labels, int n) {
        base[b >> 6] |= 1ull << (b & 63u);
        for (int k = 0; k < n; ++k) {
            const uint64_t p = b + labels[k];
            occ[p >> 6] |= 1ull << (p & 63u);
        }
    }
};

// A state's (or set's) distinct labels and, for each, what it leads to: a state, or the
// index of a set plus the number of states.
struct Rows {
    std::vector<int64_t> begin{0};
    std::vector<uint8_t> label;
    std::vector<int32_t> to;
    int64_t count(size_t s) const { return begin[s + 1] - begin[s]; }
};

constexpr int32_t kSetMembers = 8;  // members of a set that gets a code of its own

struct Builder {
    int32_t n;
    const uint8_t *accept;
    Rows rows;
    std::vector<std::vector<int32_t>> sets;  // members, ascending
    std::map<std::vector<int32_t>, int32_t> set_id;

    int32_t successor(std::vector<int32_t> &targets) {
        if (targets.size() == 1) return targets[0];
        const auto it = set_id.emplace(targets, (int32_t)sets.size());
        if (it.second) sets.push_back(targets);
        return n + it.first->second;
    }

    // Closes the row of (label, target) edges `e` (destroyed).
    void add_row(std::vector<std::pair<int32_t, int32_t>> &e, std::vector<int32_t> &scratch) {
        std::sort(e.begin(), e.end());
        e.erase(std::unique(e.begin(), e.end()), e.end());
        for (size_t k = 0; k < e.size();) {
            scratch.clear();
            const int32_t c = e[k].first;
            for (; k < e.size() && e[k].first == c; ++k) scratch.push_back(e[k].second);
            rows.label.push_back((uint8_t)c);
            rows.to.push_back(successor(scratch));
        }
        rows.begin.push_back((int64_t)rows.label.size());
    }

    bool accepts(int32_t set) const {
        for (int32_t t : sets[(size_t)set])
            if (accept[t]) return true;
        return false;
    }
};

int32_t build(int32_t n, const int32_t *srp, const int32_t *stg, const int32_t *ssy,
              const uint8_t *accept, int64_t cap_slots, uint32_t *slots, int64_t cap_pairs,
              uint32_t *pairs, int64_t cap_codes, uint32_t *codes, int64_t *info) {
    Builder B{n, accept, {}, {}, {}};
    std::vector<std::pair<int32_t, int32_t>> e;  // (label, target) of one row
    std::vector<int32_t> scratch;
    for (int32_t s = 0; s < n; ++s) {
        e.clear();
        for (int32_t k = srp[s]; k < srp[s + 1]; ++k) {
            if (stg[k] < 0 || stg[k] >= n) return GBFSM_INVALID_ARG;
            if (ssy[k] == GBFSM_ANY_SYMBOL) {
                for (int32_t c = 0; c < kAlphabet; ++c) e.emplace_back(c, stg[k]);
            } else if (ssy[k] >= 0 && ssy[k] < kAlphabet) {
                e.emplace_back(ssy[k], stg[k]);
            } else {
                return GBFSM_INVALID_ARG;
            }
        }
        B.add_row(e, scratch);
        if ((int64_t)B.rows.label.size() > cap_slots) return GBFSM_UNSUPPORTED;
    }
    // rows of the sets, in the order they arise: at most a quarter more states and edges,
    // and no more edges than fit in shared memory when the states' own do
    const int64_t own = (int64_t)B.rows.label.size();
    int64_t most = own + own / 4 + 64;
    if (own <= kSharedLabels) most = std::min(most, kSharedLabels);
    most = std::min(most, cap_slots);
    const size_t most_sets = std::min((size_t)n / 4 + 64, (size_t)(cap_codes - n));
    std::vector<int32_t> row_of;  // per set: its row, or -1 (no code of its own)
    std::vector<int32_t> coded;   // the sets that have one
    for (size_t i = 0; i < B.sets.size(); ++i) {
        const std::vector<int32_t> members = B.sets[i];
        int64_t width = 0;
        for (int32_t t : members) width += B.rows.count((size_t)t);
        if (members.size() > (size_t)kSetMembers || coded.size() >= most_sets ||
            (int64_t)B.rows.label.size() + width > most) {
            row_of.push_back(-1);
            continue;
        }
        e.clear();
        for (int32_t t : members)
            for (int64_t k = B.rows.begin[t]; k < B.rows.begin[(size_t)t + 1]; ++k) {
                const int32_t to = B.rows.to[(size_t)k];
                if (to < n) {
                    e.emplace_back(B.rows.label[(size_t)k], to);
                } else {
                    for (int32_t u : B.sets[(size_t)(to - n)])
                        e.emplace_back(B.rows.label[(size_t)k], u);
                }
            }
        row_of.push_back(n + (int32_t)coded.size());
        coded.push_back((int32_t)i);
        B.add_row(e, scratch);
    }

    // positions: by class (states, sets, accepting), longest rows first in each
    const size_t total = (size_t)n + coded.size();
    auto rank = [&](size_t s) {
        if (s < (size_t)n) return accept[s] ? 2 : 0;
        return B.accepts(coded[s - (size_t)n]) ? 2 : 1;
    };
    std::vector<uint8_t> ranks(total);
    std::vector<int32_t> order(total);
    for (size_t s = 0; s < total; ++s) {
        ranks[s] = (uint8_t)rank(s);
        order[s] = (int32_t)s;
    }
    std::stable_sort(order.begin(), order.end(), [&](int32_t a, int32_t b) {
        if (ranks[a] != ranks[b]) return ranks[a] < ranks[b];
        return B.rows.count((size_t)a) > B.rows.count((size_t)b);
    });
    // how often a window may fail rows of one length before the search starts past it:
    // dense packing pays where the table can still fit in shared memory
    const int patience = (int64_t)B.rows.label.size() <= kSharedLabels ? 64 : 24;
    Positions pos;
    std::vector<uint16_t> failed;
    size_t from = 0, floor_w = 0;
    uint64_t floor_bit = ~0ull;
    int64_t last_count = -1;
    uint32_t begin[3] = {0, 0, 0}, top = 0;
    int at = 0;
    for (const int32_t s : order) {
        while (at < ranks[s]) {  // a class lies above the ones before it
            begin[++at] = top;
            floor_w = (2 * (size_t)top) >> 6;
            floor_bit = ~0ull << ((2 * top) & 63u);
            last_count = -1;
        }
        const int64_t count = B.rows.count((size_t)s);
        if (count != last_count) {
            last_count = count;
            from = floor_w;
            failed.assign(failed.size(), 0);
        }
        const uint8_t *lab = B.rows.label.data() + B.rows.begin[(size_t)s];
        for (size_t w = from;; ++w) {
            uint64_t c = pos.candidates(w, lab, (int)count);
            if (w == floor_w) c &= floor_bit;
            if (c) {
                const uint64_t b =
                    (uint64_t)w * 64u + (uint64_t)(__builtin_ffsll((long long)c) - 1);
                pos.take(b, lab, (int)count);
                codes[s] = (uint32_t)(b >> 1);
                top = std::max(top, codes[s] + 1u);
                break;
            }
            if (failed.size() <= w) failed.resize(w + 64, 0);
            if (++failed[w] >= patience && w == from) ++from;
        }
    }
    while (at < 2) begin[++at] = top;
    const uint32_t multi_begin = top;
    const int64_t n_slots = 2 * (int64_t)multi_begin + kAlphabet;
    if (n_slots > cap_slots) return GBFSM_UNSUPPORTED;

    // lists: one per set, of its members' codes (sets with a code of their own have one
    // too, for the steps that handle members one by one)
    int64_t n_pairs = 0;
    std::vector<uint32_t> list(B.sets.size());
    for (size_t i = 0; i < B.sets.size(); ++i) {
        const std::vector<int32_t> &m = B.sets[i];
        uint32_t code = codes[m.back()];
        for (size_t k = m.size() - 1; k-- > 0;) {
            if (n_pairs >= cap_pairs) return GBFSM_UNSUPPORTED;
            pairs[2 * n_pairs] = codes[m[k]];
            pairs[2 * n_pairs + 1] = code;
            code = multi_begin + 1u + (uint32_t)n_pairs++;
        }
        list[i] = code;
    }
    if ((uint64_t)multi_begin + 1u + (uint64_t)n_pairs > 1u << 24) return GBFSM_UNSUPPORTED;
    for (int64_t p = 0; p < n_slots; ++p) slots[p] = (uint32_t)((p + 1) & 1);
    for (size_t s = 0; s < total; ++s)
        for (int64_t k = B.rows.begin[s]; k < B.rows.begin[s + 1]; ++k) {
            const int32_t to = B.rows.to[(size_t)k];
            const int32_t row = to < n ? to : row_of[(size_t)(to - n)];
            const uint32_t code = row >= 0 ? codes[row] : list[(size_t)(to - n)];
            const uint32_t label = B.rows.label[(size_t)k];
            slots[2 * (int64_t)codes[s] + label] = label | (code << 8);
        }
    // after the states' codes: each coded set's code, its list and its size
    uint32_t *more = codes + n;
    const std::vector<uint32_t> set_code(more, more + coded.size());
    for (size_t i = 0; i < coded.size(); ++i) {
        more[3 * i] = set_code[i];
        more[3 * i + 1] = list[(size_t)coded[i]];
        more[3 * i + 2] = (uint32_t)B.sets[(size_t)coded[i]].size();
    }
    info[0] = n_slots;
    info[1] = n_pairs;
    info[2] = begin[1];
    info[3] = begin[2];
    info[4] = multi_begin;
    info[5] = (int64_t)coded.size();
    return GBFSM_OK;
}

}  // namespace
}  // namespace gbfsm

extern "C" int32_t gbfsm_slots_build(int32_t num_states, const int32_t *sym_row_ptr,
                                     const int32_t *sym_targets, const int32_t *sym_symbols,
                                     const uint8_t *accept, int64_t cap_slots, uint32_t *slots,
                                     int64_t cap_pairs, uint32_t *pairs, int64_t cap_codes,
                                     uint32_t *codes, int64_t *info) {
    using namespace gbfsm;
    if (num_states < 1 || !sym_row_ptr || !accept || !slots || !codes || !info ||
        cap_slots < kAlphabet || cap_codes < num_states || cap_pairs < 0 || (cap_pairs > 0 && !pairs))
        return GBFSM_INVALID_ARG;
    if (sym_row_ptr[0] != 0) return GBFSM_INVALID_ARG;
    for (int32_t s = 0; s < num_states; ++s)
        if (sym_row_ptr[s + 1] < sym_row_ptr[s]) return GBFSM_INVALID_ARG;
    if (sym_row_ptr[num_states] > 0 && (!sym_targets || !sym_symbols)) return GBFSM_INVALID_ARG;
    try {
        return build(num_states, sym_row_ptr, sym_targets, sym_symbols, accept, cap_slots, slots,
                     cap_pairs, pairs, num_states + (cap_codes - num_states) / 3, codes, info);
    } catch (const std::bad_alloc &) {
        return GBFSM_OOM;
    } catch (...) {
        return GBFSM_CUDA_ERROR;
    }
}
