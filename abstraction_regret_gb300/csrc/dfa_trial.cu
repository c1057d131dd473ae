// How a DFA's set of all states shrinks over a text (host code): what the chunked walks of
// dfa_chunks.cuh depend on and cannot know from the number of states. A random DFA's set is
// down to 2n/t members after t bytes; one whose bytes permute its states (a counter modulo
// k, a parity product) keeps all n for good, and a chunk's collapse is then n lookups a byte
// for nothing: 256 inputs of 16 KiB on 4096 permuted states took 114 ms cut into chunks, 2.9
// whole. A trial is part of building a DFA's table, so larger DFAs have a thread per text: 1.4
// ms for three texts and 16384 states, 2.8 one after the other.
#include <new>
#include <system_error>
#include <thread>
#include <vector>

#include "common.cuh"
#include "dfa_device.cuh"

namespace gbfsm {
namespace {

constexpr int32_t kThreadStates = 2048;  // below, a text takes less than starting a thread
constexpr int32_t kMaxTexts = 8;

int32_t try_text(int32_t n, const int32_t *trans, const uint8_t *text, int64_t len, int32_t want,
                 int32_t schedules, int64_t *out) {
    const int64_t schedule = collapse_schedule((uint32_t)n);
    out[0] = -1;
    out[1] = 0;
    out[2] = schedule;
    try {
        std::vector<int32_t> set((size_t)n), seen((size_t)n, -1);
        for (int32_t s = 0; s < n; ++s) set[(size_t)s] = s;
        int64_t lookups = 0, pos = 0;
        while ((int64_t)set.size() > want && pos < len && lookups <= schedules * schedule) {
            lookups += (int64_t)set.size();
            const int32_t c = text[pos];
            size_t kept = 0;
            for (const int32_t s : set) {
                const int32_t t = trans[(size_t)s * kAlphabet + (size_t)c];
                if (t < 0 || t >= n) return GBFSM_INVALID_ARG;
                if (seen[(size_t)t] != (int32_t)pos) {
                    seen[(size_t)t] = (int32_t)pos;
                    set[kept++] = t;
                }
            }
            set.resize(kept);
            ++pos;
        }
        out[1] = lookups;
        if ((int64_t)set.size() <= want && lookups <= schedules * schedule) out[0] = pos;
        return GBFSM_OK;
    } catch (const std::bad_alloc &) {
        return GBFSM_OOM;
    }
}

}  // namespace
}  // namespace gbfsm

extern "C" int32_t gbfsm_dfa_collapse_trial(int32_t num_states, const int32_t *trans,
                                            const uint8_t *texts, int32_t n_texts, int64_t len,
                                            int32_t want, const int32_t *schedules, int64_t *out) {
    using namespace gbfsm;
    if (num_states < 1 || !trans || !texts || n_texts < 1 || n_texts > kMaxTexts || len < 0 ||
        len > INT32_MAX || want < 1 || !schedules || !out)
        return GBFSM_INVALID_ARG;
    for (int32_t k = 0; k < n_texts; ++k)
        if (schedules[k] < 1) return GBFSM_INVALID_ARG;
    int32_t status[kMaxTexts];
    std::thread threads[kMaxTexts];
    auto one = [&](int32_t k) {
        status[k] = try_text(num_states, trans, texts + k * len, len, want, schedules[k],
                             out + 3 * k);
    };
    for (int32_t k = 1; k < n_texts; ++k) {
        if (num_states >= kThreadStates) {
            try {
                threads[k] = std::thread(one, k);
                continue;
            } catch (const std::system_error &) {  // no thread to be had: here
            }
        }
        one(k);
    }
    one(0);
    for (int32_t k = 1; k < n_texts; ++k)
        if (threads[k].joinable()) threads[k].join();
    for (int32_t k = 0; k < n_texts; ++k)
        if (status[k] != GBFSM_OK) return status[k];
    return GBFSM_OK;
}
