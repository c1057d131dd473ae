// How a DFA's set of all states shrinks over a text (host code): what the chunked walks of
// dfa_chunks.cuh depend on and cannot know from the number of states. A random DFA's set is
// down to 2n/t members after t bytes; one whose bytes permute its states (a counter modulo
// k, a parity product) keeps all n for good, and a chunk's collapse is then n lookups a byte
// for nothing: 256 inputs of 16 KiB on 4096 permuted states took 114 ms cut into chunks, 2.9
// whole.
#include <new>
#include <vector>

#include "common.cuh"
#include "dfa_device.cuh"

extern "C" int32_t gbfsm_dfa_collapse_trial(int32_t num_states, const int32_t *trans,
                                            const uint8_t *text, int64_t len, int32_t want,
                                            int32_t schedules, int64_t *out) {
    using namespace gbfsm;
    if (num_states < 1 || !trans || (len > 0 && !text) || len < 0 || want < 1 || schedules < 1 ||
        !out)
        return GBFSM_INVALID_ARG;
    const int64_t schedule = collapse_schedule((uint32_t)num_states);
    out[0] = -1;
    out[1] = 0;
    out[2] = schedule;
    try {
        std::vector<int32_t> set((size_t)num_states), seen((size_t)num_states, -1);
        for (int32_t s = 0; s < num_states; ++s) set[(size_t)s] = s;
        int64_t lookups = 0, pos = 0;
        while ((int64_t)set.size() > want && pos < len && lookups <= schedules * schedule) {
            lookups += (int64_t)set.size();
            const int32_t c = text[pos];
            size_t kept = 0;
            for (const int32_t s : set) {
                const int32_t t = trans[(size_t)s * kAlphabet + (size_t)c];
                if (t < 0 || t >= num_states) return GBFSM_INVALID_ARG;
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
