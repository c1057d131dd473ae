// Epsilon closures for the symbol lists (host code): of the states that edges lead to, as
// long as the lists stay within their limit. The closures of a chain of epsilon edges hold a
// quarter of its length squared states, and an automaton that long has lists far above the
// limit, so the sum is looked at after every closure and the search ends there (a chain of
// 4000 states took 6 s when all closures were gathered first, in Python).
#include <new>
#include <vector>

#include "common.cuh"

extern "C" int32_t gbfsm_eps_closures(int32_t num_states, const int32_t *eps_row_ptr,
                                      const int32_t *eps_targets, const int64_t *weight,
                                      int32_t start, int64_t limit, int64_t *row, int32_t *states) {
    using namespace gbfsm;
    if (num_states < 1 || !eps_row_ptr || !weight || start < 0 || start >= num_states ||
        limit < 0 || !row || !states || eps_row_ptr[0] != 0)
        return GBFSM_INVALID_ARG;
    for (int32_t s = 0; s < num_states; ++s)
        if (eps_row_ptr[s + 1] < eps_row_ptr[s]) return GBFSM_INVALID_ARG;
    const int64_t edges = eps_row_ptr[num_states];
    if (edges > 0 && !eps_targets) return GBFSM_INVALID_ARG;
    for (int64_t k = 0; k < edges; ++k)
        if (eps_targets[k] < 0 || eps_targets[k] >= num_states) return GBFSM_INVALID_ARG;
    // edges followed in all: closures of few states with very many edges among them end the
    // search as well
    int64_t steps = 64 * (limit + num_states) + edges;
    try {
        std::vector<int32_t> seen((size_t)num_states, -1);
        int64_t n = 0, pairs = 0;
        for (int32_t s = 0; s < num_states; ++s) {
            row[s] = n;
            if (eps_row_ptr[s + 1] == eps_row_ptr[s] || (weight[s] == 0 && s != start)) continue;
            const int64_t first = n;
            // the most members that the limit has room for (the start's closure is not counted)
            const int64_t room = weight[s] > 0 ? (limit - pairs) / weight[s] : num_states;
            seen[(size_t)s] = s;
            if (room < 1) return GBFSM_UNSUPPORTED;
            states[n++] = s;
            for (int64_t k = first; k < n; ++k) {
                const int32_t u = states[k];
                for (int32_t e = eps_row_ptr[u]; e < eps_row_ptr[u + 1]; ++e) {
                    const int32_t t = eps_targets[e];
                    if (--steps < 0) return GBFSM_UNSUPPORTED;
                    if (seen[(size_t)t] == s) continue;
                    seen[(size_t)t] = s;
                    if (n - first >= room) return GBFSM_UNSUPPORTED;
                    states[n++] = t;
                }
            }
            pairs += weight[s] * (n - first);
        }
        row[num_states] = n;
        return GBFSM_OK;
    } catch (const std::bad_alloc &) {
        return GBFSM_OOM;
    }
}
