// The launches of DFA_CHUNK and DFA_FIXUP tasks (chunked walks of long DFA inputs,
// dfa_chunks.cuh): a collapse launch (a warp per chunk, with shared scratch for the walk of
// the set of all states: two bitmaps of the largest DFA's states and two member lists), a
// walk launch (two chunks per warp, no shared memory) and a fix-up launch (a warp per
// input). Each takes tasks from a grid-stride loop over the task list, whose length is read
// on the device (the plan header).
#include <atomic>
#include <map>
#include <mutex>
#include <utility>

#include "common.cuh"
#include "dfa_chunks.cuh"
#include "engine.hpp"

namespace gbfsm {
namespace {

constexpr int kDfaChunkThreads = 128;  // 4 warps per CTA
constexpr int kDfaChunkWarps = kDfaChunkThreads / 32;
// Nearly the time of the chunk's walk while the device has idle warps: 64 inputs of 64 KiB on
// 4096 permuted states 22 ms, 10.8 walked whole and 470 with collapses to the chunks' ends.
constexpr uint32_t kBudgetPerByte = 48;

// A task of the list that names a DFA and chunks inside the tables; false otherwise.
__device__ __forceinline__ bool dfa_task_ok(const gbfsm_task &task,
                                            const gbfsm_automaton *__restrict__ table,
                                            int32_t n_automata, const gbfsm_chunk *chunks,
                                            int32_t n_chunks, uint32_t words) {
    if (task.automaton < 0 || task.automaton >= n_automata || task.first < 0 || task.count < 1 ||
        task.first > n_chunks - task.count)
        return false;
    const gbfsm_automaton &T = table[task.automaton];
    return T.kind == 1 && T.dfa.num_states >= 1 && (uint32_t)T.dfa.num_states <= words * 32u &&
           chunks[task.first].input >= 0;
}

__global__ void __launch_bounds__(kDfaChunkThreads, 6) dfa_collapse_kernel(
    const gbfsm_automaton *__restrict__ table, int32_t n_automata,
    const gbfsm_task *__restrict__ tasks, int32_t n_tasks, const int32_t *__restrict__ task_count,
    const uint8_t *__restrict__ data, const int64_t *__restrict__ offsets,
    const int64_t *__restrict__ ends, const gbfsm_chunk *__restrict__ chunks, int32_t n_chunks,
    void *records, uint32_t words, int32_t *latch) {
    extern __shared__ __align__(16) uint32_t dsm[];
    if (task_count) n_tasks = min(n_tasks, *task_count);
    const int warp_in_cta = (int)(threadIdx.x >> 5);
    uint32_t *bm0 = dsm + (size_t)warp_in_cta * (2u * words + kListMembers);
    uint32_t *bm1 = bm0 + words;
    uint16_t *list = reinterpret_cast<uint16_t *>(bm1 + words);
    // (a warp per CTA first, so that few tasks spread over the SMs)
    const int nwarps = (int)gridDim.x * kDfaChunkWarps;
    const int t0 = warp_in_cta * (int)gridDim.x + (int)blockIdx.x;
    const int rounds = t0 < n_tasks ? (n_tasks - t0 + nwarps - 1) / nwarps : 0;
    // twice over the tasks, the inputs' first chunks in the first round: an input that accepts
    // early is then latched before a later wave begins its other chunks
    for (int r = 0; r < 2 * rounds; ++r) {
        const gbfsm_task task = tasks[t0 + (r < rounds ? r : r - rounds) * nwarps];
        if (task.kind != GBFSM_TASK_DFA_CHUNK ||
            !dfa_task_ok(task, table, n_automata, chunks, n_chunks, words))
            continue;
        const gbfsm_chunk ch = chunks[task.first];
        if ((ch.index == 0) != (r < rounds)) continue;
        const gbfsm_dfa_dev d = table[task.automaton].dfa;
        const int64_t off = offsets[ch.input];
        DfaChunkRecord *rec = dfa_record(records, task.first);
        int32_t *lt = latch ? latch + ch.input : nullptr;
        if (d.entry_bytes == 2)
            dfa_chunk_collapse<uint16_t>(d, data + off, ch.begin - off, ch.end - off, ch.index,
                                         bm0, bm1, list, rec, lt, kBudgetPerByte);
        else
            dfa_chunk_collapse<uint32_t>(d, data + off, ch.begin - off, ch.end - off, ch.index,
                                         bm0, bm1, list, rec, lt, kBudgetPerByte);
        __syncwarp();
    }
}

__global__ void __launch_bounds__(kDfaChunkThreads) dfa_fixup_kernel(
    const gbfsm_automaton *__restrict__ table, int32_t n_automata,
    const gbfsm_task *__restrict__ tasks, int32_t n_tasks, const int32_t *__restrict__ task_count,
    const uint8_t *__restrict__ data, const int64_t *__restrict__ offsets,
    const int64_t *__restrict__ ends, const gbfsm_chunk *__restrict__ chunks, int32_t n_chunks,
    const void *records, uint32_t words, int32_t *flags, int32_t *lens, int32_t *examined) {
    if (task_count) n_tasks = min(n_tasks, *task_count);
    const int nwarps = (int)gridDim.x * kDfaChunkWarps;
    for (int t = (int)(threadIdx.x >> 5) * (int)gridDim.x + (int)blockIdx.x; t < n_tasks;
         t += nwarps) {
        const gbfsm_task task = tasks[t];
        if (task.kind != GBFSM_TASK_DFA_FIXUP ||
            !dfa_task_ok(task, table, n_automata, chunks, n_chunks, words))
            continue;
        const gbfsm_dfa_dev d = table[task.automaton].dfa;
        const int32_t input = chunks[task.first].input;
        const int64_t off = offsets[input];
        const int64_t len = (ends ? ends[input] : offsets[input + 1]) - off;
        const Verdict v =
            d.entry_bytes == 2
                ? dfa_fixup<uint16_t>(d, data + off, len, records, task.first, task.count)
                : dfa_fixup<uint32_t>(d, data + off, len, records, task.first, task.count);
        if (lane_id() == 0) {
            flags[input] = v.flag;
            lens[input] = v.len;
            if (examined) examined[input] = (int32_t)v.examined;
        }
    }
}

__global__ void __launch_bounds__(kDfaChunkThreads) dfa_walk_chunks_kernel(
    const gbfsm_automaton *__restrict__ table, int32_t n_automata,
    const gbfsm_task *__restrict__ tasks, int32_t n_tasks, const int32_t *__restrict__ task_count,
    const uint8_t *__restrict__ data, const int64_t *__restrict__ offsets,
    const int64_t *__restrict__ ends, const gbfsm_chunk *__restrict__ chunks, int32_t n_chunks,
    void *records, uint32_t words, int32_t *latch) {
    if (task_count) n_tasks = min(n_tasks, *task_count);
    constexpr int kPerWarp = 32 / kEntries;
    const int mine = (int)lane_id() / kEntries;
    const int step = (int)gridDim.x * kDfaChunkWarps * kPerWarp;
    for (int t0 = ((int)(threadIdx.x >> 5) * (int)gridDim.x + (int)blockIdx.x) * kPerWarp;
         t0 < n_tasks; t0 += step) {
        gbfsm_task task;
        bool valid = t0 + mine < n_tasks;
        if (valid) {
            task = tasks[t0 + mine];
            valid = task.kind == GBFSM_TASK_DFA_CHUNK &&
                    dfa_task_ok(task, table, n_automata, chunks, n_chunks, words);
        }
        DfaChunkRecord *rec = nullptr;
        const uint8_t *base = nullptr;
        const void *entries = nullptr;
        int32_t target = 0, index = 0, entry_bytes = 2;
        int32_t *lt = nullptr;
        if (valid) {
            const gbfsm_chunk ch = chunks[task.first];
            rec = dfa_record(records, task.first);
            valid = rec->p >= 0;
            const int64_t off = offsets[ch.input];
            const int64_t len = (ends ? ends[ch.input] : offsets[ch.input + 1]) - off;
            const gbfsm_automaton &T = table[task.automaton];
            base = data + off;
            entries = T.dfa.table;
            entry_bytes = T.dfa.entry_bytes;
            index = ch.index;
            lt = latch ? latch + ch.input : nullptr;
            target = dfa_walk_target(chunks, n_chunks, records, task.first, ch.end - off, len,
                                     T.dfa_overlap);
        }
        const bool two = valid && entry_bytes == 2, four = valid && entry_bytes != 2;
        if (__any_sync(GBFSM_FULL_MASK, two))
            dfa_chunk_walk<uint16_t>(two, static_cast<const uint16_t *>(entries), base, target,
                                     index, rec, lt);
        if (__any_sync(GBFSM_FULL_MASK, four))
            dfa_chunk_walk<uint32_t>(four, static_cast<const uint32_t *>(entries), base, target,
                                     index, rec, lt);
        __syncwarp();
    }
}

// Shared scratch of a CTA for DFAs of up to `words` x 32 states.
size_t dfa_chunks_smem(uint32_t words) {
    return (size_t)kDfaChunkWarps * (2u * words + kListMembers) * sizeof(uint32_t);
}

// Resident CTAs per SM for that scratch, asked once per (device, scratch size): later
// launches and graph captures reuse the answer. Opts the kernel in to the shared memory
// it needs above 48 KiB; -1 when that is more than the device has.
int dfa_chunks_blocks_per_sm(uint32_t words, gbfsm_status &st) {
    static std::mutex mu;
    static std::map<std::pair<int, uint32_t>, int> occupancy;
    st = GBFSM_OK;
    const size_t smem = dfa_chunks_smem(words);
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess) {
        cudaGetLastError();
        st = GBFSM_CUDA_ERROR;
        return 0;
    }
    std::lock_guard<std::mutex> lock(mu);
    const auto key = std::make_pair(dev, words);
    const auto it = occupancy.find(key);
    if (it != occupancy.end()) return it->second;
    if (smem > 48u * 1024u) {
        if (smem + kSmemReserve > (size_t)smem_optin()) return -1;
        // the most any size may take: a later, smaller one must not lower the limit
        if (cudaFuncSetAttribute(dfa_collapse_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 smem_optin() - (int)kSmemReserve) != cudaSuccess) {
            cudaGetLastError();
            st = GBFSM_CUDA_ERROR;
            return 0;
        }
    }
    int blocks = 0;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&blocks, dfa_collapse_kernel,
                                                      kDfaChunkThreads, smem) != cudaSuccess) {
        cudaGetLastError();
        st = GBFSM_CUDA_ERROR;
        return 0;
    }
    occupancy[key] = blocks;
    return blocks;
}

// Resident CTAs per SM of the walk launch, asked once per device.
int dfa_walk_blocks_per_sm() {
    static std::atomic<int> cached[64];
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) {
        cudaGetLastError();
        return 0;
    }
    int blocks = cached[dev].load();
    if (blocks > 0) return blocks;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&blocks, dfa_walk_chunks_kernel,
                                                      kDfaChunkThreads, 0) != cudaSuccess) {
        cudaGetLastError();
        return 0;
    }
    cached[dev].store(blocks);
    return blocks;
}

}  // namespace

gbfsm_status launch_dfa_chunks(const gbfsm_automaton *table, int32_t n_automata,
                               const gbfsm_task *tasks, int32_t max_tasks,
                               const int32_t *task_count, const uint8_t *data,
                               const int64_t *offsets, const int64_t *ends,
                               const gbfsm_chunk_io &chunk_io, int32_t max_states,
                               int32_t *flags, int32_t *lens, int32_t *examined,
                               int32_t *latch, int32_t kind, cudaStream_t stream) {
    if (max_tasks <= 0) return GBFSM_OK;
    const uint32_t words = ((uint32_t)max_states + 31u) >> 5;
    // one wave (max_tasks is the capacity: how many there are is read on the device)
    auto grid_of = [&](int per_sm) {
        const int wave = sm_count() * (per_sm > 0 ? per_sm : 1);
        return wave < max_tasks ? wave : max_tasks;
    };
    if (kind != GBFSM_TASK_DFA_FIXUP) {
        const size_t smem = dfa_chunks_smem(words);
        gbfsm_status st = GBFSM_OK;
        const int blocks = dfa_chunks_blocks_per_sm(words, st);
        if (st != GBFSM_OK) return fail(st, "dfa_collapse_kernel: occupancy query failed");
        if (blocks < 0)
            return fail(GBFSM_UNSUPPORTED, "DFA chunk walks of %d states need %zu shared bytes",
                        max_states, smem);
        dfa_collapse_kernel<<<grid_of(blocks), kDfaChunkThreads, smem, stream>>>(
            table, n_automata, tasks, max_tasks, task_count, data, offsets, ends,
            chunk_io.chunks, chunk_io.n_chunks, chunk_io.records, words, latch);
        GBFSM_LAUNCH_CHECK("dfa_collapse_kernel launch");
        dfa_walk_chunks_kernel<<<grid_of(dfa_walk_blocks_per_sm()),
                                 kDfaChunkThreads, 0, stream>>>(
            table, n_automata, tasks, max_tasks, task_count, data, offsets, ends,
            chunk_io.chunks, chunk_io.n_chunks, chunk_io.records, words, latch);
        GBFSM_LAUNCH_CHECK("dfa_walk_chunks_kernel launch");
    }
    if (kind != GBFSM_TASK_DFA_CHUNK) {
        dfa_fixup_kernel<<<grid_of(4), kDfaChunkThreads, 0, stream>>>(
            table, n_automata, tasks, max_tasks, task_count, data, offsets, ends,
            chunk_io.chunks, chunk_io.n_chunks, chunk_io.records, words, flags, lens, examined);
        GBFSM_LAUNCH_CHECK("dfa_fixup_kernel launch");
    }
    return GBFSM_OK;
}

}  // namespace gbfsm

extern "C" int32_t gbfsm_dfa_chunks_warps_per_sm(int32_t max_states) {
    using namespace gbfsm;
    if (max_states < 1 || max_states > 32768) return 0;
    gbfsm_status st = GBFSM_OK;
    const int blocks = dfa_chunks_blocks_per_sm(((uint32_t)max_states + 31u) >> 5, st);
    const int walk = dfa_walk_blocks_per_sm();
    return st == GBFSM_OK && blocks > 0 && walk > 0 ? walk * kDfaChunkWarps * (32 / kEntries) : 0;
}

extern "C" gbfsm_status gbfsm_dfa_chunks_run_kind(
    const gbfsm_automaton *table, int32_t n_automata, const gbfsm_task *tasks, int32_t max_tasks,
    const int32_t *task_count, const uint8_t *data, const int64_t *offsets, const int64_t *ends,
    const gbfsm_chunk_io *chunk_io, int32_t max_states, int32_t *flags, int32_t *lens,
    int32_t *examined, int32_t *latch, int32_t kind, void *stream) {
    using namespace gbfsm;
    if (max_tasks < 0 || n_automata < 0) return fail(GBFSM_INVALID_ARG, "negative task count");
    if (max_tasks == 0) return GBFSM_OK;
    if (!table || !tasks || !data || !offsets || !chunk_io || !chunk_io->chunks ||
        !chunk_io->records || !flags || !lens)
        return fail(GBFSM_INVALID_ARG, "NULL array passed to gbfsm_dfa_chunks_run");
    if (chunk_io->n_chunks < 1)
        return fail(GBFSM_INVALID_ARG, "gbfsm_dfa_chunks_run: empty chunk table");
    if (max_states < 1 || max_states > 32768)
        return fail(GBFSM_INVALID_ARG, "max_states must be in 1..32768 (got %d)", max_states);
    if (kind != 0 && kind != GBFSM_TASK_DFA_CHUNK && kind != GBFSM_TASK_DFA_FIXUP)
        return fail(GBFSM_INVALID_ARG, "gbfsm_dfa_chunks_run_kind: kind %d", kind);
    return launch_dfa_chunks(table, n_automata, tasks, max_tasks, task_count, data, offsets, ends,
                             *chunk_io, max_states, flags, lens, examined, latch, kind,
                             static_cast<cudaStream_t>(stream));
}

extern "C" gbfsm_status gbfsm_dfa_chunks_run(const gbfsm_automaton *table, int32_t n_automata,
                                             const gbfsm_task *tasks, int32_t max_tasks,
                                             const int32_t *task_count, const uint8_t *data,
                                             const int64_t *offsets, const int64_t *ends,
                                             const gbfsm_chunk_io *chunk_io,
                                             int32_t max_states, int32_t *flags, int32_t *lens,
                                             int32_t *examined, int32_t *latch, void *stream) {
    return gbfsm_dfa_chunks_run_kind(table, n_automata, tasks, max_tasks, task_count, data,
                                     offsets, ends, chunk_io, max_states, flags, lens, examined,
                                     latch, 0, stream);
}
