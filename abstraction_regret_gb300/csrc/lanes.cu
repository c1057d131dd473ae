// One-lane-per-chunk speculative NFA launch (GBFSM_TASK_LANES tasks).
//
// Each warp takes one LANES task (up to 32 chunks) and each lane runs one chunk: over its
// automaton's slot table with slot_chunk() (lane_slots.cuh), from shared memory when the
// pool is one automaton whose table fits there, through L1 otherwise; or, for an automaton
// without one (too many wildcard edges), with lane_chunk() (chunks.cuh), which compares the
// packed edge labels of its members. A chunk that outgrows its lane is appended to the
// overflow queue as a CHUNK task, which the persistent launch then runs with a whole warp.
// There is no warp-wide loop, so this is a separate, lighter launch than the persistent
// kernel and fits more resident warps per SM.
#include <atomic>

#include "chunks.cuh"
#include "common.cuh"
#include "engine.hpp"
#include "lane_slots.cuh"

namespace gbfsm {
namespace {

constexpr int kLanesThreads = 256;   // tables in global memory: 64 registers, 4 CTAs per SM
constexpr int kLanesPerSm = 4;
constexpr int kSharedThreads = 1024;  // a table in shared memory: 64 registers, one CTA per SM

// Tasks that a CTA of `warps` warps takes: one per warp when the launch has few, so that
// they use every CTA of the grid. With `share` launches at a time (slices of one batch)
// that together fit the grid, each keeps to its part of it, so that they run side by side.
__device__ __forceinline__ int tasks_per_cta(int n_tasks, int share, int warps) {
    const int grid = (int)gridDim.x;
    const int64_t all = (int64_t)n_tasks * share;
    const int64_t spread = all <= (int64_t)grid * warps ? all : (int64_t)n_tasks;
    return max(1, (int)((spread + grid - 1) / grid));
}

// A chunk that outgrew its lane, for the overflow queue. The queue holds n_chunks entries:
// only a task list naming a chunk twice could overflow it, and then the extra entries are
// dropped rather than written past it.
__device__ __forceinline__ void spill_chunk(const ChunkIO &io, int32_t aut, int cid) {
    gbfsm_task spill;
    spill.automaton = aut;
    spill.first = cid;
    spill.count = 1;
    spill.kind = GBFSM_TASK_CHUNK;
    const int slot = atomicAdd(io.overflow_count, 1);
    if (slot < io.n_chunks) io.overflow_tasks[slot] = spill;
}

// The chunk that a lane runs of a LANES task, and its automaton; -1 when it has none (a
// short task, or one that names chunks or automata outside the tables).
__device__ __forceinline__ int lane_chunk_id(const ChunkIO &io, const gbfsm_task &task, int lane,
                                             int32_t n_automata, gbfsm_chunk &ch, int32_t &aut) {
    const int cid = task.first + lane;
    aut = 0;
    if (lane >= task.count || cid < 0 || cid >= io.n_chunks) return -1;
    ch = io.chunks[cid];
    if (ch.input < 0) return -1;
    // automaton -1: each lane runs its chunk's input's automaton
    aut = task.automaton >= 0 ? task.automaton : (io.aut_ids ? io.aut_ids[ch.input] : 0);
    if (aut >= 0 && aut < n_automata) return cid;
    aut = 0;
    return -1;
}

__global__ void __launch_bounds__(kLanesThreads, kLanesPerSm) lanes_kernel(
    const gbfsm_automaton *__restrict__ table, int32_t n_automata,
    const gbfsm_task *__restrict__ tasks, int32_t n_tasks, const int32_t *__restrict__ range,
    const uint8_t *__restrict__ data, const int64_t *__restrict__ offsets, ChunkIO io,
    int32_t share) {
    int32_t first = 0;
    if (range) {  // a task range written on the device by an earlier launch
        first = range[0];
        n_tasks = min(n_tasks, range[1]);
    }
    const int lane = (int)lane_id();
    const int warp = (int)(threadIdx.x >> 5);
    // every CTA takes a run of consecutive tasks, and the CTAs of an SM (dealt out in turn)
    // neighbouring runs when the launch fills the grid: they mostly share an automaton,
    // whose slots then stay in the SM's L1
    const int per = tasks_per_cta(n_tasks, share, kLanesThreads / 32);
    const int sms = (int)gridDim.x / kLanesPerSm;
    int run = (int)blockIdx.x;
    if (sms * kLanesPerSm == (int)gridDim.x && per * sms * (kLanesPerSm - 1) < n_tasks)
        run = (run % sms) * kLanesPerSm + run / sms;
    const int w_end = min(n_tasks, (run + 1) * per);
    for (int w = run * per + warp; w < w_end; w += kLanesThreads / 32) {
        const gbfsm_task task = tasks[first + w];
        int32_t aut;
        gbfsm_chunk ch;
        const int cid = lane_chunk_id(io, task, lane, n_automata, ch, aut);
        const bool slots = cid >= 0 && table[aut].kind == 0 && table[aut].nfa.slots != nullptr &&
                           table[aut].nfa.pair_row != nullptr;
        const uint32_t mask = __ballot_sync(GBFSM_FULL_MASK, slots);
        if (cid < 0 || table[aut].kind != 0) continue;  // LANES tasks of a DFA are ignored
        const gbfsm_nfa_dev &A = table[aut].nfa;
        const int64_t off = offsets[ch.input];
        bool done = false;
        if (slots) {
            const Bounds bd = chunk_bounds(io, A, data + off, cid, off);
            done = slot_chunk(A, GlobalSlots{A.slots, A.slot_pairs}, data + off, bd.b, bd.e,
                              bd.ov_end, ch.index, io.records + cid, mask);
        } else if (A.lane_edges != nullptr && A.pair_row != nullptr) {
            const Bounds bd = chunk_bounds(io, A, data + off, cid, off);
            done = lane_chunk(A, data + off, bd.b, bd.e, bd.ov_end, ch.index, io.records + cid);
        }
        if (!done) spill_chunk(io, aut, cid);
    }
}

// The same launch for a pool of one automaton whose slots fit in shared memory: each CTA
// (one per SM) copies them there with the TMA engine first. kNarrow: the 3-byte form.
template <bool kNarrow>
__global__ void __launch_bounds__(kSharedThreads, 1) lanes_shared_kernel(
    const gbfsm_automaton *__restrict__ table, const gbfsm_task *__restrict__ tasks,
    int32_t n_tasks, const int32_t *__restrict__ range, const uint8_t *__restrict__ data,
    const int64_t *__restrict__ offsets, ChunkIO io, int32_t share,
    uint32_t smem_bytes) {
    extern __shared__ __align__(16) uint8_t smem[];
    int32_t first = 0;
    if (range) {
        first = range[0];
        n_tasks = min(n_tasks, range[1]);
    }
    // tasks are dealt out a warp per CTA at a time over the CTAs that take part; the others
    // leave before the copy
    const int per = min(tasks_per_cta(n_tasks, share, kSharedThreads / 32), kSharedThreads / 32);
    const int ctas = min((int)gridDim.x, (n_tasks + per - 1) / per);
    if ((int)blockIdx.x >= ctas) return;
    const gbfsm_nfa_dev &A = table[0].nfa;
    const uint32_t n = A.num_slots;
    StageCopy copies[2];
    int n_copies;
    uint32_t bytes;
    if (kNarrow) {
        bytes = pad16(n) + pad16(2ull * n) + pad16(4ull * A.num_pairs);
        copies[0] = StageCopy{16u, A.slot_narrow, bytes};
        n_copies = 1;
    } else {
        bytes = pad16(4ull * n) + pad16(8ull * A.num_pairs);
        copies[0] = StageCopy{16u, A.slots, pad16(4ull * n)};
        copies[1] = StageCopy{16u + pad16(4ull * n), A.slot_pairs, pad16(8ull * A.num_pairs)};
        n_copies = 2;
    }
    // (a table that does not match what the host sized the launch for is not staged)
    bool ok = table[0].kind == 0 && A.pair_row != nullptr && 16u + bytes <= smem_bytes;
    if (ok) ok = stage_to_smem(smem, reinterpret_cast<uint64_t *>(smem), copies, n_copies);
    const int lane = (int)lane_id();
    for (int w = (int)(threadIdx.x >> 5) * ctas + (int)blockIdx.x; w < n_tasks;
         w += ctas * (kSharedThreads / 32)) {
        const gbfsm_task task = tasks[first + w];
        int32_t aut;
        gbfsm_chunk ch;
        const int cid = lane_chunk_id(io, task, lane, 1, ch, aut);
        const uint32_t mask = __ballot_sync(GBFSM_FULL_MASK, cid >= 0);
        if (cid < 0) continue;
        const int64_t off = offsets[ch.input];
        bool done = false;
        if (ok) {
            const Bounds bd = chunk_bounds(io, A, data + off, cid, off);
            const uint32_t t = smem_addr(smem + 16);
            if (kNarrow)
                done = slot_chunk(A,
                                  NarrowSlots{t, t + pad16(n), t + pad16(n) + pad16(2ull * n)},
                                  data + off, bd.b, bd.e, bd.ov_end, ch.index, io.records + cid,
                                  mask);
            else
                done = slot_chunk(A, WideSlots{t, t + pad16(4ull * n)}, data + off, bd.b, bd.e,
                                  bd.ov_end, ch.index, io.records + cid, mask);
        }
        if (!done) spill_chunk(io, 0, cid);
    }
}

}  // namespace

int lanes_warps_per_sm() {
    // asked once per device (the answer depends only on the kernel and the device)
    static int cached[64] = {0};
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) dev = -1;
    if (dev >= 0 && cached[dev] > 0) return cached[dev];
    // the kernel uses no shared memory: ask for the largest L1 share of the unified
    // L1/shared storage, where the lane records that miss in registers are gathered from
    cudaFuncSetAttribute(lanes_kernel, cudaFuncAttributePreferredSharedMemoryCarveout, 0);
    cudaGetLastError();
    int blocks = 0;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&blocks, lanes_kernel, kLanesThreads, 0) !=
        cudaSuccess)
        blocks = 0;
    cudaGetLastError();
    const int warps = blocks * (kLanesThreads / 32);
    if (dev >= 0 && warps > 0) cached[dev] = warps;
    return warps;
}

int32_t lanes_stage_limit() {
    const int most = smem_optin() - (int)kSmemReserve - 16;
    return most > 0 ? most : 0;
}

namespace {

// Opts the shared-memory kernel in to the largest table, once per device.
gbfsm_status lanes_allow_shared(bool narrow) {
    static std::atomic<uint32_t> allowed[2][64];
    int dev = 0;
    GBFSM_CUDA_TRY(cudaGetDevice(&dev));
    const bool known = dev >= 0 && dev < 64;
    if (known && allowed[narrow][dev].load() != 0) return GBFSM_OK;
    const int most = 16 + lanes_stage_limit();
    GBFSM_CUDA_TRY(narrow
                       ? cudaFuncSetAttribute(lanes_shared_kernel<true>,
                                              cudaFuncAttributeMaxDynamicSharedMemorySize, most)
                       : cudaFuncSetAttribute(lanes_shared_kernel<false>,
                                              cudaFuncAttributeMaxDynamicSharedMemorySize, most));
    if (known) allowed[narrow][dev].store(1);
    return GBFSM_OK;
}

}  // namespace

gbfsm_status launch_lanes(const gbfsm_automaton *table, int32_t n_automata,
                          const gbfsm_task *tasks, int32_t n_tasks, const int32_t *range,
                          const uint8_t *data, const int64_t *offsets,
                          const gbfsm_chunk_io &chunk_io, cudaStream_t stream) {
    if (n_tasks <= 0) return GBFSM_OK;
    lanes_warps_per_sm();  // once per device: sets the L1 share
    const int32_t share = chunk_io.lane_share > 1 ? chunk_io.lane_share : 1;
    ChunkIO io{chunk_io.chunks, static_cast<ChunkRecord *>(chunk_io.records),
               chunk_io.overflow_tasks, chunk_io.overflow_count, nullptr, chunk_io.n_chunks,
               chunk_io.aut_ids, 0};
    if (chunk_io.lane_stage != 0 && n_automata == 1) {
        const bool narrow = chunk_io.lane_stage == GBFSM_LANE_STAGE_NARROW;
        if (chunk_io.lane_stage_bytes < 0 || chunk_io.lane_stage_bytes > lanes_stage_limit())
            return fail(GBFSM_UNSUPPORTED, "lane tables of %d bytes do not fit in shared memory",
                        chunk_io.lane_stage_bytes);
        const uint32_t bytes = 16u + (uint32_t)chunk_io.lane_stage_bytes;
        const gbfsm_status st = lanes_allow_shared(narrow);
        if (st != GBFSM_OK) return st;
        const int grid = n_tasks < sm_count() ? n_tasks : sm_count();
        if (narrow)
            lanes_shared_kernel<true><<<grid, kSharedThreads, bytes, stream>>>(
                table, tasks, n_tasks, range, data, offsets, io, share, bytes);
        else
            lanes_shared_kernel<false><<<grid, kSharedThreads, bytes, stream>>>(
                table, tasks, n_tasks, range, data, offsets, io, share, bytes);
        GBFSM_LAUNCH_CHECK("lanes_shared_kernel launch");
        return GBFSM_OK;
    }
    // at most one resident wave; the warps loop over the tasks
    int grid = sm_count() * kLanesPerSm;
    if (grid > n_tasks) grid = n_tasks;
    lanes_kernel<<<grid, kLanesThreads, 0, stream>>>(table, n_automata, tasks, n_tasks, range,
                                                      data, offsets, io, share);
    GBFSM_LAUNCH_CHECK("lanes_kernel launch");
    return GBFSM_OK;
}

}  // namespace gbfsm
