// Plain DFA launch for fewer inputs than the device has room for chains: a CTA per input,
// which is cut into two chunks per warp and followed from their entry states
// (dfa_chunks.cuh: collapse, walk and fix-up, here with the records in shared memory and a
// barrier between the three). One thread per input leaves 4096 inputs as 4096 chains of
// dependent lookups, 0.19-0.23 us each, and the GPU idle; two chunks a warp halve the
// chain, and fewer inputs get more. 4096 inputs of 64 KiB on 4096 states: 7.4 ms against
// 12.6 ms by dfa_cluster_kernel; 136 inputs of up to 4 KiB on 524 states 0.23 against 0.63.
#include <map>
#include <mutex>
#include <tuple>

#include "common.cuh"
#include "dfa_chunks.cuh"
#include "engine.hpp"

namespace gbfsm {
namespace {

constexpr int kSplitMaxWarps = 4;
constexpr int kSplitPerWarp = 32 / kEntries;  // chunks a warp walks
constexpr uint32_t kBudgetPerByte = 1;  // (this launch fills the device with warps)

// Shortest chunk: a set of n states collapses in about n / 8 bytes, whose steps take a few
// times a walk's; with chunks of n / 2 bytes, inputs of about n bytes on 8000 states were 9%
// slower cut than whole.
__device__ __forceinline__ int64_t split_chunk(int32_t num_states) {
    return max((int64_t)256, 2 * (int64_t)num_states);
}

// Bytes that a lane walks before anything else: an input that accepts early is done then,
// before its chunks' collapses.
__device__ __forceinline__ int64_t split_prefix(int64_t len) {
    return min((int64_t)1024, len / 16);
}

// (72 registers: 28 CTAs of one warp per SM)
__global__ void __launch_bounds__(kSplitMaxWarps * 32, 7) dfa_split_kernel(
    gbfsm_dfa_dev d, const uint8_t *__restrict__ data, const int64_t *__restrict__ offsets,
    uint32_t words, int32_t *flags, int32_t *lens, int32_t *examined) {
    extern __shared__ __align__(16) uint32_t sm[];
    const int warps = (int)(blockDim.x >> 5), warp = (int)(threadIdx.x >> 5);
    const uint32_t lane = lane_id();
    void *records = sm;  // kSplitPerWarp per warp
    uint32_t *rest = sm + warps * kSplitPerWarp * (GBFSM_CHUNK_RECORD_BYTES / 4);
    int32_t *latch = reinterpret_cast<int32_t *>(rest);
    uint32_t *bm0 = rest + 4 + (size_t)warp * (2u * words + kListMembers);
    uint32_t *bm1 = bm0 + words;
    uint16_t *list = reinterpret_cast<uint16_t *>(bm1 + words);
    const int input = (int)blockIdx.x;
    const uint8_t *base = data + offsets[input];
    const int64_t len = offsets[input + 1] - offsets[input];
    const int count =
        (int)min((int64_t)(warps * kSplitPerWarp), len / split_chunk(d.num_states));
    const uint16_t *table = static_cast<const uint16_t *>(d.table);
    if (count < 2) {  // too short to cut: one lane
        if (threadIdx.x == 0) {
            int32_t f, l;
            int64_t ex;
            dfa_walk<uint16_t, false>(table, d.accept_bits, (uint32_t)d.start_state, base, len,
                                      f, l, ex);
            flags[input] = f;
            lens[input] = l;
            if (examined) examined[input] = (int32_t)ex;
        }
        return;
    }
    const int64_t prefix = split_prefix(len);
    if (threadIdx.x == 0) {
        *latch = INT32_MAX;
        int32_t acc = -1;
        uint32_t s = (uint32_t)d.start_state;
        if ((__ldg(d.accept_bits + (s >> 5)) >> (s & 31u)) & 1u)
            acc = 0;
        else
            s = dfa_walk_span(GlobalEntries<uint16_t>{table}, EntryTraits<uint16_t>::kAccept, s,
                              base, 0, (int32_t)prefix, acc);
        DfaChunkRecord *r = dfa_record(records, 0);
        r->p = r->at = r->done = (int32_t)prefix;
        r->count = 1;
        r->entry[0] = r->exit[0] = (uint16_t)s;
        r->acc[0] = acc;
    }
    __syncthreads();
    if (const int32_t acc = dfa_record(records, 0)->acc[0]; acc >= 0) {
        if (threadIdx.x == 0) {
            flags[input] = 1;
            lens[input] = acc;
            if (examined) examined[input] = acc;
        }
        return;
    }
    const int64_t more = len - prefix;  // the chunks are cut from these bytes
    for (int c = warp == 0 ? warps : warp; c < count; c += warps)
        dfa_chunk_collapse<uint16_t>(d, base, prefix + c * more / count,
                                     prefix + (c + 1) * more / count, c, bm0, bm1, list,
                                     dfa_record(records, c), latch, kBudgetPerByte);
    __syncthreads();
    const int c = warp + (int)(lane / kEntries) * warps;
    DfaChunkRecord *rec = dfa_record(records, c < count ? c : 0);
    const bool valid = c < count && rec->p >= 0;
    int32_t target = (int32_t)len;
    for (int j = count - 1; j > c; --j) {
        const int32_t at = dfa_record(records, j)->at;
        if (at >= 0) target = at;
    }
    dfa_chunk_walk<uint16_t>(valid, table, base, target, c, rec, latch);
    __syncthreads();
    if (warp == 0) {
        const Verdict v = dfa_fixup<uint16_t>(d, base, len, records, 0, count);
        if (lane == 0) {
            flags[input] = v.flag;
            lens[input] = v.len;
            if (examined) examined[input] = (int32_t)v.examined;
        }
    }
}

size_t split_smem(uint32_t words, int warps) {
    return (size_t)warps * kSplitPerWarp * GBFSM_CHUNK_RECORD_BYTES + 16u +
           (size_t)warps * (2u * words + kListMembers) * sizeof(uint32_t);
}

// Resident CTAs per SM, asked once per device and shape (0: cannot run).
int split_blocks_per_sm(uint32_t words, int warps) {
    static std::mutex mu;
    static std::map<std::tuple<int, uint32_t, int>, int> cache;
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess) {
        cudaGetLastError();
        return 0;
    }
    std::lock_guard<std::mutex> lock(mu);
    const auto key = std::make_tuple(dev, words, warps);
    const auto it = cache.find(key);
    if (it != cache.end()) return it->second;
    const size_t smem = split_smem(words, warps);
    int blocks = 0;
    if (smem + kSmemReserve <= (size_t)smem_optin() &&
        cudaFuncSetAttribute(dfa_split_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             smem_optin() - (int)kSmemReserve) == cudaSuccess &&
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&blocks, dfa_split_kernel, 32 * warps,
                                                      smem) != cudaSuccess)
        blocks = 0;
    cudaGetLastError();
    cache[key] = blocks;
    return blocks;
}

}  // namespace

bool launch_dfa_split(const gbfsm_dfa_dev &d, const uint8_t *data, const int64_t *offsets,
                      int32_t n_inputs, int32_t *flags, int32_t *lens, int32_t *examined,
                      cudaStream_t stream, gbfsm_status &status) {
    // A DFA whose set of all states has been seen to shrink as fast as a random one's does:
    // the cut pays while a collapse takes no more than about twice as many lookups.
    // And a DFA that accepts often ends its inputs within a few thousand bytes, about as many as
    // a collapse costs: 4096 inputs of 64 KiB with 0.05% accepting states took 4.6 ms cut and
    // 2.5 ms whole
    if (d.entry_bytes != 2 || d.num_states > 32768 || !(d.flags & GBFSM_DFA_COLLAPSES) ||
        !(d.flags & GBFSM_DFA_RARE_ACCEPT))
        return false;
    const uint32_t words = ((uint32_t)d.num_states + 31u) >> 5;
    for (int warps = kSplitMaxWarps; warps >= 1; warps /= 2) {
        if (n_inputs > sm_count() * split_blocks_per_sm(words, warps)) continue;
        dfa_split_kernel<<<n_inputs, 32 * warps, split_smem(words, warps), stream>>>(
            d, data, offsets, words, flags, lens, examined);
        const cudaError_t err = cudaGetLastError();
        status = err == cudaSuccess ? GBFSM_OK : cuda_fail(err, "dfa_split_kernel launch");
        return true;
    }
    return false;  // more than one wave of them: enough chains as they are
}

}  // namespace gbfsm
