// Fix-up of chunked inputs by a CTA per input, for automata with symbol lists
// (sym_device.cuh).
//
// Chunks of such automata often cannot be linked: a state that stays active for good once
// it is entered (a `.+` loop of a pattern) is in every speculative start set, whether the
// input has entered it or not, so the sets never become equal, and the input has to be
// stepped serially from its start. That chain is the time of the whole batch, and one warp
// needs 0.7 us a byte for a list of 200 pairs, all of it instructions issued one after
// another. Here 256 threads test a pair each. The list bounds of the next few hundred bytes
// are looked up ahead into shared memory, the pairs of the next three bytes are on their way
// while this byte's are tested against the set, and three bitmaps take turns (read, written,
// cleared), so that a byte costs one barrier; whether a step entered an accepting state or
// died is looked at every four bytes, from positions that the steps leave behind. 0.28 us a
// byte: 64 documents of 4..32 KiB on 100 patterns (1728 states, 215 pairs a byte) take 9.2
// ms, against 384 ms when a warp stepped the set member by member (an always active state
// has 2500 edges to go through), 26.8 ms by a warp over the lists, 19.4 ms by 128 threads
// that looked up every byte themselves. What bounds it: the latency of about 60 dependent
// instructions and a barrier a byte.
#include "chunks.cuh"
#include "common.cuh"
#include "engine.hpp"
#include "sym_device.cuh"

namespace gbfsm {
namespace {

constexpr int kSymThreads = 256;
constexpr int kSymRounds = 2;   // pairs per thread loaded ahead (lists of up to 512 pairs)
constexpr int kSymWindow = kSymThreads;  // bytes whose list bounds are looked up at a time
constexpr int kSymRing = 2 * kSymWindow;
constexpr uint32_t kNoPair = 0xffffffffu;
static_assert((kSymRing & (kSymRing - 1)) == 0, "ring positions are masked");

__device__ __forceinline__ uint32_t ring_at(int32_t position) {
    return (uint32_t)position & (uint32_t)(kSymRing - 1);
}

struct SymShared {
    uint2 *ring;       // [kSymRing] list bounds of the bytes at positions % kSymRing
    int32_t *accept;   // first position that entered an accepting state (INT32_MAX: none)
    int32_t *alive;    // last position with a member
    int32_t *members;  // sum of a population count
    int32_t *plan;     // warp 0's word to the others: done, last_rec
    uint32_t *maps;    // three bitmaps
};

// The CTA's run over one input: the set after the bytes before position `at`. Every thread
// calls every method with identical arguments and gets identical answers.
struct SymBlock {
    const gbfsm_nfa_dev &A;
    SymShared sh;
    int words;
    uint32_t *cur, *nxt, *old;  // the set; all zero; to be cleared in the next step
    const uint8_t *base;
    int32_t len, at;
    int32_t looked;  // positions whose list bounds are in the ring
    // the pairs of the next three bytes are loaded or on their way, byte i's in e[i % 4] (a
    // register that a load is on its way to must not be moved)
    int slot;
    uint32_t e[4][kSymRounds];

    __device__ __forceinline__ SymBlock(const gbfsm_nfa_dev &a, const SymShared &s,
                                        const uint8_t *in, int32_t n)
        : A(a), sh(s), words(2 * a.num_words), cur(s.maps), nxt(s.maps + words),
          old(s.maps + 2 * words), base(in), len(n), at(-1), looked(0), slot(0) {}

    // An empty set at position `pos`.
    __device__ __forceinline__ void clear(int32_t pos) {
        __syncthreads();
        for (int w = (int)threadIdx.x; w < 3 * words; w += kSymThreads) sh.maps[w] = 0u;
        if (threadIdx.x == 0) {
            *sh.accept = INT32_MAX;
            *sh.alive = pos;
        }
        __syncthreads();
    }

    __device__ __forceinline__ void load(uint2 bounds, uint32_t (&to)[kSymRounds]) const {
        const uint32_t i = bounds.x + threadIdx.x;
        to[0] = i < bounds.y ? __ldg(A.sym_lists + i) : kNoPair;
        if (bounds.y - bounds.x > (uint32_t)kSymThreads) {
#pragma unroll
            for (int u = 1; u < kSymRounds; ++u)
                to[u] = i + (uint32_t)kSymThreads * u < bounds.y
                            ? __ldg(A.sym_lists + i + kSymThreads * u)
                            : kNoPair;
        }
    }

    // List bounds of the next window of bytes (none past the end). The entries written are
    // those of bytes consumed a window ago; a barrier lies before their first use.
    __device__ __forceinline__ void look() {
        const int32_t p = looked + (int32_t)threadIdx.x;
        uint2 v = make_uint2(0u, 0u);
        if (p < len) {
            const uint32_t c = byte_at(base + p);
            v.x = __ldg(A.sym_list_row + c);
            v.y = __ldg(A.sym_list_row + c + 1);
        }
        sh.ring[ring_at(p)] = v;
        looked += kSymWindow;
    }

    __device__ __forceinline__ void seek(int32_t to) {
        __syncthreads();
        at = to;
        slot = 0;
        looked = to;
        look();
        __syncthreads();
        load(sh.ring[ring_at(to)], e[0]);
        load(sh.ring[ring_at(to + 1)], e[1]);
        load(sh.ring[ring_at(to + 2)], e[2]);
    }

    // One step over the pairs p0 (and any past them) of the list at `bounds`, to position pos.
    __device__ __forceinline__ void test(uint2 bounds, bool every, int32_t pos,
                                         const uint32_t (&p0)[kSymRounds]) {
        auto put = [&](uint32_t p) {
            const uint32_t t = (p >> kSymStateBits) & kSymStateMask;
            atomicOr(nxt + (t >> 5), 1u << (t & 31u));
            if (p & kSymAccept) atomicMin(sh.accept, pos);
            *sh.alive = pos;
        };
        auto pair = [&](uint32_t p) {
            if (p == kNoPair) return;
            const uint32_t s = p & kSymStateMask;
            if (every || ((cur[s >> 5] >> (s & 31u)) & 1u)) put(p);
        };
        pair(p0[0]);
        const uint32_t n = bounds.y - bounds.x;
        if (n > (uint32_t)kSymThreads) {
#pragma unroll
            for (int u = 1; u < kSymRounds; ++u) pair(p0[u]);
        }
        if (n > (uint32_t)(kSymThreads * kSymRounds))
            for (uint32_t i = bounds.x + (uint32_t)(kSymThreads * kSymRounds) + threadIdx.x;
                 i < bounds.y; i += kSymThreads)
                pair(__ldg(A.sym_lists + i));
        if ((int)threadIdx.x < words) old[threadIdx.x] = 0u;
        for (int w = (int)threadIdx.x + kSymThreads; w < words; w += kSymThreads) old[w] = 0u;
        uint32_t *t = old;
        old = cur;
        cur = nxt;
        nxt = t;
        __syncthreads();
    }

    __device__ __forceinline__ void start() {
        clear(0);
        const uint2 all = make_uint2(__ldg(A.sym_list_row + kAlphabet),
                                     __ldg(A.sym_list_row + kAlphabet + 1));
        load(all, e[0]);
        test(all, true, 0, e[0]);
    }

    // The next byte, its pairs in e[S].
    template <int S>
    __device__ __forceinline__ void one() {
        load(sh.ring[ring_at(at + 3)], e[(S + 3) % 4]);
        test(sh.ring[ring_at(at)], false, at + 1, e[S]);
        ++at;
    }

    // Up to `to` (<= len): kAlive there, or an event, `at` the position of the byte that
    // ends with it. An event is noticed up to four bytes late (its position stands): a
    // dead set stays dead, and the first accept is kept.
    __device__ __forceinline__ int run(int32_t to) {
        for (;;) {
            if (slot == 0 || at == to) {
                const int32_t acc = *static_cast<volatile int32_t *>(sh.accept);
                const int32_t live = *static_cast<volatile int32_t *>(sh.alive);
                // (a thread a step ahead may have written its later position already)
                if (acc <= at) {
                    at = acc;
                    return kAccept;
                }
                if (live < at) {
                    at = live + 1;
                    return kDead;
                }
                if (at == to) return kAlive;
                if (looked - at <= kSymWindow) look();
            }
            if (slot == 0) {
                one<0>();
                slot = 1;
                if (at == to) continue;
            }
            if (slot == 1) {
                one<1>();
                slot = 2;
                if (at == to) continue;
            }
            if (slot == 2) {
                one<2>();
                slot = 3;
                if (at == to) continue;
            }
            one<3>();
            slot = 0;
        }
    }

    __device__ __forceinline__ int count() {
        __syncthreads();
        if (threadIdx.x == 0) *sh.members = 0;
        __syncthreads();
        int c = 0;
        for (int w = (int)threadIdx.x; w < words; w += kSymThreads) c += __popc(cur[w]);
        if (c) atomicAdd(sh.members, c);
        __syncthreads();
        return *sh.members;
    }

    __device__ __forceinline__ void init_recs(const ChunkRecord &r) {
        clear(INT32_MIN);
        if ((int)threadIdx.x < min(r.end_count, kEndCap)) {
            const uint32_t s = r.end_recs[threadIdx.x].x;
            atomicOr(cur + (s >> 5), 1u << (s & 31u));
        }
        if (threadIdx.x == 0) *sh.alive = (int32_t)r.end;
        __syncthreads();
    }
};

// scan_links() out of line: its views would cost the steps below their registers (the serial
// chain of 64 documents 9.8 ms with it inlined, 9.5 without).
__device__ __noinline__ bool scan_links_apart(const ChunkRecord *recs, int first, int count,
                                              Verdict &v, int &last_rec) {
    return scan_links(recs, first, count, v, last_rec);
}

// The serial part of a fix-up (serial_fixup, chunks.cuh): from the chunk after last_rec.
__device__ Verdict sym_serial(const gbfsm_nfa_dev &A, const SymShared &sh, const uint8_t *base,
                              int64_t len, const ChunkRecord *recs, int first, int count,
                              int last_rec) {
    SymBlock w(A, sh, base, (int32_t)len);
    int k = 1;
    if (last_rec >= 0) {
        w.init_recs(recs[first + last_rec]);
        k = last_rec + 1;
    } else {  // the first chunk's final set was not recorded: recompute it exactly
        w.start();
        w.seek(0);
        w.run((int32_t)recs[first].end);  // (the scan found no event there)
    }
    // stops: the checkpoints of chunk k, then its end; matched: its record is exact from
    // there on
    int c = 0;
    bool matched = false;
    while (k < count) {
        const ChunkRecord &rk = recs[first + k];
        const int32_t b = (int32_t)rk.begin, e = (int32_t)rk.end;
        if (w.at < b || w.at > e) w.seek(b);
        const int32_t stop = matched || c >= kCheckpoints ? e : min(e, b + (1 << c));
        const int ev = w.run(stop);
        if (ev == kDead) return decided(0, w.at);
        if (ev == kAccept) return decided(1, w.at);
        if (!matched && c < kCheckpoints && stop == b + (1 << c)) {
            if (w.count() == rk.counts[c]) {
                if (rk.acc_after[c] >= 0) return decided(1, rk.acc_after[c]);
                if (rk.dead_at >= 0) return decided(0, rk.dead_at);
                matched = true;
                if (rk.end_count >= 0) {
                    w.init_recs(rk);
                    w.at = -1;  // at e: the next chunk seeks its begin
                    ++k;
                    c = 0;
                    matched = false;
                    continue;
                }
            }
            ++c;
        }
        if (stop == e) {
            ++k;
            c = 0;
            matched = false;
        }
    }
    return Verdict{0, 0, len};
}

__global__ void __launch_bounds__(kSymThreads, 2) sym_fixup_kernel(
    const gbfsm_automaton *__restrict__ table, int32_t n_automata,
    const gbfsm_task *__restrict__ tasks, int32_t n_tasks, const uint8_t *__restrict__ data,
    const int64_t *__restrict__ offsets, const int64_t *__restrict__ ends, ChunkIO io,
    int32_t max_words, int32_t list_capacity, int32_t *flags, int32_t *lens, int32_t *examined) {
    extern __shared__ __align__(16) uint32_t sm[];
    if (io.task_count) n_tasks = min(n_tasks, *io.task_count);
    SymShared sh;
    sh.ring = reinterpret_cast<uint2 *>(sm);
    int32_t *words = reinterpret_cast<int32_t *>(sm + 2 * kSymRing);
    sh.accept = words;
    sh.alive = words + 1;
    sh.members = words + 2;
    sh.plan = words + 4;
    sh.maps = sm + 2 * kSymRing + 8;
    for (int t = (int)blockIdx.x; t < n_tasks; t += (int)gridDim.x) {
        const gbfsm_task task = tasks[t];
        if (task.kind != GBFSM_TASK_FIXUP || task.automaton < 0 || task.automaton >= n_automata ||
            task.first < 0 || task.count < 1 || task.first + task.count > io.n_chunks)
            continue;
        const gbfsm_automaton &T = table[task.automaton];
        if (T.kind != 0 || !sym_usable(T.nfa, list_capacity) || T.nfa.num_words > max_words)
            continue;
        const gbfsm_nfa_dev &A = T.nfa;
        const int32_t id = io.chunks[task.first].input;
        const int64_t off = offsets[id];
        const int64_t len = (ends ? ends[id] : offsets[id + 1]) - off;
        __syncthreads();  // the last task's shared words are read
        Verdict v{0, 0, len};
        if (threadIdx.x < 32) {
            int last_rec = -1;
            const bool done = scan_links_apart(io.records, task.first, task.count, v, last_rec);
            if (threadIdx.x == 0) {
                sh.plan[0] = done ? 1 : 0;
                sh.plan[1] = last_rec;
            }
        }
        __syncthreads();
        const bool serial = sh.plan[0] == 0;
        if (serial)
            v = sym_serial(A, sh, data + off, len, io.records, task.first, task.count,
                           sh.plan[1]);
        if (threadIdx.x == 0) {
            flags[id] = v.flag;
            lens[id] = v.len;
            if (examined) examined[id] = (int32_t)v.examined;
        }
    }
}

}  // namespace

gbfsm_status launch_sym_fixup(const gbfsm_automaton *table, int32_t n_automata,
                              int32_t max_words, const gbfsm_task *tasks, int32_t n_tasks,
                              const uint8_t *data, const int64_t *offsets, const int64_t *ends,
                              const gbfsm_chunk_io &chunk_io, const gbfsm_plan &p, int32_t *flags,
                              int32_t *lens, int32_t *examined, cudaStream_t stream) {
    if (n_tasks <= 0) return GBFSM_OK;
    // as the persistent launch sizes its lists (sym_usable depends on it)
    const int32_t capacity = p.list_capacity > 0 ? p.list_capacity : kDefaultListCapacity;
    const int32_t most = (int32_t)((kSymStateMask + 1u) / 64u);
    const int32_t words = max_words < most ? (max_words > 0 ? max_words : 1) : most;
    const size_t smem = (2u * kSymRing + 8u + 3u * 2u * (size_t)words) * sizeof(uint32_t);
    ChunkIO io{chunk_io.chunks, static_cast<ChunkRecord *>(chunk_io.records), nullptr, nullptr,
               chunk_io.task_count, chunk_io.n_chunks, chunk_io.aut_ids, 1};
    const int wave = sm_count() * 4;
    sym_fixup_kernel<<<wave < n_tasks ? wave : n_tasks, kSymThreads, smem, stream>>>(
        table, n_automata, tasks, n_tasks, data, offsets, ends, io, words, capacity, flags, lens,
        examined);
    GBFSM_LAUNCH_CHECK("sym_fixup_kernel launch");
    return GBFSM_OK;
}

}  // namespace gbfsm

extern "C" gbfsm_status gbfsm_sym_fixup_run(
    const gbfsm_automaton *table, int32_t n_automata, int32_t max_words, const gbfsm_task *tasks,
    int32_t n_tasks, const uint8_t *data, const int64_t *offsets, const int64_t *ends,
    const gbfsm_chunk_io *chunk_io, const gbfsm_plan *plan, int32_t *flags, int32_t *lens,
    int32_t *examined, void *stream) {
    using namespace gbfsm;
    if (n_tasks < 0 || n_automata < 0) return fail(GBFSM_INVALID_ARG, "negative task count");
    if (n_tasks == 0) return GBFSM_OK;
    if (!table || !tasks || !data || !offsets || !chunk_io || !chunk_io->chunks ||
        !chunk_io->records || !plan || !flags || !lens)
        return fail(GBFSM_INVALID_ARG, "NULL array passed to gbfsm_sym_fixup_run");
    return launch_sym_fixup(table, n_automata, max_words, tasks, n_tasks, data, offsets, ends,
                            *chunk_io, *plan, flags, lens, examined,
                            static_cast<cudaStream_t>(stream));
}
