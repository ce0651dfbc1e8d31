// Slot-table scheduler: router top-k ids of all ranks -> per-expert padded row ranges and the
// (peer rank, peer route) tables of this rank.  Integer-only, bit-exact with the reference
// scheduler (csrc/scheduler.cuh:35-147 in Mixture-of-Kittens): routes of one peer are ordered
// "thread-major" over 1024 virtual threads, peers are interleaved round-robin inside an expert,
// experts are padded to 256 rows.
//
// The reference rescans every peer's routes 2*El times.  Here every route is read three times, or twice with the scan
// kernel below; a chunk is the routes of 4 virtual threads of one peer, a block handles 8 consecutive chunks, a warp one:
//   count   every block histograms its routes per local expert in shared memory   -> block_hist[peer][block][expert]
//           and all blocks together clear the tables
//   place   every block sums block_hist into the expert totals of every peer and its own start offsets, counts its
//           chunks again in shared memory for the offsets of its warps, then each warp walks its routes in order, ranks
//           equal experts inside the warp with match.any, and writes the slots
// The place blocks re-read W*32*El counts each, one (rank, expert) pair per thread up to W*El = 256.  Larger problems run a
// scan kernel in between that turns the chunk counts into offsets once, and launch all three kernels plainly:
//   scan    one warp per (expert, peer): exclusive offsets of the 256 chunks and the total   -> cnt[expert][peer]
// Calls back to back on one stream, top-8, us with two kernels / with three, one B200:
//   W*El                          64          256          320          384          512
//   1 rank,    512 tokens    7.4 / 16.4   7.8 / 16.4  10.4 / 18.4  10.7 / 17.4  11.0 / 17.4
//   1 rank,  16384 tokens   15.7 / 22.6  16.0 / 22.6  18.8 / 24.6  19.1 / 22.9  18.8 / 24.6
//   8 ranks,   512 tokens    9.0 / 16.4   9.6 / 16.6  10.8 / 18.4  11.6 / 18.4  11.1 / 18.4
//   8 ranks, 16384 tokens   20.1 / 26.6  20.2 / 26.6  21.6 / 26.7  22.4 / 26.6  41.6 / 26.6
// So the line, where a thread takes its second pair, is on the near side of a steep rise that comes between 384 and 512.
// Algorithmic traffic: W*T*K ids of 4 or 8 B, three times or twice, + 2 * capacity * 4 B of table writes; at these sizes
// launches and the latency of dependent loads decide (before, with three kernels always: 8 ranks x 32 experts 30.7 us, now
// 20.4; one rank x 128 experts 28.7, now 15.7, or 18.1 from int64 ids without the cast in front; 8 ranks x 256 experts 36.2,
// now 30.4).  Routes are read as int32 or, on one rank, as the caller's int64.
#include <algorithm>
#include <atomic>

#include "common.cuh"
#include "profile.cuh"

namespace mok {
namespace {

constexpr int kVThreads = 1024;           // virtual threads of the reference ordering
constexpr int kChunkVts = 4;              // virtual threads per warp-chunk
constexpr int kChunks = kVThreads / kChunkVts;   // 256 chunks per peer
constexpr int kWarpsPerBlock = 8;
constexpr int kBlockThreads = kWarpsPerBlock * 32;
constexpr int kPad = 256;                 // expert row padding

constexpr int kBlocksPerPeer = kChunks / kWarpsPerBlock;
constexpr int kMaxFusedPairs = 256;      // W * El up to which the place kernel finds its offsets by itself

struct SchedParams {
    const void* topk;       // [W, R] int32 or int64
    int W, R, El, rank, capacity;
    int* peer_rank;         // [capacity]
    int* peer_token_idx;    // [capacity]
    int* num_tokens;        // [1]
    int* tokens_per_expert; // [El]
    int* chunk_hist;        // [W, kChunks, El], or [W, kBlocksPerPeer, El] where the place kernel finds its offsets
    int* cnt;               // [El, W]
    int* status;
    int vec_routes;         // routes can be read 16 bytes at a time (aligned, R a multiple of four)
    int vec_tables;         // the tables can be cleared 16 bytes at a time
};

// local expert of a route, or -1 (an int64 id is cut to 32 bits as the cast in front of the int32 tables would)
template <class Id>
__device__ __forceinline__ int local_expert(Id id, int first, int El) {
    const int e = static_cast<int>(id) - first;
    return e >= 0 && e < El ? e : -1;
}

// Counts the routes of a warp's chunk into `hist`.  Virtual thread vt owns routes vt, vt+1024, ..., so the chunk's four
// virtual threads sit side by side in every run of 1024 routes: a lane takes the four routes of one run (one or two
// 16-byte loads where alignment and R allow).
template <class Id>
__device__ __forceinline__ void count_chunk(const Id* routes, int R, bool vec, int v0, int first, int El, int* hist, int lane) {
    static_assert(kChunkVts == 4, "four routes per load");
#pragma unroll 4
    for (long long base = v0 + lane * kVThreads; base < R; base += 32 * kVThreads) {
        Id id[4];
        if (!vec) {
#pragma unroll
            for (int j = 0; j < 4; ++j) id[j] = base + j < R ? routes[base + j] : static_cast<Id>(-1);     // -1: no expert
        } else if constexpr (sizeof(Id) == 4) {
            *reinterpret_cast<int4*>(id) = *reinterpret_cast<const int4*>(routes + base);
        } else {
            reinterpret_cast<longlong2*>(id)[0] = reinterpret_cast<const longlong2*>(routes + base)[0];
            reinterpret_cast<longlong2*>(id)[1] = reinterpret_cast<const longlong2*>(routes + base)[1];
        }
#pragma unroll
        for (int j = 0; j < 4; ++j) { const int e = local_expert(id[j], first, El); if (e >= 0) atomicAdd(&hist[e], 1); }
    }
}

template <class Id, bool kFused>
__global__ void __launch_bounds__(kBlockThreads) sched_count_kernel(SchedParams p) {
    extern __shared__ int smem[];                            // kFused: [El] of the block, else [warps][El]
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    int* hist = smem + (kFused ? 0 : warp * p.El);
    const int hists = kFused ? p.El : kWarpsPerBlock * p.El;
    for (int e = threadIdx.x; e < hists; e += kBlockThreads) smem[e] = 0;
    __syncthreads();
    pdl_wait();

    // both tables to -1 (unwritten slots), over the whole grid
    const int4 none = make_int4(-1, -1, -1, -1);
    const int vecs = p.vec_tables ? p.capacity / 4 : 0;
    for (int i = blockIdx.x * kBlockThreads + threadIdx.x; i < vecs; i += gridDim.x * kBlockThreads) {
        reinterpret_cast<int4*>(p.peer_rank)[i] = none;
        reinterpret_cast<int4*>(p.peer_token_idx)[i] = none;
    }
    for (int i = 4 * vecs + blockIdx.x * kBlockThreads + threadIdx.x; i < p.capacity; i += gridDim.x * kBlockThreads) {
        p.peer_rank[i] = -1;
        p.peer_token_idx[i] = -1;
    }

    const int gchunk = blockIdx.x * kWarpsPerBlock + warp;   // over W * kChunks; blocks beyond only clear
    if (blockIdx.x >= p.W * kBlocksPerPeer) return;
    const int peer = gchunk / kChunks, chunk = gchunk % kChunks;
    count_chunk(static_cast<const Id*>(p.topk) + static_cast<size_t>(peer) * p.R, p.R, p.vec_routes != 0, chunk * kChunkVts,
                p.rank * p.El, p.El, hist, lane);
    if (kFused) __syncthreads(); else __syncwarp();
    if (kFused) {
        int* out = p.chunk_hist + static_cast<size_t>(blockIdx.x) * p.El;
        for (int e = threadIdx.x; e < p.El; e += kBlockThreads) out[e] = hist[e];
    } else {
        int* out = p.chunk_hist + static_cast<size_t>(gchunk) * p.El;
        for (int e = lane; e < p.El; e += 32) out[e] = hist[e];
    }
}

// one warp per (expert, peer): exclusive scan over the 256 chunks, in place
__global__ void __launch_bounds__(kBlockThreads) sched_scan_kernel(SchedParams p) {
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    pdl_wait();
    const int pair = blockIdx.x * kWarpsPerBlock + warp;       // e * W + peer
    if (pair >= p.El * p.W) return;
    const int e = pair / p.W, peer = pair % p.W;
    constexpr int kPerLane = kChunks / 32;                      // 8 consecutive chunks per lane
    int v[kPerLane];
    int sum = 0;
#pragma unroll
    for (int j = 0; j < kPerLane; ++j) {
        v[j] = p.chunk_hist[(static_cast<size_t>(peer) * kChunks + lane * kPerLane + j) * p.El + e];
        sum += v[j];
    }
    int incl = sum;
#pragma unroll
    for (int off = 1; off < 32; off <<= 1) {
        const int n = __shfl_up_sync(0xffffffffu, incl, off);
        if (lane >= off) incl += n;
    }
    int run = incl - sum;
#pragma unroll
    for (int j = 0; j < kPerLane; ++j) {
        p.chunk_hist[(static_cast<size_t>(peer) * kChunks + lane * kPerLane + j) * p.El + e] = run;
        run += v[j];
    }
    if (lane == 31) p.cnt[pair] = incl;
}

template <class Id, bool kFused>
__global__ void __launch_bounds__(kBlockThreads) sched_place_kernel(SchedParams p) {
    extern __shared__ int smem[];
    int* s_cnt = smem;                        // [El * W]
    int* s_base = s_cnt + p.El * p.W;         // [El]
    int* s_run = s_base + p.El;               // [warps][El]
    __shared__ int s_warp_tot[kWarpsPerBlock];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int gchunk = blockIdx.x * kWarpsPerBlock + warp;
    const int peer = gchunk / kChunks, chunk = gchunk % kChunks;
    const int v0 = chunk * kChunkVts, first = p.rank * p.El;
    const Id* routes = static_cast<const Id*>(p.topk) + static_cast<size_t>(peer) * p.R;
    int* run = s_run + warp * p.El;

    if (kFused) {
        for (int e = threadIdx.x; e < kWarpsPerBlock * p.El; e += kBlockThreads) s_run[e] = 0;
        __syncthreads();
    }
    pdl_wait();
    if (kFused) {
        count_chunk(routes, p.R, p.vec_routes != 0, v0, first, p.El, run, lane);
        __syncthreads();
        // totals of every peer, this block's start inside its peer, and from that the starts of its eight warps
        const int mine = blockIdx.x % kBlocksPerPeer;
        for (int i = threadIdx.x; i < p.El * p.W; i += kBlockThreads) {
            const int r = i / p.El, e = i - r * p.El;
            const int* h = p.chunk_hist + static_cast<size_t>(r) * kBlocksPerPeer * p.El + e;
            int total = 0, before = 0;
#pragma unroll
            for (int b = 0; b < kBlocksPerPeer; ++b) {
                const int n = h[static_cast<size_t>(b) * p.El];
                total += n;
                if (b < mine) before += n;
            }
            s_cnt[e * p.W + r] = total;
            if (r == peer) {
                for (int w = 0; w < kWarpsPerBlock; ++w) { const int n = s_run[w * p.El + e]; s_run[w * p.El + e] = before; before += n; }
            }
        }
    } else {
        for (int i = threadIdx.x; i < p.El * p.W; i += kBlockThreads) s_cnt[i] = p.cnt[i];
        const int* start = p.chunk_hist + static_cast<size_t>(gchunk) * p.El;
        for (int e = lane; e < p.El; e += 32) run[e] = start[e];
    }
    __syncthreads();
    // padded rows per expert -> exclusive scan over experts (block-wide, El <= 1024)
    int carry = 0;
    for (int e0 = 0; e0 < p.El; e0 += kBlockThreads) {
        const int e = e0 + threadIdx.x;
        int padded = 0;
        if (e < p.El) {
            int tot = 0;
            for (int r = 0; r < p.W; ++r) tot += s_cnt[e * p.W + r];
            padded = (tot + kPad - 1) / kPad * kPad;
            if (blockIdx.x == 0) p.tokens_per_expert[e] = padded;
        }
        int incl = padded;
#pragma unroll
        for (int off = 1; off < 32; off <<= 1) {
            const int n = __shfl_up_sync(0xffffffffu, incl, off);
            if (lane >= off) incl += n;
        }
        if (lane == 31) s_warp_tot[warp] = incl;
        __syncthreads();
        int warp_off = 0, block_tot = 0;
        for (int w = 0; w < kWarpsPerBlock; ++w) {
            if (w < warp) warp_off += s_warp_tot[w];
            block_tot += s_warp_tot[w];
        }
        if (e < p.El) s_base[e] = carry + warp_off + incl - padded;
        carry += block_tot;
        __syncthreads();
    }
    if (blockIdx.x == 0 && threadIdx.x == 0) {
        p.num_tokens[0] = carry;
        if (carry > p.capacity) report_status(p.status, MOK_STATUS_SCHEDULE_OVERFLOW, carry);
    }

    // the chunk's routes in order: virtual thread by virtual thread, each one's routes ascending
    const unsigned lt_mask = (1u << lane) - 1u;
    constexpr int kAhead = 4;                                 // loads in flight per lane
    for (int vt = v0; vt < v0 + kChunkVts; ++vt) {
        for (long long base = vt; base < p.R; base += kAhead * 32 * kVThreads) {
            int es[kAhead];
#pragma unroll
            for (int u = 0; u < kAhead; ++u) {
                const long long r = base + (u * 32 + lane) * kVThreads;
                es[u] = r < p.R ? local_expert(routes[r], first, p.El) : -1;
            }
#pragma unroll
            for (int u = 0; u < kAhead; ++u) {
                const int e = es[u];
                const unsigned same = __match_any_sync(0xffffffffu, e);
                int before = 0;
                if (e >= 0) {
                    before = run[e];
                    const int j = before + __popc(same & lt_mask);
                    int dst = s_base[e];
                    if (p.W == 1) {
                        dst += j;
                    } else {
                        for (int rr = 0; rr < p.W; ++rr) {
                            const int c = s_cnt[e * p.W + rr];
                            dst += min(c, j) + ((rr < peer && c > j) ? 1 : 0);
                        }
                    }
                    if (dst < p.capacity) {
                        p.peer_rank[dst] = peer;
                        p.peer_token_idx[dst] = static_cast<int>(base) + (u * 32 + lane) * kVThreads;
                    }
                }
                __syncwarp();
                if (e >= 0 && (same & lt_mask) == 0) run[e] = before + __popc(same);   // lowest lane of each group
                __syncwarp();
            }
        }
    }
}

}  // namespace
}  // namespace mok

extern "C" size_t mok_schedule_scratch_bytes(int ep_size, int num_local_experts) {
    if (ep_size <= 0 || num_local_experts <= 0) return 0;
    return (static_cast<size_t>(ep_size) * mok::kChunks * num_local_experts +
            static_cast<size_t>(ep_size) * num_local_experts) * sizeof(int);
}

namespace mok {
// dynamic shared memory of the two kernels
constexpr size_t count_smem(int El, bool fused) { return static_cast<size_t>(fused ? 1 : kWarpsPerBlock) * El * sizeof(int); }
constexpr size_t place_smem(int El, int W) { return (static_cast<size_t>(El) * W + El + static_cast<size_t>(kWarpsPerBlock) * El) * sizeof(int); }

template <class Id, bool kFused>
int launch_schedule_as(const SchedParams& p, cudaStream_t stream) {
    // The dynamic shared-memory ceiling is a sticky per-device attribute: set it once to what the largest accepted
    // problem needs, so that concurrent calls with different expert counts cannot lower it under one another.
    static std::atomic<bool> configured[64];
    int dev = 0;
    MOK_CUDA_CHECK(cudaGetDevice(&dev));
    if (dev < 0 || dev >= 64 || !configured[dev].load(std::memory_order_acquire)) {
        MOK_CUDA_CHECK(cudaFuncSetAttribute(sched_count_kernel<Id, kFused>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                            static_cast<int>(count_smem(MOK_MAX_LOCAL_EXPERTS, false))));
        MOK_CUDA_CHECK(cudaFuncSetAttribute(sched_place_kernel<Id, kFused>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                            static_cast<int>(place_smem(MOK_MAX_LOCAL_EXPERTS, MOK_MAX_PEERS))));
        if (dev >= 0 && dev < 64) configured[dev].store(true, std::memory_order_release);
    }
    const int chunk_blocks = p.W * kBlocksPerPeer;
    ProfScope prof(kSlotScheduler, stream, kFused ? 2 : 3);
    // enough blocks to clear the tables at a few KB each, at most one per SM beyond the counting ones
    const int clear_blocks = std::min(device_sm_count(), (p.capacity / 4 + kBlockThreads - 1) / kBlockThreads);
    MOK_TRY(launch_kernel(sched_count_kernel<Id, kFused>, std::max(chunk_blocks, clear_blocks), kBlockThreads, count_smem(p.El, kFused),
                          stream, false, kFused, p));
    if (!kFused) {
        const int pair_blocks = (p.El * p.W + kWarpsPerBlock - 1) / kWarpsPerBlock;
        MOK_TRY(launch_kernel(sched_scan_kernel, pair_blocks, kBlockThreads, 0, stream, false, false, p));
    }
    return launch_kernel(sched_place_kernel<Id, kFused>, chunk_blocks, kBlockThreads, place_smem(p.El, p.W), stream, false, kFused, p);
}

// shared by the entry points; `scratch` is a device pointer, `id_bytes` the width of a route
int launch_schedule(const void* topk_all, int id_bytes, int ep_size, int num_local_tokens, int topk,
                    int num_local_experts, int schedule_capacity, int rank,
                    int32_t* schedule_peer_rank, int32_t* schedule_peer_token_idx,
                    int32_t* num_tokens, int32_t* tokens_per_expert,
                    void* scratch, int32_t* status, cudaStream_t stream) {
    SchedParams p;
    p.topk = topk_all;
    p.W = ep_size;
    p.R = num_local_tokens * topk;
    p.El = num_local_experts;
    p.rank = rank;
    p.capacity = schedule_capacity;
    p.peer_rank = schedule_peer_rank;
    p.peer_token_idx = schedule_peer_token_idx;
    p.num_tokens = num_tokens;
    p.tokens_per_expert = tokens_per_expert;
    p.chunk_hist = static_cast<int*>(scratch);
    p.cnt = p.chunk_hist + static_cast<size_t>(ep_size) * kChunks * num_local_experts;
    p.status = status;
    auto aligned = [](const void* ptr) { return reinterpret_cast<uintptr_t>(ptr) % 16 == 0; };
    p.vec_routes = aligned(topk_all) && p.R % 4 == 0;        // a peer's routes start R ids after the previous one's
    p.vec_tables = aligned(schedule_peer_rank) && aligned(schedule_peer_token_idx);
    const bool fused = ep_size * num_local_experts <= kMaxFusedPairs;
    if (id_bytes == 8) return fused ? launch_schedule_as<long long, true>(p, stream) : launch_schedule_as<long long, false>(p, stream);
    return fused ? launch_schedule_as<int, true>(p, stream) : launch_schedule_as<int, false>(p, stream);
}
}  // namespace mok

namespace {
int schedule_with_scratch(const void* topk_all, int id_bytes, int ep_size, int num_local_tokens, int topk, int num_local_experts,
                          int schedule_capacity, int rank, int32_t* schedule_peer_rank, int32_t* schedule_peer_token_idx,
                          int32_t* num_tokens, int32_t* tokens_per_expert, void* scratch, size_t scratch_bytes, int32_t* status,
                          void* stream) {
    if (!topk_all || !schedule_peer_rank || !schedule_peer_token_idx || !num_tokens || !tokens_per_expert || !scratch)
        return MOK_ERR_INVALID;
    if (ep_size < 1 || ep_size > MOK_MAX_PEERS || rank < 0 || rank >= ep_size) return MOK_ERR_INVALID;
    if (num_local_tokens <= 0 || topk <= 0 || schedule_capacity <= 0) return MOK_ERR_INVALID;
    if (num_local_experts < 1 || num_local_experts > MOK_MAX_LOCAL_EXPERTS) return MOK_ERR_INVALID;
    if (scratch_bytes < mok_schedule_scratch_bytes(ep_size, num_local_experts)) return MOK_ERR_INVALID;
    return mok::launch_schedule(topk_all, id_bytes, ep_size, num_local_tokens, topk, num_local_experts, schedule_capacity, rank,
                                schedule_peer_rank, schedule_peer_token_idx, num_tokens, tokens_per_expert,
                                scratch, status, static_cast<cudaStream_t>(stream));
}
}  // namespace

extern "C" int mok_schedule(const int32_t* topk_all, int ep_size, int num_local_tokens, int topk,
                            int num_local_experts, int schedule_capacity, int rank,
                            int32_t* schedule_peer_rank, int32_t* schedule_peer_token_idx,
                            int32_t* num_tokens, int32_t* tokens_per_expert,
                            void* scratch, size_t scratch_bytes, int32_t* status, void* stream) {
    return schedule_with_scratch(topk_all, 4, ep_size, num_local_tokens, topk, num_local_experts, schedule_capacity, rank,
                                 schedule_peer_rank, schedule_peer_token_idx, num_tokens, tokens_per_expert, scratch, scratch_bytes,
                                 status, stream);
}

extern "C" int mok_schedule_i64(const int64_t* topk_all, int ep_size, int num_local_tokens, int topk,
                                int num_local_experts, int schedule_capacity, int rank,
                                int32_t* schedule_peer_rank, int32_t* schedule_peer_token_idx,
                                int32_t* num_tokens, int32_t* tokens_per_expert,
                                void* scratch, size_t scratch_bytes, int32_t* status, void* stream) {
    return schedule_with_scratch(topk_all, 8, ep_size, num_local_tokens, topk, num_local_experts, schedule_capacity, rank,
                                 schedule_peer_rank, schedule_peer_token_idx, num_tokens, tokens_per_expert, scratch, scratch_bytes,
                                 status, stream);
}

// ---------------------------------------------------------------------------------------------
// Scheduler variant for callers that must not allocate device memory.
//
// Some hosts of this library run under a fixed memory plan: an inference server that sized its
// arena at start-up, a real-time loop where cudaMalloc's implicit device synchronisation is not
// acceptable, or a plug-in boundary that hands out no allocator at all.  Such a caller cannot
// provide the chunk-histogram scratch mok_schedule() asks for.  This entry point keeps that
// scratch in a fixed array inside the library image instead, so the call needs nothing beyond the
// caller's inputs and outputs.
//
// The array is a file-scope __device__ object: every GPU that loads the library carries it
// (kStaticScratchBytes) until the process exits.  In host code its name is only a handle, not a
// device address, so the address is looked up with cudaGetSymbolAddress once per device, with that
// device current, on the first call made on that device; later calls reuse the cached address.
// That first call should therefore be made outside any stream capture.
//
// All calls on one GPU share the array.  The kernels overwrite every element they later read, so
// nothing has to be cleared between calls, but two calls whose kernels overlap on the GPU (two
// streams, or two threads) race on it: run them one after the other.
// ---------------------------------------------------------------------------------------------
namespace mok {
namespace {
constexpr size_t kStaticScratchBytes = 4u << 20;   // enough for ep_size * num_local_experts <= 4080
static __device__ __align__(256) unsigned char g_static_sched_scratch[kStaticScratchBytes];
std::atomic<void*> g_static_scratch_addr[64];    // per device; two threads that race on the first call store the same address

int static_scratch_for_current_device(void** out) {
    int dev = -1;
    MOK_CUDA_CHECK(cudaGetDevice(&dev));
    if (dev < 0 || dev >= 64) return MOK_ERR_UNSUPPORTED;
    void* ptr = g_static_scratch_addr[dev].load(std::memory_order_acquire);
    if (ptr == nullptr) {
        const cudaError_t err = cudaGetSymbolAddress(&ptr, g_static_sched_scratch);
        if (err != cudaSuccess || ptr == nullptr) { note_cuda_error(err, __FILE__, __LINE__); return MOK_ERR_CUDA; }
        g_static_scratch_addr[dev].store(ptr, std::memory_order_release);
    }
    *out = ptr;
    return MOK_OK;
}
}  // namespace
}  // namespace mok

extern "C" size_t mok_schedule_static_max_scratch_bytes(void) { return mok::kStaticScratchBytes; }

extern "C" int mok_schedule_static(const int32_t* topk_all, int ep_size, int num_local_tokens, int topk,
                                   int num_local_experts, int schedule_capacity, int rank,
                                   int32_t* schedule_peer_rank, int32_t* schedule_peer_token_idx,
                                   int32_t* num_tokens, int32_t* tokens_per_expert, int32_t* status, void* stream) {
    if (!topk_all || !schedule_peer_rank || !schedule_peer_token_idx || !num_tokens || !tokens_per_expert)
        return MOK_ERR_INVALID;
    if (ep_size < 1 || ep_size > MOK_MAX_PEERS || rank < 0 || rank >= ep_size) return MOK_ERR_INVALID;
    if (num_local_tokens <= 0 || topk <= 0 || schedule_capacity <= 0) return MOK_ERR_INVALID;
    if (num_local_experts < 1 || num_local_experts > MOK_MAX_LOCAL_EXPERTS) return MOK_ERR_INVALID;
    if (mok_schedule_scratch_bytes(ep_size, num_local_experts) > mok::kStaticScratchBytes) return MOK_ERR_TOO_LARGE;
    void* scratch = nullptr;
    const int rc = mok::static_scratch_for_current_device(&scratch);
    if (rc != MOK_OK) return rc;
    return mok::launch_schedule(topk_all, 4, ep_size, num_local_tokens, topk, num_local_experts, schedule_capacity, rank,
                                schedule_peer_rank, schedule_peer_token_idx, num_tokens, tokens_per_expert,
                                scratch, status, static_cast<cudaStream_t>(stream));
}
