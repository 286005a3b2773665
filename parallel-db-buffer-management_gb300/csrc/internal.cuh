// internal.cuh -- host/device internals shared by the libpbm translation units.
#pragma once
#include <cuda_runtime.h>
#include <atomic>
#include <memory>
#include <mutex>
#include <vector>
#include <cstdint>
#include <cstdio>

#include "pbm.h"
#include "pbm/pbm_device.cuh"

namespace pbm {

// Invariant-check counters.
struct CheckCounters {
    unsigned long long ok, failed, out_of_range, duplicates, not_marked, used;
};

extern std::atomic<unsigned long long> g_launches;
inline void count_launch(unsigned long long n = 1) { g_launches.fetch_add(n, std::memory_order_relaxed); }

int sm_count();
bool device_writable(const void* p);

constexpr uint32_t kDefaultMaxSteps = 4096;

// Sum of a value over the warp by shuffles (every lane calls converged; every lane gets it).
__device__ __forceinline__ unsigned long long warp_total_wide(unsigned long long v) {
#pragma unroll
    for (int d = 16; d > 0; d >>= 1) v += __shfl_xor_sync(0xffffffffu, v, d);
    return v;
}

// Adds every thread's N counters to dst[0..N) with one global atomic per
// counter per block: each warp leaves its sums in shared memory and, after the block's
// one barrier, thread k adds up counter k.  The warp's sums take one 32-bit reduction
// each; values too large for that (one vote for all the counters) take the shuffles, in a
// branch of their own: with a vote and a branch per counter the code between the
// reductions cost the end of a short kernel 1 us (claim, write and free of 32,768
// pages 15.6 against 14.4 us, eight buffer-manager rounds 119 against 116).  Every
// thread of the block calls it once (after its loop, converged); blocks whose size is
// not a multiple of 32 (one-thread replays) add directly.  Per-thread atomics on a
// shared counter would serialise on one L2 address (~1.5 G/s).
template <int N>
__device__ __forceinline__ void block_add_counters(const unsigned long long (&v)[N],
                                                   unsigned long long* const (&dst)[N]) {
    if (blockDim.x & 31u) {
        for (int k = 0; k < N; ++k)
            if (v[k]) atomicAdd(dst[k], v[k]);
        return;
    }
    __shared__ unsigned long long sh[32][N];
    unsigned long long all = 0ull;
#pragma unroll
    for (int k = 0; k < N; ++k) all |= v[k];
    const bool wide = __any_sync(0xffffffffu, (all >> 27) != 0ull);
    if (!wide) {
#pragma unroll
        for (int k = 0; k < N; ++k) {
            const uint32_t x = __reduce_add_sync(0xffffffffu, (uint32_t)v[k]);
            if ((threadIdx.x & 31u) == 0u) sh[threadIdx.x >> 5][k] = x;
        }
    } else {
#pragma unroll
        for (int k = 0; k < N; ++k) {
            const unsigned long long x = warp_total_wide(v[k]);
            if ((threadIdx.x & 31u) == 0u) sh[threadIdx.x >> 5][k] = x;
        }
    }
    __syncthreads();
    if (threadIdx.x < (unsigned)N) {
        unsigned long long x = 0ull;
        for (uint32_t w = 0; w < blockDim.x >> 5; ++w) x += sh[w][threadIdx.x];
        if (x) atomicAdd(dst[threadIdx.x], x);
    }
}

// Programmatic dependent launch.  A kernel launched with launch_next may be set up and
// get its blocks onto the SMs while the kernel before it in the stream still runs;
// it calls stream_wait() before its first access to global memory, which returns once
// that kernel has ended and its writes are visible (at once after an ordinary
// predecessor), and then lets the kernel after it do the same.  Because the kernel before may
// still write while this one is alive, nothing it could write is read with __ldg or
// through a const __restrict__ pointer, which promise data that never changes in the
// kernel's lifetime.  Most calls here are
// kernels of 3-20 us launched one after another, and the start of a launch is 2-3 us of
// each.  Measured on GB300, a call and the calls after it in a stream: 32 claims + frees
// 8.2 -> 6.3 us; claim, read and free of 16,384 pages 18.5 -> 12.7; eight
// buffer-manager rounds of 131,072 fetches 157 -> 136; with 4 KiB copies 205 -> 168.
__device__ __forceinline__ void stream_wait() {
    asm volatile("griddepcontrol.wait;" ::: "memory");
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
}

template <typename... P, typename... A>
inline cudaError_t launch_next_if(bool overlap, void (*kernel)(P...), unsigned grid, unsigned block, size_t smem,
                                  cudaStream_t s, A&&... args) {
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3(grid);
    cfg.blockDim = dim3(block);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = s;
    cudaLaunchAttribute at{};
    at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at.val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = &at;
    cfg.numAttrs = overlap ? 1 : 0;
    return cudaLaunchKernelEx(&cfg, kernel, P(args)...);
}

template <typename... P, typename... A>
inline cudaError_t launch_next(void (*kernel)(P...), unsigned grid, unsigned block, size_t smem, cudaStream_t s,
                               A&&... args) {
    return launch_next_if(true, kernel, grid, block, smem, s, args...);
}

// Copies the first `bytes` bytes of rows ids[0 .. n) of a table (row i at base + i *
// stride, n_rows rows; zeros for ids that name none) to out, row after row.  V: int4
// where addresses, stride and size are multiples of 16, else int32_t.  One piece per
// thread, the grid as large as the work.  Measured on GB300, 16,384 rows of 256
// bytes: 9 -> 4 us a launch, which spent most of it on 64-bit divisions per 4 bytes.
template <typename V>
__global__ void __launch_bounds__(256) k_gather_rows(const char* base, size_t stride, uint32_t n_rows, const int32_t* ids,
                                                     uint32_t n, uint32_t per_row, V* out) {
    stream_wait();
    const unsigned long long total = (unsigned long long)n * per_row;
    const unsigned long long step = (unsigned long long)gridDim.x * blockDim.x;
    for (unsigned long long i = (unsigned long long)blockIdx.x * blockDim.x + threadIdx.x; i < total; i += step) {
        const uint32_t r = total <= 0xffffffffull ? (uint32_t)i / per_row : (uint32_t)(i / per_row);
        const uint32_t k = (uint32_t)(i - (unsigned long long)r * per_row);
        const int32_t id = ids[r];
        V v{};
        if (id >= 0 && (uint32_t)id < n_rows) v = reinterpret_cast<const V*>(base + (size_t)(uint32_t)id * stride)[k];
        out[i] = v;
    }
}

inline cudaError_t gather_rows(const char* base, size_t stride, uint32_t n_rows, const int32_t* d_ids, uint32_t n,
                               uint32_t bytes, int32_t* d_out, cudaStream_t s) {
    const bool wide = (((uintptr_t)base | (uintptr_t)d_out | stride | bytes) & 15u) == 0u;
    const uint32_t per_row = bytes / (wide ? 16u : 4u);
    const unsigned long long blocks = ((unsigned long long)n * per_row + 255ull) / 256ull;
    const unsigned grid = (unsigned)(blocks < (1ull << 20) ? blocks : (1ull << 20));
    return wide ? launch_next(k_gather_rows<int4>, grid, 256, 0, s, base, stride, n_rows, d_ids, n, per_row, (int4*)d_out)
                : launch_next(k_gather_rows<int32_t>, grid, 256, 0, s, base, stride, n_rows, d_ids, n, per_row, d_out);
}

// Makes a device current for the rest of the calling scope and restores the
// caller's device when the scope ends.  Every entry point that takes a pool
// (or an object built on one) opens one with the pool's device, so a process
// may hold one pool per GPU and call into any of them from any current
// device.  A negative ordinal (no pool) switches nothing.
struct DeviceScope {
    int prev = -1;
    bool switched = false;
    explicit DeviceScope(int dev) {
        if (dev >= 0 && cudaGetDevice(&prev) == cudaSuccess && prev != dev && cudaSetDevice(dev) == cudaSuccess)
            switched = true;
    }
    ~DeviceScope() {
        if (switched) cudaSetDevice(prev);
    }
    DeviceScope(const DeviceScope&) = delete;
    DeviceScope& operator=(const DeviceScope&) = delete;
};

// Workspaces of a pool's fail-fast launches: a launch of one stream may run beside one of
// another.  kBudgetSlots of them go round; a launch that gets one last used in
// another stream waits for that launch's end.  A launch under capture has one that goes
// back when the graph that was captured, and every graph made of it, is gone: at first
// there are kBudgetCaptures of those, and as many more come with each device allocation.
constexpr uint32_t kBudgetSlots = 8, kBudgetCaptures = 24, kBudgetSpaces = kBudgetSlots + kBudgetCaptures;
struct BudgetSlot {
    cudaEvent_t done;
    unsigned long long stream;   // id of the stream that used it last
    bool used;
};
struct BudgetSpace {
    LaunchBudget* budget;         // free pages at launch start
    unsigned long long* counts;   // free pages per block slice of the budget pass
};
// The captured launches' workspaces.  The graphs that hold some may outlive the pool, so each
// shares this list; the device memory goes with the pool.
struct BudgetCaptureSpaces {
    std::mutex mu;
    std::vector<BudgetSpace> unused;   // room for all of them reserved: returning one cannot fail
    size_t total = 0;
    std::vector<char*> chunks;
};

// Stretches of the single clock's sweep that blocks took and did not need (see k_alloc_clock),
// first in, first out: position and length in one word, 0 = empty.  Half of the slots are
// for the blocks that find room at the same moment, 32 an SM at most; a stretch that finds
// no room is passed until the arm comes round.
constexpr uint32_t kClockSlots = 16384;
struct ClockList {
    alignas(128) unsigned long long head;    // next ticket to take
    alignas(128) unsigned long long tail;    // next ticket to fill
    alignas(128) unsigned long long avail;   // filled slots
    alignas(128) unsigned long long slot[kClockSlots];
};

constexpr int kDefaultBlock = 256;
constexpr int kCappedBlocks = 5;   // resident blocks the register-capped batch kernels are built for

}  // namespace pbm

struct pbm_pool {
    pbm::PoolView view;
    uint64_t n_pages;
    uint32_t page_size;
    uint32_t flags;
    uint32_t max_slots;
    size_t bitmap_bytes;            // n_words32 (even) * 4
    uint64_t padding_bits;          // set bits past n_pages
    uint32_t* d_words;
    char* d_base;
    pbm::DevStats* d_stats;
    int32_t* d_cursors;             // clustered walk, per slot
    uint32_t* d_arms;               // distributed clock, per slot
    unsigned long long* d_arm;      // single clock
    pbm::ClockList* d_clock_list;
    int32_t* d_ring;                // FIFO ring, n_pages entries (lazily built)
    pbm::FifoState* d_fifo;
    bool fifo_valid;
    uint32_t* d_seen;               // check scratch: one bit per page
    pbm::CheckCounters* d_check;
    unsigned long long* d_scan;     // scratch for prefix sums (per-block partials)
    unsigned long long* d_prefix;   // batch prefix (n_groups + 1)
    // fail-fast launches: one workspace per launch (see budget_prepare)
    std::mutex budget_mu;
    pbm::BudgetSlot budget_slots[pbm::kBudgetSlots];
    uint32_t budget_next;
    pbm::BudgetSpace budget_space[pbm::kBudgetSlots];
    std::shared_ptr<pbm::BudgetCaptureSpaces> budget_captures;
    uint64_t list_cap;              // free pages up to which the budget pass may hand them out itself
    uint32_t budget_blocks;
    uint32_t prefix_cap;
    int device;
};

#define PBM_CUDA_TRY(expr)                                                          \
    do {                                                                            \
        cudaError_t _e = (expr);                                                    \
        if (_e != cudaSuccess) {                                                    \
            std::fprintf(stderr, "[pbm] %s failed: %s (%s:%d)\n", #expr,           \
                         cudaGetErrorString(_e), __FILE__, __LINE__);               \
            cudaGetLastError(); /* do not leave the error for the next caller */   \
            return PBM_ERR_CUDA;                                                    \
        }                                                                           \
    } while (0)

#define PBM_ON_POOL_DEVICE(pool) pbm::DeviceScope pbm_device_scope_((pool) ? (pool)->device : -1)

#define PBM_LAUNCH_CHECK()                                                          \
    do {                                                                            \
        cudaError_t _e = cudaGetLastError();                                        \
        if (_e != cudaSuccess) {                                                    \
            std::fprintf(stderr, "[pbm] launch failed: %s (%s:%d)\n",              \
                         cudaGetErrorString(_e), __FILE__, __LINE__);               \
            return PBM_ERR_CUDA;                                                    \
        }                                                                           \
        pbm::count_launch();                                                        \
    } while (0)

namespace pbm {
// Implemented in pool.cu
int fifo_build(pbm_pool* pool, cudaStream_t s);
int popcount_used(pbm_pool* pool, uint64_t* used, cudaStream_t s);
// Counts the pool's free pages into *budget on stream s (no sync); a launch of
// n_requests that asks for at least half of them is served in order by the same
// pass (list mode).  *slot is for budget_launched.
int budget_prepare(pbm_pool* pool, uint32_t n_requests, int32_t* d_ids, int32_t* d_steps, cudaStream_t s,
                   LaunchBudget** budget, uint32_t* slot);
int budget_launched(pbm_pool* pool, uint32_t slot, cudaStream_t s);
}  // namespace pbm
