// pool.cu -- page pool lifecycle, prefill, occupancy, snapshots, invariant
// checks and the free-list build.
//
// Reference counterparts: initPages/pageAddress/getPageID (source/Paging.cuh:30-85),
// initMemoryManagement/resetMemoryManager/getFreePagePercentage/prefillBuffer
// (source/RandomWalkBasic_BM.cuh:42-164 and copies), popc_kernel + cub sum
// (RandomWalkBasic_BM.cuh:109-145).
#include <cstdlib>
#include <cstring>
#include <new>

#include <atomic>

#include <algorithm>

#include "internal.cuh"

namespace pbm {

std::atomic<unsigned long long> g_launches{0};

// SM count of the current device, cached per device ordinal (one atomic
// word each, so host threads launching at once never see a torn value).
int sm_count() {
    static std::atomic<int> cached[64];
    int dev = 0;
    cudaGetDevice(&dev);
    std::atomic<int>* slot = (dev >= 0 && dev < 64) ? &cached[dev] : nullptr;
    int c = slot ? slot->load(std::memory_order_relaxed) : 0;
    if (!c) {
        int n = 0;
        cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev);
        c = n > 0 ? n : 1;
        if (slot) slot->store(c, std::memory_order_relaxed);
    }
    return c;
}

// Whether a kernel may write p: device or managed memory, or host memory that
// is pinned and mapped (cudaHostAlloc, cudaHostRegister).  Plain pageable host
// memory is refused, so a wrong buffer is an error status and never a kernel
// touching an unmapped address.
bool device_writable(const void* p) {
    cudaPointerAttributes at{};
    if (cudaPointerGetAttributes(&at, p) != cudaSuccess) {
        cudaGetLastError();
        return false;
    }
    if (at.type == cudaMemoryTypeDevice || at.type == cudaMemoryTypeManaged) return true;
    return at.type == cudaMemoryTypeHost && at.devicePointer == p;
}

// Bernoulli(occ) bitmap: one thread per 32-bit word, one hash per page.
__global__ void k_prefill(uint32_t* words, uint32_t n_words, uint64_t n_pages,
                          uint64_t thresh53, uint64_t seed) {
    for (uint64_t w = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; w < n_words;
         w += (uint64_t)gridDim.x * blockDim.x) {
        uint32_t val = 0;
        uint64_t p0 = (uint64_t)w * 32u;
#pragma unroll 8
        for (uint32_t b = 0; b < 32; ++b) {
            uint64_t p = p0 + b;
            bool held = p >= n_pages || (hash64(seed, p) >> 11) < thresh53;
            val |= (uint32_t)held << b;
        }
        words[w] = val;
    }
}

// Padding bits only (reset): clear every word, then set bits >= n_pages.
__global__ void k_reset_words(uint32_t* words, uint32_t n_words, uint64_t n_pages) {
    for (uint64_t w = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; w < n_words;
         w += (uint64_t)gridDim.x * blockDim.x) {
        uint64_t p0 = (uint64_t)w * 32u;
        uint32_t val = 0;
        if (p0 + 32u > n_pages) {
            for (uint32_t b = 0; b < 32; ++b) if (p0 + b >= n_pages) val |= 1u << b;
        }
        words[w] = val;
    }
}

// Sets the padding bits (pages >= n_pages) of the last words again, e.g.
// after a caller wrote the bitmap: the walks rely on them never being free.
__global__ void k_set_padding(uint32_t* words, uint32_t n_words, uint64_t n_pages) {
    const uint32_t w = (uint32_t)(n_pages >> 5) + threadIdx.x;
    if (w >= n_words) return;
    const uint64_t p0 = (uint64_t)w * 32u;
    uint32_t pad = 0;
    for (uint32_t b = 0; b < 32; ++b) if (p0 + b >= n_pages) pad |= 1u << b;
    if (pad) words[w] |= pad;
}

__device__ __forceinline__ unsigned long long warp_sum64(unsigned long long v) {
#pragma unroll
    for (int d = 16; d > 0; d >>= 1) v += __shfl_down_sync(0xffffffffu, v, d);
    return v;  // valid in lane 0
}

// Block-wide sum (blockDim.x a multiple of 32, <= 1024); result in thread 0.
__device__ __forceinline__ unsigned long long block_sum(unsigned long long v) {
    __shared__ unsigned long long red[32];
    v = warp_sum64(v);
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    if (lane == 0) red[warp] = v;
    __syncthreads();
    unsigned long long t = 0;
    if (warp == 0) {
        t = lane < (int)(blockDim.x >> 5) ? red[lane] : 0ull;
        t = warp_sum64(t);
    }
    __syncthreads();
    return t;
}

// Fused popcount-reduce over the bitmap (one pass, 64-bit words).
__global__ void k_popcount(const unsigned long long* words, uint32_t n_words64,
                           unsigned long long* out) {
    unsigned long long c = 0;
    for (uint64_t w = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; w < n_words64;
         w += (uint64_t)gridDim.x * blockDim.x)
        c += (unsigned long long)__popcll(__ldcg(words + w));
    c = block_sum(c);
    if (threadIdx.x == 0 && c) atomicAdd(out, c);
}

// Invariant check of an id list: range, duplicates (scratch bitmap `seen`),
// and that every returned page is marked held.
__global__ void k_check_ids(const uint32_t* words, uint32_t* seen, uint64_t n_pages,
                            const int32_t* ids, uint32_t n, CheckCounters* out) {
    unsigned long long ok = 0, failed = 0, oor = 0, dup = 0, unmarked = 0;
    for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (uint64_t)gridDim.x * blockDim.x) {
        int32_t id = ids[i];
        if (id == -1) { ++failed; continue; }
        if (id < 0 || (uint64_t)id >= n_pages) { ++oor; continue; }
        ++ok;
        uint32_t w = (uint32_t)id >> 5, bit = 1u << ((uint32_t)id & 31u);
        if (atomicOr(seen + w, bit) & bit) ++dup;
        if (!(__ldcg(words + w) & bit)) ++unmarked;
    }
    ok = block_sum(ok);
    failed = block_sum(failed);
    oor = block_sum(oor);
    dup = block_sum(dup);
    unmarked = block_sum(unmarked);
    if (threadIdx.x == 0) {
        if (ok) atomicAdd(&out->ok, ok);
        if (failed) atomicAdd(&out->failed, failed);
        if (oor) atomicAdd(&out->out_of_range, oor);
        if (dup) atomicAdd(&out->duplicates, dup);
        if (unmarked) atomicAdd(&out->not_marked, unmarked);
    }
}

// ---- free-list build: the FIFO ring holds the free pages in ascending order ----
// pass 1: free pages per block of 32-bit words
__global__ void k_fifo_count(const uint32_t* words, uint32_t n_words, uint32_t words_per_block,
                             unsigned long long* counts) {
    uint32_t w0 = blockIdx.x * words_per_block;
    unsigned long long c = 0;
    for (uint32_t w = w0 + threadIdx.x; w < n_words && w < w0 + words_per_block; w += blockDim.x)
        c += (unsigned long long)__popc(~__ldcg(words + w));
    c = block_sum(c);
    if (threadIdx.x == 0) counts[blockIdx.x] = c;
}
// pass 2: exclusive scan of the per-block counts (one block)
__global__ void k_fifo_scan(unsigned long long* counts, uint32_t n_blocks, FifoState* st,
                            int32_t* ring, uint64_t n_pages) {
    if (threadIdx.x == 0) {
        unsigned long long acc = 0;
        for (uint32_t b = 0; b < n_blocks; ++b) {
            unsigned long long c = counts[b];
            counts[b] = acc;
            acc += c;
        }
        st->head = 0;
        st->tail = acc;
        st->avail = acc;
    }
}
// pass 3: each block writes its free pages; the rest of the ring is empty (-1)
__global__ void k_fifo_fill(const uint32_t* words, uint32_t n_words, uint32_t words_per_block,
                            const unsigned long long* offs, int32_t* ring, uint64_t n_pages) {
    uint32_t w0 = blockIdx.x * words_per_block;
    __shared__ unsigned long long base;
    if (threadIdx.x == 0) base = offs[blockIdx.x];
    __syncthreads();
    // sequential within the block by warps of words, ordered by word index
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nwarps = blockDim.x >> 5;
    __shared__ unsigned long long warp_base[32];
    for (uint32_t chunk = w0; chunk < w0 + words_per_block && chunk < n_words;
         chunk += (uint32_t)nwarps * 32u) {
        uint32_t w = chunk + (uint32_t)warp * 32u + (uint32_t)lane;
        uint32_t fr = (w < n_words && w < w0 + words_per_block) ? ~__ldcg(words + w) : 0u;
        int c = __popc(fr);
        int incl = c;
        for (int d = 1; d < 32; d <<= 1) {
            int y = __shfl_up_sync(0xffffffffu, incl, d);
            if (lane >= d) incl += y;
        }
        if (lane == 31) warp_base[warp] = (unsigned long long)incl;
        __syncthreads();
        if (threadIdx.x == 0) {
            unsigned long long acc = base;
            for (int i = 0; i < nwarps; ++i) { unsigned long long t = warp_base[i]; warp_base[i] = acc; acc += t; }
            base = acc;
        }
        __syncthreads();
        unsigned long long pos = warp_base[warp] + (unsigned long long)(incl - c);
        while (fr) {
            int b = __ffs((int)fr) - 1;
            fr &= fr - 1u;
            ring[pos++] = (int32_t)(w * 32u + (uint32_t)b);
        }
        __syncthreads();
    }
}
__global__ void k_fifo_clear_tail(int32_t* ring, const FifoState* st, uint64_t n_pages) {
    unsigned long long start = st->tail;
    for (unsigned long long i = start + blockIdx.x * blockDim.x + threadIdx.x; i < n_pages;
         i += (unsigned long long)gridDim.x * blockDim.x)
        ring[i] = -1;
}

int fifo_build(pbm_pool* pool, cudaStream_t s) {
    if (!pool->d_ring) {
        if (cudaMalloc(&pool->d_ring, sizeof(int32_t) * pool->n_pages) != cudaSuccess) {
            cudaGetLastError();
            pool->d_ring = nullptr;
            return PBM_ERR_NOMEM;
        }
    }
    const uint32_t nw = pool->view.n_words32;
    const uint32_t wpb = 4096;
    const uint32_t nb = (nw + wpb - 1) / wpb;
    k_fifo_count<<<nb, 256, 0, s>>>(pool->d_words, nw, wpb, pool->d_scan);
    PBM_LAUNCH_CHECK();
    k_fifo_scan<<<1, 32, 0, s>>>(pool->d_scan, nb, pool->d_fifo, pool->d_ring, pool->n_pages);
    PBM_LAUNCH_CHECK();
    k_fifo_fill<<<nb, 256, 0, s>>>(pool->d_words, nw, wpb, pool->d_scan, pool->d_ring, pool->n_pages);
    PBM_LAUNCH_CHECK();
    k_fifo_clear_tail<<<sm_count() * 4, 256, 0, s>>>(pool->d_ring, pool->d_fifo, pool->n_pages);
    PBM_LAUNCH_CHECK();
    pool->fifo_valid = true;
    return PBM_OK;
}

// ---- fail-fast launch budget ----
// Both passes run at most kBudgetPerSm blocks of kBudgetThreads per SM: 55 warps, the most
// whose stages (4 KiB a warp) the second one's shared memory holds.  A thread takes a word
// at a time, so the time goes up by a step where the pool's words pass a multiple of the
// threads on the chip (17.1 M pages each), and the more threads, the later.  us for a fail-fast launch of a
// quarter of the pages at 90% and its frees, 48 warps an SM (6 blocks of 256) / 54 (6 of 288) / 55 (5 of 352):
//   2^20 pages 13.7 / 13.9 / 14.0    16 M 23.2 / 21.6 / 21.2    2^25 30.7 / 29.2 / 29.1
//   2^22       15.6 / 16.0 / 15.8    17 M 23.5 / 24.1 / 21.3    2^26 45.3 / 44.9 / 45.7
//   12 M       19.3 / 20.1 / 19.7    20 M 24.0 / 24.8 / 24.7    2^27 91.4 / 91.0 / 92.1
constexpr int kBudgetThreads = 352;
constexpr int kBudgetPerSm = 5;

// Pass 1: the free pages (clear bits; padding bits stay set) of each block's
// contiguous slice of `per` 64-bit words, into counts[block].
__global__ void __launch_bounds__(kBudgetThreads) k_free_budget(const unsigned long long* words, uint32_t n_words64, uint32_t per,
                                                     unsigned long long* counts, LaunchBudget* b) {
    stream_wait();
    const uint64_t w0 = (uint64_t)blockIdx.x * per;
    const uint64_t w1 = min((uint64_t)n_words64, w0 + per);
    unsigned long long c = 0;
    for (uint64_t w = w0 + threadIdx.x; w < w1; w += blockDim.x)
        c += (unsigned long long)__popcll(~__ldcg(words + w));
    c = block_sum(c);
    if (threadIdx.x == 0) {
        counts[blockIdx.x] = c;
        if (blockIdx.x == 0) b->lost = 0u;
    }
}

// Pass 2: F, the sum of the counts, and, when the launch asks for at least half of
// the F free pages (and F is below `cap`), the pages themselves: request r takes
// the r-th free page in ascending order.  Each block claims its slice's
// pages word by word with one atomicOr and writes their ids to the requests that
// start at its offset (the counts of the blocks before it); the ids of a warp's 32 words
// go through shared memory so that they leave as whole lines.  A slice gives exactly
// the pages counted in it: pages another stream took since then leave their
// requests kLostPage, which the launch's kernel serves by walking.  Writing
// a list of pages here and taking each page of it with an atomic of its own in that kernel
// moved 8 more bytes per page and took an atomic per page instead of per
// word.  Measured on GB300, 2^22 requests on 2^24 pages at 90% (1.68 M granted) and
// their frees: 63 -> 37 us, 28 with a word per thread here and refusals stored four at
// a time behind it, 23 with the refusals stored here, under way while the words are claimed.
__global__ void __launch_bounds__(kBudgetThreads, kBudgetPerSm) k_take_free(unsigned long long* words, uint32_t n_words64, uint32_t per,
                                                   const unsigned long long* counts, LaunchBudget* b, uint32_t n_requests,
                                                   unsigned long long cap, int32_t* ids, int32_t* steps, DevStats* stats) {
    constexpr uint32_t kWarps = kBudgetThreads / 32;
    __shared__ uint32_t warp_tot[kWarps];
    __shared__ unsigned long long s_sum[2];
    __shared__ uint16_t stage[kWarps][2048];   // per warp: page offsets within its 32 words
    stream_wait();
    unsigned long long off = 0, F = 0;
    for (uint32_t k = threadIdx.x; k < gridDim.x; k += blockDim.x) {
        const unsigned long long c = __ldcg(counts + k);
        F += c;
        if (k < blockIdx.x) off += c;
    }
    F = block_sum(F);
    off = block_sum(off);
    if (threadIdx.x == 0) {
        s_sum[0] = F;
        s_sum[1] = off;
    }
    __syncthreads();
    F = s_sum[0];
    off = s_sum[1];
    const bool mode = 2ull * n_requests >= F && F < cap;
    if (blockIdx.x == 0 && threadIdx.x == 0) {
        b->free_at_start = (long long)F;
        b->list_mode = mode ? 1 : 0;
    }
    if (!mode) return;
    // the requests past the free pages: refused here, their stores under way behind the words'
    if (F < n_requests) {
        const uint32_t nthr = gridDim.x * kBudgetThreads, tid = blockIdx.x * kBudgetThreads + threadIdx.x;
        const uint32_t f = (uint32_t)F, n = n_requests;
        uint32_t lo = f, hi = f;                   // [lo, hi): stored four at a time
        if ((((uintptr_t)ids | (uintptr_t)steps) & 15u) == 0u && n - f >= 8u) {
            lo = (f + 3u) & ~3u;
            hi = n & ~3u;
            for (uint32_t i = (lo >> 2) + tid; i < hi >> 2; i += nthr) {
                reinterpret_cast<int4*>(ids)[i] = make_int4(-1, -1, -1, -1);
                if (steps) reinterpret_cast<int4*>(steps)[i] = make_int4(0, 0, 0, 0);
            }
        }
        for (uint64_t i = tid; i < (lo - f) + (n - hi); i += nthr) {
            const uint64_t r = i < lo - f ? f + i : hi + (i - (lo - f));
            ids[r] = -1;
            if (steps) steps[r] = 0;
        }
        if (tid == 0) atomicAdd(&stats->failures, (unsigned long long)(n - f));
    }
    if (off >= n_requests) return;
    // this slice's requests: off .. off + quota - 1
    const uint32_t quota = (uint32_t)min(__ldcg(counts + blockIdx.x), (unsigned long long)n_requests - off);
    int32_t* out = ids + off;
    const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
    const uint64_t w0 = (uint64_t)blockIdx.x * per;
    const uint64_t w1 = min((uint64_t)n_words64, w0 + per);
    uint32_t done = 0, lost = 0;               // requests behind this chunk (block-uniform); lost: this thread's
    for (uint64_t base = w0; base < w1 && done < quota; base += kBudgetThreads) {
        const uint64_t w = base + threadIdx.x;
        const uint64_t fr = w < w1 ? ~(uint64_t)__ldcg(words + w) : 0ull;
        const int c = __popcll(fr);
        int incl = c;
#pragma unroll
        for (int d = 1; d < 32; d <<= 1) {
            const int y = __shfl_up_sync(kFull32, incl, d);
            if ((int)lane >= d) incl += y;
        }
        if (lane == 31u) warp_tot[warp] = (uint32_t)incl;
        __syncthreads();
        uint32_t before = 0, total = 0;
#pragma unroll
        for (uint32_t i = 0; i < kWarps; ++i) {
            const uint32_t x = warp_tot[i];
            if (i < warp) before += x;
            total += x;
        }
        const uint32_t wpos = done + before;                       // the warp's first request
        const uint32_t wlim = wpos < quota ? min(quota - wpos, warp_tot[warp]) : 0u;   // and how many it has
        const uint32_t excl = (uint32_t)(incl - c);
        uint64_t take = excl < wlim ? low_bits(fr, (int)(wlim - excl)) : 0ull;
        uint64_t gone = 0ull;
        if (take) gone = take & (uint64_t)atomicOr(words + w, (unsigned long long)take);
        // offsets of the taken bits, half a word at a time; a page lost to another stream is marked
        uint16_t* st = stage[warp] + excl;
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            const uint32_t off0 = lane * 64u + 32u * (uint32_t)h;
            for (uint32_t m = (uint32_t)(take >> (32 * h)); m; m &= m - 1u) *st++ = (uint16_t)(off0 + (uint32_t)__ffs((int)m) - 1u);
        }
        if (gone) {
            uint16_t* sg = stage[warp] + excl;
            for (uint64_t m = take; m; m &= m - 1ull, ++sg)
                if (gone & (m & (0ull - m))) *sg = 0xffffu;
            lost += (uint32_t)__popcll(gone);
        }
        __syncwarp();
        const uint32_t page0 = (uint32_t)(base + warp * 32u) * 64u;
        for (uint32_t i = lane; i < wlim; i += 32u) {
            const uint32_t o = stage[warp][i];
            out[wpos + i] = o == 0xffffu ? kLostPage : (int32_t)(page0 + o);
            if (steps) steps[off + wpos + i] = 1;
        }
        done += total;
        __syncthreads();   // warp_tot and the stage are used again
    }
    // pages counted here but gone before they were read
    uint32_t missing = 0;
    for (uint32_t i = done + threadIdx.x; i < quota; i += kBudgetThreads) {
        out[i] = kLostPage;
        ++missing;
    }
    lost += missing;
    const unsigned long long all_lost = block_sum(lost);
    if (threadIdx.x == 0) {
        if (all_lost) atomicAdd(&b->lost, (uint32_t)all_lost);
        const unsigned long long got = quota - all_lost;
        if (got) {
            atomicAdd(&stats->successes, got);
            atomicAdd(&stats->steps, got);
        }
    }
}

namespace {

constexpr size_t kBudgetCounts = 128;   // the counts begin a line of their own
size_t budget_space_bytes(uint32_t blocks) {
    return (kBudgetCounts + sizeof(unsigned long long) * blocks + 255u) & ~(size_t)255u;
}

BudgetSpace budget_space_at(char* base, uint32_t blocks, size_t i) {
    char* p = base + i * budget_space_bytes(blocks);
    return {reinterpret_cast<LaunchBudget*>(p), reinterpret_cast<unsigned long long*>(p + kBudgetCounts)};
}

// Puts the kBudgetCaptures workspaces at `base` among the unused ones; `own`: a device
// allocation that goes with the pool.  False: no host memory.
bool budget_add_captures(BudgetCaptureSpaces& c, char* base, uint32_t blocks, bool own) {
    std::lock_guard<std::mutex> lk(c.mu);
    try {
        c.unused.reserve(c.total + kBudgetCaptures);
        if (own) c.chunks.push_back(base);
    } catch (...) {
        return false;
    }
    c.total += kBudgetCaptures;
    for (uint32_t i = 0; i < kBudgetCaptures; ++i) c.unused.push_back(budget_space_at(base, blocks, i));
    return true;
}

// One of the unused ones, if there is one.
bool budget_take_unused(BudgetCaptureSpaces& c, BudgetSpace* space) {
    std::lock_guard<std::mutex> lk(c.mu);
    if (c.unused.empty()) return false;
    *space = c.unused.back();
    c.unused.pop_back();
    return true;
}

// A workspace held by a graph.
struct BudgetLoan {
    std::shared_ptr<BudgetCaptureSpaces> of;
    BudgetSpace space;
};

// The last graph that held the loan is gone (called by the CUDA runtime, on any thread).
void CUDART_CB budget_return(void* p) {
    BudgetLoan* loan = static_cast<BudgetLoan*>(p);
    {
        std::lock_guard<std::mutex> lk(loan->of->mu);
        loan->of->unused.push_back(loan->space);
    }
    delete loan;
}

// A workspace for a launch captured into `graph`, which holds it from here on.
int budget_borrow(pbm_pool* pool, cudaGraph_t graph, BudgetSpace* space) {
    BudgetCaptureSpaces& c = *pool->budget_captures;
    if (!budget_take_unused(c, space)) {
        char* chunk = nullptr;
        // an allocation is no part of the capture, nor of one in another thread
        cudaStreamCaptureMode mode = cudaStreamCaptureModeRelaxed;
        cudaThreadExchangeStreamCaptureMode(&mode);
        bool ok = cudaMalloc(&chunk, budget_space_bytes(pool->budget_blocks) * kBudgetCaptures) == cudaSuccess;
        if (ok && !budget_add_captures(c, chunk, pool->budget_blocks, true)) {
            cudaFree(chunk);
            ok = false;
        }
        cudaThreadExchangeStreamCaptureMode(&mode);
        if (!ok || !budget_take_unused(c, space)) {
            cudaGetLastError();
            return PBM_ERR_NOMEM;
        }
    }
    BudgetLoan* loan = new (std::nothrow) BudgetLoan{pool->budget_captures, *space};
    if (!loan) {
        std::lock_guard<std::mutex> lk(c.mu);
        c.unused.push_back(*space);
        return PBM_ERR_NOMEM;
    }
    cudaUserObject_t held = nullptr;
    if (cudaUserObjectCreate(&held, loan, budget_return, 1, cudaUserObjectNoDestructorSync) != cudaSuccess) {
        cudaGetLastError();
        budget_return(loan);
        return PBM_ERR_CUDA;
    }
    if (cudaGraphRetainUserObject(graph, held, 1, cudaGraphUserObjectMove) != cudaSuccess) {
        cudaGetLastError();
        cudaUserObjectRelease(held, 1);
        return PBM_ERR_CUDA;
    }
    return PBM_OK;
}

}  // namespace

// Both passes of a launch, in a workspace of its own; pool->budget_mu is held until
// budget_launched, so that the launches of two threads do not mix in one stream.  The
// workspace's counts and places must be the launch's own: with another launch's, two
// blocks could give one request its page.
int budget_prepare(pbm_pool* pool, uint32_t n_requests, int32_t* d_ids, int32_t* d_steps, cudaStream_t s,
                   LaunchBudget** budget, uint32_t* slot) {
    cudaStreamCaptureStatus capture = cudaStreamCaptureStatusNone;
    cudaGraph_t graph = nullptr;
    const cudaGraphNode_t* deps = nullptr;        // asked for only so that nothing is left out of the answer
    const cudaGraphEdgeData* edges = nullptr;
    size_t n_deps = 0;
    PBM_CUDA_TRY(cudaStreamGetCaptureInfo(s, &capture, nullptr, &graph, &deps, &edges, &n_deps));
    BudgetSpace space;
    if (capture == cudaStreamCaptureStatusNone) {
        *slot = pool->budget_next++ % kBudgetSlots;
        space = pool->budget_space[*slot];
        const BudgetSlot& last = pool->budget_slots[*slot];
        unsigned long long id = 0;
        PBM_CUDA_TRY(cudaStreamGetId(s, &id));
        if (last.used && last.stream != id) PBM_CUDA_TRY(cudaStreamWaitEvent(s, last.done, 0));
    } else if (capture == cudaStreamCaptureStatusActive) {
        *slot = kBudgetSlots;
        const int rc = budget_borrow(pool, graph, &space);
        if (rc) return rc;
    } else {
        return PBM_ERR_CUDA;   // a capture that already failed
    }
    *budget = space.budget;
    const uint32_t nw64 = (uint32_t)(pool->bitmap_bytes / 8u);
    const uint32_t nb = pool->budget_blocks;
    const uint32_t per = (nw64 + nb - 1u) / nb;
    unsigned long long* words = reinterpret_cast<unsigned long long*>(pool->d_words);
    launch_next(k_free_budget, nb, (unsigned)kBudgetThreads, 0, s, words, nw64, per, space.counts, space.budget);
    PBM_LAUNCH_CHECK();
    launch_next(k_take_free, nb, (unsigned)kBudgetThreads, 0, s, words, nw64, per, space.counts, space.budget,
                n_requests, (unsigned long long)pool->list_cap + 1ull, d_ids, d_steps, pool->d_stats);
    PBM_LAUNCH_CHECK();
    return PBM_OK;
}

// The launch that uses the workspace is queued in s (or was refused).
int budget_launched(pbm_pool* pool, uint32_t slot, cudaStream_t s) {
    if (slot >= kBudgetSlots) return PBM_OK;
    BudgetSlot& last = pool->budget_slots[slot];
    PBM_CUDA_TRY(cudaStreamGetId(s, &last.stream));
    PBM_CUDA_TRY(cudaEventRecord(last.done, s));
    last.used = true;
    return PBM_OK;
}

int popcount_used(pbm_pool* pool, uint64_t* used, cudaStream_t s) {
    PBM_CUDA_TRY(cudaMemsetAsync(&pool->d_check->used, 0, sizeof(unsigned long long), s));
    uint32_t nw64 = (uint32_t)(pool->bitmap_bytes / 8u);
    int blocks = sm_count() * 4;
    k_popcount<<<blocks, 256, 0, s>>>(reinterpret_cast<const unsigned long long*>(pool->d_words), nw64,
                                      &pool->d_check->used);
    PBM_LAUNCH_CHECK();
    unsigned long long h = 0;
    PBM_CUDA_TRY(cudaMemcpyAsync(&h, &pool->d_check->used, sizeof(h), cudaMemcpyDeviceToHost, s));
    PBM_CUDA_TRY(cudaStreamSynchronize(s));
    *used = (uint64_t)(h - pool->padding_bits);
    return PBM_OK;
}

}  // namespace pbm

using namespace pbm;

static void pool_free_all(pbm_pool* p) {
    if (!p) return;
    cudaFree(p->d_words);   // and all that lies behind it
    cudaFree(p->d_base);
    cudaFree(p->d_ring);
    cudaFree(p->d_prefix);
    for (BudgetSlot& slot : p->budget_slots)
        if (slot.done) cudaEventDestroy(slot.done);
    if (p->budget_captures)
        for (char* chunk : p->budget_captures->chunks) cudaFree(chunk);
    delete p;
}

__global__ void k_init_slots(int32_t* cursors, uint32_t* arms, uint32_t max_slots, uint32_t n_pages) {
    for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < max_slots; i += (uint64_t)gridDim.x * blockDim.x) {
        cursors[i] = -1;
        // distributed clock: arm0 = idx(lcg(seed(0, slot)), T) (parallelPage.cu:546-555 randomises arms)
        arms[i] = idx_hi(lcg(request_seed(0u, i)), n_pages);
    }
}

static int pool_reset_impl(pbm_pool* p, cudaStream_t s) {
    const uint32_t nw = (uint32_t)(p->bitmap_bytes / 4u);
    k_reset_words<<<sm_count() * 4, 256, 0, s>>>(p->d_words, nw, p->n_pages);
    PBM_LAUNCH_CHECK();
    k_init_slots<<<sm_count() * 4, 256, 0, s>>>(p->d_cursors, p->d_arms, p->max_slots, (uint32_t)p->n_pages);
    PBM_LAUNCH_CHECK();
    PBM_CUDA_TRY(cudaMemsetAsync(p->d_stats, 0, sizeof(DevStats), s));
    PBM_CUDA_TRY(cudaMemsetAsync(p->d_arm, 0, sizeof(unsigned long long), s));
    PBM_CUDA_TRY(cudaMemsetAsync(p->d_clock_list, 0, sizeof(ClockList), s));
    p->fifo_valid = false;
    return PBM_OK;
}

extern "C" {

const char* pbm_version(void) { return "pbm-gb300 0.1 (sm_103a)"; }
uint64_t pbm_kernel_launches(void) { return (uint64_t)g_launches.load(); }
int pbm_device_sm_count(int* h_sms) {
    if (!h_sms) return PBM_ERR_INVALID;
    *h_sms = sm_count();
    return PBM_OK;
}

int pbm_pool_create(const pbm_pool_config* cfg, pbm_pool** out) {
    if (!cfg || !out) return PBM_ERR_INVALID;
    *out = nullptr;
    if (cfg->n_pages == 0 || cfg->n_pages > 0x7fffffffull || cfg->page_size == 0) return PBM_ERR_INVALID;
    pbm_pool* p = new (std::nothrow) pbm_pool();   // value-initialised: all zero
    if (!p) return PBM_ERR_NOMEM;
    p->n_pages = cfg->n_pages;
    p->page_size = cfg->page_size;
    p->flags = cfg->flags;
    p->max_slots = cfg->max_slots ? cfg->max_slots : (1u << 22);
    cudaGetDevice(&p->device);
    const uint64_t nw64 = (cfg->n_pages + 63u) / 64u;
    p->bitmap_bytes = (size_t)nw64 * 8u;
    p->padding_bits = nw64 * 64u - cfg->n_pages;
    p->view.n_pages = (uint32_t)cfg->n_pages;
    p->view.n_words32 = (uint32_t)((cfg->n_pages + 31u) / 32u);
    p->view.n_words64 = (uint32_t)nw64;
    p->view.page_size = cfg->page_size;
    const uint32_t nb_scan = (uint32_t)((p->view.n_words32 + 4095u) / 4096u) + 1u;
    p->prefix_cap = 0;
    // the budget pass: a block per kBudgetThreads 64-bit words, at most kBudgetPerSm per SM; it hands
    // pages out itself in a pool at least half full
    p->budget_blocks = (uint32_t)std::min<uint64_t>((uint64_t)sm_count() * kBudgetPerSm,
                                                 (nw64 + kBudgetThreads - 1u) / kBudgetThreads);
    p->list_cap = std::max<uint64_t>(1024u, cfg->n_pages / 2u);
    // everything but the page memory and the free list in one allocation, the bitmap first
    size_t at = 0;
    auto place = [&](size_t bytes) {
        const size_t o = at;
        at += (bytes + 255u) & ~(size_t)255u;
        return o;
    };
    const size_t o_words = place(p->bitmap_bytes), o_seen = place(p->bitmap_bytes);
    const size_t o_cursors = place(sizeof(int32_t) * p->max_slots), o_arms = place(sizeof(uint32_t) * p->max_slots);
    const size_t o_stats = place(sizeof(DevStats)), o_arm = place(sizeof(unsigned long long));
    const size_t o_clock = place(sizeof(ClockList));
    const size_t o_fifo = place(sizeof(FifoState)), o_check = place(sizeof(CheckCounters));
    const size_t o_budget = place(budget_space_bytes(p->budget_blocks) * kBudgetSpaces);
    const size_t o_scan = place(sizeof(unsigned long long) * nb_scan);
    char* all = nullptr;
    bool ok = cudaMalloc(&all, at) == cudaSuccess;
    if (ok) {
        p->d_words = reinterpret_cast<uint32_t*>(all + o_words);
        p->d_seen = reinterpret_cast<uint32_t*>(all + o_seen);
        p->d_cursors = reinterpret_cast<int32_t*>(all + o_cursors);
        p->d_arms = reinterpret_cast<uint32_t*>(all + o_arms);
        p->d_stats = reinterpret_cast<DevStats*>(all + o_stats);
        p->d_arm = reinterpret_cast<unsigned long long*>(all + o_arm);
        p->d_clock_list = reinterpret_cast<ClockList*>(all + o_clock);
        p->d_fifo = reinterpret_cast<FifoState*>(all + o_fifo);
        p->d_check = reinterpret_cast<CheckCounters*>(all + o_check);
        for (uint32_t i = 0; i < kBudgetSlots; ++i) p->budget_space[i] = budget_space_at(all + o_budget, p->budget_blocks, i);
        p->d_scan = reinterpret_cast<unsigned long long*>(all + o_scan);
    }
    try {
        p->budget_captures = std::make_shared<BudgetCaptureSpaces>();
    } catch (...) {
        ok = false;
    }
    ok = ok && budget_add_captures(*p->budget_captures, all + o_budget + kBudgetSlots * budget_space_bytes(p->budget_blocks),
                                   p->budget_blocks, false);
    for (BudgetSlot& slot : p->budget_slots)
        ok = ok && cudaEventCreateWithFlags(&slot.done, cudaEventDisableTiming) == cudaSuccess;
    if (ok && (cfg->flags & PBM_POOL_MATERIALIZE)) {
        ok = cudaMalloc(&p->d_base, (size_t)cfg->n_pages * cfg->page_size) == cudaSuccess;
    }
    if (!ok) {
        cudaGetLastError();
        pool_free_all(p);
        return PBM_ERR_NOMEM;
    }
    p->view.words = p->d_words;
    p->view.base = p->d_base;
    int rc = pool_reset_impl(p, 0);
    if (rc == PBM_OK && cudaStreamSynchronize(0) != cudaSuccess) rc = PBM_ERR_CUDA;
    if (rc != PBM_OK) { pool_free_all(p); return rc; }
    *out = p;
    return PBM_OK;
}

int pbm_pool_destroy(pbm_pool* pool) {
    PBM_ON_POOL_DEVICE(pool);
    if (!pool) return PBM_ERR_INVALID;
    cudaDeviceSynchronize();
    pbm_malloc_release(pool);   // malloc side tables, if any
    pool_free_all(pool);
    return PBM_OK;
}

int pbm_pool_info(const pbm_pool* pool, uint64_t* n_pages, uint32_t* page_size, void** d_bitmap,
                  size_t* bitmap_bytes, void** d_base) {
    if (!pool) return PBM_ERR_INVALID;
    if (n_pages) *n_pages = pool->n_pages;
    if (page_size) *page_size = pool->page_size;
    if (d_bitmap) *d_bitmap = pool->d_words;
    if (bitmap_bytes) *bitmap_bytes = pool->bitmap_bytes;
    if (d_base) *d_base = pool->d_base;
    return PBM_OK;
}

int pbm_pool_reset(pbm_pool* pool, void* stream) {
    PBM_ON_POOL_DEVICE(pool);
    if (!pool) return PBM_ERR_INVALID;
    return pool_reset_impl(pool, (cudaStream_t)stream);
}

int pbm_pool_prefill_bernoulli(pbm_pool* pool, double occupancy, uint64_t seed, void* stream) {
    PBM_ON_POOL_DEVICE(pool);
    if (!pool || !(occupancy >= 0.0) || occupancy > 1.0) return PBM_ERR_INVALID;
    cudaStream_t s = (cudaStream_t)stream;
    uint64_t thresh = occupancy <= 0.0 ? 0ull
                      : occupancy >= 1.0 ? (1ull << 53)
                                         : (uint64_t)(occupancy * 9007199254740992.0);
    const uint32_t nw = (uint32_t)(pool->bitmap_bytes / 4u);
    k_prefill<<<sm_count() * 8, 256, 0, s>>>(pool->d_words, nw, pool->n_pages, thresh, seed);
    PBM_LAUNCH_CHECK();
    pool->fifo_valid = false;
    return PBM_OK;
}

int pbm_pool_used(pbm_pool* pool, uint64_t* h_used, void* stream) {
    PBM_ON_POOL_DEVICE(pool);
    if (!pool || !h_used) return PBM_ERR_INVALID;
    return popcount_used(pool, h_used, (cudaStream_t)stream);
}

int pbm_pool_read_bitmap(pbm_pool* pool, void* h_dst, size_t bytes, void* stream) {
    PBM_ON_POOL_DEVICE(pool);
    if (!pool || !h_dst || bytes != pool->bitmap_bytes) return PBM_ERR_INVALID;
    cudaStream_t s = (cudaStream_t)stream;
    PBM_CUDA_TRY(cudaMemcpyAsync(h_dst, pool->d_words, bytes, cudaMemcpyDeviceToHost, s));
    PBM_CUDA_TRY(cudaStreamSynchronize(s));
    return PBM_OK;
}

int pbm_pool_write_bitmap(pbm_pool* pool, const void* h_src, size_t bytes, void* stream) {
    PBM_ON_POOL_DEVICE(pool);
    if (!pool || !h_src || bytes != pool->bitmap_bytes) return PBM_ERR_INVALID;
    cudaStream_t s = (cudaStream_t)stream;
    PBM_CUDA_TRY(cudaMemcpyAsync(pool->d_words, h_src, bytes, cudaMemcpyHostToDevice, s));
    k_set_padding<<<1, 64, 0, s>>>(pool->d_words, (uint32_t)(bytes / 4u), pool->n_pages);
    PBM_LAUNCH_CHECK();
    PBM_CUDA_TRY(cudaStreamSynchronize(s));
    pool->fifo_valid = false;
    return PBM_OK;
}

int pbm_pool_device_state(pbm_pool* pool, int build_fifo, pbm_device_state* h_out, void* stream) {
    PBM_ON_POOL_DEVICE(pool);
    if (!pool || !h_out) return PBM_ERR_INVALID;
    if (build_fifo && !pool->fifo_valid) {
        int rc = fifo_build(pool, (cudaStream_t)stream);
        if (rc) return rc;
        PBM_CUDA_TRY(cudaStreamSynchronize((cudaStream_t)stream));
    }
    h_out->words = pool->d_words;
    h_out->base = pool->d_base;
    h_out->n_pages = pool->n_pages;
    h_out->page_size = pool->page_size;
    h_out->n_words32 = pool->view.n_words32;
    h_out->n_words64 = pool->view.n_words64;
    h_out->max_slots = pool->max_slots;
    h_out->cursors = pool->d_cursors;
    h_out->arms = pool->d_arms;
    h_out->single_arm = pool->d_arm;
    h_out->fifo_state = pool->d_fifo;
    h_out->fifo_ring = pool->d_ring;
    h_out->stats = pool->d_stats;
    return PBM_OK;
}

int pbm_pool_stats(pbm_pool* pool, pbm_stats* h_out, void* stream) {
    PBM_ON_POOL_DEVICE(pool);
    if (!pool || !h_out) return PBM_ERR_INVALID;
    cudaStream_t s = (cudaStream_t)stream;
    DevStats d;
    PBM_CUDA_TRY(cudaMemcpyAsync(&d, pool->d_stats, sizeof(d), cudaMemcpyDeviceToHost, s));
    PBM_CUDA_TRY(cudaStreamSynchronize(s));
    h_out->successes = d.successes;
    h_out->failures = d.failures;
    h_out->steps = d.steps;
    h_out->frees = d.frees;
    return d.timeouts ? PBM_ERR_TIMEOUT : PBM_OK;
}

int pbm_check_ids(pbm_pool* pool, const int32_t* d_ids, uint32_t n, pbm_check_result* h_out,
                  void* stream) {
    PBM_ON_POOL_DEVICE(pool);
    if (!pool || !h_out || (n && !d_ids)) return PBM_ERR_INVALID;
    cudaStream_t s = (cudaStream_t)stream;
    PBM_CUDA_TRY(cudaMemsetAsync(pool->d_seen, 0, pool->bitmap_bytes, s));
    PBM_CUDA_TRY(cudaMemsetAsync(pool->d_check, 0, sizeof(CheckCounters), s));
    if (n) {
        int blocks = (int)((n + 255u) / 256u);
        if (blocks > sm_count() * 8) blocks = sm_count() * 8;
        k_check_ids<<<blocks, 256, 0, s>>>(pool->d_words, pool->d_seen, pool->n_pages, d_ids, n,
                                           pool->d_check);
        PBM_LAUNCH_CHECK();
    }
    CheckCounters c;
    PBM_CUDA_TRY(cudaMemcpyAsync(&c, pool->d_check, sizeof(c), cudaMemcpyDeviceToHost, s));
    PBM_CUDA_TRY(cudaStreamSynchronize(s));
    uint64_t used = 0;
    int rc = popcount_used(pool, &used, s);
    if (rc) return rc;
    h_out->n_ok = (int64_t)c.ok;
    h_out->n_failed = (int64_t)c.failed;
    h_out->n_out_of_range = (int64_t)c.out_of_range;
    h_out->n_duplicates = (int64_t)c.duplicates;
    h_out->n_not_marked = (int64_t)c.not_marked;
    h_out->used_pages = (int64_t)used;
    return (c.out_of_range || c.duplicates || c.not_marked) ? PBM_ERR_CORRUPT : PBM_OK;
}

}  // extern "C"
