// malloc.cu -- batched size-classed malloc / free over a pool's pages, with
// two backends: page runs with live counts (pbm/pbm_malloc.cuh) and per-class
// block queues (pbm/pbm_qmalloc.cuh).  Forms: plain (one launch per group),
// persistent (one launch), a one-warp deterministic replay, and the
// CUDA-graph form.
//
// Reference: mallocRW / freeRW (source/RWMalloc.cuh:299-334), the
// KernelMallocCollab allocator (source/malloc.cu:223-320) and the
// malloc/free drivers (unitTests/unitTest3.cu, unitTestMalloc1.cu).
#include <atomic>
#include <cstddef>
#include <mutex>
#include <new>

#include "batch_common.cuh"
#include "pbm/pbm_malloc.cuh"
#include "pbm/pbm_qmalloc.cuh"

namespace pbm {
namespace {

struct MArgs {
    MallocView m;
    QMallocView qm;
    const pbm_group* groups;
    uint32_t n_groups;
    uint32_t step;                    // graph form: the replay (set on the host before each launch)
    uint32_t n_steps;                 // descriptor tables (replay k uses table k mod n_steps; >= 1)
    uint32_t seed;
    const uint32_t* sizes;            // per slot
    unsigned long long* ptrs;         // per slot (device addresses, 0 = none)
    unsigned long long arena_len;
    const unsigned long long* prefix;   // not fused: n_groups + 1 exclusive prefix
    int32_t fuse;                     // each block scans the groups itself
    uint32_t max_steps;
    DevStats* stats;
    int32_t op;                       // plain form: the one group this launch serves
    uint32_t count;
    unsigned long long offset;
    unsigned long long q_base;
};

struct MAcc {
    unsigned long long ok = 0, fail = 0, steps = 0, frees = 0, bad = 0;
};

__device__ __forceinline__ unsigned long long wrap(unsigned long long slot, unsigned long long len) {
    if (slot >= len) slot = slot - len < len ? slot - len : slot % len;
    return slot;
}

// Q: the queue backend (pbm_qmalloc.cuh), else page runs (pbm_malloc.cuh).
template <bool SERIAL, bool Q>
__device__ __forceinline__ void malloc_round(const MArgs& a, uint32_t seed, bool active, int op,
                                             unsigned long long q0, unsigned long long q,
                                             unsigned long long slot, MAcc& acc) {
    const bool do_malloc = active && op == PBM_OP_MALLOC;
    const bool do_free = active && op == PBM_OP_MFREE;
    const uint64_t size = do_malloc ? (uint64_t)a.sizes[slot] : 0ull;
    int32_t s = 0;
    void* p = nullptr;
    // a chunk usually lies in one group, so it is all mallocs or all frees
    if (!__any_sync(0xffffffffu, do_malloc)) {
    } else if constexpr (Q) {
        p = qmalloc_group(a.qm, 0xffffffffu, size, request_seed(seed, (uint32_t)q), a.max_steps, SERIAL, &s);
    } else {
        p = malloc_group(a.m, 0xffffffffu, size, request_seed(seed ^ 0x9E3779B9u, (uint32_t)q0),
                         request_seed(seed, (uint32_t)q), a.max_steps, SERIAL, &s);
    }
    if (do_malloc) {
        a.ptrs[slot] = (unsigned long long)p;
        if (size) {
            acc.ok += p != nullptr;
            acc.fail += p == nullptr;
            acc.steps += (unsigned long long)s;
        }
    }
    if (!__any_sync(0xffffffffu, do_free)) return;
    const void* fp = do_free ? (const void*)a.ptrs[slot] : nullptr;
    bool ok;
    if constexpr (Q) ok = qfree_group(a.qm, 0xffffffffu, fp);
    else ok = free_group(a.m, 0xffffffffu, fp);
    if (do_free) {
        a.ptrs[slot] = 0ull;
        if (fp) {
            acc.frees += ok;
            acc.bad += !ok;
        }
    }
}

// Two rounds of frees (page runs), their pointers and then their runs read together.
__device__ __forceinline__ void free_rounds(const MArgs& a, bool act_a, unsigned long long slot_a, bool act_b,
                                            unsigned long long slot_b, MAcc& acc) {
    const void* pa = act_a ? (const void*)a.ptrs[slot_a] : nullptr;
    const void* pb = act_b ? (const void*)a.ptrs[slot_b] : nullptr;
    bool ok_a, ok_b;
    const int32_t ra = run_of_block(a.m, pa, ok_a), rb = run_of_block(a.m, pb, ok_b);
    if (act_a) a.ptrs[slot_a] = 0ull;
    if (act_b) a.ptrs[slot_b] = 0ull;
    ok_a = release_run(a.m, 0xffffffffu, ra) && ok_a;
    ok_b = release_run(a.m, 0xffffffffu, rb) && ok_b;
    acc.frees += (pa && ok_a) + (pb && ok_b);
    acc.bad += (pa && !ok_a) + (pb && !ok_b);
}

__device__ __forceinline__ void flush_macc(const MAcc& c, DevStats* st) {
    block_add_counters<5>({c.ok, c.fail, c.steps, c.frees, c.bad},
                          {&st->successes, &st->failures, &st->steps, &st->frees, &st->bad_frees});
}

// With a.fuse each block scans the step's group counts into shared memory itself, and
// the graph form's step comes with the launch's parameters, so a replay is one
// launch (a prefix kernel before it and a step kernel after it took 7 us of 39).  With page
// runs and at least 96 requests for every warp (467,000 on 152 SMs), a warp serves 64 at
// a time, two rounds, and two rounds of frees, each a chain of dependent reads, go side by side.  A
// smaller batch keeps more warps busy with 32; us for mallocs and their frees, 256 groups, 32 / 64 at a time:
//   requests  3,000  100,000  200,000  300,000    320,000  400,000  524,288    1,000,000  2,000,000
//             14/18    19/23    25/25  27.6/27.2    30/33    34/36  40.0/38.9      64/64    131/127
// The replay in request order takes 32: a slot that two of its groups free is empty for the second.
// The chunks are dealt round robin over the blocks (mallocs and frees, whose chunks cost
// differently, come in long runs) and a block's warps take its next one from a shared counter.
template <bool SERIAL, bool Q>
__global__ void __launch_bounds__(256, 4) k_malloc_persistent(MArgs a) {
    stream_wait();
    extern __shared__ unsigned long long s_prefix[];
    __shared__ unsigned int s_next;
    MAcc acc;
    const pbm_group* groups = a.groups + (size_t)(a.step % a.n_steps) * a.n_groups;
    const uint32_t seed = a.seed + a.step;
    const unsigned long long* pre = a.prefix;
    if (threadIdx.x == 0) s_next = 0u;
    if (a.fuse) {
        block_exclusive_prefix(groups, a.n_groups, s_prefix);
        pre = s_prefix;
    } else {
        __syncthreads();
    }
    const unsigned long long total = pre[a.n_groups];
    const uint32_t lane = threadIdx.x & 31u;
    const unsigned long long nwarps = (unsigned long long)gridDim.x * (blockDim.x >> 5);
    const unsigned long long ch = !Q && !SERIAL && total >= nwarps * 96ull ? 64ull : 32ull;   // requests per chunk
    for (;;) {
        unsigned int k = 0;
        if (lane == 0) k = atomicAdd(&s_next, 1u);
        k = __shfl_sync(0xffffffffu, k, 0);
        const unsigned long long q0 = ((unsigned long long)k * gridDim.x + blockIdx.x) * ch;
        if (q0 >= total) break;
        const uint32_t g0 = find_group_warp(pre, a.n_groups, q0, 0u);
        const unsigned long long g0_end = pre[g0 + 1u];
        auto locate = [&](unsigned long long q, int& op, unsigned long long& slot) {
            const uint32_t g = q < g0_end ? g0 : find_group_any(pre, a.n_groups, q, g0);
            const pbm_group gd = groups[g];
            op = gd.op;
            slot = wrap(gd.offset + (q - pre[g]), a.arena_len);
        };
        const unsigned long long qa = q0 + lane, qb = qa + 32ull;
        const bool act_a = qa < total, act_b = ch == 64ull && qb < total;
        int op_a = PBM_OP_MALLOC, op_b = PBM_OP_MALLOC;
        unsigned long long slot_a = 0, slot_b = 0;
        if (act_a) locate(qa, op_a, slot_a);
        if (act_b) locate(qb, op_b, slot_b);
        if (!Q && !__any_sync(0xffffffffu, (act_a && op_a == PBM_OP_MALLOC) || (act_b && op_b == PBM_OP_MALLOC))) {
            free_rounds(a, act_a && op_a == PBM_OP_MFREE, slot_a, act_b && op_b == PBM_OP_MFREE, slot_b, acc);
        } else {
            malloc_round<SERIAL, Q>(a, seed, act_a, op_a, q0, qa, slot_a, acc);
            if (ch == 64ull && q0 + 32ull < total) malloc_round<SERIAL, Q>(a, seed, act_b, op_b, q0 + 32ull, qb, slot_b, acc);
        }
    }
    flush_macc(acc, a.stats);
}

template <bool Q>
__global__ void __launch_bounds__(256) k_malloc_plain(MArgs a) {
    stream_wait();
    MAcc acc;
    const uint32_t lane = threadIdx.x & 31u;
    const unsigned long long warp0 = ((unsigned long long)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const unsigned long long nwarps = ((unsigned long long)gridDim.x * blockDim.x) >> 5;
    for (unsigned long long chunk = warp0; chunk * 32ull < a.count; chunk += nwarps) {
        const unsigned long long ql = chunk * 32ull + lane;
        const bool active = ql < a.count;
        malloc_round<false, Q>(a, a.seed, active, a.op, a.q_base + chunk * 32ull, a.q_base + ql,
                            wrap(a.offset + ql, a.arena_len), acc);
    }
    flush_macc(acc, a.stats);
}

__global__ void k_malloc_init(int32_t* start_of, int32_t* live, uint8_t* len_of, uint32_t n) {
    for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (uint64_t)gridDim.x * blockDim.x) {
        start_of[i] = -1;
        live[i] = 0;
        len_of[i] = 0;
    }
}

struct MallocTables {
    // page-run backend
    int32_t* start_of = nullptr;
    int32_t* live = nullptr;
    uint8_t* len_of = nullptr;
    // queue backend
    QueueRing* rings = nullptr;
    uint32_t* slots = nullptr;
    uint8_t* class_of = nullptr;
    unsigned long long* qcounters = nullptr;
    uint32_t qcap = 0;
    // shared
    unsigned long long* prefix = nullptr;
    uint32_t prefix_cap = 0;
};

__global__ void k_qmalloc_init(QueueRing* rings, uint32_t capacity) {
    const int c = threadIdx.x;
    if (c < kQClasses) {
        rings[c].head = rings[c].tail = rings[c].avail = 0ull;
        rings[c].space = capacity;
    }
}

}  // namespace
}  // namespace pbm

using namespace pbm;

namespace {

// Malloc tables of a pool live beside it, keyed by the pool handle.  Every
// entry point takes g_reg_mu for its whole call (launches only enqueue work),
// so tables are never moved or freed under another thread's call.
std::mutex g_reg_mu;
struct Registry {
    pbm_pool* pool;
    MallocTables t;
};
Registry g_reg[64];
int g_nreg = 0;

MallocTables* tables_of(pbm_pool* p) {
    for (int i = 0; i < g_nreg; ++i) if (g_reg[i].pool == p) return &g_reg[i].t;
    return nullptr;
}

MallocTables* tables_add(pbm_pool* p) {
    if (MallocTables* t = tables_of(p)) return t;
    if (g_nreg >= 64) return nullptr;
    g_reg[g_nreg].pool = p;
    g_reg[g_nreg].t = MallocTables{};
    return &g_reg[g_nreg++].t;
}

uint32_t page_shift_of(const pbm_pool* p) {
    uint32_t sh = 0;
    while ((1u << sh) < p->page_size) ++sh;
    return sh;
}

MallocView view_of(pbm_pool* p, const MallocTables* t) {
    MallocView m;
    m.pool = p->view;
    m.start_of = t->start_of;
    m.live = t->live;
    m.len_of = t->len_of;
    m.page_shift = page_shift_of(p);
    return m;
}

QMallocView qview_of(pbm_pool* p, const MallocTables* t) {
    QMallocView q;
    q.pool = p->view;
    q.rings = t->rings;
    q.slots = t->slots;
    q.class_of = t->class_of;
    q.counters = t->qcounters;
    q.capacity = t->qcap;
    q.page_shift = page_shift_of(p);
    return q;
}

int check_pool(pbm_pool* p) {
    if (!p || !p->d_base) return PBM_ERR_INVALID;
    if ((p->page_size & (p->page_size - 1u)) || p->page_size < 2048u || p->page_size > (1u << 16))
        return PBM_ERR_INVALID;
    return PBM_OK;
}

void free_queue(MallocTables* t) {
    cudaFree(t->rings);
    cudaFree(t->slots);
    cudaFree(t->class_of);
    cudaFree(t->qcounters);
    t->rings = nullptr;
    t->slots = nullptr;
    t->class_of = nullptr;
    t->qcounters = nullptr;
    t->qcap = 0;
}

void drop_if_empty(pbm_pool* p) {
    for (int i = 0; i < g_nreg; ++i) {
        if (g_reg[i].pool != p) continue;
        MallocTables& t = g_reg[i].t;
        if (!t.start_of && !t.rings) {
            cudaFree(t.prefix);
            g_reg[i] = g_reg[--g_nreg];
        }
        return;
    }
}

bool ensure_prefix(MallocTables* t, uint32_t n_groups) {
    if (t->prefix_cap >= n_groups + 1u) return true;
    cudaFree(t->prefix);
    t->prefix = nullptr;
    if (cudaMalloc(&t->prefix, sizeof(unsigned long long) * (n_groups + 1u)) != cudaSuccess) {
        cudaGetLastError();
        t->prefix_cap = 0;
        return false;
    }
    t->prefix_cap = n_groups + 1u;
    return true;
}

// Resident blocks per SM of the persistent kernel (asked once).
template <bool Q>
int persistent_blocks() {
    static std::atomic<int> cache{0};
    int per_sm = cache.load(std::memory_order_relaxed);
    if (!per_sm) {
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_malloc_persistent<false, Q>, 256, kFusedPrefixBytes);
        if (per_sm < 1) per_sm = 1;
        cache.store(per_sm, std::memory_order_relaxed);
    }
    return per_sm;
}

// The persistent kernel's launch (plain stream order when captured).
void launch_persistent(const MArgs& a, bool queue, bool serial, bool captured, cudaStream_t s) {
    const size_t smem = a.fuse ? sizeof(unsigned long long) * (a.n_groups + 1u) : 0u;
    const unsigned block = serial ? 32u : 256u;
    const unsigned grid = serial ? 1u : (unsigned)(sm_count() * (queue ? persistent_blocks<true>() : persistent_blocks<false>()));
    auto kernel = queue ? (serial ? k_malloc_persistent<true, true> : k_malloc_persistent<false, true>)
                        : (serial ? k_malloc_persistent<true, false> : k_malloc_persistent<false, false>);
    launch_next_if(!captured, kernel, grid, block, smem, s, a);
}

int batch_impl(pbm_pool* pool, bool queue, const pbm_group* d_groups, const pbm_group* h_groups, uint32_t n_groups,
               const uint32_t* d_sizes, unsigned long long* d_ptrs, uint64_t arena_len, uint32_t seed,
               uint32_t max_steps, int mode, void* stream) {
    MallocTables* t = tables_of(pool);
    if (!t || (queue ? !t->rings : !t->start_of) || !d_ptrs || !arena_len) return PBM_ERR_INVALID;
    if (n_groups == 0) return PBM_OK;
    cudaStream_t s = (cudaStream_t)stream;
    pool->fifo_valid = false;
    MArgs a{};
    if (queue) a.qm = qview_of(pool, t);
    else a.m = view_of(pool, t);
    a.seed = seed;
    a.sizes = d_sizes;
    a.ptrs = d_ptrs;
    a.arena_len = arena_len;
    a.max_steps = max_steps ? max_steps : kDefaultMaxSteps;
    a.stats = pool->d_stats;
    if (mode == PBM_LAUNCH_PLAIN) {
        if (!h_groups) return PBM_ERR_INVALID;
        unsigned long long q = 0;
        for (uint32_t g = 0; g < n_groups; ++g) {
            const pbm_group& gd = h_groups[g];
            if (gd.op != PBM_OP_MALLOC && gd.op != PBM_OP_MFREE) return PBM_ERR_INVALID;
            if (gd.count == 0) continue;
            a.op = gd.op;
            a.count = gd.count;
            a.offset = gd.offset;
            a.q_base = q;
            const unsigned long long warps = (gd.count + 31ull) / 32ull;
            const unsigned grid = (unsigned)((warps * 32ull + 255ull) / 256ull);
            launch_next(queue ? k_malloc_plain<true> : k_malloc_plain<false>, grid, 256, 0, s, a);
            PBM_LAUNCH_CHECK();
            q += gd.count;
        }
        return PBM_OK;
    }
    if ((mode != PBM_LAUNCH_PERSISTENT && mode != PBM_LAUNCH_SERIAL) || !d_groups) return PBM_ERR_INVALID;
    a.groups = d_groups;
    a.n_groups = n_groups;
    a.n_steps = 1u;
    a.fuse = n_groups <= kFusedGroups ? 1 : 0;
    if (!a.fuse) {
        if (!ensure_prefix(t, n_groups)) return PBM_ERR_NOMEM;
        k_batch_prefix<<<1, 1024, 0, s>>>(d_groups, n_groups, 0u, 1u, t->prefix);
        PBM_LAUNCH_CHECK();
        a.prefix = t->prefix;
    }
    launch_persistent(a, queue, mode == PBM_LAUNCH_SERIAL, false, s);
    PBM_LAUNCH_CHECK();
    return PBM_OK;
}

int graph_impl(pbm_pool* pool, bool queue, const pbm_group* d_groups, uint32_t n_groups, uint32_t n_steps,
               const uint32_t* d_sizes, unsigned long long* d_ptrs, uint64_t arena_len, uint32_t seed0,
               uint32_t max_steps, void* stream, pbm_graph** out) {
    MallocTables* t = tables_of(pool);
    if (!t || (queue ? !t->rings : !t->start_of) || !d_groups || !d_ptrs || !out || !n_groups || !n_steps ||
        !arena_len)
        return PBM_ERR_INVALID;
    *out = nullptr;
    pbm_graph* g = new (std::nothrow) pbm_graph();
    if (!g) return PBM_ERR_NOMEM;
    g->device = pool->device;
    const bool fuse = n_groups <= kFusedGroups;
    if (!fuse && cudaMalloc(&g->d_prefix, sizeof(unsigned long long) * (n_groups + 1u)) != cudaSuccess) {
        cudaGetLastError();
        delete g;
        return PBM_ERR_NOMEM;
    }
    MArgs a{};
    if (queue) a.qm = qview_of(pool, t);
    else a.m = view_of(pool, t);
    a.groups = d_groups;
    a.n_groups = n_groups;
    a.n_steps = n_steps;
    a.fuse = fuse ? 1 : 0;
    a.seed = seed0;
    a.sizes = d_sizes;
    a.ptrs = d_ptrs;
    a.arena_len = arena_len;
    a.prefix = g->d_prefix;
    a.max_steps = max_steps ? max_steps : kDefaultMaxSteps;
    a.stats = pool->d_stats;
    if (queue) persistent_blocks<true>();   // asked before the capture
    else persistent_blocks<false>();
    const int rc = graph_capture(g, a, offsetof(MArgs, step), d_groups, n_groups, n_steps, fuse,
                                 [&](cudaStream_t cap) {
                                     launch_persistent(a, queue, false, true, cap);
                                     return cudaGetLastError() == cudaSuccess ? PBM_OK : PBM_ERR_CUDA;
                                 });
    if (rc != PBM_OK) {
        cudaFree(g->d_prefix);
        delete g;
        return rc;
    }
    pool->fifo_valid = false;
    *out = g;
    return PBM_OK;
}

}  // namespace

extern "C" {

int pbm_malloc_init(pbm_pool* pool) {
    PBM_ON_POOL_DEVICE(pool);
    std::lock_guard<std::mutex> lk(g_reg_mu);
    int rc = check_pool(pool);
    if (rc) return rc;
    MallocTables* t = tables_add(pool);
    if (!t) return PBM_ERR_NOMEM;
    if (t->start_of) return PBM_OK;
    const size_t n = pool->n_pages;
    if (cudaMalloc(&t->start_of, n * 9) != cudaSuccess) {   // the three tables, one allocation
        cudaGetLastError();
        t->start_of = nullptr;
        drop_if_empty(pool);
        return PBM_ERR_NOMEM;
    }
    t->live = t->start_of + n;
    t->len_of = reinterpret_cast<uint8_t*>(t->live + n);
    k_malloc_init<<<sm_count() * 4, 256>>>(t->start_of, t->live, t->len_of, (uint32_t)n);
    PBM_LAUNCH_CHECK();
    PBM_CUDA_TRY(cudaDeviceSynchronize());
    return PBM_OK;
}

int pbm_malloc_tables(pbm_pool* pool, void** d_start_of, void** d_live, void** d_len_of) {
    PBM_ON_POOL_DEVICE(pool);
    std::lock_guard<std::mutex> lk(g_reg_mu);
    MallocTables* t = tables_of(pool);
    if (!t || !t->start_of) return PBM_ERR_INVALID;
    if (d_start_of) *d_start_of = t->start_of;
    if (d_live) *d_live = t->live;
    if (d_len_of) *d_len_of = t->len_of;
    return PBM_OK;
}

int pbm_malloc_release(pbm_pool* pool) {
    PBM_ON_POOL_DEVICE(pool);
    std::lock_guard<std::mutex> lk(g_reg_mu);
    MallocTables* t = tables_of(pool);
    if (!t) return PBM_ERR_INVALID;
    cudaDeviceSynchronize();
    cudaFree(t->start_of);   // and live, len_of behind it
    t->start_of = nullptr;
    t->live = nullptr;
    t->len_of = nullptr;
    free_queue(t);
    drop_if_empty(pool);
    return PBM_OK;
}

int pbm_malloc_batch(pbm_pool* pool, const pbm_group* d_groups, const pbm_group* h_groups, uint32_t n_groups,
                     const uint32_t* d_sizes, unsigned long long* d_ptrs, uint64_t arena_len, uint32_t seed,
                     uint32_t max_steps, int mode, void* stream) {
    PBM_ON_POOL_DEVICE(pool);
    std::lock_guard<std::mutex> lk(g_reg_mu);
    return batch_impl(pool, false, d_groups, h_groups, n_groups, d_sizes, d_ptrs, arena_len, seed, max_steps, mode,
                      stream);
}

int pbm_malloc_graph_create(pbm_pool* pool, const pbm_group* d_groups, uint32_t n_groups, uint32_t n_steps,
                            const uint32_t* d_sizes, unsigned long long* d_ptrs, uint64_t arena_len,
                            uint32_t seed0, uint32_t max_steps, void* stream, pbm_graph** out) {
    PBM_ON_POOL_DEVICE(pool);
    std::lock_guard<std::mutex> lk(g_reg_mu);
    return graph_impl(pool, false, d_groups, n_groups, n_steps, d_sizes, d_ptrs, arena_len, seed0, max_steps, stream,
                      out);
}

int pbm_malloc_counts(pbm_pool* pool, uint64_t* h_live_runs, uint64_t* h_bad_frees, void* stream) {
    PBM_ON_POOL_DEVICE(pool);
    std::lock_guard<std::mutex> lk(g_reg_mu);
    MallocTables* t = tables_of(pool);
    if (!t || !t->start_of) return PBM_ERR_INVALID;
    cudaStream_t s = (cudaStream_t)stream;
    DevStats d;
    PBM_CUDA_TRY(cudaMemcpyAsync(&d, pool->d_stats, sizeof(d), cudaMemcpyDeviceToHost, s));
    PBM_CUDA_TRY(cudaStreamSynchronize(s));
    if (h_bad_frees) *h_bad_frees = d.bad_frees;
    if (h_live_runs) {
        // runs still holding blocks: count first pages with live > 0 (host scan of a snapshot)
        const size_t n = pool->n_pages;
        int32_t* h = new (std::nothrow) int32_t[n];
        if (!h) return PBM_ERR_NOMEM;
        cudaError_t e = cudaMemcpy(h, t->live, n * 4, cudaMemcpyDeviceToHost);
        uint64_t c = 0;
        for (size_t i = 0; i < n; ++i) c += h[i] > 0;
        delete[] h;
        if (e != cudaSuccess) { cudaGetLastError(); return PBM_ERR_CUDA; }
        *h_live_runs = c;
    }
    return PBM_OK;
}

// ---- queue backend ----

int pbm_qmalloc_init(pbm_pool* pool, uint32_t ring_capacity) {
    PBM_ON_POOL_DEVICE(pool);
    std::lock_guard<std::mutex> lk(g_reg_mu);
    int rc = check_pool(pool);
    if (rc) return rc;
    if (pool->n_pages * (uint64_t)pool->page_size > (1ull << 36)) return PBM_ERR_INVALID;   // 32-bit handles of 16 B
    const uint32_t cap = ring_capacity ? ring_capacity : (1u << 20);
    if (cap & (cap - 1u)) return PBM_ERR_INVALID;
    MallocTables* t = tables_add(pool);
    if (!t) return PBM_ERR_NOMEM;
    if (t->rings) return t->qcap == cap ? PBM_OK : PBM_ERR_INVALID;
    const size_t n = pool->n_pages;
    if (cudaMalloc(&t->rings, sizeof(QueueRing) * kQClasses) != cudaSuccess ||
        cudaMalloc(&t->slots, sizeof(uint32_t) * (size_t)kQClasses * cap) != cudaSuccess ||
        cudaMalloc(&t->class_of, n) != cudaSuccess ||
        cudaMalloc(&t->qcounters, sizeof(unsigned long long) * kQCounterWords) != cudaSuccess) {
        cudaGetLastError();
        free_queue(t);
        drop_if_empty(pool);
        return PBM_ERR_NOMEM;
    }
    t->qcap = cap;
    PBM_CUDA_TRY(cudaMemset(t->slots, 0xff, sizeof(uint32_t) * (size_t)kQClasses * cap));
    PBM_CUDA_TRY(cudaMemset(t->class_of, 0, n));
    PBM_CUDA_TRY(cudaMemset(t->qcounters, 0, sizeof(unsigned long long) * kQCounterWords));
    k_qmalloc_init<<<1, 32>>>(t->rings, cap);
    PBM_LAUNCH_CHECK();
    PBM_CUDA_TRY(cudaDeviceSynchronize());
    return PBM_OK;
}

int pbm_qmalloc_release(pbm_pool* pool) {
    PBM_ON_POOL_DEVICE(pool);
    std::lock_guard<std::mutex> lk(g_reg_mu);
    MallocTables* t = tables_of(pool);
    if (!t || !t->rings) return PBM_ERR_INVALID;
    cudaDeviceSynchronize();
    free_queue(t);
    drop_if_empty(pool);
    return PBM_OK;
}

int pbm_qmalloc_batch(pbm_pool* pool, const pbm_group* d_groups, const pbm_group* h_groups, uint32_t n_groups,
                      const uint32_t* d_sizes, unsigned long long* d_ptrs, uint64_t arena_len, uint32_t seed,
                      uint32_t max_steps, int mode, void* stream) {
    PBM_ON_POOL_DEVICE(pool);
    std::lock_guard<std::mutex> lk(g_reg_mu);
    return batch_impl(pool, true, d_groups, h_groups, n_groups, d_sizes, d_ptrs, arena_len, seed, max_steps, mode,
                      stream);
}

int pbm_qmalloc_graph_create(pbm_pool* pool, const pbm_group* d_groups, uint32_t n_groups, uint32_t n_steps,
                             const uint32_t* d_sizes, unsigned long long* d_ptrs, uint64_t arena_len,
                             uint32_t seed0, uint32_t max_steps, void* stream, pbm_graph** out) {
    PBM_ON_POOL_DEVICE(pool);
    std::lock_guard<std::mutex> lk(g_reg_mu);
    return graph_impl(pool, true, d_groups, n_groups, n_steps, d_sizes, d_ptrs, arena_len, seed0, max_steps, stream,
                      out);
}

int pbm_qmalloc_counts(pbm_pool* pool, uint64_t* h_queued, uint64_t* h_chunks, uint64_t* h_overflow,
                       uint64_t* h_timeouts, uint64_t* h_bad_frees, void* stream) {
    PBM_ON_POOL_DEVICE(pool);
    std::lock_guard<std::mutex> lk(g_reg_mu);
    MallocTables* t = tables_of(pool);
    if (!t || !t->rings) return PBM_ERR_INVALID;
    cudaStream_t s = (cudaStream_t)stream;
    QueueRing r[kQClasses];
    unsigned long long c[kQCounterWords];
    PBM_CUDA_TRY(cudaMemcpyAsync(r, t->rings, sizeof(r), cudaMemcpyDeviceToHost, s));
    PBM_CUDA_TRY(cudaMemcpyAsync(c, t->qcounters, sizeof(c), cudaMemcpyDeviceToHost, s));
    PBM_CUDA_TRY(cudaStreamSynchronize(s));
    if (h_queued)
        for (int k = 0; k < kQClasses; ++k) h_queued[k] = (uint64_t)(long long)r[k].avail;
    if (h_chunks) *h_chunks = c[kQChunks];
    if (h_overflow) *h_overflow = c[kQOverflow];
    if (h_timeouts) *h_timeouts = c[kQTimeouts];
    if (h_bad_frees) *h_bad_frees = c[kQBadFrees];
    return PBM_OK;
}

}  // extern "C"
