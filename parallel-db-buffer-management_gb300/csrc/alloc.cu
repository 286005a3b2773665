// alloc.cu -- page allocation and free kernels for every strategy.
//
// One launch serves n requests; request r uses LCG seed request_seed(seed, r)
// regardless of which thread runs it, so a one-thread (one-warp) launch of
// the same kernel is a deterministic replay of the same requests in order.
//
// Reference routines restated: getPage/freePage of RandomWalkBasic.cuh:54-84,
// RandomWalkBasic_BM.cuh:60-102, CollabRW_BM.cuh:114-160, CRW_BM.cuh:75-156;
// parallelPage.cu getPageLinkedList (:342-369), getPageSingleClock (:491-509),
// getPageDistClock (:571-592), getXPageRandomWalk_BM (:1104-1142).
#include "internal.cuh"

namespace pbm {

struct AllocArgs {
    PoolView v;
    uint32_t n;
    uint32_t seed;
    uint32_t max_steps;
    uint32_t stride;
    int32_t* ids;
    int32_t* steps;
    DevStats* stats;
    int32_t* cursors;            // clustered walk
    uint32_t* arms;              // distributed clock
    unsigned long long* arm;     // single clock
    uint32_t max_slots;
    int32_t dedupe;              // collaborative walk: W*stride may exceed L
    LaunchBudget* budget;        // fail-fast launch budget (null: every request walks)
};

// Per-thread accumulators reduced once per block.
struct Acc {
    uint32_t ok = 0, fail = 0;      // a launch has at most 2^32 - 1 requests
    unsigned long long steps = 0;
};

__device__ __forceinline__ void flush_acc(const Acc& a, DevStats* st) {
    block_add_counters<3>({a.ok, a.fail, a.steps}, {&st->successes, &st->failures, &st->steps});
}

// A launch whose budget pass served the requests in order (list mode) is done, unless
// some lost their page meanwhile: those walk.
__device__ __forceinline__ bool all_listed(const AllocArgs& a) {
    return a.budget && __ldcg(&a.budget->list_mode) && !__ldcg(&a.budget->lost);
}

// Whether request r walks: granted by the budget and not served by its pass.
__device__ __forceinline__ bool must_walk(const AllocArgs& a, bool listed, uint64_t r) {
    return r < a.n && budget_grants(a.budget, r) && (!listed || a.ids[r] == kLostPage);
}

enum class Walk { Page, Word32, Word64, Crw, SingleClock, DistClock };

// Per-thread strategies.  The loop runs whole warps (uniform trip count) so
// the block-level flush can use full-warp shuffles.
// Eight blocks an SM for the walks; the page walk spills a little to fit 32 registers, and its
// counts of requests are 32-bit for that (2^20 page walks at 50% 43.7 -> 41.4 us).  With 40 or
// 48 registers it is faster in an empty pool (250,007 requests 12.3 -> 10.3 / 11.0 us) and
// slower in a crowded one (at 90% 33 -> 40 / 34, at 95% 52 -> 67 / 54).
template <Walk K>
__global__ void __launch_bounds__(256, 8) k_alloc_thread(AllocArgs a) {
    stream_wait();
    Acc acc;
    if (all_listed(a)) return;
    const bool listed = a.budget && __ldcg(&a.budget->list_mode);
    // whole warps iterate together (nthr is a multiple of 32), or one thread in the serial
    // replay; r stays below the requests rounded up to 32s, at most 2^32
    const uint32_t nthr = gridDim.x * blockDim.x;
    uint32_t r = blockIdx.x * blockDim.x + threadIdx.x;
    const uint32_t r0 = r & ~31u;
    const uint32_t trips = r0 < a.n ? (a.n - 1u - r0) / nthr + 1u : 0u;
    for (uint32_t k = 0; k < trips; ++k, r += nthr) {
        const bool go = must_walk(a, listed, r);
        int32_t s = 0, id = -1;
        if (K == Walk::Page && blockDim.x >= 32u) {
            id = walk_page_warp(a.v, go, request_seed(a.seed, (uint32_t)r), a.max_steps, &s);
        } else if (!go) {
            // past the last request, or past the launch budget: no free page is left for this request
        } else if constexpr (K == Walk::Page) {
            const int32_t seed0 = request_seed(a.seed, r);
            id = walk_page(a.v, seed0, a.max_steps, &s);
        } else if constexpr (K == Walk::Word32) {
            const int32_t seed0 = request_seed(a.seed, r);
            id = walk_word<uint32_t>(a.v, seed0, a.max_steps, &s);
        } else if constexpr (K == Walk::Word64) {
            const int32_t seed0 = request_seed(a.seed, r);
            id = walk_word<uint64_t>(a.v, seed0, a.max_steps, &s);
        } else if constexpr (K == Walk::Crw) {
            const int32_t seed0 = request_seed(a.seed, r);
            int32_t* cur = a.cursors + (r % a.max_slots);
            int32_t c = *cur;
            id = walk_crw(a.v, &c, seed0, a.max_steps, &s);
            *cur = c;
        } else if constexpr (K == Walk::SingleClock) {
            id = sweep_single(a.v, a.arm, a.max_steps, &s);   // the one-thread replay; blocks: k_alloc_clock
        } else {
            uint32_t* arm = a.arms + (r % a.max_slots);
            uint32_t ar = *arm;
            id = sweep_dist(a.v, &ar, a.max_steps, &s);
            *arm = ar;
        }
        if (r >= a.n || (listed && !go)) continue;   // answered by the budget pass
        a.ids[r] = id;
        if (a.steps) a.steps[r] = s;
        acc.ok += id >= 0;
        acc.fail += id < 0;
        acc.steps += (unsigned long long)s;
    }
    flush_acc(acc, a.stats);
}

// ---- the single clock's sweep ----
// While there are plenty of free pages each warp sweeps for itself (sweep_single_warp), and
// the pages that its window holds beyond its need are passed until the arm comes round.  A
// launch that asks for most of the free pages cannot pass any: it would go round the pool
// again and again for the last of them, and fail requests that use up their positions on
// the way.  Its blocks share the positions out: a block moves the arm over those that it
// needs on average, its threads read one word each, and the end of the window
// that was not needed goes to a list, where a block that is short looks before it moves
// the arm again.  On average as many blocks leave an end as are short; with many ends in the list first
// windows are a standard deviation shorter.
// Measured on GB300, launches for exactly the free pages, us and requests that fail, one
// position an atomic / every warp for itself / as here:
//   2^20 pages at 50%: 107, 0 / 213-249, 50-200 / 85-95, 0
//   2^24 pages at 90%: 1400, 0 / 390-450, 400-2,200 / 146, 0
//   2^20 pages at 50% with a bound of 64 positions: 89, 0 / 46-50, 19,400-20,200 / 70, 0
// and 300,007 requests for 1 M free pages with their frees, alone in a stream: 116 / 16.8 / 17.3 (shared out: 27).
// The line lies at two thirds of the free pages: a warp's window is on average a fifth to a
// quarter longer than its need, so what is asked for and what is passed stay
// below what is there (launches for half of the free pages of 2^24 at 90%: 41 us both ways).
constexpr int kClockBlocks = 5;              // of 256 threads an SM
constexpr uint32_t kClockSpins = 1u << 12;   // polls of a slot that is being filled
constexpr long long kClockMany = 1024;       // ends in the list from which first windows are a little shorter
constexpr uint32_t kClockWaits = 32;         // looks at the list when no positions are left,
constexpr uint32_t kClockPause = 1000;       // and ns between them: for ends that other blocks are just leaving

// Whether the list has room for one more, `avail` being its count a moment ago.
__device__ __forceinline__ bool clock_room(long long avail) { return avail < (long long)(kClockSlots / 2u); }

__device__ __forceinline__ void clock_fill(ClockList* q, unsigned long long ticket, uint32_t pos, uint32_t len) {
    atomicExch(q->slot + ticket % kClockSlots, ((unsigned long long)pos << 32) | len);
    atomicAdd(&q->avail, 1ull);
}

__device__ __forceinline__ bool clock_take(ClockList* q, uint32_t* pos, uint32_t* len) {
    if ((long long)atomicAdd(&q->avail, ~0ull) <= 0) {
        atomicAdd(&q->avail, 1ull);
        return false;
    }
    unsigned long long* slot = q->slot + atomicAdd(&q->head, 1ull) % kClockSlots;
    unsigned long long e = 0ull;
    for (uint32_t k = 0; !e && k < kClockSpins; ++k) e = atomicExch(slot, 0ull);
    *pos = (uint32_t)(e >> 32);
    *len = (uint32_t)e;
    return e != 0ull;
}

// Exclusive prefix of v over the block, and its total.  `warp_tot`: a word per warp, not in use
// between the caller's last barrier and its next one.
__device__ __forceinline__ uint32_t block_prefix(uint32_t v, uint32_t* warp_tot, uint32_t* total) {
    const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5, nwarps = blockDim.x >> 5;
    const uint32_t incl = (uint32_t)group_incl_scan<32>((int)v, lane, kFull32);
    if (lane == 31u) warp_tot[warp] = incl;
    __syncthreads();
    uint32_t before = 0, all = 0;
    for (uint32_t i = 0; i < nwarps; ++i) {
        const uint32_t x = warp_tot[i];
        if (i < warp) before += x;
        all += x;
    }
    *total = all;
    return before + incl - v;
}

// The sweep of a block that shares out the positions, for its threads with `go`; the block calls
// converged.  seen_free of `seen` positions looked at were free.  A request's steps are the positions from
// the page before its own; together the requests examine max_steps positions each, and those that find no page
// end after max_steps -- once they have looked at the list kClockWaits times more.
__device__ __forceinline__ int32_t clock_share(const AllocArgs& a, ClockList* list, bool go, uint32_t seen_free, uint32_t seen,
                                               int32_t* steps_out) {
    __shared__ uint32_t s_need[8], s_free[8], s_got[8];
    __shared__ uint32_t s_pos[256];              // positions of the pages claimed in a window, from 1
    __shared__ uint32_t s_p0, s_len, s_end, s_room;
    const uint32_t T = a.v.n_pages;
    const unsigned long long most = 32u * (blockDim.x - 2u);       // positions at once: a word per thread, wrapped or not
    uint32_t M = 0;                                                // requests without a page
    uint32_t rank = block_prefix(go ? 1u : 0u, s_need, &M);        // this one's place among them
    unsigned long long left = (unsigned long long)M * a.max_steps;
    unsigned long long passed = 0;                                 // positions since the last page claimed
    int32_t id = -1, s = go ? (int32_t)a.max_steps : 0;
    bool want = go;
    bool none = false;                                             // the last window had no free page
    long long avail = 0;                                           // thread 0's: the list's count seen last
    if (threadIdx.x == 0) avail = (long long)__ldcg(&list->avail);
    uint32_t waits = 0;
    for (bool first = true; M; first = false) {
        if (threadIdx.x == 0) {
            uint32_t p0 = 0, P = 0;
            if (!left) __nanosleep(kClockPause);
            const long long now = (long long)__ldcg(&list->avail);
            if (none || !left) avail = now;
            if (!first && avail > 0 && clock_take(list, &p0, &P)) {
                const uint32_t fit = (uint32_t)min(most, (unsigned long long)P);
                if (fit < P) {
                    const uint32_t rest = p0 + fit;
                    clock_fill(list, atomicAdd(&list->tail, 1ull), rest >= T ? rest - T : rest, P - fit);
                }
                P = fit;
            } else if (left) {
                const unsigned long long mean = (unsigned long long)M * seen / (seen_free ? seen_free : 1u);
                unsigned long long len = mean + 1ull;
                if (!first) len = mean + (mean >> 3) + 8ull;
                else if (avail > kClockMany) len -= min(mean / 2u, (unsigned long long)sqrtf((float)(mean * seen / (seen_free + 1u))));
                P = (uint32_t)min(min(min(len, most), left), (unsigned long long)T);
                p0 = (uint32_t)(atomicAdd(a.arm, (unsigned long long)P) % T);
            }
            avail = now;
            s_room = clock_room(avail);
            s_p0 = p0;
            s_len = P;
        }
        __syncthreads();
        const uint32_t p0 = s_p0, P = s_len;
        if (!P && ++waits >= kClockWaits) break;
        // thread i: word i of the pages p0 .. p0 + P - 1, wrapping past the last page
        const uint32_t i = threadIdx.x, w0 = p0 >> 5;
        const uint32_t end_a = min(T, p0 + P);                     // first stretch [p0, end_a)
        const uint32_t n_a = ((end_a + 31u) >> 5) - w0;
        const uint32_t end_b = P - (end_a - p0);                   // second stretch [0, end_b)
        const uint32_t w = i < n_a ? w0 + i : i - n_a;
        const uint32_t lo = i < n_a ? max(p0, w << 5) : w << 5, hi = i < n_a ? end_a : end_b;
        uint32_t fr = 0u;
        if ((w << 5) < hi) fr = ~load_word(a.v.words + w) & bit_range(lo & 31u, min(31u, hi - 1u - (w << 5)));
        uint32_t total = 0, got_total = 0;
        const uint32_t excl = block_prefix((uint32_t)__popc(fr), s_free, &total);
        const uint32_t to_pos = i < n_a ? 1u - p0 : T - p0 + 1u;   // page + to_pos: its position in the window
        uint32_t end = P;
        if (excl < M && M - excl <= (uint32_t)__popc(fr)) {        // the last page needed is here
            end = (w << 5) + nth_set_bit(fr, (int)(M - excl - 1u)) + to_pos;
            s_end = end;
        }
        const bool leave = end < P && s_room;
        unsigned long long ticket = 0;
        if (leave) ticket = atomicAdd(&list->tail, 1ull);
        uint32_t got = low_bits(fr, (int)M - (int)excl);
        if (got) got &= ~atomicOr(a.v.words + w, got);             // less what another claim took first
        if (leave) clock_fill(list, ticket, p0 + end >= T ? p0 + end - T : p0 + end, P - end);
        const uint32_t at0 = block_prefix((uint32_t)__popc(got), s_got, &got_total);
        const uint32_t used = total >= M ? s_end : P;
        for (uint32_t m = got, k = at0; m; m &= m - 1u, ++k) s_pos[k] = (w << 5) + (uint32_t)__ffs((int)m) - 1u + to_pos;
        __syncthreads();
        if (want && rank < got_total) {
            const uint32_t at = s_pos[rank];
            const uint32_t p = p0 + at - 1u;
            id = (int32_t)(p >= T ? p - T : p);
            s = (int32_t)min((unsigned long long)a.max_steps, rank ? (unsigned long long)(at - s_pos[rank - 1u]) : passed + at);
            want = false;
        }
        passed = got_total ? used - min(used, s_pos[got_total - 1u]) : passed + used;
        none = total == 0u;
        M -= got_total;
        left = min(left - min(left, (unsigned long long)used), (unsigned long long)M * a.max_steps);
        rank -= got_total;
        seen_free += total;
        seen += P;
        if (seen > (1u << 24)) {
            seen >>= 1;
            seen_free >>= 1;
        }
    }
    *steps_out = s;
    return id;
}

__global__ void __launch_bounds__(256, kClockBlocks) k_alloc_clock(AllocArgs a, ClockList* list, uint32_t at_work) {
    stream_wait();
    __shared__ uint32_t s_sample[8];
    Acc acc;
    if (all_listed(a)) return;
    const bool listed = a.budget && __ldcg(&a.budget->list_mode);
    for (uint64_t base = (uint64_t)blockIdx.x * blockDim.x; base < a.n; base += (uint64_t)gridDim.x * blockDim.x) {
        const uint64_t r = base + threadIdx.x;
        const bool go = must_walk(a, listed, r);
        int32_t s = 0, id;
        // a word drawn at random by each thread: free pages of 1024 positions (warp), of all (block)
        const uint32_t f = __reduce_add_sync(
            kFull32, (uint32_t)__popc(~load_word(a.v.words + idx_hi(request_seed(a.seed, (uint32_t)r) & 0x7fffffff, a.v.n_words32))));
        if ((threadIdx.x & 31u) == 0u) s_sample[threadIdx.x >> 5] = f;
        __syncthreads();
        uint32_t seen_free = 0;
        for (uint32_t i = 0; i < blockDim.x >> 5; ++i) seen_free += s_sample[i];
        const uint32_t seen = 32u * blockDim.x;
        // the pages that were free when the launch began: those free now, and those that the blocks before have
        // taken, but for the ones that may still be at work
        const uint64_t taken = base > at_work ? base - at_work : 0u;
        if (a.n > 32u && 3.0f * (float)a.n >= 2.0f * ((float)seen_free / (float)seen * (float)a.v.n_pages + (float)taken))
            id = clock_share(a, list, go, seen_free, seen, &s);
        else
            id = sweep_single_warp(a.v, a.arm, go, f, a.max_steps, a.n <= 32u, &s);
        if (r < a.n && !(listed && !go)) {                         // else answered by the budget pass
            a.ids[r] = id;
            if (a.steps) a.steps[r] = s;
            acc.ok += id >= 0;
            acc.fail += id < 0;
            acc.steps += (unsigned long long)s;
        }
        __syncthreads();                                           // s_sample is used again
    }
    flush_acc(acc, a.stats);
}

// Warp-collaborative walk: groups of W lanes take W consecutive requests.
// Launched with blockDim a multiple of W (>= W); a one-group launch
// (blockDim == W, one block) replays the groups in request order.
// Six blocks of 256 fit an SM (40 registers), and the grid is that: with eight per SM
// launched, a last quarter of the blocks ran after the others (250,007 requests at 90%
// and their frees 10.2 -> 8.6 us, 2^20 at 50% 18.7 -> 18.2).
constexpr int kCollabBlocks = 6;

template <int W, typename Word>
__global__ void __launch_bounds__(256, kCollabBlocks) k_alloc_collab(AllocArgs a) {
    stream_wait();
    __shared__ int32_t slots[256];
    Acc acc;
    const uint64_t tid = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
    const uint64_t nthr = (uint64_t)gridDim.x * blockDim.x;
    const uint32_t gl = threadIdx.x & (uint32_t)(W - 1);
    const uint32_t L = WordTraits<Word>::count(a.v);
    const uint32_t lane_off = (uint32_t)(((unsigned long long)gl * a.stride) % L);
    volatile int32_t* my_slots = slots + (threadIdx.x & ~(uint32_t)(W - 1));
    if (all_listed(a)) return;
    const bool listed = a.budget && __ldcg(&a.budget->list_mode);
    // trip count uniform across each group of W lanes
    for (uint64_t base = tid - gl; base < a.n; base += nthr) {
        const uint64_t r = base + gl;
        const bool need = must_walk(a, listed, r);
        int32_t s = 0;
        const int32_t id = walk_collab<W, Word>(a.v, need, request_seed(a.seed, base), lane_off, a.dedupe != 0, a.max_steps,
                                                my_slots, &s);
        if (r < a.n && (need || !listed)) {          // else answered by the budget pass
            a.ids[r] = id;
            if (a.steps) a.steps[r] = need ? s : 0;   // refused by the budget: no walk
            acc.ok += id >= 0;
            acc.fail += id < 0;
            acc.steps += (unsigned long long)s;
        }
    }
    flush_acc(acc, a.stats);
}

// ---- the free list (fifo_get / fifo_put of pbm_device.cuh, for whole blocks) ----
// A block takes its requests' pages with one reservation and one run of tickets,
// so its ring slots are neighbours, and returns pages the same way.  With an
// atomic per thread on each shared counter the launch lasted as long as the queue
// at those counters' addresses (long-scoreboard stalls of 70-125 cycles per
// instruction).  A thread serves kFifoItems requests, their slots' exchanges
// in flight together, once that still leaves every SM a block; one otherwise.
// Measured on GB300, 2^20 gets + puts on 2^24 pages at 50%: 118 -> 30 us; 250,007:
// 23.4 -> 16.3; 1,000: 8.4 both.  Merging a warp's pages of one bitmap word
// (__match_any_sync) before the bitmap atomics: 58 us, the match costs more
// than the atomics once the list's order is mixed.  One-thread replays go page
// by page.
constexpr int kFifoItems = 4;

template <int ITEMS>
__global__ void __launch_bounds__(256) k_fifo_alloc(AllocArgs a, FifoState* st, int32_t* ring) {
    stream_wait();
    Acc acc;
    if (blockDim.x & 31u) {
        for (uint64_t r = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; r < a.n; r += (uint64_t)gridDim.x * blockDim.x) {
            int32_t s = 0;
            const int32_t id = fifo_get(a.v, st, ring, a.stats, &s);
            a.ids[r] = id;
            if (a.steps) a.steps[r] = s;
            acc.ok += id >= 0;
            acc.fail += id < 0;
            acc.steps += (unsigned long long)s;
        }
    } else {
        __shared__ uint32_t s_got, s_slot;
        const uint32_t tile = blockDim.x * (uint32_t)ITEMS;
        const uint64_t base = (uint64_t)blockIdx.x * tile;
        const uint32_t k = (uint32_t)(a.n - base < tile ? a.n - base : tile);
        if (threadIdx.x == 0) {
            const long long old = (long long)atomicAdd(&st->avail, 0ull - (unsigned long long)k);
            const uint32_t got = old <= 0 ? 0u : (old < (long long)k ? (uint32_t)old : k);
            if (got < k) atomicAdd(&st->avail, (unsigned long long)(k - got));
            s_got = got;
            s_slot = got ? (uint32_t)(atomicAdd(&st->head, (unsigned long long)got) % a.v.n_pages) : 0u;
        }
        __syncthreads();
        const uint32_t got = s_got, slot0 = s_slot;
        int32_t id[ITEMS];
        int32_t* slot[ITEMS];
#pragma unroll
        for (int j = 0; j < ITEMS; ++j) {
            const uint32_t i = (uint32_t)j * blockDim.x + threadIdx.x;
            uint32_t pos = slot0 + i;                    // i < got <= n_pages
            if (pos >= a.v.n_pages) pos -= a.v.n_pages;
            slot[j] = ring + pos;
            id[j] = i < got ? atomicExch(slot[j], -1) : -1;
        }
#pragma unroll
        for (int j = 0; j < ITEMS; ++j) {
            const uint32_t i = (uint32_t)j * blockDim.x + threadIdx.x;
            if (i >= k) continue;
            int32_t s = 0;
            if (i < got) {
                uint32_t spins = 0;
                while (id[j] < 0 && spins < kFifoSpinLimit) {   // the put that holds the ticket is on its way
                    __nanosleep(64);
                    ++spins;
                    id[j] = atomicExch(slot[j], -1);
                }
                s = (int32_t)spins + 1;
                if (id[j] < 0) atomicAdd(&a.stats->timeouts, 1ull);
                else atomicOr(a.v.words + ((uint32_t)id[j] >> 5), 1u << ((uint32_t)id[j] & 31u));
            }
            a.ids[base + i] = id[j];
            if (a.steps) a.steps[base + i] = s;
            acc.ok += id[j] >= 0;
            acc.fail += id[j] < 0;
            acc.steps += (unsigned long long)s;
        }
    }
    flush_acc(acc, a.stats);
}

template <int ITEMS>
__global__ void __launch_bounds__(256) k_fifo_free(PoolView v, uint32_t n, const int32_t* ids,
                                                   FifoState* st, int32_t* ring, DevStats* stats) {
    stream_wait();
    __shared__ uint32_t s_warp[32];
    __shared__ uint32_t s_slot;
    const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5, nwarps = blockDim.x >> 5;
    const uint64_t base = (uint64_t)blockIdx.x * blockDim.x * ITEMS;
    int32_t id[ITEMS];
    uint32_t cnt = 0;                        // this thread's pages
#pragma unroll
    for (int j = 0; j < ITEMS; ++j) {
        const uint64_t r = base + (uint64_t)j * blockDim.x + threadIdx.x;
        id[j] = r < n ? ids[r] : -1;
        if (id[j] >= (int32_t)v.n_pages) id[j] = -1;
        // the bit, a round trip and two barriers before the page is in its slot: a get of another
        // stream sets it again as soon as it has the page
        if (id[j] >= 0) atomicAnd(v.words + ((uint32_t)id[j] >> 5), ~(1u << ((uint32_t)id[j] & 31u)));
        const uint32_t b = __ballot_sync(kFull32, id[j] >= 0);
        cnt += (uint32_t)__popc(b);          // the warp's
    }
    if (lane == 0u) s_warp[warp] = cnt;
    __syncthreads();
    if (threadIdx.x == 0) {
        uint32_t total = 0;
        for (uint32_t w = 0; w < nwarps; ++w) {
            const uint32_t c = s_warp[w];
            s_warp[w] = total;               // the warp's first ticket
            total += c;
        }
        s_slot = total ? (uint32_t)(atomicAdd(&st->tail, (unsigned long long)total) % v.n_pages) : 0u;
    }
    __syncthreads();
    uint32_t rank = s_warp[warp];
    uint32_t put = 0;
#pragma unroll
    for (int j = 0; j < ITEMS; ++j) {
        const uint32_t b = __ballot_sync(kFull32, id[j] >= 0);
        if (id[j] >= 0) {
            const uint64_t pos = (uint64_t)s_slot + rank + (uint32_t)__popc(b & ((1u << lane) - 1u));
            int32_t* slot = ring + (pos >= v.n_pages ? pos % v.n_pages : pos);
            uint32_t k = 0;
            bool in = true;
            while (atomicCAS(slot, -1, id[j]) != -1) {   // a get of the previous lap is on its way
                if (++k >= kFifoSpinLimit) {
                    atomicAdd(&stats->timeouts, 1ull);
                    in = false;
                    break;
                }
                __nanosleep(64);
            }
            put += in;
        }
        rank += (uint32_t)__popc(b);
    }
    // the block's pages are in their slots: count them available, and freed
    const uint32_t w_put = __reduce_add_sync(kFull32, put);
    __syncthreads();                         // s_warp: every warp has read its first ticket
    if (lane == 0u) s_warp[warp] = w_put;
    __syncthreads();
    if (threadIdx.x == 0) {
        unsigned long long total = 0;
        for (uint32_t w = 0; w < nwarps; ++w) total += s_warp[w];
        if (total) {
            atomicAdd(&st->avail, total);
            atomicAdd(&stats->frees, total);
        }
    }
}

// ---- frees ----
// A thread frees four neighbouring ids of the list: one 16-byte load, and
// neighbours that share a bitmap word (a claim that took several pages of one word
// wrote them side by side) go back with one atomicAnd.  One id per thread spent most
// of its ~200 instructions per warp on the block's counter.  The grid is at most
// what the SMs hold at once, so the blocks' counter atomics, which queue at
// one address, number some thousand at most.  Measured on GB300, us per launch
// of 2^20 ids in a stream of launches: 12.4 -> 8.0 as the collaborative walk wrote them,
// 12.4 -> 10.3 at random (8 us at the ceiling of one atomic per id).
// MERGE: lanes of a warp that free pages of one word merge their bits first
// (the configuration's free_merge).
template <bool MERGE>
__global__ void __launch_bounds__(256) k_free_pages(PoolView v, uint32_t n, const int32_t* ids, DevStats* stats) {
    stream_wait();
    unsigned long long f = 0;
    const uint64_t tid = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
    const uint64_t nthr = (uint64_t)gridDim.x * blockDim.x;
    if constexpr (MERGE) {
        const uint64_t n_round = ((uint64_t)n + 31u) & ~31ull;
        for (uint64_t r = tid; r < n_round; r += nthr) {
            int32_t id = r < n ? ids[r] : -1;
            if (id >= (int32_t)v.n_pages) id = -1;
            free_page_warp(v, 0xffffffffu, id);
            f += id >= 0;
        }
    } else {
        uint32_t cnt = 0;
        uint32_t done = 0;
        if (((uintptr_t)ids & 15u) == 0u) {
            const int4* ids4 = reinterpret_cast<const int4*>(ids);
            const uint32_t n4 = n >> 2;
            for (uint64_t i = tid; i < n4; i += nthr) {
                const int4 q = ids4[i];
                const int32_t id[4] = {q.x, q.y, q.z, q.w};
                uint32_t w = 0u, m = 0u;
#pragma unroll
                for (int k = 0; k < 4; ++k) {
                    if (id[k] < 0 || id[k] >= (int32_t)v.n_pages) continue;
                    const uint32_t wk = (uint32_t)id[k] >> 5, bit = 1u << ((uint32_t)id[k] & 31u);
                    if (m && wk != w) {
                        atomicAnd(v.words + w, ~m);
                        m = 0u;
                    }
                    w = wk;
                    m |= bit;
                    ++cnt;
                }
                if (m) atomicAnd(v.words + w, ~m);
            }
            done = n4 << 2;
        }
        for (uint64_t r = done + tid; r < n; r += nthr) {
            const int32_t id = ids[r];
            if (id < 0 || id >= (int32_t)v.n_pages) continue;
            free_page(v, id);
            ++cnt;
        }
        f = cnt;
    }
    block_add_counters<1>({f}, {&stats->frees});
}

// ---- contiguous runs ----
// SPAN: runs may cross word boundaries (1 <= k <= kMaxSpanPages); else one
// word holds the run (1 <= k <= 32, the reference's getXPage semantics).
template <bool SPAN>
__global__ void __launch_bounds__(256) k_alloc_runs(AllocArgs a, const int32_t* npages) {
    stream_wait();
    Acc acc;
    const uint64_t n_round = ((uint64_t)a.n + 31u) & ~31ull;   // whole warps walk together
    const bool warps = SPAN && blockDim.x >= 32u;              // else the one-thread replay
    for (uint64_t r = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; r < n_round;
         r += (uint64_t)gridDim.x * blockDim.x) {
        const int32_t k = r < a.n ? npages[r] : 0;
        int32_t s = 0, id = -1;
        if (warps)
            id = walk_span_warp(a.v, k >= 1 && k <= 32 ? (uint32_t)k : 0u, request_seed(a.seed, (uint32_t)r), a.max_steps, &s);
        if (SPAN) {
            if (k >= 1 && (uint32_t)k <= kMaxSpanPages && (!warps || k > 32))
                id = walk_span(a.v, (uint32_t)k, request_seed(a.seed, r), a.max_steps, &s);
        } else if (k >= 1 && k <= 32) {
            id = walk_run(a.v, (uint32_t)k, request_seed(a.seed, r), a.max_steps, &s);
        }
        if (r >= a.n) continue;
        a.ids[r] = id;
        if (a.steps) a.steps[r] = s;
        acc.ok += id >= 0;
        acc.fail += id < 0;
        acc.steps += (unsigned long long)s;
    }
    flush_acc(acc, a.stats);
}

__global__ void __launch_bounds__(256) k_free_runs(PoolView v, uint32_t n, const int32_t* ids,
                                                   const int32_t* npages, DevStats* stats) {
    stream_wait();
    unsigned long long f = 0;
    for (uint64_t r = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; r < n; r += (uint64_t)gridDim.x * blockDim.x) {
        int32_t id = ids[r], k = npages[r];
        if (id < 0 || k < 1 || (uint32_t)k > kMaxSpanPages || (unsigned long long)id + (uint32_t)k > v.n_pages)
            continue;
        free_span(v, id, (uint32_t)k);
        f += (unsigned long long)k;
    }
    block_add_counters<1>({f}, {&stats->frees});
}

// ---- config-1 step: claim one page, write the payload, free ----
// Each request claims a page with the page-probe walk, writes its request
// index into every 4-byte word of the first payload_words words of the page,
// and frees the page unless `hold` (unitTest1.5.cu:138-150 get/free kernels
// plus the payload write of the page-pool workload).
// HOLD: the warp's walks go on together (walk_page_warp).  A page that is freed
// again is better walked for alone: its thread frees it at once, and not when its
// warp's longest walk is done (32,768 requests for 32,768 free pages: 3.6 probes and 20 us
// alone, 5.4 probes and 24 us together).
// The counters are 64-bit throughout: with 32-bit ones (38 registers instead of 40) claiming,
// reading and freeing 16,384 pages took 14.3 us instead of 12.2.
template <bool HOLD>
__global__ void __launch_bounds__(256) k_claim_write_free(AllocArgs a, uint32_t payload_words) {
    stream_wait();
    unsigned long long ok = 0, fail = 0, walked = 0, frees = 0;
    const uint64_t n_round = ((uint64_t)a.n + 31u) & ~31ull;   // whole warps walk together
    for (uint64_t r = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; r < n_round;
         r += (uint64_t)gridDim.x * blockDim.x) {
        int32_t s = 0;
        int32_t id = -1;
        if constexpr (HOLD) id = walk_page_warp(a.v, r < a.n, request_seed(a.seed, (uint32_t)r), a.max_steps, &s);
        if (r >= a.n) continue;
        if constexpr (!HOLD) id = walk_page(a.v, request_seed(a.seed, (uint32_t)r), a.max_steps, &s);
        a.ids[r] = id;
        if (a.steps) a.steps[r] = s;
        if (id >= 0) {
            int32_t* pg = reinterpret_cast<int32_t*>(a.v.base + (size_t)(uint32_t)id * a.v.page_size);
            uint32_t k = 0;
            if (((a.v.page_size | (uint32_t)(uintptr_t)a.v.base) & 15u) == 0u) {   // 16-byte aligned pages: 16 bytes a store
                const int4 v4 = make_int4((int32_t)r, (int32_t)r, (int32_t)r, (int32_t)r);
                for (; k + 4u <= payload_words; k += 4u) *reinterpret_cast<int4*>(pg + k) = v4;
            }
            for (; k < payload_words; ++k) pg[k] = (int32_t)r;
            if (!HOLD) { free_page(a.v, id); ++frees; }
        }
        ok += id >= 0;
        fail += id < 0;
        walked += (unsigned long long)s;
    }
    block_add_counters<4>({ok, fail, walked, frees},
                          {&a.stats->successes, &a.stats->failures, &a.stats->steps, &a.stats->frees});
}

}  // namespace pbm

using namespace pbm;

namespace {

int check_cfg(const pbm_walk_config* c) {
    if (!c) return PBM_ERR_INVALID;
    if (c->strategy < 0 || c->strategy >= PBM_N_STRATEGIES) return PBM_ERR_INVALID;
    if (c->word_bits != 0 && c->word_bits != 32 && c->word_bits != 64) return PBM_ERR_INVALID;
    if (c->collab_width != 0 && c->collab_width != 8 && c->collab_width != 16 && c->collab_width != 32)
        return PBM_ERR_INVALID;
    if (c->block_size < 0 || c->block_size > 1024 || (c->block_size % 32) != 0) return PBM_ERR_INVALID;
    return PBM_OK;
}

// Blocks for `threads` threads of work, at most what the SMs hold at once: the
// kernels loop over the rest.  For kernels with little work per request, where
// block starts and the counter atomic of each block's end were a good part
// of the launch (the collaborative walk of 2^20 requests: 22.6 -> 15 us).
// For the per-thread walks it is two such grids: their length varies, and blocks that
// start as others end even it out (2^22 word probes at 50%: 102 us, 106 with one grid,
// 128 with a block per 256 requests and a counter flush that is dear; 2^22 page walks
// 171, 171, 190).  Behind a budget one grid is enough, most requests being answered by
// it: 2^22 page walks at 90% fail-fast 124 -> 31 us, word probes 108 -> 30 (the refusals
// have since moved to the budget's pass: 23).
constexpr int kThreadBlocks = 16 * 256, kListedBlocks = 8 * 256;

int capped_grid(uint64_t threads, int block, int per_sm) {
    const uint64_t need = (threads + (uint64_t)block - 1u) / (uint64_t)block;
    const uint64_t fit = (uint64_t)sm_count() * (uint64_t)(per_sm / block > 0 ? per_sm / block : 1);
    return (int)(need < 1u ? 1u : need < fit ? need : fit);
}

AllocArgs make_args(pbm_pool* p, const pbm_walk_config* c, uint32_t n, uint32_t seed, int32_t* ids,
                    int32_t* steps) {
    AllocArgs a;
    a.v = p->view;
    a.n = n;
    a.seed = seed;
    a.max_steps = c->max_steps ? c->max_steps : kDefaultMaxSteps;
    a.stride = c->stride ? c->stride : 1u;
    a.ids = ids;
    a.steps = steps;
    a.stats = p->d_stats;
    a.cursors = p->d_cursors;
    a.arms = p->d_arms;
    a.arm = p->d_arm;
    a.max_slots = p->max_slots;
    int W = c->collab_width ? c->collab_width : 32;
    uint32_t L = c->word_bits == 64 ? p->view.n_words64 : p->view.n_words32;
    a.dedupe = ((unsigned long long)(W - 1) * a.stride >= L) ? 1 : 0;
    a.budget = nullptr;
    return a;
}

template <int W, typename Word>
int launch_collab_w(const AllocArgs& a, int grid, int block, cudaStream_t s) {
    launch_next(k_alloc_collab<W, Word>, grid, block, 0, s, a);
    PBM_LAUNCH_CHECK();
    return PBM_OK;
}

int launch_alloc(pbm_pool* p, const pbm_walk_config* c, const AllocArgs& a, bool serial,
                 cudaStream_t s) {
    const int block_cfg = c->block_size ? c->block_size : kDefaultBlock;
    const int W = c->collab_width ? c->collab_width : 32;
    const bool w64 = c->word_bits == 64;
    int block = serial ? 1 : block_cfg;
    const int grid = serial ? 1 : capped_grid(a.n, block, a.budget ? kListedBlocks : kThreadBlocks);
    switch (c->strategy) {
    case PBM_RANDOM_WALK:
        launch_next(k_alloc_thread<Walk::Page>, grid, block, 0, s, a);
        break;
    case PBM_RANDOM_WALK_BM:
        if (w64) launch_next(k_alloc_thread<Walk::Word64>, grid, block, 0, s, a);
        else launch_next(k_alloc_thread<Walk::Word32>, grid, block, 0, s, a);
        break;
    case PBM_CLUSTERED_RW_BM:
        launch_next(k_alloc_thread<Walk::Crw>, grid, block, 0, s, a);
        break;
    case PBM_SINGLE_CLOCK:
        // always in blocks of 256, which share out positions best (a larger one is refused, as the others are)
        if (serial) launch_next(k_alloc_thread<Walk::SingleClock>, grid, block, 0, s, a);
        else launch_next(k_alloc_clock, capped_grid(a.n, 256, a.budget ? kListedBlocks : kThreadBlocks), block > 256 ? block : 256, 0, s, a,
                         p->d_clock_list, (uint32_t)(sm_count() * kClockBlocks * 256));
        break;
    case PBM_DIST_CLOCK:
        launch_next(k_alloc_thread<Walk::DistClock>, grid, block, 0, s, a);
        break;
    case PBM_COLLAB_RW_BM: {
        int cb = serial ? W : block_cfg;
        const int cg = serial ? 1 : capped_grid(a.n, cb, kCollabBlocks * 256);
        if (W == 8) return w64 ? launch_collab_w<8, uint64_t>(a, cg, cb, s) : launch_collab_w<8, uint32_t>(a, cg, cb, s);
        if (W == 16) return w64 ? launch_collab_w<16, uint64_t>(a, cg, cb, s) : launch_collab_w<16, uint32_t>(a, cg, cb, s);
        return w64 ? launch_collab_w<32, uint64_t>(a, cg, cb, s) : launch_collab_w<32, uint32_t>(a, cg, cb, s);
    }
    case PBM_LINKED_LIST: {
        if (!p->fifo_valid) {
            int rc = fifo_build(p, s);
            if (rc) return rc;
        }
        const int blocks = serial ? 1 : (int)((a.n + (uint32_t)block - 1u) / (uint32_t)block);
        if (serial || a.n < (uint32_t)(sm_count() * block * kFifoItems))
            launch_next(k_fifo_alloc<1>, blocks, block, 0, s, a, p->d_fifo, p->d_ring);
        else
            launch_next(k_fifo_alloc<kFifoItems>, (blocks + kFifoItems - 1) / kFifoItems, block, 0, s, a, p->d_fifo, p->d_ring);
        break;
    }
    default:
        return PBM_ERR_INVALID;
    }
    PBM_LAUNCH_CHECK();
    return PBM_OK;
}

}  // namespace

extern "C" {

int pbm_alloc(pbm_pool* pool, const pbm_walk_config* cfg, uint32_t n, uint32_t seed, int32_t* d_ids,
              int32_t* d_steps, void* stream) {
    PBM_ON_POOL_DEVICE(pool);
    if (!pool || (n && !d_ids)) return PBM_ERR_INVALID;
    int rc = check_cfg(cfg);
    if (rc) return rc;
    if (n == 0) return PBM_OK;
    if (cfg->fail_fast && cfg->block_size > kDefaultBlock) {
        // the walks are built for at most that many threads, and a launch of more is refused: refuse it
        // before the budget's passes take pages for it
        std::fprintf(stderr, "[pbm] pbm_alloc: blocks of %d threads cannot be launched\n", cfg->block_size);
        return PBM_ERR_CUDA;
    }
    AllocArgs a = make_args(pool, cfg, n, seed, d_ids, d_steps);
    if (cfg->strategy != PBM_LINKED_LIST) pool->fifo_valid = false;
    if (cfg->fail_fast && cfg->strategy != PBM_LINKED_LIST) {   // the free list counts its pages itself
        std::lock_guard<std::mutex> lk(pool->budget_mu);
        uint32_t slot = 0;
        rc = budget_prepare(pool, n, d_ids, d_steps, (cudaStream_t)stream, &a.budget, &slot);
        if (rc) return rc;
        rc = launch_alloc(pool, cfg, a, false, (cudaStream_t)stream);
        const int rc2 = budget_launched(pool, slot, (cudaStream_t)stream);
        return rc ? rc : rc2;
    }
    return launch_alloc(pool, cfg, a, false, (cudaStream_t)stream);
}

int pbm_alloc_serial(pbm_pool* pool, const pbm_walk_config* cfg, uint32_t n, uint32_t seed,
                     int32_t* d_ids, int32_t* d_steps, void* stream) {
    PBM_ON_POOL_DEVICE(pool);
    if (!pool || (n && !d_ids)) return PBM_ERR_INVALID;
    int rc = check_cfg(cfg);
    if (rc) return rc;
    if (n == 0) return PBM_OK;
    AllocArgs a = make_args(pool, cfg, n, seed, d_ids, d_steps);
    if (cfg->strategy != PBM_LINKED_LIST) pool->fifo_valid = false;
    return launch_alloc(pool, cfg, a, true, (cudaStream_t)stream);
}

int pbm_free(pbm_pool* pool, const pbm_walk_config* cfg, uint32_t n, const int32_t* d_ids, void* stream) {
    PBM_ON_POOL_DEVICE(pool);
    if (!pool || (n && !d_ids)) return PBM_ERR_INVALID;
    int rc = check_cfg(cfg);
    if (rc) return rc;
    if (n == 0) return PBM_OK;
    cudaStream_t s = (cudaStream_t)stream;
    int block = cfg->block_size ? cfg->block_size : kDefaultBlock;
    int grid = (int)((n + (uint32_t)block - 1u) / (uint32_t)block);
    if (cfg->strategy == PBM_LINKED_LIST) {
        if (!pool->fifo_valid) {
            rc = fifo_build(pool, s);
            if (rc) return rc;
        }
        if (n < (uint32_t)(sm_count() * block * kFifoItems))
            launch_next(k_fifo_free<1>, grid, block, 0, s, pool->view, n, d_ids, pool->d_fifo, pool->d_ring, pool->d_stats);
        else
            launch_next(k_fifo_free<kFifoItems>, (grid + kFifoItems - 1) / kFifoItems, block, 0, s, pool->view, n, d_ids, pool->d_fifo, pool->d_ring, pool->d_stats);
    } else {
        pool->fifo_valid = false;
        if (cfg->free_merge && block >= 32) {
            launch_next(k_free_pages<true>, grid, block, 0, s, pool->view, n, d_ids, pool->d_stats);
        } else {
            launch_next(k_free_pages<false>, capped_grid(((uint64_t)n + 3u) / 4u, block, 2048), block, 0, s, pool->view, n, d_ids, pool->d_stats);
        }
    }
    PBM_LAUNCH_CHECK();
    return PBM_OK;
}

static int alloc_runs_impl(pbm_pool* pool, uint32_t n, const int32_t* d_npages, uint32_t seed,
                           uint32_t max_steps, int32_t* d_ids, int32_t* d_steps, bool serial,
                           bool span, void* stream) {
    if (!pool || (n && (!d_ids || !d_npages))) return PBM_ERR_INVALID;
    if (n == 0) return PBM_OK;
    pbm_walk_config c{};
    c.strategy = PBM_RANDOM_WALK_BM;
    c.max_steps = max_steps;
    AllocArgs a = make_args(pool, &c, n, seed, d_ids, d_steps);
    int block = serial ? 1 : kDefaultBlock;
    int grid = serial ? 1 : (int)((n + (uint32_t)block - 1u) / (uint32_t)block);
    if (span) launch_next(k_alloc_runs<true>, grid, block, 0, (cudaStream_t)stream, a, d_npages);
    else launch_next(k_alloc_runs<false>, grid, block, 0, (cudaStream_t)stream, a, d_npages);
    PBM_LAUNCH_CHECK();
    pool->fifo_valid = false;
    return PBM_OK;
}

int pbm_alloc_runs(pbm_pool* pool, uint32_t n, const int32_t* d_npages, uint32_t seed,
                   uint32_t max_steps, int32_t* d_ids, int32_t* d_steps, void* stream) {
    PBM_ON_POOL_DEVICE(pool);
    return alloc_runs_impl(pool, n, d_npages, seed, max_steps, d_ids, d_steps, false, false, stream);
}

int pbm_alloc_runs_serial(pbm_pool* pool, uint32_t n, const int32_t* d_npages, uint32_t seed,
                          uint32_t max_steps, int32_t* d_ids, int32_t* d_steps, void* stream) {
    PBM_ON_POOL_DEVICE(pool);
    return alloc_runs_impl(pool, n, d_npages, seed, max_steps, d_ids, d_steps, true, false, stream);
}

int pbm_alloc_spans(pbm_pool* pool, uint32_t n, const int32_t* d_npages, uint32_t seed,
                    uint32_t max_steps, int32_t* d_ids, int32_t* d_steps, void* stream) {
    PBM_ON_POOL_DEVICE(pool);
    return alloc_runs_impl(pool, n, d_npages, seed, max_steps, d_ids, d_steps, false, true, stream);
}

int pbm_alloc_spans_serial(pbm_pool* pool, uint32_t n, const int32_t* d_npages, uint32_t seed,
                           uint32_t max_steps, int32_t* d_ids, int32_t* d_steps, void* stream) {
    PBM_ON_POOL_DEVICE(pool);
    return alloc_runs_impl(pool, n, d_npages, seed, max_steps, d_ids, d_steps, true, true, stream);
}

int pbm_free_runs(pbm_pool* pool, uint32_t n, const int32_t* d_ids, const int32_t* d_npages, void* stream) {
    PBM_ON_POOL_DEVICE(pool);
    if (!pool || (n && (!d_ids || !d_npages))) return PBM_ERR_INVALID;
    if (n == 0) return PBM_OK;
    int grid = (int)((n + 255u) / 256u);
    launch_next(k_free_runs, grid, 256, 0, (cudaStream_t)stream, pool->view, n, d_ids, d_npages, pool->d_stats);
    PBM_LAUNCH_CHECK();
    pool->fifo_valid = false;
    return PBM_OK;
}

int pbm_claim_write_free(pbm_pool* pool, uint32_t n, uint32_t seed, uint32_t payload_bytes, int hold,
                         uint32_t max_steps, int32_t* d_ids, int32_t* d_steps, void* stream) {
    PBM_ON_POOL_DEVICE(pool);
    if (!pool || (n && !d_ids) || !pool->d_base || payload_bytes > pool->page_size || (payload_bytes & 3u))
        return PBM_ERR_INVALID;
    if (n == 0) return PBM_OK;
    pbm_walk_config c{};
    c.strategy = PBM_RANDOM_WALK;
    c.max_steps = max_steps;
    AllocArgs a = make_args(pool, &c, n, seed, d_ids, d_steps);
    // a batch too small to give every SM two 256-thread blocks runs in
    // 64-thread blocks, so its walks spread over every SM
    const int block = n < (uint32_t)sm_count() * 512u ? 64 : 256;
    int grid = (int)((n + (uint32_t)block - 1u) / (uint32_t)block);
    launch_next(hold ? k_claim_write_free<true> : k_claim_write_free<false>, grid, block, 0, (cudaStream_t)stream, a,
                payload_bytes / 4u);
    PBM_LAUNCH_CHECK();
    pool->fifo_valid = false;
    return PBM_OK;
}

int pbm_gather_pages(pbm_pool* pool, const int32_t* d_ids, uint32_t n, uint32_t bytes_per_page,
                     int32_t* d_out, void* stream) {
    PBM_ON_POOL_DEVICE(pool);
    if (!pool || !pool->d_base || (n && (!d_ids || !d_out)) || bytes_per_page > pool->page_size ||
        (bytes_per_page & 3u) || bytes_per_page == 0)
        return PBM_ERR_INVALID;
    if (n == 0) return PBM_OK;
    gather_rows(pool->view.base, pool->page_size, pool->view.n_pages, d_ids, n, bytes_per_page, d_out, (cudaStream_t)stream);
    PBM_LAUNCH_CHECK();
    return PBM_OK;
}

}  // extern "C"
