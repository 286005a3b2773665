// pbm_device.cuh -- device-side core of the GB300 page manager.
//
// Everything a kernel needs to allocate and free pages of a pool from any
// thread: the pool descriptor, the reference's LCG, the index mapping, and
// the walks (per-thread page probe, per-thread word probe, warp-collaborative
// walk, clustered walk, clock sweeps, contiguous runs) plus frees.
//
// The same inline routines run inside this library's batch kernels and in a
// caller's own kernels through the drop-in headers (RandomWalkBasic.cuh,
// RandomWalkBasic_BM.cuh, CollabRW_BM.cuh, CRW_BM.cuh, RWMalloc.cuh,
// parallelPage.cuh).
//
// Bitmap layout: bit b of 32-bit word w <-> page 32*w + b; bit set = held.
// The 64-bit view reads the same bytes (page 64*w + b), so the storage is
// padded to an even number of 32-bit words and every bit past the last page
// is kept set.  All walks are bounded: after max_steps random jumps a
// request returns -1 instead of trapping or spinning.
#pragma once
#include <cstdint>

namespace pbm {

// Pool descriptor, passed by value (or read from a __device__ global by the
// drop-in API).  32 bytes.
struct PoolView {
    uint32_t* words;      // bitmap, n_words32 (even) 32-bit words
    char*     base;       // page memory (pageAddress), may be null
    uint32_t  n_pages;    // T
    uint32_t  n_words32;  // ceil(T/32)
    uint32_t  n_words64;  // ceil(T/64)
    uint32_t  page_size;  // bytes
};

// Device statistics block (one per pool), updated with block-aggregated atomics.
struct DevStats {
    unsigned long long successes;
    unsigned long long failures;
    unsigned long long steps;
    unsigned long long frees;
    unsigned long long timeouts;   // bounded waits that gave up
    unsigned long long bad_frees;  // malloc frees rejected (outside the pool / double free)
    unsigned long long pad[2];
};

// FIFO free list of the linked-list strategy: a ring of page ids with
// ticket counters.  `avail` is a signed count stored in two's complement.
// Every get and put of every thread hits these counters, so each has a
// 128-byte line (an L2 slice's atomic unit) of its own.
struct FifoState {
    alignas(128) unsigned long long head;    // next get ticket
    alignas(128) unsigned long long tail;    // next put ticket
    alignas(128) unsigned long long avail;   // free pages in the ring
};

constexpr uint32_t kFifoSpinLimit = 1u << 20;   // bounded waits in the free list
constexpr uint32_t kFull32 = 0xffffffffu;
constexpr uint64_t kFull64 = 0xffffffffffffffffull;

// ---------------------------------------------------------------------------
// RNG
// ---------------------------------------------------------------------------

// source/RNG_LCG.cuh:9-12: (1103515245*x + 12345) % (1<<31) in signed 64-bit
// with C truncation, cast to int.  The remainder by 2^31 is a mask of the
// magnitude, so no 64-bit division is issued.
__host__ __device__ __forceinline__ int32_t lcg(int32_t x) {
    long long v = 1103515245LL * (long long)x + 12345LL;
    long long r = v >= 0 ? (v & 0x7fffffffLL) : -((-v) & 0x7fffffffLL);
    return (int32_t)r;
}

// The same step for a state in [0, 2^31), which is every state the walks
// see (request seeds are 31-bit and the LCG keeps non-negative states
// non-negative): (A*x + C) mod 2^31 is then the low 31 bits of the 32-bit
// product, so one multiply-add and a mask replace the 64-bit arithmetic.
__host__ __device__ __forceinline__ int32_t lcg31(int32_t x) {
    return (int32_t)((1103515245u * (uint32_t)x + 12345u) & 0x7fffffffu);
}

// Index in [0, n) from the LCG state's 31 bits by multiply-high.  The
// reference reduces with `(unsigned)x % n`; for power-of-two n that keeps
// only the LCG's low bits, whose short periods make threads with equal low
// seed bits walk identical sequences.  The high bits do not have that flaw.
__host__ __device__ __forceinline__ uint32_t idx_hi(int32_t x, uint32_t n) {
    return (uint32_t)((((unsigned long long)((uint32_t)x & 0x7fffffffu)) * n) >> 31);
}

// Per-request seed: murmur3 fmix32 of (stream seed, request index), 31 bits.
__host__ __device__ __forceinline__ int32_t request_seed(uint32_t S, uint32_t r) {
    uint32_t h = r * 0x9E3779B1u + S * 0x85EBCA77u + 0x165667B1u;
    h ^= h >> 16; h *= 0x85EBCA6Bu;
    h ^= h >> 13; h *= 0xC2B2AE35u;
    h ^= h >> 16;
    return (int32_t)(h & 0x7fffffffu);
}

// splitmix64 output function on a Weyl counter (Bernoulli prefill).
__host__ __device__ __forceinline__ uint64_t hash64(uint64_t seed, uint64_t ctr) {
    uint64_t z = seed * 0xD1B54A32D192ED03ull + (ctr + 1ull) * 0x9E3779B97F4A7C15ull;
    z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
    z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
    return z ^ (z >> 31);
}

// bits lo..hi (inclusive) of a 32-bit word
__host__ __device__ __forceinline__ uint32_t bit_range(uint32_t lo, uint32_t hi) {
    return (hi >= 31u ? kFull32 : ((1u << (hi + 1u)) - 1u)) & ~((1u << lo) - 1u);
}

#ifdef __CUDACC__

// ---------------------------------------------------------------------------
// Word access
// ---------------------------------------------------------------------------

// Bitmap loads bypass L1 (it is not coherent with the L2 atomics); a stale
// value would only waste a probe, the atomic stays authoritative.
__device__ __forceinline__ uint32_t load_word(const uint32_t* p) { return __ldcg(p); }
__device__ __forceinline__ uint64_t load_word(const uint64_t* p) {
    return (uint64_t)__ldcg(reinterpret_cast<const unsigned long long*>(p));
}
__device__ __forceinline__ uint32_t atomic_or(uint32_t* p, uint32_t m) { return atomicOr(p, m); }
__device__ __forceinline__ uint64_t atomic_or(uint64_t* p, uint64_t m) {
    return (uint64_t)atomicOr(reinterpret_cast<unsigned long long*>(p), (unsigned long long)m);
}
__device__ __forceinline__ void atomic_and_noret(uint32_t* p, uint32_t m) { atomicAnd(p, m); }
__device__ __forceinline__ void atomic_and_noret(uint64_t* p, uint64_t m) {
    atomicAnd(reinterpret_cast<unsigned long long*>(p), (unsigned long long)m);
}
__device__ __forceinline__ int popc_w(uint32_t x) { return __popc(x); }
__device__ __forceinline__ int popc_w(uint64_t x) { return __popcll(x); }
__device__ __forceinline__ int ctz_w(uint32_t x) { return __ffs((int)x) - 1; }
__device__ __forceinline__ int ctz_w(uint64_t x) { return __ffsll((long long)x) - 1; }

// Position of the (k+1)-th set bit of m (0 <= k < popc(m)): five halving
// steps, each counting the set bits of the lower half and moving into the
// upper half when k lies beyond them (branch-free, no loop; measured faster
// than __fns in the walks).
__device__ __forceinline__ uint32_t nth_set_bit(uint32_t m, int k) {
    uint32_t pos = 0;
    int c = __popc(m & 0xffffu);
    if (k >= c) { k -= c; pos += 16u; m >>= 16; }
    c = __popc(m & 0xffu);
    if (k >= c) { k -= c; pos += 8u; m >>= 8; }
    c = __popc(m & 0xfu);
    if (k >= c) { k -= c; pos += 4u; m >>= 4; }
    c = __popc(m & 0x3u);
    if (k >= c) { k -= c; pos += 2u; m >>= 2; }
    if (k >= (int)(m & 1u)) pos += 1u;
    return pos;
}

// Lowest k set bits of m (0 <= k <= popc(m)).
__device__ __forceinline__ uint32_t low_bits(uint32_t m, int k) {
    if (k <= 0) return 0u;
    if (k >= __popc(m)) return m;
    return m & ((1u << nth_set_bit(m, k)) - 1u);   // below the (k+1)-th set bit
}
__device__ __forceinline__ uint64_t low_bits(uint64_t m, int k) {
    if (k <= 0) return 0ull;
    uint32_t lo = (uint32_t)m, hi = (uint32_t)(m >> 32);
    int clo = __popc(lo);
    if (k <= clo) return (uint64_t)low_bits(lo, k);
    return (uint64_t)lo | ((uint64_t)low_bits(hi, k - clo) << 32);
}

template <typename Word> struct WordTraits;
template <> struct WordTraits<uint32_t> {
    static constexpr int kBits = 32;
    static constexpr int kShift = 5;
    __device__ static uint32_t full() { return kFull32; }
    __device__ static uint32_t count(const PoolView& v) { return v.n_words32; }
};
template <> struct WordTraits<uint64_t> {
    static constexpr int kBits = 64;
    static constexpr int kShift = 6;
    __device__ static uint64_t full() { return kFull64; }
    __device__ static uint32_t count(const PoolView& v) { return v.n_words64; }
};

// ---------------------------------------------------------------------------
// Per-thread page-probe walk (RandomWalkBasic semantics, on the bitmap):
// probe a random page with one atomicOr of its bit, which takes the page
// when the bit was clear and changes nothing when it was set (the reference
// exchanges each probed map entry, source/RandomWalkBasic.cuh:54-74); steps =
// probes.  One round trip per probe.  Measured on GB300 (churn at 50 / 75 /
// 90 / 95% occupancy): 54 / 30 / 13 / 6.9 G ops/s against 37 / 21 / 11 / 6.7
// reading the word first; only walks that run to their bound in an exhausted
// pool pay for it, with an atomic instead of a load per missed probe.
// ---------------------------------------------------------------------------
__device__ __forceinline__ int32_t walk_page(const PoolView& v, int32_t seed0,
                                             uint32_t max_steps, int32_t* steps_out) {
    int32_t x = seed0 & 0x7fffffff;   // walks run on 31-bit states
    uint32_t s = 0;
    while (s < max_steps) {
        ++s;
        x = lcg31(x);
        uint32_t p = idx_hi(x, v.n_pages);
        uint32_t* wp = v.words + (p >> 5);
        uint32_t bit = 1u << (p & 31u);
        const uint32_t old = atomicOr(wp, bit);
        if (!(old & bit)) {
            if (steps_out) *steps_out = (int32_t)s;
            return (int32_t)p;
        }
    }
    if (steps_out) *steps_out = (int32_t)s;
    return -1;
}

// Affine jump-ahead of the LCG by n steps: lcg31 applied n times to x is
// (an * x + cn) mod 2^31.  The maps of 1, 2, 4, ... steps, each the square of the
// one before, are composed by the bits of n (n < 2^BITS).
template <int BITS>
__device__ __forceinline__ void lcg_jump(uint32_t n, uint32_t& an, uint32_t& cn) {
    uint32_t a = 1103515245u, c = 12345u;
    an = 1u;
    cn = 0u;
#pragma unroll
    for (int k = 0; k < BITS; ++k) {
        if ((n >> k) & 1u) {
            cn = a * cn + c;
            an *= a;
        }
        c = a * c + c;
        a *= a;
    }
}

// The page-probe walks of a whole warp (lanes with `need`, each on its own LCG
// sequence from its seed0); the warp calls converged.  A lane's walk alone is a
// chain of dependent round trips, and the warp, and with it the launch, lasts as
// long as its longest chain while the served lanes idle (250,007 requests on 5 M
// pages at 90%: 8 of 32 lanes worked on average, the longest walk was some 240
// probes).  Here each lane makes its first kOwnProbes probes itself, and then the
// served lanes look ahead for the others: with m lanes unserved, each walk gets
// 2^floor(log2(32 / m)) lanes, and each of these reads the pages of
// kPageAhead consecutive probes (the LCG's state advanced to the first of them at
// once) with all its loads in flight; the first page of a walk that reads as free
// is claimed with the atomicOr.  Every walk tries the same pages in the
// same order and counts the same probes as walk_page; a page read as free but
// lost to another claim counts as held, and the walk goes on just past it.  The
// lanes per walk double from one round to the next at most: reading far ahead
// after a few misses would read pages that a walk in a half-empty pool rarely
// needs.  Measured on GB300 (alloc + free of that launch, us): 114 -> 45; 16,384
// requests at 95%: 88 -> 24; at 2% nothing is left after the own probes (10.4
// both).  Two probes read ahead per lane: 52 and 39; eight: 50 and 21, but 20%
// slower for a million requests at 50%, where the extra loads cost more.
constexpr uint32_t kOwnProbes = 3;
constexpr uint32_t kPageAhead = 4;

__device__ __forceinline__ int32_t walk_page_warp(const PoolView& v, bool need, int32_t seed0,
                                                  uint32_t max_steps, int32_t* steps_out) {
    int32_t x = seed0 & 0x7fffffff;   // walks run on 31-bit states
    uint32_t s = 0;
    int32_t id = -1;
#pragma unroll 1
    for (uint32_t k = 0; k < kOwnProbes; ++k) {
        if (!(need && id < 0 && s < max_steps)) break;
        ++s;
        x = lcg31(x);
        const uint32_t p = idx_hi(x, v.n_pages);
        const uint32_t bit = 1u << (p & 31u);
        if (!(atomicOr(v.words + (p >> 5), bit) & bit)) id = (int32_t)p;
    }
    uint32_t pend = __ballot_sync(kFull32, need && id < 0 && s < max_steps);
    if (pend) {
        const uint32_t lane = threadIdx.x & 31u;
        const uint32_t lt = (1u << lane) - 1u;
        uint32_t aj, cj;                  // jump of lane * kPageAhead steps
        lcg_jump<7>(lane * kPageAhead, aj, cj);
        uint32_t max_sh = 0u;             // log2 of the most lanes one walk may get
        do {
            const uint32_t m = (uint32_t)__popc(pend);
            uint32_t sh = (uint32_t)__clz((int)(m - 1u)) - 27u;   // floor(log2(32 / m)): clz(0) is 32
            if (sh > max_sh) sh = max_sh;
            if (max_sh < 5u) ++max_sh;
            // this lane's place: lane j of the walk of the pending lane of that rank
            const uint32_t j = lane & ((1u << sh) - 1u);
            const uint32_t rank = lane >> sh;
            const uint32_t owner = rank < m ? nth_set_bit(pend, (int)rank) : 0u;
            const uint32_t x0 = (uint32_t)__shfl_sync(kFull32, x, (int)owner);
            const uint32_t s0 = __shfl_sync(kFull32, s, (int)owner) + j * kPageAhead;
            const uint32_t a = __shfl_sync(kFull32, aj, (int)j), c = __shfl_sync(kFull32, cj, (int)j);
            int32_t xj = (int32_t)((a * x0 + c) & 0x7fffffffu);
            uint32_t p[kPageAhead], val[kPageAhead];
#pragma unroll
            for (uint32_t u = 0; u < kPageAhead; ++u) {
                xj = lcg31(xj);
                p[u] = idx_hi(xj, v.n_pages);
                val[u] = (rank < m && s0 < max_steps && u < max_steps - s0) ? load_word(v.words + (p[u] >> 5)) : kFull32;
            }
            uint32_t pc = 0u, k = kPageAhead;   // the first page read as free, the probes up to it
            bool fre = false;
#pragma unroll
            for (int u = (int)kPageAhead - 1; u >= 0; --u) {
                if (!((val[u] >> (p[u] & 31u)) & 1u)) {
                    pc = p[u];
                    k = (uint32_t)u + 1u;
                    fre = true;
                }
            }
            const uint32_t fm = __ballot_sync(kFull32, fre);
            const bool first = fre && !(fm & lt & ~((1u << (lane - j)) - 1u));   // of its walk's lanes
            const uint32_t bit = 1u << (pc & 31u);
            const bool won = first && !(atomicOr(v.words + (pc >> 5), bit) & bit);
            const uint32_t wm = __ballot_sync(kFull32, won);
            // the walk's own lane takes up the result: the first page read as free, else the last one read
            const uint32_t base = ((uint32_t)__popc(pend & lt) << sh) & 31u;   // its walk's first lane
            const uint32_t last = base + (1u << sh) - 1u;
            const uint32_t seen = (fm >> base) << base;
            const uint32_t low = seen ? (uint32_t)__ffs((int)seen) - 1u : 32u;
            const uint32_t src = low <= last ? low : last;
            const uint32_t past = (src - base) * kPageAhead + __shfl_sync(kFull32, k, (int)src);
            const uint32_t ps = __shfl_sync(kFull32, pc, (int)src);
            if ((pend >> lane) & 1u) {
                const uint32_t d = min(past, max_steps - s);   // probes made: 1 .. 32 * kPageAhead
                if ((wm >> src) & 1u) id = (int32_t)ps;
                uint32_t an, cn;
                lcg_jump<8>(d, an, cn);
                x = (int32_t)((an * (uint32_t)x + cn) & 0x7fffffffu);
                s += d;
            }
            pend = __ballot_sync(kFull32, need && id < 0 && s < max_steps);
        } while (pend);
    }
    if (steps_out) *steps_out = (int32_t)s;
    return id;
}

// ---------------------------------------------------------------------------
// Per-thread word-probe walk (RandomWalkBasic_BM semantics): jump to a random
// word, claim its lowest clear bit; on a lost race retry in the same word;
// steps = jumps.  source/RandomWalkBasic_BM.cuh:60-89.  (Taking every clear
// bit with one atomicOr of all ones and handing the rest back is one round
// trip instead of two, but a racer that jumps to a word while its bits are
// held sees it full and jumps again: measured on GB300, 7% more jumps with
// 4,096 walkers on 32,768 words, outside the word-probe model's 3-SE band;
// the collaborative walks use it, where the gain is measured and the model
// still holds.)
// ---------------------------------------------------------------------------
template <typename Word>
__device__ __forceinline__ int32_t walk_word(const PoolView& v, int32_t seed0,
                                             uint32_t max_steps, int32_t* steps_out) {
    using T = WordTraits<Word>;
    Word* words = reinterpret_cast<Word*>(v.words);
    const uint32_t L = T::count(v);
    int32_t x = seed0 & 0x7fffffff;   // walks run on 31-bit states
    uint32_t s = 0;
    while (s < max_steps) {
        ++s;
        x = lcg31(x);
        uint32_t w = idx_hi(x, L);
        Word val = load_word(words + w);
        while (val != T::full()) {
            int b = ctz_w((Word)~val);
            Word bit = (Word)1 << b;
            Word old = atomic_or(words + w, bit);
            if (!(old & bit)) {
                if (steps_out) *steps_out = (int32_t)s;
                return (int32_t)(((uint32_t)w << T::kShift) + (uint32_t)b);
            }
            val = old | bit;
        }
    }
    if (steps_out) *steps_out = (int32_t)s;
    return -1;
}

// ---------------------------------------------------------------------------
// Warp-collaborative walk (CollabRW_BM, source/CollabRW_BM.cuh:114-160,
// restated lock-free).  A group of W lanes (W = 8, 16 or 32, aligned within
// the warp) shares one LCG stream.  Per jump lane i takes word
// (base + i*stride) mod L -- one cache line for the group when stride == 1 --
// with one atomicOr of all ones: the read and the claim of every clear bit
// of the word in a single round trip, as the reference grabs whole words.
// The group keeps as many of those bits as it still needs -- lowest lanes
// and lowest bits first -- and hands the rest straight back with one
// atomicAnd per word (the reference writes whole words back with atomicExch,
// which drops pages freed meanwhile; an AND of exactly the surplus cannot).
// The kept bits go to the needing lanes in lane order (needing lane of rank
// r takes the r-th kept bit).  Needs left unmet go to the next jump.  Every
// bit a lane takes is its own, so no claim is ever lost to a concurrent one;
// surplus bits are held only between the two atomics, and a walker that
// reads them in that window skips them.  (Reading the words first and then
// claiming only the planned bits costs a second dependent round trip per
// jump; on GB300 the single grab is 5-7% faster at 90% occupancy.)
// Lanes whose words coincide (only possible when W*stride > L): only the
// lowest of them grabs (__match_any_sync), so every word is taken once and
// the result is that of lane order.
//
// Every lane of the group must call this converged; `need` says whether the
// lane requests a page.  All lanes of the group report the same step count
// (jumps of the group), as in the reference.  `slots` is unused (kept for
// the callers' shared scratch layout).
// ---------------------------------------------------------------------------
template <int W>
__device__ __forceinline__ int group_incl_scan(int v, uint32_t gl, uint32_t gmask) {
#pragma unroll
    for (int d = 1; d < W; d <<= 1) {
        int y = __shfl_up_sync(gmask, v, d, W);
        if ((int)gl >= d) v += y;
    }
    return v;
}

// Position of the (k+1)-th set bit of m (k < popc(m)).
__device__ __forceinline__ uint32_t nth_bit(uint32_t m, int k) { return nth_set_bit(m, k); }
__device__ __forceinline__ uint32_t nth_bit(uint64_t m, int k) {
    const uint32_t lo = (uint32_t)m;
    const int c = __popc(lo);
    return k < c ? nth_set_bit(lo, k) : 32u + nth_set_bit((uint32_t)(m >> 32), k - c);
}

template <int W, typename Word>
__device__ __forceinline__ int32_t walk_collab(const PoolView& v, bool need, int32_t group_seed,
                                               uint32_t lane_off /* (lane_in_group*stride) % L */,
                                               bool dedupe, uint32_t max_steps,
                                               volatile int32_t* slots, int32_t* steps_out) {
    (void)slots;
    using T = WordTraits<Word>;
    Word* words = reinterpret_cast<Word*>(v.words);
    const uint32_t L = T::count(v);
    const uint32_t lane = threadIdx.x & 31u;
    const uint32_t gl = lane & (uint32_t)(W - 1);                    // lane in group
    const uint32_t gmask = (W == 32) ? kFull32 : (((1u << W) - 1u) << (lane & ~(uint32_t)(W - 1)));
    const uint32_t lt = (1u << lane) - 1u;                           // lanes below me
    int32_t id = -1;
    int32_t x = group_seed & 0x7fffffff;
    uint32_t needm = __ballot_sync(gmask, need);
    uint32_t s = 0;
    while (needm && s < max_steps) {
        ++s;
        x = lcg31(x);
        uint32_t w = idx_hi(x, L) + lane_off;
        if (w >= L) w -= L;
        bool grab = true;
        if (dedupe) grab = (__match_any_sync(gmask, w) & lt) == 0u;   // a lower lane takes this word
        const Word fr = grab ? (Word)~atomic_or(words + w, T::full()) : (Word)0;
        {
            const int cnt = popc_w(fr);
            const int incl = group_incl_scan<W>(cnt, gl, gmask);
            const int n = __popc(needm);
            const Word got = low_bits(fr, n - (incl - cnt));        // kept: the first n in lane order
            const Word extra = fr & (Word)~got;
            if (extra) atomic_and_noret(words + w, (Word)~extra);   // surplus handed back
            const int g = popc_w(got);
            // inclusive prefix of the kept bits, and their total
            const int gincl = min(incl, n);
            const int G = min(__shfl_sync(gmask, incl, W - 1, W), n);
            if (G > 0) {
                // needing lane of rank r takes gained bit r: its source is the
                // first group lane whose inclusive gain exceeds r
                const int r = need && id < 0 ? __popc(needm & lt) : 0;
                int src = 0;
#pragma unroll
                for (int step = W / 2; step >= 1; step >>= 1) {
                    const int gv = __shfl_sync(gmask, gincl, src + step - 1, W);
                    if (gv <= r) src += step;
                }
                const int src_excl = __shfl_sync(gmask, gincl - g, src, W);
                const uint32_t src_w = __shfl_sync(gmask, w, src, W);
                Word src_got;
                if constexpr (sizeof(Word) == 8) {
                    const uint32_t lo = __shfl_sync(gmask, (uint32_t)got, src, W);
                    const uint32_t hi = __shfl_sync(gmask, (uint32_t)(got >> 32), src, W);
                    src_got = ((Word)hi << 32) | (Word)lo;
                } else {
                    src_got = __shfl_sync(gmask, got, src, W);
                }
                if (need && id < 0 && r < G)
                    id = (int32_t)((src_w << T::kShift) + nth_bit(src_got, r - src_excl));
            }
            needm = __ballot_sync(gmask, need && id < 0);
        }
    }
    if (steps_out) *steps_out = (int32_t)s;
    return id;
}

// ---------------------------------------------------------------------------
// The collaborative walk for two requests per lane (a warp serving 64
// requests at a time): the same jump, window, plan and atomics as
// walk_collab<32, Word>, with the needing requests ranked a-requests first
// (lane order), then b-requests; request of rank r takes gained bit r.  The
// jump's fixed costs (window load, scan, claims) are shared by up to 64
// requests.  The whole warp calls converged.
// ---------------------------------------------------------------------------
template <typename Word>
__device__ __forceinline__ void collab_take(int r, int gincl, int g, uint32_t w, Word got, int32_t& id) {
    using T = WordTraits<Word>;
    int src = 0;
#pragma unroll
    for (int step = 16; step >= 1; step >>= 1) {
        const int gv = __shfl_sync(kFull32, gincl, src + step - 1);
        if (gv <= r) src += step;
    }
    const int src_excl = __shfl_sync(kFull32, gincl - g, src);
    const uint32_t src_w = __shfl_sync(kFull32, w, src);
    Word src_got;
    if constexpr (sizeof(Word) == 8) {
        const uint32_t lo = __shfl_sync(kFull32, (uint32_t)got, src);
        const uint32_t hi = __shfl_sync(kFull32, (uint32_t)(got >> 32), src);
        src_got = ((Word)hi << 32) | (Word)lo;
    } else {
        src_got = __shfl_sync(kFull32, got, src);
    }
    id = (int32_t)((src_w << T::kShift) + nth_bit(src_got, r - src_excl));
}

template <typename Word>
__device__ __forceinline__ void walk_collab2(const PoolView& v, bool need_a, bool need_b, int32_t group_seed,
                                             uint32_t lane_off, bool dedupe, uint32_t max_steps, int32_t& id_a,
                                             int32_t& id_b, int32_t* steps_out) {
    using T = WordTraits<Word>;
    Word* words = reinterpret_cast<Word*>(v.words);
    const uint32_t L = T::count(v);
    const uint32_t lane = threadIdx.x & 31u;
    const uint32_t lt = (1u << lane) - 1u;
    id_a = -1;
    id_b = -1;
    int32_t x = group_seed & 0x7fffffff;
    uint32_t ma = __ballot_sync(kFull32, need_a), mb = __ballot_sync(kFull32, need_b);
    uint32_t s = 0;
    while ((ma | mb) && s < max_steps) {
        ++s;
        x = lcg31(x);
        uint32_t w = idx_hi(x, L) + lane_off;
        if (w >= L) w -= L;
        bool grab = true;
        if (dedupe) grab = (__match_any_sync(kFull32, w) & lt) == 0u;   // a lower lane takes this word
        const Word fr = grab ? (Word)~atomic_or(words + w, T::full()) : (Word)0;
        const int cnt = popc_w(fr);
        const int incl = group_incl_scan<32>(cnt, lane, kFull32);
        const int na = __popc(ma);
        const int n = na + __popc(mb);
        const Word got = low_bits(fr, n - (incl - cnt));
        const Word extra = fr & (Word)~got;
        if (extra) atomic_and_noret(words + w, (Word)~extra);
        const int g = popc_w(got);
        const int gincl = min(incl, n);
        const int G = min(__shfl_sync(kFull32, incl, 31), n);
        if (G > 0) {
            const bool wa = need_a && id_a < 0, wb = need_b && id_b < 0;
            const int ra = wa ? __popc(ma & lt) : 0;
            const int rb = wb ? na + __popc(mb & lt) : 0;
            int32_t ta = -1, tb = -1;
            collab_take<Word>(ra, gincl, g, w, got, ta);
            if (__any_sync(kFull32, wb && rb < G)) collab_take<Word>(rb, gincl, g, w, got, tb);
            if (wa && ra < G) id_a = ta;
            if (wb && rb < G) id_b = tb;
        }
        ma = __ballot_sync(kFull32, need_a && id_a < 0);
        mb = __ballot_sync(kFull32, need_b && id_b < 0);
    }
    if (steps_out) *steps_out = (int32_t)s;
}

// ---------------------------------------------------------------------------
// The collaborative walk over an arbitrary set of converged lanes `active`
// (the drop-in form: the reference's getPage runs on __activemask(),
// CollabRW_BM.cuh:119).  Active lane k (k-th set bit of `active`) takes word
// (base + k) mod L with the same grab and hand-back as walk_collab; prefix
// sums use bit-sliced ballots, so inactive lanes never participate.  `slots`
// = 32 ints of shared memory for this warp.
// ---------------------------------------------------------------------------
template <typename Word>
__device__ __forceinline__ int32_t walk_collab_masked(const PoolView& v, uint32_t active, bool need,
                                                      int32_t seed, uint32_t max_steps,
                                                      volatile int32_t* slots, int32_t* steps_out) {
    using T = WordTraits<Word>;
    Word* words = reinterpret_cast<Word*>(v.words);
    const uint32_t L = T::count(v);
    const uint32_t lane = threadIdx.x & 31u;
    const uint32_t lt = (1u << lane) - 1u;
    const uint32_t k = (uint32_t)__popc(active & lt);
    const uint32_t off = k % L;
    const bool dedupe = __popc(active) > (int)L;
    int32_t id = -1;
    int32_t x = seed & 0x7fffffff;
    uint32_t needm = __ballot_sync(active, need);
    uint32_t s = 0;
    while (needm && s < max_steps) {
        ++s;
        x = lcg31(x);
        uint32_t w = idx_hi(x, L) + off;
        if (w >= L) w -= L;
        bool grab = true;
        if (dedupe) grab = (__match_any_sync(active, w) & lt) == 0u;   // a lower lane takes this word
        const Word fr = grab ? (Word)~atomic_or(words + w, T::full()) : (Word)0;
        int cnt = popc_w(fr);
        int pre = 0;
#pragma unroll
        for (int b = 0; b < 7; ++b) pre += __popc(__ballot_sync(active, (cnt >> b) & 1) & lt) << b;
        int n = __popc(needm);
        Word got = low_bits(fr, n - pre);                            // kept; the surplus goes back
        const Word extra = fr & (Word)~got;
        if (extra) atomic_and_noret(words + w, (Word)~extra);
        int g = popc_w(got);
        int gpre = 0, G = 0;
#pragma unroll
        for (int b = 0; b < 7; ++b) {
            uint32_t bm = __ballot_sync(active, (g >> b) & 1);
            gpre += __popc(bm & lt) << b;
            G += __popc(bm) << b;
        }
        int pos = gpre;
        while (got) {
            int b = ctz_w(got);
            got &= got - (Word)1;
            slots[pos++] = (int32_t)(((uint32_t)w << T::kShift) + (uint32_t)b);
        }
        __syncwarp(active);
        if (id < 0 && need) {
            int rank = __popc(needm & lt);
            if (rank < G) id = slots[rank];
        }
        __syncwarp(active);
        needm = __ballot_sync(active, need && id < 0);
    }
    if (steps_out) *steps_out = (int32_t)s;
    return id;
}

// ---------------------------------------------------------------------------
// Clustered walk (CRW_BM, source/CRW_BM.cuh:75-142): resume at the word of
// this slot's last page (the next word once the last page was the word's
// top bit) and claim its lowest clear bit; otherwise random word-probe
// jumps.  steps = claim attempts (the reference does not count jumps).
// `cursor` = last page of the slot or -1; updated on success.
// ---------------------------------------------------------------------------
__device__ __forceinline__ int32_t walk_crw(const PoolView& v, int32_t* cursor, int32_t seed0,
                                            uint32_t max_steps, int32_t* steps_out) {
    const uint32_t L = v.n_words32;
    int32_t s = 0;
    int32_t last = *cursor;
    if (last >= 0) {
        uint32_t w = (uint32_t)last >> 5;
        if (((uint32_t)last & 31u) == 31u) { w += 1u; if (w == L) w = 0; }
        uint32_t val = load_word(v.words + w);
        while (val != kFull32) {
            ++s;
            int b = __ffs((int)~val) - 1;
            uint32_t bit = 1u << b;
            uint32_t old = atomicOr(v.words + w, bit);
            if (!(old & bit)) {
                *cursor = (int32_t)(w * 32u + (uint32_t)b);
                if (steps_out) *steps_out = s;
                return *cursor;
            }
            val = old | bit;
        }
    }
    int32_t x = seed0 & 0x7fffffff;   // walks run on 31-bit states
    for (uint32_t j = 0; j < max_steps; ++j) {
        x = lcg31(x);
        uint32_t w = idx_hi(x, L);
        uint32_t val = load_word(v.words + w);
        while (val != kFull32) {
            ++s;
            int b = __ffs((int)~val) - 1;
            uint32_t bit = 1u << b;
            uint32_t old = atomicOr(v.words + w, bit);
            if (!(old & bit)) {
                *cursor = (int32_t)(w * 32u + (uint32_t)b);
                if (steps_out) *steps_out = s;
                return *cursor;
            }
            val = old | bit;
        }
    }
    if (steps_out) *steps_out = s;
    return -1;
}

// ---------------------------------------------------------------------------
// Clock sweeps.  Single clock: one shared arm, atomicAdd then test-and-set
// (parallelPage.cu:491-509 checks and then exchanges without looking at the
// old value; here the claim is the atomicOr's old bit).  Distributed clock:
// a private arm per slot, linear probe (parallelPage.cu:571-592).
// ---------------------------------------------------------------------------
__device__ __forceinline__ int32_t sweep_single(const PoolView& v, unsigned long long* arm,
                                                uint32_t max_steps, int32_t* steps_out) {
    uint32_t s = 0;
    while (s < max_steps) {
        ++s;
        unsigned long long a = atomicAdd(arm, 1ull);
        uint32_t p = (uint32_t)(a % v.n_pages);
        uint32_t* wp = v.words + (p >> 5);
        uint32_t bit = 1u << (p & 31u);
        if (load_word(wp) & bit) continue;
        if (!(atomicOr(wp, bit) & bit)) {
            if (steps_out) *steps_out = (int32_t)s;
            return (int32_t)p;
        }
    }
    if (steps_out) *steps_out = (int32_t)s;
    return -1;
}

// The single clock's sweep for a warp's requests (lanes with `need`); the warp calls
// converged.  The shared arm is one address, and one atomic per position examined
// (and warp) queued there: 300,007 requests at 75% moved it some 190,000 times.
// Here a warp moves the arm once over a window of positions, long enough to hold the
// free pages it needs at the density seen last, each lane reads one word of the window, and the first free pages in
// sweep order are claimed, one atomicOr per word, and go to the needing lanes in lane
// order.  Pages of the window beyond the need are passed until the arm comes round
// again.  `alone`: no other warp of the launch moves the arm, so the unused end of
// the last window is given back (when the arm is still where this warp left it): a
// launch of one warp leaves the arm just past its last page and passes no free
// page, as the one-thread sweep does.  A request's steps are the positions from the
// page before its own; requests that find no page end after max_steps positions each,
// taken together.  fr_seen: the free pages in 1024 positions, to begin with.
constexpr uint32_t kClockWindow = 896;   // positions: at most 30 words, wrapped windows included

__device__ __forceinline__ uint32_t clock_window(uint32_t m, uint32_t free_pages, uint32_t positions) {
    // m / density, an eighth and 8 positions to spare
    const uint32_t f = free_pages ? free_pages : 1u;
    const uint32_t w = (uint32_t)(((unsigned long long)m * positions) / f);
    const uint32_t p = w + (w >> 3) + 8u;
    return p < kClockWindow ? p : kClockWindow;
}

__device__ __forceinline__ int32_t sweep_single_warp(const PoolView& v, unsigned long long* arm, bool need, uint32_t fr_seen,
                                                     uint32_t max_steps, bool alone, int32_t* steps_out) {
    const uint32_t lane = threadIdx.x & 31u;
    const uint32_t lt = (1u << lane) - 1u;
    const uint32_t T = v.n_pages;
    int32_t id = -1, steps = need ? (int32_t)max_steps : 0;
    uint32_t needm = __ballot_sync(kFull32, need);
    if (!needm) {
        if (steps_out) *steps_out = 0;
        return -1;
    }
    unsigned long long left = (unsigned long long)__popc(needm) * max_steps;   // positions the requests may examine
    uint32_t p_seen = 1024u;
    unsigned long long passed = 0;                                 // positions since the last page claimed
    while (needm && left) {
        const uint32_t m = (uint32_t)__popc(needm);
        uint32_t P = clock_window(m, fr_seen, p_seen);
        if (P > T) P = T;
        if (P > left) P = (uint32_t)left;
        left -= P;
        unsigned long long a0 = 0;
        if (lane == 0u) a0 = atomicAdd(arm, (unsigned long long)P);
        a0 = __shfl_sync(kFull32, a0, 0);
        const uint32_t p0 = (uint32_t)(a0 % T);
        // lane i: word i of the pages p0 .. p0 + P - 1, wrapping past the last page
        const uint32_t w0 = p0 >> 5;
        const uint32_t end_a = min(T, p0 + P);                     // first stretch [p0, end_a)
        const uint32_t n_a = ((end_a + 31u) >> 5) - w0;
        const uint32_t end_b = P - (end_a - p0);                   // second stretch [0, end_b)
        const uint32_t w = lane < n_a ? w0 + lane : lane - n_a;
        const uint32_t lo = lane < n_a ? max(p0, w << 5) : w << 5, hi = lane < n_a ? end_a : end_b;
        uint32_t fr = 0u;
        if ((w << 5) < hi) fr = ~load_word(v.words + w) & bit_range(lo & 31u, min(31u, hi - 1u - (w << 5)));
        int cnt = __popc(fr);
        int incl = group_incl_scan<32>(cnt, lane, kFull32);
        fr_seen = (uint32_t)__shfl_sync(kFull32, incl, 31);
        p_seen = P;
        uint32_t got = low_bits(fr, (int)m - (incl - cnt));
        if (got) got &= ~atomicOr(v.words + w, got);               // less what another claim took first
        const int g = __popc(got);
        const int gincl = group_incl_scan<32>(g, lane, kFull32);
        const int G = __shfl_sync(kFull32, gincl, 31);
        // needing lane of rank r takes page r of those claimed
        const bool mine = (needm >> lane) & 1u;
        const int r = mine ? __popc(needm & lt) : 0;
        int src = 0;
#pragma unroll
        for (int step = 16; step >= 1; step >>= 1)
            if (__shfl_sync(kFull32, gincl, src + step - 1) <= r) src += step;
        const int src_excl = __shfl_sync(kFull32, gincl - g, src);
        const uint32_t src_w = __shfl_sync(kFull32, w, src), src_got = __shfl_sync(kFull32, got, src);
        const bool served = mine && r < G;
        uint32_t at = 0u;                                          // position past the lane's page, from p0
        if (served) {
            id = (int32_t)((src_w << 5) + nth_set_bit(src_got, r - src_excl));
            at = (uint32_t)id >= p0 ? (uint32_t)id - p0 + 1u : (uint32_t)id + (T - p0) + 1u;
        }
        const uint32_t before = needm & lt;
        const uint32_t prev = __shfl_sync(kFull32, at, before ? 31 - __clz((int)before) : 0);
        if (served) steps = (int32_t)min((unsigned long long)max_steps, before ? at - prev : passed + at);
        const uint32_t at_last = __reduce_max_sync(kFull32, at);
        passed = at_last ? P - at_last : passed + P;
        if (alone && G >= (int)m && lane == 31u - (uint32_t)__clz((int)needm) && at < P)
            atomicCAS(arm, a0 + P, a0 + at);                       // the end of the window was not needed
        needm = __ballot_sync(kFull32, mine && !served);
    }
    if (steps_out) *steps_out = steps;
    return id;
}

// The distributed clock's sweep: position by position as far as its steps and its arm
// go, but read a word at a time: a read per position was a round trip per held page.
// Measured on GB300, 250,007 requests and their frees: 50% 21 -> 12.5 us, 90% 52 -> 13,
// 95% 89 -> 15.
__device__ __forceinline__ int32_t sweep_dist(const PoolView& v, uint32_t* arm,
                                              uint32_t max_steps, int32_t* steps_out) {
    uint32_t s = 0, a = *arm;
    int32_t out = -1;
    while (s < max_steps && out < 0) {
        const uint32_t p = a >= v.n_pages ? a - v.n_pages : a;
        uint32_t b = p & 31u;
        // the positions of this word that are left: to its end, the pool's, the bound's
        const uint32_t room = min(min(32u - b, v.n_pages - p), max_steps - s);
        const uint32_t end = b + room;
        uint32_t* wp = v.words + (p >> 5);
        uint32_t val = load_word(wp);
        a = p;
        while (b < end && out < 0) {
            const uint32_t fr = ~val & bit_range(b, end - 1u);
            const uint32_t c = fr ? (uint32_t)__ffs((int)fr) : end;   // past the first free page, or the end
            s += c - b;
            a += c - b;
            if (fr) {
                const uint32_t bit = 1u << (c - 1u);
                val = atomicOr(wp, bit);
                if (!(val & bit)) out = (int32_t)(a - 1u);
            }
            b = c;
        }
    }
    *arm = a;
    if (steps_out) *steps_out = (int32_t)s;
    return out;
}

// ---------------------------------------------------------------------------
// Contiguous run of n pages (1..32) inside one 32-bit word, word-probe walk,
// lowest fitting start, claimed with compare-and-swap so a run is either
// taken whole or not at all (parallelPage.cu:1104-1142 sets the bits with
// atomicOr and reverts the wrong ones on a collision; RWMalloc.cuh:203-248).
// ---------------------------------------------------------------------------
__device__ __forceinline__ uint32_t run_starts(uint32_t f, uint32_t n) {
    uint32_t r = f, len = 1;
    while (len < n) {
        uint32_t sh = len < n - len ? len : n - len;
        r &= r >> sh;
        len += sh;
    }
    return r;
}

__device__ __forceinline__ int32_t walk_run(const PoolView& v, uint32_t n, int32_t seed0,
                                            uint32_t max_steps, int32_t* steps_out) {
    const uint32_t L = v.n_words32;
    int32_t x = seed0 & 0x7fffffff;   // walks run on 31-bit states
    uint32_t s = 0;
    while (s < max_steps) {
        ++s;
        x = lcg31(x);
        uint32_t w = idx_hi(x, L);
        uint32_t val = load_word(v.words + w);
        for (int tries = 0; tries < 64; ++tries) {
            uint32_t r = run_starts(~val, n);
            if (!r) break;
            uint32_t st = (uint32_t)(__ffs((int)r) - 1);
            uint32_t m = (n >= 32u ? kFull32 : ((1u << n) - 1u)) << st;
            uint32_t old = atomicCAS(v.words + w, val, val | m);
            if (old == val) {
                if (steps_out) *steps_out = (int32_t)s;
                return (int32_t)(w * 32u + st);
            }
            val = old;
        }
    }
    if (steps_out) *steps_out = (int32_t)s;
    return -1;
}

// ---------------------------------------------------------------------------
// Runs that may cross word boundaries (getXPage*_BM / getNPage without the
// one-word limit of parallelPage.cu:1104-1142 and RWMalloc.cuh:203-248).
// Per jump the walk scans words w, w+1, ... (at most ceil(n/32) + 1 of them,
// never past the last word), tracking the free run that reaches the top bit
// of the previous word: a run is found where that run plus the current
// word's free low bits reaches n, or -- for n <= 32 -- inside the current
// word (lowest start).  The run is then claimed word by word with atomicOr;
// if a word had lost some of its bits to another claim, every bit this claim
// set is released again and the walk jumps anew.  steps = jumps.
// ---------------------------------------------------------------------------
constexpr uint32_t kMaxSpanPages = 1u << 16;

// mask of the pages of run [p0, p0+n) that lie in word ww
__host__ __device__ __forceinline__ uint32_t span_mask(uint32_t p0, uint32_t n, uint32_t ww) {
    const uint32_t a = p0 >> 5, b = (p0 + n - 1u) >> 5;
    return bit_range(ww == a ? (p0 & 31u) : 0u, ww == b ? ((p0 + n - 1u) & 31u) : 31u);
}

// First run of n <= 32 free pages in words w (value v0) and w+1 (value v1,
// all ones past the last word): inside w, across the boundary, inside w+1.
__device__ __forceinline__ int32_t span_in_pair(uint32_t w, uint32_t v0, uint32_t v1, uint32_t n, uint32_t L) {
    uint32_t r = run_starts(~v0, n);
    if (r) return (int32_t)(w * 32u + (uint32_t)(__ffs((int)r) - 1));
    const uint32_t hi = v0 ? (uint32_t)__clz((int)v0) : 32u;
    if (w + 1u >= L) return -1;
    const uint32_t lo = v1 ? (uint32_t)(__ffs((int)v1) - 1) : 32u;
    if (hi > 0u && hi + lo >= n) return (int32_t)(w * 32u + 32u - hi);
    r = run_starts(~v1, n);
    if (r) return (int32_t)((w + 1u) * 32u + (uint32_t)(__ffs((int)r) - 1));
    return -1;
}

// First run of n free pages seen from word w on (-1 if none in the window).
__device__ __forceinline__ int32_t find_span(const PoolView& v, uint32_t w, uint32_t n) {
    const uint32_t L = v.n_words32;
    if (n <= 32u) {
        // two-word window, both loads in flight together (same result as the loop below)
        const uint32_t v0 = load_word(v.words + w);
        const uint32_t v1 = w + 1u < L ? load_word(v.words + w + 1u) : kFull32;
        return span_in_pair(w, v0, v1, n, L);
    }
    const uint32_t nscan = (n + 31u) / 32u + 1u;
    uint32_t run = 0, start = 0;   // free pages ending at the top of the previous word
    for (uint32_t k = 0; k < nscan && w + k < L; ++k) {
        const uint32_t ww = w + k;
        const uint32_t val = load_word(v.words + ww);
        const uint32_t lo = val ? (uint32_t)(__ffs((int)val) - 1) : 32u;   // free low bits
        if (run > 0u && run + lo >= n) return (int32_t)start;
        if (n <= 32u) {
            const uint32_t r = run_starts(~val, n);
            if (r) return (int32_t)(ww * 32u + (uint32_t)(__ffs((int)r) - 1));
        }
        if (val == 0u) {
            if (run == 0u) start = ww * 32u;
            run += 32u;
        } else {
            const uint32_t hi = (uint32_t)__clz((int)val);            // free top bits
            run = hi;
            start = ww * 32u + 32u - hi;
        }
    }
    return -1;
}

__device__ __forceinline__ void free_span(const PoolView& v, int32_t id, uint32_t n) {
    const uint32_t p0 = (uint32_t)id;
    for (uint32_t ww = p0 >> 5; ww <= (p0 + n - 1u) >> 5; ++ww) atomicAnd(v.words + ww, ~span_mask(p0, n, ww));
}

// Claims the run of n pages at p0 word by word; on a word that lost bits to
// another claim, every bit this claim set is released again.
__device__ __forceinline__ bool claim_span(const PoolView& v, uint32_t p0, uint32_t n) {
    const uint32_t a = p0 >> 5, b = (p0 + n - 1u) >> 5;
    uint32_t ww = a;
    for (; ww <= b; ++ww) {
        const uint32_t m = span_mask(p0, n, ww);
        const uint32_t old = atomicOr(v.words + ww, m);
        if (old & m) {                                   // lost part of the run
            if (m & ~old) atomicAnd(v.words + ww, ~(m & ~old));
            break;
        }
    }
    if (ww > b) return true;
    for (uint32_t k = a; k < ww; ++k) atomicAnd(v.words + k, ~span_mask(p0, n, k));   // roll back
    return false;
}

// claim_span for a run of at most 32 pages (one word or two): both words' atomics are in
// flight together (524,288 mallocs + frees 55.9 -> 53.9 us, 20,000 runs of 1..32 pages and
// their frees at 10% 22.8 -> 19.7).
__device__ __forceinline__ bool claim_pair(const PoolView& v, uint32_t p0, uint32_t n) {
    const uint32_t a = p0 >> 5, b = (p0 + n - 1u) >> 5;
    const uint32_t ma = span_mask(p0, n, a), mb = b != a ? span_mask(p0, n, b) : 0u;
    const uint32_t oa = atomicOr(v.words + a, ma);
    const uint32_t ob = mb ? atomicOr(v.words + b, mb) : 0u;
    if (!((oa & ma) | (ob & mb))) return true;
    if (ma & ~oa) atomicAnd(v.words + a, ~(ma & ~oa));   // lost part of the run: what was set goes back
    if (mb & ~ob) atomicAnd(v.words + b, ~(mb & ~ob));
    return false;
}

// Random jumps until a run of n free pages is claimed (steps = jumps).  For
// n <= 32 the walk is pipelined: the LCG fixes every jump's words in
// advance, so the next kSpanAhead jumps' two words are in flight while a
// jump is judged and claimed, and the same words are examined in the same
// order.  Measured on the malloc workload (GB300): 1.64 G ops/s one jump
// ahead, 1.46 two ahead, 1.41 three ahead, 1.36 unpipelined.
constexpr int kSpanAhead = 1;
__device__ __forceinline__ int32_t walk_span(const PoolView& v, uint32_t n, int32_t seed0,
                                             uint32_t max_steps, int32_t* steps_out) {
    const uint32_t L = v.n_words32;
    int32_t x = seed0 & 0x7fffffff;   // walks run on 31-bit states
    uint32_t s = 0;
    if (n <= 32u && max_steps > 0u) {
        // ring of the next kSpanAhead jumps' words, loads in flight
        uint32_t pw[kSpanAhead], p0[kSpanAhead], p1[kSpanAhead];
#pragma unroll
        for (int k = 0; k < kSpanAhead; ++k) {
            x = lcg31(x);
            pw[k] = idx_hi(x, L);
            p0[k] = (uint32_t)k < max_steps ? load_word(v.words + pw[k]) : kFull32;
            p1[k] = (uint32_t)k < max_steps && pw[k] + 1u < L ? load_word(v.words + pw[k] + 1u) : kFull32;
        }
        while (s < max_steps) {
            const uint32_t w = pw[0], v0 = p0[0], v1 = p1[0];
            ++s;
#pragma unroll
            for (int k = 0; k + 1 < kSpanAhead; ++k) {
                pw[k] = pw[k + 1];
                p0[k] = p0[k + 1];
                p1[k] = p1[k + 1];
            }
            x = lcg31(x);                                  // jump s + kSpanAhead
            pw[kSpanAhead - 1] = idx_hi(x, L);
            const bool more = s + (uint32_t)kSpanAhead <= max_steps;
            p0[kSpanAhead - 1] = more ? load_word(v.words + pw[kSpanAhead - 1]) : kFull32;
            p1[kSpanAhead - 1] = more && pw[kSpanAhead - 1] + 1u < L ? load_word(v.words + pw[kSpanAhead - 1] + 1u)
                                                                     : kFull32;
            const int32_t found = span_in_pair(w, v0, v1, n, L);
            if (found >= 0 && claim_span(v, (uint32_t)found, n)) {
                if (steps_out) *steps_out = (int32_t)s;
                return found;
            }
        }
        if (steps_out) *steps_out = (int32_t)s;
        return -1;
    }
    while (s < max_steps) {
        ++s;
        x = lcg31(x);
        const int32_t found = find_span(v, idx_hi(x, L), n);
        if (found < 0) continue;
        if (claim_span(v, (uint32_t)found, n)) {
            if (steps_out) *steps_out = (int32_t)s;
            return found;
        }
    }
    if (steps_out) *steps_out = (int32_t)s;
    return -1;
}

// Runs of need_n <= 32 pages (0 = none) for the lanes of a whole warp, each
// lane on its own LCG sequence from seed0; steps = jumps.  Every needing
// lane first takes kOwnJumps jumps of its own (all in parallel; one, two, three:
// 30,000 runs of 1..8 pages and their frees on 2^18 pages took 19.8, 14.6, 13.3 us, 20,000
// of 1..32 on 2^20 pages 22.2, 22.9, 23.3).  The walks still unserved
// then share the warp for kShareRounds rounds: with m of them each gets
// 2^floor(log2(32 / m)) lanes, lane j of a walk judging its jump s + j + 1 (its LCG
// state advanced j + 1 steps at once), and the runs found are claimed in jump order, the
// walks side by side.  Those that are left look for runs that are rare, in a pool that is
// nearly full, and are walked one after the other with all lanes and kSpanWide jumps a
// lane in flight.  In a run without races a lane gets the page the one-lane walk would
// give it, after the same jumps.  Measured on GB300: mallocs of 16 B .. 64 KiB and their
// frees, 524,288 into 2^22 pages, one walk at a time 62 us, sharing 58; 192,155 into
// 1.5 M pages 48 and 33; but the malloc trace that outgrows its pool, where a quarter of
// the requests fail after 512 jumps, 5.1 and 4.6 G ops/s, and 6.2 with both.
// The whole warp calls converged.
constexpr uint32_t kOwnJumps = 2;
constexpr uint32_t kShareRounds = 3;
constexpr uint32_t kSpanWide = 2;

__device__ __forceinline__ int32_t walk_span_warp(const PoolView& v, uint32_t need_n, int32_t seed0,
                                                  uint32_t max_steps, int32_t* steps_out) {
    const uint32_t lane = threadIdx.x & 31u;
    const uint32_t lt = (1u << lane) - 1u;
    const uint32_t L = v.n_words32;
    int32_t x = seed0 & 0x7fffffff;   // walks run on 31-bit states
    uint32_t s = 0;
    int32_t id = -1;
#pragma unroll 1
    for (uint32_t k = 0; k < kOwnJumps; ++k) {
        if (!(need_n > 0u && id < 0 && s < max_steps)) break;
        ++s;
        x = lcg31(x);
        const uint32_t w = idx_hi(x, L);
        const uint32_t v0 = load_word(v.words + w);
        const uint32_t v1 = w + 1u < L ? load_word(v.words + w + 1u) : kFull32;
        const int32_t f = span_in_pair(w, v0, v1, need_n, L);
        if (f >= 0 && claim_pair(v, (uint32_t)f, need_n)) id = f;
    }
    uint32_t pend = __ballot_sync(kFull32, need_n > 0u && id < 0 && s < max_steps);
    uint32_t aj = 0u, cj = 0u;                             // jump ahead by lane + 1 steps
    if (pend) lcg_jump<6>(lane + 1u, aj, cj);
    for (uint32_t round = 0; pend && round < kShareRounds; ++round) {
        const uint32_t m = (uint32_t)__popc(pend);
        const uint32_t sh = (uint32_t)__clz((int)(m - 1u)) - 27u;   // floor(log2(32 / m)): clz(0) is 32
        const uint32_t j = lane & ((1u << sh) - 1u);
        const uint32_t rank = lane >> sh;
        const uint32_t owner = rank < m ? nth_set_bit(pend, (int)rank) : 0u;
        const uint32_t x0 = (uint32_t)__shfl_sync(kFull32, x, (int)owner);
        const uint32_t n0 = __shfl_sync(kFull32, need_n, (int)owner);
        const uint32_t s0 = __shfl_sync(kFull32, s, (int)owner);
        const uint32_t a = __shfl_sync(kFull32, aj, (int)j), c = __shfl_sync(kFull32, cj, (int)j);
        const int32_t xj = (int32_t)((a * x0 + c) & 0x7fffffffu);
        const uint32_t wj = idx_hi(xj, L);
        int32_t fj = -1;
        if (rank < m && j < max_steps - s0) {
            const uint32_t a0 = load_word(v.words + wj);
            const uint32_t a1 = wj + 1u < L ? load_word(v.words + wj + 1u) : kFull32;
            fj = span_in_pair(wj, a0, a1, n0, L);
        }
        // claims in jump order: each walk's first candidate, the next one where that was lost
        const uint32_t gm = (uint32_t)(((1ull << (1u << sh)) - 1ull) << (lane - j));   // this walk's lanes
        uint32_t open = __ballot_sync(kFull32, fj >= 0), won = 0u;
        while (open) {
            const bool first = ((open >> lane) & 1u) && !(open & gm & lt);
            const bool ok = first && claim_pair(v, (uint32_t)fj, n0);
            won |= __ballot_sync(kFull32, ok);
            open = __ballot_sync(kFull32, ((open >> lane) & 1u) && !first && !(won & gm));
        }
        const uint32_t base = ((uint32_t)__popc(pend & lt) << sh) & 31u;   // the first lane of this lane's walk
        const uint32_t last = base + (1u << sh) - 1u;
        const uint32_t mine = (won >> base) << base;
        const uint32_t low = mine ? (uint32_t)__ffs((int)mine) - 1u : 32u;
        const uint32_t src = low <= last ? low : last;
        const int32_t xs = __shfl_sync(kFull32, xj, (int)src);
        const int32_t fs = __shfl_sync(kFull32, fj, (int)src);
        if ((pend >> lane) & 1u) {
            s += min(src - base + 1u, max_steps - s);
            x = xs;
            if (low <= last) id = fs;
        }
        pend = __ballot_sync(kFull32, need_n > 0u && id < 0 && s < max_steps);
    }
    // the walks that are left, in a pool where their runs are rare: one after the other with the
    // whole warp, kSpanWide jumps a lane in flight
    while (pend) {
        const int l0 = __ffs((int)pend) - 1;
        uint32_t x0 = (uint32_t)__shfl_sync(kFull32, x, l0);
        const uint32_t n0 = __shfl_sync(kFull32, need_n, l0);
        uint32_t s0 = __shfl_sync(kFull32, s, l0);
        int32_t got = -1;
        while (got < 0 && s0 < max_steps) {
            uint32_t wj[kSpanWide], a0[kSpanWide], a1[kSpanWide];
#pragma unroll
            for (uint32_t u = 0; u < kSpanWide; ++u) {
                const uint32_t xj = (aj * x0 + cj) & 0x7fffffffu;      // jump s0 + 32 u + lane + 1
                x0 = __shfl_sync(kFull32, xj, 31);
                wj[u] = idx_hi((int32_t)xj, L);
                const bool in = 32u * u + lane < max_steps - s0;
                a0[u] = in ? load_word(v.words + wj[u]) : kFull32;
                a1[u] = in && wj[u] + 1u < L ? load_word(v.words + wj[u] + 1u) : kFull32;
            }
#pragma unroll
            for (uint32_t u = 0; u < kSpanWide; ++u) {
                if (got >= 0) break;
                const int32_t fj = span_in_pair(wj[u], a0[u], a1[u], n0, L);
                uint32_t open = __ballot_sync(kFull32, fj >= 0);
                while (open) {                                         // claims in jump order
                    const int j = __ffs((int)open) - 1;
                    open &= open - 1u;
                    const bool ok = (int)lane == j && claim_pair(v, (uint32_t)fj, n0);
                    if (__any_sync(kFull32, ok)) {
                        got = __shfl_sync(kFull32, fj, j);
                        s0 += 32u * u + (uint32_t)j + 1u;
                        break;
                    }
                }
            }
            if (got < 0) s0 = max_steps - s0 < 32u * kSpanWide ? max_steps : s0 + 32u * kSpanWide;
        }
        if ((int)lane == l0) {
            id = got;
            s = s0;
        }
        pend &= pend - 1u;
    }
    if (steps_out) *steps_out = (int32_t)s;
    return id;
}

// ---------------------------------------------------------------------------
// FIFO free list (linked-list strategy, parallelPage.cu:342-440, restated
// lock-free).  get: reserve one free page on `avail`, take a head ticket,
// exchange the ring slot with -1 (bounded wait for the put that holds the
// ticket); put: take a tail ticket, CAS the id into the empty slot (bounded
// wait).  A wait that runs out records a timeout and returns -1 / false.
// The bitmap is kept in step so occupancy and invariants read the same.
// ---------------------------------------------------------------------------
__device__ __forceinline__ int32_t fifo_get(const PoolView& v, FifoState* st, int32_t* ring,
                                            DevStats* stats, int32_t* spins) {
    unsigned long long old = atomicAdd(&st->avail, ~0ull);   // avail -= 1
    if ((long long)old <= 0) {
        atomicAdd(&st->avail, 1ull);
        if (spins) *spins = 0;
        return -1;
    }
    unsigned long long t = atomicAdd(&st->head, 1ull);
    int32_t* slot = ring + (t % v.n_pages);
    uint32_t k = 0;
    int32_t id = atomicExch(slot, -1);
    while (id < 0 && k < kFifoSpinLimit) {
        __nanosleep(64);
        ++k;
        id = atomicExch(slot, -1);
    }
    if (spins) *spins = (int32_t)k + 1;
    if (id < 0) {
        atomicAdd(&stats->timeouts, 1ull);
        return -1;
    }
    atomicOr(v.words + ((uint32_t)id >> 5), 1u << ((uint32_t)id & 31u));
    return id;
}

__device__ __forceinline__ bool fifo_put(const PoolView& v, FifoState* st, int32_t* ring,
                                         DevStats* stats, int32_t id) {
    atomicAnd(v.words + ((uint32_t)id >> 5), ~(1u << ((uint32_t)id & 31u)));
    unsigned long long t = atomicAdd(&st->tail, 1ull);
    int32_t* slot = ring + (t % v.n_pages);
    uint32_t k = 0;
    while (atomicCAS(slot, -1, id) != -1) {
        if (++k >= kFifoSpinLimit) {
            atomicAdd(&stats->timeouts, 1ull);
            return false;
        }
        __nanosleep(64);
    }
    atomicAdd(&st->avail, 1ull);
    return true;
}

// ---------------------------------------------------------------------------
// Frees.
// ---------------------------------------------------------------------------
__device__ __forceinline__ void free_page(const PoolView& v, int32_t id) {
    atomicAnd(v.words + ((uint32_t)id >> 5), ~(1u << ((uint32_t)id & 31u)));
}

__device__ __forceinline__ void free_run(const PoolView& v, int32_t id, uint32_t n) {
    uint32_t st = (uint32_t)id & 31u;
    uint32_t m = (n >= 32u ? kFull32 : ((1u << n) - 1u)) << st;
    atomicAnd(v.words + ((uint32_t)id >> 5), ~m);
}

// Warp-aggregated free: lanes freeing pages of the same word merge their
// bits (__match_any_sync + __reduce_or_sync) and one lane issues the AND.
// `active` = lanes calling converged; lanes with id < 0 free nothing.
__device__ __forceinline__ void free_page_warp(const PoolView& v, uint32_t active, int32_t id) {
    const uint32_t lane = threadIdx.x & 31u;
    uint32_t w = id >= 0 ? ((uint32_t)id >> 5) : 0xffffffffu;
    uint32_t bit = id >= 0 ? (1u << ((uint32_t)id & 31u)) : 0u;
    uint32_t peers = __match_any_sync(active, w);
    uint32_t merged = __reduce_or_sync(peers, bit);
    if (id >= 0 && (__ffs((int)peers) - 1) == (int)lane) atomicAnd(v.words + w, ~merged);
}

// ---------------------------------------------------------------------------
// Launch budget: fail fast in an exhausted pool.  A pass over the bitmap just
// before the launch counts the free pages F.  Request r of the launch may
// take a page only if r < F: the requests past the pages that were free
// fail at once instead of walking to their step bound, and no more pages are
// granted than were free at the start -- with no atomic at all, so the
// launch never contends on a shared counter.  When the launch asks for at
// least half of the F free pages (`list_mode`), the pass also claims them, the
// r-th free page in ascending order for request r, and refuses the requests past F; only
// those whose page another stream took in between (`lost` of them, their ids kLostPage) are
// left to walk.  A null budget grants every request.
// ---------------------------------------------------------------------------
struct LaunchBudget {
    long long free_at_start;    // F
    int32_t list_mode;          // 1: requests 0 .. F - 1 served in order, the others refused
    uint32_t lost;              // but for these
};
constexpr int32_t kLostPage = -2;

__device__ __forceinline__ bool budget_grants(const LaunchBudget* b, unsigned long long r) {
    return !b || (long long)r < __ldcg(&b->free_at_start);
}

__device__ __forceinline__ void* page_address(const PoolView& v, int32_t id) {
    return (void*)(v.base + (size_t)(uint32_t)id * v.page_size);
}

__device__ __forceinline__ int32_t page_id(const PoolView& v, const void* p) {
    size_t off = (size_t)((const char*)p - v.base);
    if ((const char*)p < v.base || off >= (size_t)v.n_pages * v.page_size) return -1;
    return (int32_t)(off / v.page_size);
}

#endif  // __CUDACC__
}  // namespace pbm
