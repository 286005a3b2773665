// batch_common.cuh -- pieces shared by the batch kernels (pages and malloc):
// the groups' prefix sums (as a block-level routine and as a kernel), the
// group lookup, the step advance of the graph form, and the graph handle.
#pragma once
#include <cstring>

#include "internal.cuh"

namespace pbm {
namespace {

// Batches with at most this many groups keep their prefix sums in shared
// memory of every block of the persistent kernel.
constexpr uint32_t kFusedGroups = 4096;
constexpr size_t kFusedPrefixBytes = sizeof(unsigned long long) * (kFusedGroups + 1u);

// Group of request q: the g in [lo, n_groups) with prefix[g] <= q < prefix[g+1]
// (prefix in global or shared memory).
__device__ __forceinline__ uint32_t find_group_any(const unsigned long long* prefix, uint32_t n_groups,
                                                   unsigned long long q, uint32_t lo) {
    uint32_t hi = n_groups;
    while (lo + 1u < hi) {
        uint32_t mid = (lo + hi) >> 1;
        if (prefix[mid] <= q) lo = mid; else hi = mid;
    }
    return lo;
}

// Last g in [lo, n_groups) with prefix[g] <= q (prefix[lo] <= q), searched
// by the whole warp: 32 evenly spaced probes and a ballot narrow the range
// 32-fold per round (two rounds for 256 groups).
__device__ __forceinline__ uint32_t find_group_warp(const unsigned long long* prefix, uint32_t n_groups,
                                                    unsigned long long q, uint32_t lo) {
    const uint32_t lane = threadIdx.x & 31u;
    uint32_t hi = n_groups;
    while (hi - lo > 1u) {
        const uint32_t stride = (hi - lo + 31u) >> 5;
        const uint32_t idx = lo + lane * stride;
        const uint32_t b = __ballot_sync(0xffffffffu, idx < hi && prefix[idx] <= q);
        lo += (31u - (uint32_t)__clz((int)b)) * stride;
        hi = min(hi, lo + stride);
    }
    return lo;
}

// Exclusive prefix of the groups' counts into out[0..n] by the whole block
// (blockDim.x a multiple of 32, at most 1024).  Ends with a block barrier.
__device__ __forceinline__ void block_exclusive_prefix(const pbm_group* g, uint32_t n, unsigned long long* out) {
    __shared__ unsigned long long warp_tot[32];
    __shared__ unsigned long long carry;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nwarps = blockDim.x >> 5;
    if (threadIdx.x == 0) carry = 0;
    __syncthreads();
    for (uint32_t base = 0; base < n; base += blockDim.x) {
        uint32_t i = base + threadIdx.x;
        unsigned long long c = i < n ? (unsigned long long)g[i].count : 0ull;
        unsigned long long incl = c;
        for (int d = 1; d < 32; d <<= 1) {
            unsigned long long y = __shfl_up_sync(0xffffffffu, incl, d);
            if (lane >= d) incl += y;
        }
        if (lane == 31) warp_tot[warp] = incl;
        __syncthreads();
        if (warp == 0) {
            unsigned long long t = lane < nwarps ? warp_tot[lane] : 0ull;
            unsigned long long ti = t;
            for (int d = 1; d < 32; d <<= 1) {
                unsigned long long y = __shfl_up_sync(0xffffffffu, ti, d);
                if (lane >= d) ti += y;
            }
            if (lane < nwarps) warp_tot[lane] = ti - t;   // exclusive warp offsets
        }
        __syncthreads();
        unsigned long long excl = carry + warp_tot[warp] + incl - c;
        if (i < n) out[i] = excl;
        __syncthreads();
        if (threadIdx.x == blockDim.x - 1) carry = excl + c;
        __syncthreads();
    }
    if (threadIdx.x == 0) out[n] = carry;
    __syncthreads();
}

// Exclusive prefix of one step's groups (one block of 1024 threads), for
// batches of more groups than a block scans itself.  Replay k of a graph reads
// descriptor table k mod n_steps (so a graph may be replayed any number of times).
__global__ void k_batch_prefix(const pbm_group* groups, uint32_t n_groups, uint32_t step, uint32_t n_steps,
                               unsigned long long* prefix) {
    block_exclusive_prefix(groups + (size_t)(step % n_steps) * n_groups, n_groups, prefix);
}

}  // namespace
}  // namespace pbm

// A captured graph: one kernel (and, for batches of many groups, the prefix kernel
// before it).  Its replays are counted on the host, and the count is written into the
// kernels' parameters before each one, so a launch reads its step with its
// parameters and not from memory.
struct pbm_graph {
    cudaGraph_t graph;
    cudaGraphExec_t exec;
    uint32_t host_step;
    unsigned long long* d_pools;      // the batch kernel's tail-pool counters (may be null)
    unsigned long long* d_prefix;     // the prefix kernel's output (may be null)
    unsigned long long launches_per_replay;
    int device;                       // the pool's device: replays run there
    // the kernel nodes whose parameters carry the step, their launch settings, and
    // the main kernel's argument structure, with the step at step_offset
    cudaGraphNode_t main_node, prefix_node;
    cudaKernelNodeParams main_kp, prefix_kp;
    alignas(16) unsigned char main_args[320];
    size_t step_offset;
    const pbm_group* prefix_groups;
    uint32_t prefix_n_groups, prefix_n_steps;
    // the last replay's end, the stream a plain launch of a one-kernel graph was in (by id: a handle
    // may come back for another stream), and whether replays stay with the graph
    cudaEvent_t done;
    unsigned long long last_stream;
    bool launched, graph_only;
};

namespace pbm {
namespace {

// Captures the graph's kernels -- the prefix kernel unless `fused`, then what launch(stream)
// launches, one kernel whose argument structure is `args` -- and instantiates
// them.  On failure the graph holds no capture.  Captured on a private stream:
// the legacy default stream cannot be.
template <typename Args, typename Launch>
int graph_capture(pbm_graph* g, const Args& args, size_t step_offset, const pbm_group* d_groups, uint32_t n_groups,
                  uint32_t n_steps, bool fused, Launch launch) {
    static_assert(sizeof(Args) <= sizeof(g->main_args), "graph keeps the kernel's arguments");
    std::memcpy(g->main_args, &args, sizeof(Args));
    g->step_offset = step_offset;
    g->prefix_groups = d_groups;
    g->prefix_n_groups = n_groups;
    g->prefix_n_steps = n_steps;
    auto fail = [&](int code) {
        if (g->exec) cudaGraphExecDestroy(g->exec);
        if (g->graph) cudaGraphDestroy(g->graph);
        if (g->done) cudaEventDestroy(g->done);
        g->exec = nullptr;
        g->graph = nullptr;
        g->done = nullptr;
        cudaGetLastError();
        return code;
    };
    cudaStream_t cap = nullptr;
    if (cudaStreamCreateWithFlags(&cap, cudaStreamNonBlocking) != cudaSuccess) return fail(PBM_ERR_CUDA);
    if (cudaStreamBeginCapture(cap, cudaStreamCaptureModeThreadLocal) != cudaSuccess) {
        cudaStreamDestroy(cap);
        return fail(PBM_ERR_CUDA);
    }
    if (!fused) k_batch_prefix<<<1, 1024, 0, cap>>>(d_groups, n_groups, 0u, n_steps, g->d_prefix);
    const int rc = launch(cap);
    const cudaError_t e = cudaStreamEndCapture(cap, &g->graph);
    cudaStreamDestroy(cap);
    if (rc != PBM_OK || e != cudaSuccess) return fail(rc != PBM_OK ? rc : PBM_ERR_CUDA);
    cudaGraphNode_t nodes[2] = {};
    size_t nn = 2;
    if (cudaGraphGetNodes(g->graph, nodes, &nn) != cudaSuccess) return fail(PBM_ERR_CUDA);
    for (size_t i = 0; i < nn && i < 2; ++i) {
        cudaGraphNodeType t;
        cudaKernelNodeParams kp{};
        if (cudaGraphNodeGetType(nodes[i], &t) != cudaSuccess || t != cudaGraphNodeTypeKernel) continue;
        if (cudaGraphKernelNodeGetParams(nodes[i], &kp) != cudaSuccess) return fail(PBM_ERR_CUDA);
        kp.kernelParams = nullptr;   // pointed into the graph; replays pass their own
        kp.extra = nullptr;
        if (kp.func == (void*)k_batch_prefix) {
            g->prefix_node = nodes[i];
            g->prefix_kp = kp;
        } else {
            g->main_node = nodes[i];
            g->main_kp = kp;
        }
    }
    if (!g->main_node || (!fused && !g->prefix_node)) return fail(PBM_ERR_CUDA);
    if (cudaGraphInstantiate(&g->exec, g->graph, 0) != cudaSuccess ||
        cudaEventCreateWithFlags(&g->done, cudaEventDisableTiming) != cudaSuccess)
        return fail(PBM_ERR_CUDA);
    g->launches_per_replay = fused ? 1u : 2u;
    return PBM_OK;
}

}  // namespace
}  // namespace pbm
