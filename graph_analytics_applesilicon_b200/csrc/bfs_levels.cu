// bfs_levels.cu -- the host-driven BFS forms: one launch or launch sequence and
// one host wait per level, as the reference's GpuBfs::run* loops
// (src/metal/bfs_gpu.mm:115-429).  They are the "plain" forms the persistent
// kernel is measured against, and the drop-in for gpu_vertex / gpu_naive /
// gpu_binned / gpu_edge / gpu_do.
//
// Kernels are new sm_100a code: warp-aggregated queue appends (__ballot_sync
// + one atomic per warp), CAS claims on dist, shared-memory staging of the
// scanned frontier degrees in the edge-balanced expansion, and bitmap
// frontiers with __ballot_sync word assembly in the bottom-up step.
#include <algorithm>
#include <atomic>
#include <chrono>

#include "bfs.hpp"
#include "bfs_device.cuh"
#include "host_cpu.hpp"

namespace gb {

uint32_t checkTg(uint32_t tg) {
    if (tg < 32 || tg > 1024 || tg % 32 != 0)
        throw Error(GB_ERR_ARG, "threadgroup size must be a multiple of 32 in [32, 1024]");
    return tg;
}

void validateOptions(const gb_bfs_options& o) {
    checkTg(o.tg);
    if (o.ept == 0) throw Error(GB_ERR_ARG, "ept must be >= 1");
    if (o.ept > 64) throw Error(GB_ERR_ARG, "ept must be <= 64");
    if (!(o.alpha > 0) || !(o.beta > 0)) throw Error(GB_ERR_ARG, "alpha and beta must be > 0");
    if (o.force_strategy >= GB_NUM_STRATS) throw Error(GB_ERR_ARG, "force_strategy out of range");
    if (o.block != 0 && o.block != 256 && o.block != 512)
        throw Error(GB_ERR_ARG, "persistent block size must be 256 or 512");
    if (o.selector > GB_SELECT_LEARNED) throw Error(GB_ERR_ARG, "unknown selector");
    if (o.in_flight > (uint32_t)kMaxInFlight)
        throw Error(GB_ERR_ARG, "in_flight must be at most " + std::to_string(kMaxInFlight));
}

namespace {

using Stats = GbLevelStats;

__device__ __forceinline__ bool claimDist(uint32_t* dist, uint32_t u, uint32_t value) {
    // Plain load first: skips the atomic for already-visited vertices.
    if (*reinterpret_cast<volatile uint32_t*>(&dist[u]) != kInf) return false;
    return atomicCAS(&dist[u], kInf, value) == kInf;
}

__device__ __forceinline__ void addStats(Stats* s, unsigned long long frontier, unsigned long long edges,
                                         unsigned long long nextEdges) {
    frontier = warpSum(frontier);
    edges = warpSum(edges);
    nextEdges = warpSum(nextEdges);
    if (laneId() == 0) {
        if (frontier) atomicAdd(&s->frontier, frontier);
        if (edges) atomicAdd(&s->edges, edges);
        if (nextEdges) atomicAdd(&s->nextEdges, nextEdges);
    }
}

__global__ void initDistKernel(uint32_t* dist, uint64_t n, uint32_t source) {
    const uint64_t stride = (uint64_t)gridDim.x * blockDim.x;
    const uint64_t n4 = n / 4;
    uint4* d4 = reinterpret_cast<uint4*>(dist);
    for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n4; i += stride)
        d4[i] = make_uint4(kInf, kInf, kInf, kInf);
    for (uint64_t i = n4 * 4 + (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += stride) dist[i] = kInf;
}

__global__ void setSourceKernel(uint32_t* dist, uint32_t source) { dist[source] = 0; }

// gpu_vertex: thread per vertex every level; plain stores (all writers store
// level + 1, readers only test for "unreached"), so `found` may overcount and
// is used only as "something changed" (src/shaders/bfs.metal:45-54).
__global__ void vertexLevelKernel(const uint32_t* row_ptr, const uint32_t* col_idx, uint32_t* dist, uint64_t n,
                                  uint32_t level, Stats* s) {
    const uint64_t stride = (uint64_t)gridDim.x * blockDim.x;
    unsigned long long frontier = 0, edges = 0, found = 0;
    for (uint64_t base = (uint64_t)blockIdx.x * blockDim.x; base < n; base += stride) {
        uint64_t v = base + threadIdx.x;
        if (v < n && dist[v] == level) {
            uint32_t b = row_ptr[v], e = row_ptr[v + 1];
            frontier++;
            edges += e - b;
            for (uint32_t i = b; i < e; ++i) {
                uint32_t u = col_idx[i];
                if (dist[u] == kInf) {
                    dist[u] = level + 1;
                    found++;
                }
            }
        }
    }
    found = warpSum(found);
    if (laneId() == 0 && found) atomicAdd(&s->found, (unsigned)min(found, 0xFFFFFFFFull));
    addStats(s, frontier, edges, 0);
}

// gpu_naive: thread per frontier vertex, CAS claim, one atomic append per claim.
__global__ void naiveLevelKernel(const uint32_t* row_ptr, const uint32_t* col_idx, uint32_t* dist, Stats* s,
                                 const uint32_t* queue, uint32_t* next, uint32_t size, uint32_t level) {
    unsigned long long frontier = 0, edges = 0;
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < size) {
        uint32_t v = queue[i], b = row_ptr[v], e = row_ptr[v + 1];
        frontier = 1;
        edges = e - b;
        for (uint32_t k = b; k < e; ++k) {
            uint32_t u = col_idx[k];
            if (claimDist(dist, u, level + 1)) next[atomicAdd(&s->found, 1u)] = u;
        }
    }
    addStats(s, frontier, edges, 0);
}

// ----------------------------------------------------------- gpu_binned

struct BinArgs {
    const uint32_t* row_ptr;
    const uint32_t* col_idx;
    uint32_t* dist;
    Stats* s;
    const uint32_t* queue;
    uint32_t* q[3];
    uint32_t size, level, smallMax, largeMin;
};

// Discovery: claim u and append it to the next-level queue of its degree bin.
// Called by all 32 lanes together.
__device__ __forceinline__ void binVisit(const BinArgs& a, bool has, uint32_t e) {
    uint32_t u = has ? a.col_idx[e] : 0u;
    bool claimed = has && claimDist(a.dist, u, a.level + 1);
    if (!__any_sync(kFull, claimed)) return;
    uint32_t udeg = claimed ? a.row_ptr[u + 1] - a.row_ptr[u] : 0u;
    uint32_t bin = udeg < a.smallMax ? 0u : (udeg < a.largeMin ? 1u : 2u);
#pragma unroll
    for (int b = 0; b < 3; ++b) {
        bool want = claimed && bin == (uint32_t)b;
        if (!__any_sync(kFull, want)) continue;
        uint32_t pos = warpAppend(want, &a.s->bin[b]);
        if (want) a.q[b][pos] = u;
    }
    unsigned long long ne = warpSum((unsigned long long)udeg);
    if (laneId() == 0 && ne) atomicAdd(&a.s->nextEdges, ne);
}

// Small bin: the warp expands its 32 short lists together: lane j takes edge
// j of the lists' concatenation; the owner lane is found by a shuffle binary
// search over the lanes' exclusive degree prefix.
__global__ void binnedSmallKernel(BinArgs a) {
    const uint32_t gid = blockIdx.x * blockDim.x + threadIdx.x;
    const unsigned lane = laneId();
    bool active = gid < a.size;
    uint32_t v = active ? a.queue[gid] : 0u;
    uint32_t begin = active ? a.row_ptr[v] : 0u;
    uint32_t deg = active ? a.row_ptr[v + 1] - begin : 0u;
    uint32_t incl = deg;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        uint32_t y = __shfl_up_sync(kFull, incl, o);
        if ((int)lane >= o) incl += y;
    }
    uint32_t pre = incl - deg, total = __shfl_sync(kFull, incl, 31);
    for (uint32_t base = 0; base < total; base += 32) {
        uint32_t j = base + lane;
        uint32_t owner = 0;
#pragma unroll
        for (uint32_t step = 16; step > 0; step >>= 1) {
            uint32_t cand = owner + step;
            if (__shfl_sync(kFull, pre, cand) <= j) owner = cand;
        }
        uint32_t ob = __shfl_sync(kFull, begin, owner), op = __shfl_sync(kFull, pre, owner);
        binVisit(a, j < total, ob + (j - op));
    }
}

// Medium bin: warp per vertex, lanes stride the list (coalesced col_idx).
__global__ void binnedMediumKernel(BinArgs a) {
    const uint32_t vi = (blockIdx.x * blockDim.x + threadIdx.x) / 32;
    if (vi >= a.size) return;  // uniform per warp
    uint32_t v = a.queue[vi], b = a.row_ptr[v], e = a.row_ptr[v + 1];
    for (uint32_t base = b; base < e; base += 32) binVisit(a, base + laneId() < e, base + laneId());
}

// Large bin: block per vertex.
__global__ void binnedLargeKernel(BinArgs a) {
    if (blockIdx.x >= a.size) return;
    uint32_t v = a.queue[blockIdx.x], b = a.row_ptr[v], e = a.row_ptr[v + 1];
    for (uint32_t base = b; base < e; base += blockDim.x) binVisit(a, base + threadIdx.x < e, base + threadIdx.x);
}

// ------------------------------------------------------------- gpu_edge

// One launch per level (gpu_edge, gpu_do).  A level of these forms is short (a
// few us on R-MAT 16), so what a call takes is what surrounds its kernels: with a
// counter memset, a three-part scan of the frontier's degrees, a counter copy, two
// events and a stream wait around each expansion a level cost 41 us (6 levels,
// 265 us a call).  Here
//  - an append reserves queue slots and edge offsets with one 64-bit atomic, so
//    the next level's offsets are scanned as they are written;
//  - the last block to finish stores the level's counters and its time into pinned
//    memory, where the host polls for them, and zeroes them for the next level;
//  - the first launch of a run does all the setting up.
// A level takes 18 us so, a call 126.

// Sums over a level, zero between levels.  `append` is (vertices << 32) | sum of
// their degrees: at most n vertices and m adjacency entries, both below 2^32.
struct EdgeStats {
    unsigned long long append, examined, t0;
    unsigned long long queued;  // queueFromBitmapKernel's append word
    unsigned ticket;
};
static_assert(sizeof(EdgeStats) <= sizeof(unsigned long long) * kEdgeStatWords, "room in the handle's buffer");

struct EdgeArgs {
    const uint32_t* row_ptr;
    const uint32_t* col_idx;
    uint32_t* dist;
    EdgeStats* s;
    unsigned long long* pub;  // pinned: append, examined, device time in ns, sequence number
    unsigned long long seq;
    uint32_t level;
    bool first;  // no launch of this level before this one
};

__device__ __forceinline__ void levelStart(const EdgeArgs& a) {
    if (a.first && blockIdx.x == 0 && threadIdx.x == 0) a.s->t0 = globaltimer();
}

// Ends a level: every block calls it after its own additions to *a.s.
__device__ __forceinline__ void levelEnd(const EdgeArgs& a) {
    __syncthreads();
    if (threadIdx.x != 0) return;
    __threadfence();
    if (atomicAdd(&a.s->ticket, 1u) != gridDim.x - 1) return;
    __threadfence();
    volatile EdgeStats* s = a.s;
    volatile unsigned long long* pub = a.pub;
    pub[0] = s->append;
    pub[1] = s->examined;
    pub[2] = globaltimer() - s->t0;
    s->append = s->examined = s->queued = 0;
    s->ticket = 0;
    __threadfence_system();
    pub[3] = a.seq;
}

// Depths to infinity, the source and its queue entry, the counters to zero.
__global__ void edgeInitKernel(EdgeArgs a, uint64_t n, uint32_t source, uint32_t* queue, uint32_t* offsets) {
    const uint64_t stride = (uint64_t)gridDim.x * blockDim.x, t = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
    uint4* d4 = reinterpret_cast<uint4*>(a.dist);  // its buffer is a multiple of 16 bytes
    for (uint64_t i = t; i < (n + 3) / 4; i += stride) {
        const uint64_t v = 4 * i;
        d4[i] = make_uint4(v == source ? 0u : kInf, v + 1 == source ? 0u : kInf, v + 2 == source ? 0u : kInf,
                           v + 3 == source ? 0u : kInf);
    }
    if (t == 0) {
        *a.s = EdgeStats{};
        a.s->t0 = globaltimer();
        queue[0] = source;
        offsets[0] = 0;
    }
}

constexpr uint32_t kStageCap = 2048;

// Edge-balanced expansion: block b owns edges [b*chunk, (b+1)*chunk) of the
// level (chunk = blockDim * ept); thread t takes edges t, t+blockDim, ... so a
// warp reads 32 consecutive edges per round.  Two warps find the chunk's owner
// range; the range's scanned offsets and adjacency starts are staged in shared
// memory so every per-edge owner search runs there.  R rounds go through each
// stage together (their loads and claims overlap, one append for all R).
template <int R>
__global__ void __launch_bounds__(1024) edgeExpandKernel(EdgeArgs a, const uint32_t* queue, const uint32_t* offsets,
                                                         uint32_t* nextQ, uint32_t* nextOff, uint32_t size,
                                                         uint32_t total, uint32_t ept) {
    __shared__ uint32_t sOff[kStageCap], sStart[kStageCap];
    __shared__ uint32_t sRange[2];
    levelStart(a);
    const uint64_t chunk = (uint64_t)blockDim.x * ept, c0 = blockIdx.x * chunk;
    const uint64_t c1 = min(c0 + chunk, (uint64_t)total);
    const unsigned warp = threadIdx.x >> 5, lane = laneId();
    for (unsigned k = warp; k < 2; k += blockDim.x >> 5) {
        const uint32_t o = warpOwnerOf(offsets, 0u, size - 1, (uint32_t)(k ? c1 - 1 : c0));
        if (lane == 0) sRange[k] = o;
    }
    __syncthreads();
    const uint32_t lo = sRange[0], hi = sRange[1], cnt = hi - lo + 1;
    const bool staged = cnt <= kStageCap;
    if (staged)
        for (uint32_t i = threadIdx.x; i < cnt; i += blockDim.x) {
            sOff[i] = offsets[lo + i];
            sStart[i] = a.row_ptr[queue[lo + i]];
        }
    __syncthreads();
    for (uint32_t k0 = 0; k0 < ept; k0 += R) {  // block-uniform rounds: appends stay convergent
        uint32_t u[R], st[R], en[R];
        bool has[R];
#pragma unroll
        for (int k = 0; k < R; ++k) {
            const uint64_t e = c0 + (uint64_t)(k0 + k) * blockDim.x + threadIdx.x;
            has[k] = k0 + k < ept && e < c1;
            u[k] = 0;
            if (!has[k]) continue;
            if (staged) {
                const uint32_t i = ownerOf(sOff, 0u, cnt - 1, (uint32_t)e);
                u[k] = a.col_idx[sStart[i] + ((uint32_t)e - sOff[i])];
            } else {
                const uint32_t i = ownerOf(offsets, lo, hi, (uint32_t)e);
                u[k] = a.col_idx[a.row_ptr[queue[i]] + ((uint32_t)e - offsets[i])];
            }
        }
#pragma unroll
        for (int k = 0; k < R; ++k) has[k] = has[k] && *reinterpret_cast<volatile uint32_t*>(&a.dist[u[k]]) == kInf;
#pragma unroll
        for (int k = 0; k < R; ++k) {
            st[k] = has[k] ? a.row_ptr[u[k]] : 0u;
            en[k] = has[k] ? a.row_ptr[u[k] + 1] : 0u;
            has[k] = has[k] && atomicCAS(&a.dist[u[k]], kInf, a.level + 1) == kInf;
        }
        unsigned long long mine = 0;
#pragma unroll
        for (int k = 0; k < R; ++k) mine += has[k] ? (1ull << 32) | (en[k] - st[k]) : 0ull;
        if (!__any_sync(kFull, mine != 0)) continue;
        unsigned long long incl = mine;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const unsigned long long y = __shfl_up_sync(kFull, incl, o);
            if (lane >= (unsigned)o) incl += y;
        }
        unsigned long long at = 0;
        if (lane == 31) at = atomicAdd(&a.s->append, incl);
        at = __shfl_sync(kFull, at, 31) + incl - mine;
#pragma unroll
        for (int k = 0; k < R; ++k) {
            if (!has[k]) continue;
            nextQ[at >> 32] = u[k];
            nextOff[at >> 32] = (uint32_t)at;
            at += (1ull << 32) | (en[k] - st[k]);
        }
    }
    levelEnd(a);
}

// A top-down level whose frontier has no edges.
__global__ void noEdgesKernel(EdgeArgs a) {
    levelStart(a);
    levelEnd(a);
}

// ------------------------------------------------------------- bottom-up

// Thread per vertex: an unreached vertex scans its list for the first parent
// in the frontier bitmap (early exit).  The 32 lanes of a warp are one bitmap
// word of the next frontier, assembled with __ballot_sync and stored by lane
// 0, so every word of `next` is written and needs no clearing.  One addition
// per block and counter: per warp, an R-MAT 22 level's 113,000 additions to one
// line take 80 us by themselves.
__global__ void __launch_bounds__(1024) bottomUpKernel(EdgeArgs a, const uint32_t* front, uint32_t* next, uint64_t n) {
    __shared__ unsigned long long sum[2];
    levelStart(a);
    if (threadIdx.x < 2) sum[threadIdx.x] = 0;
    __syncthreads();
    const uint64_t stride = (uint64_t)gridDim.x * blockDim.x;
    unsigned long long append = 0, examined = 0;
    for (uint64_t base = (uint64_t)blockIdx.x * blockDim.x; base < n; base += stride) {
        const uint64_t v = base + threadIdx.x;
        bool found = false;
        if (v < n && a.dist[v] == kInf) {
            const uint32_t b = a.row_ptr[v], e = a.row_ptr[v + 1];
            if (b < e) {
                examined += buScanFrom(a.col_idx, front, b, e, found) - b;
                if (found) {
                    a.dist[v] = a.level + 1;
                    append += (1ull << 32) | (e - b);
                }
            }
        }
        const unsigned word = __ballot_sync(kFull, found);
        if (laneId() == 0 && v < n) next[v >> 5] = word;
    }
    append = warpSum(append);
    examined = warpSum(examined);
    if (laneId() == 0) {
        if (append) atomicAdd(&sum[0], append);
        if (examined) atomicAdd(&sum[1], examined);
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        if (sum[0]) atomicAdd(&a.s->append, sum[0]);
        if (sum[1]) atomicAdd(&a.s->examined, sum[1]);
    }
    levelEnd(a);
}

// The frontier's bitmap from the depths (the first bottom-up level).
__global__ void frontBitmapKernel(EdgeArgs a, uint32_t* front, uint64_t n) {
    levelStart(a);
    for (uint64_t base = (uint64_t)blockIdx.x * blockDim.x; base < n; base += (uint64_t)gridDim.x * blockDim.x) {
        const uint64_t v = base + threadIdx.x;
        const unsigned word = __ballot_sync(kFull, v < n && a.dist[v] == a.level);
        if (laneId() == 0 && v < n) front[v >> 5] = word;
    }
}

// The frontier's queue and edge offsets from its bitmap (the first top-down
// level after bottom-up ones): one append per block and 256 vertices.
constexpr int kQueueThreads = 256;

__global__ void queueFromBitmapKernel(EdgeArgs a, const uint32_t* front, uint64_t n, uint32_t* queue,
                                      uint32_t* offsets) {
    __shared__ unsigned long long scan[kQueueThreads / 32 + 1], at0;
    levelStart(a);
    for (uint64_t base = (uint64_t)blockIdx.x * kQueueThreads; base < n; base += (uint64_t)gridDim.x * kQueueThreads) {
        const uint64_t v = base + threadIdx.x;
        const bool in = v < n && ((front[v >> 5] >> (v & 31)) & 1u);
        const unsigned long long mine = in ? (1ull << 32) | (a.row_ptr[v + 1] - a.row_ptr[v]) : 0ull;
        unsigned long long total;
        unsigned long long at = blockScan<kQueueThreads>(mine, &total, scan);
        if (total == 0) continue;  // block-uniform
        if (threadIdx.x == 0) at0 = atomicAdd(&a.s->queued, total);
        __syncthreads();
        at += at0;
        if (in) {
            queue[at >> 32] = (uint32_t)v;
            offsets[at >> 32] = (uint32_t)at;
        }
        __syncthreads();  // at0 is the next round's
    }
}

uint32_t gridCap(uint64_t work, uint32_t threads) {
    uint64_t b = (work + threads - 1) / threads;
    uint64_t cap = (uint64_t)deviceSmCount() * (2048 / threads) * 4;
    return (uint32_t)std::max<uint64_t>(1, std::min(b, cap));
}

double msSince(std::chrono::steady_clock::time_point t0) {
    return std::chrono::duration<double, std::milli>(std::chrono::steady_clock::now() - t0).count();
}

}  // namespace
}  // namespace gb

using namespace gb;

void gb_bfs::initDist(uint32_t src) {
    initDistKernel<<<gridCap(n / 4 + 1, 256), 256, 0, stream.s>>>(dist.get(), n, src);
    setSourceKernel<<<1, 1, 0, stream.s>>>(dist.get(), src);
    GB_LAUNCH_CHECK();
}

void gb_bfs::beginLevel() {
    GB_CUDA(cudaMemsetAsync(stats.get(), 0, sizeof(GbLevelStats), stream.s));
}

void gb_bfs::endLevel() {
    GB_CUDA(cudaMemcpyAsync(hstats.p, stats.get(), sizeof(GbLevelStats), cudaMemcpyDeviceToHost, stream.s));
    GB_CUDA(cudaEventRecord(ev.b, stream.s));
    GB_CUDA(cudaStreamSynchronize(stream.s));
    lastGpuMs += ev.ms();
    ++lastLevels;
}

void gb_bfs::ensureEdgeBuffers() {
    qA.ensure(n);
    qB.ensure(n);
    offA.ensure(n);
    offB.ensure(n);
    edgeStats.ensure(kEdgeStatWords);
    edgePub.ensure(4);
}

void gb_bfs::runVertex(uint32_t src, const gb_bfs_options& o, std::vector<gb_level>* tr) {
    const uint32_t tg = checkTg(o.tg);
    lastGpuMs = 0;
    lastLevels = 0;
    for (uint32_t level = 0;; ++level) {
        auto t0 = std::chrono::steady_clock::now();
        GB_CUDA(cudaEventRecord(ev.a, stream.s));
        beginLevel();
        if (level == 0) initDist(src);
        vertexLevelKernel<<<gridCap(n, tg), tg, 0, stream.s>>>(rowPtr.get(), colIdx.get(), dist.get(), n, level,
                                                               stats.get());
        GB_LAUNCH_CHECK();
        endLevel();
        const GbLevelStats& s = *hstats.p;
        if (tr) tr->push_back({level, 'T', 'G', 0, 0, s.frontier, s.edges, msSince(t0)});
        if (s.found == 0) break;
    }
}

void gb_bfs::runNaive(uint32_t src, const gb_bfs_options& o, std::vector<gb_level>* tr) {
    const uint32_t tg = checkTg(o.tg);
    qA.ensure(n);
    qB.ensure(n);
    uint32_t *cur = qA.get(), *next = qB.get();
    hstage.p[0] = src;
    GB_CUDA(cudaMemcpyAsync(cur, hstage.p, 4, cudaMemcpyHostToDevice, stream.s));
    uint32_t size = 1;
    lastGpuMs = 0;
    lastLevels = 0;
    for (uint32_t level = 0; size > 0; ++level) {
        auto t0 = std::chrono::steady_clock::now();
        GB_CUDA(cudaEventRecord(ev.a, stream.s));
        beginLevel();
        if (level == 0) initDist(src);
        naiveLevelKernel<<<divUp(size, tg), tg, 0, stream.s>>>(rowPtr.get(), colIdx.get(), dist.get(), stats.get(),
                                                               cur, next, size, level);
        GB_LAUNCH_CHECK();
        endLevel();
        const GbLevelStats& s = *hstats.p;
        if (tr) tr->push_back({level, 'T', 'G', 0, 0, s.frontier, s.edges, msSince(t0)});
        size = s.found;
        std::swap(cur, next);
    }
}

void gb_bfs::runBinned(uint32_t src, const gb_bfs_options& o, std::vector<gb_level>* tr) {
    const uint32_t tg = checkTg(o.tg);
    for (auto& set : bins)
        for (auto& q : set) q.ensure(n);
    auto bin = [&](uint32_t d) { return d < o.small_max ? 0 : (d < o.large_min ? 1 : 2); };
    uint32_t count[3] = {0, 0, 0};
    const uint32_t srcDeg = degree(src);
    hstage.p[0] = src;
    GB_CUDA(cudaMemcpyAsync(bins[0][bin(srcDeg)].get(), hstage.p, 4, cudaMemcpyHostToDevice, stream.s));
    count[bin(srcDeg)] = 1;
    uint64_t edges = srcDeg;
    int cur = 0;
    lastGpuMs = 0;
    lastLevels = 0;
    for (uint32_t level = 0; count[0] + count[1] + count[2] > 0; ++level) {
        auto t0 = std::chrono::steady_clock::now();
        GB_CUDA(cudaEventRecord(ev.a, stream.s));
        beginLevel();
        if (level == 0) initDist(src);
        BinArgs a{rowPtr.get(), colIdx.get(), dist.get(), stats.get(), nullptr,
                  {bins[cur ^ 1][0].get(), bins[cur ^ 1][1].get(), bins[cur ^ 1][2].get()},
                  0, level, o.small_max, o.large_min};
        for (int b = 0; b < 3; ++b) {
            if (count[b] == 0) continue;
            a.size = count[b];
            a.queue = bins[cur][b].get();
            if (b == 0) binnedSmallKernel<<<divUp(count[b], tg), tg, 0, stream.s>>>(a);
            else if (b == 1) binnedMediumKernel<<<divUp((uint64_t)count[b] * 32, tg), tg, 0, stream.s>>>(a);
            else binnedLargeKernel<<<count[b], tg, 0, stream.s>>>(a);
            GB_LAUNCH_CHECK();
        }
        endLevel();
        const GbLevelStats& s = *hstats.p;
        if (tr) tr->push_back({level, 'T', 'G', 0, 0, (uint64_t)count[0] + count[1] + count[2], edges, msSince(t0)});
        for (int b = 0; b < 3; ++b) count[b] = s.bin[b];
        edges = s.nextEdges;
        cur ^= 1;
    }
}

namespace {
// The levels of a gpu_edge or gpu_do run on the handle's stream.
struct EdgeRun {
    gb_bfs& h;
    const uint32_t tg, ept;
    EdgeArgs a{};
    uint32_t *q, *off, *qNext, *offNext;
    uint64_t size = 1, total;  // frontier: vertices, sum of their degrees
    uint64_t examined = 0;     // by the last level, if bottom-up

    EdgeRun(gb_bfs& h_, uint32_t src, const gb_bfs_options& o) : h(h_), tg(checkTg(o.tg)), ept(o.ept), total(h_.degree(src)) {
        if (ept == 0) throw Error(GB_ERR_ARG, "ept must be >= 1");
        h.ensureEdgeBuffers();
        q = h.qA.get(), qNext = h.qB.get(), off = h.offA.get(), offNext = h.offB.get();
        a.row_ptr = h.rowPtr.get();
        a.col_idx = h.colIdx.get();
        a.dist = h.dist.get();
        a.s = reinterpret_cast<EdgeStats*>(h.edgeStats.get());
        a.pub = h.edgePub.p;
        h.edgePub.p[3] = 0;  // no level's number
        h.lastGpuMs = 0;
        h.lastLevels = 0;
        edgeInitKernel<<<gridCap(h.n / 4 + 1, 256), 256, 0, h.stream.s>>>(a, h.n, src, q, off);
        GB_LAUNCH_CHECK();
    }

    void begin(uint32_t level) {
        a.level = level;
        a.first = level > 0;  // the first level's time begins with the setting up
        a.seq = ++h.edgeSeq;
    }
    void topDown() {
        if (total == 0) {
            noEdgesKernel<<<1, 32, 0, h.stream.s>>>(a);
            GB_LAUNCH_CHECK();
            return;
        }
        const uint32_t grid = divUp(total, (uint64_t)tg * ept);
        if (ept <= 2)
            edgeExpandKernel<2><<<grid, tg, 0, h.stream.s>>>(a, q, off, qNext, offNext, (uint32_t)size, (uint32_t)total, ept);
        else
            edgeExpandKernel<4><<<grid, tg, 0, h.stream.s>>>(a, q, off, qNext, offNext, (uint32_t)size, (uint32_t)total, ept);
        GB_LAUNCH_CHECK();
    }
    // Waits for the level's counters; the frontier is then the next one.
    void end() {
        ++h.lastLevels;
        const volatile unsigned long long* pub = h.edgePub.p;
        for (uint64_t spins = 1; pub[3] != a.seq; ++spins) {
            cpuPause();
            if (spins & 1023) continue;
            const cudaError_t e = cudaStreamQuery(h.stream.s);
            if (e == cudaErrorNotReady) continue;
            GB_CUDA(e);
            if (pub[3] != a.seq) throw Error(GB_ERR_CUDA, "a level ended without its counters");
        }
        std::atomic_thread_fence(std::memory_order_acquire);
        size = pub[0] >> 32;
        total = (uint32_t)pub[0];
        examined = pub[1];
        h.lastGpuMs += pub[2] * 1e-6;
    }
    void swapQueues() {
        std::swap(q, qNext);
        std::swap(off, offNext);
    }
};
}  // namespace

void gb_bfs::runEdge(uint32_t src, const gb_bfs_options& o, std::vector<gb_level>* tr, bool wait) {
    EdgeRun r(*this, src, o);
    for (uint32_t level = 0; r.size > 0; ++level) {
        auto t0 = std::chrono::steady_clock::now();
        const uint64_t size = r.size, total = r.total;
        r.begin(level);
        r.topDown();
        r.end();
        if (tr) tr->push_back({level, 'T', 'G', 0, 0, size, total, msSince(t0)});
        r.swapQueues();
    }
    if (wait) GB_CUDA(cudaStreamSynchronize(stream.s));
}

// gpu_do: the alpha/beta rule of cpu::bfsDO / GpuBfs::runDirOpt
// (src/cpu/bfs_cpu.cpp:227-283, src/metal/bfs_gpu.mm:326-429), decided on the
// host from the counters each level leaves.
void gb_bfs::runDirOpt(uint32_t src, const gb_bfs_options& o, std::vector<gb_level>* tr, bool wait) {
    const uint64_t words = (n + 31) / 32;
    bmFront.ensure(words);
    bmNext.ensure(words);
    EdgeRun r(*this, src, o);
    uint32_t *front = bmFront.get(), *next = bmNext.get();
    uint64_t scout = r.total, toCheck = m;
    bool bottomUp = false, toBitmap = false, toQueue = false;
    for (uint32_t level = 0; r.size > 0; ++level) {
        auto t0 = std::chrono::steady_clock::now();
        if (!bottomUp && (double)scout > (double)toCheck / o.alpha) {
            bottomUp = true;
            toBitmap = true;
        }
        if (!bottomUp) toCheck -= std::min(toCheck, scout);
        const uint64_t size = r.size, total = r.total;
        r.begin(level);
        if (bottomUp) {
            if (toBitmap) {
                frontBitmapKernel<<<gridCap(n, 256), 256, 0, stream.s>>>(r.a, front, n);
                GB_LAUNCH_CHECK();
                r.a.first = false;
            }
            bottomUpKernel<<<gridCap(n, r.tg), r.tg, 0, stream.s>>>(r.a, front, next, n);
            GB_LAUNCH_CHECK();
        } else {
            if (toQueue && total > 0) {
                queueFromBitmapKernel<<<gridCap(n, kQueueThreads), kQueueThreads, 0, stream.s>>>(r.a, front, n, r.q, r.off);
                GB_LAUNCH_CHECK();
                r.a.first = false;
            }
            r.topDown();
        }
        r.end();
        toBitmap = toQueue = false;
        if (tr)
            tr->push_back({level, bottomUp ? 'B' : 'T', 'G', (uint8_t)(bottomUp ? GB_STRAT_BU : GB_STRAT_TD_EPT2), 0,
                           size, bottomUp ? r.examined : total, msSince(t0)});
        if (bottomUp) {
            std::swap(front, next);
            if (!(r.size >= size || (double)r.size > (double)n / o.beta)) {
                bottomUp = false;
                toQueue = true;
                scout = 1;
            }
        } else {
            scout = r.total;
            r.swapQueues();
        }
    }
    if (wait) GB_CUDA(cudaStreamSynchronize(stream.s));
}
