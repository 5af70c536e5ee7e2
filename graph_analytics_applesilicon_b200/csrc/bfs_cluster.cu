// bfs_cluster.cu -- BFS of bounded-degree graphs (road networks): a
// thread-block cluster runs one source's levels, several sources side by side.
//
// A road network's traversal is 1,000-3,000 levels of about a thousand
// vertices each, nothing but latency.  On the whole grid such a level costs
// 6.4 us: the grid barrier, the level's counters, the queue tail's atomic, the
// queue itself, the adjacency bounds and the claim are each a round trip to L2
// (350-800 cycles, the far half of L2 being the slow one).  Here they stay on
// the SMs:
//   - the frontier queue is in shared memory, a part per block, and an entry is
//     the vertex's neighbours themselves, copied from a 4-slot neighbour table
//     by cp.async when the vertex is claimed, so the copy runs behind the end
//     of the level;
//   - the visited bitmap is spread over the cluster's shared memory and claimed
//     by distributed-shared-memory atomics (300-700 cycles against 750-1100);
//   - a level ends with every block sending its count to the others by
//     st.async onto their mbarriers: no fence and no cluster barrier, whose
//     release waits for all the block's global writes (1,500-2,500 cycles).
// Measured, road 1400 x 1400 (1,854 levels, 1,060 vertices each on average),
// device time: one source 12.6 -> 3.7 ms (2.0 us per level), 64 sources of one
// call 107 (batched kernel) -> 7.7 ms.
#include <cooperative_groups.h>

#include <algorithm>
#include <cstring>
#include <vector>

#include "bfs.hpp"
#include "cluster_leave.hpp"
#include "cluster_shape.hpp"

namespace cg = cooperative_groups;

namespace gb {
namespace {

// 512 threads: 256 make more passes of a level (1400 x 1400: 3.85 against 3.71
// ms), 1024 cost more per barrier (4.37 ms).
constexpr int kClThreads = 512;
constexpr uint32_t kClLanes = 4;     // lanes per queue entry, a neighbour slot each
// A vertex of more than 4 neighbours keeps 3 in its slots; the fourth slot then
// holds kClMore | (neighbours left) << kClPosBits | position of the fourth in
// col_idx, which bounds the degree (31) and m (2^26).
constexpr uint32_t kClMore = 0x80000000u, kClPosBits = 26, kClMaxDegree = 31;
// A wait gives up after this time and then this many polls: the timer runs on
// while the process is preempted, the polls do not.
constexpr unsigned long long kClWaitNs = 2000000000ull;
constexpr uint32_t kClWaitPolls = 1u << 14;
constexpr unsigned long long kClSettleNs = 20000ull;  // a count takes under a microsecond to arrive

struct ClArgs {
    const uint4* __restrict__ nbr;  // neighbour table
    const uint32_t* __restrict__ col_idx;
    uint32_t* dist;  // source i's depths at dist + i * n, all infinity before the launch
    const uint32_t* sources;
    GbClusterStat* stat;
    uint64_t n;
    uint32_t words;  // bitmap words per block
};

__device__ __forceinline__ uint32_t smemAddr(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }

// The address of `local`, an address in this block's shared memory, in block `rank` of the cluster.
__device__ __forceinline__ uint32_t mapaAddr(uint32_t local, uint32_t rank) {
    uint32_t r;
    asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(local), "r"(rank));
    return r;
}
__device__ __forceinline__ uint32_t ldShared(uint32_t addr) {
    uint32_t v;
    asm volatile("ld.shared.u32 %0, [%1];" : "=r"(v) : "r"(addr) : "memory");
    return v;
}
__device__ __forceinline__ uint32_t ldCluster(uint32_t addr) {
    uint32_t v;
    asm volatile("ld.shared::cluster.u32 %0, [%1];" : "=r"(v) : "r"(addr) : "memory");
    return v;
}

// Sets u's bit in the cluster's bitmap (word w is in block w % NC at w / NC);
// true when it was clear.
template <uint32_t NC>
__device__ __forceinline__ bool claim(uint32_t bmAddr, uint32_t u) {
    const uint32_t w = u >> 5;
    uint32_t old;
    asm volatile("atom.relaxed.cluster.shared::cluster.or.b32 %0, [%1], %2;"
                 : "=r"(old)
                 : "r"(mapaAddr(bmAddr + (w / NC) * 4, w % NC)), "r"(1u << (u & 31))
                 : "memory");
    return !((old >> (u & 31)) & 1u);
}

// The cluster as one block sees it when blocks give up (cluster_leave.hpp):
// `flag` is a word of this block's shared memory, 0 until a block gives up.
template <uint32_t NC>
struct ClusterEnd {
    cg::cluster_group& cl;
    uint32_t flag;
    __device__ void sync() { cl.sync(); }
    __device__ void raise() {
        if (threadIdx.x < NC)
            asm volatile("st.relaxed.cluster.shared::cluster.u32 [%0], %1;" ::"r"(mapaAddr(flag, threadIdx.x)), "r"(1u)
                         : "memory");
    }
    __device__ bool raised() { return __syncthreads_or(ldShared(flag) != 0); }
    __device__ void settle() {
        for (const uint64_t t = globaltimer(); globaltimer() - t < kClSettleNs;) __nanosleep(1000);
    }
};

// Level L reads the queue parts of parity L & 1 and appends to the others, a
// block always to its own part.  Block r's count for level L is cnt[L % 3]
// (the count level L + 2 will fill is zeroed during level L) and reaches block
// b's slot[L & 1][r] with 8 bytes on b's mbar[L & 1]; a block goes on once all
// NC counts are there, so it also never runs more than a level ahead of
// another, which is what makes two parities enough.  A block expands its own
// part.  When the parts have drifted apart the level reads all parts as one
// list instead, entry i of the concatenation going to lane group i; only then
// is a cluster barrier needed, for the other blocks' queue entries.  Entries
// beyond a part's room are dropped but counted: every block sees that count,
// all leave together, and the caller runs the sources another way.  A block
// whose wait runs out takes all others with it (cluster_leave.hpp).
template <uint32_t NC>
__global__ void __launch_bounds__(kClThreads, 2) clusterBfsKernel(ClArgs a) {
    extern __shared__ __align__(16) uint4 clMem[];  // [2][kClQueue] entries, then the bitmap
    __shared__ uint32_t cnt[3], gaveUp;
    __shared__ __align__(8) unsigned long long slot[2][NC], mbar[2];
    cg::cluster_group cl = cg::this_cluster();
    const uint32_t rank = cl.block_rank(), s = blockIdx.x / NC;
    const unsigned tid = threadIdx.x, lane = laneId();
    uint32_t* dist = a.dist + (uint64_t)s * a.n;
    uint32_t* bitmap = reinterpret_cast<uint32_t*>(clMem + 2 * kClQueue);
    const uint32_t bmAddr = smemAddr(bitmap), qAddr = smemAddr(clMem), slotAddr = smemAddr(slot), flagAddr = smemAddr(&gaveUp);
    ClusterEnd<NC> end{cl, flagAddr};
    const uint64_t t0 = globaltimer();
    for (uint32_t i = tid; i < a.words; i += kClThreads) bitmap[i] = 0;
    if (tid < 3) cnt[tid] = 0;
    if (tid == 0) gaveUp = 0;
    if (tid < 2) asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(smemAddr(&mbar[tid])) : "memory");
    if (tid < NC) slot[0][tid] = tid == 0;  // level 0: the source, in block 0's part
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    cl.sync();
    if (rank == 0 && tid == 0) {
        const uint32_t v = a.sources[s];
        clMem[0] = a.nbr[v];
        dist[v] = 0;
        claim<NC>(bmAddr, v);
    }
    __syncthreads();
    const uint32_t sub = lane % kClLanes, grp = tid / kClLanes, first = (tid - lane) / kClLanes;
    constexpr uint32_t kGroups = kClThreads / kClLanes;
    uint32_t level = 0, c0 = 0, status = 0, spreadAt = 0;  // c0 = level % 3
    for (;; ++level) {
        const uint32_t c1 = c0 == 2 ? 0 : c0 + 1, c2 = c1 == 2 ? 0 : c1 + 1, par = level & 1;
        const uint32_t mine = lane < NC ? ldShared(slotAddr + (par * NC + lane) * 8) : 0u;
        const uint32_t total = __reduce_add_sync(kFull, mine), most = __reduce_max_sync(kFull, mine);
        if (total == 0) break;
        if (most > kClQueue) {
            status = kClusterOverflow;
            break;
        }
        if (tid == 0) cnt[c2] = 0;
        const uint32_t cntAddr = smemAddr(&cnt[c1]);
        const uint32_t qc = qAddr + par * (kClQueue * 16), qn = qAddr + (par ^ 1) * (kClQueue * 16);
        // claims u (kInf: none) in every lane of the warp; winners store their
        // depth and start the copy of their neighbours into the next queue
        auto visit = [&](uint32_t u) {
            const bool won = u != kInf && claim<NC>(bmAddr, u);
            const unsigned b = __ballot_sync(kFull, won);
            if (!b) return;
            uint32_t p = 0;
            if (lane == 0)
                asm volatile("atom.shared::cta.add.u32 %0, [%1], %2;" : "=r"(p) : "r"(cntAddr), "r"(__popc(b)) : "memory");
            p = __shfl_sync(kFull, p, 0) + __popc(b & lanemaskLt());
            if (won) {
                if (p < kClQueue)
                    asm volatile("cp.async.ca.shared.global [%0], [%1], 16;" ::"r"(qn + p * 16), "l"(a.nbr + u) : "memory");
                dist[u] = level + 1;
            }
        };
        auto expand = [&](uint32_t x) {  // x: slot `sub` of the lane group's entry (kInf: none)
            const bool more = (x & kClMore) && x != kInf;
            uint32_t e = x & ((1u << kClPosBits) - 1), left = more ? (x >> kClPosBits) & 31u : 0u;
            visit(more ? a.col_idx[e] : x);
            while (__any_sync(kFull, left > 1)) {  // the rest of a longer list, in the lane of slot 3
                ++e;
                visit(left > 1 ? a.col_idx[e] : kInf);
                if (left) --left;
            }
        };
        // Reading the parts as one list costs about 2,000 cycles (the barrier
        // and the remote reads) and evens out the 16 levels that follow it;
        // below 32 entries over the mean a block's level is one pass anyway.
        const uint32_t over = most - total / NC;
        if (NC > 1 && (over > 256 || (over > 32 && level - spreadAt >= 16))) {
            spreadAt = level;
            if (!clusterMeet(end)) break;  // block-uniform
            uint32_t x = mine;
#pragma unroll
            for (int o = 1; o < (int)NC; o <<= 1) {
                const uint32_t y = __shfl_up_sync(kFull, x, o);
                if ((int)lane >= o) x += y;
            }
            const uint32_t pre = x - mine;
            for (uint32_t i0 = rank * kGroups; i0 + first < total; i0 += kGroups * NC) {  // warp-uniform
                const uint32_t i = i0 + grp;
                uint32_t j = 0, p = 0;
#pragma unroll
                for (uint32_t b = 1; b < NC; ++b) {
                    const uint32_t pb = __shfl_sync(kFull, pre, b);
                    if (i >= pb) {
                        j = b;
                        p = pb;
                    }
                }
                expand(i < total ? ldCluster(mapaAddr(qc + (i - p) * 16 + sub * 4, j)) : kInf);
            }
        } else {
            const uint32_t own = __shfl_sync(kFull, mine, rank);
            for (uint32_t i0 = 0; i0 + first < own; i0 += kGroups)
                expand(i0 + grp < own ? ldShared(qc + (i0 + grp) * 16 + sub * 4) : kInf);
        }
        __syncthreads();  // the block's appends are counted
        const uint32_t mb = smemAddr(&mbar[par ^ 1]);
        if (tid < 32) {
            const unsigned long long c = cnt[c1];
            if (lane == 0)
                asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(mb), "r"(NC * 8u) : "memory");
            if (lane < NC)
                asm volatile("st.async.weak.shared::cluster.mbarrier::complete_tx::bytes.b64 [%0], %1, [%2];" ::"r"(
                                 mapaAddr(smemAddr(&slot[par ^ 1][rank]), lane)),
                             "l"(c), "r"(mapaAddr(mb, lane))
                             : "memory");
        }
        uint32_t done = 0, polls = 0;
        for (uint64_t tw = 0; !done;) {  // bounded
            asm volatile(
                "{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\tselp.u32 %0, 1, 0, p;\n\t}"
                : "=r"(done)
                : "r"(mb), "r"((level >> 1) & 1u)
                : "memory");
            if (done) break;
            const uint64_t t = globaltimer();
            if (!tw) tw = t;
            if ((t - tw > kClWaitNs && ++polls > kClWaitPolls) || ldShared(flagAddr)) break;
        }
        asm volatile("cp.async.wait_all;" ::: "memory");
        if (__syncthreads_or(!done)) {  // also: every thread's copies into the queue have landed
            status = kClusterTimeout;
            break;
        }
        c0 = c1;
    }
    // no block leaves while another may still send to it or read its queue
    if (clusterLeave(end, status == kClusterTimeout)) status = kClusterTimeout;
    if (rank == 0 && tid == 0) a.stat[s] = {level, status, (unsigned long long)(globaltimer() - t0)};
}

// The neighbour table: a vertex's first 4 neighbours (kInf beyond its degree).
__global__ void nbrTableKernel(const uint32_t* __restrict__ row_ptr, const uint32_t* __restrict__ col_idx, uint64_t n,
                               uint4* nbr) {
    for (uint64_t v = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; v < n; v += (uint64_t)gridDim.x * blockDim.x) {
        const uint32_t st = row_ptr[v], d = row_ptr[v + 1] - st;
        uint4 x;
        x.x = d > 0 ? col_idx[st] : kInf;
        x.y = d > 1 ? col_idx[st + 1] : kInf;
        x.z = d > 2 ? col_idx[st + 2] : kInf;
        x.w = d > 4 ? kClMore | (d - 3) << kClPosBits | (st + 3) : d > 3 ? col_idx[st + 3] : kInf;
        nbr[v] = x;
    }
}

template <uint32_t NC>
cudaLaunchConfig_t clusterConfig(uint64_t n, uint32_t k, cudaStream_t st, cudaLaunchAttribute* attr) {
    attr->id = cudaLaunchAttributeClusterDimension;
    attr->val.clusterDim.x = NC;
    attr->val.clusterDim.y = attr->val.clusterDim.z = 1;
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3(k * NC);
    cfg.blockDim = dim3(kClThreads);
    cfg.dynamicSmemBytes = clusterSmem(n, NC);
    cfg.stream = st;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    return cfg;
}

template <uint32_t NC>
void allowCluster() {
    GB_CUDA(cudaFuncSetAttribute(clusterBfsKernel<NC>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kClSmem));
    if (NC > 8) GB_CUDA(cudaFuncSetAttribute(clusterBfsKernel<NC>, cudaFuncAttributeNonPortableClusterSizeAllowed, 1));
}

template <uint32_t NC>
void launchCluster(const ClArgs& a, uint32_t k, cudaStream_t st) {
    allowCluster<NC>();
    cudaLaunchAttribute attr{};
    cudaLaunchConfig_t cfg = clusterConfig<NC>(a.n, k, st, &attr);
    GB_CUDA(cudaLaunchKernelEx(&cfg, clusterBfsKernel<NC>, a));
}

// Whether the device can run a cluster of NC blocks of this graph.
template <uint32_t NC>
bool clusterRuns(uint64_t n) {
    allowCluster<NC>();
    cudaLaunchAttribute attr{};
    cudaLaunchConfig_t cfg = clusterConfig<NC>(n, 1, nullptr, &attr);
    int clusters = 0;
    if (cudaOccupancyMaxActiveClusters(&clusters, clusterBfsKernel<NC>, &cfg) == cudaSuccess) return clusters > 0;
    cudaGetLastError();  // a size the device does not know
    return false;
}

bool clusterRuns(uint64_t n, uint32_t nc) {
    switch (nc) {
        case 1: return clusterRuns<1>(n);
        case 2: return clusterRuns<2>(n);
        case 4: return clusterRuns<4>(n);
        case 8: return clusterRuns<8>(n);
        default: return clusterRuns<16>(n);
    }
}

}  // namespace
}  // namespace gb

using namespace gb;

// Whether k sources may run a cluster each.  The line is the shape of road
// networks and grids, whose frontiers stay narrow: at most 31 neighbours and
// 8 on average.  A graph of that shape whose frontier outgrows the queues
// after all (a random 3-regular graph) is noticed in its first levels and
// marked, so later calls on the handle do not try again.  A caller's spin limit
// under kSoloSpin asks for waits shorter than this form's: the grid forms have them.
bool gb_bfs::clusterFits(uint32_t k, const gb_bfs_options& o) {
    return !cOff && (o.spin_limit == 0 || o.spin_limit >= kSoloSpin) && o.force_strategy < 0 && o.grid_blocks == 0 && maxDegree <= kClMaxDegree && m <= 8 * n &&
           m < (1ull << kClPosBits) && n < kClMore && clusterBlocks(k) != 0;
}

// clusterSize for this handle, which asks the device about a size once.
uint32_t gb_bfs::clusterBlocks(uint32_t k) {
    return clusterSize(n, k, (uint32_t)deviceSmCount(), [&](uint32_t nc) {
        signed char& known = cRuns[31 - __builtin_clz(nc)];
        if (known < 0) known = clusterRuns(n, nc);
        return known != 0;
    });
}

// Runs k sources' traversals into out (source i's depths at out + i * n) and
// their level counts and times into cStatHost; false when a frontier outgrew
// the queues or there is no memory for the neighbour table (out is then not valid).
bool gb_bfs::runCluster(const uint32_t* src, uint32_t k, uint32_t* out) {
    if (!cNbrReady) {
        if (!cNbr.tryEnsure(n)) return false;
        nbrTableKernel<<<(uint32_t)std::min<uint64_t>((n + 255) / 256, (uint64_t)deviceSmCount() * 8), 256, 0,
                         stream.s>>>(rowPtr.get(), colIdx.get(), n, cNbr.get());
        GB_LAUNCH_CHECK();
        cNbrReady = true;
    }
    cSrc.ensure(64);
    cStat.ensure(64);
    cStatHost.ensure(64);
    hstage.ensure(64);
    std::memcpy(hstage.p, src, k * 4);
    GB_CUDA(cudaMemcpyAsync(cSrc.get(), hstage.p, k * 4, cudaMemcpyHostToDevice, stream.s));
    const uint32_t nc = clusterBlocks(k);
    const ClArgs a{cNbr.get(), colIdx.get(), out, cSrc.get(), cStat.get(), n, (uint32_t)(((n + 31) / 32 + nc - 1) / nc)};
    GB_CUDA(cudaEventRecord(ev.a, stream.s));
    GB_CUDA(cudaMemsetAsync(out, 0xFF, (uint64_t)k * n * 4, stream.s));  // every depth infinity
    switch (nc) {
        case 1: launchCluster<1>(a, k, stream.s); break;
        case 2: launchCluster<2>(a, k, stream.s); break;
        case 4: launchCluster<4>(a, k, stream.s); break;
        case 8: launchCluster<8>(a, k, stream.s); break;
        default: launchCluster<16>(a, k, stream.s); break;
    }
    GB_CUDA(cudaEventRecord(ev.b, stream.s));
    GB_CUDA(cudaMemcpyAsync(cStatHost.p, cStat.get(), k * sizeof(GbClusterStat), cudaMemcpyDeviceToHost, stream.s));
    GB_CUDA(cudaStreamSynchronize(stream.s));
    uint32_t levels = 0;
    for (uint32_t i = 0; i < k; ++i) {
        if (cStatHost.p[i].status == kClusterTimeout)
            throw Error(GB_ERR_TIMEOUT, "cluster BFS: a wait for the other blocks' counts exceeded its limit");
        if (cStatHost.p[i].status) cOff = true;
        levels = std::max(levels, cStatHost.p[i].levels);
    }
    if (cOff) {  // for the handle's life
        cNbr.release();
        return false;
    }
    lastGpuMs = ev.ms();
    lastLevels = levels;
    return true;
}

// gb_bfs_run_many with the learned selector: up to 64 sources to a launch,
// each with its own device time and level count; false (nothing valid) when a
// frontier outgrew the queues or there is no memory for this form.
bool gb_bfs::runClusterMany(const uint32_t* src, uint32_t count, uint32_t* out, uint64_t stride, float* msOut,
                            uint32_t* levelsOut) {
    if (!bDist.tryEnsure((uint64_t)std::min<uint32_t>(count, 64) * n + 4)) return false;
    for (uint32_t g0 = 0; g0 < count; g0 += 64) {
        const uint32_t k = std::min<uint32_t>(64, count - g0);
        if (!runCluster(src + g0, k, bDist.get())) {
            bDist.release();  // the grid form rotates in_flight + 2 rows; a batch takes its own again
            return false;
        }
        for (uint32_t j = 0; j < k; ++j) {
            if (msOut) msOut[g0 + j] = (float)((double)cStatHost.p[j].ns * 1e-6);
            if (levelsOut) levelsOut[g0 + j] = cStatHost.p[j].levels;
        }
        if (g0 + k == count) {
            GB_CUDA(cudaMemcpyAsync(dist.get(), bDist.get() + (uint64_t)(k - 1) * n, n * 4, cudaMemcpyDeviceToDevice,
                                    stream.s));
            lastGpuMs = (double)cStatHost.p[k - 1].ns * 1e-6;
        }
        if (out) returnRows(k, out + (uint64_t)g0 * stride, stride);
        if (g0 + k == count) lastLevels = cStatHost.p[k - 1].levels;  // the last source's, as its depths
    }
    GB_CUDA(cudaStreamSynchronize(stream.s));
    GB_CUDA(cudaStreamSynchronize(copyStream.s));
    return true;
}
