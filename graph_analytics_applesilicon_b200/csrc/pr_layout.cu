// pr_layout.cu -- the adaptive pull's layout, built on the GPU
// (GpuPageRank::prepareAdaptive, src/metal/pagerank_gpu.mm:70-86).
//
// Vertices are relabeled by descending in-degree (ties by id), so the most
// gathered contributions sit together and lists of one length are neighbours.
// Lists are sorted by new id (one radix sort of (row, column) keys) and padded
// to whole 16-byte vectors with the id n, whose contribution is 0.  All lists
// of one padded length form a run (GbPrRun): a vertex's list is found from its
// id, with no row pointer to load and no ragged ends to mask.  Classes by
// in-degree d (the reference's three bins, refined):
//   d >= large_min            split into warp chunks (a warp per list while one
//                             chunk holds it);
//   small_max <= d            a group of lanes per list, four vectors per lane
//                             (two or eight: 3% slower on Chung-Lu, 1-2% on the web graph);
//   d < small_max             a lane per list, interleaved in blocks of 32.
#include <algorithm>
#include <vector>

#include "graph_prep.cuh"
#include "pagerank.hpp"

namespace gb {
namespace {

constexpr uint32_t kPrInterVecs = 8;   // longest interleaved list, in vectors
// An adaptive sweep of a large graph keeps the contributions that are gathered
// most in shared memory, whose gathers cost the L1 and the L2 nothing.  A place
// costs each SM 4 bytes of copying per sweep, as long as some 28 gathers
// elsewhere on the GPU, so a vertex needs this out-degree to be worth one; and
// the copying and the one block per SM it leaves room for need a sweep of this
// many entries to pay (us a sweep without / with: Chung-Lu of 3M entries 19.1 /
// 23.7, 9M 38.9 / 39.9, 30M 109 / 109, 76M 277 / 223; R-MAT of 4M 22.2 / 23.1,
// 17M 56.4 / 48.4, 34M 123 / 98).
constexpr uint64_t kPrHotEntries = 12ull << 20;
constexpr uint32_t kPrHotMin = 32;
constexpr uint32_t kPrHotBins = 1u << 14;
constexpr uint32_t kPrLaneVecs = 4;    // vectors per lane a group is sized for

// Vectors per chunk of a split list: as many as leave each of the GPU's warps
// about ten tasks, so that the longest task is a small part of a sweep (web
// graph, 5M entries: 34.2 us a sweep with 256 vectors, 36.9 with 512; Chung-Lu,
// 233M: 873 and 831).
uint32_t chunkVecs(uint64_t m) {
    uint32_t c = 256;
    while (c < 512 && (uint64_t)c * 8 * 65536 <= m) c *= 2;
    return c;
}

__global__ void gatherU32Kernel(const uint32_t* __restrict__ in, const uint32_t* __restrict__ order, uint64_t n,
                                uint32_t* out) {
    for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (uint64_t)gridDim.x * blockDim.x)
        out[i] = in[order[i]];
}

// deg[i] = degree of order[i].
__global__ void orderedDegreesKernel(const uint32_t* __restrict__ rp, const uint32_t* __restrict__ order, uint64_t n,
                                     uint32_t* deg) {
    for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (uint64_t)gridDim.x * blockDim.x)
        deg[i] = rp[order[i] + 1] - rp[order[i]];
}

// Sorted keys to padded lists, a block per split list (by a warp, a list of 2M
// entries takes 1.7 ms), a warp per other list: row i's entries are the sorted
// keys [start[i], start[i + 1]).  Runs are found by their first vertex; the
// split lists' run (run 0 when hubs > 0) gives each list its own place.
__global__ void fillListsKernel(const unsigned long long* __restrict__ keys, const uint32_t* __restrict__ start,
                                uint64_t n, unsigned long long mask, const GbPrRun* __restrict__ runs, uint32_t nRuns,
                                uint32_t hubs, const uint32_t* __restrict__ hubVec, const uint32_t* __restrict__ pos,
                                uint32_t pad, uint32_t* out) {
    const uint64_t nw = ((uint64_t)gridDim.x * blockDim.x) >> 5;
    const unsigned lane = threadIdx.x & 31;
    auto entry = [&](uint32_t s, uint32_t d, uint32_t k) {
        if (k >= d) return pad;
        const uint32_t u = (uint32_t)(keys[s + k] & mask);
        return pos ? pos[u] : u;
    };
    for (uint32_t i = blockIdx.x; i < hubs; i += gridDim.x) {
        const uint32_t s = start[i], d = start[i + 1] - s;
        uint32_t* to = out + 4ull * hubVec[i];
        for (uint32_t k = threadIdx.x; k < (d + 3) / 4 * 4; k += blockDim.x) to[k] = entry(s, d, k);
    }
    for (uint64_t i = hubs + (((uint64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5); i < n; i += nw) {
        const uint32_t s = start[i], d = start[i + 1] - s;
        uint32_t lo = 0, hi = nRuns - 1;
        while (lo < hi) {  // last run with v0 <= i
            const uint32_t mid = (lo + hi + 1) / 2;
            if (runs[mid].v0 <= i) lo = mid;
            else hi = mid - 1;
        }
        const GbPrRun r = runs[lo];
        const uint32_t idx = (uint32_t)i - r.v0, step = r.inter ? 128 : 4;  // entries from one vector to the next
        uint32_t* to = out + 4ull * (r.e0 + (r.inter ? (uint64_t)(idx / 32) * 32 * r.vecs + idx % 32 : (uint64_t)idx * r.vecs));
        for (uint32_t k = lane; k < 4 * r.vecs; k += 32) to[(uint64_t)(k / 4) * step + k % 4] = entry(s, d, k);
    }
}

// The lists of at least splitMin entries of a CSR: counts (hubs, chunks), then
// the chunk table.  A list's chunks are consecutive; the lists' own order is
// that of the atomics and does not matter.
__global__ void countSplitKernel(const uint32_t* __restrict__ rp, uint64_t n, uint32_t splitMin, uint32_t per,
                                 uint32_t* counts) {
    for (uint64_t v = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; v < n; v += (uint64_t)gridDim.x * blockDim.x) {
        const uint32_t d = rp[v + 1] - rp[v];
        if (d < splitMin) continue;
        atomicAdd(&counts[0], 1u);
        atomicAdd(&counts[1], (d - 1) / per + 1);
    }
}

__global__ void fillSplitKernel(const uint32_t* __restrict__ rp, uint64_t n, uint32_t splitMin, uint32_t per,
                                uint32_t* counts, uint4* chunks, uint32_t* first) {
    for (uint64_t v = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; v < n; v += (uint64_t)gridDim.x * blockDim.x) {
        const uint32_t b = rp[v], e = rp[v + 1];
        if (e - b < splitMin) continue;
        const uint32_t cnt = (e - b - 1) / per + 1, h = atomicAdd(&counts[0], 1u), c = atomicAdd(&counts[1], cnt);
        first[2 * h] = c;
        first[2 * h + 1] = cnt;
        for (uint32_t k = 0; k < cnt; ++k)
            chunks[c + k] = make_uint4((uint32_t)v, b + k * per, k + 1 < cnt ? b + (k + 1) * per : e, h);
    }
}

// bins[d] += vertices of out-degree d, for d >= kPrHotMin; the last bin takes all beyond.
__global__ void outdegreeBinsKernel(const uint32_t* __restrict__ outdeg, uint64_t n, uint32_t* bins) {
    for (uint64_t v = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; v < n; v += (uint64_t)gridDim.x * blockDim.x)
        if (outdeg[v] >= kPrHotMin) atomicAdd(&bins[min(outdeg[v], kPrHotBins - 1)], 1u);
}

// Places of the contributions: the vertices of out-degree [lo, hi) get the first
// free of the `hot` first places while there are any, all others (first launch)
// the place hot + v.
__global__ void hotPlacesKernel(const uint32_t* __restrict__ outdeg, uint64_t n, uint32_t lo, uint32_t hi, uint32_t hot,
                                bool first, uint32_t* taken, uint32_t* pos) {
    for (uint64_t base = (uint64_t)blockIdx.x * blockDim.x; base < n; base += (uint64_t)gridDim.x * blockDim.x) {
        const uint64_t v = base + threadIdx.x;
        const uint32_t d = v < n ? outdeg[v] : 0u;
        const bool in = v < n && d >= lo && d < hi;
        const uint32_t slot = warpAppend(in, taken);
        if (in && slot < hot) pos[v] = slot;
        else if (v < n && first) pos[v] = hot + (uint32_t)v;
    }
}

template <class T>
void upload(DevBuf<T>& buf, const std::vector<T>& v, cudaStream_t st) {
    buf.ensure(v.size() + 1);
    if (!v.empty()) GB_CUDA(cudaMemcpyAsync(buf.get(), v.data(), v.size() * sizeof(T), cudaMemcpyHostToDevice, st));
}

uint32_t groupLog2(uint32_t d, uint32_t vecs, uint32_t smallMax, uint32_t largeMin) {
    if (d >= largeMin) return 5;  // a split list of one chunk
    if (d < smallMax) return 0;
    uint32_t lg = 1;
    while (lg < 5 && (kPrLaneVecs << lg) < vecs) ++lg;
    return lg;
}

// Chooses the contributions to keep in shared memory (h.hotA of them, 0 when they
// are too few of the gathers to matter or there is no memory for them) and every
// contribution's place.  The contributions' buffers, which every variant uses, are
// replaced only by larger ones that are there.
void choosePlaces(gb_pr& h, cudaStream_t st) {
    const uint64_t n = h.n;
    h.hotA = 0;
    for (auto& c : h.contrib) GB_CUDA(cudaMemsetAsync(c.get() + n, 0, 16, st));  // the padding's place without any
    if (h.mIn < kPrHotEntries || n + kPrHotMax + 4 >= (1ull << 32)) return;
    DevBuf<uint32_t> bins;
    std::vector<uint32_t> count(kPrHotBins);
    bins.ensure(kPrHotBins);
    GB_CUDA(cudaMemsetAsync(bins.get(), 0, kPrHotBins * 4, st));
    outdegreeBinsKernel<<<prepGrid(n, 256), 256, 0, st>>>(h.outdegA.get(), n, bins.get());
    GB_LAUNCH_CHECK();
    GB_CUDA(cudaMemcpyAsync(count.data(), bins.get(), kPrHotBins * 4, cudaMemcpyDeviceToHost, st));
    GB_CUDA(cudaStreamSynchronize(st));
    // from the largest down: all of out-degree above `cut`, of `cut` as many as there is room for
    uint64_t taken = 0, gathers = 0;
    uint32_t cut = kPrHotBins - 1;
    for (;; --cut) {
        const uint64_t room = std::min<uint64_t>(count[cut], kPrHotMax - taken);
        taken += room;
        gathers += room * cut;
        if (taken == kPrHotMax || cut == kPrHotMin) break;
    }
    if (gathers < h.mIn / 8) return;
    const uint32_t hot = (uint32_t)((taken + 3) / 4 * 4);
    DevBuf<float> larger[2];
    for (int i = 0; i < 2; ++i)
        if (h.contrib[i].n < n + hot + 4 && !larger[i].tryEnsure(n + hot + 4)) return;
    if (!h.posA.tryEnsure(n)) return;
    for (int i = 0; i < 2; ++i) {
        if (larger[i].get()) h.contrib[i].swap(larger[i]);
        GB_CUDA(cudaMemsetAsync(h.contrib[i].get() + n + hot, 0, 16, st));
    }
    GB_CUDA(cudaMemsetAsync(bins.get(), 0, 4, st));
    hotPlacesKernel<<<prepGrid(n, 256), 256, 0, st>>>(h.outdegA.get(), n, cut + 1, 0xFFFFFFFFu, hot, true, bins.get(), h.posA.get());
    GB_LAUNCH_CHECK();
    hotPlacesKernel<<<prepGrid(n, 256), 256, 0, st>>>(h.outdegA.get(), n, cut, cut + 1, hot, false, bins.get(), h.posA.get());
    GB_LAUNCH_CHECK();
    h.hotA = hot;
}

}  // namespace
}  // namespace gb

using namespace gb;

void gb_pr::prepareAdaptive(uint32_t smallMax, uint32_t largeMin) {
    if (binsReady && binSmall == smallMax && binLarge == largeMin) return;
    if (!hasIn) throw Error(GB_ERR_ARG, "gpu_pull_adaptive needs the in-CSR");
    if (n == 0) return;
    binsReady = false;
    invalidateGraphs();
    cudaStream_t st = stream.s;
    ScanScratch sc;
    DevBuf<uint32_t> order, start;
    order.ensure(n);
    permADev.ensure(n);
    degreeRank(rowIn.get(), n, order.get(), permADev.get(), sc, st);
    start.ensure(n + 1);
    orderedDegreesKernel<<<prepGrid(n, 256), 256, 0, st>>>(rowIn.get(), order.get(), n, start.get());
    GB_LAUNCH_CHECK();
    GB_CUDA(cudaMemsetAsync(start.get() + n, 0, 4, st));
    scanExclusive(start.get(), start.get(), n + 1, nullptr, sc, st);
    outdegA.ensure(n);
    gatherU32Kernel<<<prepGrid(n, 256), 256, 0, st>>>(outdeg.get(), order.get(), n, outdegA.get());
    GB_LAUNCH_CHECK();

    choosePlaces(*this, st);

    // how many vertices have each in-degree, from which the hubs and runs follow
    uint32_t longest = 0;
    for (uint64_t v = 0; v < n; ++v) longest = std::max(longest, hostRowIn[v + 1] - hostRowIn[v]);
    std::vector<uint32_t> withDegree((uint64_t)longest + 1, 0);
    for (uint64_t v = 0; v < n; ++v) ++withDegree[hostRowIn[v + 1] - hostRowIn[v]];
    std::vector<uint4> chunks;
    std::vector<uint32_t> first, hubVec;
    std::vector<GbPrRun> runs;
    uint64_t e = 0, tasks = 0, i = 0;  // vectors, tasks and vertices placed so far
    const uint32_t perChunk = chunkVecs(mIn);
    auto closeRun = [&] {              // gives the last run its end and the places of its lists
        GbPrRun& r = runs.back();
        r.vEnd = (uint32_t)i;
        const uint64_t lists = i - r.v0;
        e += (r.inter ? (lists + 31) / 32 * 32 : lists) * r.vecs;
        tasks += (lists + (32u >> r.lg) - 1) >> (5 - r.lg);
    };
    for (int64_t d = longest; d >= 0; --d) {
        const uint32_t count = withDegree[d], vecs = ((uint32_t)d + 3) / 4;
        if (count == 0) continue;
        if ((uint32_t)d >= largeMin && vecs > perChunk) {
            for (uint32_t x = 0; x < count; ++x, ++i) {
                hubVec.push_back((uint32_t)e);
                first.push_back((uint32_t)chunks.size());
                uint32_t c = 0;
                for (uint32_t b = 0; b < vecs; b += perChunk, ++c)
                    chunks.push_back(make_uint4((uint32_t)i, (uint32_t)e + b, (uint32_t)e + std::min(vecs, b + perChunk),
                                                (uint32_t)i));
                first.push_back(c);
                e += vecs;
            }
            continue;
        }
        const uint32_t lg = groupLog2((uint32_t)d, vecs, smallMax, largeMin);
        if (runs.empty() || runs.back().vecs != vecs || runs.back().lg != lg) {
            if (!runs.empty()) closeRun();
            runs.push_back({(uint32_t)tasks, (uint32_t)i, 0, (uint32_t)e, vecs, lg, lg == 0 && vecs <= kPrInterVecs, 0});
        }
        i += count;
    }
    if (!runs.empty()) closeRun();
    nHubs = (uint32_t)hubVec.size();
    nChunks = (uint32_t)chunks.size();
    if (e >= (1ull << 32)) throw Error(GB_ERR_ARG, "adaptive layout exceeds 2^32 16-byte vectors");
    nRuns = (uint32_t)runs.size();
    nRunTasks = (uint32_t)tasks;
    DevBuf<uint32_t> dHubVec;
    upload(dHubVec, hubVec, st);
    upload(hubChunks, chunks, st);
    upload(hubFirst, first, st);
    upload(runsA, runs, st);
    hubDone.ensure(nHubs + 1);
    GB_CUDA(cudaMemsetAsync(hubDone.get(), 0, (nHubs + 1) * sizeof(unsigned), st));
    hubPart.ensure(2 * (size_t)nChunks + 2);
    vecA.ensure(e + 1);
    if (mIn) {
        const int b = keyBits(n);
        DevBuf<unsigned long long> keys, tmp;
        keys.ensure(mIn);
        permutedKeys(rowIn.get(), colIn.get(), n, mIn, b, permADev.get(), keys.get(), st);
        radixSortKeys(keys, tmp, mIn, 2 * b, sc, st);
        fillListsKernel<<<prepGrid(n * 32, 256), 256, 0, st>>>(keys.get(), start.get(), n, (1ull << b) - 1, runsA.get(),
                                                               nRuns, nHubs, dHubVec.get(), hotA ? posA.get() : nullptr,
                                                               (uint32_t)n + hotA, reinterpret_cast<uint32_t*>(vecA.get()));
        GB_LAUNCH_CHECK();
    }
    GB_CUDA(cudaStreamSynchronize(st));
    binSmall = smallMax;
    binLarge = largeMin;
    binsReady = true;
}

// Lanes per list and split lists of the scalar (a lane per list) and vector
// pulls on the graph as given.  A list shares its warp with its neighbours, so
// one much longer than the others would hold them all, and one of 30,000
// entries the whole sweep (R-MAT 18: 165 us of 185): lists of 64 entries per
// lane of a group or more go to warps of their own, in chunks.
void gb_pr::prepareSplit(bool vector) {
    PrSplit& s = split[vector ? 1 : 0];
    if (s.ready) return;
    s.lg = 0;
    if (vector) {  // two vectors per lane at the mean degree
        s.lg = 1;
        while (s.lg < 5 && n && mIn / n > (8ull << s.lg)) ++s.lg;
    }
    s.splitMin = 64u << s.lg;
    constexpr uint32_t kPer = 1024;
    cudaStream_t st = stream.s;
    DevBuf<uint32_t> counts;
    counts.ensure(2);
    uint32_t c[2] = {0, 0};
    GB_CUDA(cudaMemsetAsync(counts.get(), 0, 8, st));
    if (n) {
        countSplitKernel<<<prepGrid(n, 256), 256, 0, st>>>(rowIn.get(), n, s.splitMin, kPer, counts.get());
        GB_LAUNCH_CHECK();
        GB_CUDA(cudaMemcpyAsync(c, counts.get(), 8, cudaMemcpyDeviceToHost, st));
        GB_CUDA(cudaMemsetAsync(counts.get(), 0, 8, st));
        GB_CUDA(cudaStreamSynchronize(st));
    }
    s.chunks.ensure(c[1] + 1);
    s.first.ensure(2 * (size_t)c[0] + 1);
    s.done.ensure(c[0] + 1);
    s.part.ensure(2 * (size_t)c[1] + 1);
    GB_CUDA(cudaMemsetAsync(s.done.get(), 0, (c[0] + 1) * sizeof(unsigned), st));
    if (c[1]) {
        fillSplitKernel<<<prepGrid(n, 256), 256, 0, st>>>(rowIn.get(), n, s.splitMin, kPer, counts.get(), s.chunks.get(),
                                                          s.first.get());
        GB_LAUNCH_CHECK();
        GB_CUDA(cudaStreamSynchronize(st));
    }
    s.nChunks = c[1];
    s.ready = true;
    invalidateGraphs();
}
