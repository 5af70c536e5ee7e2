// graph_prep.cu -- graph preparation on the GPU: fromEdgeList, transpose,
// symmetrize and permute (the reference's src/graph/csr.cpp:112-163 and
// src/graph/transform.cpp:9-76, which run on the host and dominate the wall
// time of preparing the 234M-edge graphs).
//
// All four reduce to one step: write one 64-bit key (row << b | column) per
// output entry (b = bits of n - 1), sort the keys, optionally drop repeated
// keys and self-loops, and count rows into row_ptr.  Sorting (row, column)
// keys gives exactly the reference's outputs: rows in id order, every row
// sorted by column.
//
// Sort: least-significant-digit radix sort with 8-bit digits, one pass per
// digit of the key's used bits.  Each pass: (1) per-tile digit histograms
// (tiles of 4096 keys, shared-memory atomics), (2) one exclusive scan of the
// digit-major histogram table (the single-pass scan of prims.cu), (3) a
// stable scatter: a tile is ranked in 16 rounds of 256 keys, within a warp by
// __match_any_sync peers, across the block's warps by a shared-memory table
// of per-warp digit counts (entries tagged with the round, so nothing is
// cleared between rounds), across rounds by running digit bases.
#include <algorithm>
#include <cstdlib>
#include <cstring>
#include <vector>

#include "capi_util.hpp"
#include "graph_host.hpp"
#include "graph_prep.cuh"
#include "host_copy.hpp"

namespace gb {
namespace {

constexpr int kRsThreads = 256;
constexpr int kRsRounds = 16;
constexpr int kRsTile = kRsThreads * kRsRounds;  // keys per block
constexpr int kRsWarps = kRsThreads / 32;
constexpr unsigned long long kNoKey = ~0ull;

__global__ void __launch_bounds__(kRsThreads) rsHistKernel(const unsigned long long* keys, uint64_t n, int shift,
                                                           uint32_t* counts, uint32_t tiles) {
    __shared__ uint32_t h[256];
    h[threadIdx.x] = 0;
    __syncthreads();
    const uint64_t base = (uint64_t)blockIdx.x * kRsTile;
    for (int r = 0; r < kRsRounds; ++r) {
        const uint64_t i = base + (uint64_t)r * kRsThreads + threadIdx.x;
        if (i < n) atomicAdd(&h[(keys[i] >> shift) & 255u], 1u);
    }
    __syncthreads();
    counts[(uint64_t)threadIdx.x * tiles + blockIdx.x] = h[threadIdx.x];  // digit-major
}

__global__ void __launch_bounds__(kRsThreads) rsScatterKernel(const unsigned long long* keys,
                                                              unsigned long long* out, uint64_t n, int shift,
                                                              const uint32_t* offsets, uint32_t tiles) {
    __shared__ uint32_t base[256];              // running position of each digit in this tile
    __shared__ uint32_t wcnt[kRsWarps][256];    // (round + 1) << 16 | count of the digit in warp w
    __shared__ uint32_t wpre[kRsWarps][256];    // exclusive prefix over warps, this round
    const unsigned tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    base[tid] = offsets[(uint64_t)tid * tiles + blockIdx.x];
    for (int w = 0; w < kRsWarps; ++w) wcnt[w][tid] = 0;
    __syncthreads();
    const uint64_t tileBase = (uint64_t)blockIdx.x * kRsTile;
    for (int r = 0; r < kRsRounds; ++r) {
        const uint64_t i = tileBase + (uint64_t)r * kRsThreads + tid;
        const bool valid = i < n;
        const unsigned long long k = valid ? keys[i] : kNoKey;
        const uint32_t d = valid ? (uint32_t)((k >> shift) & 255u) : 256u + lane;  // invalid lanes: own group
        const unsigned peers = __match_any_sync(0xFFFFFFFFu, d);
        const uint32_t rank = __popc(peers & ((1u << lane) - 1u));
        const uint32_t tag = (uint32_t)(r + 1) << 16;
        if (valid && rank == 0) wcnt[warp][d] = tag | __popc(peers);
        __syncthreads();
        {  // digit tid: prefix over warps
            uint32_t run = 0;
            for (int w = 0; w < kRsWarps; ++w) {
                wpre[w][tid] = run;
                const uint32_t e = wcnt[w][tid];
                run += (e >> 16) == (uint32_t)(r + 1) ? (e & 0xFFFFu) : 0u;
            }
            __syncthreads();
            if (valid) out[base[d] + wpre[warp][d] + rank] = k;
            __syncthreads();
            base[tid] += run;
        }
        __syncthreads();
    }
}

// Sorted keys to CSR without intermediate arrays.  A key is kept when it starts
// a new value (unique) and is not a self-loop (dropSelf); b = column bits.  One
// pass counts each tile's kept keys, and after a scan of those counts a second
// writes the kept columns at their places and, wherever the row changes, the
// row pointers of the rows that begin there (empty rows among them; more than
// kCsrGap of those are left to a block of a third kernel).  Measured on 17.6M keys: 0.78 ms with keep and position arrays and a degree atomic per
// key, 0.2 ms so.
constexpr int kCsrThreads = 256, kCsrItems = 8, kCsrTile = kCsrThreads * kCsrItems;
constexpr uint64_t kCsrGap = 64;

__device__ __forceinline__ bool keptKey(const unsigned long long* keys, uint64_t i, int b, bool unique, bool dropSelf) {
    const unsigned long long k = keys[i], mask = (1ull << b) - 1ull;
    if (unique && i > 0 && keys[i - 1] == k) return false;
    return !(dropSelf && (k >> b) == (k & mask));
}

__global__ void __launch_bounds__(kCsrThreads) csrCountKernel(const unsigned long long* keys, uint64_t n, int b,
                                                              bool unique, bool dropSelf, uint32_t* counts) {
    const uint64_t base = (uint64_t)blockIdx.x * kCsrTile;
    uint32_t c = 0;
#pragma unroll
    for (int r = 0; r < kCsrItems; ++r) {
        const uint64_t i = base + (uint64_t)r * kCsrThreads + threadIdx.x;
        c += __syncthreads_count(i < n && keptKey(keys, i, b, unique, dropSelf));
    }
    if (threadIdx.x == 0) counts[blockIdx.x] = c;
}

// rp[x] = value for x in [lo, hi), or an entry of the gap list: gaps[0] counts them.
__device__ __forceinline__ void fillRows(uint32_t* rp, uint64_t lo, uint64_t hi, uint32_t value, uint32_t* gaps) {
    if (hi > lo + kCsrGap) {
        uint32_t* g = gaps + 1 + 3 * (uint64_t)atomicAdd(gaps, 1u);
        g[0] = (uint32_t)lo;
        g[1] = (uint32_t)hi;
        g[2] = value;
        return;
    }
    for (uint64_t x = lo; x < hi; ++x) rp[x] = value;
}

__global__ void csrGapsKernel(const uint32_t* gaps, uint32_t* rp) {
    const uint32_t count = gaps[0];
    for (uint32_t i = blockIdx.x; i < count; i += gridDim.x) {
        const uint32_t* g = gaps + 1 + 3 * (uint64_t)i;
        for (uint64_t x = (uint64_t)g[0] + threadIdx.x; x < g[1]; x += blockDim.x) rp[x] = g[2];
    }
}

__global__ void __launch_bounds__(kCsrThreads) csrEmitKernel(const unsigned long long* keys, uint64_t n, uint64_t rows,
                                                             int b, bool unique, bool dropSelf, const uint32_t* starts,
                                                             uint32_t* col, uint32_t* rp, uint32_t* gaps) {
    __shared__ uint32_t sWarp[kCsrThreads / 32];
    const unsigned long long mask = (1ull << b) - 1ull;
    const unsigned lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const uint64_t base = (uint64_t)blockIdx.x * kCsrTile;
    uint32_t run = starts[blockIdx.x];
    for (int r = 0; r < kCsrItems; ++r) {
        const uint64_t i = base + (uint64_t)r * kCsrThreads + threadIdx.x;
        const bool in = i < n, keep = in && keptKey(keys, i, b, unique, dropSelf);
        const unsigned ball = __ballot_sync(kFull, keep);
        if (lane == 0) sWarp[warp] = __popc(ball);
        __syncthreads();
        uint32_t before = 0, all = 0;
#pragma unroll
        for (int w = 0; w < kCsrThreads / 32; ++w) {
            before += w < (int)warp ? sWarp[w] : 0u;
            all += sWarp[w];
        }
        __syncthreads();
        if (in) {
            const unsigned long long k = keys[i];
            const uint32_t pos = run + before + __popc(ball & lanemaskLt());
            if (keep) col[pos] = (uint32_t)(k & mask);
            const uint64_t row = k >> b;
            // rows after the previous key's begin here; the first key also opens row 0
            fillRows(rp, i > 0 ? (keys[i - 1] >> b) + 1 : 0, row + 1, pos, gaps);
            if (i + 1 == n) fillRows(rp, row + 1, rows + 1, pos + (keep ? 1u : 0u), gaps);
        }
        run += all;
    }
}

__global__ void initIotaKernel(uint32_t* p, uint64_t n) {
    for (uint64_t v = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; v < n; v += (uint64_t)gridDim.x * blockDim.x)
        p[v] = (uint32_t)v;
}

// Keys of a CSR's entries: (map(row) or col-as-row) per mode.
//   mode 0: (row, col)             mode 1: (col, row)  (transpose)
//   mode 2: (perm[row], perm[col])  mode 3: (row, col) and (col, row) (symmetrize)
// out has m (modes 0-2) or 2m (mode 3) keys; a warp per row, but rows of more
// than kLongRow entries are left for the whole block at its end (by a warp, a row
// of 2M entries takes 2.3 ms).
constexpr uint32_t kLongRow = 4096, kLongRows = 64;

__global__ void csrKeysKernel(const uint32_t* rp, const uint32_t* ci, uint64_t n, uint64_t m, int b, int mode,
                              const uint32_t* perm, unsigned long long* out) {
    __shared__ uint32_t longRow[kLongRows], longs;
    if (threadIdx.x == 0) longs = 0;
    __syncthreads();
    auto emit = [&](unsigned long long u, uint32_t i) {
        const unsigned long long w = ci[i];
        unsigned long long k;
        if (mode == 1) k = (w << b) | u;
        else if (mode == 2) k = ((unsigned long long)perm[u] << b) | perm[w];
        else k = (u << b) | w;
        out[i] = k;
        if (mode == 3) out[m + i] = (w << b) | u;
    };
    const uint64_t nw = ((uint64_t)gridDim.x * blockDim.x) >> 5;
    const unsigned lane = threadIdx.x & 31;
    for (uint64_t v = ((uint64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5; v < n; v += nw) {
        const uint32_t s = rp[v], e = rp[v + 1];
        if (e - s > kLongRow) {  // warp-uniform
            uint32_t slot = 0;
            if (lane == 0) slot = atomicAdd(&longs, 1u);
            slot = __shfl_sync(kFull, slot, 0);
            if (slot < kLongRows) {
                if (lane == 0) longRow[slot] = (uint32_t)v;
                continue;
            }
        }
        for (uint32_t i = s + lane; i < e; i += 32) emit(v, i);
    }
    __syncthreads();
    for (uint32_t k = 0; k < min(longs, kLongRows); ++k) {
        const uint32_t v = longRow[k], e = rp[v + 1];
        for (uint64_t i = (uint64_t)rp[v] + threadIdx.x; i < e; i += blockDim.x) emit(v, (uint32_t)i);
    }
}

__global__ void edgeKeysKernel(const uint32_t* eu, const uint32_t* ev, uint64_t ne, int b, bool both,
                               unsigned long long* out) {
    for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < ne; i += (uint64_t)gridDim.x * blockDim.x) {
        const unsigned long long u = eu[i], v = ev[i];
        out[i] = (u << b) | v;
        if (both) out[ne + i] = (v << b) | u;
    }
}

// Input checks on the device (every id that reaches the key kernels must be
// below n): bad |= 1 row_ptr decreases, 2 column >= n, 4 edge endpoint >= n,
// 8 perm value >= n or repeated (seen: ceil(n/32) zeroed words).  bad[1]
// becomes the longest list's length.
__global__ void checkCsrKernel(const uint32_t* rp, const uint32_t* ci, uint64_t n, uint64_t m, unsigned* bad) {
    const uint64_t stride = (uint64_t)gridDim.x * blockDim.x;
    unsigned f = 0, longest = 0;
    for (uint64_t v = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; v < n; v += stride) {
        const uint32_t b = rp[v], e = rp[v + 1];
        if (b > e) f |= 1u;
        else longest = max(longest, e - b);
    }
    longest = __reduce_max_sync(0xFFFFFFFFu, longest);
    if ((threadIdx.x & 31) == 0 && longest) atomicMax(bad + 1, longest);
    for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < m; i += stride)
        if (ci[i] >= n) f |= 2u;
    if (f) atomicOr(bad, f);
}

__global__ void checkEdgesKernel(const uint32_t* eu, const uint32_t* ev, uint64_t ne, uint64_t n, unsigned* bad) {
    unsigned f = 0;
    for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < ne; i += (uint64_t)gridDim.x * blockDim.x)
        if (eu[i] >= n || ev[i] >= n) f |= 4u;
    if (f) atomicOr(bad, f);
}

__global__ void checkPermKernel(const uint32_t* perm, uint64_t n, uint32_t* seen, unsigned* bad) {
    for (uint64_t v = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; v < n; v += (uint64_t)gridDim.x * blockDim.x) {
        const uint32_t p = perm[v];
        if (p >= n) {
            atomicOr(bad, 8u);
            continue;
        }
        if (atomicOr(&seen[p >> 5], 1u << (p & 31)) & (1u << (p & 31))) atomicOr(bad, 8u);
    }
}

// Connected components (symmetric graph) by hooking and pointer jumping:
// every edge hooks the larger of its endpoints' roots under the smaller
// (atomicMin), then every vertex jumps to its root; repeated until no hook
// changes anything.  A root only ever moves to a smaller id, so each
// component ends rooted at its smallest vertex: the reference's component
// order (components numbered by their first, i.e. smallest, vertex).
__device__ __forceinline__ uint32_t ccRoot(const uint32_t* parent, uint32_t v) {
    uint32_t p = parent[v];
    while (p != v) {
        v = p;
        p = parent[v];
    }
    return v;
}

__global__ void ccHookKernel(const uint32_t* rp, const uint32_t* ci, uint64_t n, uint32_t* parent, unsigned* changed) {
    const uint64_t nw = ((uint64_t)gridDim.x * blockDim.x) >> 5;
    const unsigned lane = threadIdx.x & 31;
    bool any = false;
    for (uint64_t u = ((uint64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5; u < n; u += nw) {
        for (uint32_t i = rp[u] + lane; i < rp[u + 1]; i += 32) {
            const uint32_t v = ci[i];
            if (v <= u) continue;  // each undirected edge once
            const uint32_t ru = ccRoot(parent, (uint32_t)u), rv = ccRoot(parent, v);
            if (ru == rv) continue;
            const uint32_t hi = ru > rv ? ru : rv, lo = ru > rv ? rv : ru;
            if (atomicMin(&parent[hi], lo) > lo) any = true;
        }
    }
    if (__any_sync(0xFFFFFFFFu, any) && lane == 0) atomicOr(changed, 1u);
}

__global__ void ccJumpKernel(uint64_t n, uint32_t* parent) {
    for (uint64_t v = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; v < n; v += (uint64_t)gridDim.x * blockDim.x)
        parent[v] = ccRoot(parent, (uint32_t)v);
}

// size per root, then the best (largest; the smallest root among equals)
// packed as (size << 32) | (~root) into one atomicMax.
__global__ void ccSizeKernel(uint64_t n, const uint32_t* parent, uint32_t* size) {
    for (uint64_t v = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; v < n; v += (uint64_t)gridDim.x * blockDim.x)
        atomicAdd(&size[parent[v]], 1u);
}

__global__ void ccBestKernel(uint64_t n, const uint32_t* size, unsigned long long* best) {
    unsigned long long b = 0;
    for (uint64_t v = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; v < n; v += (uint64_t)gridDim.x * blockDim.x)
        if (size[v]) {
            const unsigned long long key = ((unsigned long long)size[v] << 32) | (0xFFFFFFFFu - (uint32_t)v);
            b = key > b ? key : b;
        }
    if (b) atomicMax(best, b);
}

__global__ void ccMaskKernel(uint64_t n, const uint32_t* parent, const unsigned long long* best, uint8_t* ok) {
    const uint32_t root = 0xFFFFFFFFu - (uint32_t)(*best & 0xFFFFFFFFull);
    for (uint64_t v = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; v < n; v += (uint64_t)gridDim.x * blockDim.x)
        ok[v] = parent[v] == root ? 1 : 0;
}

}  // namespace

uint32_t prepGrid(uint64_t work, uint32_t threads) {
    const uint64_t g = (work + threads - 1) / threads;
    return (uint32_t)std::max<uint64_t>(1, std::min<uint64_t>(g, (uint64_t)deviceSmCount() * 16));
}

int keyBits(uint64_t n) {
    int b = 1;
    while (b < 32 && (1ull << b) < n) ++b;
    return b;
}

void permutedKeys(const uint32_t* rp, const uint32_t* ci, uint64_t n, uint64_t m, int b, const uint32_t* perm,
                  unsigned long long* keys, cudaStream_t st) {
    csrKeysKernel<<<prepGrid(n * 32, 256), 256, 0, st>>>(rp, ci, n, m, b, 2, perm, keys);
    GB_LAUNCH_CHECK();
}

// Sorts N keys whose used bits are [0, bits); a holds the result (after an odd
// number of passes the two buffers have changed places).
void radixSortKeys(DevBuf<unsigned long long>& a, DevBuf<unsigned long long>& tmp, uint64_t N, int bits,
                   ScanScratch& sc, cudaStream_t st, DevBuf<uint32_t>* countsScratch) {
    if (N < 2) return;
    if (N >= (1ull << 32)) throw Error(GB_ERR_ARG, "graph prep: more than 2^32 entries");
    const uint32_t tiles = (uint32_t)((N + kRsTile - 1) / kRsTile);
    DevBuf<uint32_t> own;
    DevBuf<uint32_t>& counts = countsScratch ? *countsScratch : own;
    counts.ensure((uint64_t)tiles * 256 + 1);
    tmp.ensure(N);
    unsigned long long* src = a.get();
    unsigned long long* dst = tmp.get();
    int passes = 0;
    for (int shift = 0; shift < bits; shift += 8, ++passes) {
        rsHistKernel<<<tiles, kRsThreads, 0, st>>>(src, N, shift, counts.get(), tiles);
        GB_LAUNCH_CHECK();
        scanExclusive(counts.get(), counts.get(), (uint64_t)tiles * 256, nullptr, sc, st);
        rsScatterKernel<<<tiles, kRsThreads, 0, st>>>(src, dst, N, shift, counts.get(), tiles);
        GB_LAUNCH_CHECK();
        std::swap(src, dst);
    }
    if (passes & 1) {
        if (tmp.n >= a.n) a.swap(tmp);  // no caller loses room
        else GB_CUDA(cudaMemcpyAsync(a.get(), src, N * 8, cudaMemcpyDeviceToDevice, st));
    }
}

constexpr uint64_t kStagedMin = 16u << 20;  // bytes of a result from which its copy is staged

// Sorted keys -> CSR (host arrays in *out), optionally unique / without
// self-loops.  The columns take the sort's second buffer.
void keysToCsr(DevBuf<unsigned long long>& keys, DevBuf<unsigned long long>& tmp, uint64_t N, uint64_t n, int b,
               bool unique, bool dropSelf, uint32_t flags, ScanScratch& sc, cudaStream_t st, gb_csr* out) {
    DevBuf<uint32_t> counts, rp, gaps;
    rp.ensure(n + 1);
    uint32_t m2 = 0;
    uint32_t* col = nullptr;
    if (N) {
        tmp.ensure((N + 1) / 2);
        col = reinterpret_cast<uint32_t*>(tmp.get());
        const uint32_t tiles = (uint32_t)((N + kCsrTile - 1) / kCsrTile);
        counts.ensure(tiles + 1);
        csrCountKernel<<<tiles, kCsrThreads, 0, st>>>(keys.get(), N, b, unique, dropSelf, counts.get());
        GB_LAUNCH_CHECK();
        scanExclusive(counts.get(), counts.get(), tiles, counts.get() + tiles, sc, st);
        gaps.ensure(1 + 3 * (n / kCsrGap + 2));
        GB_CUDA(cudaMemsetAsync(gaps.get(), 0, 4, st));
        csrEmitKernel<<<tiles, kCsrThreads, 0, st>>>(keys.get(), N, n, b, unique, dropSelf, counts.get(), col, rp.get(),
                                                     gaps.get());
        GB_LAUNCH_CHECK();
        csrGapsKernel<<<deviceSmCount(), 256, 0, st>>>(gaps.get(), rp.get());
        GB_LAUNCH_CHECK();
        GB_CUDA(cudaMemcpyAsync(&m2, counts.get() + tiles, 4, cudaMemcpyDeviceToHost, st));
    } else {
        GB_CUDA(cudaMemsetAsync(rp.get(), 0, (n + 1) * 4, st));
    }
    GB_CUDA(cudaStreamSynchronize(st));
    uint32_t* hrp = static_cast<uint32_t*>(std::malloc((n + 1) * 4));
    uint32_t* hci = static_cast<uint32_t*>(std::malloc(std::max<uint64_t>(m2, 1) * 4));
    if (!hrp || !hci) {
        std::free(hrp);
        std::free(hci);
        throw Error(GB_ERR_OOM, "graph prep: host allocation failed");
    }
    try {
        // A ring of its own has to be page-locked, 2.5 ms.  A plain copy costs less
        // into memory that is mapped already, up to some 30 MB, and more into pages
        // that it touches first.  Ms a build with plain copies / with the ring, by
        // bytes of the result, with the results kept: 4.1 MB 6.3 / 7.9, 8.2 MB 8.1 /
        // 8.8, 12.2 MB 10.4 / 9.1, 16.3 MB 12.1 / 9.7, 24.5 MB 16.8 / 11.2, 47.6 MB
        // 30.5 / 18.2, 71.3 MB 45.6 / 24.2; each freed before the next: 12.2 MB 5.0 /
        // 8.4, 16.3 MB 5.3 / 8.5, 24.5 MB 6.8 / 9.9, 47.6 MB 30.7 / 18.0, 71.3 MB 43.7 /
        // 23.4.  The line lies where neither loses much to the other.
        if ((n + m2) * 4 < kStagedMin) {
            GB_CUDA(cudaMemcpyAsync(hrp, rp.get(), (n + 1) * 4, cudaMemcpyDeviceToHost, st));
            GB_CUDA(cudaMemcpyAsync(hci, col, (uint64_t)m2 * 4, cudaMemcpyDeviceToHost, st));
            GB_CUDA(cudaStreamSynchronize(st));
        } else {
            StagedCopy staged;
            staged.run(rp.get(), (n + 1) * 4, hrp, st);
            staged.run(col, (uint64_t)m2 * 4, hci, st);
        }
    } catch (...) {
        std::free(hrp);
        std::free(hci);
        throw;
    }
    out->n = n;
    out->m = m2;
    out->flags = flags;
    out->row_ptr = hrp;
    out->col_idx = hci;
}

// Connected components of a symmetric device CSR: parent[v] = the smallest
// vertex of v's component (hook + jump rounds; each round at least halves the
// number of roots that still have a smaller neighbouring root, so 64 rounds
// cover any n < 2^32 many times over).
void connectedComponents(const uint32_t* rp, const uint32_t* ci, uint64_t n, uint32_t* parent, cudaStream_t st) {
    DevBuf<unsigned> changed;
    changed.ensure(1);
    initIotaKernel<<<prepGrid(n, 256), 256, 0, st>>>(parent, n);
    GB_LAUNCH_CHECK();
    for (int round = 0; round < 64; ++round) {
        GB_CUDA(cudaMemsetAsync(changed.get(), 0, 4, st));
        ccHookKernel<<<prepGrid(n * 32, 256), 256, 0, st>>>(rp, ci, n, parent, changed.get());
        GB_LAUNCH_CHECK();
        ccJumpKernel<<<prepGrid(n, 256), 256, 0, st>>>(n, parent);
        GB_LAUNCH_CHECK();
        unsigned h = 0;
        GB_CUDA(cudaMemcpyAsync(&h, changed.get(), 4, cudaMemcpyDeviceToHost, st));
        GB_CUDA(cudaStreamSynchronize(st));
        if (h == 0) return;
    }
    throw Error(GB_ERR_STATE, "connected components did not settle in 64 rounds");
}

namespace {

// Reads the device check words; throws if any check failed.  Returns the
// second word (checkCsrKernel's longest list; 0 after the other checks).
uint32_t requireChecks(DevBuf<unsigned>& bad, cudaStream_t st) {
    unsigned w[2];
    GB_CUDA(cudaMemcpyAsync(w, bad.get(), 8, cudaMemcpyDeviceToHost, st));
    GB_CUDA(cudaStreamSynchronize(st));
    const unsigned h = w[0];
    if (h & 1u) throw Error(GB_ERR_ARG, "graph prep: row_ptr must not decrease");
    if (h & 2u) throw Error(GB_ERR_ARG, "graph prep: column id >= n");
    if (h & 4u) throw Error(GB_ERR_ARG, "gb_csr_from_edges_gpu: edge endpoint >= n");
    if (h & 8u) throw Error(GB_ERR_ARG, "gb_csr_permute_gpu: perm is not a permutation of [0, n)");
    return w[1];
}

// Uploads a host CSR.
void uploadCsr(const gb_csr* g, DevBuf<uint32_t>& rp, DevBuf<uint32_t>& ci, cudaStream_t st) {
    rp.ensure(g->n + 1);
    ci.ensure(g->m + 1);
    GB_CUDA(cudaMemcpyAsync(rp.get(), g->row_ptr, (g->n + 1) * 4, cudaMemcpyHostToDevice, st));
    if (g->m) GB_CUDA(cudaMemcpyAsync(ci.get(), g->col_idx, g->m * 4, cudaMemcpyHostToDevice, st));
}

}  // namespace

void checkDeviceCsr(const uint32_t* rp, const uint32_t* ci, uint64_t n, uint64_t m, cudaStream_t st,
                    uint32_t* maxDegree) {
    DevBuf<unsigned> bad;
    bad.ensure(2);
    GB_CUDA(cudaMemsetAsync(bad.get(), 0, 8, st));
    checkCsrKernel<<<prepGrid(std::max(n, m), 256), 256, 0, st>>>(rp, ci, n, m, bad.get());
    GB_LAUNCH_CHECK();
    const uint32_t longest = requireChecks(bad, st);
    if (maxDegree) *maxDegree = longest;
}

void uploadCheckedCsr(const gb_csr* g, DevBuf<uint32_t>& rp, DevBuf<uint32_t>& ci, cudaStream_t st) {
    GB_REQUIRE(g && g->row_ptr && (g->m == 0 || g->col_idx), "null CSR arrays");
    GB_REQUIRE(g->n >= 1 && g->n < 0xFFFFFFFFull, "graph prep: n must be in [1, 2^32 - 1)");
    GB_REQUIRE(g->m < (1ull << 32), "graph prep: m must fit in uint32");
    GB_REQUIRE(g->row_ptr[0] == 0 && g->row_ptr[g->n] == g->m, "graph prep: row_ptr must run from 0 to m");
    DevBuf<unsigned> bad;
    bad.ensure(2);
    GB_CUDA(cudaMemsetAsync(bad.get(), 0, 8, st));
    uploadCsr(g, rp, ci, st);
    checkCsrKernel<<<prepGrid(std::max(g->n, g->m), 256), 256, 0, st>>>(rp.get(), ci.get(), g->n, g->m, bad.get());
    GB_LAUNCH_CHECK();
    requireChecks(bad, st);
}

namespace {

constexpr uint32_t kFlagDirected = 1u, kFlagSorted = 2u, kFlagDedup = 4u;

// mode as csrKeysKernel; see the entry points for flags and uniqueness.
void csrOp(const gb_csr* g, int mode, const uint32_t* permHost, bool unique, bool dropSelf, uint32_t flags,
           gb_csr* out) {
    GB_REQUIRE(g && out, "null argument");
    GB_REQUIRE(g->n >= 1 && g->n < 0xFFFFFFFFull, "graph prep: n must be in [1, 2^32 - 1)");
    GB_REQUIRE(g->m < (1ull << 32), "graph prep: m must fit in uint32");
    GB_REQUIRE(g->row_ptr && (g->m == 0 || g->col_idx), "null CSR arrays");
    GB_REQUIRE(g->row_ptr[0] == 0 && g->row_ptr[g->n] == g->m, "graph prep: row_ptr must run from 0 to m");
    Stream st;
    ScanScratch sc;
    DevBuf<uint32_t> rp, ci, perm, seen;
    DevBuf<unsigned> bad;
    bad.ensure(2);
    GB_CUDA(cudaMemsetAsync(bad.get(), 0, 8, st.s));
    uploadCsr(g, rp, ci, st.s);
    checkCsrKernel<<<prepGrid(std::max(g->n, g->m), 256), 256, 0, st.s>>>(rp.get(), ci.get(), g->n, g->m, bad.get());
    GB_LAUNCH_CHECK();
    if (mode == 2) {
        perm.ensure(g->n);
        seen.ensure((g->n + 31) / 32);
        GB_CUDA(cudaMemcpyAsync(perm.get(), permHost, g->n * 4, cudaMemcpyHostToDevice, st.s));
        GB_CUDA(cudaMemsetAsync(seen.get(), 0, (g->n + 31) / 32 * 4, st.s));
        checkPermKernel<<<prepGrid(g->n, 256), 256, 0, st.s>>>(perm.get(), g->n, seen.get(), bad.get());
        GB_LAUNCH_CHECK();
    }
    requireChecks(bad, st.s);
    const int b = keyBits(g->n);
    const uint64_t N = mode == 3 ? 2 * g->m : g->m;
    DevBuf<unsigned long long> keys, tmp;
    keys.ensure(N + 1);
    if (g->m) {
        csrKeysKernel<<<prepGrid(g->n * 32, 256), 256, 0, st.s>>>(rp.get(), ci.get(), g->n, g->m, b, mode, perm.get(),
                                                                 keys.get());
        GB_LAUNCH_CHECK();
    }
    radixSortKeys(keys, tmp, N, 2 * b, sc, st.s);
    keysToCsr(keys, tmp, N, g->n, b, unique, dropSelf, flags, sc, st.s, out);
}

}  // namespace
}  // namespace gb

using namespace gb;

extern "C" {

int gb_csr_from_edges_gpu(uint64_t n, const uint32_t* eu, const uint32_t* ev, uint64_t ne, int directed,
                          gb_csr* out) {
    return guard([&] {
        GB_REQUIRE(out && (ne == 0 || (eu && ev)), "null argument");
        GB_REQUIRE(n >= 1 && n < 0xFFFFFFFFull, "graph prep: n must be in [1, 2^32 - 1)");
        Stream st;
        ScanScratch sc;
        DevBuf<uint32_t> du, dv;
        DevBuf<unsigned> bad;
        bad.ensure(2);
        du.ensure(ne + 1);
        dv.ensure(ne + 1);
        GB_CUDA(cudaMemsetAsync(bad.get(), 0, 8, st.s));
        if (ne) {
            GB_CUDA(cudaMemcpyAsync(du.get(), eu, ne * 4, cudaMemcpyHostToDevice, st.s));
            GB_CUDA(cudaMemcpyAsync(dv.get(), ev, ne * 4, cudaMemcpyHostToDevice, st.s));
            checkEdgesKernel<<<prepGrid(ne, 256), 256, 0, st.s>>>(du.get(), dv.get(), ne, n, bad.get());
            GB_LAUNCH_CHECK();
        }
        requireChecks(bad, st.s);
        const int b = keyBits(n);
        const uint64_t N = directed ? ne : 2 * ne;
        DevBuf<unsigned long long> keys, tmp;
        keys.ensure(N + 1);
        if (ne) {
            edgeKeysKernel<<<prepGrid(ne, 256), 256, 0, st.s>>>(du.get(), dv.get(), ne, b, !directed, keys.get());
            GB_LAUNCH_CHECK();
        }
        radixSortKeys(keys, tmp, N, 2 * b, sc, st.s);
        keysToCsr(keys, tmp, N, n, b, true, true, (directed ? kFlagDirected : 0u) | kFlagSorted | kFlagDedup, sc, st.s,
                  out);
    });
}

int gb_csr_transpose_gpu(const gb_csr* g, gb_csr* out) {
    return guard([&] { csrOp(g, 1, nullptr, false, false, g ? g->flags : 0u, out); });
}

int gb_csr_symmetrize_gpu(const gb_csr* g, gb_csr* out) {
    return guard([&] {
        GB_REQUIRE(g && out, "null argument");
        if (!(g->flags & kFlagDirected)) {  // undirected: the same graph, as given (transform.cpp:27)
            out->row_ptr = static_cast<uint32_t*>(std::malloc((g->n + 1) * 4));
            out->col_idx = static_cast<uint32_t*>(std::malloc(std::max<uint64_t>(g->m, 1) * 4));
            if (!out->row_ptr || !out->col_idx) {
                std::free(out->row_ptr);
                std::free(out->col_idx);
                out->row_ptr = out->col_idx = nullptr;
                throw Error(GB_ERR_OOM, "graph prep: host allocation failed");
            }
            std::memcpy(out->row_ptr, g->row_ptr, (g->n + 1) * 4);
            if (g->m) std::memcpy(out->col_idx, g->col_idx, g->m * 4);
            out->n = g->n;
            out->m = g->m;
            out->flags = g->flags;
            return;
        }
        GB_REQUIRE(g->flags & kFlagDedup,
                   "gb_csr_symmetrize_gpu: the input must be duplicate-free (kFlagDedup); "
                   "gb_csr_symmetrize handles lists with repeated entries");
        csrOp(g, 3, nullptr, true, false, kFlagSorted | kFlagDedup, out);
    });
}

int gb_csr_permute_gpu(const gb_csr* g, const uint32_t* perm, gb_csr* out) {
    return guard([&] {
        GB_REQUIRE(g && perm, "null argument");
        csrOp(g, 2, perm, false, false, g->flags, out);  // perm is checked on the device
    });
}

int gb_pick_sources_gpu(const gb_csr* g, int count, uint64_t seed, int any_component, uint32_t* out, int* k) {
    return guard([&] {
        GB_REQUIRE(g && g->row_ptr && out, "null argument");
        GB_REQUIRE(g->n >= 1 && g->n < 0xFFFFFFFFull, "graph prep: n must be in [1, 2^32 - 1)");
        GB_REQUIRE(g->row_ptr[0] == 0 && g->row_ptr[g->n] == g->m, "graph prep: row_ptr must run from 0 to m");
        const uint64_t n = g->n;
        std::vector<uint8_t> ok(n, 1);
        if (!any_component) {
            GB_REQUIRE(!(g->flags & kFlagDirected),
                       "gb_pick_sources_gpu: components need a symmetric graph (gb_pick_sources follows "
                       "out-edges of directed ones)");
            Stream st;
            DevBuf<uint32_t> rp, ci, parent, size;
            DevBuf<unsigned long long> best;
            DevBuf<uint8_t> dok;
            best.ensure(1);
            uploadCheckedCsr(g, rp, ci, st.s);
            parent.ensure(n);
            size.ensure(n);
            dok.ensure(n);
            connectedComponents(rp.get(), ci.get(), n, parent.get(), st.s);
            GB_CUDA(cudaMemsetAsync(size.get(), 0, n * 4, st.s));
            GB_CUDA(cudaMemsetAsync(best.get(), 0, 8, st.s));
            ccSizeKernel<<<prepGrid(n, 256), 256, 0, st.s>>>(n, parent.get(), size.get());
            ccBestKernel<<<prepGrid(n, 256), 256, 0, st.s>>>(n, size.get(), best.get());
            ccMaskKernel<<<prepGrid(n, 256), 256, 0, st.s>>>(n, parent.get(), best.get(), dok.get());
            GB_LAUNCH_CHECK();
            GB_CUDA(cudaMemcpyAsync(ok.data(), dok.get(), n, cudaMemcpyDeviceToHost, st.s));
            GB_CUDA(cudaStreamSynchronize(st.s));
        }
        auto s = drawSources(n, g->row_ptr, ok, count, seed);
        if (!s.empty()) std::memcpy(out, s.data(), s.size() * 4);
        if (k) *k = (int)s.size();
    });
}

}  // extern "C"
