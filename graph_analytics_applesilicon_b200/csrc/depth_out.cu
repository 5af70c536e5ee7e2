// depth_out.cu -- returning results to host memory.
//
// A depth array is 4 bytes per vertex, but a traversal of L levels only needs
// depths below L: when L < 15 (255, 65535) the depths travel over PCIe as 4
// bits (1 byte, 2 bytes) per vertex, sentinel all ones for unreached, in chunks
// whose host-side widening to uint32 (host_cpu.hpp, OpenMP threads) overlaps the copy
// of the next chunk.  The pack kernel also checks every depth against the
// width, so a wrong level count can only cost a plain copy, never a wrong
// result; a caller may therefore enqueue the packing behind a traversal whose
// level count it does not know yet (beginDepths) and widen after one wait.
#include <omp.h>

#include <algorithm>
#include <cstring>

#include "bfs.hpp"
#include "host_copy.hpp"
#include "host_cpu.hpp"

namespace gb {
namespace {

constexpr uint64_t kPackChunk = 1u << 20;    // vertices per pipelined chunk (a multiple of 32)
constexpr uint64_t kOneThread = 1u << 16;    // up to this many depths one thread widens: an OpenMP region costs more

int hostThreads(int most) { return std::max(1, std::min(most, omp_get_max_threads())); }

// Eight depths per thread and step: two 16-byte loads (where d is aligned to
// them; a batch's rows need not be), one store of 4, 8 or 16 bytes.  FMT 0: two
// depths per byte, low nibble first; 1: a byte; 2: two bytes.  The last group
// is filled up with the sentinel (out has room for it).
template <int FMT>
__global__ void packDepthsKernel(const uint32_t* d, uint64_t count, uint8_t* out, uint64_t pitch, unsigned* overflow) {
    d += blockIdx.y * count;  // a row per y, `pitch` bytes apart when packed
    out += blockIdx.y * pitch;
    constexpr uint32_t kBits = FMT == 0 ? 4 : FMT == 1 ? 8 : 16, kSentinel = (1u << kBits) - 1u;
    const bool aligned = (reinterpret_cast<uintptr_t>(d) & 15) == 0;
    bool bad = false;
    const uint64_t groups = (count + 7) / 8;
    for (uint64_t g = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; g < groups; g += (uint64_t)gridDim.x * blockDim.x) {
        uint32_t v[8];
        if (aligned && 8 * g + 8 <= count) {
            const uint4 a = reinterpret_cast<const uint4*>(d)[2 * g], b = reinterpret_cast<const uint4*>(d)[2 * g + 1];
            v[0] = a.x; v[1] = a.y; v[2] = a.z; v[3] = a.w;
            v[4] = b.x; v[5] = b.y; v[6] = b.z; v[7] = b.w;
        } else {
#pragma unroll
            for (int i = 0; i < 8; ++i) v[i] = 8 * g + i < count ? d[8 * g + i] : kInf;
        }
        uint32_t w[FMT == 0 ? 1 : FMT == 1 ? 2 : 4] = {};
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            bad |= v[i] != kInf && v[i] >= kSentinel;
            w[i * kBits / 32] |= (v[i] & kSentinel) << (i * kBits % 32);  // infinity ends as the sentinel
        }
        if (FMT == 0) reinterpret_cast<uint32_t*>(out)[g] = w[0];
        else if (FMT == 1) reinterpret_cast<uint2*>(out)[g] = make_uint2(w[0], w[1]);
        else reinterpret_cast<uint4*>(out)[g] = make_uint4(w[0], w[1], w[2], w[3]);
    }
    if (__syncthreads_or(bad) && threadIdx.x == 0) *overflow = 1u;  // may be pinned memory
}

}  // namespace

void widenPacked(int fmt, const uint8_t* in, uint64_t count, uint32_t* out) {
    if (count <= kOneThread) {
        widenRange(fmt, in, 0, count, out);
        return;
    }
    const int threads = hostThreads(16);
    const uint64_t step = ((count + threads - 1) / threads + 31) / 32 * 32;
#pragma omp parallel for num_threads(threads) schedule(static)
    for (int t = 0; t < threads; ++t) {
        const uint64_t lo = std::min(count, (uint64_t)t * step), hi = std::min(count, lo + step);
        if (lo < hi) widenRange(fmt, in, lo, hi, out);
    }
}

void widenRows(int fmt, const uint8_t* in, uint64_t pitch, uint32_t rows, uint64_t count, uint32_t* out, uint64_t stride) {
    if (rows == 1 || stride == 0 || rows * count <= kOneThread) {  // stride 0: one row after the other, the last stays
        for (uint32_t r = 0; r < rows; ++r) widenPacked(fmt, in + r * pitch, count, out + r * stride);
        return;
    }
    constexpr uint64_t kPiece = 1u << 14;  // a multiple of 32
    const uint64_t per = (count + kPiece - 1) / kPiece;
#pragma omp parallel for num_threads(hostThreads(16)) schedule(static)
    for (uint64_t t = 0; t < rows * per; ++t) {
        const uint64_t r = t / per, lo = t % per * kPiece;
        widenRange(fmt, in + r * pitch, lo, std::min(count, lo + kPiece), out + r * stride);
    }
}

int packFormat(uint32_t levels) {
    if (levels < 15) return 0;
    if (levels < 255) return 1;
    if (levels < 65535) return 2;
    return -1;
}

uint64_t packedBytes(int fmt, uint64_t count) {
    return fmt == 0 ? (count + 1) / 2 : fmt == 1 ? count : 2 * count;
}

void enqueuePack(int fmt, const uint32_t* d, uint64_t count, uint8_t* dev, unsigned* overflow, cudaStream_t st,
                 uint32_t rows, uint64_t pitch) {
    const uint32_t blocks = (uint32_t)std::max<uint64_t>(1, std::min<uint64_t>((count / 8 + 255) / 256, (uint64_t)deviceSmCount() * 8));
    const dim3 grid(blocks, rows);
    if (fmt == 0) packDepthsKernel<0><<<grid, 256, 0, st>>>(d, count, dev, pitch, overflow);
    else if (fmt == 1) packDepthsKernel<1><<<grid, 256, 0, st>>>(d, count, dev, pitch, overflow);
    else packDepthsKernel<2><<<grid, 256, 0, st>>>(d, count, dev, pitch, overflow);
    GB_LAUNCH_CHECK();
}

static void addPackEvent(gb_bfs* h) {
    cudaEvent_t e;
    GB_CUDA(cudaEventCreateWithFlags(&e, cudaEventDisableTiming));
    h->packEv.push_back(e);
}

void beginDepths(gb_bfs* h, const uint32_t* d, uint64_t count, uint32_t levels, DepthReturn& r) {
    cudaStream_t st = h->stream.s;
    r.d = d;
    r.count = count;
    r.fmt = packFormat(levels);
    if (r.fmt < 0) return;
    const uint64_t bytes = packedBytes(r.fmt, count);
    h->packHost.ensure(count <= kSmallDepths ? bytes + 16 : bytes);
    h->packFlagHost.ensure(1);
    if (count <= kSmallDepths) {
        *h->packFlagHost.p = 0;
        enqueuePack(r.fmt, d, count, h->packHost.p, h->packFlagHost.p, st);
        while (h->packEv.empty()) addPackEvent(h);
        GB_CUDA(cudaEventRecord(h->packEv[0], st));
        return;
    }
    h->packDev.ensure(bytes + 16);
    if (!h->packFlag.get()) {  // zero but after an overflow, which endDepths clears again
        h->packFlag.ensure(1);
        GB_CUDA(cudaMemsetAsync(h->packFlag.get(), 0, 4, st));
    }
    enqueuePack(r.fmt, d, count, h->packDev.get(), h->packFlag.get(), st);
    GB_CUDA(cudaMemcpyAsync(h->packFlagHost.p, h->packFlag.get(), 4, cudaMemcpyDeviceToHost, st));
    const uint64_t chunks = (count + kPackChunk - 1) / kPackChunk;
    while (h->packEv.size() < chunks) addPackEvent(h);
    for (uint64_t c = 0; c < chunks; ++c) {
        const uint64_t lo = packedBytes(r.fmt, c * kPackChunk), hi = packedBytes(r.fmt, std::min(count, (c + 1) * kPackChunk));
        GB_CUDA(cudaMemcpyAsync(h->packHost.p + lo, h->packDev.get() + lo, hi - lo, cudaMemcpyDeviceToHost, st));
        GB_CUDA(cudaEventRecord(h->packEv[c], st));
    }
}

void waitDepths(gb_bfs* h, const DepthReturn& r) {
    if (r.fmt < 0) GB_CUDA(cudaStreamSynchronize(h->stream.s));
    else GB_CUDA(cudaEventSynchronize(h->packEv[0]));
}

void endDepths(gb_bfs* h, const DepthReturn& r, uint32_t levels, uint32_t* out) {
    if (r.fmt >= 0) {
        const uint64_t chunks = (r.count + kPackChunk - 1) / kPackChunk;
        for (uint64_t c = 0; c < chunks; ++c) {
            GB_CUDA(cudaEventSynchronize(h->packEv[c]));
            if (*h->packFlagHost.p) break;  // copied ahead of the chunks
            const uint64_t lo = c * kPackChunk, len = std::min(kPackChunk, r.count - lo);
            widenPacked(r.fmt, h->packHost.p + packedBytes(r.fmt, lo), len, out + lo);
        }
        if (*h->packFlagHost.p == 0) return;
        GB_CUDA(cudaStreamSynchronize(h->stream.s));
        if (r.count > kSmallDepths) GB_CUDA(cudaMemsetAsync(h->packFlag.get(), 0, 4, h->stream.s));
        // the guessed width was too narrow: once more with the level count, which fits
        if (packFormat(levels) > r.fmt) {
            DepthReturn again;
            beginDepths(h, r.d, r.count, levels, again);
            endDepths(h, again, levels, out);
            return;
        }
    }
    h->staged.run(r.d, r.count * 4, out, h->stream.s);
}

void copyDepthsToHost(gb_bfs* h, const uint32_t* d, uint64_t count, uint32_t* out, uint32_t levels) {
    DepthReturn r;
    beginDepths(h, d, count, levels, r);
    endDepths(h, r, levels, out);
}

void StagedCopy::run(const void* dev, size_t bytes, void* out, cudaStream_t st) {
    constexpr size_t kChunk = 1u << 19;
    const size_t chunks = (bytes + kChunk - 1) / kChunk;
    hold_.ensure(1);
    HostPinned<uint8_t> ring;
    ring.ensure(std::min(bytes, kSlots * kChunk));
    for (cudaEvent_t& e : ev_)
        if (!e) GB_CUDA(cudaEventCreateWithFlags(&e, cudaEventDisableTiming));
    const uint8_t* src = static_cast<const uint8_t*>(dev);
    uint8_t* dst = static_cast<uint8_t*>(out);
    auto length = [&](size_t c) { return std::min(kChunk, bytes - c * kChunk); };
    auto enqueue = [&](size_t c) {
        GB_CUDA(cudaMemcpyAsync(ring.p + c % kSlots * kChunk, src + c * kChunk, length(c), cudaMemcpyDeviceToHost, st));
        GB_CUDA(cudaEventRecord(ev_[c % kSlots], st));
    };
    for (size_t c = 0; c < std::min<size_t>(chunks, kSlots); ++c) enqueue(c);
    const int threads = hostThreads(8);
    for (size_t c = 0; c < chunks; ++c) {
        GB_CUDA(cudaEventSynchronize(ev_[c % kSlots]));
        const uint8_t* from = ring.p + c % kSlots * kChunk;
        uint8_t* to = dst + c * kChunk;
        const size_t len = length(c);
        constexpr size_t kPiece = 1 << 15;
        const int pieces = (int)((len + kPiece - 1) / kPiece);
#pragma omp parallel for num_threads(threads) schedule(static) if (pieces > 3)
        for (int p = 0; p < pieces; ++p)
            std::memcpy(to + p * kPiece, from + p * kPiece, std::min(kPiece, len - p * kPiece));
        if (c + kSlots < chunks) enqueue(c + kSlots);
    }
}

}  // namespace gb
