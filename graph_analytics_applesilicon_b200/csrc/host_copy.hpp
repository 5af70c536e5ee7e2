// host_copy.hpp -- device memory to the caller's pageable memory.
//
// A plain device-to-host copy into pageable memory is staged by the driver on
// one thread (6-7 GB/s measured, 67 us for 400 KB).  Here the chunks land in a
// ring of pinned buffers and host threads move them on while the next chunks
// cross PCIe.
#pragma once

#include "common.cuh"

namespace gb {

class StagedCopy {
public:
    ~StagedCopy() {
        for (cudaEvent_t e : ev_)
            if (e) cudaEventDestroy(e);
    }
    // Copies bytes from dev to out, ordered after the work on st; returns when out is complete.
    void run(const void* dev, size_t bytes, void* out, cudaStream_t st);

private:
    static constexpr int kSlots = 2;
    HostPinned<uint8_t> hold_;  // keeps the pool while this object lives; the ring itself is taken for a call
    cudaEvent_t ev_[kSlots] = {};
};

}  // namespace gb
