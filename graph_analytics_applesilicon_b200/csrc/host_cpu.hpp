// host_cpu.hpp -- what depends on the host's processor: packed depths to uint32,
// with SSE2 where there is it, else one depth at a time, and a pause while polling.
#pragma once

#ifdef __SSE2__
#include <emmintrin.h>
#endif

#include <cstdint>
#include <cstring>

namespace gb {

constexpr uint32_t kWideInf = 0xFFFFFFFFu;  // an unreached vertex's depth

// A pause between two looks at a word that a device will write.
inline void cpuPause() {
#ifdef __SSE2__
    _mm_pause();
#elif defined(__aarch64__)
    asm volatile("yield" ::: "memory");
#else
    asm volatile("" ::: "memory");
#endif
}

inline uint32_t widenOne(int fmt, const uint8_t* in, uint64_t i) {
    if (fmt == 0) {
        const uint32_t v = (in[i / 2] >> (4 * (i & 1))) & 15u;
        return v == 15u ? kWideInf : v;
    }
    if (fmt == 1) return in[i] == 0xFFu ? kWideInf : in[i];
    uint16_t v;
    std::memcpy(&v, in + 2 * i, 2);
    return v == 0xFFFFu ? kWideInf : v;
}

#ifdef __SSE2__
inline void store4(uint32_t* o, __m128i x) { _mm_storeu_si128(reinterpret_cast<__m128i*>(o), x); }

// Sixteen bytes b (sentinel 0xFF) to sixteen uint32 (sentinel all ones): the
// sentinel's compare mask is the high part in both unpacking steps.
inline void widen16(__m128i b, uint32_t* o) {
    const __m128i m = _mm_cmpeq_epi8(b, _mm_set1_epi8(-1));
    const __m128i lo = _mm_unpacklo_epi8(b, m), hi = _mm_unpackhi_epi8(b, m);
    const __m128i ml = _mm_unpacklo_epi8(m, m), mh = _mm_unpackhi_epi8(m, m);
    store4(o, _mm_unpacklo_epi16(lo, ml));
    store4(o + 4, _mm_unpackhi_epi16(lo, ml));
    store4(o + 8, _mm_unpacklo_epi16(hi, mh));
    store4(o + 12, _mm_unpackhi_epi16(hi, mh));
}
#endif

// Depths [lo, hi) of a packed array; lo is a multiple of 32.  Plain stores: with
// stores that bypass the cache the 16.8 MB of R-MAT 22 take 358 us a call, so 307.
// Not inlined into its callers' loops: 65,536 depths so cost 4 us less a call.
__attribute__((noinline)) inline void widenRange(int fmt, const uint8_t* in, uint64_t lo, uint64_t hi, uint32_t* out) {
    uint64_t i = lo;
#ifdef __SSE2__
    if (fmt == 0) {
        const __m128i low = _mm_set1_epi8(15);
        for (; i + 32 <= hi; i += 32) {
            const __m128i x = _mm_loadu_si128(reinterpret_cast<const __m128i*>(in + i / 2));
            const __m128i a = _mm_and_si128(x, low), b = _mm_and_si128(_mm_srli_epi16(x, 4), low);
            const __m128i y0 = _mm_unpacklo_epi8(a, b), y1 = _mm_unpackhi_epi8(a, b);
            widen16(_mm_or_si128(y0, _mm_cmpeq_epi8(y0, low)), out + i);
            widen16(_mm_or_si128(y1, _mm_cmpeq_epi8(y1, low)), out + i + 16);
        }
    } else if (fmt == 1) {
        for (; i + 16 <= hi; i += 16)
            widen16(_mm_loadu_si128(reinterpret_cast<const __m128i*>(in + i)), out + i);
    } else {
        const __m128i ones = _mm_set1_epi16(-1);
        for (; i + 8 <= hi; i += 8) {
            const __m128i x = _mm_loadu_si128(reinterpret_cast<const __m128i*>(in + 2 * i));
            const __m128i m = _mm_cmpeq_epi16(x, ones);
            store4(out + i, _mm_unpacklo_epi16(x, m));
            store4(out + i + 4, _mm_unpackhi_epi16(x, m));
        }
    }
#endif
    for (; i < hi; ++i) out[i] = widenOne(fmt, in, i);
}

}  // namespace gb
