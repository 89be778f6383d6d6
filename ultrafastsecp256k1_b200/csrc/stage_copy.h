// Copies into pinned staging memory that a host -> device copy reads next.
//
// With ordinary stores the staged lines are left modified in the caches of the
// cores that packed them, and the copy engine's reads have to snoop them out:
// 2 MB packed by four threads took 60 us to pack and 200 us to copy in (48 us
// from memory).  Non-temporal stores go to memory: 33 + 48 us, and a single
// thread packs 1.3x faster as well (no line is read before it is overwritten).
#pragma once
#include <stddef.h>
#include <stdint.h>
#include <string.h>

#if defined(__SSE2__)
#include <emmintrin.h>
#endif

namespace uf {

// Orders this thread's stage_copy stores before the copy that reads them is
// enqueued (by this thread, or by another that this one signals afterwards).
inline void stage_fence() {
#if defined(__SSE2__)
    _mm_sfence();
#endif
}

inline void stage_copy(void* dst, const void* src, size_t n) {
#if defined(__SSE2__)
    constexpr size_t kSmall = 256;   // below this, the unaligned ends cost more
    if (n >= kSmall) {
        uint8_t* d = (uint8_t*)dst;
        const uint8_t* s = (const uint8_t*)src;
        const size_t head = (size_t)(-(uintptr_t)d & 63u);
        if (head) memcpy(d, s, head);
        d += head;
        s += head;
        n -= head;
        for (; n >= 64; n -= 64, d += 64, s += 64) {
            const __m128i* a = (const __m128i*)s;
            __m128i* b = (__m128i*)d;
            const __m128i x0 = _mm_loadu_si128(a), x1 = _mm_loadu_si128(a + 1);
            const __m128i x2 = _mm_loadu_si128(a + 2), x3 = _mm_loadu_si128(a + 3);
            _mm_stream_si128(b, x0);
            _mm_stream_si128(b + 1, x1);
            _mm_stream_si128(b + 2, x2);
            _mm_stream_si128(b + 3, x3);
        }
        if (n) memcpy(d, s, n);
        return;
    }
#endif
    memcpy(dst, src, n);
}

// n rows of `width` bytes, `stride` apart in src, to consecutive ones at dst.
inline void stage_rows(uint8_t* dst, const uint8_t* src, size_t width, size_t stride, size_t n) {
#if defined(__SSE2__)
    if (((uintptr_t)dst & 15u) == 0 && (width == 32 || width == 64)) {
        for (size_t i = 0; i < n; ++i, dst += width, src += stride)
            for (size_t q = 0; q < width; q += 16)
                _mm_stream_si128((__m128i*)(dst + q), _mm_loadu_si128((const __m128i*)(src + q)));
        return;
    }
#endif
    for (size_t i = 0; i < n; ++i) memcpy(dst + i * width, src + i * stride, width);
}

}  // namespace uf
