// Bit-sliced counting on words of 32 mask pixels, shared by the SuBSENSE and LOBSTER median kernels.
#pragma once
#include <stdint.h>

namespace lvbgs {

// bit-sliced arithmetic on 32 pixels at once: carry of a full adder
__device__ __forceinline__ uint32_t maj3(uint32_t a, uint32_t b, uint32_t c) { return (a & b) | (a & c) | (b & c); }

// number of set pixels of each pixel's row window [x - r, x + r], r < 2^(HB-1): bit planes h[0..HB-1] of
// word C with its neighbour words L and R
template <int HB>
__device__ __forceinline__ void row_window_planes(uint32_t L, uint32_t C, uint32_t R, int r, uint32_t (&h)[HB]) {
    h[0] = C;
#pragma unroll
    for (int i = 1; i < HB; ++i) h[i] = 0u;
    int d = 1;
    for (; d + 1 <= r; d += 2) {
        const uint32_t a = __funnelshift_r(C, R, d), b = __funnelshift_l(L, C, d);
        const uint32_t e = __funnelshift_r(C, R, d + 1), f = __funnelshift_l(L, C, d + 1);
        const uint32_t s = h[0] ^ a ^ b, c1 = maj3(h[0], a, b);
        h[0] = s ^ e ^ f;
        const uint32_t c2 = maj3(s, e, f);
        uint32_t c = maj3(h[1], c1, c2);
        h[1] ^= c1 ^ c2;
#pragma unroll
        for (int i = 2; i < HB; ++i) {
            const uint32_t t = h[i] & c;
            h[i] ^= c;
            c = t;
        }
    }
    if (d <= r) {
        const uint32_t a = __funnelshift_r(C, R, d), b = __funnelshift_l(L, C, d);
        uint32_t c = maj3(h[0], a, b);
        h[0] ^= a ^ b;
#pragma unroll
        for (int i = 1; i < HB; ++i) {
            const uint32_t t = h[i] & c;
            h[i] ^= c;
            c = t;
        }
    }
}

// a += v: sums of up to 2 HB planes, a row's counts of HB planes
template <int HB>
__device__ __forceinline__ void add_planes(uint32_t (&a)[2 * HB], const uint32_t (&v)[HB]) {
    uint32_t c = 0u;
#pragma unroll
    for (int b = 0; b < HB; ++b) {
        const uint32_t s = a[b] ^ v[b] ^ c;
        c = maj3(a[b], v[b], c);
        a[b] = s;
    }
#pragma unroll
    for (int b = HB; b < 2 * HB; ++b) {
        const uint32_t t = a[b] & c;
        a[b] ^= c;
        c = t;
    }
}

// the pixels whose sum is above `than`, from the lowest bit up
template <int NB>
__device__ __forceinline__ uint32_t planes_above(const uint32_t (&a)[NB], int than) {
    uint32_t m = 0u;
#pragma unroll
    for (int b = 0; b < NB; ++b) m = ((than >> b) & 1) ? (a[b] & m) : (a[b] | m);
    return m;
}

}  // namespace lvbgs
