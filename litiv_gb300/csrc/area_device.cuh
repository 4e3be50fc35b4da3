// cv::resize(INTER_AREA) of an 8-bit frame by groups of eight lanes, shared by the SuBSENSE and PAWCS kernels.
#pragma once
#include <stdint.h>

#include "lvbgs_internal.h"

namespace lvbgs {

// One output pixel (dx, dy) of the frame's area resampling, every channel, by a group of eight lanes (one
// source row per lane and step); each lane of the group gets the values. The same numbers as area_resample:
// the block mean where the sides are integral multiples (sums of bytes, exact in any order), else the exact
// area-weighted mean rounded half to even, in 32-bit integers while 255 * W * H fits them. One lane per
// output walked 64 C bytes, 12 us on any frame (100 us on 1279x719, in 64-bit arithmetic). The groups of a
// warp are independent of one another (its shuffles name the group's lanes only).
template <int C>
__device__ __forceinline__ void area_resample_group(const uint8_t* __restrict__ fr, int W, int H, int dW, int dH,
                                                    int dx, int dy, uint32_t (&v)[C]) {
    const int sub = threadIdx.x & 7;
    const unsigned mask = 0xffu << (threadIdx.x & 24);
    const bool whole = W % dW == 0 && H % dH == 0;
    const size_t pitch = (size_t)W * C;
    if (whole) {
        const int sx = W / dW, sy = H / dH;
        uint32_t sum[C];
#pragma unroll
        for (int c = 0; c < C; ++c) sum[c] = 0u;
        for (int j = sub; j < sy; j += 8) {
            const uint8_t* row = fr + (size_t)(dy * sy + j) * pitch + (size_t)dx * sx * C;
            if (sx == 8 && (pitch & 7) == 0 && ((uintptr_t)fr & 7) == 0) {
                // 8 C bytes at an 8-byte boundary: byte b of the row belongs to channel b % C
                uint2 w[C];
#pragma unroll
                for (int i = 0; i < C; ++i) w[i] = __ldg((const uint2*)row + i);
#pragma unroll
                for (int i = 0; i < 2 * C; ++i) {
                    const uint32_t word = (i & 1) ? w[i / 2].y : w[i / 2].x;
#pragma unroll
                    for (int c = 0; c < C; ++c) {
                        uint32_t sel = 0u;
#pragma unroll
                        for (int b = 0; b < 4; ++b) sel |= ((4 * i + b) % C == c) ? 1u << (8 * b) : 0u;
                        sum[c] = __dp4a(word, sel, sum[c]);
                    }
                }
            } else {
                for (int i = 0; i < sx; ++i)
#pragma unroll
                    for (int c = 0; c < C; ++c) sum[c] += __ldg(row + i * C + c);
            }
        }
#pragma unroll
        for (int c = 0; c < C; ++c) {
#pragma unroll
            for (int o = 4; o > 0; o >>= 1) sum[c] += __shfl_xor_sync(mask, sum[c], o, 8);
            const int r = __float2int_rn((float)(int)sum[c] * (1.f / (float)(sx * sy)));
            v[c] = (uint32_t)(r < 0 ? 0 : r > 255 ? 255 : r);
        }
        return;
    }
    // in units of 1/dW (1/dH) a source pixel i spans [i dW, (i+1) dW), the output pixel [x0, x1)
    const long long x0 = (long long)dx * W, x1 = x0 + W, y0 = (long long)dy * H, y1 = y0 + H;
    const int i0 = (int)(x0 / dW), i1 = (int)((x1 + dW - 1) / dW);
    const int j0 = (int)(y0 / dH), j1 = (int)((y1 + dH - 1) / dH);
    const bool narrow = 255ull * (unsigned long long)W * (unsigned long long)H < (1ull << 31);
    unsigned long long num[C];
#pragma unroll
    for (int c = 0; c < C; ++c) num[c] = 0ull;
    for (int j = j0 + sub; j < j1; j += 8) {
        const long long a = (long long)j * dH, b = a + dH;
        const uint32_t oy = (uint32_t)((b < y1 ? b : y1) - (a > y0 ? a : y0));
        unsigned long long line[C];
#pragma unroll
        for (int c = 0; c < C; ++c) line[c] = 0ull;
        const uint8_t* row = fr + (size_t)j * pitch;
        for (int i = i0; i < i1; ++i) {
            const long long l = (long long)i * dW, r = l + dW;
            const uint32_t ox = (uint32_t)((r < x1 ? r : x1) - (l > x0 ? l : x0));
#pragma unroll
            for (int c = 0; c < C; ++c) {
                const uint32_t s = __ldg(row + (size_t)i * C + c);
                line[c] += narrow ? (unsigned long long)(ox * s) : (unsigned long long)ox * s;
            }
        }
#pragma unroll
        for (int c = 0; c < C; ++c) num[c] += line[c] * oy;
    }
#pragma unroll
    for (int c = 0; c < C; ++c) {
#pragma unroll
        for (int o = 4; o > 0; o >>= 1) num[c] += __shfl_xor_sync(mask, num[c], o, 8);
        if (narrow) {
            const uint32_t den = (uint32_t)W * (uint32_t)H, n = (uint32_t)num[c];
            uint32_t q = n / den;
            const uint32_t r2 = (n - q * den) * 2u;
            if (r2 > den || (r2 == den && (q & 1u))) ++q;
            v[c] = q > 255u ? 255u : q;
        } else {
            v[c] = area_round_ties_even(num[c], (unsigned long long)W * (unsigned long long)H);
        }
    }
}

}  // namespace lvbgs
