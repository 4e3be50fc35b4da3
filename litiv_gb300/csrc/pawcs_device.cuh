// Device helpers shared by the one- and three-channel PAWCS kernels (pawcs_kernels.cu,
// pawcs3_kernels.cu): the reference's tables, draws, word weights, thresholds and LBSP.
#pragma once
#include <cuda_runtime.h>
#include <float.h>
#include <stdint.h>

#include "lbsp_device.cuh"
#include "pawcs_internal.h"

namespace lvbgs {

// sampling weights (opencv.hpp:915-923)
static __constant__ int pw_pat7[49] = {2, 4, 6, 7, 6, 4, 2, 4, 8, 12, 14, 12, 8, 4, 6, 12, 21, 25, 21, 12, 6, 7, 14, 25, 28,
                                25, 14, 7, 6, 12, 21, 25, 21, 12, 6, 4, 8, 12, 14, 12, 8, 4, 2, 4, 6, 7, 6, 4, 2};

constexpr float kTLower = 1.0f, kTUpper = 256.0f, kTIncr = 0.5f, kTDecr = 0.25f;
constexpr float kVIncr = 1.0f, kVDecr = 0.1f, kRVar = 0.01f, kUnstRatio = 0.1f, kUnstR = 3.0f;
constexpr int kBootWin = kPwBootWin;

__device__ __forceinline__ int pw_stream_by_tile(const PwParams& P, int t) {
    int lo = 0, hi = P.nStreams - 1;
    while (lo < hi) {
        const int mid = (lo + hi + 1) >> 1;
        if (P.streams[mid].sd.tileBase <= t) lo = mid;
        else hi = mid - 1;
    }
    return lo;
}
__device__ __forceinline__ int pw_stream_by_row(const PwParams& P, int r) {
    int lo = 0, hi = P.nStreams - 1;
    while (lo < hi) {
        const int mid = (lo + hi + 1) >> 1;
        if (P.streams[mid].sd.rowBase <= r) lo = mid;
        else hi = mid - 1;
    }
    return lo;
}

// one rand() of the reference: draw k of pixel px in frame f
__device__ __forceinline__ uint32_t pw_draw(unsigned long long seed, uint32_t f, uint32_t px, uint32_t k) {
    uint32_t c[4] = {k >> 2, px, f, 0u};
    philox4x32_10(c, (uint32_t)seed, (uint32_t)(seed >> 32));
    const uint32_t lo = (k & 1u) ? c[1] : c[0], hi = (k & 1u) ? c[3] : c[2];  // registers, not an indexed array
    return ((k & 2u) ? hi : lo) & 0x7fffffffu;
}
// draw % m for the reference's size_t moduli (rand() < 2^31, so a modulus above 2^32 leaves it as is)
__device__ __forceinline__ uint32_t pw_mod(uint32_t r, unsigned long long m) {
    return m > 0xffffffffull ? r : r % (uint32_t)m;
}

// GetLocalWordWeight (:1596-1598): (float)occ / (float)((last-first) + (t-last)*2 + offset). The denominator
// nearly always fits 32 bits, whose conversion is the same number and a quarter of the work.
__device__ __forceinline__ float pw_weight(uint32_t occ, uint32_t first, uint32_t last, uint32_t t,
                                           unsigned long long off) {
    const unsigned long long den = (unsigned long long)(last - first) + (unsigned long long)(t - last) * 2ull + off;
    const float fd = (den >> 32) ? (float)den : (float)(uint32_t)den;
    return (float)occ / fd;
}

struct PwThr {
    uint32_t color, desc;
};

// (size_t)(sqrt(R) * m) as the reference evaluates it: an unqualified sqrt of a float there is the
// C library's double sqrt, and the product is taken in double (:119, :267, :663, :993). For a float R
// and a small integer m that truncation equals the exact floor(m * sqrt(R)), the largest k with
// k^2 <= m^2 R (a float R lies at least 2^-24/m^2 in relative terms from any such boundary, far more
// than the two double roundings move the product). A float candidate is corrected by one with an
// exact comparison: hi + lo = m^2 R exactly (two-product), k^2 exact in float below 2^24.
__device__ __forceinline__ uint32_t pw_sqrt_floor(float R, uint32_t m) {
    uint32_t k = (uint32_t)(__fsqrt_rn(R) * (float)m);
    const float mm = (float)(m * m);
    if (m * m >= (1u << 24) || k >= 4095u) return (uint32_t)(__dsqrt_rn((double)R) * (double)m);
    const float hi = mm * R, lo = __fmaf_rn(mm, R, -hi);
    const auto le = [&](uint32_t kk) {  // kk^2 <= m^2 R
        const float k2 = (float)(kk * kk);
        return k2 < hi || (k2 == hi && lo >= 0.0f);
    };
    if (!le(k)) --k;
    else if (le(k + 1)) ++k;
    return k;
}
// nCurrColorDistThreshold / nCurrDescDistThreshold of one channel (:633-634)
__device__ __forceinline__ PwThr pw_thresholds(float R, uint32_t unstable, uint32_t minColor, uint32_t descOff) {
    PwThr t;
    t.color = pw_sqrt_floor(R, minColor) / 2u;
    const unsigned long long sh = (unsigned long long)floorf(R + 0.5f);
    const unsigned long long d = (sh < 64 ? (1ull << sh) : 0ull) + descOff + (unsigned long long)unstable * descOff;
    t.desc = d > 0xffffffffull ? 0xffffffffu : (uint32_t)d;
    return t;
}

__device__ __forceinline__ uint32_t pw_absdiff(uint32_t a, uint32_t b) { return a > b ? a - b : b - a; }

// the 16 LBSP taps of channel c at pixel (x, y) of a dense C-channel image, four to a word (lbsp_thr's packing)
template <int C>
__device__ __forceinline__ void pw_taps(const uint8_t* img, int W, int x, int y, int c, uint32_t (&v)[4]) {
    const uint8_t* base = img + ((size_t)y * W + x) * C + c;
#pragma unroll
    for (int j = 0; j < 4; ++j) {
        uint32_t w = 0;
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const int n = 4 * j + i;
            w |= (uint32_t)__ldg(base + (lbsp_dy(n) * W + lbsp_dx(n)) * C) << (8 * i);
        }
        v[j] = w;
    }
}

// rolling-average factors of frame f (:570-573)
__device__ __forceinline__ void pw_factors(unsigned long long f, int nmv, float* fLT, float* fST) {
    const int boot = f <= (unsigned long long)kBootWin;
    const unsigned long long nlt = boot ? (unsigned long long)(nmv / 2) : (unsigned long long)nmv, nst = nlt / 4;
    *fLT = 1.0f / (float)(f < nlt ? f : nlt);
    *fST = 1.0f / (float)(f < nst ? f : nst);
}

__device__ __forceinline__ size_t pw_slot(const PawcsDev& S, int buf, int j, int p) {
    return ((size_t)buf * S.L + j) * S.sd.npx + p;
}

// one local word of a one-channel dictionary
struct PwWord {
    uint32_t occ, first, last, desc, col;
};
__device__ __forceinline__ PwWord pw_load(const PawcsDev& S, size_t slot) {
    const uint4 v = S.wA[slot];
    return {v.x, v.y, v.z, v.w & 0xffffu, v.w >> 16};
}
__device__ __forceinline__ void pw_store(const PawcsDev& S, size_t slot, const PwWord& w) {
    S.wA[slot] = make_uint4(w.occ, w.first, w.last, w.desc | (w.col << 16));
}
// one local word of a three-channel dictionary
struct Pw3Word {
    uint32_t col;   // packed colour
    uint32_t d01;   // descriptors of channels 0 and 1
    uint32_t d2;    // descriptor of channel 2
    uint32_t occ, first, last;
};
struct Pw3Raw {  // as stored
    uint4 a;
    uint32_t last, c2;
};
__device__ __forceinline__ Pw3Raw pw3_fetch(const PawcsDev& S, size_t slot) {
    return {S.wA[slot], S.wLast[slot], S.wC2[slot]};
}
__device__ __forceinline__ Pw3Word pw3_unpack(const Pw3Raw& r) {
    return {(r.a.y >> 16) | (r.c2 << 16), r.a.x, r.a.y & 0xffffu, r.a.z, r.a.w, r.last};
}
__device__ __forceinline__ Pw3Word pw3_load(const PawcsDev& S, int buf, int j, int p) {
    return pw3_unpack(pw3_fetch(S, pw_slot(S, buf, j, p)));
}
__device__ __forceinline__ void pw3_put(const PawcsDev& S, size_t slot, const Pw3Word& w) {
    S.wA[slot] = make_uint4(w.d01, (w.d2 & 0xffffu) | (w.col << 16), w.occ, w.first);
    S.wLast[slot] = w.last;
    S.wC2[slot] = (uint8_t)(w.col >> 16);
}
__device__ __forceinline__ void pw3_store(const PawcsDev& S, int buf, int j, int p, const Pw3Word& w) {
    pw3_put(S, pw_slot(S, buf, j, p), w);
}

// Appends the pixels q of a block of 256 threads (every thread calls it) to a list, one atomic a block.
__device__ __forceinline__ void pw_list_append(uint32_t* list, unsigned int* count, bool want, int q) {
    __shared__ unsigned int off[8], base;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const unsigned m = __ballot_sync(0xffffffffu, want);
    if (lane == 0) off[warp] = (unsigned)__popc(m);
    __syncthreads();
    if (threadIdx.x == 0) {
        unsigned int all = 0;
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            const unsigned int c = off[i];
            off[i] = all;
            all += c;
        }
        base = all ? atomicAdd(count, all) : 0u;
    }
    __syncthreads();
    if (want) list[base + off[warp] + (unsigned)__popc(m & ((1u << lane) - 1u))] = (uint32_t)q;
}
// The place of a thread in a list of n pixels: as few pixels a warp as fill the machine (warps: resident at once),
// because the updaters' loops diverge and a warp serves its lanes' paths one after the other; -1: none.
__device__ __forceinline__ int pw_list_index(unsigned int n, unsigned int warps) {
    warps = min(warps, gridDim.x * (blockDim.x / 32u));  // the grid has a thread for every pixel, so 32 a warp serve all
    const unsigned int k = min(32u, (n + warps - 1u) / warps), lane = threadIdx.x & 31u;
    const unsigned int i = (blockIdx.x * (blockDim.x / 32u) + threadIdx.x / 32u) * k + lane;
    return lane < k && i < n ? (int)i : -1;
}

// End of a fixed-point round, called by every thread of the dirty pass: counts the pixels to rerun; the block
// that finishes last closes the round. No dirty pixel means the fixed point is reached: its round count and
// flag are set, here for the rounds and the tail enqueued after this one, and in host memory.
// list: the dirty pixels (q), any order, their count in PWF_NDIRTY; null: not listed.
__device__ __forceinline__ void pw_round_end(const PwParams& P, bool dirty, uint32_t* list = nullptr, int q = 0) {
    if (list) {
        pw_list_append(list, &P.flags[PWF_DIRTY], dirty, q);
        __syncthreads();
        if (threadIdx.x != 0) return;
    } else {
        const int any = __syncthreads_count(dirty);
        if (threadIdx.x != 0) return;
        if (any) atomicAdd(&P.flags[PWF_DIRTY], (unsigned)any);
    }
    __threadfence();
    if (atomicAdd(&P.flags[PWF_DONE], 1u) != gridDim.x - 1u) return;
    P.flags[PWF_DONE] = 0u;
    const unsigned int total = atomicExch(&P.flags[PWF_DIRTY], 0u);
    P.flags[PWF_NDIRTY] = total;
    if (total == 0u) {
        P.flags[PWF_ROUNDS] = (unsigned)P.round + 1u;
        P.hflags[PWF_ROUNDS] = (unsigned)P.round + 1u;
        P.hflags[PWF_CONV] = 1u;
        __threadfence();
        P.flags[PWF_CONV] = 1u;
    }
}

}  // namespace lvbgs

namespace lvbgs {

// ---- three channels: packed colours (c0 | c1 << 8 | c2 << 16), descriptors (d0 | d1 << 16, d2) ----

// nCurrColorDistThreshold / nCurrDescDistThreshold of three channels (:1011-1012)
__device__ __forceinline__ PwThr pw3_thresholds(float R, uint32_t unstable, uint32_t minColor, uint32_t descOff) {
    PwThr t;
    t.color = pw_sqrt_floor(R, minColor) * 3u;
    const unsigned long long sh = (unsigned long long)floorf(R + 0.5f);
    const unsigned long long d = ((sh < 64 ? (1ull << sh) : 0ull) + descOff + (unsigned long long)unstable * descOff) * 3ull;
    t.desc = d > 0xffffffffull ? 0xffffffffu : (uint32_t)d;
    return t;
}
__device__ __forceinline__ uint32_t pw3_ch(uint32_t c, int k) { return (c >> (8 * k)) & 255u; }
// lv::L1dist of two three-byte colours (math.hpp:226-250): the reference accumulates the sum in
// the type of L1dist(uchar, uchar), unsigned char, so it wraps modulo 256 (every three-channel colour
// L1 of PAWCS goes through it, directly or through cmixdist)
__device__ __forceinline__ uint32_t pw3_l1(uint32_t a, uint32_t b) {
    return __dp4a(__vabsdiffu4(a, b), 0x00010101u, 0u) & 0xffu;
}
// lv::cdist<3> of two byte colours (math.hpp:474-496): sqrt of the colour distortion, 0 for a grey
// pair or identical colours: floor(sqrt(|a|^2 - floor((a.b)^2 / |b|^2))). The products are byte dot products;
// the quotient is at most |a|^2 < 2^18 (Cauchy-Schwarz), so a single-precision estimate is off by less than
// one and the remainder corrects it (it lies within one divisor of its range, so 32-bit arithmetic holds it);
// the root of an integer below 2^18 likewise. 64-bit division and the rounded square root cost ~100
// instructions for each word, of ~250 in all.
__device__ __forceinline__ uint32_t pw3_cdist(uint32_t a, uint32_t b) {
    const bool grey = a == (a & 0xffu) * 0x010101u && b == (b & 0xffu) * 0x010101u;
    if (grey || a == b) return 0u;
    const uint32_t cs = __dp4a(a, a, 0u), bs = max(__dp4a(b, b, 0u), 1u), mix = __dp4a(a, b, 0u);
    const float fm = (float)mix;
    uint32_t q = (uint32_t)(fm * __fdividef(fm, (float)bs));
    const int r = (int)(mix * mix - q * bs);
    if (r < 0) --q;
    else if (r >= (int)bs) ++q;
    const uint32_t n = cs - q;
    float root;
    asm("sqrt.approx.f32 %0, %1;" : "=f"(root) : "f"((float)n));
    uint32_t k = (uint32_t)root;
    if (k * k > n) --k;
    else if ((k + 1u) * (k + 1u) <= n) ++k;
    return k;
}
// lv::cmixdist (math.hpp:596-605)
__device__ __forceinline__ uint32_t pw3_cmix(uint32_t a, uint32_t b) { return pw3_l1(a, b) / 2u + pw3_cdist(a, b) * 4u; }
__device__ __forceinline__ uint32_t pw3_hd(uint32_t a01, uint32_t a2, uint32_t b01, uint32_t b2) {
    return (uint32_t)__popc(a01 ^ b01) + (uint32_t)__popc((a2 ^ b2) & 0xffffu);
}
__device__ __forceinline__ uint32_t pw3_color(const uint8_t* img, int p) {
    const uint8_t* q = img + (size_t)p * 3;
    return (uint32_t)q[0] | ((uint32_t)q[1] << 8) | ((uint32_t)q[2] << 16);
}

}  // namespace lvbgs
