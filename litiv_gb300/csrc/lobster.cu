// LOBSTER, ViBe and PBAS frame steps for sm_103a (BackgroundSubtractorLOBSTER.cpp:459-581, the
// non-parallel path; BackgroundSubtractorViBe.cpp:77-191; BackgroundSubtractorPBAS.cpp:111-496). The
// kernels are written for LOBSTER and take the algorithm as a template parameter: ViBe evaluates every
// pixel (no ROI), matches colours only, keeps plain colour samples and outputs its raw mask, and its
// neighbour positions are clamped to the frame instead of the LBSP border; PBAS adds a gradient image,
// gradient samples, per-pixel R/T/D maps and a frame-level mean gradient distance, and its neighbour
// update writes the target's own values (self diffusion). The scheme below is the same for all three.
//
// The reference scans the ROI pixels in raster order. A pixel reads its own samples, which an earlier
// pixel's neighbour update may have overwritten in the same frame (:510-512 / :569-574); nothing else
// it reads changes during the frame. Random draws are keyed by (seed, frame, pixel, draw index), so
// they do not depend on the scan order. A frame step therefore
//   1. evaluates every pixel against the frame-start samples (lob_k_eval): decision, samples scanned
//      e, and the model writes it makes (own sample, neighbour target and sample), in an intent word;
//   2. re-evaluates the pixels whose scan read a sample that an earlier neighbour writes, with the samples
//      the raster scan would see (the latest earlier writer of each sample; lob_k_first);
//   3. repeats that for the later pixels whose incoming writes changed, round after round until nothing
//      changes (lob_k_round; the dependencies follow raster order, so this is the raster-order fixed
//      point). Rounds are enqueued ahead; a converged flag makes the rest return;
//   4. commits every sample write in raster order, each pixel gathering the writes aimed at it from
//      its 3x3 neighbourhood (lob_k_commit), then the median blur of the mask (:577-579).
// The writers of a pixel are within one pixel of it: getNeighborPosition_3x3 moves one step and
// clamps into the LBSP border, and ROI pixels lie inside that border.
//
// A scan that ends within a few samples (most of a background) stays with its pixel's lane; a longer one is
// finished by eight lanes, eight samples a step, whose ballots give the samples scanned before the stop, so that
// one long scan does not hold 31 lanes for N steps. The samples of a pixel are one aligned word or word pair
// (load_sample), and a frame's launches are chained (each starts while the one before drains).
#include <cuda_runtime.h>

#include <cmath>
#include <cstring>

#include "bitslice.cuh"
#include "lbsp_device.cuh"
#include "lobster_internal.h"
#include "staging.h"

namespace lvbgs {

namespace {

// 7x7 Gaussian sampling weights (opencv.hpp:915-923)
__constant__ int c_lob_pat7[49] = {2,  4,  6,  7,  6,  4,  2,  4,  8,  12, 14, 12, 8,  4,  6, 12, 21,
                                   25, 21, 12, 6,  7,  14, 25, 28, 25, 14, 7,  6,  12, 21, 25, 21, 12,
                                   6,  4,  8,  12, 14, 12, 8,  4,  2,  4,  6,  7,  6,  4,  2};
constexpr int kThreadsL = 256;
constexpr int kMaxRoundsL = 4096;  // repair rounds of one frame step before LVBGS_DEVICE_ERROR

// ---- intent word ----
// bit 0 valid (ROI pixel evaluated), bit 1 foreground, bits 2-8 samples scanned, bit 9 own-sample write,
// bits 10-15 its sample, bit 16 neighbour write, bits 17-20 neighbour code (dy+1)*3+(dx+1), bits 21-26
// its sample, bits 27-29 draws consumed
constexpr uint32_t kIValid = 1u, kIFG = 2u, kIOwn = 1u << 9, kINb = 1u << 16;
__device__ __forceinline__ int i_e(uint32_t w) { return (int)((w >> 2) & 127u); }
__device__ __forceinline__ int i_sown(uint32_t w) { return (int)((w >> 10) & 63u); }
__device__ __forceinline__ int i_code(uint32_t w) { return (int)((w >> 17) & 15u); }
__device__ __forceinline__ int i_snb(uint32_t w) { return (int)((w >> 21) & 63u); }
__device__ __forceinline__ int i_draws(uint32_t w) { return (int)((w >> 27) & 7u); }
// the neighbour-write part of an intent (target and sample)
__device__ __forceinline__ uint32_t i_nbpart(uint32_t w) { return (w & kIValid) ? (w & (kINb | (1023u << 17))) : 0u; }
__device__ __forceinline__ int nb_target(uint32_t w, int q, int W) {
    const int c = i_code(w);
    return q + (c / 3 - 1) * W + (c % 3 - 1);
}

__device__ __forceinline__ unsigned int ld_vol(const unsigned int* p) { return *(const volatile unsigned int*)p; }

// draw k of pixel p in frame t (the counter-based generator that replaces rand())
struct Draws {
    uint32_t blk, v[4];
};
__device__ __forceinline__ uint32_t draw(const LobDev& D, uint32_t p, uint32_t k, Draws& ds) {
    const uint32_t blk = k >> 2;
    if (blk != ds.blk) {
        uint32_t c[4] = {blk, p, D.frameKey, 0u};
        philox4x32_10(c, (uint32_t)D.seed, (uint32_t)(D.seed >> 32));
        ds.v[0] = c[0];
        ds.v[1] = c[1];
        ds.v[2] = c[2];
        ds.v[3] = c[3];
        ds.blk = blk;
    }
    return ds.v[k & 3u] & 0x7fffffffu;
}
// rand() % m for a 31-bit draw and a size_t modulus
__device__ __forceinline__ unsigned long long mod64(uint32_t a, unsigned long long m) {
    if (m > 0xffffffffull) return a;
    const uint32_t m32 = (uint32_t)m;
    if ((m32 & (m32 - 1u)) == 0u) return a & (m32 - 1u);
    return a % m32;
}
__device__ __forceinline__ int clampi(int v, int lo, int hi) { return v < lo ? lo : v > hi ? hi : v; }
// tiles of n pixels along a side. Tiles are numbered row by row in a grid of one dimension: the second one ends at 65,535
LV_HD constexpr int tiles_across(int side, int n) { return (side + n - 1) / n; }

// the 16 LBSP taps of channel c at pixel index p of a dense image, packed four to a word
template <int C>
__device__ __forceinline__ void taps(const uint8_t* img, int W, int p, int c, uint32_t (&v)[4]) {
    const uint8_t* base = img + (size_t)p * C + c;
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

// Sample s of pixel p as (d, c2): LOBSTER, the packed word and the colour byte; ViBe, colour c at bits 8c of
// d; PBAS, also gradient c at bits 24 + 8c. A sample is one or two accesses that a warp makes in whole lines:
// LOBSTER u64 + u8 (one channel u16 + u8); PBAS u32 (colours, gradient 0) + u16 (gradients 1 and 2), one
// channel u16; ViBe u16 + u8, one channel u8. With a byte plane per value a PBAS sample took six accesses.
template <int C, int ALG>
__device__ __forceinline__ void load_sample(const LobDev& D, int s, int p, unsigned long long& d, uint32_t& c2) {
    const size_t o = (size_t)s * D.npx + p;
    c2 = 0;
    if (ALG == ALG_PBAS) {
        if (C == 3) {
            d = (unsigned long long)__ldg((const uint32_t*)D.sC + o) | ((unsigned long long)__ldg((const uint16_t*)D.sG + o) << 32);
        } else {
            const uint32_t v = __ldg((const uint16_t*)D.sC + o);
            d = (v & 0xffu) | ((unsigned long long)(v >> 8) << 24);
        }
    } else if (ALG == ALG_VIBE) {
        if (C == 3) d = (uint32_t)__ldg((const uint16_t*)D.sC + o) | ((uint32_t)__ldg(D.sG + o) << 16);
        else d = __ldg(D.sC + o);
    } else {
        if (C == 3) d = __ldg((const unsigned long long*)D.sD + o);
        else d = __ldg((const uint16_t*)D.sD + o);
        c2 = __ldg(D.sC + o);
    }
}
template <int C, int ALG>
__device__ __forceinline__ void store_sample(const LobDev& D, int s, int p, unsigned long long d, uint32_t c2) {
    const size_t o = (size_t)s * D.npx + p;
    if (ALG == ALG_PBAS) {
        if (C == 3) {
            ((uint32_t*)D.sC)[o] = (uint32_t)d;
            ((uint16_t*)D.sG)[o] = (uint16_t)(d >> 32);
        } else {
            ((uint16_t*)D.sC)[o] = (uint16_t)((d & 0xffu) | ((d >> 16) & 0xff00u));
        }
    } else if (ALG == ALG_VIBE) {
        if (C == 3) {
            ((uint16_t*)D.sC)[o] = (uint16_t)d;
            D.sG[o] = (uint8_t)(d >> 16);
        } else {
            D.sC[o] = (uint8_t)d;
        }
    } else {
        if (C == 3) ((unsigned long long*)D.sD)[o] = d;
        else ((uint16_t*)D.sD)[o] = (uint16_t)d;
        D.sC[o] = (uint8_t)c2;
    }
}
// bytes of the two sample planes (sC, sG) per sample and pixel
inline size_t sample_bytes_lo(int alg, int C) { return alg == ALG_PBAS ? (C == 3 ? 4 : 2) : alg == ALG_VIBE ? (C == 3 ? 2 : 1) : 1; }
inline size_t sample_bytes_hi(int alg, int C) { return C != 3 ? 0 : alg == ALG_PBAS ? 2 : alg == ALG_VIBE ? 1 : 0; }

// what the scan needs of a pixel: LOBSTER, its colour by channel and its LBSP taps; ViBe and PBAS, its colour
// packed (channel c at bits 8c); PBAS, also its gradient packed, its threshold R(x) * R0 and the weight of
// gradient distances BGSPBAS_GRAD_WEIGHT_ALPHA / m_fFormerMeanGradDist
template <int C, int ALG>
struct PxIn {
    uint32_t vals[C][4];
    uint32_t curr[ALG == ALG_LOBSTER ? C : 1], g;
    float thr, gw;
};
// the squared distance of two packed three-channel values (bits 24 to 31 of b ignored, of a zero)
__device__ __forceinline__ uint32_t sqdist3(uint32_t a, uint32_t b) {
    const uint32_t d = __vabsdiffu4(a, b & 0xffffffu);
    return __dp4a(d, d, 0u);
}
// sqrtf of an integer below 65536; zero, frequent here, keeps off the root's path for special values
__device__ __forceinline__ float root16(uint32_t v) {
    const float r = __fsqrt_rn((float)max(v, 1u));
    return v ? r : 0.0f;
}

// one sample against the pixel: LOBSTER (:479-494 / :522-541); ViBe (BackgroundSubtractorViBe.cpp:87 /
// :165-170): |in - bg| < R on one channel; on three, lv::L2dist<3>(uchar*, uchar*) < 3R, whose squared
// differences add up in uint16_t (utils/math.hpp:391-396), so the sum s wraps modulo 65536 before the
// square root. For integers s < 65536 and T = 3R, (float)sqrt(s) < (float)T is exactly s < T*T when
// T < 256 (sqrt(T*T - 1) < T - 1/(2T), and 1/(2T) is far above the float spacing near T), and always true
// when T >= 256
template <int C, int ALG>
__device__ __forceinline__ bool match(const LobDev& D, const PxIn<C, ALG>& in, unsigned long long d, uint32_t c2) {
    if constexpr (ALG == ALG_VIBE) {
        if (C == 1) return (uint32_t)abs((int)in.curr[0] - (int)(d & 0xffu)) < D.colThr;
        const unsigned long long T = 3ull * D.colThr;
        return T >= 256ull || (unsigned long long)(sqdist3(in.curr[0], (uint32_t)d) & 0xffffu) < T * T;
    } else if constexpr (C == 1) {
        const uint32_t bgc = c2, bgd = (uint32_t)d & 0xffffu;
        if ((uint32_t)abs((int)in.curr[0] - (int)bgc) > D.colThr / 2u) return false;
        return (uint32_t)__popc(lbsp_thr(in.vals[0], bgc, __ldg(D.lut + bgc)) ^ bgd) <= D.descThr;
    } else {
        const uint32_t descThr = D.descThr * 3u, colThr = D.colThr * 3u;
        const uint32_t scDesc = descThr / 2u, scCol = colThr / 2u;
        uint32_t totCol = 0, totDesc = 0;
#pragma unroll
        for (int c = 0; c < 3; ++c) {
            const uint32_t bgc = c == 0 ? (uint32_t)(d >> 48) & 0xffu : c == 1 ? (uint32_t)(d >> 56) & 0xffu : c2;
            const uint32_t bgd = (uint32_t)(d >> (16 * c)) & 0xffffu;
            const uint32_t colDist = (uint32_t)abs((int)in.curr[c] - (int)bgc);
            if (colDist > scCol) return false;
            const uint32_t descDist = (uint32_t)__popc(lbsp_thr(in.vals[c], bgc, __ldg(D.lut + bgc)) ^ bgd);
            if (descDist > scDesc) return false;
            totCol += colDist;
            totDesc += descDist;
        }
        return totDesc <= descThr && totCol <= colThr;
    }
}

template <int C, int ALG>
__device__ __forceinline__ void pixel_inputs(const LobDev& D, int p, bool on, PxIn<C, ALG>& in) {
    in.thr = in.gw = 0.0f;
    in.g = 0u;
#pragma unroll
    for (int c = 0; c < (ALG == ALG_LOBSTER ? C : 1); ++c) in.curr[c] = 0u;
#pragma unroll
    for (int c = 0; c < C; ++c)
#pragma unroll
        for (int j = 0; j < 4; ++j) in.vals[c][j] = 0u;
    if (!on) return;
#pragma unroll
    for (int c = 0; c < C; ++c) {
        if constexpr (ALG == ALG_LOBSTER) {
            taps<C>(D.frame, D.W, p, c, in.vals[c]);
            in.curr[c] = __ldg(D.frame + (size_t)p * C + c);
        } else {
            in.curr[0] |= (uint32_t)__ldg(D.frame + (size_t)p * C + c) << (8 * c);
        }
        if (ALG == ALG_PBAS) in.g |= (uint32_t)__ldg(D.grad + (size_t)p * C + c) << (8 * c);
    }
    if (ALG == ALG_PBAS) {
        in.thr = D.fm[(size_t)D.cur * 3 * D.npx + p] * D.R0;
        in.gw = 10.0f / *D.meanGrad;
    }
}
// The sample word the pixel writes: LOBSTER, its descriptors (:499-500 / :548-550) and colour; ViBe, its colour;
// PBAS, its colour and gradient (also what a neighbour update writes into it)
template <int C, int ALG>
__device__ __forceinline__ unsigned long long sample_word(const LobDev& D, const PxIn<C, ALG>& in) {
    if constexpr (ALG == ALG_VIBE) {
        return in.curr[0];
    } else if constexpr (ALG == ALG_PBAS) {
        return (unsigned long long)in.curr[0] | ((unsigned long long)in.g << 24);
    } else {
        unsigned long long wd = 0;
#pragma unroll
        for (int c = 0; c < C; ++c)
            wd |= (unsigned long long)lbsp_thr(in.vals[c], in.curr[c], __ldg(D.lut + in.curr[c])) << (16 * c);
        if (C == 3) wd |= ((unsigned long long)in.curr[0] << 48) | ((unsigned long long)in.curr[1] << 56);
        return wd;
    }
}

// One sample against the pixel. PBAS (:146-166 / :365-394): the colour distance plus the weighted gradient
// distance, at most 255, against the threshold; grad is the gradient distance (one channel) or its square
// modulo 65536, with dist its root (three: lv::L2dist of two Vec3b adds in uint16_t). (float)sqrt((double)s) of that integer
// equals sqrtf((float)s), since double rounding through double is innocuous for the square root
// (53 >= 2 * 24 + 2 bits).
template <int C, int ALG>
__device__ __forceinline__ bool judge(const LobDev& D, const PxIn<C, ALG>& in, unsigned long long d, uint32_t c2, float& fSum,
                                      uint32_t& grad, float& dist) {
    if constexpr (ALG != ALG_PBAS) {
        return match<C, ALG>(D, in, d, c2);
    } else if constexpr (C == 1) {
        const uint32_t nCol = (uint32_t)abs((int)in.curr[0] - (int)(d & 0xffu));
        grad = (uint32_t)abs((int)in.g - (int)((d >> 24) & 0xffu));
        fSum = in.gw * (float)grad + (float)nCol;
    } else {
        grad = sqdist3(in.g, (uint32_t)(d >> 24)) & 0xffffu;
        dist = root16(grad);
        fSum = in.gw * dist + root16(sqdist3(in.curr[0], (uint32_t)d) & 0xffffu);
    }
    if (fSum > 255.0f) fSum = 255.0f;
    return fSum <= in.thr;
}

// Samples that earlier neighbours write this frame (repair): which, and which of them match the pixel now. PBAS
// writes the pixel's own values into them (self diffusion): distance 0, always good.
struct Over {
    unsigned long long mask, good;
};
// state of a pixel's ordered scan; PBAS: smallest good distance, bad samples and the sum of their gradient
// distances (one channel: exact; three: about, it only predicts where the ordered sum will be)
struct Scan {
    int s, nGood, nb;
    uint32_t badSum;
    float badAbout, fMin;
};
__device__ __forceinline__ Scan scan_start() { return {0, 0, 0, 0u, 0.0f, 255.0f}; }
// the gradient distance of the pixel's i-th bad sample, three channels, as its square in 16 bits
__device__ __forceinline__ uint16_t& bad_value(const LobDev& D, int i, int p) { return D.badVals[(size_t)p * D.N + i]; }

// the ordered scan by the pixel's own lane, from st up to sample end
template <int C, int ALG>
__device__ __forceinline__ void lane_scan(const LobDev& D, int p, const PxIn<C, ALG>& in, const Over& ov, int end, Scan& st) {
    unsigned long long dB = 0;
    uint32_t cB = 0;
    if (st.s < end && st.nGood < D.nreq) load_sample<C, ALG>(D, st.s, p, dB, cB);
    while (st.nGood < D.nreq && st.s < end) {
        const unsigned long long d = dB;
        const uint32_t c2 = cB;
        if (st.s + 1 < end) load_sample<C, ALG>(D, st.s + 1, p, dB, cB);
        float fSum = 0.0f, dist = 0.0f;
        uint32_t grad = 0u;
        const bool good = ((ov.mask >> st.s) & 1ull) ? (ov.good >> st.s) & 1ull : judge<C, ALG>(D, in, d, c2, fSum, grad, dist);
        if (good) {
            if (ALG == ALG_PBAS && st.fMin > fSum) st.fMin = fSum;
            ++st.nGood;
        } else if (ALG == ALG_PBAS) {
            if (C == 1) st.badSum += grad;
            else bad_value(D, st.nb, p) = (uint16_t)grad;
            st.badAbout += dist;
            ++st.nb;
        }
        ++st.s;
    }
}

// The rest of the scans of a warp's pixels (on: this lane's pixel p may need more), by groups of eight lanes: a
// group takes the next unsettled pixel, broadcasts its inputs and judges eight samples a step; the ballot gives
// the ordered result (the scan stops at the nreq-th good sample). A warp whose lanes scan alone runs to its
// slowest lane, all N samples as soon as one lane is foreground, and a single scan is a chain of ~0.4 us a
// sample. Every lane of the warp calls it.
template <int C, int ALG>
__device__ __forceinline__ void group_scan(const LobDev& D, bool on, int p, const PxIn<C, ALG>& in, const Over& ov, Scan& st) {
    constexpr unsigned kAll = 0xffffffffu;
    const int lane = threadIdx.x & 31, grp = lane >> 3, sub = lane & 7, N = D.N, nreq = D.nreq;
    unsigned todo = __ballot_sync(kAll, on && st.nGood < nreq && st.s < N);
    while (todo) {
        unsigned own = todo;
        for (int i = 0; i < grp; ++i) own &= own - 1u;
        const bool go = own != 0u;
        const int src = go ? __ffs(own) - 1 : lane;
        unsigned taken = todo;
#pragma unroll
        for (int i = 0; i < 4; ++i) todo &= todo - 1u;
        taken ^= todo;
        __syncwarp();
        PxIn<C, ALG> b;
#pragma unroll
        for (int c = 0; c < (ALG == ALG_LOBSTER ? C : 1); ++c) b.curr[c] = __shfl_sync(kAll, in.curr[c], src);
#pragma unroll
        for (int c = 0; c < C; ++c)
#pragma unroll
            for (int j = 0; j < 4; ++j) b.vals[c][j] = ALG == ALG_LOBSTER ? __shfl_sync(kAll, in.vals[c][j], src) : 0u;
        b.g = ALG == ALG_PBAS ? __shfl_sync(kAll, in.g, src) : 0u;
        b.thr = b.gw = 0.0f;
        if (ALG == ALG_PBAS) {
            b.thr = __shfl_sync(kAll, in.thr, src);
            b.gw = __shfl_sync(kAll, in.gw, src);
        }
        const int bp = __shfl_sync(kAll, p, src);
        Over bo;
        bo.mask = __shfl_sync(kAll, ov.mask, src);
        bo.good = __shfl_sync(kAll, ov.good, src);
        Scan t;
        t.s = __shfl_sync(kAll, st.s, src);
        t.nGood = __shfl_sync(kAll, st.nGood, src);
        t.nb = ALG == ALG_PBAS ? __shfl_sync(kAll, st.nb, src) : 0;
        t.badSum = 0u;
        t.badAbout = 0.0f;
        t.fMin = 255.0f;
        int k = t.s + sub;
        unsigned long long d = 0;
        uint32_t c2 = 0;
        if (go && k < N) load_sample<C, ALG>(D, k, bp, d, c2);
        while (__any_sync(kAll, go && t.nGood < nreq && t.s < N)) {
            __syncwarp();
            const bool act = go && t.nGood < nreq && t.s < N;
            unsigned long long dn = 0;
            uint32_t cn = 0;
            if (act && k + 8 < N) load_sample<C, ALG>(D, k + 8, bp, dn, cn);
            float fSum = 0.0f, dist = 0.0f;
            uint32_t grad = 0u;
            bool good = false;
            if (act && k < N)
                good = ((bo.mask >> k) & 1ull) ? (bo.good >> k) & 1ull : judge<C, ALG>(D, b, d, c2, fSum, grad, dist);
            __syncwarp();
            const uint32_t m = (__ballot_sync(kAll, good) >> (8 * grp)) & 0xffu;
            if (act) {
                const int need = nreq - t.nGood, cnt = __popc(m);
                int stop = min(8, N - t.s);
                if (cnt >= need) {
                    uint32_t r = m;
                    for (int i = 1; i < need; ++i) r &= r - 1u;
                    stop = __ffs(r);
                    t.nGood = nreq;
                } else {
                    t.nGood += cnt;
                }
                if (ALG == ALG_PBAS && sub < stop) {
                    if (good) {
                        if (t.fMin > fSum) t.fMin = fSum;
                    } else if (C == 1) {
                        t.badSum += grad;
                    } else {
                        t.badAbout += dist;
                        bad_value(D, t.nb + __popc(~m & ((1u << sub) - 1u)), bp) = (uint16_t)grad;
                    }
                }
                if (ALG == ALG_PBAS) t.nb += __popc(~m & ((1u << stop) - 1u));
                t.s += stop;
            }
            d = dn;
            c2 = cn;
            k += 8;
        }
        if (ALG == ALG_PBAS) {
#pragma unroll
            for (int o = 4; o > 0; o >>= 1) {
                t.badSum += __shfl_xor_sync(kAll, t.badSum, o);
                t.badAbout += __shfl_xor_sync(kAll, t.badAbout, o);
                const float f = __shfl_xor_sync(kAll, t.fMin, o);
                if (t.fMin > f) t.fMin = f;
            }
        }
        // back to the owners: the r-th owner's scan was done by group r
        const bool mine = (taken >> lane) & 1u;
        const int from = mine ? 8 * __popc(taken & ((1u << lane) - 1u)) : lane;
        const int rs = __shfl_sync(kAll, t.s, from), rg = __shfl_sync(kAll, t.nGood, from);
        if (mine) {
            st.s = rs;
            st.nGood = rg;
        }
        if (ALG == ALG_PBAS) {
            const int rb = __shfl_sync(kAll, t.nb, from);
            const uint32_t rq = __shfl_sync(kAll, t.badSum, from);
            const float rf = __shfl_sync(kAll, t.fMin, from), ra = __shfl_sync(kAll, t.badAbout, from);
            if (mine) {
                st.nb = rb;
                st.badSum += rq;
                st.badAbout += ra;
                if (st.fMin > rf) st.fMin = rf;
            }
        }
    }
    __syncwarp();
}

// The decision of a scanned pixel p (x, y) and its model writes with their draws (:497-513 / :545-575; PBAS
// :174-194 / :402-424): returns the intent word. PBAS also writes its D(x), T(x) and R(x) of the next parity
// (:198-231 / :427-458) and the bad samples for the frame level.
template <int C, int ALG>
__device__ uint32_t decide(const LobDev& D, int p, int x, int y, const Scan& st) {
    uint32_t w = kIValid | ((uint32_t)st.s << 2), k = 0;
    const bool fg = st.nGood < D.nreq;
    const size_t npx = (size_t)D.npx;
    float R = 0.0f, T = 0.0f, Dn = 0.0f;
    if (ALG == ALG_PBAS) {
        const float* fc = D.fm + (size_t)D.cur * 3 * npx;
        R = fc[p];
        T = fc[npx + p];
        const float Dm = fc[2 * npx + p], Nf = (float)D.N;
        Dn = (Dm * (Nf - 1.0f) + st.fMin / 255.0f) / Nf;
    }
    if (fg) {
        w |= kIFG;
    } else {
        const unsigned long long nLR =
            ALG == ALG_PBAS && !D.lrOverride ? (unsigned long long)__float2uint_rz(ceilf(T)) : D.nLR;
        Draws ds;
        ds.blk = 0xffffffffu;
        if (mod64(draw(D, (uint32_t)p, k++, ds), nLR) == 0ull) {
            const uint32_t so = draw(D, (uint32_t)p, k++, ds) % (uint32_t)D.N;
            w |= kIOwn | (so << 10);
        }
        if (mod64(draw(D, (uint32_t)p, k++, ds), nLR) == 0ull) {
            // getNeighborPosition_3x3 (opencv.hpp:945-953), clamped into the LBSP border (LOBSTER) or the frame
            constexpr int bord = ALG == ALG_LOBSTER ? kBorder : 0;
            int dx, dy;
            nb3_offset((int)(draw(D, (uint32_t)p, k++, ds) % 8u), dx, dy);
            const int nx = clampi(x + dx, bord, D.W - bord - 1), ny = clampi(y + dy, bord, D.H - bord - 1);
            const uint32_t sn = draw(D, (uint32_t)p, k++, ds) % (uint32_t)D.N;
            w |= kINb | ((uint32_t)((ny - y + 1) * 3 + (nx - x + 1)) << 17) | (sn << 21);
        }
    }
    if (ALG == ALG_PBAS) {
        float Tn;
        if (fg) {
            Tn = T + 1.0000f / (Dn * 255.00f + 1.0000f);
            if (Tn > 200.00f) Tn = 200.00f;
        } else {
            Tn = T - 0.0500f / (Dn * 255.00f + 1.0000f);
            if (Tn < 2.0000f) Tn = 2.0000f;
        }
        float Rn = R;
        if (R < 0.6000f + Dn * 5.0000f + 0.0000f) {
            if (R < 99.0000f) Rn = R * 1.0500f;
        } else if (R > 0.6000f) {
            Rn = R * 0.9500f;
        }
        float* fn = D.fm + (size_t)(D.cur ^ 1) * 3 * npx;
        fn[p] = Rn;
        fn[npx + p] = Tn;
        fn[2 * npx + p] = Dn;
        if (C == 1) D.badSum[p] = st.badSum;  // three channels keep the values (badVals)
        D.badCnt[p] = (uint8_t)st.nb;
    }
    return w | (k << 27);
}

// per-thread counts (each below 2^24) into one or two 64-bit counters, one atomic each per block: the counters
// are shared by the whole frame, and same-address atomics serialize. Every thread of the block calls it.
__device__ __forceinline__ void block_add(unsigned long long* a, unsigned int va, unsigned long long* b = nullptr,
                                          unsigned int vb = 0u) {
    __shared__ unsigned int red[2][kThreadsL / 32];
    const unsigned int sa = __reduce_add_sync(0xffffffffu, va), sb = b ? __reduce_add_sync(0xffffffffu, vb) : 0u;
    __syncthreads();  // an earlier call's values have been read
    if ((threadIdx.x & 31) == 0) {
        red[0][threadIdx.x >> 5] = sa;
        red[1][threadIdx.x >> 5] = sb;
    }
    __syncthreads();
    if (threadIdx.x < 2) {
        unsigned long long t = 0;
        for (int w = 0; w < kThreadsL / 32; ++w) t += red[threadIdx.x][w];
        unsigned long long* c = threadIdx.x ? b : a;
        if (t) atomicAdd(c, t);
    }
}

// list push with per-round dedupe; the lanes that push together share one counter atomic
__device__ __forceinline__ void push(const LobDev& D, uint32_t* list, unsigned int* count, uint32_t stamp, int t) {
    if (atomicExch(&D.stamp[t], stamp) == stamp) return;
    const unsigned am = __activemask();
    const int lane = threadIdx.x & 31, leader = __ffs(am) - 1;
    unsigned int base = 0;
    if (lane == leader) base = atomicAdd(count, (unsigned int)__popc(am));
    base = __shfl_sync(am, base, leader);
    const unsigned int i = base + (unsigned int)__popc(am & ((1u << lane) - 1u));
    if (i < D.listCap) list[i] = (uint32_t)t;
    else atomicOr(&D.flags[LOB_F_ERR], 1u);
}

}  // namespace

// 1. every ROI pixel (ViBe, PBAS: every pixel) against the frame-start samples: the lane itself up to lane_cap
// samples, which settle most pixels, the others by groups. Block 0 opens the frame step's flags. Caps of 2, 4, 8
// and none: LOBSTER 1277x719 BGR 53 / 45 / 42 / 46 us; PBAS 1920x1080 BGR 177 / 140 / 149 / 164 us; ViBe, whose
// judgements are too cheap for the broadcasts, 320x240 BGR 11.7 / 10.8 / 10.5 / 9.9 us. PBAS's judgement on packed
// bytes (four bytes a difference, a dot product for the squares) took its 140 us to 136 us, six blocks per SM
// instead of four to 110 us: the loads' latency bounds it (DRAM at a third of its rate, 57 % of the issue slots).
LV_HD constexpr int lane_cap(int alg) { return alg == ALG_LOBSTER ? 8 : alg == ALG_PBAS ? 4 : kMaxSamples; }
template <int C, int ALG>
__global__ void __launch_bounds__(kThreadsL, ALG == ALG_PBAS ? 6 : 5) lob_k_eval(LobDev D) {
    pdl_entry();
    if (blockIdx.x == 0 && threadIdx.x < LOB_F_WORDS) D.flags[threadIdx.x] = 0u;
    if (ALG == ALG_PBAS && blockIdx.x == 0 && threadIdx.x < 2) D.stats[2 + threadIdx.x] = 0ull;
    const int p = blockIdx.x * blockDim.x + threadIdx.x;
    const bool in = p < D.npx;
    const bool on = in && (ALG != ALG_LOBSTER || D.roi[p]);
    PxIn<C, ALG> px;
    pixel_inputs<C, ALG>(D, p, on, px);
    const Over none = {0ull, 0ull};
    Scan st = scan_start();
    if (on) {
        D.wD[p] = sample_word<C, ALG>(D, px);
        lane_scan<C, ALG>(D, p, px, none, min(lane_cap(ALG), D.N), st);
    }
    group_scan<C, ALG>(D, on, p, px, none, st);
    if (in) D.intent[p] = on ? decide<C, ALG>(D, p, p % D.W, p / D.W, st) : 0u;
    if (ALG == ALG_PBAS && C == 3) {  // about what the block's chunk adds to the ordered sum: repairs hardly change it
        __shared__ float sm[kThreadsL / 32];
        float about = in ? st.badAbout : 0.0f;
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) about += __shfl_xor_sync(0xffffffffu, about, o);
        if ((threadIdx.x & 31) == 0) sm[threadIdx.x >> 5] = about;
        __syncthreads();
        if (threadIdx.x == 0) {
            float c = 0.0f;
            for (int w = 0; w < kThreadsL / 32; ++w) c += sm[w];
            D.chunkAbout[blockIdx.x] = c;
        }
    }
    block_add(&D.stats[0], on ? (unsigned int)st.s : 0u);
}

// the four earlier pixels within one step of p (x, y): the row above, then the left neighbour
struct Earlier {
    int q[4];
    bool ok[4];
};
__device__ __forceinline__ Earlier earlier(const LobDev& D, int p, int x, int y) {
    return {{p - D.W - 1, p - D.W, p - D.W + 1, p - 1}, {y > 0 && x > 0, y > 0, y > 0 && x + 1 < D.W, x > 0}};
}

// Re-evaluates the pixels of a warp's owner lanes (on: this lane holds pixel p; every lane calls it) with the
// samples that their earlier neighbours write now, and lists the later pixels whose incoming writes changed.
// alone: every lane scans its own pixel (a list that fills the machine), otherwise groups of eight lanes do.
template <int C, int ALG>
__device__ void reevaluate(const LobDev& D, bool on, int p, bool alone, uint32_t* out, unsigned int* outCount, uint32_t stamp,
                           unsigned int& scanned) {
    const int x = on ? p % D.W : 0, y = on ? p / D.W : 0;
    PxIn<C, ALG> px;
    pixel_inputs<C, ALG>(D, p, on, px);
    Over ov = {0ull, 0ull};
    if (on) {
        const Earlier e = earlier(D, p, x, y);
        uint32_t wq[4];
#pragma unroll
        for (int j = 0; j < 4; ++j) wq[j] = e.ok[j] ? ld_vol(&D.intent[e.q[j]]) : 0u;
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            if (!((wq[j] & kIValid) && (wq[j] & kINb) && nb_target(wq[j], e.q[j], D.W) == p)) continue;
            const unsigned long long bit = 1ull << i_snb(wq[j]);
            bool good = true;
            if (ALG != ALG_PBAS) {
                const uint32_t c = ALG != ALG_LOBSTER ? 0u : __ldg(D.frame + (size_t)e.q[j] * C + (C == 3 ? 2 : 0));
                float f, dist;
                uint32_t gr;
                good = judge<C, ALG>(D, px, __ldcg(D.wD + e.q[j]), c, f, gr, dist);
            }
            // the latest writer of a sample decides
            ov.mask |= bit;
            ov.good = good ? ov.good | bit : ov.good & ~bit;
        }
    }
    Scan st = scan_start();
    if (alone && on) lane_scan<C, ALG>(D, p, px, ov, D.N, st);
    group_scan<C, ALG>(D, on, p, px, ov, st);
    if (!on) return;
    scanned += (unsigned int)st.s;
    const uint32_t wNew = decide<C, ALG>(D, p, x, y, st), wOld = ld_vol(&D.intent[p]);
    if (wNew == wOld) return;
    *(volatile uint32_t*)&D.intent[p] = wNew;
    if (i_nbpart(wNew) == i_nbpart(wOld)) return;
    // the targets of the old and the new neighbour write that come later in raster order
    if (wOld & kINb) {
        const int t = nb_target(wOld, p, D.W);
        if (t > p) push(D, out, outCount, stamp, t);
    }
    if (wNew & kINb) {
        const int t = nb_target(wNew, p, D.W);
        if (t > p) push(D, out, outCount, stamp, t);
    }
}

// End of repair round `round`, by every block of its kernel; the block that finishes last closes it: converged
// when the round listed nothing, otherwise its input list becomes the next round's output
__device__ __forceinline__ void round_end(const LobDev& D, int round) {
    __syncthreads();
    if (threadIdx.x != 0) return;
    __threadfence();
    if (atomicAdd(&D.flags[LOB_F_DONE], 1u) != gridDim.x - 1u) return;
    D.flags[LOB_F_DONE] = 0u;
    const int cur = round & 1;
    const unsigned int next = ld_vol(&D.flags[cur ^ 1]);
    D.flags[LOB_F_ROUNDS] = (unsigned int)round + 1u;
    if (next > D.listCap) {
        D.flags[LOB_F_ERR] |= 1u;
        D.flags[LOB_F_CONV] = 1u;
    } else if (next == 0u) {
        D.flags[LOB_F_CONV] = 1u;
    } else {
        D.flags[cur] = 0u;
    }
}

// 2. Round 0: a block finds the pixels of its own (PER a thread) whose scan read a sample that an earlier
// neighbour writes, and re-evaluates them, with the other blocks' re-evaluations under way: a pixel that changes
// its neighbour write after a later pixel looked at it lists that pixel for round 1. One launch where the marks
// went through a list in memory. A block lasts as long as its slowest re-evaluation, so it takes 1,024 pixels:
// with 256, LOBSTER 1277x719 BGR took 36 us and PBAS 1920x1080 BGR 67 us. A chain of latencies: more blocks at
// once are worth some spilled registers (3 / 5 / 6 / 8 blocks per SM: LOBSTER 19.6 / 17.8 / 14.6 / 15.4 us, PBAS
// 34 / 30 / 28 / 24 us). A frame of which four pixels a thread would make fewer than two blocks on each of this
// chip's 152 SMs takes one a thread: 320x240 BGR ViBe 8.6 -> 7.7 us, 45 -> 40 us a frame (the one size measured in both forms;
// on a chip with another count the line would lie elsewhere).
constexpr int kFirstSmall = 304 * 1024;
template <int C, int ALG, int PER>
__global__ void __launch_bounds__(kThreadsL, ALG == ALG_PBAS ? 8 : 6) lob_k_first(LobDev D) {
    pdl_entry();
    constexpr int kFirstPx = PER * kThreadsL;
    __shared__ int items[kFirstPx];
    __shared__ int count;
    if (threadIdx.x == 0) count = 0;
    __syncthreads();
    const int lane = threadIdx.x & 31, p0 = blockIdx.x * kFirstPx + (int)threadIdx.x;
    uint32_t w[PER], wq[PER][4];
#pragma unroll
    for (int i = 0; i < PER; ++i) {
        const int p = p0 + i * kThreadsL;
        w[i] = p < D.npx ? ld_vol(&D.intent[p]) : 0u;
        const Earlier e = earlier(D, p, p % D.W, p / D.W);
#pragma unroll
        for (int j = 0; j < 4; ++j) wq[i][j] = p < D.npx && e.ok[j] ? ld_vol(&D.intent[e.q[j]]) : 0u;
    }
#pragma unroll
    for (int i = 0; i < PER; ++i) {
        const int p = p0 + i * kThreadsL;
        bool dirty = false;
        if (w[i] & kIValid) {
            const int n = i_e(w[i]);
            // the four earlier neighbours reach p with the codes of one step down right, down, down left, right
            const int code[4] = {8, 7, 6, 5};
#pragma unroll
            for (int j = 0; j < 4; ++j)
                dirty = dirty || ((wq[i][j] & kIValid) && (wq[i][j] & kINb) && i_code(wq[i][j]) == code[j] && i_snb(wq[i][j]) < n);
        }
        const unsigned m = __ballot_sync(0xffffffffu, dirty);
        int base = 0;
        if (lane == 0 && m) base = atomicAdd(&count, __popc(m));
        base = __shfl_sync(0xffffffffu, base, 0);
        if (dirty) items[base + __popc(m & ((1u << lane) - 1u))] = p;
    }
    __syncthreads();
    unsigned int scanned = 0;
    const uint32_t stamp = D.stampBase + 1u;
    const int n = count;
    const bool alone = n > kThreadsL / 2;  // more than four pixels a group: every lane its own
    const int per = alone ? 32 : 4;
    for (int i0 = (threadIdx.x >> 5) * per; i0 < n; i0 += per * (kThreadsL / 32)) {
        const int i = alone ? i0 + lane : i0 + (lane >> 3);
        const bool on = i < n && (alone || (lane & 7) == 0);
        reevaluate<C, ALG>(D, on, on ? items[i] : 0, alone, D.list1, &D.flags[LOB_F_COUNT1], stamp, scanned);
    }
    block_add(&D.stats[0], scanned);
    round_end(D, 0);
}

// 3. one later repair round: the pixels of list (round & 1)
template <int C, int ALG>
__global__ void __launch_bounds__(kThreadsL) lob_k_round(LobDev D, int round) {
    pdl_entry();
    if (ld_vol(&D.flags[LOB_F_CONV])) return;
    const int cur = round & 1;
    const unsigned int n0 = ld_vol(&D.flags[cur]);
    const unsigned int n = n0 < D.listCap ? n0 : D.listCap;
    const uint32_t* in = cur ? D.list1 : D.list0;
    uint32_t* out = cur ? D.list0 : D.list1;
    unsigned int* outCount = &D.flags[cur ^ 1];
    const uint32_t stamp = D.stampBase + (uint32_t)round + 1u;
    unsigned int scanned = 0;
    const int lane = threadIdx.x & 31;
    const unsigned int warp = blockIdx.x * (kThreadsL / 32) + (threadIdx.x >> 5), warps = gridDim.x * (kThreadsL / 32);
    const bool alone = n > 16u * warps;  // more than four pixels a group: every lane its own
    const unsigned int per = alone ? 32u : 4u;
    for (unsigned int i0 = warp * per; i0 < n; i0 += warps * per) {
        const unsigned int i = alone ? i0 + lane : i0 + (lane >> 3);
        const bool on = i < n && (alone || (lane & 7) == 0);
        reevaluate<C, ALG>(D, on, on ? (int)__ldcg(in + i) : 0, alone, out, outCount, stamp, scanned);
    }
    block_add(&D.stats[0], scanned);
    round_end(D, round);
}

// 4. every pixel gathers the sample writes aimed at it, in raster order of the writers (own update
// before neighbour update within a writer); the raw mask (ViBe: the output, :84 / :176) and the draw
// counters of the frame. The nine intents are requested together; the writes go to a register list of 12 bits
// each (window slot, sample, own write) that the warp executes together, and more than five (rare) take the
// slots one by one. A pixel's writes are its own thread's, in order, so the last writer of a sample wins.
template <int C, int ALG>
__global__ void __launch_bounds__(kThreadsL) lob_k_commit(LobDev D) {
    pdl_entry();
    const unsigned int conv = ld_vol(&D.flags[LOB_F_CONV]);
    if (blockIdx.x == 0 && threadIdx.x < LOB_F_WORDS) ((volatile unsigned int*)D.hflags)[threadIdx.x] = ld_vol(&D.flags[threadIdx.x]);
    if (!conv) return;
    const int p = blockIdx.x * blockDim.x + threadIdx.x;
    unsigned int writes = 0;
    bool fg = false;
    if (p < D.npx) {
        const int x = p % D.W, y = p / D.W;
        uint32_t w9[9];
#pragma unroll
        for (int k = 0; k < 9; ++k) {
            const int dx = k % 3 - 1, dy = k / 3 - 1;
            const bool ok = y + dy >= 0 && y + dy < D.H && x + dx >= 0 && x + dx < D.W;
            w9[k] = ok ? D.intent[p + dy * D.W + dx] : 0u;
        }
        const uint32_t wp = w9[4];
        const bool valid = (wp & kIValid) != 0;
        fg = valid && (wp & kIFG);
        if (ALG == ALG_VIBE) D.maskOut[p] = fg ? 255 : 0;
        D.kctr[p] = (uint16_t)(valid ? i_draws(wp) : 0);
        if (valid) writes = ((wp & kIOwn) ? 1u : 0u) + ((wp & kINb) ? 1u : 0u);
        // the pixels a write can reach: inside the LBSP border (LOBSTER), the whole frame (ViBe, PBAS)
        constexpr int bord = ALG == ALG_LOBSTER ? kBorder : 0;
        const bool reach = x >= bord && y >= bord && x < D.W - bord && y < D.H - bord;
        unsigned long long list = 0;
        int nwr = 0;
#pragma unroll
        for (int k = 0; k < 9; ++k) {
            const uint32_t w = w9[k];
            if (!reach || !(w & kIValid)) continue;
            if (k == 4 && (w & kIOwn)) {
                if (nwr < 5) list |= (unsigned long long)(2048u | (4u << 6) | (uint32_t)i_sown(w)) << (12 * nwr);
                ++nwr;
            }
            if ((w & kINb) && i_code(w) == 8 - k) {
                if (nwr < 5) list |= (unsigned long long)(((uint32_t)k << 6) | (uint32_t)i_snb(w)) << (12 * nwr);
                ++nwr;
            }
        }
        struct Write {
            unsigned long long d;
            uint32_t c2;
            int s;
        };
        auto read = [&](int k, int s) -> Write {
            // PBAS: every write into pixel p holds p's own colour and gradient
            const int q = ALG == ALG_PBAS ? p : p + (k / 3 - 1) * D.W + k % 3 - 1;
            const uint32_t c2 = ALG == ALG_LOBSTER ? __ldg(D.frame + (size_t)q * C + (C == 3 ? 2 : 0)) : 0u;
            // (an ordinary load: the evaluation, which writes the words, may still run when this kernel's blocks arrive)
            return {D.wD[q], c2, s};
        };
        auto entry = [&](int j) {
            const uint32_t e = (uint32_t)(list >> (12 * j)) & 0xfffu;
            return read((int)((e >> 6) & 15u), (int)(e & 63u));
        };
        // the next write's word is requested before this one is stored (an ordinary load does not pass a store)
        const int nlist = nwr <= 5 ? nwr : 0;
        const int iters = (int)__reduce_max_sync(__activemask(), (unsigned)nlist);
        Write next = nlist > 0 ? entry(0) : Write{0ull, 0u, 0};
        for (int j = 0; j < iters; ++j) {
            const Write w = next;
            if (j + 1 < nlist) next = entry(j + 1);
            if (j < nlist) store_sample<C, ALG>(D, w.s, p, w.d, w.c2);
        }
        auto write = [&](int k, int s) {
            const Write w = read(k, s);
            store_sample<C, ALG>(D, w.s, p, w.d, w.c2);
        };
        if (nwr > 5) {
#pragma unroll 1
            for (int k = 0; k < 9; ++k) {
                const int q = p + (k / 3 - 1) * D.W + k % 3 - 1;
                const int qy = y + k / 3 - 1, qx = x + k % 3 - 1;
                if (qy < 0 || qy >= D.H || qx < 0 || qx >= D.W) continue;
                const uint32_t w = D.intent[q];
                if (!(w & kIValid)) continue;
                if (k == 4 && (w & kIOwn)) write(4, i_sown(w));
                if ((w & kINb) && i_code(w) == 8 - k) write(k, i_snb(w));
            }
        }
    }
    if (ALG != ALG_VIBE) {
        const uint32_t m = __ballot_sync(0xffffffffu, fg);
        if ((threadIdx.x & 31) == 0 && p < D.npx) D.rawBits[p >> 5] = m;
    }
    block_add(&D.stats[1], writes);
}

// cv::medianBlur(raw mask, k) with replicated borders: 255 where more than half of the k*k window is
// set (:577), which becomes the last mask and the output (:578); the frame becomes the last colour
// frame (:580). The raw mask comes as bits of the pixels in order (a warp of the commit writes a word), so a row's
// word is two loads and a shift; one block per tile of kMedW words x kMedH rows counts the row windows and then
// their sums on bit planes, 32 pixels an operation, and writes four pixels a store. With a byte and a count a
// pixel in shared memory and byte copies: 1920x1080 16 us and now 7, 1277x719 BGR 11 us and now 8.
constexpr int kMedW = 4, kMedH = 16, kMedMaxR = 15, kMedRows = kMedH + 2 * kMedMaxR;
struct MedSmem {
    uint32_t raw[kMedRows][kMedW + 2];
    uint32_t h[5][kMedRows][kMedW];
    uint32_t fg[kMedH][kMedW];
};
template <int HB>
__device__ __forceinline__ void lob_median_words(MedSmem& sm, int r, int half) {
    for (int i = threadIdx.x; i < (kMedH + 2 * r) * kMedW; i += kThreadsL) {
        const int y = i / kMedW, w = i % kMedW;
        uint32_t h[HB];
        row_window_planes<HB>(sm.raw[y][w], sm.raw[y][w + 1], sm.raw[y][w + 2], r, h);
#pragma unroll
        for (int b = 0; b < HB; ++b) sm.h[b][y][w] = h[b];
    }
    __syncthreads();
    if (threadIdx.x < kMedH * kMedW) {
        const int y = threadIdx.x / kMedW, w = threadIdx.x % kMedW;
        uint32_t a[2 * HB];
#pragma unroll
        for (int b = 0; b < 2 * HB; ++b) a[b] = 0u;
        for (int j = 0; j <= 2 * r; ++j) {
            uint32_t v[HB];
#pragma unroll
            for (int b = 0; b < HB; ++b) v[b] = sm.h[b][y + j][w];
            add_planes<HB>(a, v);
        }
        sm.fg[y][w] = planes_above<2 * HB>(a, half);
    }
    __syncthreads();
}
template <bool KEEP>
__global__ void __launch_bounds__(kThreadsL) lob_k_median(LobDev D) {
    pdl_entry();
    if (!ld_vol(&D.flags[LOB_F_CONV])) return;
    __shared__ MedSmem sm;
    const int r = D.medianK / 2, t = threadIdx.x, W = D.W;
    const int tilesX = tiles_across(W, 32 * kMedW);
    const int x0 = (int)(blockIdx.x % tilesX) * 32 * kMedW, y0 = (int)(blockIdx.x / tilesX) * kMedH;
    for (int i = t; i < (kMedH + 2 * r) * (kMedW + 2); i += kThreadsL) {
        const int ry = i / (kMedW + 2), x = x0 + 32 * (i % (kMedW + 2) - 1);
        const int row = clampi(y0 - r + ry, 0, D.H - 1) * W;
        auto bits = [&](int p) {  // 32 pixels from p on (the plane has a word past the frame)
            return __funnelshift_r(__ldcg(&D.rawBits[p >> 5]), __ldcg(&D.rawBits[(p >> 5) + 1]), p & 31);
        };
        uint32_t v;
        if (x < 0) {
            v = (bits(row) & 1u) ? 0xffffffffu : 0u;
        } else {
            const uint32_t last = (bits(row + W - 1) & 1u) ? 0xffffffffu : 0u, in = x + 32 <= W ? 0xffffffffu : x < W ? (1u << (W - x)) - 1u : 0u;
            v = x < W ? (bits(row + x) & in) | (last & ~in) : last;
        }
        sm.raw[ry][i % (kMedW + 2)] = v;
    }
    __syncthreads();
    // 2 * sum > k * k
    if (r < 8) lob_median_words<4>(sm, r, D.medianK * D.medianK / 2);
    else lob_median_words<5>(sm, r, D.medianK * D.medianK / 2);
    const int y = y0 + t / 16, len = min(32 * kMedW, W - x0);
    if (y < D.H) {
        // 16 threads a row; aligned words whatever the width, the row's first and last in bytes
        auto put = [&](uint8_t* plane) {
            uint8_t* out = plane + (size_t)y * W + x0;
            const int off = (int)((uintptr_t)out & 3);
            for (int i = t % 16; 4 * i - off < len; i += 16) {
                const int b = 4 * i - off;  // from -3 on
                const uint32_t lo = b >= 0 ? sm.fg[t / 16][b >> 5] : 0u, hi = b < 32 * (kMedW - 1) ? sm.fg[t / 16][(b >> 5) + 1] : 0u;
                const uint32_t v = (((__funnelshift_r(lo, hi, b & 31) & 15u) * 0x00204081u) & 0x01010101u) * 255u;
                if (b >= 0 && b + 4 <= len) {
                    *(uint32_t*)(out + b) = v;
                } else {
                    for (int j = max(0, -b); j < 4 && b + j < len; ++j) out[b + j] = (uint8_t)(v >> (8 * j));
                }
            }
        };
        put(D.maskOut);
        if (KEEP) put(D.lastFG);  // PBAS keeps neither
    }
    if (KEEP) {
        const size_t bytes = (size_t)D.npx * D.C, g = (size_t)blockIdx.x * kThreadsL + t;
        const size_t threads = (size_t)gridDim.x * kThreadsL;
        // lastColor is aligned; a frame at any address is read as the aligned words that lie wholly inside it
        const uint32_t sh = 8u * (uint32_t)((uintptr_t)D.frame & 3);
        const uint32_t* src = (const uint32_t*)((uintptr_t)D.frame & ~(uintptr_t)3);
        size_t first = 0, end = bytes / 4;  // words of lastColor
        if (sh) {
            first = 1;
            end = bytes >= 12 ? (bytes - 8) / 4 + 1 : 1;
        }
        for (size_t i = first + g; i < end; i += threads)
            ((uint32_t*)D.lastColor)[i] = sh ? __funnelshift_r(__ldg(src + i), __ldg(src + i + 1), sh) : __ldg(src + i);
        for (size_t i = g; i < 4 * first + (bytes - 4 * end); i += threads) {
            const size_t j = i < 4 * first ? i : 4 * end + i - 4 * first;
            if (j < bytes) D.lastColor[j] = __ldg(D.frame + j);
        }
    }
}

// initialize() (:442-457 with BackgroundSubtractionUtils.cpp:70-155, BackgroundSubtractorLBSP.cpp:21-65):
// last colour frame = the ROI part of the frame, last descriptors of the strict interior ROI pixels
template <int C>
__global__ void __launch_bounds__(kThreadsL) lob_k_init(LobDev D, const uint8_t* img) {
    const int p = blockIdx.x * blockDim.x + threadIdx.x;
    if (p >= D.npx) return;
    const int x = p % D.W, y = p / D.W;
    const bool in = D.roi[p] != 0;
    const bool desc = in && x > kBorder && y > kBorder && x < D.W - kBorder && y < D.H - kBorder;
#pragma unroll
    for (int c = 0; c < C; ++c) {
        const uint32_t v = __ldg(img + (size_t)p * C + c);
        D.lastColor[(size_t)p * C + c] = in ? (uint8_t)v : 0;
        uint16_t d = 0;
        if (desc) {
            uint32_t t[4];
            taps<C>(img, D.W, p, c, t);
            d = (uint16_t)lbsp_thr(t, v, __ldg(D.lut + v));
        }
        D.lastDesc[(size_t)p * C + c] = d;
    }
    D.lastFG[p] = 0;
    D.kctr[p] = 0;
}

// ViBe's initialize() (BackgroundSubtractorViBe.cpp:57-75 / :112-134): sample s of every pixel from a
// 7x7 Gaussian position of the frame clamped to the frame (draw s of the pixel in frame 0)
template <int C>
__global__ void __launch_bounds__(kThreadsL) lob_k_vibe_init(LobDev D, const uint8_t* img) {
    const int p = blockIdx.x * blockDim.x + threadIdx.x;
    if (p >= D.npx) return;
    const int x0 = p % D.W, y0 = p / D.W;
    Draws ds;
    ds.blk = 0xffffffffu;
    for (int s = 0; s < D.N; ++s) {
        int r = 1 + (int)(draw(D, (uint32_t)p, (uint32_t)s, ds) % 512u);
        int sx = 0, sy = 0;
        for (int i = 0; i < 49; ++i) {
            r -= c_lob_pat7[i];
            if (r <= 0) {
                sy = i / 7;
                sx = i % 7;
                break;
            }
        }
        sx = clampi(sx + x0 - 3, 0, D.W - 1);
        sy = clampi(sy + y0 - 3, 0, D.H - 1);
        const uint8_t* src = img + ((size_t)sy * D.W + sx) * C;
        unsigned long long d = 0;
#pragma unroll
        for (int c = 0; c < C; ++c) d |= (unsigned long long)__ldg(src + c) << (8 * c);
        store_sample<C, ALG_VIBE>(D, s, p, d, 0u);
    }
}

// ---- PBAS (BackgroundSubtractorPBAS.cpp) ----

__device__ __forceinline__ int reflect101(int i, int n) {
    if (n == 1) return 0;
    while (i < 0 || i >= n) i = i < 0 ? -i : 2 * n - 2 - i;
    return i;
}

// The gradient image of a frame (:127-135 / :338-346): GaussianBlur 3x3 (sigma 0), the separable [1 2 1] / 4
// kernel in 8-bit fixed point, (sum + 8) >> 4; the Scharr derivatives ([-3 0 3; -10 0 10; -3 0 3] and its
// transpose), convertScaleAbs (|v| saturated to 255) and addWeighted(0.5, 0.5) ((a + b) * 0.5 rounded half to
// even), all with BORDER_REFLECT_101. One block per tile of kGradW x kGradH pixels: the frame tile with its
// reflected 2-pixel halo in shared memory, blurred there with a 1-pixel halo (both kernels are symmetric, so
// the blur of a reflected position is the reflected blur), then the derivatives; four bytes at a time, two per
// word in 16 bits (the sums are at most 16 * 255). Bytes of a channel are C apart in the interleaved rows. The
// blur went through memory before, a byte and nine loads a thread: 30 + 38 us on a 1920x1080 BGR frame, 34 with tiles
// loaded by bytes, 25 with words.
constexpr int kGradW = 64, kGradH = 16;
template <int C>
struct GradTile {
    static constexpr int kPad = 8;                                   // bytes before the tile's first pixel
    static constexpr int kRow = (kPad + (kGradW + 2) * C + 4 + 3) / 4;  // words of a row
    uint32_t src[kGradH + 4][kRow], blur[kGradH + 2][kRow];
};
// bytes b .. b + 3 of a shared row (any byte offset), and their spread to two 16-bit pairs
__device__ __forceinline__ uint32_t row4(const uint32_t* row, int b) {
    return __funnelshift_r(row[b >> 2], row[(b >> 2) + 1], 8 * (b & 3));
}
__device__ __forceinline__ uint32_t even2(uint32_t w) { return w & 0x00ff00ffu; }
__device__ __forceinline__ uint32_t odd2(uint32_t w) { return (w >> 8) & 0x00ff00ffu; }
template <int C>
__global__ void __launch_bounds__(kThreadsL) pbas_k_grad(LobDev D, const uint8_t* img) {
    using T = GradTile<C>;
    __shared__ T sm;
    const int tilesX = tiles_across(D.W, kGradW), t = threadIdx.x;
    const int x0 = (int)(blockIdx.x % tilesX) * kGradW, y0 = (int)(blockIdx.x / tilesX) * kGradH;
    // frame bytes of rows y0 - 2 .. y0 + 17, pixels x0 - 2 .. x0 + 65, from byte kPad - 2 C of a row on
    constexpr int kBytes = (kGradW + 4) * C;
    // inside the frame's width a tile row is kRow aligned words from byte x0 C - kPad on (x0 C is a multiple of 64)
    const long b0 = (long)x0 * C - T::kPad, rowBytes = (long)D.W * C;
    const bool words = b0 >= 0 && b0 + 4 * T::kRow <= rowBytes && ((rowBytes | (uintptr_t)img) & 3) == 0;
    if (words) {
        for (int i = t; i < (kGradH + 4) * T::kRow; i += kThreadsL) {
            const int r = i / T::kRow, w = i % T::kRow, gy = reflect101(y0 - 2 + r, D.H);
            sm.src[r][w] = __ldg((const uint32_t*)(img + (size_t)gy * rowBytes + b0) + w);
        }
    } else {
        for (int i = t; i < (kGradH + 4) * kBytes; i += kThreadsL) {
            const int r = i / kBytes, b = i % kBytes;
            const int gy = reflect101(y0 - 2 + r, D.H), gx = reflect101(x0 - 2 + b / C, D.W);
            ((uint8_t*)sm.src[r])[T::kPad - 2 * C + b] = __ldg(img + ((size_t)gy * D.W + gx) * C + b % C);
        }
    }
    __syncthreads();
    // blur of rows y0 - 1 .. y0 + 16, pixels x0 - 1 .. x0 + 64, in words from byte kFirst on
    constexpr int kFirst = (T::kPad - C) / 4 * 4, kBlurW = (T::kPad + (kGradW + 1) * C - kFirst + 3) / 4;
    for (int i = t; i < (kGradH + 2) * kBlurW; i += kThreadsL) {
        const int r = i / kBlurW, b = kFirst + 4 * (i % kBlurW);
        uint32_t e = 0x00080008u, o = 0x00080008u;
#pragma unroll
        for (int j = 0; j < 3; ++j) {
            const uint32_t* row = sm.src[r + j];
            const uint32_t L = row4(row, b - C), M = row[b >> 2], R = row4(row, b + C);
            const uint32_t he = even2(L) + 2u * even2(M) + even2(R), ho = odd2(L) + 2u * odd2(M) + odd2(R);
            e += j == 1 ? 2u * he : he;
            o += j == 1 ? 2u * ho : ho;
        }
        sm.blur[r][b >> 2] = ((e >> 4) & 0x00ff00ffu) | (((o >> 4) & 0x00ff00ffu) << 8);
    }
    __syncthreads();
    constexpr int kOutW = kGradW * C / 4;
    for (int i = t; i < kGradH * kOutW; i += kThreadsL) {
        const int r = i / kOutW, k = 4 * (i % kOutW), b = T::kPad + k;
        if (y0 + r >= D.H) break;
        uint32_t l[3], c[3], h[3];  // the rows' words to the left, at and to the right of the four bytes
#pragma unroll
        for (int j = 0; j < 3; ++j) {
            const uint32_t* row = sm.blur[r + j];
            l[j] = row4(row, b - C);
            c[j] = row[b >> 2];
            h[j] = row4(row, b + C);
        }
        uint32_t out = 0;
#pragma unroll
        for (int half = 0; half < 2; ++half) {
            auto u = [&](uint32_t w) { return half ? odd2(w) : even2(w); };
            const uint32_t colL = 3u * (u(l[0]) + u(l[2])) + 10u * u(l[1]), colR = 3u * (u(h[0]) + u(h[2])) + 10u * u(h[1]);
            const uint32_t top = 3u * (u(l[0]) + u(h[0])) + 10u * u(c[0]), bot = 3u * (u(l[2]) + u(h[2])) + 10u * u(c[2]);
            const uint32_t sum = __vminu2(__vabsdiffu2(colR, colL), 0x00ff00ffu) + __vminu2(__vabsdiffu2(bot, top), 0x00ff00ffu);
            const uint32_t hf = (sum >> 1) & 0x00ff00ffu;
            out |= (hf + (sum & hf & 0x00010001u)) << (8 * half);
        }
        const int left = (D.W - x0) * C - k;  // bytes of the frame row from here on
        uint8_t* dst = D.grad + ((size_t)(y0 + r) * D.W + x0) * C + k;
        if (left >= 4 && ((uintptr_t)dst & 3) == 0) {
            *(uint32_t*)dst = out;
        } else {
            for (int q = 0; q < min(left, 4); ++q) dst[q] = (uint8_t)(out >> (8 * q));
        }
    }
}

// PBAS's initialize() (:61-109 / :287-324): R = 1, T = the default update rate, D = 0 in the maps of
// parity 0, the mean gradient distance mean0 (20, or the last one), and sample s of every pixel (colour and gradient) from a 7x7
// Gaussian position of the frame clamped to the frame (draw s of the pixel in frame 0)
template <int C>
__global__ void __launch_bounds__(kThreadsL) pbas_k_init(LobDev D, const uint8_t* img, float mean0) {
    const int p = blockIdx.x * blockDim.x + threadIdx.x;
    if (p >= D.npx) return;
    const size_t npx = (size_t)D.npx;
    D.fm[p] = 1.0f;
    D.fm[npx + p] = D.updateRate;
    D.fm[2 * npx + p] = 0.0f;
    if (p == 0) *D.meanGrad = mean0;
    const int x0 = p % D.W, y0 = p / D.W;
    Draws ds;
    ds.blk = 0xffffffffu;
    for (int s = 0; s < D.N; ++s) {
        int r = 1 + (int)(draw(D, (uint32_t)p, (uint32_t)s, ds) % 512u);
        int sx = 0, sy = 0;
        for (int i = 0; i < 49; ++i) {
            r -= c_lob_pat7[i];
            if (r <= 0) {
                sy = i / 7;
                sx = i % 7;
                break;
            }
        }
        sx = clampi(sx + x0 - 3, 0, D.W - 1);
        sy = clampi(sy + y0 - 3, 0, D.H - 1);
        const size_t src = ((size_t)sy * D.W + sx) * C;
        unsigned long long d = 0;
#pragma unroll
        for (int c = 0; c < C; ++c)
            d |= ((unsigned long long)__ldg(img + src + c) << (8 * c)) | ((unsigned long long)D.grad[src + c] << (24 + 8 * c));
        store_sample<C, ALG_PBAS>(D, s, p, d, 0u);
    }
}

// the frame-level mean gradient distance of the bad samples, single channel (:232): the size_t sum
// of their gradient distances and their count (which starts at 1), per block into two counters
__global__ void __launch_bounds__(kThreadsL) pbas_k_mean1(LobDev D) {
    pdl_entry();
    if (!ld_vol(&D.flags[LOB_F_CONV])) return;
    unsigned long long sum = 0, cnt = 0;
    for (int p = blockIdx.x * blockDim.x + threadIdx.x; p < D.npx; p += gridDim.x * blockDim.x) {
        sum += D.badSum[p];
        cnt += D.badCnt[p];
    }
    for (int o = 16; o > 0; o >>= 1) {
        sum += __shfl_xor_sync(0xffffffffu, sum, o);
        cnt += __shfl_xor_sync(0xffffffffu, cnt, o);
    }
    if ((threadIdx.x & 31) == 0) {
        if (sum) atomicAdd(&D.stats[2], sum);
        if (cnt) atomicAdd(&D.stats[3], cnt);
    }
}
__global__ void pbas_k_mean1_end(LobDev D) {
    pdl_entry();
    if (!ld_vol(&D.flags[LOB_F_CONV])) return;
    const float mean = (float)D.stats[2] / (float)(D.stats[3] + 1ull);
    *D.meanGrad = mean > 20.0f ? mean : 20.0f;
}

// three channels (:460): the float sum of the bad samples' gradient distances in raster order (pixel,
// then scan order), s <- RN(s + v) value after value. The values are non-negative, so s only grows, and
// while s stays in one binade [2^e, 2^(e+1)) with ulp u = 2^(e-23), RN(s + v) = s + u * q where q is
// v / u rounded to an integer: up when the fraction is above 1/2, down when below, and on an exact 1/2
// to the even quotient, which depends on the parity of s / u. The sum over a chunk of values is
// therefore a function of that parity only: a transfer (d0, d1), the increment in ulps for an even or
// odd start, composed value by value (d'_p = d_p + d2_{(p + d_p) & 1}).
//   lob_k_eval: about how much each chunk of 256 pixels adds, before the repairs;
//   pbas_k_sum_scan: the exclusive prefix of that, which predicts the binade of s at each chunk's start;
//   pbas_k_sum_tr: the transfers of each chunk, and of its 32-pixel granules, for the predicted binade and
//     the two beside it;
//   pbas_k_sum_win: those of each window of 32 chunks, composed from its chunks';
//   pbas_k_sum_walk: from s = 0, one warp over the windows, as many at once as have transfers for the binade of
//     s and keep s in it; where s crosses into the next binade (or the prediction was off), the same over that
//     window's chunks, over that chunk's granules, and value by value over that granule.
// 1920x1080 BGR: 8 + 46 + 3 + 59 us, the first beside the repairs, the others beside the commit, the median and the
// mask's copy. A frame is over when both streams are: one handle's frames take 289 us back to back (253 us when a frame's
// mean was left to run beside the next frame's upload and gradient, after the call had returned).
// The result is the sequential sum bit for bit. An increment of 2^24 ulps leaves the binade whatever the start,
// so transfers saturate at 2^25 and fit 32 bits.
constexpr int kSumChunk = 256, kSumNB = 3, kSumEMin = 10, kSumScan = 1024;
static_assert(kSumChunk == kThreadsL, "a block of the evaluation is a chunk");
constexpr uint32_t kTrSat = 1u << 25;
struct Tr {
    uint32_t d0, d1;
};
__device__ __forceinline__ Tr tr_then(Tr a, Tr b) {
    Tr r;
    r.d0 = min(a.d0 + ((a.d0 & 1u) ? b.d1 : b.d0), kTrSat);
    r.d1 = min(a.d1 + ((a.d1 & 1u) ? b.d0 : b.d1), kTrSat);
    return r;
}
// The sums after one more value in binades e, e + 1, .. (e >= 10, the value 0 or in [1, 256)), from an even start
// (a[b].d0) and an odd one (a[b].d1, counted from 1): the value is m 2^-sh ulps, and adding half an ulp less
// one, plus the parity of the floor of the sum, rounds to the nearest and halves to even.
__device__ __forceinline__ void tr_add(Tr (&a)[3], float v, int e) {
    const uint32_t bits = __float_as_uint(v), m = v > 0.0f ? (bits & 0x7fffffu) | 0x800000u : 0u;
    int sh = min(e + 127 - (int)(bits >> 23), 29);  // from 26 on every value vanishes
    uint32_t half = 1u << (sh - 1);
#pragma unroll
    for (int b = 0; b < 3; ++b, ++sh, half <<= 1) {
        const uint32_t q = m >> sh, t = m + half - 1u;
        a[b].d0 += (t + ((a[b].d0 ^ q) & 1u)) >> sh;
        a[b].d1 += (t + ((a[b].d1 ^ q) & 1u)) >> sh;
    }
}
// binade of a positive float
__device__ __forceinline__ int binade(float s) { return (int)((__float_as_uint(s) >> 23) & 0xffu) - 127; }
// s after a transfer, when s >= 1024 and the transfer keeps s in its binade
__device__ __forceinline__ bool tr_apply(float& s, Tr t) {
    if (s < 1024.0f) return false;
    const uint32_t bits = __float_as_uint(s), m = (bits & 0x7fffffu) | 0x800000u;
    const uint32_t m2 = m + ((m & 1u) ? t.d1 : t.d0);
    if (m2 + 1u >= (1u << 24)) return false;
    s = __uint_as_float((bits & 0xff800000u) | (m2 & 0x7fffffu));
    return true;
}

constexpr int kSumGran = kSumChunk / 32;
struct SumWork {
    float* about;  // [nChunks], then their exclusive prefix
    Tr* tr;        // [nChunks][kSumNB]
    Tr* trw;       // [nChunks][kSumGran][kSumNB]: the transfers of each chunk's 32-pixel granules
    Tr* win;       // [nWin][kSumNB]: of each window of 32 chunks
    int* eb;       // [nChunks]: the first of the chunk's binades
    int* winEb;    // [nWin]: the first of the window's binades << 3 | which of the three all its chunks have
    static size_t bytes(size_t nChunks) {
        const size_t nWin = (nChunks + 31) / 32;
        return nChunks * (2 * 4 + (1 + kSumGran) * kSumNB * sizeof(Tr)) + nWin * (kSumNB * sizeof(Tr) + 4);
    }
};
inline SumWork sum_work(void* base, size_t nChunks) {
    const size_t nWin = (nChunks + 31) / 32;
    SumWork W;
    W.tr = (Tr*)base;
    W.trw = W.tr + nChunks * kSumNB;
    W.win = W.trw + nChunks * kSumGran * kSumNB;
    W.about = (float*)(W.win + nWin * kSumNB);
    W.eb = (int*)(W.about + nChunks);
    W.winEb = W.eb + nChunks;
    return W;
}
// the k-th bad sample's gradient distance of pixel p
__device__ __forceinline__ float bad_dist(const LobDev& D, int k, int p) { return root16(bad_value(D, k, p)); }

__global__ void __launch_bounds__(kSumScan) pbas_k_sum_scan(SumWork W, int nChunks) {
    pdl_entry();
    __shared__ float sm[kSumScan / 32];
    const int t = threadIdx.x, lane = t & 31, warp = t >> 5, per = (nChunks + kSumScan - 1) / kSumScan;
    const int c0 = min(t * per, nChunks), c1 = min(c0 + per, nChunks);
    float own = 0.0f;
#pragma unroll 8
    for (int c = c0; c < c1; ++c) own += W.about[c];
    float inc = own;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const float y = __shfl_up_sync(0xffffffffu, inc, o);
        if (lane >= o) inc += y;
    }
    if (lane == 31) sm[warp] = inc;
    __syncthreads();
    if (warp == 0) {
        const float v = sm[lane];
        float i2 = v;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const float y = __shfl_up_sync(0xffffffffu, i2, o);
            if (lane >= o) i2 += y;
        }
        sm[lane] = i2 - v;
    }
    __syncthreads();
    float run = sm[warp] + inc - own;
    for (int c = c0; c < c1; ++c) {
        const float v = W.about[c];
        W.about[c] = run;
        run += v;
    }
}

// A warp takes a granule of 32 pixels: their values, in order, are split evenly over its lanes (a foreground pixel
// has up to N, most have none or a few), each lane composes its own run, and the runs are composed in order.
__global__ void __launch_bounds__(kSumChunk) pbas_k_sum_tr(LobDev D, SumWork W) {
    pdl_entry();
    if (!ld_vol(&D.flags[LOB_F_CONV])) return;
    __shared__ Tr sm[kSumGran][kSumNB];
    __shared__ int first[kSumGran][33];
    const int t = threadIdx.x, lane = t & 31, wid = t >> 5;
    const int p0 = blockIdx.x * kSumChunk + 32 * wid, p = p0 + lane;
    const int n = p < D.npx ? (int)D.badCnt[p] : 0;
    int inc = n;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const int y = __shfl_up_sync(0xffffffffu, inc, o);
        if (lane >= o) inc += y;
    }
    first[wid][lane + 1] = inc;
    if (lane == 0) first[wid][0] = 0;
    __syncwarp();
    const int total = __shfl_sync(0xffffffffu, inc, 31), per = (total + 31) / 32;
    const float pre = W.about[blockIdx.x];
    const int e0 = max(pre >= 1.0f ? binade(pre) - 1 : kSumEMin, kSumEMin);
    Tr acc[kSumNB];  // a lane adds at most 64 values of 2^21 ulps: no overflow
#pragma unroll
    for (int j = 0; j < kSumNB; ++j) acc[j] = {0u, 1u};
    const int i0 = min(lane * per, total), i1 = min(i0 + per, total);
    if (i0 < i1) {
        int q = 0;  // the pixel of value i0: the last one whose first value is at most i0
#pragma unroll
        for (int step = 16; step > 0; step >>= 1)
            if (first[wid][q + step] <= i0) q += step;
        int k = i0 - first[wid][q], left = first[wid][q + 1] - i0;
        for (int i = i0; i < i1;) {
            const int m = min(min(left, i1 - i), 4);  // values of this pixel in flight together
            float x[4];
#pragma unroll
            for (int j = 0; j < 4; ++j) x[j] = j < m ? bad_dist(D, k + j, p0 + q) : 0.0f;
#pragma unroll
            for (int j = 0; j < 4; ++j)
                if (j < m) tr_add(acc, x[j], e0);
            i += m;
            k += m;
            left -= m;
            while (left == 0 && i < i1) {
                ++q;
                k = 0;
                left = first[wid][q + 1] - first[wid][q];
            }
        }
    }
    __syncwarp();
    // ordered reduction: lane 0 of each warp, then the warps in order
#pragma unroll
    for (int j = 0; j < kSumNB; ++j) {
        acc[j].d1 -= 1u;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            Tr y;
            y.d0 = __shfl_down_sync(0xffffffffu, acc[j].d0, o);
            y.d1 = __shfl_down_sync(0xffffffffu, acc[j].d1, o);
            if ((lane & (2 * o - 1)) == 0) acc[j] = tr_then(acc[j], y);
        }
        if (lane == 0) {
            sm[wid][j] = acc[j];
            W.trw[((size_t)blockIdx.x * kSumGran + wid) * kSumNB + j] = acc[j];
        }
    }
    __syncthreads();
    if (t < kSumNB) {
        Tr r = sm[0][t];
        for (int w = 1; w < kSumGran; ++w) r = tr_then(r, sm[w][t]);
        W.tr[(size_t)blockIdx.x * kSumNB + t] = r;
        if (t == 0) W.eb[blockIdx.x] = e0;
    }
    block_add(&D.stats[3], (unsigned int)n);
}

// the transfers of a window of 32 chunks, one warp each, for three binades from its first chunk's on
__global__ void __launch_bounds__(256) pbas_k_sum_win(LobDev D, SumWork W, int nChunks) {
    pdl_entry();
    if (!ld_vol(&D.flags[LOB_F_CONV])) return;
    const int w = blockIdx.x * 8 + (threadIdx.x >> 5), lane = threadIdx.x & 31, c = 32 * w + lane;
    if (32 * w >= nChunks) return;
    const bool in = c < nChunks;
    const int eb = in ? W.eb[c] : 0, e0 = __shfl_sync(0xffffffffu, eb, 0);
    Tr t[kSumNB];
#pragma unroll
    for (int i = 0; i < kSumNB; ++i) t[i] = in ? W.tr[(size_t)c * kSumNB + i] : Tr{0u, 0u};
    int have = 0;
#pragma unroll
    for (int j = 0; j < kSumNB; ++j) {
        const int k = e0 + j - eb;
        Tr a = {0u, 0u};
#pragma unroll
        for (int i = 0; i < kSumNB; ++i)
            if (in && k == i) a = t[i];
        if (__all_sync(0xffffffffu, !in || (k >= 0 && k < kSumNB))) have |= 1 << j;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            Tr y;
            y.d0 = __shfl_down_sync(0xffffffffu, a.d0, o);
            y.d1 = __shfl_down_sync(0xffffffffu, a.d1, o);
            if ((lane & (2 * o - 1)) == 0) a = tr_then(a, y);
        }
        if (lane == 0) W.win[(size_t)w * kSumNB + j] = a;
    }
    if (lane == 0) W.winEb[w] = (e0 << 3) | have;
}

// Advances s over the elements pos .. cnt - 1 of a warp's 32 (element l on lane l: transfers t for the binades eb,
// eb + 1, eb + 2 as far as `have` says), as far as transfers for the binade of s exist and keep s in it: an
// inclusive scan composes them, and a ballot finds how many fit. Returns the element it stopped at.
__device__ int tr_run(float& s, const Tr (&t)[kSumNB], int eb, int have, int cnt, int pos) {
    const int lane = threadIdx.x & 31;
    while (pos < cnt && s >= 1024.0f) {
        const int k = binade(s) - eb;
        const bool usable = lane >= pos && lane < cnt && k >= 0 && k < kSumNB && ((have >> k) & 1);
        const unsigned m = __ballot_sync(0xffffffffu, usable) >> pos;
        const int run = ~m ? __ffs(~m) - 1 : 32;
        if (run == 0) break;
        Tr a = {0u, 0u};
#pragma unroll
        for (int i = 0; i < kSumNB; ++i)
            if (lane >= pos && lane < pos + run && k == i) a = t[i];
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            Tr y;
            y.d0 = __shfl_up_sync(0xffffffffu, a.d0, o);
            y.d1 = __shfl_up_sync(0xffffffffu, a.d1, o);
            if (lane >= o) a = tr_then(y, a);
        }
        float mine = s;
        const bool fits = lane >= pos && lane < pos + run && tr_apply(mine, a);
        const unsigned f = __ballot_sync(0xffffffffu, fits) >> pos;  // the increments grow: a prefix fits
        const int n = ~f ? __ffs(~f) - 1 : 32;
        if (n == 0) break;
        s = __shfl_sync(0xffffffffu, mine, pos + n - 1);
        pos += n;
        if (n < run) break;
    }
    return pos;
}

// the walk (one warp; every lane holds the same sum), then the mean and its floor of 20
__global__ void __launch_bounds__(32) pbas_k_sum_walk(LobDev D, SumWork W, int nChunks) {
    pdl_entry();
    if (!ld_vol(&D.flags[LOB_F_CONV])) return;
    __shared__ __align__(16) float vals[32 * kMaxSamples];
    __shared__ int first[33];
    const int lane = threadIdx.x, nWin = (nChunks + 31) / 32;
    float s = 0.0f;
    Tr tn[kSumNB];
    int en = 0;
    auto fetch = [&](int w) {
        en = w < nWin ? W.winEb[w] : 0;
#pragma unroll
        for (int i = 0; i < kSumNB; ++i) tn[i] = w < nWin ? W.win[(size_t)w * kSumNB + i] : Tr{0u, 0u};
    };
    fetch(lane);
    for (int w0 = 0; w0 < nWin; w0 += 32) {
        Tr tw[kSumNB];
#pragma unroll
        for (int i = 0; i < kSumNB; ++i) tw[i] = tn[i];
        const int ew = en, wcnt = min(32, nWin - w0);
        fetch(w0 + 32 + lane);  // the next 32 windows while these are walked
        for (int wp = 0; wp < wcnt; ++wp) {
            wp = tr_run(s, tw, ew >> 3, ew & 7, wcnt, wp);
            if (wp >= wcnt) break;
            // window wp chunk by chunk
            const int c0 = 32 * (w0 + wp), c = c0 + lane, ccnt = min(32, nChunks - c0);
            Tr tc[kSumNB];
            const int ec = c < nChunks ? W.eb[c] : 0;
#pragma unroll
            for (int i = 0; i < kSumNB; ++i) tc[i] = c < nChunks ? W.tr[(size_t)c * kSumNB + i] : Tr{0u, 0u};
            for (int cp = 0; cp < ccnt; ++cp) {
                cp = tr_run(s, tc, ec, 7, ccnt, cp);
                if (cp >= ccnt) break;
                // chunk cp granule by granule
                const int chunk = c0 + cp, eg = __shfl_sync(0xffffffffu, ec, cp);
                const int pEnd = min((chunk + 1) * kSumChunk, D.npx);
                const int gcnt = (pEnd - chunk * kSumChunk + 31) / 32;
                Tr tg[kSumNB];
#pragma unroll
                for (int i = 0; i < kSumNB; ++i)
                    tg[i] = lane < gcnt ? W.trw[((size_t)chunk * kSumGran + lane) * kSumNB + i] : Tr{0u, 0u};
                int cnt8[kSumGran];  // the value counts of the chunk's pixels, requested with its transfers
#pragma unroll
                for (int i = 0; i < kSumGran; ++i) {
                    const int p = chunk * kSumChunk + 32 * i + lane;
                    cnt8[i] = p < pEnd ? (int)D.badCnt[p] : 0;
                }
                for (int g = 0; g < gcnt; ++g) {
                    g = tr_run(s, tg, eg, 7, gcnt, g);
                    if (g >= gcnt) break;
                    // value by value: the granule's values staged in shared memory, every lane adding them in order
                    int off = 0;
#pragma unroll
                    for (int i = 0; i < kSumGran; ++i)
                        if (g == i) off = cnt8[i];
#pragma unroll
                    for (int o = 1; o < 32; o <<= 1) {
                        const int y = __shfl_up_sync(0xffffffffu, off, o);
                        if (lane >= o) off += y;
                    }
                    first[lane + 1] = off;
                    if (lane == 0) first[0] = 0;
                    __syncwarp();
                    const int total = first[32], padded = (total + 31) & ~31;  // adding 0 changes nothing
#pragma unroll 4
                    for (int i = lane; i < padded; i += 32) {
                        int q = 0;
#pragma unroll
                        for (int step = 16; step > 0; step >>= 1)
                            if (first[q + step] <= i) q += step;
                        vals[i] = i < total ? bad_dist(D, i - first[q], chunk * kSumChunk + 32 * g + q) : 0.0f;
                    }
                    __syncwarp();
                    for (int q = 0; q < padded; q += 32) {
                        float4 v[8];
#pragma unroll
                        for (int i = 0; i < 8; ++i) v[i] = *(const float4*)&vals[q + 4 * i];
#pragma unroll
                        for (int i = 0; i < 8; ++i) s = (((s + v[i].x) + v[i].y) + v[i].z) + v[i].w;
                    }
                    __syncwarp();
                }
            }
        }
    }
    if (lane == 0) {
        const float mean = s / (float)(D.stats[3] + 1ull);
        *D.meanGrad = mean > 20.0f ? mean : 20.0f;
    }
}

// refreshModel(frac, force) (:410-440): samples [start, start+nref) of every ROI pixel (not in the last
// foreground unless forced) from a 7x7 Gaussian position of the last colour frame, with its descriptor,
// which also goes to the last descriptor frame (:427-433); the draws continue the frame's counters
template <int C>
__global__ void __launch_bounds__(kThreadsL) lob_k_refresh(LobDev D, int start, int nref, int force) {
    const int p = blockIdx.x * blockDim.x + threadIdx.x;
    if (p >= D.npx || !D.roi[p]) return;
    if (!force && D.lastFG[p]) return;
    const int x0 = p % D.W, y0 = p / D.W;
    uint32_t k = D.kctr[p];
    Draws ds;
    ds.blk = 0xffffffffu;
    for (int s = start; s < start + nref; ++s) {
        int r = 1 + (int)(draw(D, (uint32_t)p, k++, ds) % 512u);
        int sx = 0, sy = 0;
        for (int i = 0; i < 49; ++i) {
            r -= c_lob_pat7[i];
            if (r <= 0) {
                sy = i / 7;
                sx = i % 7;
                break;
            }
        }
        sx = clampi(sx + x0 - 3, kBorder, D.W - kBorder - 1);
        sy = clampi(sy + y0 - 3, kBorder, D.H - kBorder - 1);
        const int sp = sy * D.W + sx;
        if (!force && D.lastFG[sp]) continue;
        const int rs = s % D.N;
        unsigned long long wd = 0;
        uint32_t col[C];
#pragma unroll
        for (int c = 0; c < C; ++c) {
            col[c] = D.lastColor[(size_t)sp * C + c];
            uint32_t t[4];
            taps<C>(D.lastColor, D.W, sp, c, t);
            const uint16_t d = (uint16_t)lbsp_thr(t, col[c], __ldg(D.lut + col[c]));
            D.lastDesc[(size_t)sp * C + c] = d;
            wd |= (unsigned long long)d << (16 * c);
        }
        const size_t o = (size_t)rs * D.npx + p;
        if (C == 3) {
            ((unsigned long long*)D.sD)[o] = wd | ((unsigned long long)col[0] << 48) | ((unsigned long long)col[1] << 56);
            D.sC[o] = (uint8_t)col[2];
        } else {
            ((uint16_t*)D.sD)[o] = (uint16_t)wd;
            D.sC[o] = (uint8_t)col[0];
        }
    }
    D.kctr[p] = (uint16_t)k;
}

// getBackgroundImage / getBackgroundDescriptorsImage (:583-620): per channel the float sum of
// sample / N in sample order, converted with rounding and saturation
template <int C>
__global__ void lob_k_background(LobDev D, void* out, int descriptors) {
    const size_t n = (size_t)D.npx * C;
    for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x) {
        const int p = (int)(i / C), c = (int)(i % C);
        float acc = 0.0f;
        for (int s = 0; s < D.N; ++s) {
            const size_t o = (size_t)s * D.npx + p;
            uint32_t v;
            if (D.alg != ALG_LOBSTER) {
                unsigned long long d;
                uint32_t c2;
                if (D.alg == ALG_VIBE) load_sample<C, ALG_VIBE>(D, s, p, d, c2);
                else load_sample<C, ALG_PBAS>(D, s, p, d, c2);
                v = (uint32_t)(d >> (8 * c)) & 0xffu;
            } else if (descriptors) {
                v = C == 3 ? (uint32_t)(((const unsigned long long*)D.sD)[o] >> (16 * c)) & 0xffffu
                           : ((const uint16_t*)D.sD)[o];
            } else if (C == 3 && c < 2) {
                v = (uint32_t)(((const unsigned long long*)D.sD)[o] >> (48 + 8 * c)) & 0xffu;
            } else {
                v = D.sC[o];
            }
            acc += (float)v / (float)D.N;
        }
        const int r = __float2int_rn(acc);
        if (descriptors) ((uint16_t*)out)[i] = (uint16_t)clampi(r, 0, 65535);
        else ((uint8_t*)out)[i] = (uint8_t)clampi(r, 0, 255);
    }
}

// the sample planes in the reference's layout ([N][H*W*C] colours; what 1: descriptors, 2: PBAS's gradients)
template <int C>
__global__ void lob_k_export_samples(LobDev D, void* out, int what) {
    const int descriptors = what == 1;
    const size_t n = (size_t)D.N * D.npx * C;
    for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x) {
        const size_t sp = i / C;
        const int c = (int)(i % C);
        if (D.alg != ALG_LOBSTER) {
            const int smp = (int)(sp / D.npx), p = (int)(sp % D.npx);
            unsigned long long d;
            uint32_t c2;
            if (D.alg == ALG_VIBE) load_sample<C, ALG_VIBE>(D, smp, p, d, c2);
            else load_sample<C, ALG_PBAS>(D, smp, p, d, c2);
            ((uint8_t*)out)[i] = (uint8_t)(d >> ((what == 2 ? 24 : 0) + 8 * c));
        } else if (descriptors) {
            ((uint16_t*)out)[i] = C == 3 ? (uint16_t)(((const unsigned long long*)D.sD)[sp] >> (16 * c))
                                         : ((const uint16_t*)D.sD)[sp];
        } else {
            ((uint8_t*)out)[i] = (C == 3 && c < 2) ? (uint8_t)(((const unsigned long long*)D.sD)[sp] >> (48 + 8 * c))
                                                   : D.sC[sp];
        }
    }
}

// ------------------------------------------------------------------------------------------------
// host side
// ------------------------------------------------------------------------------------------------
namespace {

inline size_t al(size_t v) { return (v + 255) & ~(size_t)255; }

inline uint8_t sat_round_u8f(float v) {
    const float r = std::nearbyint(v);
    return (uint8_t)(r < 0.f ? 0.f : r > 255.f ? 255.f : r);
}

#define LOB_CUDA(call, what)                                                      \
    do {                                                                          \
        const cudaError_t e_ = (call);                                            \
        if (e_ != cudaSuccess) {                                                  \
            err = std::string(what) + ": " + cudaGetErrorString(e_);              \
            return e_ == cudaErrorMemoryAllocation ? LVBGS_OOM : LVBGS_DEVICE_ERROR; \
        }                                                                         \
    } while (0)

inline cudaError_t staging(void** p, size_t bytes, cudaStream_t st) {
    int dev = 0;
    const cudaError_t e = cudaGetDevice(&dev);
    return e == cudaSuccess ? staging_alloc(dev, p, bytes, st) : e;
}

inline int blocks_for(size_t n) { return (int)((n + kThreadsL - 1) / kThreadsL); }

}  // namespace

void lob_release(LobState& L) {
    if (L.meanDone) cudaEventSynchronize(L.meanDone);
    if (L.repaired) cudaEventDestroy(L.repaired);
    if (L.meanStream) cudaStreamDestroy(L.meanStream);
    if (L.meanDone) cudaEventDestroy(L.meanDone);
    L.meanDone = L.repaired = nullptr;
    L.meanStream = nullptr;
    cudaFree(L.mem);
    L.mem = nullptr;
    L.bytes = 0;
    if (L.h_flags) cudaFreeHost(L.h_flags);
    L.h_flags = nullptr;
}

lvbgs_status lob_setup(LobState& L, int alg, const lvbgs_params& prm, int W, int H, int C,
                       const std::vector<uint8_t>& roi, size_t orig, size_t fin, cudaStream_t st, std::string& err) {
    // PBAS keeps its former mean gradient distance when initialized again (it is set by the
    // constructor only, BackgroundSubtractorPBAS.cpp:29)
    if (L.mem && L.d.alg == ALG_PBAS && L.d.meanGrad) {
        LOB_CUDA(cudaEventSynchronize(L.meanDone), "frame step");
        LOB_CUDA(cudaMemcpy(&L.pbasMean, L.d.meanGrad, sizeof(float), cudaMemcpyDeviceToHost), "state read-back");
    }
    cudaFree(L.mem);
    L.mem = nullptr;
    const size_t npx = (size_t)W * H, N = prm.bg_samples;
    // ViBe keeps only colour samples, PBAS colour and gradient samples and its maps (words in two planes,
    // load_sample), LOBSTER the packed descriptor plane and a colour byte
    const bool vibe = alg != ALG_LOBSTER, pbas = alg == ALG_PBAS;
    const size_t lob = vibe ? 0 : 1, pb = pbas ? 1 : 0;
    size_t off = 0;
    auto take = [&](size_t bytes) {
        const size_t o = off;
        off += al(bytes);
        return o;
    };
    const size_t oRoi = take(npx), oLastColor = take(lob * npx * C), oLastFG = take(lob * npx),
                 oRawBits = take(vibe && !pbas ? 0 : (npx / 32 + 2) * 4), oLut = take(256), oLastDesc = take(lob * npx * C * 2), oKctr = take(npx * 2),
                 oSD = take(lob * N * npx * (C == 3 ? 8 : 2)), oSC = take(N * npx * sample_bytes_lo(alg, C)),
                 oIntent = take(npx * 4),
                 oWD = take(npx * 8), oList0 = take(npx * 4), oList1 = take(npx * 4), oStamp = take(npx * 4),
                 oFlags = take(LOB_F_WORDS * 4), oStats = take(32), oFrame = take(npx * C), oMask = take(npx),
                 oSG = take(N * npx * sample_bytes_hi(alg, C)), oGrad = take(pb * npx * C),
                 oFm = take(pb * 6 * npx * 4), oMean = take(pb * 4), oBadSum = take(pb * npx * 4),
                 oBadCnt = take(pb * npx), oBadVals = take(pb * (C == 3 ? npx * N * 2 : 0)),
                 oSumTr = take(pb * (C == 3 ? SumWork::bytes((npx + kSumChunk - 1) / kSumChunk) : 0));
    LOB_CUDA(cudaMalloc(&L.mem, off), "model allocation");
    if (!L.h_flags) LOB_CUDA(cudaHostAlloc((void**)&L.h_flags, LOB_F_WORDS * 4, cudaHostAllocMapped), "pinned allocation");
    if (!L.meanDone) LOB_CUDA(cudaEventCreateWithFlags(&L.meanDone, cudaEventDisableTiming), "event creation");
    if (pbas && !L.meanStream) {
        LOB_CUDA(cudaEventCreateWithFlags(&L.repaired, cudaEventDisableTiming), "event creation");
        LOB_CUDA(cudaStreamCreateWithFlags(&L.meanStream, cudaStreamNonBlocking), "stream creation");
    }
    L.bytes = off;
    LobDev& D = L.d;
    D = LobDev{};
    D.alg = alg;
    D.W = W;
    D.H = H;
    D.C = C;
    D.N = (int)N;
    D.nreq = (int)prm.required_bg_samples;
    D.npx = (int)npx;
    D.descThr = (unsigned int)prm.desc_dist_threshold_offset;
    D.colThr = (unsigned int)prm.min_color_dist_threshold;
    D.seed = prm.seed;
    D.medianK = prm.default_median_blur_kernel_size;
    D.listCap = (unsigned int)npx;
    D.stampBase = 1;  // nonzero: the stamps start at 0
    uint8_t* b = L.mem;
    D.roi = b + oRoi;
    D.lastColor = b + oLastColor;
    D.lastFG = b + oLastFG;
    D.rawBits = (uint32_t*)(b + oRawBits);
    D.lut = b + oLut;
    D.lastDesc = (uint16_t*)(b + oLastDesc);
    D.kctr = (uint16_t*)(b + oKctr);
    D.sD = b + oSD;
    D.sC = b + oSC;
    D.sG = b + oSG;
    D.intent = (uint32_t*)(b + oIntent);
    D.wD = (unsigned long long*)(b + oWD);
    D.list0 = (uint32_t*)(b + oList0);
    D.list1 = (uint32_t*)(b + oList1);
    D.stamp = (uint32_t*)(b + oStamp);
    D.flags = (unsigned int*)(b + oFlags);
    D.hflags = L.h_flags;
    D.stats = (unsigned long long*)(b + oStats);
    L.d_frame = b + oFrame;
    L.d_mask = b + oMask;
    if (pbas) {
        D.grad = b + oGrad;
        D.fm = (float*)(b + oFm);
        D.meanGrad = (float*)(b + oMean);
        D.badSum = (uint32_t*)(b + oBadSum);
        D.badCnt = b + oBadCnt;
        D.badVals = (uint16_t*)(b + oBadVals);
        D.sumTr = b + oSumTr;
        if (C == 3) D.chunkAbout = sum_work(D.sumTr, (npx + kSumChunk - 1) / kSumChunk).about;
        // the constructor's arguments (BackgroundSubtractorPBAS.cpp:21-32) and medianBlur(.., 9) (:266 / :494)
        D.R0 = (float)prm.min_color_dist_threshold;
        D.updateRate = prm.update_rate;
        D.medianK = 9;
        D.cur = 0;
    }
    L.ksent = 0;
    L.lastRounds = 1;
    L.frames = 0;
    L.n_rel = fin;
    L.orig_roi = orig;
    // BackgroundSubtractorLBSP.cpp:30-34 / :47-48: the LBSP threshold LUT (one channel divides by 3)
    uint8_t lut[256];
    const float rel = prm.rel_lbsp_threshold;
    for (int t = 0; t <= 255; ++t)
        lut[t] = C == 1 ? sat_round_u8f(((float)t * rel + (float)prm.lbsp_threshold_offset) / 3)
                        : sat_round_u8f((float)t * rel + (float)prm.lbsp_threshold_offset);
    LOB_CUDA(cudaMemsetAsync(L.mem, 0, off, st), "model reset");
    LOB_CUDA(cudaMemcpyAsync(D.roi, roi.data(), npx, cudaMemcpyHostToDevice, st), "roi upload");
    LOB_CUDA(cudaMemcpyAsync(D.lut, lut, 256, cudaMemcpyHostToDevice, st), "lut upload");
    return LVBGS_OK;
}

namespace {
// one kernel of the frame step for the stream's (channels, algorithm)
template <template <int, int> class K, typename... A>
void launch(const LobDev& D, int blocks, cudaStream_t st, A... args) {
    if (D.alg == ALG_VIBE) {
        if (D.C == 3) K<3, ALG_VIBE>::run(blocks, st, D, args...);
        else K<1, ALG_VIBE>::run(blocks, st, D, args...);
    } else if (D.alg == ALG_PBAS) {
        if (D.C == 3) K<3, ALG_PBAS>::run(blocks, st, D, args...);
        else K<1, ALG_PBAS>::run(blocks, st, D, args...);
    } else {
        if (D.C == 3) K<3, ALG_LOBSTER>::run(blocks, st, D, args...);
        else K<1, ALG_LOBSTER>::run(blocks, st, D, args...);
    }
}
template <int C, int ALG>
struct Eval {
    // Not chained: what comes before may be a kernel of the caller's that writes the frame and lets dependents start
    // early, and the read-only loads (ld.global.nc) of a kernel want memory that nothing writes while it is there.
    static void run(int b, cudaStream_t st, const LobDev& D) { lob_k_eval<C, ALG><<<b, kThreadsL, 0, st>>>(D); }
};
template <int C, int ALG>
struct First {
    static void run(int b, cudaStream_t st, const LobDev& D) {
        if (D.npx < kFirstSmall) launch_chained(lob_k_first<C, ALG, 1>, dim3(b), dim3(kThreadsL), st, D);
        else launch_chained(lob_k_first<C, ALG, 4>, dim3((b + 3) / 4), dim3(kThreadsL), st, D);
    }
};
template <int C, int ALG>
struct Round {
    static void run(int b, cudaStream_t st, const LobDev& D, int r) { launch_chained(lob_k_round<C, ALG>, dim3(b), dim3(kThreadsL), st, D, r); }
};
template <int C, int ALG>
struct Commit {
    static void run(int b, cudaStream_t st, const LobDev& D) { launch_chained(lob_k_commit<C, ALG>, dim3(b), dim3(kThreadsL), st, D); }
};

// PBAS's gradient image of a device frame into D.grad
void pbas_gradient(const LobDev& D, const uint8_t* img, cudaStream_t st) {
    const dim3 g((unsigned)tiles_across(D.W, kGradW) * tiles_across(D.H, kGradH));
    if (D.C == 3) pbas_k_grad<3><<<g, kThreadsL, 0, st>>>(D, img);
    else pbas_k_grad<1><<<g, kThreadsL, 0, st>>>(D, img);
}

// PBAS's frame-level mean gradient distance, after the commit
void pbas_mean_launch(const LobDev& D, int sms, cudaStream_t st) {
    if (D.C == 1) {
        pbas_k_mean1<<<2 * sms, kThreadsL, 0, st>>>(D);  // after another stream's event
        launch_chained(pbas_k_mean1_end, dim3(1), dim3(1), st, D);
    } else {
        const int nChunks = (D.npx + kSumChunk - 1) / kSumChunk;
        const SumWork W = sum_work(D.sumTr, nChunks);
        pbas_k_sum_tr<<<nChunks, kSumChunk, 0, st>>>(D, W);  // after another stream's event
        launch_chained(pbas_k_sum_win, dim3((nChunks + 255) / 256), dim3(256), st, D, W, nChunks);
        launch_chained(pbas_k_sum_walk, dim3(1), dim3(32), st, D, W, nChunks);
    }
}

lvbgs_status lob_refresh_launch(LobState& L, float frac, int force, cudaStream_t st, std::string& err) {
    LobDev& D = L.d;
    const int N = D.N;
    const int nref = frac < 1.0f ? (int)(frac * (float)N) : N;
    int start = 0;
    if (frac < 1.0f) {
        // the frame-level draw of the start position (:416)
        uint32_t c[4] = {L.ksent >> 2, kSentinelPx, D.frameKey, 0u};
        philox4x32_10(c, (uint32_t)D.seed, (uint32_t)(D.seed >> 32));
        start = (int)((c[L.ksent & 3u] & 0x7fffffffu) % (uint32_t)N);
        ++L.ksent;
    }
    if (nref > 0) {
        if (D.C == 3) lob_k_refresh<3><<<blocks_for(D.npx), kThreadsL, 0, st>>>(D, start, nref, force);
        else lob_k_refresh<1><<<blocks_for(D.npx), kThreadsL, 0, st>>>(D, start, nref, force);
        LOB_CUDA(cudaGetLastError(), "refresh launch");
    }
    return LVBGS_OK;
}
}  // namespace

lvbgs_status lob_init_model(LobState& L, const uint8_t* dimg, cudaStream_t st, std::string& err) {
    LobDev& D = L.d;
    D.frameKey = 0;
    L.ksent = 0;
    if (D.alg == ALG_PBAS) {
        D.cur = 0;
        pbas_gradient(D, dimg, st);
        if (D.C == 3) pbas_k_init<3><<<blocks_for(D.npx), kThreadsL, 0, st>>>(D, dimg, L.pbasMean);
        else pbas_k_init<1><<<blocks_for(D.npx), kThreadsL, 0, st>>>(D, dimg, L.pbasMean);
        LOB_CUDA(cudaGetLastError(), "init launch");
        LOB_CUDA(cudaStreamSynchronize(st), "initialization");
        return LVBGS_OK;
    }
    if (D.alg == ALG_VIBE) {
        if (D.C == 3) lob_k_vibe_init<3><<<blocks_for(D.npx), kThreadsL, 0, st>>>(D, dimg);
        else lob_k_vibe_init<1><<<blocks_for(D.npx), kThreadsL, 0, st>>>(D, dimg);
        LOB_CUDA(cudaGetLastError(), "init launch");
        LOB_CUDA(cudaStreamSynchronize(st), "initialization");
        return LVBGS_OK;
    }
    if (D.C == 3) lob_k_init<3><<<blocks_for(D.npx), kThreadsL, 0, st>>>(D, dimg);
    else lob_k_init<1><<<blocks_for(D.npx), kThreadsL, 0, st>>>(D, dimg);
    LOB_CUDA(cudaGetLastError(), "init launch");
    // refreshModel(1.0f, true) (:455)
    lvbgs_status s = lob_refresh_launch(L, 1.0f, 1, st, err);
    if (s != LVBGS_OK) return s;
    LOB_CUDA(cudaStreamSynchronize(st), "initialization");
    return LVBGS_OK;
}

lvbgs_status lob_refresh(LobState& L, float frac, int force, cudaStream_t st, std::string& err) {
    lvbgs_status s = lob_refresh_launch(L, frac, force, st, err);
    if (s != LVBGS_OK) return s;
    LOB_CUDA(cudaStreamSynchronize(st), "refresh");
    return LVBGS_OK;
}

lvbgs_status lob_apply(LobState& L, const uint8_t* dimg, uint8_t* dmask, uint8_t* hostMask, double lr,
                       cudaStream_t st, std::string& err) {
    LobDev& D = L.d;
    D.frame = dimg;
    D.maskOut = dmask;
    D.nLR = std::isinf(lr) ? ~0ull : (unsigned long long)std::ceil(lr);  // :470
    if (D.alg == ALG_PBAS) {
        // learningRateOverride > 0 replaces ceil(T(x)) (:174 / :402)
        D.lrOverride = lr > 0 ? 1 : 0;
        if (!(lr > 0)) D.nLR = 0;
    }
    ++L.frames;
    D.frameKey = (uint32_t)L.frames;
    L.ksent = 0;
    const int C = D.C, nb = blocks_for(D.npx);
    int dev = 0, sms = 1;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    const int roundBlocks = 2 * (sms > 0 ? sms : 1);
    std::memset(L.h_flags, 0, LOB_F_WORDS * 4);  // the commit writes the frame step's flags here
    // PBAS's frame-level mean gradient distance is only needed by the next evaluation: it runs on a stream of its
    // own, beside the commit, the median and the mask's copy (its last kernel is one warp's serial walk). The host
    // waits for both streams. Only the evaluation and the repairs write what the mean reads.
    if (D.alg == ALG_PBAS) pbas_gradient(D, dimg, st);
    launch<Eval>(D, nb, st);
    if (D.alg == ALG_PBAS && C == 3) {
        LOB_CUDA(cudaEventRecord(L.repaired, st), "event record");
        LOB_CUDA(cudaStreamWaitEvent(L.meanStream, L.repaired, 0), "event wait");
        const int nChunks = (D.npx + kSumChunk - 1) / kSumChunk;
        pbas_k_sum_scan<<<1, kSumScan, 0, L.meanStream>>>(sum_work(D.sumTr, nChunks), nChunks);
    }
    launch<First>(D, nb, st);
    LOB_CUDA(cudaGetLastError(), "evaluation launch");
    int round = 1, chunk = L.lastRounds;
    for (;;) {
        for (int i = 0; i < chunk; ++i, ++round) launch<Round>(D, roundBlocks, st, round);
        if (D.alg == ALG_PBAS) {
            LOB_CUDA(cudaEventRecord(L.repaired, st), "event record");
            LOB_CUDA(cudaStreamWaitEvent(L.meanStream, L.repaired, 0), "event wait");
            pbas_mean_launch(D, sms, L.meanStream);
            LOB_CUDA(cudaGetLastError(), "mean launch");
            LOB_CUDA(cudaEventRecord(L.meanDone, L.meanStream), "event record");
        }
        launch<Commit>(D, nb, st);
        // LOBSTER's median blur, last mask and last colour frame; PBAS's median blur (ViBe outputs its
        // raw mask)
        const dim3 mg((unsigned)tiles_across(D.W, 32 * kMedW) * tiles_across(D.H, kMedH));
        if (D.alg == ALG_LOBSTER) launch_chained(lob_k_median<true>, mg, dim3(kThreadsL), st, D);
        else if (D.alg == ALG_PBAS) launch_chained(lob_k_median<false>, mg, dim3(kThreadsL), st, D);
        LOB_CUDA(cudaGetLastError(), "repair launch");
        if (hostMask) LOB_CUDA(cudaMemcpyAsync(hostMask, dmask, (size_t)D.npx, cudaMemcpyDeviceToHost, st), "mask download");
        LOB_CUDA(cudaStreamSynchronize(st), "frame step");
        if (D.alg == ALG_PBAS) LOB_CUDA(cudaEventSynchronize(L.meanDone), "frame step");
        const volatile unsigned int* hf = L.h_flags;
        if (hf[LOB_F_ERR]) {
            err = "LOBSTER repair list overflow";
            return LVBGS_DEVICE_ERROR;
        }
        if (hf[LOB_F_CONV]) break;
        if (round >= kMaxRoundsL) {
            err = "LOBSTER raster-order repair did not converge";
            return LVBGS_DEVICE_ERROR;
        }
        chunk = std::max(1, chunk * 2);
    }
    L.lastRounds = (int)L.h_flags[LOB_F_ROUNDS];
    D.stampBase += (uint32_t)round + 2u;
    if (D.alg == ALG_PBAS) D.cur ^= 1;  // the maps this frame step wrote are the next one's start
    return LVBGS_OK;
}

lvbgs_status lob_background(LobState& L, void* hostOut, bool descriptors, cudaStream_t st, std::string& err) {
    LobDev& D = L.d;
    const size_t n = (size_t)D.npx * D.C * (descriptors ? 2 : 1);
    void* tmp = nullptr;
    LOB_CUDA(staging(&tmp, n, st), "staging allocation");
    if (D.C == 3) lob_k_background<3><<<1024, 256, 0, st>>>(D, tmp, descriptors ? 1 : 0);
    else lob_k_background<1><<<1024, 256, 0, st>>>(D, tmp, descriptors ? 1 : 0);
    cudaError_t e = cudaGetLastError();
    if (e == cudaSuccess) e = cudaMemcpyAsync(hostOut, tmp, n, cudaMemcpyDeviceToHost, st);
    cudaFreeAsync(tmp, st);
    if (e == cudaSuccess) e = cudaStreamSynchronize(st);
    LOB_CUDA(e, "background image");
    return LVBGS_OK;
}

size_t lob_map_bytes(const LobState& L, int which) {
    const size_t npx = (size_t)L.d.npx, C = (size_t)L.d.C, N = (size_t)L.d.N;
    if (L.d.alg == ALG_VIBE) return which == LVBGS_MAP_SAMPLE_COLOR ? N * npx * C : which == LVBGS_MAP_ROI ? npx : 0;
    if (L.d.alg == ALG_PBAS) switch (which) {
            case LVBGS_MAP_SAMPLE_COLOR:
            case LVBGS_MAP_SAMPLE_GRAD: return N * npx * C;
            case LVBGS_MAP_R:
            case LVBGS_MAP_T:
            case LVBGS_MAP_DMIN_LT: return npx * 4;
            case LVBGS_MAP_GRAD: return npx * C;
            case LVBGS_MAP_MEAN_GRAD: return 4;
            case LVBGS_MAP_ROI: return npx;
            default: return 0;
        }
    switch (which) {
        case LVBGS_MAP_LAST_FG:
        case LVBGS_MAP_ROI: return npx;
        case LVBGS_MAP_LAST_COLOR: return npx * C;
        case LVBGS_MAP_LAST_DESC: return npx * C * 2;
        case LVBGS_MAP_SAMPLE_COLOR: return N * npx * C;
        case LVBGS_MAP_SAMPLE_DESC: return N * npx * C * 2;
        case LVBGS_MAP_LUT: return 256;
        default: return 0;
    }
}

lvbgs_status lob_get_map(LobState& L, int which, void* hostOut, size_t bytes, cudaStream_t st, std::string& err) {
    LobDev& D = L.d;
    const size_t need = lob_map_bytes(L, which);
    if (need == 0) {
        err = "map not kept by LOBSTER";
        return LVBGS_BAD_ARG;
    }
    if (bytes < need) {
        err = "output buffer too small";
        return LVBGS_BAD_ARG;
    }
    const void* src = nullptr;
    const float* fm = D.fm ? D.fm + (size_t)D.cur * 3 * D.npx : nullptr;
    if (D.alg == ALG_VIBE) src = which == LVBGS_MAP_ROI ? (const void*)D.roi : nullptr;
    else if (D.alg == ALG_PBAS) switch (which) {
            case LVBGS_MAP_SAMPLE_COLOR:
            case LVBGS_MAP_SAMPLE_GRAD: break;
            case LVBGS_MAP_R: src = fm; break;
            case LVBGS_MAP_T: src = fm + D.npx; break;
            case LVBGS_MAP_DMIN_LT: src = fm + 2 * (size_t)D.npx; break;
            case LVBGS_MAP_GRAD: src = D.grad; break;
            case LVBGS_MAP_MEAN_GRAD: src = D.meanGrad; break;
            default: src = D.roi; break;
        }
    else switch (which) {
        case LVBGS_MAP_LAST_FG: src = D.lastFG; break;
        case LVBGS_MAP_ROI: src = D.roi; break;
        case LVBGS_MAP_LAST_COLOR: src = D.lastColor; break;
        case LVBGS_MAP_LAST_DESC: src = D.lastDesc; break;
        case LVBGS_MAP_LUT: src = D.lut; break;
        default: break;
    }
    if (src) {
        LOB_CUDA(cudaMemcpyAsync(hostOut, src, need, cudaMemcpyDeviceToHost, st), "map download");
        LOB_CUDA(cudaStreamSynchronize(st), "map download");
        return LVBGS_OK;
    }
    void* tmp = nullptr;
    LOB_CUDA(staging(&tmp, need, st), "staging allocation");
    const int desc = which == LVBGS_MAP_SAMPLE_DESC ? 1 : which == LVBGS_MAP_SAMPLE_GRAD ? 2 : 0;
    if (D.C == 3) lob_k_export_samples<3><<<1024, 256, 0, st>>>(D, tmp, desc);
    else lob_k_export_samples<1><<<1024, 256, 0, st>>>(D, tmp, desc);
    cudaError_t e = cudaGetLastError();
    if (e == cudaSuccess) e = cudaMemcpyAsync(hostOut, tmp, need, cudaMemcpyDeviceToHost, st);
    cudaFreeAsync(tmp, st);
    if (e == cudaSuccess) e = cudaStreamSynchronize(st);
    LOB_CUDA(e, "sample export");
    return LVBGS_OK;
}

lvbgs_status lob_stats(LobState& L, unsigned long long out[2], cudaStream_t st, std::string& err) {
    LOB_CUDA(cudaMemcpyAsync(out, L.d.stats, 16, cudaMemcpyDeviceToHost, st), "statistics download");
    LOB_CUDA(cudaStreamSynchronize(st), "statistics download");
    return LVBGS_OK;
}

}  // namespace lvbgs
