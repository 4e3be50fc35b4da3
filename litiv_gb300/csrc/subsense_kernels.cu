// SuBSENSE frame step for sm_103a: one tick processes one frame of every stream in the batch as a
// sequence of ordinary launches over a per-stream descriptor table (a tile, row or segment index is
// mapped to its stream by binary search); only the repair rounds run as one cooperative kernel whose
// rounds are separated by a bounded grid barrier.
//
// Exactness of the reference's sequential raster scan (BackgroundSubtractorSuBSENSE.cpp:201-481):
// a pixel p reads two things another pixel writes during the same frame -- its own samples, which
// an earlier pixel's neighbour update may have overwritten (:296-299/:442-448), and the D_last /
// raw-segmentation-ST values of its randomly chosen neighbour q, which are this frame's values when
// q precedes p (:292-293/:438-439). Random draws are keyed by (stream, frame, pixel, draw index),
// so they do not depend on the scan order. The tick therefore
//   A  evaluates every pixel against the frame-start model and records an "intent" (decision,
//      samples evaluated, own/neighbour sample writes, neighbour-update state),
//   B  resolves the ghost test of each neighbour update against the values the scan would see,
//      and marks every pixel whose evaluated samples were overwritten by an earlier pixel,
//   M/R repairs: re-evaluates marked pixels with the overwritten samples (M) and re-resolves the
//      ghost tests that read a pixel whose decision changed (R), marking the pixels whose incoming
//      writes changed, until nothing changes (the dependencies follow raster order, so this is a
//      fixed point reached in at most the length of the longest dependency chain),
//   F  commits every sample write in raster order (last writer wins) and starts post-processing.
// Post-processing, frame-level statistics and the automatic model reset follow in later launches of
// the same tick.
#include <cuda_runtime.h>

#include "area_device.cuh"
#include "bitslice.cuh"
#include "lbsp_device.cuh"
#include "lvbgs_internal.h"

namespace lvbgs {

// 7x7 Gaussian sampling weights (opencv.hpp:915-923)
__constant__ int c_pat7[49] = {2, 4, 6, 7, 6, 4, 2,     4, 8, 12, 14, 12, 8, 4, 6, 12, 21, 25, 21, 12, 6, 7, 14, 25, 28,
                               25, 14, 7, 6, 12, 21, 25, 21, 12, 6, 4, 8, 12, 14, 12, 8, 4, 2, 4, 6, 7, 6, 4, 2};

constexpr int kUFLimit = 1 << 22;

// ------------------------------------------------------------------------------------------
// small helpers
// ------------------------------------------------------------------------------------------
__device__ __forceinline__ unsigned long long gtimer() {
    unsigned long long t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    return t;
}
__device__ __forceinline__ unsigned int ld_volatile(const unsigned int* p) { return *(const volatile unsigned int*)p; }

// Barrier over the first nCtas CTAs of a cooperative launch (all co-resident). The wait is bounded: after
// timeoutNs the CTA records ERR_BARRIER_TIMEOUT and every CTA leaves at its next check. The arrivals only count up
// (from the tick's start, zero): the due value, kept by the CTA, is what the barriers so far need, so nothing is
// reset or released, and the error word is read together with the count. With a count that the last
// arrival resets and a generation that it raises, a barrier was a chain of seven trips to L2.
__device__ bool grid_sync(TickWork* w, unsigned int nCtas, unsigned long long timeoutNs, unsigned int& due) {
    __shared__ int s_ok;
    due += nCtas;
    __syncthreads();
    if (threadIdx.x == 0) {
        __threadfence();
        atomicAdd(&w->bar_count, 1u);
        const unsigned long long t0 = gtimer();
        int ok = 1;
        for (;;) {
            const unsigned int arrived = ld_volatile(&w->bar_count), err = ld_volatile(&w->err);
            if (err != 0u) {
                ok = 0;
                break;
            }
            if ((int)(arrived - due) >= 0) break;
            if (gtimer() - t0 > timeoutNs) {
                atomicOr(&w->err, ERR_BARRIER_TIMEOUT);
                ok = 0;
                break;
            }
            __nanosleep(20);
        }
        __threadfence();
        s_ok = ok;
    }
    __syncthreads();
    if (blockIdx.x == 0 && threadIdx.x == 0 && w->nts < 40u) w->ts[w->nts++] = gtimer();
    return s_ok != 0;
}

__device__ __forceinline__ int find_stream_by_tile(const TickParams& P, int t) {
    int lo = 0, hi = P.nStreams - 1;
    while (lo < hi) {
        const int mid = (lo + hi + 1) >> 1;
        if (P.streams[mid].tileBase <= t) lo = mid;
        else hi = mid - 1;
    }
    return lo;
}

struct DrawState {
    uint32_t blk;
    uint32_t v[4];
};
__device__ __forceinline__ uint32_t draw_k(unsigned long long seed, uint32_t frame, uint32_t px, uint32_t k,
                                           DrawState& ds) {
    const uint32_t blk = k >> 2;
    if (blk != ds.blk) {
        uint32_t c[4] = {blk, px, frame, 0u};
        philox4x32_10(c, (uint32_t)seed, (uint32_t)(seed >> 32));
        ds.v[0] = c[0];
        ds.v[1] = c[1];
        ds.v[2] = c[2];
        ds.v[3] = c[3];
        ds.blk = blk;
    }
    return ds.v[k & 3u] & 0x7fffffffu;
}
// a % m for a 31-bit draw and a size_t modulus (m >= 2^32 leaves a unchanged)
__device__ __forceinline__ unsigned long long mod_draw(uint32_t a, unsigned long long m) {
    if (m > 0xffffffffull) return (unsigned long long)a;
    const uint32_t m32 = (uint32_t)m;
    if ((m32 & (m32 - 1u)) == 0u) return (unsigned long long)(a & (m32 - 1u));  // powers of two (T = 2, 4, ...)
    return (unsigned long long)(a % m32);
}
// a % N for a 31-bit draw with the stream's multiplier M = ceil(2^40 / N): for N <= 64 the
// quotient error a*(M - 2^40/N)/2^40 < 2^-9 < 1/N, so floor(a*M / 2^40) is the exact quotient
__device__ __forceinline__ uint32_t mod_n(uint32_t a, const StreamDev& S) {
    const uint32_t q = (uint32_t)(((unsigned long long)a * S.nMagic) >> 40);
    return a - q * (uint32_t)S.N;
}

__device__ __forceinline__ void clamp_xy(int& x, int& y, int W, int H) {
    if (x < kBorder) x = kBorder;
    else if (x >= W - kBorder) x = W - kBorder - 1;
    if (y < kBorder) y = kBorder;
    else if (y >= H - kBorder) y = H - kBorder - 1;
}

__device__ __forceinline__ float fmin_std(float a, float b) { return (b < a) ? b : a; }
__device__ __forceinline__ float fmax_std(float a, float b) { return (a < b) ? b : a; }

// A pixel's samples: the descriptor word of sample 0 (sample k: k * S.sStride bytes on) and the distance in
// bytes from there to its colour byte, in the same 32-byte sector
template <int C>
struct Samples {
    uint8_t* at;
    int toCol;
};
template <int C>
__device__ __forceinline__ Samples<C> samples_of(const StreamDev& S, int p) {
    const unsigned sec = (unsigned)p / kSecPx<C>, j = (unsigned)p - sec * kSecPx<C>;
    constexpr int kDescB = C == 3 ? 8 : 2;
    return {S.samples + (size_t)sec * 32 + j * kDescB, kDescB * kSecPx<C> - (kDescB - 1) * (int)j};
}
template <int C>
__device__ __forceinline__ void load_sample(const Samples<C>& m, size_t off, uint64_t& d, uint32_t& c) {
    d = C == 3 ? *(const uint64_t*)(m.at + off) : (uint64_t) * (const uint16_t*)(m.at + off);
    c = m.at[off + m.toCol];
}
template <int C>
__device__ __forceinline__ void store_sample(const Samples<C>& m, size_t off, uint64_t d, uint32_t c) {
    if (C == 3) *(uint64_t*)(m.at + off) = d;
    else *(uint16_t*)(m.at + off) = (uint16_t)d;
    m.at[off + m.toCol] = (uint8_t)c;
}

struct FrameK {
    float fLT, fST, t_lo, t_hi;
    uint32_t frame;  // frame index of this tick (m_nFrameIdx after ++)
    int cur, nxt;
    int cooldown;  // m_nModelResetCooldown != 0
    int use3x3;
};
// exact quotients i/765, i/255, i/48 and i/16 (IEEE division on the device, done once): the
// normalized distances of :254/:258/:272 and :396/:400/:416 divide small integers by constants
__device__ float g_div_col3[766], g_div_col1[256], g_div_desc3[49], g_div_desc1[17];
extern "C" __global__ void lvbgs_init_tables() {
    for (int i = threadIdx.x; i < 766; i += blockDim.x) g_div_col3[i] = (float)i / 765.0f;
    for (int i = threadIdx.x; i < 256; i += blockDim.x) g_div_col1[i] = (float)i / 255.0f;
    for (int i = threadIdx.x; i < 49; i += blockDim.x) g_div_desc3[i] = (float)i / 48.0f;
    for (int i = threadIdx.x; i < 17; i += blockDim.x) g_div_desc1[i] = (float)i / 16.0f;
}

__device__ __forceinline__ FrameK frame_consts(const StreamDev& S) {
    const StreamCtl* ctl = S.ctl;
    FrameK F;
    const unsigned long long f = ctl->frame_idx + 1ull;
    F.fLT = ctl->fLT;
    F.fST = ctl->fST;
    F.frame = (uint32_t)f;
    F.cur = (int)(ctl->frame_idx & 1ull);
    F.nxt = F.cur ^ 1;
    F.cooldown = ctl->cooldown != 0ull;
    F.t_lo = ctl->t_lo;
    F.t_hi = ctl->t_hi;
    F.use3x3 = ctl->use3x3;
    return F;
}

// one override of a sample read: an earlier pixel's neighbour update of this pixel
struct Ovr {
    int s;
    uint32_t col;      // packed colour bytes
    uint64_t desc;     // packed descriptors
};

// ------------------------------------------------------------------------------------------
// per-pixel evaluation: one iteration of the reference's raster loop for pixel p, against the
// frame-start samples (optionally overridden). Writes the pixel's next-frame maps and returns
// its intent word. (1ch: BackgroundSubtractorSuBSENSE.cpp:201-330, 3ch: :333-481)
// ------------------------------------------------------------------------------------------
// per-pixel inputs of one evaluation, loaded up front so that all of them are in flight together
template <int C>
struct PixIn {
    float R, V, T, DL, DmLT, DmST, RwLT, RwST, FnLT, FnST;
    uint32_t uOld, lastFG, blink;
    uint32_t lc[C], ld[C];
};
template <int C>
__device__ __forceinline__ void load_pix(const StreamDev& S, const FrameK& F, int p, PixIn<C>& in) {
    const int npx = S.npx;
    const float* fc = S.fm + (size_t)F.cur * kNumFloatMaps * npx;
    in.R = fc[FM_R * npx + p];
    in.V = fc[FM_V * npx + p];
    in.T = fc[FM_T * npx + p];
    in.DL = fc[FM_DLAST * npx + p];
    in.DmLT = fc[FM_DMIN_LT * npx + p];
    in.DmST = fc[FM_DMIN_ST * npx + p];
    in.RwLT = fc[FM_RAW_LT * npx + p];
    in.RwST = fc[FM_RAW_ST * npx + p];
    in.FnLT = fc[FM_FIN_LT * npx + p];
    in.FnST = fc[FM_FIN_ST * npx + p];
    in.uOld = S.unst[(size_t)F.cur * npx + p];
    in.lastFG = S.lastFG[p];
    in.blink = S.blinks[p];
    const uint8_t* lc = S.lastCol + (size_t)F.cur * npx * C + (size_t)p * C;
    const uint16_t* ld = S.lastDesc + (size_t)F.cur * npx * C + (size_t)p * C;
#pragma unroll
    for (int c = 0; c < C; ++c) {
        in.lc[c] = lc[c];
        in.ld[c] = ld[c];
    }
}

// thresholds of one evaluation from R(x) and the previous unstable flag, and the new unstable flag
// descThr is clamped to 255: a descriptor distance is at most 16 per channel (48 summed), so every
// comparison against the clamped value (or three times it) has the result of the unclamped one
struct EvalThr {
    uint32_t colThr;
    uint32_t descThr;
    uint32_t uNew;
};
__device__ __forceinline__ EvalThr eval_thresholds(const StreamDev& S, float R, float RwLT, float RwST, float FnLT,
                                                   float FnST, uint32_t uOld) {
    EvalThr t;
    t.colThr =
        (uint32_t)__float2ull_rz(R * (float)S.minColor - (float)((uint32_t)(uOld == 0u) * (uint32_t)S.stabColorOff));
    const unsigned long long descThr = (1ull << (unsigned)__float2ull_rz(floorf(R + 0.5f))) +
                                       (unsigned long long)S.descOff + (unsigned long long)uOld * S.descOff;
    t.descThr = descThr < 255ull ? (uint32_t)descThr : 255u;
    t.uNew = (R > 3.000f || (RwLT - FnLT) > 0.100f || (RwST - FnST) > 0.100f) ? 1u : 0u;
    return t;
}

// state of the ordered sample scan: next sample, good samples so far, minima over the good ones
struct ScanSt {
    int s, nGood;
    uint32_t minDesc, minSum;
    int g0, g1;                   // indices of the first two good samples (-1: none)
    uint32_t g0d, g0s, g1d, g1s;  // their descriptor and summed distances
};

// one sample against the pixel (the body of the sample loops, :226-250 / :357-393): whether it is a
// good match, and its descriptor and summed distances. The reference rejects a sample at the first
// failed check; the verdict is the conjunction of all checks, so the three-channel form tests the
// three colour distances first (one branch), then evaluates the three channels without branches.
template <int C>
__device__ __forceinline__ bool sample_match(const uint8_t* __restrict__ lut, const uint32_t (&vals)[C][4],
                                             const uint32_t (&curr)[C], const uint32_t (&intra)[C],
                                             const EvalThr& th, uint64_t d, uint32_t c2, uint32_t& dd,
                                             uint32_t& sd) {
    if (C == 1) {
        const uint32_t cthr = th.colThr / 2u;
        const uint32_t bgc = c2, bgd = (uint32_t)d & 0xffffu;
        const uint32_t colDist = (uint32_t)abs((int)curr[0] - (int)bgc);
        if (colDist > cthr) return false;
        const uint32_t intraD = __popc(intra[0] ^ bgd);
        const uint32_t interD = __popc((lbsp_thr_raw(vals[0], bgc, lut[bgc]) ^ bgd) & 0xffffu);
        const uint32_t descDist = (intraD + interD) / 2u;
        if (descDist > th.descThr) return false;
        uint32_t sumDist = (descDist / 4u) * 15u + colDist;
        if (sumDist > 255u) sumDist = 255u;
        if (sumDist > cthr) return false;
        dd = descDist;
        sd = sumDist;
        return true;
    } else {
        const uint32_t totColThr = th.colThr * 3u, scThr = totColThr / 2u;
        const uint32_t hiw = (uint32_t)(d >> 32), low = (uint32_t)d;
        // bytes 0-2: the sample's colours (d bits 48-55, 56-63, c2); byte 3 repeats byte 2
        const uint32_t bgW = __byte_perm(hiw, c2, 0x4432);
        const uint32_t currW = curr[0] | (curr[1] << 8) | (curr[2] * 0x01010000u);
        const uint32_t cd = __vabsdiffu4(currW, bgW);
        const uint32_t col0 = cd & 0xffu, col1 = (cd >> 8) & 0xffu, col2 = (cd >> 16) & 0xffu;
        if (max(max(col0, col1), col2) > scThr) return false;
        const uint32_t col[3] = {col0, col1, col2};
        const uint32_t bgc[3] = {bgW & 0xffu, (bgW >> 8) & 0xffu, (bgW >> 16) & 0xffu};
        const uint32_t bgd[3] = {low & 0xffffu, low >> 16, hiw & 0xffffu};
        uint32_t totDesc = 0, totSum = 0;
        bool bad = false;
#pragma unroll
        for (int c = 0; c < 3; ++c) {
            const uint32_t intraD = __popc(intra[c] ^ bgd[c]);
            const uint32_t interD = __popc((lbsp_thr_raw(vals[c], bgc[c], lut[bgc[c]]) ^ bgd[c]) & 0xffffu);
            const uint32_t descDist = (intraD + interD) / 2u;
            const uint32_t sumDist = min((descDist / 2u) * 15u + col[c], 255u);
            bad |= sumDist > scThr;
            totDesc += descDist;
            totSum += sumDist;
        }
        if (bad || totDesc > th.descThr * 3u || totSum > totColThr) return false;
        dd = totDesc;
        sd = totSum;
        return true;
    }
}

template <int C>
__device__ __forceinline__ void scan_init(ScanSt& st) {
    st.s = 0;
    st.nGood = 0;
    st.g0 = st.g1 = -1;
    st.g0d = st.g0s = st.g1d = st.g1s = 0;
    st.minDesc = C == 1 ? 16u : 48u;
    st.minSum = C == 1 ? 255u : 765u;
}
// the evaluation's ordered sample scan: until nreq good samples or kScanCap samples; dA/cA and dB/cB hold
// samples 0 and 1 (they arrive with the feedback maps), and the loop requests sample s+2 while it evaluates
// sample s. The first good sample's index is tracked (a deferred scan's record keeps it), not the distances.
template <int C>
__device__ __forceinline__ void scan_samples(const StreamDev& S, const uint8_t* __restrict__ lut, const Samples<C>& sp,
                                             const uint32_t (&vals)[C][4], const uint32_t (&curr)[C],
                                             const uint32_t (&intra)[C], const EvalThr& th, uint64_t dA, uint32_t cA,
                                             uint64_t dB, uint32_t cB, ScanSt& st) {
    const int nreq = S.nreq;
    const int sMax = kScanCap < S.N ? kScanCap : S.N;
    int nGood = 0, s = 0, g0 = -1;
    uint32_t minDesc = st.minDesc, minSum = st.minSum;
    while (nGood < nreq && s < sMax) {
        const uint64_t d = dA;
        const uint32_t c2 = cA;
        dA = dB;
        cA = cB;
        if (s + 2 < sMax) {
            load_sample<C>(sp, (size_t)(s + 2) * S.sStride, dB, cB);
        }
        uint32_t dd, sd;
        if (sample_match<C>(lut, vals, curr, intra, th, d, c2, dd, sd)) {
            if (minDesc > dd) minDesc = dd;
            if (minSum > sd) minSum = sd;
            if (g0 < 0) g0 = s;
            ++nGood;
        }
        ++s;
    }
    st.s = s;
    st.nGood = nGood;
    st.minDesc = minDesc;
    st.minSum = minSum;
    st.g0 = g0;
}

// With nreq <= 2 a scan's outcome is fixed by its stop position and its (at most two) good samples:
// every other sample it evaluated is bad. Recording them for the long scans lets the repair re-match
// such a pixel from the samples that earlier pixels overwrite (the others keep their frame-start
// values, so their verdicts), scanning on only when an overwrite removed a good sample.
// Record: frame tag | stop | count | indices | descriptor distances | summed distances.
__device__ __forceinline__ void record_scan(const StreamDev& S, const FrameK& F, int p, const ScanSt& st) {
    if (S.nreq > 2) return;
    const int n = st.nGood < 2 ? st.nGood : 2;
    uint4 r;
    r.x = F.frame;
    r.y = (uint32_t)st.s | ((uint32_t)n << 8) | ((uint32_t)(st.g0 < 0 ? 255 : st.g0) << 16) |
          ((uint32_t)(st.g1 < 0 ? 255 : st.g1) << 24);
    r.z = (st.g0d & 0xffffu) | (st.g1d << 16);
    r.w = (st.g0s & 0xffffu) | (st.g1s << 16);
    S.goodRec[p] = r;
}

// L2 prefetch of a sample: a hint without registers
template <int C>
__device__ __forceinline__ void prefetch_sample(const Samples<C>& m, size_t off) {
    asm volatile("prefetch.global.L2 [%0];" ::"l"(m.at + off));
}

constexpr int kScanPrefetch = 8;  // samples prefetched ahead of the loads of a lane's own scan

// The ordered scan of one pixel's samples by one lane, continued from st (see coop_scan for the masks)
template <int C, bool REC>
__device__ __forceinline__ void lane_scan(const StreamDev& S, int p, const uint32_t (&vals)[C][4],
                                          const uint32_t (&curr)[C], const uint32_t (&intra)[C], const EvalThr& th,
                                          uint64_t ovMask, uint64_t ovGood, ScanSt& st) {
    const int N = S.N, nreq = S.nreq;
    const uint8_t* lut = S.ctl->lut;
    const Samples<C> sp = samples_of<C>(S, p);
    const size_t stride = S.sStride;
    int s = st.s;
    uint64_t dA = 0, dB = 0;
    uint32_t cA = 0, cB = 0;
    if (s < N) load_sample<C>(sp, s * stride, dA, cA);
    if (s + 1 < N) load_sample<C>(sp, (s + 1) * stride, dB, cB);
    for (int k = s + 2; k < min(N, s + 2 + kScanPrefetch); ++k) prefetch_sample<C>(sp, k * stride);
    while (st.nGood < nreq && s < N) {
        const uint64_t d = dA;
        const uint32_t c2 = cA;
        dA = dB;
        cA = cB;
        if (s + 2 < N) {
            load_sample<C>(sp, (s + 2) * stride, dB, cB);
            if (s + 2 + kScanPrefetch < N) prefetch_sample<C>(sp, (s + 2 + kScanPrefetch) * stride);
        }
        if (!REC && ((ovMask >> s) & 1ull)) {
            st.nGood += (int)((ovGood >> s) & 1ull);
        } else {
            uint32_t dd, sd;
            if (sample_match<C>(lut, vals, curr, intra, th, d, c2, dd, sd)) {
                st.minDesc = min(st.minDesc, dd);
                st.minSum = min(st.minSum, sd);
                if (REC) {
                    if (st.g0 < 0) {
                        st.g0 = s;
                        st.g0d = dd;
                        st.g0s = sd;
                    } else if (st.g1 < 0) {
                        st.g1 = s;
                        st.g1d = dd;
                        st.g1s = sd;
                    }
                }
                ++st.nGood;
            }
        }
        ++s;
    }
    st.s = s;
}

// The ordered scan of one pixel's samples by eight lanes. One lane that walks 50 samples waits ~0.4 us for
// each (a chain of a sample's loads, LUT look-ups and ~130 instructions), 20 us in all, whatever the
// machine holds beside it; eight lanes take eight samples a step, and the ballot of their verdicts gives the
// ordered result: the scan stops at the nreq-th good sample, and samples past it count for nothing.
// A warp has four groups of eight lanes; lane j < m of a group owns an item (want: it has a scan to
// continue, from st), and the group scans its owners' items in turn. Every lane of the warp calls it. With
// eight owners a group (m == 8: a list that fills the machine) every lane scans its own item instead: the
// latency is then hidden by the other warps, and the groups' shuffles and the samples past the stop would
// cost issue slots (64-stream tick 6.39 ms with groups only, 6.35 ms before).
// ovMask: samples that earlier pixels overwrite this frame (repair), ovGood: those of them that match now
// (their distances stay with the owner). REC: also reports the first two good samples.
template <int C, bool REC>
__device__ __forceinline__ void coop_scan(const TickParams& P, bool want, int m, int si, int p,
                                          const uint32_t (&vals)[C][4], const uint32_t (&curr)[C],
                                          const uint32_t (&intra)[C], const EvalThr& th, uint64_t ovMask,
                                          uint64_t ovGood, ScanSt& st) {
    constexpr unsigned kAll = 0xffffffffu;
    const int lane = threadIdx.x & 31, sub = lane & 7;
    __syncwarp();
    if (m == 8) {
        if (want) lane_scan<C, REC>(P.streams[si], p, vals, curr, intra, th, ovMask, ovGood, st);
        return;
    }
    for (int j = 0; j < m; ++j) {
        const int src = (lane & 24) + j;
        const bool go = __shfl_sync(kAll, (int)want, src) != 0;
        if (!__any_sync(kAll, go)) continue;
        const int bsi = __shfl_sync(kAll, si, src), bp = __shfl_sync(kAll, p, src);
        uint32_t bv[C][4], bc[C], bi[C];
#pragma unroll
        for (int c = 0; c < C; ++c) {
#pragma unroll
            for (int i = 0; i < 4; ++i) bv[c][i] = __shfl_sync(kAll, vals[c][i], src);
            bc[c] = __shfl_sync(kAll, curr[c], src);
            bi[c] = __shfl_sync(kAll, intra[c], src);
        }
        EvalThr bt;
        bt.colThr = __shfl_sync(kAll, th.colThr, src);
        bt.descThr = __shfl_sync(kAll, th.descThr, src);
        bt.uNew = 0u;
        int s = __shfl_sync(kAll, st.s, src), ng = __shfl_sync(kAll, st.nGood, src);
        const uint64_t bm = REC ? 0ull : __shfl_sync(kAll, ovMask, src);
        const uint64_t bg = REC ? 0ull : __shfl_sync(kAll, ovGood, src);
        const StreamDev& S = P.streams[go ? bsi : 0];
        const int N = go ? S.N : 0, nreq = S.nreq;
        const uint8_t* lut = S.ctl->lut;
        const Samples<C> sp = samples_of<C>(S, bp);
        const size_t stride = S.sStride;
        int k = s + sub;
        uint64_t d = 0;
        uint32_t c2 = 0;
        if (k < N) load_sample<C>(sp, k * stride, d, c2);
        uint32_t mins = 0xffffffffu;  // descriptor minimum | summed minimum, 16 bits each
        uint32_t first = 0xffffffffu, second = 0xffffffffu;  // this lane's good samples: index, distances
        while (__any_sync(kAll, ng < nreq && s < N)) {
            __syncwarp();
            const bool act = ng < nreq && s < N;
            uint64_t dn = 0;
            uint32_t cn = 0;
            if (act && k + 8 < N) load_sample<C>(sp, (k + 8) * stride, dn, cn);
            uint32_t dd = 0, sd = 0;
            const bool good = act && k < N && (REC || !((bm >> k) & 1ull)) &&
                              sample_match<C>(lut, bv, bc, bi, bt, d, c2, dd, sd);
            uint32_t b = (__ballot_sync(kAll, good) >> (lane & 24)) & 0xffu;
            if (act) {
                if (!REC) b |= (uint32_t)(bg >> s) & 0xffu;
                const int need = nreq - ng, cnt = __popc(b);
                int stop = min(8, N - s);
                if (cnt >= need) {
                    uint32_t t = b;
                    for (int i = 1; i < need; ++i) t &= t - 1u;
                    stop = __ffs(t);
                    ng = nreq;
                } else {
                    ng += cnt;
                }
                if (good && sub < stop) {
                    mins = __vminu2(mins, (dd << 16) | sd);
                    if (REC) {
                        const uint32_t key = ((uint32_t)k << 24) | (dd << 16) | sd;
                        if (first == 0xffffffffu) first = key;
                        else if (second == 0xffffffffu) second = key;
                    }
                }
                s += stop;
            }
            d = dn;
            c2 = cn;
            k += 8;
        }
#pragma unroll
        for (int o = 4; o > 0; o >>= 1) mins = __vminu2(mins, __shfl_xor_sync(kAll, mins, o));
        uint32_t k0 = 0xffffffffu, k1 = 0xffffffffu;
        if (REC) {
            k0 = first;
#pragma unroll
            for (int o = 4; o > 0; o >>= 1) k0 = min(k0, __shfl_xor_sync(kAll, k0, o));
            k1 = first == k0 ? second : first;
#pragma unroll
            for (int o = 4; o > 0; o >>= 1) k1 = min(k1, __shfl_xor_sync(kAll, k1, o));
        }
        if (go && sub == j) {
            st.s = s;
            st.nGood = ng;
            st.minDesc = min(st.minDesc, mins >> 16);
            st.minSum = min(st.minSum, mins & 0xffffu);
            if (REC) {
                if (st.g0 < 0 && k0 != 0xffffffffu) {
                    st.g0 = (int)(k0 >> 24);
                    st.g0d = (k0 >> 16) & 0xffu;
                    st.g0s = k0 & 0xffffu;
                    k0 = k1;
                }
                if (st.g0 >= 0 && st.g1 < 0 && k0 != 0xffffffffu) {
                    st.g1 = (int)(k0 >> 24);
                    st.g1d = (k0 >> 16) & 0xffu;
                    st.g1s = k0 & 0xffffu;
                }
            }
        }
    }
}
// Items of a list that one group of eight lanes owns at a time: one while the machine has a group for
// every item, up to four, then eight (every lane owns one and scans it alone). Re-match round 0 with all
// groups / lanes alone from 5 / from 3 on: 24,000 items (three a group) 46 / 46 / 52 us, 42,000 (five)
// 75 / 70 / 70 us, 122,000 on a quarter of the machine 321 / 231 / 231 us.
__device__ __forceinline__ int coop_share(unsigned int n, unsigned int ctas) {
    const unsigned int groups = ctas * (blockDim.x >> 5) * 4u;
    const unsigned int m = (n + groups - 1u) / groups;
    return m > 4u ? 8 : (int)max(1u, m);
}

// the rest of one evaluation after the sample scan (:254-330 / :396-481): D_last, D_min, the raw
// segmentation averages, the model/neighbour update decisions and draws, T, v and R; writes the
// next-frame maps and returns the intent word
template <int C>
__device__ uint32_t eval_tail(const StreamDev& S, const FrameK& F, int x, int y, int p, const PixIn<C>& in,
                              const uint32_t (&curr)[C], const uint32_t (&intra)[C], uint32_t uNew,
                              const ScanSt& st) {
    const int npx = S.npx;
    float* fn = S.fm + (size_t)F.nxt * kNumFloatMaps * npx;
    float R = in.R, V = in.V, T = in.T;
    const float DL = in.DL;
    float DmLT = in.DmLT, DmST = in.DmST, RwLT = in.RwLT, RwST = in.RwST;
    const uint32_t lastFG = in.lastFG, blink = in.blink;
    const int nreq = S.nreq, nGood = st.nGood, s = st.s;
    const uint32_t minDesc = st.minDesc, minSum = st.minSum;

    // D_last (:254-255 / :396-397): depends on the pixel alone. With three channels the reference
    // takes the colour term from lv::L1dist<3>(const uchar*, const uchar*) (math.hpp:226-232), whose
    // accumulator type is that of L1dist(uchar, uchar), unsigned char: the sum wraps modulo 256.
    uint32_t l1 = 0, hd = 0;
#pragma unroll
    for (int c = 0; c < C; ++c) {
        l1 += (uint32_t)abs((int)in.lc[c] - (int)curr[c]);
        hd += __popc(in.ld[c] ^ intra[c]);
    }
    if (C == 3) l1 &= 0xffu;
    const float* divCol = C == 1 ? g_div_col1 : g_div_col3;    // i / 255 or i / 765
    const float* divDesc = C == 1 ? g_div_desc1 : g_div_desc3;  // i / 16 or i / 48
    const float normLast = (__ldg(&divCol[l1]) + __ldg(&divDesc[hd])) / 2;
    const float DLn = DL * (1.0f - F.fST) + normLast * F.fST;

    uint32_t intent = kInValid | ((uint32_t)s << kInEShift);
    DrawState ds;
    ds.blk = 0xffffffffu;
    const uint32_t seedFrame = F.frame;
    const bool fg = nGood < nreq;
    if (fg) {
        const float md = (__ldg(&divCol[minSum]) + __ldg(&divDesc[minDesc])) / 2 + (float)(nreq - nGood) / (float)nreq;
        const float nmd = fmin_std(1.0f, md);
        DmLT = DmLT * (1.0f - F.fLT) + nmd * F.fLT;
        DmST = DmST * (1.0f - F.fST) + nmd * F.fST;
        RwLT = RwLT * (1.0f - F.fLT) + F.fLT;
        RwST = RwST * (1.0f - F.fST) + F.fST;
        intent |= kInFG;
        if (F.cooldown && (draw_k(S.seed, seedFrame, (uint32_t)p, 0u, ds) % 2u) == 0u) {
            const uint32_t so = mod_n(draw_k(S.seed, seedFrame, (uint32_t)p, 1u, ds), S);
            intent |= kInOwn | (so << kInSOwnShift);
        }
    } else {
        const float nmd = (__ldg(&divCol[minSum]) + __ldg(&divDesc[minDesc])) / 2;
        DmLT = DmLT * (1.0f - F.fLT) + nmd * F.fLT;
        DmST = DmST * (1.0f - F.fST) + nmd * F.fST;
        RwLT = RwLT * (1.0f - F.fLT);
        RwST = RwST * (1.0f - F.fST);
        const unsigned long long nLR = S.lrMode ? S.lrFixed : (unsigned long long)__float2ull_rz(ceilf(T));
        uint32_t k = 0;
        if (mod_draw(draw_k(S.seed, seedFrame, (uint32_t)p, k++, ds), nLR) == 0ull) {
            const uint32_t so = mod_n(draw_k(S.seed, seedFrame, (uint32_t)p, k++, ds), S);
            intent |= kInOwn | (so << kInSOwnShift);
        }
        const bool use3 = F.use3x3 && !uNew;
        const uint32_t rn = draw_k(S.seed, seedFrame, (uint32_t)p, k++, ds);
        int nx, ny;
        if (use3) nb3_offset((int)(rn % 8u), nx, ny);
        else nb5_offset((int)(rn % 24u), nx, ny);
        nx += x;
        ny += y;
        clamp_xy(nx, ny, S.W, S.H);
        const uint32_t code = (uint32_t)((ny - y + 2) * 5 + (nx - x + 2));
        const uint32_t nrand = draw_k(S.seed, seedFrame, (uint32_t)p, k++, ds);
        const unsigned long long X = use3 ? nLR : (nLR / 2ull + 1ull);
        uint32_t st;
        if (mod_draw(nrand, X) == 0ull) st = NB_WRITE;
        else if (mod_draw(nrand, (unsigned long long)__float2ull_rz(F.t_lo)) == 0ull) st = NB_PENDING;
        else st = NB_NO;
        const uint32_t snb = mod_n(draw_k(S.seed, seedFrame, (uint32_t)p, k, ds), S);
        intent |= (code << kInCodeShift) | (st << kInNStShift) | (snb << kInSNbShift);
    }

    // feedback: T (:302-311), v (:312-318), R (:319-325)
    const float mn = fmin_std(DmLT, DmST), mx = fmax_std(DmLT, DmST);
    if (lastFG || (mn < 0.100f && fg)) {
        if (T < F.t_hi) T += 0.5000f / (mx * V);
    } else if (T > F.t_lo) {
        T -= 0.2500f * V / mx;
    }
    if (T < F.t_lo) T = F.t_lo;
    else if (T > F.t_hi) T = F.t_hi;
    if (mx > 0.100f && blink) {
        V += 1.000f;
    } else if (V > 0.100f) {
        V -= lastFG ? 0.100f / 4 : uNew ? 0.100f / 2 : 0.100f;
        if (V < 0.100f) V = 0.100f;
    }
    // R < pow(1+2*min, 2) is evaluated in double by the reference; x*x of a float is exact in
    // double, so compare exactly with the two-product split hi + lo of x*x
    const float rx = 1.0f + mn * 2;
    const float hi = rx * rx;
    const float lo = fmaf(rx, rx, -hi);
    if (R < hi || (R == hi && lo > 0.0f)) {
        R += 0.01f * (V - 0.100f);
    } else {
        R -= 0.01f / V;
        if (R < 1.0f) R = 1.0f;
    }
    fn[FM_R * npx + p] = R;
    fn[FM_V * npx + p] = V;
    fn[FM_T * npx + p] = T;
    __stcg(&fn[FM_DLAST * npx + p], DLn);
    fn[FM_DMIN_LT * npx + p] = DmLT;
    fn[FM_DMIN_ST * npx + p] = DmST;
    fn[FM_RAW_LT * npx + p] = RwLT;
    __stcg(&fn[FM_RAW_ST * npx + p], RwST);
    S.unst[(size_t)F.nxt * npx + p] = (uint8_t)uNew;
    uint8_t* lcn = S.lastCol + (size_t)F.nxt * npx * C + (size_t)p * C;
    uint16_t* ldn = S.lastDesc + (size_t)F.nxt * npx * C + (size_t)p * C;
#pragma unroll
    for (int c = 0; c < C; ++c) {
        lcn[c] = (uint8_t)curr[c];
        __stcg(&ldn[c], (uint16_t)intra[c]);
    }
    return intent;
}

// non-zero LBSP descriptor test of the frame-level statistics (:264-265 / :405-407)
template <int C>
__device__ __forceinline__ int desc_nonzero(const uint32_t (&intra)[C]) {
    uint32_t pc = 0;
#pragma unroll
    for (int c = 0; c < C; ++c) pc += __popc(intra[c]);
    return pc >= (C == 1 ? 2u : 4u) ? 1 : 0;
}

// adds two per-thread counts (below 2^24) of a tile block to per-stream counters with one atomic each per
// block (every thread of the block calls it)
__device__ __forceinline__ void block_add_stats(unsigned long long* a, unsigned int va, unsigned long long* b,
                                                unsigned int vb) {
    __shared__ unsigned int red[2][kThreads / 32];
    const unsigned int sa = __reduce_add_sync(0xffffffffu, va), sb = __reduce_add_sync(0xffffffffu, vb);
    if ((threadIdx.x & 31) == 0) {
        red[0][threadIdx.x >> 5] = sa;
        red[1][threadIdx.x >> 5] = sb;
    }
    __syncthreads();
    if (threadIdx.x < 2) {
        unsigned long long t = 0;
        for (int i = 0; i < (int)(blockDim.x >> 5); ++i) t += red[threadIdx.x][i];
        if (t) atomicAdd(threadIdx.x ? b : a, t);
    }
}

// gathers the 16 LBSP taps of channel c at (x, y) from a byte image (tile or frame)
template <int C>
__device__ __forceinline__ void gather_taps(const uint8_t* base, int rowStride, int c, uint32_t (&v)[4]) {
#pragma unroll
    for (int j = 0; j < 4; ++j) {
        uint32_t w = 0;
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const int n = j * 4 + i;
            w |= (uint32_t)base[lbsp_dy(n) * rowStride + lbsp_dx(n) * C + c] << (8 * i);
        }
        v[j] = w;
    }
}

// the evaluation's shared-memory frame tile: byte 0 of a tile row buffer is kTileDelta<C> bytes before
// the frame byte (x0-2)*C - 2 of the tile's leftmost tap, which puts it on a 16-byte boundary of the
// frame row (x0 = 32 * tile column: (96k - 8) - 8 for C = 3, (32k - 4) - 12 for C = 1); kTileRW<C> is
// the row stride, a multiple of 16 that covers the (kTileW + 4) * C + 2 bytes of taps after the delta
template <int C>
constexpr int kTileDelta = C == 3 ? 8 : 12;
template <int C>
constexpr int kTileRW = (kTileDelta<C> + (kTileW + 2 * kBorder) * C + 2 + 15) / 16 * 16;
static_assert(kTileW == 32 && kBorder == 2, "the tile deltas assume 32-pixel tile columns and a 2-pixel border");

// ------------------------------------------------------------------------------------------
// phase A: evaluate every pixel of a tile against the frame-start model
// ------------------------------------------------------------------------------------------
template <int C>
__device__ void phaseA_tile(const TickParams& P, int si, const StreamDev& S, int lt, uint8_t* smem) {
    const int tx = lt % S.tilesX, ty = lt / S.tilesX;
    const int x0 = tx * kTileW, y0 = ty * kTileH;
    // The tile holds rows y0-2 .. y0+9 of the frame. The taps of the tile's pixels span frame bytes
    // b0 = (x0-2)*C - 2 .. b0 + (kTileW+4)*C + 1 of a row; a tile row buffer starts kTileDelta<C> bytes
    // before b0, at a 16-byte boundary of the row (x0 is a multiple of 32), so it is filled with
    // aligned 128-bit loads when the frame rows are 16-byte aligned (else 32-bit words, or bytes).
    constexpr int RW = kTileRW<C>;  // tile row stride (bytes)
    constexpr int NCH = RW / 16;    // 16-byte chunks per tile row
    constexpr int RH = kTileH + 2 * kBorder;
    const FrameK F = frame_consts(S);
    const int lx = threadIdx.x % kTileW, ly = threadIdx.x / kTileW;
    const int x = x0 + lx, y = y0 + ly;
    const bool inFrame = x < S.W && y < S.H;
    const int p = y * S.W + x;
    const bool active = inFrame && S.roi[p] != 0;
    // the scan's inputs first (they overlap the tile load below); the other maps after the scan
    float tR = 0, tRwLT = 0, tRwST = 0, tFnLT = 0, tFnST = 0;
    uint32_t tU = 0, c0 = 0, c1 = 0;
    uint64_t d0 = 0, d1 = 0;
    const Samples<C> sp = samples_of<C>(S, active ? p : 0);
    if (active) {
        const int npx = S.npx;
        const float* fc = S.fm + (size_t)F.cur * kNumFloatMaps * npx;
        tR = fc[FM_R * npx + p];
        tRwLT = fc[FM_RAW_LT * npx + p];
        tRwST = fc[FM_RAW_ST * npx + p];
        tFnLT = fc[FM_FIN_LT * npx + p];
        tFnST = fc[FM_FIN_ST * npx + p];
        tU = S.unst[(size_t)F.cur * npx + p];
        if (S.N > 0) load_sample<C>(sp, 0, d0, c0);
        if (S.N > 1) load_sample<C>(sp, S.sStride, d1, c1);
    }
    uint8_t* tile = smem;
    uint8_t* lut = smem + RW * RH;
    for (int i = threadIdx.x; i < 256; i += blockDim.x) lut[i] = S.ctl->lut[i];
    const long rowBytes = (long)S.W * C;
    const long ws = (long)(x0 - kBorder) * C - 2 - kTileDelta<C>;  // frame byte of a tile row buffer's byte 0
    const bool vecPath = (rowBytes & 15) == 0 && (((uintptr_t)S.frame) & 15) == 0;
    const bool wordPath = (rowBytes & 3) == 0 && (((uintptr_t)S.frame) & 3) == 0;
    for (int i = threadIdx.x; i < NCH * RH; i += blockDim.x) {
        const int r = i / NCH, ci = i % NCH;
        const int gy = y0 - kBorder + r;
        const long b = ws + 16 * ci;
        uint4 v = make_uint4(0u, 0u, 0u, 0u);
        if (gy >= 0 && gy < S.H) {
            const uint8_t* row = S.frame + (size_t)gy * rowBytes;
            if (vecPath && b >= 0 && b + 16 <= rowBytes) {
                v = __ldg((const uint4*)(row + b));
            } else {
                uint32_t w[4];
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    const long bw = b + 4 * j;
                    w[j] = 0;
                    if (wordPath && bw >= 0 && bw + 4 <= rowBytes) {
                        w[j] = __ldg((const uint32_t*)(row + bw));
                    } else {
                        for (int k = 0; k < 4; ++k)
                            if (bw + k >= 0 && bw + k < rowBytes) w[j] |= (uint32_t)__ldg(row + bw + k) << (8 * k);
                    }
                }
                v = make_uint4(w[0], w[1], w[2], w[3]);
            }
        }
        *(uint4*)(tile + r * RW + 16 * ci) = v;
    }
    __syncthreads();
    int nz = 0;
    bool defer = false;
    unsigned long long scanWord = 0;
    if (inFrame) {
        uint32_t intent = 0;
        if (active) {
            const uint8_t* base = tile + (ly + kBorder) * RW + kTileDelta<C> + (lx + kBorder) * C + 2;
            uint32_t vals[C][4], curr[C], intra[C];
#pragma unroll
            for (int c = 0; c < C; ++c) {
                gather_taps<C>(base, RW, c, vals[c]);
                curr[c] = base[c];
                intra[c] = lbsp_thr(vals[c], curr[c], lut[curr[c]]);
            }
            nz = desc_nonzero<C>(intra);
            const EvalThr th = eval_thresholds(S, tR, tRwLT, tRwST, tFnLT, tFnST, tU);
            ScanSt st;
            scan_init<C>(st);
            scan_samples<C>(S, lut, sp, vals, curr, intra, th, d0, c0, d1, c1, st);
            if (st.nGood < S.nreq) {
                // a long scan, or a scan that ended unsettled within the cap (N <= kScanCap): continued,
                // recorded and finished by lvbgs_k_longscan over the compacted list, so that its warps
                // hold only long scans
                defer = true;
                // s | nGood | first good index (255: none) | minDesc | minSum
                scanWord = (unsigned long long)st.s | ((unsigned long long)st.nGood << 8) |
                           ((unsigned long long)(st.g0 < 0 ? 255 : st.g0) << 16) |
                           ((unsigned long long)st.minDesc << 32) | ((unsigned long long)st.minSum << 48);
            } else {
                PixIn<C> in;
                load_pix<C>(S, F, p, in);
                intent = eval_tail<C>(S, F, x, y, p, in, curr, intra, th.uNew, st);
            }
        }
        __stcg(&S.intent[p], intent);
    }
    {
        // warp-aggregated append to the long-scan list (pixel key, scan state)
        const unsigned m = __ballot_sync(0xffffffffu, defer);
        if (m) {
            const int lane = threadIdx.x & 31, leader = __ffs(m) - 1;
            unsigned int base = 0;
            if (lane == leader) base = atomicAdd(&P.work->lcount, (unsigned int)__popc(m));
            base = __shfl_sync(0xffffffffu, base, leader);
            if (defer) {
                const unsigned int i = base + (unsigned int)__popc(m & ((1u << lane) - 1u));
                if (i < P.listCap) {
                    P.rlist[0][i] = ((unsigned long long)si << 40) | (unsigned long long)(unsigned)p;
                    P.rlist[1][i] = scanWord;
                } else {
                    atomicOr(&P.work->err, ERR_REPAIR_LIMIT);
                }
            }
        }
    }
    // per-warp reduction of the non-zero descriptor count (final: the descriptor does not depend
    // on the repair)
    for (int o = 16; o > 0; o >>= 1) nz += __shfl_xor_sync(0xffffffffu, nz, o);
    if ((threadIdx.x & 31) == 0 && nz) atomicAdd(&S.ctl->nz_acc, (unsigned long long)nz);
}

// ------------------------------------------------------------------------------------------
// list helpers for the repair loop
// ------------------------------------------------------------------------------------------
// push of one item from divergent code: the lanes that arrive together share one counter atomic
// (the counters are shared by all streams, and same-address atomics serialize)
__device__ __forceinline__ void push_item(unsigned long long* list, unsigned int* count, unsigned int cap,
                                          uint32_t* stamps, uint32_t stamp, int si, int p, TickWork* w) {
    if (atomicExch(&stamps[p], stamp) == stamp) return;
    const unsigned am = __activemask();
    const int lane = threadIdx.x & 31, leader = __ffs(am) - 1;
    unsigned int base = 0;
    if (lane == leader) base = atomicAdd(count, (unsigned int)__popc(am));
    base = __shfl_sync(am, base, leader);
    const unsigned int i = base + (unsigned int)__popc(am & ((1u << lane) - 1u));
    if (i < cap) list[i] = ((unsigned long long)si << 40) | (unsigned long long)(unsigned)p;
    else atomicOr(&w->err, ERR_REPAIR_LIMIT);
}

// target pixel of a neighbour code relative to (x, y)
__device__ __forceinline__ int code_target(int code, int x, int y, int W) {
    const int dy = code / 5 - 2, dx = code % 5 - 2;
    return (y + dy) * W + (x + dx);
}

// ghost test of pixel p's neighbour update (:292-295 / :438-441), reading the target's values as
// the raster scan would: this frame's value when the target precedes (or is) p, else the previous
// frame's
__device__ __forceinline__ uint32_t resolve_ghost(const StreamDev& S, const FrameK& F, int p, int q) {
    const int npx = S.npx;
    const int buf = (q <= p) ? F.nxt : F.cur;
    const float* fb = S.fm + (size_t)buf * kNumFloatMaps * npx;
    const float qD = __ldcg(&fb[FM_DLAST * npx + q]);
    const float qR = __ldcg(&fb[FM_RAW_ST * npx + q]);
    return (qR > 0.995f && qD < 0.010f) ? NB_GHOST_WRITE : NB_GHOST_NO;
}

__device__ __forceinline__ uint32_t set_nst(uint32_t w, uint32_t st) {
    return (w & ~(7u << kInNStShift)) | (st << kInNStShift);
}

// phase B: resolve pending ghost tests with the phase-A values; mark the pixels whose evaluated
// samples an earlier pixel overwrites (initial repair frontier). A block takes kResolveTiles tiles,
// one pixel of each per thread, with the loads of all of them issued before any is used: the work
// is a short chain of dependent loads per pixel, so more pixels in flight per thread hide it.
__device__ void phaseB_tiles(const TickParams& P, int t0) {
    // the stream of each tile and its stamp, found once per block
    __shared__ int sSi[kResolveTiles];
    __shared__ uint32_t sStamp[kResolveTiles];
    if (threadIdx.x < kResolveTiles) {
        const int t = t0 + (int)threadIdx.x;
        int si = 0;
        uint32_t stamp = 0;
        if (t < P.totalTiles) {
            si = find_stream_by_tile(P, t);
            stamp = P.streams[si].ctl->stamp_base + 1u;
        }
        sSi[threadIdx.x] = si;
        sStamp[threadIdx.x] = stamp;
    }
    __syncthreads();
    uint32_t w[kResolveTiles];
    int ps[kResolveTiles], xs[kResolveTiles], ys[kResolveTiles];
#pragma unroll
    for (int j = 0; j < kResolveTiles; ++j) {
        const int t = t0 + j;
        w[j] = 0u;
        ps[j] = xs[j] = ys[j] = 0;
        if (t < P.totalTiles) {
            const StreamDev& S = P.streams[sSi[j]];
            const int lt = t - S.tileBase;
            const int x = (lt % S.tilesX) * kTileW + threadIdx.x % kTileW;
            const int y = (lt / S.tilesX) * kTileH + threadIdx.x / kTileW;
            xs[j] = x;
            ys[j] = y;
            if (x < S.W && y < S.H) {
                ps[j] = y * S.W + x;
                w[j] = __ldcg(&S.intent[ps[j]]);
            }
        }
    }
    int qs[kResolveTiles];
    uint32_t wq[kResolveTiles];
#pragma unroll
    for (int j = 0; j < kResolveTiles; ++j) {
        qs[j] = 0;
        wq[j] = 0u;
        if (!(w[j] & kInValid)) continue;
        const StreamDev& S = P.streams[sSi[j]];
        if (in_nst(w[j]) == NB_PENDING) {
            const FrameK F = frame_consts(S);
            w[j] = set_nst(w[j], resolve_ghost(S, F, ps[j], code_target((int)in_code(w[j]), xs[j], ys[j], S.W)));
            __stcg(&S.intent[ps[j]], w[j]);
        }
        if (in_nb_writes(w[j])) {
            qs[j] = code_target((int)in_code(w[j]), xs[j], ys[j], S.W);
            if (qs[j] > ps[j]) wq[j] = __ldcg(&S.intent[qs[j]]);
        }
    }
    // one list item per target and stamp generation. The four tiles' items are reserved together: one
    // counter atomic per block (the counter is shared by all streams, and same-address atomics serialize)
    bool ok[kResolveTiles];
#pragma unroll
    for (int j = 0; j < kResolveTiles; ++j) {
        const bool want = (w[j] & kInValid) && in_nb_writes(w[j]) && qs[j] > ps[j] && (wq[j] & kInValid) &&
                          in_snb(w[j]) < in_e(wq[j]);
        ok[j] = want && atomicExch(&P.streams[sSi[j]].stampD[qs[j]], sStamp[j]) != sStamp[j];
    }
    __shared__ unsigned int sWarp[kThreads / 32], sBase;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    unsigned int mine[kResolveTiles], cnt = 0;
#pragma unroll
    for (int j = 0; j < kResolveTiles; ++j) {
        const unsigned m = __ballot_sync(0xffffffffu, ok[j]);
        mine[j] = cnt + (unsigned)__popc(m & ((1u << lane) - 1u));
        cnt += (unsigned)__popc(m);
    }
    if (lane == 0) sWarp[warp] = cnt;
    __syncthreads();
    if (threadIdx.x == 0) {
        unsigned int run = 0;
#pragma unroll
        for (int i = 0; i < kThreads / 32; ++i) {
            const unsigned int v = sWarp[i];
            sWarp[i] = run;
            run += v;
        }
        sBase = run ? atomicAdd(&P.work->dcount[0], run) : 0u;
    }
    __syncthreads();
#pragma unroll
    for (int j = 0; j < kResolveTiles; ++j) {
        if (!ok[j]) continue;
        const unsigned int i = sBase + sWarp[warp] + mine[j];
        if (i < P.listCap) P.dlist[0][i] = ((unsigned long long)sSi[j] << 40) | (unsigned long long)(unsigned)qs[j];
        else atomicOr(&P.work->err, ERR_REPAIR_LIMIT);
    }
}

// frame down-sampling for the frame-level analysis (:568-584): one output pixel by a group of eight lanes;
// the averages of channel c are on lane c
template <int C>
__device__ void ds_item(const StreamDev& S, int i) {
    const int sub = threadIdx.x & 7;
    const unsigned mask = 0xffu << (threadIdx.x & 24);
    uint32_t v[C];
    area_resample_group<C>(S.frame, S.W, S.H, S.dsW, S.dsH, i % S.dsW, i / S.dsW, v);
    uint32_t d = 0;
    if (sub < C) {
        const FrameK F = frame_consts(S);
        uint32_t vc = v[0];
#pragma unroll
        for (int c = 1; c < C; ++c) vc = sub == c ? v[c] : vc;
        const size_t k = (size_t)i * C + sub;
        // accumulateWeighted: dst = src*a + dst*(1-a)
        const float aL = F.fLT, bL = 1.0f - aL, aS = F.fST, bS = 1.0f - aS;
        const float lt = (float)vc * aL + S.dsLT[k] * bL;
        const float st = (float)vc * aS + S.dsST[k] * bS;
        S.dsLT[k] = lt;
        S.dsST[k] = st;
        d = (uint32_t)__float2ull_rz(fabsf(st - lt));
        if (C == 1) d /= 2u;
    }
    // the largest difference of the channels (lanes 0-3 of the group hold them)
#pragma unroll
    for (int o = 1; o < 4; o <<= 1) d = max(d, __shfl_xor_sync(mask, d, o, 8));
    if (sub == 0 && d) atomicAdd(&S.ctl->colordiff_acc, (unsigned long long)d);
}

// Place of the length of round i's list: the lists themselves alternate, but a round without re-resolutions
// ends in one barrier, so the length that a round resets (that of round i + 2) must not be one that a CTA
// may still read: three places rotate after round 0's.
__device__ __forceinline__ int dcount_slot(int i) { return i == 0 ? 0 : 1 + (i - 1) % 3; }

// ------------------------------------------------------------------------------------------
// repair loop bodies
// ------------------------------------------------------------------------------------------
// Re-matches the items of a warp's owner lanes (own: this lane holds pixel q of stream si; every lane of
// the warp calls it): the scan of q's samples with those that earlier pixels overwrite this frame, the tail
// of its evaluation, and the list entries that follow from a changed decision.
template <int C>
__device__ bool rematch_items(const TickParams& P, bool own, int m, int si, int q, uint32_t stampNext, int iter) {
    const StreamDev& S = P.streams[si];
    const int W = S.W, x = q % W, y = q / W;
    const FrameK F = frame_consts(S);
    const uint32_t wOld = own ? __ldcg(&S.intent[q]) : 0u;
    own = own && (wOld & kInValid);
    // overrides: earlier pixels of the 5x5 window whose neighbour update targets q, raster order. All
    // twelve intents are requested before any is looked at.
    Ovr ov[12];
    int nov = 0;
    uint64_t mask = 0, good = 0;
    uint32_t vals[C][4], curr[C], intra[C];
    PixIn<C> in;
    EvalThr th;
    ScanSt st;
    scan_init<C>(st);
    th.colThr = th.descThr = th.uNew = 0u;
#pragma unroll
    for (int c = 0; c < C; ++c) {
        curr[c] = intra[c] = 0u;
#pragma unroll
        for (int j = 0; j < 4; ++j) vals[c][j] = 0u;
    }
    bool scan = own;
    if (own) {
        uint32_t wn[12];
#pragma unroll
        for (int j = 0; j < 12; ++j) {
            const int dy = j / 5 - 2, dx = j % 5 - 2;
            const int px = x + dx, py = y + dy;
            wn[j] = (px >= 0 && px < W && py >= 0) ? __ldcg(&S.intent[py * W + px]) : 0u;
        }
        const uint4 gr = S.nreq <= 2 ? __ldcg(&S.goodRec[q]) : make_uint4(0u, 0u, 0u, 0u);
        const uint8_t* base = S.frame + (size_t)q * C;
#pragma unroll
        for (int c = 0; c < C; ++c) {
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                uint32_t wv = 0;
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    const int n = j * 4 + i;
                    wv |= (uint32_t)__ldg(base + (lbsp_dy(n) * W + lbsp_dx(n)) * C + c) << (8 * i);
                }
                vals[c][j] = wv;
            }
            curr[c] = __ldg(base + c);
        }
        load_pix<C>(S, F, q, in);
        th = eval_thresholds(S, in.R, in.RwLT, in.RwST, in.FnLT, in.FnST, in.uOld);
#pragma unroll
        for (int c = 0; c < C; ++c) intra[c] = lbsp_thr(vals[c], curr[c], S.ctl->lut[curr[c]]);
        for (int j = 0; j < 12; ++j) {
            const uint32_t w = wn[j];
            if (!in_nb_writes(w) || (int)in_code(w) != 24 - j) continue;
            const int p = (y + j / 5 - 2) * W + x + j % 5 - 2;
            const int sn = (int)in_snb(w);
            uint32_t col = 0;
            uint64_t desc = 0;
            const uint16_t* ldn = S.lastDesc + (size_t)F.nxt * S.npx * C + (size_t)p * C;
            for (int c = 0; c < C; ++c) {
                col |= (uint32_t)__ldg(S.frame + (size_t)p * C + c) << (8 * c);
                desc |= (uint64_t)__ldcg(&ldn[c]) << (16 * c);
            }
            int k = 0;
            while (k < nov && ov[k].s != sn) ++k;
            if (k == nov) ++nov;
            ov[k].s = sn;
            ov[k].col = col;
            ov[k].desc = desc;
            mask |= 1ull << sn;
        }
        // order matters only within one sample index (last writer wins); entries with distinct s are
        // independent, and an overwritten entry keeps its slot but takes the latest writer's values.
        // The overwritten samples that match now: their entries keep the distances (col, desc)
        for (int k = 0; k < nov; ++k) {
            uint64_t d;
            uint32_t c2;
            if (C == 3) {
                d = ov[k].desc | ((uint64_t)(ov[k].col & 0xffffu) << 48);
                c2 = (ov[k].col >> 16) & 0xffu;
            } else {
                d = ov[k].desc & 0xffffu;
                c2 = ov[k].col & 0xffu;
            }
            uint32_t dd, sd;
            if (sample_match<C>(S.ctl->lut, vals, curr, intra, th, d, c2, dd, sd)) {
                good |= 1ull << ov[k].s;
                ov[k].col = dd;
                ov[k].desc = sd;
            }
        }
        if (S.nreq <= 2 && gr.x == F.frame) {
            // q's frame-start scan is recorded: up to its stop eA, its good samples are the recorded ones
            // not overwritten and the overwritten ones that match now. The ordered scan over them stops
            // at the nreq-th good index, with minima over the good samples up to there; with fewer, it
            // goes on from eA (with the overwrites) as a scan from the start would.
            const int eA = (int)(gr.y & 255u), nA = (int)((gr.y >> 8) & 255u);
            int gi[2] = {S.N, S.N};  // the two smallest good indices
            uint32_t gd[2] = {0u, 0u}, gs[2] = {0u, 0u};
            int cnt = 0;
            auto add = [&](int idx, uint32_t dd, uint32_t sd) {
                ++cnt;
                if (idx < gi[0]) {
                    gi[1] = gi[0];
                    gd[1] = gd[0];
                    gs[1] = gs[0];
                    gi[0] = idx;
                    gd[0] = dd;
                    gs[0] = sd;
                } else if (idx < gi[1]) {
                    gi[1] = idx;
                    gd[1] = dd;
                    gs[1] = sd;
                }
            };
            for (int j = 0; j < nA; ++j) {
                const int g = (int)((gr.y >> (16 + 8 * j)) & 255u);
                if (!((mask >> g) & 1ull)) add(g, (j ? gr.z >> 16 : gr.z) & 0xffffu, (j ? gr.w >> 16 : gr.w) & 0xffffu);
            }
            for (int k = 0; k < nov; ++k)
                if (ov[k].s < eA && ((good >> ov[k].s) & 1ull)) add(ov[k].s, ov[k].col, (uint32_t)ov[k].desc);
            const int take = cnt < S.nreq ? cnt : S.nreq;
            for (int j = 0; j < take; ++j) {
                if (st.minDesc > gd[j]) st.minDesc = gd[j];
                if (st.minSum > gs[j]) st.minSum = gs[j];
            }
            st.nGood = take;
            st.s = cnt >= S.nreq ? gi[S.nreq > 0 ? S.nreq - 1 : 0] + 1 : eA;
            scan = cnt < S.nreq && eA < S.N;
        }
    }
    const int s0 = st.s;
    coop_scan<C, false>(P, scan, m, si, q, vals, curr, intra, th, mask, good, st);
    if (!own) return false;
    // the overwritten samples that the scan counted
    if (scan)
        for (int k = 0; k < nov; ++k)
            if (ov[k].s >= s0 && ov[k].s < st.s && ((good >> ov[k].s) & 1ull)) {
                st.minDesc = min(st.minDesc, ov[k].col);
                st.minSum = min(st.minSum, (uint32_t)ov[k].desc);
            }
    const int e = st.s;
    uint32_t wNew = eval_tail<C>(S, F, x, y, q, in, curr, intra, th.uNew, st);
    const bool decChanged = ((wNew ^ wOld) & kInFG) != 0u;
    if (!decChanged) {
        // same decision: same draws, same updates; keep the resolved neighbour state
        wNew = (wOld & ~(127u << kInEShift)) | ((uint32_t)e << kInEShift);
        __stcg(&S.intent[q], wNew);
        return true;
    }
    __stcg(&S.intent[q], wNew);
    unsigned int* dcnt = &P.work->dcount[dcount_slot(iter + 1)];
    unsigned long long* dl = P.dlist[(iter & 1) ^ 1];
    // the write that disappeared or appeared changes what its (later) target reads
    if (in_nb_writes(wOld)) {
        const int t = code_target((int)in_code(wOld), x, y, W);
        if (t > q) push_item(dl, dcnt, P.listCap, S.stampD, stampNext, si, t, P.work);
    }
    if (in_nb_writes(wNew)) {
        const int t = code_target((int)in_code(wNew), x, y, W);
        if (t > q) push_item(dl, dcnt, P.listCap, S.stampD, stampNext, si, t, P.work);
    }
    // the raw-segmentation value of q changed: re-resolve ghost tests that read it (q itself and
    // later pixels of its 5x5 window), and q's own new pending test
    unsigned long long* rl = P.rlist[iter & 1];
    unsigned int* rcnt = &P.work->rcount[iter & 1];
    const uint32_t rstamp = stampNext;  // separate stamp array: one generation per iteration
    uint32_t wl[13];  // q and the later pixels of its window, requested together
#pragma unroll
    for (int j = 0; j < 13; ++j) {
        const int px = x + (j + 12) % 5 - 2, py = y + (j + 12) / 5 - 2;
        wl[j] = j == 0 ? wNew : (px >= 0 && px < W && py < S.H) ? __ldcg(&S.intent[py * W + px]) : 0u;
    }
#pragma unroll
    for (int j = 0; j < 13; ++j)  // window slot 12 + j targets q with code 24 - (12 + j)
        if (in_ghost(wl[j]) && (int)in_code(wl[j]) == 12 - j)
            push_item(rl, rcnt, P.listCap, S.stampR, rstamp, si, (y + (j + 12) / 5 - 2) * W + x + (j + 12) % 5 - 2, P.work);
    if (in_nst(wNew) == NB_PENDING) push_item(rl, rcnt, P.listCap, S.stampR, rstamp, si, q, P.work);
    return true;
}

__device__ void reresolve_item(const TickParams& P, int si, const StreamDev& S, int p, uint32_t stampNext, int iter) {
    const int W = S.W, x = p % W, y = p / W;
    const uint32_t w = __ldcg(&S.intent[p]);
    if (!in_ghost(w)) return;
    const FrameK F = frame_consts(S);
    const int q = code_target((int)in_code(w), x, y, W);
    const uint32_t st = resolve_ghost(S, F, p, q);
    const uint32_t old = in_nst(w);
    if (st == old) return;
    __stcg(&S.intent[p], set_nst(w, st));
    // readers during the last re-match pass saw PENDING as "no write"
    const bool wroteBefore = old == NB_GHOST_WRITE, writesNow = st == NB_GHOST_WRITE;
    if (wroteBefore != writesNow && q > p)
        push_item(P.dlist[(iter & 1) ^ 1], &P.work->dcount[dcount_slot(iter + 1)], P.listCap, S.stampD, stampNext, si, q, P.work);
}

// ------------------------------------------------------------------------------------------
// phase F: commit the sample writes of the frame in raster order, the draw counters, the blink
// maps and the 3x3 closing (:536-540); initializes the union-find labels of the hole filling.
//
// The writes of a pixel come from its 5x5 window. Each intent of the tile and its 2-pixel halo sets its bit in
// the target's mask in shared memory (one atomic or for the intents that write), so a pixel walks the few
// set bits in raster order instead of comparing 25 intents. The closing works on the rows' foreground
// words: 36 pixels of a row in one 64-bit word, the same in every lane of the row's warp. Together 114 -> 111 us on a
// 1920x1080 BGR frame: what bounds it is DRAM's random sectors, one for each of the frame's sample writes (filled
// and written back), 88 us with a sample's descriptors and colours in one sector instead of two.
// ------------------------------------------------------------------------------------------
constexpr int kCommitIW = kTileW + 4, kCommitIH = kTileH + 4;  // intents with a 2-pixel halo
struct CommitSmem {
    uint32_t it[kCommitIH * kCommitIW];
    uint32_t wr[kTileH * kTileW];    // bit k (own write: 12, slots 12 to 24 one further): the writers of the pixel
    unsigned long long fg[kCommitIH];  // foreground words, bit b: pixel x0 - 2 + b
};
template <int C>
__device__ void phaseF_tile(const TickParams& P, const StreamDev& S, int lt, CommitSmem& sm) {
    constexpr int IW = kCommitIW, IH = kCommitIH;
    static_assert(kTileW == 32 && kThreads == kTileW * kTileH && IH <= 2 * kTileH, "a warp per tile row, two rows of intents");
    const int tx = lt % S.tilesX, ty = lt / S.tilesX;
    const int x0 = tx * kTileW, y0 = ty * kTileH;
    const int W = S.W, H = S.H, npx = S.npx;
    const int lx = threadIdx.x % kTileW, ly = threadIdx.x / kTileW;
    const int x = x0 + lx, y = y0 + ly, q = y * W + x;
    const bool inF = x < W && y < H;
    const uint8_t lastRaw = inF ? S.lastRawFG[q] : 0, lastRawBlink = inF ? S.lastRawBlink[q] : 0;
    // warp ly brings rows ly and ly + 8 of the intents: 32 of a row's, then its last 4
    uint32_t w0[2], w1[2];
#pragma unroll
    for (int h = 0; h < 2; ++h) {
        const int r = ly + h * kTileH, gy = y0 - 2 + r, gx = x0 - 2 + lx;
        const bool row = r < IH && gy >= 0 && gy < H;
        w0[h] = row && gx >= 0 && gx < W ? __ldcg(&S.intent[gy * W + gx]) : 0u;
        w1[h] = row && lx < 4 && gx + kTileW < W ? __ldcg(&S.intent[gy * W + gx + kTileW]) : 0u;
    }
    sm.wr[threadIdx.x] = 0u;
    __syncthreads();
#pragma unroll
    for (int h = 0; h < 2; ++h) {
        const int r = ly + h * kTileH;
        if (r >= IH) break;
        const unsigned long long lo = __ballot_sync(0xffffffffu, w0[h] & kInFG), hi = __ballot_sync(0xffffffffu, w1[h] & kInFG);
        if (lx == 0) sm.fg[r] = lo | (hi << 32);
#pragma unroll
        for (int g = 0; g < 2; ++g) {
            if (g == 1 && lx >= 4) break;
            const uint32_t w = g ? w1[h] : w0[h];
            const int cx = lx + 32 * g;
            sm.it[r * IW + cx] = w;
            if (!(w & kInValid)) continue;
            // a writer at window slot k = (dy + 2) * 5 + (dx + 2) of its target has code 24 - k
            const uint32_t code = in_code(w), cy5 = (code * 13u) >> 6;
            const int qx = cx + (int)(code - 5u * cy5) - 4, qy = r + (int)cy5 - 4;  // the target in the tile
            if (in_nb_writes(w) && (unsigned)qx < (unsigned)kTileW && (unsigned)qy < (unsigned)kTileH) {
                const uint32_t k = 24u - code;
                atomicOr(&sm.wr[qy * kTileW + qx], 1u << (k + (k >= 12u ? 1u : 0u)));
            }
            const int ox = cx - 2, oy = r - 2;
            if ((w & kInOwn) && (unsigned)ox < (unsigned)kTileW && (unsigned)oy < (unsigned)kTileH)
                atomicOr(&sm.wr[oy * kTileW + ox], 1u << 12);
        }
    }
    __syncthreads();
    const FrameK F = frame_consts(S);
    // closing of the raw mask: dilated rows of the window's three rows, eroded; out-of-frame pixels never win
    unsigned long long closed = ~0ull;
    {
        const int left = max(0, 2 - x0), right = min(IW, W - x0 + 2);  // the window's columns inside the frame
        const unsigned long long outside = ~(((1ull << (right - left)) - 1ull) << left);
        unsigned long long f[5];
#pragma unroll
        for (int j = 0; j < 5; ++j) f[j] = sm.fg[ly + j];
#pragma unroll
        for (int j = 0; j < 3; ++j) {
            const int gy = y - 1 + j;
            const unsigned long long m = f[j] | f[j + 1] | f[j + 2], d = m | (m << 1) | (m >> 1) | outside;
            if (gy >= 0 && gy < H) closed &= d & (d << 1) & (d >> 1);
        }
    }
    const uint32_t closedW = (uint32_t)(closed >> 2);
    const uint32_t wq = sm.it[(ly + 2) * IW + lx + 2];
    uint32_t todo = sm.wr[threadIdx.x];
    const Samples<C> sp = samples_of<C>(S, inF ? q : 0);
    // the writes, by the warp together: a write body per step instead of one per window slot that any lane uses
    while (__any_sync(0xffffffffu, todo)) {
        if (todo) {
            const int b = __ffs(todo) - 1, k = b - (b >= 13 ? 1 : 0);
            todo &= todo - 1u;
            const int ky = (k * 13) >> 6, kx = k - 5 * ky;
            const uint32_t w = sm.it[(ly + ky) * IW + lx + kx];
            const size_t s = b == 12 ? in_sown(w) : in_snb(w);
            const int p = (y + ky - 2) * W + x + kx - 2;
            // the writers' descriptors were written by earlier kernels of the tick and are not written by this
            // one, so they are read through L1 (neighbouring writers share lines)
            const uint16_t* ldn = S.lastDesc + (size_t)F.nxt * npx * C + (size_t)p * C;
            uint64_t d = __ldg(&ldn[0]);
            if (C == 3)
                d |= ((uint64_t)__ldg(&ldn[1]) << 16) | ((uint64_t)__ldg(&ldn[2]) << 32) |
                     ((uint64_t)__ldg(S.frame + (size_t)p * 3) << 48) | ((uint64_t)__ldg(S.frame + (size_t)p * 3 + 1) << 56);
            store_sample<C>(sp, s * S.sStride, d, __ldg(S.frame + (size_t)p * C + C - 1));
        }
        __syncwarp();
    }
    const bool raw = (wq & kInFG) != 0u;
    if (inF) {
        uint16_t kend = 0;
        if (wq & kInValid) {
            if (raw) kend = F.cooldown ? (uint16_t)(1 + ((wq & kInOwn) ? 1 : 0)) : 0;
            else kend = (uint16_t)(1 + ((wq & kInOwn) ? 1 : 0) + 2 + (in_nb_writes(wq) ? 1 : 0));
        }
        S.kctr[q] = kend;
        // blinks (:536-539)
        const uint8_t rawB = raw ? 255 : 0, cb = rawB ^ lastRaw;
        S.blinks[q] = cb | lastRawBlink;
        S.lastRawBlink[q] = cb;
        S.lastRawFG[q] = rawB;
    }
    // each warp is one 32-pixel tile row: the row's words of the raw and closed masks
    const uint32_t valid = x0 + kTileW <= W ? 0xffffffffu : (1u << (W - x0)) - 1u;
    const uint32_t rawW = __ballot_sync(0xffffffffu, inF && raw), closedV = y < H ? closedW & valid : 0u;
    if (lx == 0 && y < H) {
        const size_t o = (size_t)y * S.rowWords + tx;
        bit_plane(S, BP_RAW)[o] = rawW;
        bit_plane(S, BP_CLOSED)[o] = closedV;
    }
    // hole filling: every run start of the row's 0-pixels is its own node. A word's first pixel counts as
    // a start here (the word to its left belongs to another block); nodes that no run uses are not read.
    if (inF && ((~closedV & ~(~closedV << 1)) >> lx) & 1u) S.label[q] = q;
    block_add_stats(&S.ctl->st_writes, (unsigned int)__popc(sm.wr[threadIdx.x]), &S.ctl->st_samples, inF ? in_e(wq) : 0u);
}

// ------------------------------------------------------------------------------------------
// hole filling: cv::floodFill(closed, (0,0), 255) + bitwise_not (:541-543), rebuilt as union-find
// over the runs of 0-pixels of each row. The closed mask is 0 on the 2-pixel frame border (no ROI
// pixel lies there, and a 3x3 closing cannot reach it), so the flood-filled region is the
// 4-connected component of 0-pixels that contains that border ring. Every row's first and last
// run touch the ring and are root 0 itself; interior runs are united with the runs they
// overlap in the row above. Holes are the 0-pixels whose run's root is not 0.
// ------------------------------------------------------------------------------------------
__device__ __forceinline__ int uf_find(int* L, int a, TickWork* w) {
    int n, it = 0;
    while ((n = __ldcg(&L[a])) != a) {
        a = n;
        if (++it > kUFLimit) {
            atomicOr(&w->err, ERR_UF_LIMIT);
            break;
        }
    }
    return a;
}
__device__ void uf_union(int* L, int a, int b, TickWork* w) {
    for (int it = 0; it < kUFLimit; ++it) {
        a = uf_find(L, a, w);
        b = uf_find(L, b, w);
        if (a == b) return;
        if (a < b) {
            const int old = atomicMin(&L[b], a);
            if (old == b) return;
            b = old;
        } else {
            const int old = atomicMin(&L[a], b);
            if (old == a) return;
            a = old;
        }
    }
    atomicOr(&w->err, ERR_UF_LIMIT);
}

__device__ __forceinline__ int find_stream_by_row(const TickParams& P, int r) {
    int lo = 0, hi = P.nStreams - 1;
    while (lo < hi) {
        const int mid = (lo + hi + 1) >> 1;
        if (P.streams[mid].rowBase <= r) lo = mid;
        else hi = mid - 1;
    }
    return lo;
}

// bits of word w that lie inside a frame of width W
__device__ __forceinline__ uint32_t valid_bits(int w, int W) {
    const int n = W - 32 * w;
    return n >= 32 ? 0xffffffffu : (n <= 0 ? 0u : (1u << n) - 1u);
}

// The 0-runs of a row, 32 words at a time with one word per lane. A lane holds its word's 0-pixels and
// run starts; the start of a run that enters the word from the left comes from the nearest lower lane
// that has a start (or from the previous chunk), by one ballot and one shuffle. So a 1920-pixel row takes
// two steps of a warp, where a walk with one lane per pixel took sixty.
struct RowRuns {
    const uint32_t* row;
    int RW, W;
    uint32_t z, starts;  // this lane's word: 0-pixels, run starts
    int entry;           // start of the run that continues from the previous word (if bit 0 of z is set and no start)
    uint32_t carryZ;
    int carryStart;
    __device__ __forceinline__ void reset(const uint32_t* r, int rw, int w) {
        row = r;
        RW = rw;
        W = w;
        carryZ = 0u;
        carryStart = -1;
    }
    // loads words c .. c+31 (every lane of the warp calls it)
    __device__ __forceinline__ void load(int c, int lane) {
        const int w = c + lane;
        z = w < RW ? ~__ldcg(&row[w]) & valid_bits(w, W) : 0u;
        uint32_t prev = __shfl_up_sync(0xffffffffu, z >> 31, 1);
        if (lane == 0) prev = carryZ;
        starts = z & ~((z << 1) | prev);
        const unsigned m = __ballot_sync(0xffffffffu, starts != 0u);
        const int v = 32 * w + 31 - __clz(starts);
        const unsigned lower = m & ((1u << lane) - 1u);
        const int fromLane = __shfl_sync(0xffffffffu, v, lower ? 31 - __clz(lower) : 0);
        entry = lower ? fromLane : carryStart;
        const int last = __shfl_sync(0xffffffffu, v, m ? 31 - __clz(m) : 0);
        if (m) carryStart = last;
        carryZ = __shfl_sync(0xffffffffu, z >> 31, 31);
    }
    // start of the run that holds bit b of word w (this lane's word)
    __device__ __forceinline__ int run_start(int w, int b) const {
        const uint32_t upto = starts & (0xffffffffu >> (31 - b));
        return upto ? 32 * w + 31 - __clz(upto) : entry;
    }
    // the last run start of the row: the run that reaches x = W-1 (every lane calls it)
    __device__ __forceinline__ int last_start(int lane) const {
        for (int c = (RW - 1) & ~31; c >= 0; c -= 32) {
            const int w = c + lane;
            int v = -1;
            if (w < RW) {
                const uint32_t zz = ~__ldcg(&row[w]) & valid_bits(w, W);
                const uint32_t prev = w > 0 ? ~__ldcg(&row[w - 1]) >> 31 : 0u;
                const uint32_t st = zz & ~((zz << 1) | prev);
                if (st) v = 32 * w + 31 - __clz(st);
            }
            v = __reduce_max_sync(0xffffffffu, v);
            if (v >= 0) return v;
        }
        return -1;
    }
};

__device__ void stream_epilogue(const TickParams& P, const StreamDev& S);

// Unites each run with the runs it overlaps in the row above: a warp per row, a word per lane. A run's
// node is the index of its first pixel, labelled with itself by the kernel that wrote the closed mask;
// a run that touches the ring (it holds x = 0 or x = W-1, or lies in the first or last row) stands for
// node 0 without any memory access, so on a mostly empty mask few unions remain. The blocks past the rows
// run the frame-level epilogue of one stream each (it touches nothing that these rows read).
// Latency-bound: 1920x1080 BGR frame, 46 us (one lane per pixel, after an 18 us label pass) before, 7 to 11 us now;
// 320x240 4.7 us; a 640x480 BGR PAWCS frame 40 us.
extern "C" __global__ void __launch_bounds__(256) lvbgs_k_unite(TickParams P) {
    pdl_entry();
    if (P.gate && ld_volatile(P.gate) == 0u) return;
    const int rowBlocks = (P.totalRows + 7) / 8;
    if ((int)blockIdx.x >= rowBlocks) {
        stream_epilogue(P, P.streams[blockIdx.x - rowBlocks]);
        return;
    }
    const int gr = blockIdx.x * 8 + threadIdx.x / 32, lane = threadIdx.x & 31;
    if (gr >= P.totalRows) return;
    const StreamDev& S = P.streams[find_stream_by_row(P, gr)];
    const int y = gr - S.rowBase, W = S.W, H = S.H, RW = S.rowWords;
    const uint32_t* row = bit_plane(S, BP_CLOSED) + (size_t)y * RW;
    const bool edgeRow = y < 2 || y >= H - 2;
    RowRuns rc, ru;
    rc.reset(row, RW, W);
    ru.reset(row - (y > 0 ? RW : 0), RW, W);
    const int lastC = y > 0 ? rc.last_start(lane) : -1, lastU = y > 0 ? ru.last_start(lane) : -1;
    uint32_t carryOv = 0u;
    bool ringOk = true;
    for (int c = 0; c < RW; c += 32) {
        const int w = c + lane;
        rc.load(c, lane);
        ru.load(c, lane);
        const uint32_t vb = valid_bits(w, W);
        uint32_t ring = edgeRow ? vb : 0u;  // pixels of the 2-pixel border ring in this word
        if (w == 0) ring |= 3u & vb;
        if (w == (W - 1) >> 5) ring |= 1u << ((W - 1) & 31);
        if (W > 1 && w == (W - 2) >> 5) ring |= 1u << ((W - 2) & 31);
        if (ring & ~rc.z) ringOk = false;
        const uint32_t ov = rc.z & ru.z;
        uint32_t prev = __shfl_up_sync(0xffffffffu, ov >> 31, 1);
        if (lane == 0) prev = carryOv;
        carryOv = __shfl_sync(0xffffffffu, ov >> 31, 31);
        uint32_t seg = y > 0 ? ov & ~((ov << 1) | prev) : 0u;
        while (seg) {
            const int b = __ffs(seg) - 1;
            seg &= seg - 1u;
            const int sc = rc.run_start(w, b), su = ru.run_start(w, b);
            const int ic = (sc == 0 || sc == lastC || y == H - 1) ? 0 : y * W + sc;
            const int iu = (su == 0 || su == lastU || y == 1) ? 0 : (y - 1) * W + su;
            if (ic != iu) uf_union(S.label, ic, iu, P.work);
        }
    }
    if (__any_sync(0xffffffffu, !ringOk) && lane == 0) atomicOr(&P.work->err, ERR_RING);
}

// Combined mask |= holes | 3-fold 3x3 erosion of the closed mask (a clipped 7x7 minimum) (:541-546): a
// warp per row, a word per lane. Holes are the 0-runs whose root is not 0 (one lookup per run and word;
// runs on the ring need none). The erosion is separable: seven row words are ANDed, then the neighbour
// words come from the neighbour lanes (the two edge lanes of a chunk load theirs). One kernel where the
// hole words took a pass of their own through memory: 20 + 6 us on a 1920x1080 frame before, 13.5 us now.
extern "C" __global__ void __launch_bounds__(256) lvbgs_k_fill(TickParams P) {
    pdl_entry();
    if (P.gate && ld_volatile(P.gate) == 0u) return;
    const int gr = blockIdx.x * 8 + threadIdx.x / 32, lane = threadIdx.x & 31;
    if (gr >= P.totalRows) return;
    const StreamDev& S = P.streams[find_stream_by_row(P, gr)];
    const int y = gr - S.rowBase, W = S.W, H = S.H, RW = S.rowWords;
    const uint32_t* closed = bit_plane(S, BP_CLOSED);
    RowRuns rr;
    rr.reset(closed + (size_t)y * RW, RW, W);
    const int last = rr.last_start(lane);
    const int ya = max(0, y - 3), yb = min(H - 1, y + 3);
    // word w of the rows' minimum; pixels outside the frame never win
    auto column_and = [&](int w) {
        uint32_t v = 0xffffffffu;
        if (w < 0 || w >= RW) return v;
        for (int yy = ya; yy <= yb; ++yy) v &= __ldcg(&closed[(size_t)yy * RW + w]);
        return v | ~valid_bits(w, W);
    };
    for (int c = 0; c < RW; c += 32) {
        const int w = c + lane;
        const uint32_t er0 = column_and(w);
        uint32_t erL = __shfl_up_sync(0xffffffffu, er0, 1), erR = __shfl_down_sync(0xffffffffu, er0, 1);
        if (lane == 0) erL = column_and(w - 1);
        if (lane == 31) erR = column_and(w + 1);
        uint32_t er = er0;
#pragma unroll
        for (int d = 1; d <= 3; ++d) er &= __funnelshift_r(er0, erR, d) & __funnelshift_l(erL, er0, d);
        rr.load(c, lane);
        uint32_t holes = 0u, rem = rr.z;
        while (rem) {
            const int b = __ffs(rem) - 1;
            const uint32_t inv = ~(rem >> b);
            const int len = inv ? __ffs(inv) - 1 : 32;  // pixels of the run in this word
            const uint32_t m = (len >= 32 ? 0xffffffffu : (1u << len) - 1u) << b;
            rem &= ~m;
            const int s = rr.run_start(w, b);
            if (s != 0 && s != last && y > 0 && y < H - 1 && uf_find(S.label, y * W + s, P.work) != 0) holes |= m;
        }
        if (w < RW) {
            const size_t o = (size_t)y * RW + w;
            bit_plane(S, BP_COMB)[o] = (__ldcg(&bit_plane(S, BP_RAW)[o]) | holes | er) & valid_bits(w, W);
        }
    }
}

// shared memory of one tile of the final-mask kernel: the combined mask's words with their halo, the row
// window counts as bit planes, the final mask with the dilation's halo, the dilated words
constexpr int kFinMaxR = 15;                            // median radius (kernel size at most 31)
constexpr int kFinRows = kFinH + 6 + 2 * kFinMaxR;      // combined-mask rows
constexpr int kFinFG = kFinH + 6;                       // final-mask rows
struct FinSmem {
    uint32_t comb[kFinRows][kFinWords + 4];
    uint32_t h[5][kFinRows][kFinWords + 2];
    uint32_t fg[kFinFG][kFinWords + 2];
    uint32_t dil[kFinH][kFinWords];
};

// row window counts, then the window sums of the final mask's words and their comparison with half the
// window (threads take one word each)
template <int HB>
__device__ __forceinline__ void median_words(FinSmem& sm, int r, int half, int y0, int w0, int W, int H, int RW) {
    const int nRows = kFinFG + 2 * r;
    for (int i = threadIdx.x; i < nRows * (kFinWords + 2); i += blockDim.x) {
        const int rr = i / (kFinWords + 2), ww = i % (kFinWords + 2);
        uint32_t h[HB];
        row_window_planes<HB>(sm.comb[rr][ww], sm.comb[rr][ww + 1], sm.comb[rr][ww + 2], r, h);
#pragma unroll
        for (int b = 0; b < HB; ++b) sm.h[b][rr][ww] = h[b];
    }
    __syncthreads();
    for (int i = threadIdx.x; i < kFinFG * (kFinWords + 2); i += blockDim.x) {
        const int fr = i / (kFinWords + 2), fw = i % (kFinWords + 2);
        const int y = y0 - 3 + fr, w = w0 - 1 + fw;
        uint32_t fg = 0u;
        if (y >= 0 && y < H && w >= 0 && w < RW) {
            uint32_t a[2 * HB];
#pragma unroll
            for (int b = 0; b < 2 * HB; ++b) a[b] = b < HB ? sm.h[b < HB ? b : 0][fr][fw] : 0u;
            for (int j = 1; j <= 2 * r; ++j) {
                uint32_t v[HB];
#pragma unroll
                for (int b = 0; b < HB; ++b) v[b] = sm.h[b][fr + j][fw];
                add_planes<HB>(a, v);
            }
            fg = planes_above<2 * HB>(a, half);
            fg &= valid_bits(w, W);
        }
        sm.fg[fr][fw] = fg;
    }
}

// The final mask and everything that follows from it (:547-554): binary median blur of the combined mask
// (majority of the k x k window, replicated border), the final-segmentation averages (addWeighted), the
// mask bytes, its 3-fold 3x3 dilation (a clipped 7x7 maximum) and the blink masking with the previous and
// the new inverted dilated masks. A block takes 8 rows of 4 words (128 pixels) and counts on bit planes:
// 32 pixels per word operation, full adders over the row window, then over the rows, with the halo of the
// dilation recomputed (84 words for 32), so that no per-pixel count goes through memory and the three
// passes of before (7.8 + 15.9 + 10.2 us on a 1920x1080 frame) are one of 15.6 us. The pixels' maps are requested
// first and used last; a thread holds four neighbouring pixels, so the mask leaves in 128-byte rows also
// when it is in host memory. Bound by the 22 B/px of maps and by the latency of the short word phases.
extern "C" __global__ void __launch_bounds__(kThreads) lvbgs_k_final(TickParams P) {
    pdl_entry();
    if (P.gate && ld_volatile(P.gate) == 0u) return;
    __shared__ FinSmem sm;
    const int gt = blockIdx.x;
    if (gt >= P.totalSegs) return;
    int lo = 0, hi = P.nStreams - 1;
    while (lo < hi) {
        const int mid = (lo + hi + 1) >> 1;
        if (P.streams[mid].segBase <= gt) lo = mid;
        else hi = mid - 1;
    }
    const StreamDev& S = P.streams[lo];
    const int W = S.W, H = S.H, npx = S.npx, RW = S.rowWords;
    const int tilesX = (RW + kFinWords - 1) / kFinWords;
    const int lt = gt - S.segBase, y0 = (lt / tilesX) * kFinH, w0 = (lt % tilesX) * kFinWords;
    const int k = S.ctl->median_k, r = k / 2;
    const FrameK F = frame_consts(S);
    // the four pixels of this thread
    const int row = threadIdx.x >> 5, quad = threadIdx.x & 31;
    const int y = y0 + row, x = w0 * 32 + quad * 4, q = y * W + x;
    const int n = y < H ? min(4, W - x) : 0;  // pixels of the quad inside the frame
    const float* cLT = S.fm + ((size_t)F.cur * kNumFloatMaps + FM_FIN_LT) * npx;
    const float* cST = S.fm + ((size_t)F.cur * kNumFloatMaps + FM_FIN_ST) * npx;
    float* nLT = S.fm + ((size_t)F.nxt * kNumFloatMaps + FM_FIN_LT) * npx;
    float* nST = S.fm + ((size_t)F.nxt * kNumFloatMaps + FM_FIN_ST) * npx;
    const bool vec = (W & 3) == 0;  // then a quad is whole, and aligned in every plane
    float fl[4] = {0, 0, 0, 0}, fs[4] = {0, 0, 0, 0};
    uint32_t bl = 0u, di = 0u;
    if (vec && n > 0) {
        const float4 a = *(const float4*)(cLT + q), b = *(const float4*)(cST + q);
        fl[0] = a.x, fl[1] = a.y, fl[2] = a.z, fl[3] = a.w;
        fs[0] = b.x, fs[1] = b.y, fs[2] = b.z, fs[3] = b.w;
        bl = *(const uint32_t*)(S.blinks + q);
        di = *(const uint32_t*)(S.dilInv + q);
    } else {
#pragma unroll
        for (int i = 0; i < 4; ++i)
            if (i < n) {
                fl[i] = cLT[q + i];
                fs[i] = cST[q + i];
                bl |= (uint32_t)S.blinks[q + i] << (8 * i);
                di |= (uint32_t)S.dilInv[q + i] << (8 * i);
            }
    }
    const uint32_t* comb = bit_plane(S, BP_COMB);
    const int nRows = kFinFG + 2 * r;
    for (int i = threadIdx.x; i < nRows * (kFinWords + 4); i += blockDim.x) {
        const int rr = i / (kFinWords + 4), ww = i % (kFinWords + 4);
        const uint32_t* src = comb + (size_t)min(max(y0 - 3 - r + rr, 0), H - 1) * RW;
        const int w = w0 - 2 + ww;
        uint32_t v;
        if (w < 0) {
            v = (__ldcg(&src[0]) & 1u) ? 0xffffffffu : 0u;
        } else if (w < RW - 1) {
            v = __ldcg(&src[w]);
        } else {
            const uint32_t lw = __ldcg(&src[RW - 1]);
            const uint32_t fill = ((lw >> ((W - 1) & 31)) & 1u) ? 0xffffffffu : 0u;
            const uint32_t vb = valid_bits(w, W);
            v = (lw & vb) | (fill & ~vb);
        }
        sm.comb[rr][ww] = v;
    }
    __syncthreads();
    // 2 * sum > k * k
    if (r < 8) median_words<4>(sm, r, k * k / 2, y0, w0, W, H, RW);
    else median_words<5>(sm, r, k * k / 2, y0, w0, W, H, RW);
    __syncthreads();
    if (threadIdx.x < kFinH * kFinWords) {
        const int dr = threadIdx.x / kFinWords, dw = threadIdx.x % kFinWords;
        uint32_t a = 0u, b = 0u, c = 0u;
#pragma unroll
        for (int j = 0; j < 7; ++j) {
            a |= sm.fg[dr + j][dw];
            b |= sm.fg[dr + j][dw + 1];
            c |= sm.fg[dr + j][dw + 2];
        }
        uint32_t v = b;
#pragma unroll
        for (int d = 1; d <= 3; ++d) v |= __funnelshift_r(b, c, d) | __funnelshift_l(a, b, d);
        sm.dil[dr][dw] = v;
    }
    __syncthreads();
    if (S.maskOut && y < H) {
        // The mask bytes of the tile row as aligned words, whatever the frame's width and the buffer's address (32 or
        // 33 of them, the row's first and last in bytes): single bytes cost a transaction each when the mask
        // is in host memory, 12 mixed streams with two frames of 1279x719 82 to 157 us.
        uint8_t* out = S.maskOut + (size_t)y * W + w0 * 32;
        const int len = min(32 * kFinWords, W - w0 * 32), off = (int)((uintptr_t)out & 3);
        for (int i = quad; 4 * i - off < len; i += 32) {
            const int b = 4 * i - off;  // the word's first byte, from -3 on
            const uint32_t* f = &sm.fg[row + 3][1 + (b >> 5)];
            const uint32_t bits = __funnelshift_r(f[0], f[1], b & 31) & 15u;
            const uint32_t v = ((bits * 0x00204081u) & 0x01010101u) * 255u;
            if (b >= 0 && b + 4 <= len) {
                *(uint32_t*)(out + b) = v;
            } else {
                for (int j = max(0, -b); j < 4 && b + j < len; ++j) out[b + j] = (uint8_t)(v >> (8 * j));
            }
        }
    }
    if (n <= 0) return;
    const uint32_t fg4 = (sm.fg[row + 3][1 + (quad >> 3)] >> ((quad & 7) * 4)) & 15u;
    const uint32_t dl4 = (sm.dil[row][quad >> 3] >> ((quad & 7) * 4)) & 15u;
    // bit i -> byte i, as 0 or 255
    const uint32_t fgb = ((fg4 * 0x00204081u) & 0x01010101u) * 255u;
    const uint32_t inv = ~(((dl4 * 0x00204081u) & 0x01010101u) * 255u);
    const float aL = 1.0f - F.fLT, bL = S.ctl->bLT;
    const float aS = 1.0f - F.fST, bS = S.ctl->bST;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const float m = (float)((fgb >> (8 * i)) & 255u);
        fl[i] = (fl[i] * aL + m * bL) + 0.0f;
        fs[i] = (fs[i] * aS + m * bS) + 0.0f;
    }
    const uint32_t nb = bl & di & inv;
    if (vec) {
        *(float4*)(nLT + q) = make_float4(fl[0], fl[1], fl[2], fl[3]);
        *(float4*)(nST + q) = make_float4(fs[0], fs[1], fs[2], fs[3]);
        *(uint32_t*)(S.lastFG + q) = fgb;
        *(uint32_t*)(S.blinks + q) = nb;
        *(uint32_t*)(S.dilInv + q) = inv;
    } else {
#pragma unroll
        for (int i = 0; i < 4; ++i)
            if (i < n) {
                nLT[q + i] = fl[i];
                nST[q + i] = fs[i];
                S.lastFG[q + i] = (uint8_t)(fgb >> (8 * i));
                S.blinks[q + i] = (uint8_t)(nb >> (8 * i));
                S.dilInv[q + i] = (uint8_t)(inv >> (8 * i));
            }
    }
}

// frame-level epilogue of one stream (:555-611), one block of 256 threads: LBSP threshold LUT adaptation
// (one entry per thread), then, on thread 0, camera-motion analysis, automatic model reset decision and
// learning-rate caps
__device__ void stream_epilogue(const TickParams& P, const StreamDev& S) {
    StreamCtl* ctl = S.ctl;
    const float relThr = S.relThr;
    const unsigned int lbspOff = S.lbspOff;
    const unsigned long long nz = ctl->nz_acc;
    const float ratio = __ull2float_rn(nz) / __ull2float_rn(ctl->n_rel);
    const float last = ctl->last_nz_ratio;
    const int t = threadIdx.x;
    if (ratio < 0.100f && last < 0.100f) {
        const float v = ceilf((float)t * relThr / 4) + (float)lbspOff;
        const int lim = v > 255.0f ? 255 : (int)v;
        if ((int)ctl->lut[t] > lim) --ctl->lut[t];
    } else if (ratio > 0.500f && last > 0.500f) {
        int lim = __float2int_rn((float)lbspOff + 255 * relThr);
        lim = lim < 0 ? 0 : lim > 255 ? 255 : lim;
        if ((int)ctl->lut[t] < lim) ++ctl->lut[t];
    }
    __syncthreads();  // every thread has read the ratios
    if (t != 0) return;
    ctl->last_nz = nz;
    ctl->nz_acc = 0;
    ctl->last_nz_ratio = ratio;
    ctl->refresh_pending = 0;
    ctl->ksent = 0;
    ctl->last_colordiff = 0;
    if (ctl->lr_scaling) {
        const unsigned long long tot = ctl->colordiff_acc;
        ctl->last_colordiff = tot;
        ctl->colordiff_acc = 0;
        const float cr = __ull2float_rn(tot) / (float)(S.dsW * S.dsH);
        const unsigned long long thr = (unsigned long long)(S.minColor / 2);
        if (ctl->auto_reset) {
            if (ctl->frames_since_reset > 1000ull) {
                ctl->auto_reset = 0;
            } else if (cr >= (float)thr && ctl->cooldown == 0ull) {
                ctl->frames_since_reset = 0;
                ctl->refresh_pending = 1;
                ctl->cooldown = (unsigned long long)(S.nmv / 4);
            } else {
                ++ctl->frames_since_reset;
            }
        } else if (cr >= (float)(thr * 2ull)) {
            ctl->frames_since_reset = 0;
            ctl->auto_reset = 1;
        }
        if (cr >= (float)(thr / 2ull)) {
            const int sh = ((int)(cr / 2)) & 31;
            const int lo = 2 >> sh, hi = 256 >> sh;
            ctl->t_lo = (float)(lo > 1 ? lo : 1);
            ctl->t_hi = (float)(hi > 1 ? hi : 1);
        } else {
            ctl->t_lo = 2.0f;
            ctl->t_hi = 256.0f;
        }
        if (ctl->cooldown > 0ull) --ctl->cooldown;
    }
    if (ctl->refresh_pending) {
        // nRefreshSampleStartPos = rand() % N, drawn with the frame-level (sentinel) counter (:86)
        DrawState ds;
        ds.blk = 0xffffffffu;
        const uint32_t f = (uint32_t)(ctl->frame_idx + 1ull);
        ctl->refresh_start = draw_k(S.seed, f, kSentinelPx, 0u, ds) % (uint32_t)S.N;
        ctl->ksent = 1;
        atomicExch(&P.work->anyReset, 1u);
    }
}

// refreshModel (:80-105) of one pixel; lastBuf holds the latest colour/descriptor frame
template <int C>
__device__ void refresh_pixel(const StreamDev& S, int p, uint32_t frame, int start, int nref, int force, int lastBuf) {
    if (!S.roi[p]) return;
    if (!force && S.lastFG[p]) return;
    const int W = S.W, H = S.H, npx = S.npx, N = S.N;
    const int x0 = p % W, y0 = p / W;
    uint32_t k = S.kctr[p];
    DrawState ds;
    ds.blk = 0xffffffffu;
    const uint8_t* lc = S.lastCol + (size_t)lastBuf * npx * C;
    const uint16_t* ldd = S.lastDesc + (size_t)lastBuf * npx * C;
    for (int s = start; s < start + nref; ++s) {
        int r = 1 + (int)(draw_k(S.seed, frame, (uint32_t)p, k++, ds) % 512u);
        int sx = 0, sy = 0;
        for (int i = 0; i < 49; ++i) {
            r -= c_pat7[i];
            if (r <= 0) {
                sy = i / 7;
                sx = i % 7;
                break;
            }
        }
        sx += x0 - 3;
        sy += y0 - 3;
        clamp_xy(sx, sy, W, H);
        const int sp = sy * W + sx;
        if (!force && S.lastFG[sp]) continue;
        const int rs = s % N;
        uint64_t d = ldd[(size_t)sp * C];
        if (C == 3)
            d |= ((uint64_t)ldd[(size_t)sp * 3 + 1] << 16) | ((uint64_t)ldd[(size_t)sp * 3 + 2] << 32) |
                 ((uint64_t)lc[(size_t)sp * 3] << 48) | ((uint64_t)lc[(size_t)sp * 3 + 1] << 56);
        store_sample<C>(samples_of<C>(S, p), rs * S.sStride, d, lc[(size_t)sp * C + C - 1]);
    }
    S.kctr[p] = (uint16_t)k;
}

// ------------------------------------------------------------------------------------------
// the frame step: one kernel per phase, launched back to back over all streams of the batch (each
// kernel indexes the per-stream descriptor table); the repair loop is a cooperative kernel with
// grid barriers
// ------------------------------------------------------------------------------------------
#define LV_TILE_KERNEL_PROLOGUE                                              \
    const int t = blockIdx.x;                                               \
    if (t >= P.totalTiles) return;                                          \
    const int si = find_stream_by_tile(P, t);                               \
    const StreamDev& S = P.streams[si];                                     \
    const int lt = t - S.tileBase;

extern "C" __global__ void __launch_bounds__(kThreads, 5) lvbgs_k_eval(TickParams P) {
    pdl_entry();
    __shared__ __align__(16) uint8_t smem[kTileRW<3> * (kTileH + 2 * kBorder) + 256];
    LV_TILE_KERNEL_PROLOGUE
    if (S.C == 3) phaseA_tile<3>(P, si, S, lt, smem);
    else phaseA_tile<1>(P, si, S, lt, smem);
}

// ------------------------------------------------------------------------------------------
// long sample scans: the pixels whose ordered scan did not settle within the first kScanCap samples
// (foreground pixels scan all N) continue here from the saved scan state, over the compacted list: by
// groups of eight lanes while the list is short, else a pixel a lane (coop_share); then the rest of their
// evaluation. Spatially sparse long scans would otherwise keep whole warps of the evaluation waiting on a few lanes.
// ------------------------------------------------------------------------------------------
template <int C>
__device__ void longscan_items(const TickParams& P, bool own, int m, unsigned long long key, unsigned long long sw) {
    const int si = own ? (int)(key >> 40) : 0, p = own ? (int)(key & 0xffffffffffull) : 0;
    const StreamDev& S = P.streams[si];
    const FrameK F = frame_consts(S);
    const int W = S.W, x = p % W, y = p / W, npx = S.npx;
    ScanSt st;
    st.s = (int)(sw & 0xffu);
    st.nGood = (int)((sw >> 8) & 0xffu);
    const int g0 = (int)((sw >> 16) & 0xffu);
    st.g0 = g0 == 255 ? -1 : g0;
    st.minDesc = (uint32_t)((sw >> 32) & 0xffffu);
    st.minSum = (uint32_t)(sw >> 48);
    // a deferred scan has fewer than nreq good samples; with one, the minima are its distances
    st.g0d = st.minDesc;
    st.g0s = st.minSum;
    st.g1 = -1;
    st.g1d = st.g1s = 0;
    EvalThr th;
    th.colThr = th.descThr = th.uNew = 0u;
    uint32_t curr[C], intra[C];
    {
        uint32_t vals[C][4];
#pragma unroll
        for (int c = 0; c < C; ++c) {
            curr[c] = intra[c] = 0u;
#pragma unroll
            for (int j = 0; j < 4; ++j) vals[c][j] = 0u;
        }
        if (own) {
            // the scan needs the thresholds only; the feedback maps of the tail are loaded after it
            const float* fc = S.fm + (size_t)F.cur * kNumFloatMaps * npx;
            th = eval_thresholds(S, fc[FM_R * npx + p], fc[FM_RAW_LT * npx + p], fc[FM_RAW_ST * npx + p],
                                 fc[FM_FIN_LT * npx + p], fc[FM_FIN_ST * npx + p], S.unst[(size_t)F.cur * npx + p]);
            const uint8_t* base = S.frame + (size_t)p * C;
            const uint8_t* lut = S.ctl->lut;
#pragma unroll
            for (int c = 0; c < C; ++c) {
                gather_taps<C>(base, W * C, c, vals[c]);
                curr[c] = __ldg(base + c);
                intra[c] = lbsp_thr(vals[c], curr[c], lut[curr[c]]);
            }
        }
        coop_scan<C, true>(P, own, m, si, p, vals, curr, intra, th, 0ull, 0ull, st);
    }
    if (!own) return;
    record_scan(S, F, p, st);
    PixIn<C> in;
    load_pix<C>(S, F, p, in);
    __stcg(&S.intent[p], eval_tail<C>(S, F, x, y, p, in, curr, intra, th.uNew, st));
}

extern "C" __global__ void __launch_bounds__(256, 3) lvbgs_k_longscan(TickParams P) {
    pdl_entry();
    const unsigned int n = min(ld_volatile(&P.work->lcount), P.listCap);
    const int m = coop_share(n, gridDim.x), lane = threadIdx.x & 31, sub = lane & 7;
    const unsigned int warp = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
    const unsigned int step = gridDim.x * (blockDim.x >> 5) * 4u * m;
    for (unsigned int base = warp * 4u * m; base < n; base += step) {
        const unsigned int i = base + (unsigned)(lane >> 3) * m + sub;
        const bool own = sub < m && i < n;
        const unsigned long long key = own ? __ldcg(&P.rlist[0][i]) : 0ull, sw = own ? __ldcg(&P.rlist[1][i]) : 0ull;
        const bool c3 = own && P.streams[(int)(key >> 40)].C == 3;
        if (__any_sync(0xffffffffu, c3)) longscan_items<3>(P, c3, m, key, sw);
        if (__any_sync(0xffffffffu, own && !c3)) longscan_items<1>(P, own && !c3, m, key, sw);
    }
}

extern "C" __global__ void __launch_bounds__(kThreads) lvbgs_k_resolve(TickParams P, unsigned long long dsTotal) {
    pdl_entry();
    const int tileBlocks = (P.totalTiles + kResolveTiles - 1) / kResolveTiles;
    if ((int)blockIdx.x < tileBlocks) {
        phaseB_tiles(P, blockIdx.x * kResolveTiles);
        return;
    }
    const unsigned long long i = ((unsigned long long)(blockIdx.x - tileBlocks) * blockDim.x + threadIdx.x) >> 3;
    if (i >= dsTotal) return;
    int lo = 0, hi = P.nStreams - 1;
    while (lo < hi) {
        const int mid = (lo + hi + 1) >> 1;
        if (P.streams[mid].dsBase <= i) lo = mid;
        else hi = mid - 1;
    }
    const StreamDev& S = P.streams[lo];
    if (S.C == 3) ds_item<3>(S, (int)(i - S.dsBase));
    else ds_item<1>(S, (int)(i - S.dsBase));
}

// Repair to the raster-order fixed point (cooperative launch: all CTAs resident). Every round re-matches
// the listed pixels (M), then re-resolves the ghost tests that read a changed one (R). Most rounds change
// no decision, so R has nothing to do and its barrier is left out. Only as many CTAs take part as the first
// list has work for (later lists are shorter): a barrier over 28 CTAs costs a third of one over 304.
extern "C" __global__ void __launch_bounds__(kThreads, 2) lvbgs_k_repair(TickParams P) {
    TickWork* w = P.work;
    unsigned int due = 0u;  // barrier arrivals
    if (blockIdx.x == 0 && threadIdx.x == 0 && w->nts < 40u) w->ts[w->nts++] = gtimer();  // phase profile
    if (P.dbgFault == LVBGS_FAULT_BARRIER_TIMEOUT) {
        // injected fault: every CTA but CTA 0 waits at a barrier CTA 0 never reaches; each wait gives
        // up after P.barrierNs and records ERR_BARRIER_TIMEOUT, and every CTA returns
        if (blockIdx.x != 0) grid_sync(w, gridDim.x, P.barrierNs, due);
        return;
    }
    const int lane = threadIdx.x & 31;
    // the CTAs of this repair: a group of eight lanes for every item of the first list (whose length stays
    // as it is while the kernel runs, so that a CTA that starts late decides alike)
    const unsigned int n0 = ld_volatile(&w->dcount[0]);
    const unsigned int ctas = min(gridDim.x, max(1u, (n0 + 31u) / 32u));
    if (blockIdx.x >= ctas) return;
    int iter = 0;
    for (;;) {
        const int par = iter & 1;
        const unsigned int n = ld_volatile(&w->dcount[dcount_slot(iter)]);
        if (n == 0u) break;
        if (iter >= P.maxRepairIters) {
            if (blockIdx.x == 0 && threadIdx.x == 0) atomicOr(&w->err, ERR_REPAIR_LIMIT);
            return;
        }
        const unsigned int nItems = n < P.listCap ? n : P.listCap;
        if (blockIdx.x == 0 && threadIdx.x == 0) {
            w->rcount[par ^ 1] = 0u;
            w->dcount[dcount_slot(iter + 2)] = 0u;
            w->fetchD[par ^ 1] = 0u;
            w->fetchR[par ^ 1] = 0u;
            w->rematched += nItems;
            if (iter < 16) w->phase_ctr[iter] = nItems;
        }
        // items are fetched by each warp from a counter (not strided): per-item costs vary widely, and
        // every round waits for its slowest warp at the barrier. A fetch is 4 items (one for each
        // group of eight lanes) while there is a group for every item, up to 32.
        const int m = coop_share(nItems, ctas);
        for (;;) {
            unsigned int base = 0;
            if (lane == 0) base = atomicAdd(&w->fetchD[par], 4u * m);
            base = __shfl_sync(0xffffffffu, base, 0);
            if (base >= nItems) break;
            const unsigned int i = base + (unsigned)(lane >> 3) * m + (lane & 7);
            const bool own = (lane & 7) < m && i < nItems;
            const unsigned long long item = own ? __ldcg(&P.dlist[par][i]) : 0ull;
            const int si = (int)(item >> 40), q = (int)(item & 0xffffffffffull);
            const StreamDev& S = P.streams[si];
            const bool c3 = own && S.C == 3;
            const uint32_t stampNext = S.ctl->stamp_base + (uint32_t)iter + 2u;
            bool counted = false;
            if (__any_sync(0xffffffffu, c3)) counted = rematch_items<3>(P, c3, m, si, q, stampNext, iter);
            if (__any_sync(0xffffffffu, own && !c3)) counted |= rematch_items<1>(P, own && !c3, m, si, q, stampNext, iter);
            // re-match statistics: one atomic per stream among the lanes here
            const unsigned grp = __match_any_sync(0xffffffffu, counted ? si : -1 - lane);
            if (counted && lane == __ffs(grp) - 1) atomicAdd(&S.ctl->st_rematched, (unsigned long long)__popc(grp));
        }
        if (!grid_sync(w, ctas, P.barrierNs, due)) return;
        const unsigned int nr0 = ld_volatile(&w->rcount[par]);
        const unsigned int nr = nr0 < P.listCap ? nr0 : P.listCap;
        if (nr != 0u) {  // the same value in every CTA: rcount[par] is reset only in the next round, from 0
            for (;;) {
                unsigned int base = 0;
                if (lane == 0) base = atomicAdd(&w->fetchR[par], 32u);
                base = __shfl_sync(0xffffffffu, base, 0);
                if (base >= nr) break;
                const unsigned int i = base + lane;
                if (i < nr) {
                    const unsigned long long item = __ldcg(&P.rlist[par][i]);
                    const int si = (int)(item >> 40), p = (int)(item & 0xffffffffffull);
                    const StreamDev& S = P.streams[si];
                    reresolve_item(P, si, S, p, S.ctl->stamp_base + (uint32_t)iter + 2u, iter);
                }
            }
            if (!grid_sync(w, ctas, P.barrierNs, due)) return;
        } else if (blockIdx.x == 0 && threadIdx.x == 0 && w->nts < 40u) {
            w->ts[w->nts++] = gtimer();  // the phase profile has two entries a round
        }
        ++iter;
    }
    if (blockIdx.x == 0 && threadIdx.x == 0) w->iters = (unsigned)iter;
}

extern "C" __global__ void __launch_bounds__(kThreads) lvbgs_k_commit(TickParams P) {
    pdl_entry();
    __shared__ CommitSmem smem;
    LV_TILE_KERNEL_PROLOGUE
    if (S.C == 3) phaseF_tile<3>(P, S, lt, smem);
    else phaseF_tile<1>(P, S, lt, smem);
}


// closes the frame of every stream: frame index (and so the buffer parity), repair statistics
__device__ __forceinline__ void close_streams(const TickParams& P) {
    const unsigned int its = P.work->iters;
    // the tick's error flags go to the host with the kernel's end: no copy to enqueue and wait for
    if (threadIdx.x == 0 && P.hostErr) *(volatile unsigned int*)P.hostErr = ld_volatile(&P.work->err);
    for (int si = threadIdx.x; si < P.nStreams; si += blockDim.x) {
        StreamCtl* ctl = P.streams[si].ctl;
        ctl->frame_idx += 1ull;
        ctl->st_rounds += its;
        ctl->stamp_base += its + 4u;
        frame_factors(ctl->frame_idx + 1ull, P.streams[si].nmv, &ctl->fLT, &ctl->fST, &ctl->bLT, &ctl->bST);
    }
}

// The end of the frame. Nearly always block 0 closes the streams and the others leave at once. When a
// stream resets its model -- refreshModel(0.1) and T(x) := 1 everywhere (:588-593) -- the grid strides over
// the tiles of those streams, and the block that finishes last closes the streams (the others still read
// the frame index until then).
extern "C" __global__ void __launch_bounds__(kThreads) lvbgs_k_close(TickParams P) {
    pdl_entry();
    if (ld_volatile(&P.work->anyReset) == 0u) {
        if (blockIdx.x == 0) close_streams(P);
        return;
    }
    for (int t = blockIdx.x; t < P.totalTiles; t += gridDim.x) {
        const int si = find_stream_by_tile(P, t);
        const StreamDev& S = P.streams[si];
        if (!S.ctl->refresh_pending) continue;
        const int lt = t - S.tileBase;
        const int x = (lt % S.tilesX) * kTileW + threadIdx.x % kTileW;
        const int y = (lt / S.tilesX) * kTileH + threadIdx.x / kTileW;
        if (x >= S.W || y >= S.H) continue;
        const int p = y * S.W + x;
        const uint32_t f = (uint32_t)(S.ctl->frame_idx + 1ull);
        const int nxt = (int)((S.ctl->frame_idx + 1ull) & 1ull);
        const int nref = (int)(0.1f * (float)S.N);
        if (S.C == 3) refresh_pixel<3>(S, p, f, (int)S.ctl->refresh_start, nref, 0, nxt);
        else refresh_pixel<1>(S, p, f, (int)S.ctl->refresh_start, nref, 0, nxt);
        S.fm[(size_t)0 * kNumFloatMaps * S.npx + FM_T * S.npx + p] = 1.0f;
        S.fm[(size_t)1 * kNumFloatMaps * S.npx + FM_T * S.npx + p] = 1.0f;
    }
    __shared__ int sLast;
    __threadfence();
    __syncthreads();
    if (threadIdx.x == 0) sLast = atomicAdd(&P.work->done_ctas, 1u) == gridDim.x - 1u;
    __syncthreads();
    if (sLast) close_streams(P);
}

// ------------------------------------------------------------------------------------------
// initialization, manual refresh, background images, LBSP extraction
// ------------------------------------------------------------------------------------------
// BackgroundSubtractorLBSP.cpp:21-65 + BackgroundSubtractorSuBSENSE.cpp:129-182 (map initial values)
extern "C" __global__ void lvbgs_init_maps(StreamDev S, const uint8_t* img, float tLo) {
    const int npx = S.npx;
    for (int p = blockIdx.x * blockDim.x + threadIdx.x; p < npx; p += gridDim.x * blockDim.x) {
        const int C = S.C, x = p % S.W, y = p / S.W;
        for (int b = 0; b < 2; ++b) {
            float* f = S.fm + (size_t)b * kNumFloatMaps * npx;
            for (int m = 0; m < kNumFloatMaps; ++m) f[m * npx + p] = 0.0f;
            f[FM_T * npx + p] = tLo;
            f[FM_R * npx + p] = 1.0f;
            f[FM_V * npx + p] = 10.0f;
            S.unst[(size_t)b * npx + p] = 0;
        }
        const bool in = S.roi[p] != 0;
        const bool desc = in && x > kBorder && y > kBorder && x < S.W - kBorder && y < S.H - kBorder;
        for (int c = 0; c < C; ++c) {
            const uint8_t v = in ? img[(size_t)p * C + c] : 0;
            uint16_t d = 0;
            if (desc) {
                uint32_t vals[4];
                const uint8_t* base = img + (size_t)p * C;
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    uint32_t wv = 0;
#pragma unroll
                    for (int i = 0; i < 4; ++i) {
                        const int n = j * 4 + i;
                        wv |= (uint32_t)base[(lbsp_dy(n) * S.W + lbsp_dx(n)) * C + c] << (8 * i);
                    }
                    vals[j] = wv;
                }
                d = (uint16_t)lbsp_thr(vals, v, S.ctl->lut[v]);
            }
            for (int b = 0; b < 2; ++b) {
                S.lastCol[(size_t)b * npx * C + (size_t)p * C + c] = v;
                S.lastDesc[(size_t)b * npx * C + (size_t)p * C + c] = d;
            }
        }
        S.blinks[p] = 0;
        S.lastRawFG[p] = 0;
        S.lastFG[p] = 0;
        S.dilInv[p] = 0;
        S.lastRawBlink[p] = 0;
        S.kctr[p] = 0;
        S.stampD[p] = 0;
        S.stampR[p] = 0;
    }
}

// refreshModel(frac, force) outside a frame step (initialize(), or a user call)
extern "C" __global__ void lvbgs_refresh(StreamDev S, uint32_t frame, int start, int nref, int force, int lastBuf) {
    for (int p = blockIdx.x * blockDim.x + threadIdx.x; p < S.npx; p += gridDim.x * blockDim.x) {
        if (S.C == 3) refresh_pixel<3>(S, p, frame, start, nref, force, lastBuf);
        else refresh_pixel<1>(S, p, frame, start, nref, force, lastBuf);
    }
}

// getBackgroundImage / getBackgroundDescriptorsImage (:614-649): float mean in sample order
// A channel's mean takes the samples in order, eight of them in flight.
template <int C>
__device__ void background_pixel(const StreamDev& S, int p, uint8_t* outCol, uint16_t* outDesc) {
    const int N = S.N;
    const float Nf = (float)N;
    const Samples<C> sp = samples_of<C>(S, p);
    float acc[C], accd[C];
#pragma unroll
    for (int c = 0; c < C; ++c) acc[c] = accd[c] = 0.0f;
    for (int s0 = 0; s0 < N; s0 += 8) {
        uint64_t d[8];
        uint32_t col[8];
#pragma unroll
        for (int j = 0; j < 8; ++j) {
            d[j] = 0;
            col[j] = 0;
            if (s0 + j < N) load_sample<C>(sp, (s0 + j) * S.sStride, d[j], col[j]);
        }
#pragma unroll
        for (int j = 0; j < 8; ++j) {
            if (s0 + j >= N) break;
#pragma unroll
            for (int c = 0; c < C; ++c) {
                const uint32_t v = c == C - 1 ? col[j] : (uint32_t)(d[j] >> (48 + 8 * c)) & 0xffu;
                if (outCol) acc[c] += ((float)v) / Nf;
                if (outDesc) accd[c] += ((float)((uint32_t)(d[j] >> (16 * c)) & 0xffffu)) / Nf;
            }
        }
    }
#pragma unroll
    for (int c = 0; c < C; ++c) {
        if (outCol) {
            const int r = __float2int_rn(acc[c]);
            outCol[(size_t)p * C + c] = (uint8_t)(r < 0 ? 0 : r > 255 ? 255 : r);
        }
        if (outDesc) {
            const int r = __float2int_rn(accd[c]);
            outDesc[(size_t)p * C + c] = (uint16_t)(r < 0 ? 0 : r > 65535 ? 65535 : r);
        }
    }
}
extern "C" __global__ void lvbgs_background(StreamDev S, uint8_t* outCol, uint16_t* outDesc) {
    for (int p = blockIdx.x * blockDim.x + threadIdx.x; p < S.npx; p += gridDim.x * blockDim.x) {
        if (S.C == 3) background_pixel<3>(S, p, outCol, outDesc);
        else background_pixel<1>(S, p, outCol, outDesc);
    }
}

// sample s of pixel p for either channel count
__device__ __forceinline__ void sample_at(const StreamDev& S, int s, int p, uint64_t& d, uint32_t& c) {
    if (S.C == 3) load_sample<3>(samples_of<3>(S, p), s * S.sStride, d, c);
    else load_sample<1>(samples_of<1>(S, p), s * S.sStride, d, c);
}

// samples -> the reference's N sample images (inspection)
extern "C" __global__ void lvbgs_unpack_samples(StreamDev S, uint8_t* col, uint16_t* desc) {
    const size_t total = (size_t)S.N * S.npx;
    const int C = S.C;
    for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < total; i += (size_t)gridDim.x * blockDim.x) {
        const int k = (int)(i / S.npx), p = (int)(i - (size_t)k * S.npx);
        uint64_t v;
        uint32_t last;
        sample_at(S, k, p, v, last);
        for (int c = 0; c < C; ++c) {
            col[i * C + c] = c == C - 1 ? (uint8_t)last : (uint8_t)(v >> (48 + 8 * c));
            desc[i * C + c] = (uint16_t)(v >> (16 * c));
        }
    }
}

// the reference's N sample images -> samples (state restore)
extern "C" __global__ void lvbgs_pack_samples(StreamDev S, const uint8_t* col, const uint16_t* desc) {
    const size_t total = (size_t)S.N * S.npx;
    const int C = S.C;
    for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < total; i += (size_t)gridDim.x * blockDim.x) {
        const int k = (int)(i / S.npx), p = (int)(i - (size_t)k * S.npx);
        if (C == 3) {
            const uint64_t d = (uint64_t)desc[i * 3] | ((uint64_t)desc[i * 3 + 1] << 16) | ((uint64_t)desc[i * 3 + 2] << 32) |
                               ((uint64_t)col[i * 3] << 48) | ((uint64_t)col[i * 3 + 1] << 56);
            store_sample<3>(samples_of<3>(S, p), k * S.sStride, d, col[i * 3 + 2]);
        } else {
            store_sample<1>(samples_of<1>(S, p), k * S.sStride, desc[i], col[i]);
        }
    }
}

// LBSP::compute2 (LBSP.cpp:102-152): dense extraction, absolute (thr >= 0) or relative threshold
extern "C" __global__ void lvbgs_lbsp_dense(const uint8_t* img, int W, int H, int C, int absThr, float rel,
                                            unsigned int off, uint16_t* desc) {
    const int total = W * H;
    for (int p = blockIdx.x * blockDim.x + threadIdx.x; p < total; p += gridDim.x * blockDim.x) {
        const int x = p % W, y = p / W;
        if (x < kBorder || y < kBorder || x >= W - kBorder || y >= H - kBorder) continue;
        for (int c = 0; c < C; ++c) {
            const uint8_t* base = img + (size_t)p * C;
            uint32_t vals[4];
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                uint32_t wv = 0;
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    const int n = j * 4 + i;
                    wv |= (uint32_t)base[(lbsp_dy(n) * W + lbsp_dx(n)) * C + c] << (8 * i);
                }
                vals[j] = wv;
            }
            const uint32_t ref = base[c];
            uint32_t thr;
            if (absThr >= 0) {
                thr = absThr > 255 ? 255u : (uint32_t)absThr;
            } else {
                int r = __float2int_rn((float)ref * rel + (float)off);
                thr = (uint32_t)(r < 0 ? 0 : r > 255 ? 255 : r);
            }
            desc[(size_t)p * C + c] = (uint16_t)lbsp_thr(vals, ref, thr);
        }
    }
}

}  // namespace lvbgs
