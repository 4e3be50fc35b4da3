// PAWCS (BackgroundSubtractorPAWCS, one channel) on sm_103a: the frame step as parallel passes that
// reproduce the reference's sequential raster scan exactly (scheme in pawcs_internal.h).
//
// Reference: modules/video/src/BackgroundSubtractorPAWCS.cpp -- refreshModel :107-429, initialize
// :431-557, apply :559-1516 (one-channel pixel loop :608-934, global words :1300-1334,
// post-processing :1443-1461, frame level :1462-1516), word weights :1596-1602.
#include <cuda_runtime.h>
#include <float.h>
#include <stdint.h>

#include "area_device.cuh"
#include "pawcs_device.cuh"

namespace lvbgs {

// the neighbour-update loop of updater p over target q's words (:850-878, one channel: the
// reference updates a copy of each word, so only the weight sum and the draws matter); returns
// the replacement decision and the pixel's draw count after the loop
struct PwWordSrc {
    const PawcsDev* S;
    int q, buf, L;
    uint32_t m;        // words whose colour/descriptor are the target's current values (illumination)
    uint32_t qcol, qdesc;
    int repl;          // last slot replaced by source rsrc
    uint32_t rcol, rdesc, rincr, t;
};
__device__ __forceinline__ PwWord pw_word(const PwWordSrc& s, int j) {
    if (s.repl && j == s.L - 1) return {s.rincr, s.t, s.t, s.rdesc, s.rcol};
    PwWord w = pw_load(*s.S, pw_slot(*s.S, s.buf, j, s.q));
    if (s.m & (1u << j)) {
        w.col = s.qcol;
        w.desc = s.qdesc;
    }
    return w;
}

// ------------------------------------------------------------------------------------------
// local pass: the pixel's word scan (:632-748) against its dictionary at its turn -- the frame-start
// dictionary with the last slot replaced by the latest earlier neighbour update, if any. Writes the
// scanned dictionary (next-frame buffer, illumination updates not yet applied) and the record. The words
// stream through registers: each is read once and written one slot later (the scan's bubble pass holds back
// one word, the lightest so far), where every word was read again, in its new order, to be written.
// ------------------------------------------------------------------------------------------
__device__ void pw_item_pixel(const PawcsDev& S, int p, const PwRec& R, uint32_t col);

extern "C" __global__ void __launch_bounds__(256) pw_k_local(PwParams P) {
    PW_ROUND_GUARD(P);
    const int t0 = blockIdx.x;
    if (t0 >= P.totalTiles) return;
    const PawcsDev& S = P.streams[pw_stream_by_tile(P, t0)];
    const StreamDev& D = S.sd;
    const int lt = t0 - D.tileBase;
    const int x = (lt % D.tilesX) * kTileW + (int)threadIdx.x % kTileW;
    const int y = (lt / D.tilesX) * kTileH + (int)threadIdx.x / kTileW;
    if (x >= D.W || y >= D.H) return;
    const int p = y * D.W + x;
    const uint8_t roi = D.roi[p];
    if (!roi) return;
    const PwRec R = S.rec[p];
    const uint32_t rsrc = S.repBefore[p];
    if (P.round > 0 && R.rsrc == rsrc) return;  // inputs unchanged since its last local pass
    const StreamCtl* ctl = D.ctl;
    const PawcsCtl* pc = S.pc;
    const uint32_t t = (uint32_t)(ctl->frame_idx + 1ull);
    const int cur = (int)(ctl->frame_idx & 1ull), nxt = cur ^ 1;
    const int L = S.L;
    const unsigned long long off = pc->lword_offset;
    const int boot = t <= (uint32_t)kBootWin;
    // current descriptor
    uint32_t taps[4];
    pw_taps<1>(D.frame, D.W, x, y, 0, taps);
    const uint32_t col = D.frame[p];
    const uint32_t desc = lbsp_thr(taps, col, ctl->lut[col]);
    const uint32_t bits = __popc(desc);
    const int flat = bits < 2u;
    const int border = roi < 255;
    const float* fm = D.fm + (size_t)cur * kNumFloatMaps * D.npx;
    const float Rr = fm[FM_R * D.npx + p];
    const uint32_t unst = S.unstable[p];
    const PwThr th = pw_thresholds(Rr, unst, S.minColor, S.descOff);
    const uint32_t cooldown = (uint32_t)ctl->cooldown;
    const uint32_t incr = (1u + cooldown) << (flat || boot ? 1 : 0);
    unsigned long long rate;
    if (isinf(P.lr)) rate = ~0ull;
    else if (P.lr > 0) rate = (unsigned long long)ceil(P.lr);
    else {
        const float T = fm[FM_T * D.npx + p];
        rate = flat ? (unsigned long long)ceilf(T + kTLower) / 2ull : (unsigned long long)ceilf(T);
    }
    // the dictionary at the pixel's turn: the frame-start words (read-only in this pass), the last
    // one replaced by an earlier neighbour update (its colour and descriptor, occurrences = its incr)
    PwWord repl = {0u, t, t, 0u, 0u};
    if (rsrc != kPwNone) {
        repl.col = D.frame[rsrc];
        repl.desc = S.descT[rsrc];
        repl.occ = S.rec[rsrc].incr;
    }
    const int occOn = !D.lastFG[p] || pc->moving_cam;
    float thrW = 0.0f;
    // word scan with one bubble pass
    uint32_t k = 0;
    float sumW = 0.0f, lastW = FLT_MAX;
    uint32_t minColor = 255, minDesc = 16;
    uint32_t m0 = 0, m1 = 0;  // illumination marks by final slot
    int any0 = 0, any1 = 0;
    const unsigned long long rateHalf = rate / 2ull + 1ull;
    const bool illumOn = !unst || flat || border;
    const size_t npx = (size_t)D.npx;
    size_t src = pw_slot(S, cur, 0, p), dst = pw_slot(S, nxt, 0, p);
    PwWord held = {0u, 0u, 0u, 0u, 0u}, next = pw_load(S, src);
    uint32_t heldMarks = 0;
    for (int i = 0; i < L; ++i) {
        PwWord w = next;
        if (i + 1 < L) {
            src += npx;
            next = pw_load(S, src);
        } else if (rsrc != kPwNone) {
            w = repl;
        }
        const float cw = pw_weight(w.occ, w.first, w.last, t, off);
        if (i == 0) thrW = cw / (Rr * 2.0f);
        uint32_t marks = 0;
        bool matched = false;
        if (sumW < thrW) {
            const uint32_t cd = pw_absdiff(col, w.col);
            if (cd <= th.color) {
                const uint32_t intra = __popc(desc ^ w.desc);
                const uint32_t inter = __popc((lbsp_thr_raw(taps, w.col, ctl->lut[w.col]) ^ w.desc) & 0xffffu);
                const uint32_t dd = (intra + inter) / 2u;
                if (illumOn && cd >= th.color / 2u && intra <= th.desc / 2u) {
                    // illumination update test (:684): modulus halves (+1) once the mask is non-zero
                    const uint32_t r = pw_draw(D.seed, t, (uint32_t)p, k++);
                    if (pw_mod(r, rateHalf) == 0u) {
                        marks |= 2u;
                        any1 = 1;
                    }
                    if (pw_mod(r, any0 ? rateHalf : rate) == 0u) {
                        marks |= 1u;
                        any0 = 1;
                    }
                }
                if (dd <= th.desc) {
                    sumW += cw;
                    matched = true;
                    minColor = min(minColor, cd);
                    minDesc = min(minDesc, dd);
                }
            }
        }
        if (matched) {  // seen now, occurrences incremented
            w.last = t;
            if (occOn && cw < 1.0f) w.occ += incr;
        }
        if (cw > lastW) {  // heavier than the held word: it takes the slot before it
            pw_store(S, dst, w);
            m0 |= (marks & 1u) << (i - 1);
            m1 |= (marks >> 1) << (i - 1);
            dst += npx;
        } else {
            if (i > 0) {
                pw_store(S, dst, held);
                m0 |= (heldMarks & 1u) << (i - 1);
                m1 |= (heldMarks >> 1) << (i - 1);
                dst += npx;
            }
            held = w;
            heldMarks = marks;
            lastW = cw;
        }
    }
    m0 |= (heldMarks & 1u) << (L - 1);
    m1 |= (heldMarks >> 1) << (L - 1);
    const int bg = sumW >= thrW || border;
    const float initW = 1.0f / (float)off;
    uint8_t flags = (uint8_t)((bg ? kRfBG : 0) | (flat ? kRfFlat : 0) | (border ? kRfBorder : 0) |
                              (any0 ? kRfU0 : 0) | (any1 ? kRfU1 : 0));
    if (bg) {
        // global dictionary event (:774) and, when nothing matches, the replacement draw (:785)
        if (pw_mod(pw_draw(D.seed, t, (uint32_t)p, k), rate) == 0u) {
            flags |= kRfItem | kRfEvent;
            if (pw_mod(pw_draw(D.seed, t, (uint32_t)p, k + 1), rate * 2ull) == 0u) flags |= kRfRepDraw;
        }
    } else {
        if (flat || pw_mod(pw_draw(D.seed, t, (uint32_t)p, k), rate) == 0u) flags |= kRfItem;
        if (sumW < initW) held = {incr, t, t, desc, col};  // new local word in the last slot (:822-830)
    }
    pw_store(S, dst, held);
    S.descT[p] = (uint16_t)desc;
    S.uv[p] = (uint8_t)((any0 ? 1 : 0) | (any1 ? 2 : 0));
    R.sumW = sumW;
    R.thrW = thrW;
    R.rate = rate;
    R.m0 = m0;
    R.m1 = m1;
    R.rsrc = rsrc;
    R.kScan = (uint16_t)k;
    R.incr = (uint16_t)incr;
    R.minColor = (uint16_t)minColor;
    R.minDesc = (uint16_t)minDesc;
    R.m0hi = 0;
    R.m1hi = 0;
    R.flags = flags;
    R.bits = (uint8_t)bits;
    pw_item_pixel(S, p, R, col);
}

// ------------------------------------------------------------------------------------------
// illumination chain: the mask a pixel sees is 1 & ROI when its left neighbour made an illumination
// update this frame (the neighbour writes 1 & m_oROI, :689-690: 1 inside the ROI, 0 in its edge band
// of 128), else its frame-start value (:686-688, :893-894). Each pixel's outcome is a function of its
// left neighbour's (two states), so one warp per row scans the compositions 32 pixels at a time.
// ------------------------------------------------------------------------------------------
extern "C" __global__ void __launch_bounds__(256) pw_k_illum(PwParams P) {
    PW_ROUND_GUARD(P);
    const int gr = blockIdx.x * 8 + (int)threadIdx.x / 32, lane = threadIdx.x & 31;
    if (gr >= P.totalRows) return;
    const PawcsDev& S = P.streams[pw_stream_by_row(P, gr)];
    const StreamDev& D = S.sd;
    const int y = gr - D.rowBase;
    uint32_t carry = 0;  // outcome of the pixel before the chunk
    const int row = y * D.W;
    // four chunks a step: their loads are requested before the first is scanned
    for (int xb = 0; xb < D.W; xb += 128) {
        uint32_t roi[4], uvp[4], il[4];
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const int x = xb + 32 * j + lane;
            roi[j] = uvp[j] = il[j] = 0u;
            if (x < D.W) {
                roi[j] = D.roi[row + x];
                uvp[j] = S.uv[row + x];
                il[j] = S.illum[row + x];
            }
        }
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const int x = xb + 32 * j + lane;
            if (xb + 32 * j >= D.W) break;
            const bool in = roi[j] != 0u;
            uint32_t f = 0, m0 = 0, mL = 0;  // f: bit0 = outcome if the left neighbour made no update, bit1 = if it did
            if (in) {
                m0 = il[j] != 0u;
                mL = roi[j] & 1u;  // the mask after the left neighbour's update
                const uint32_t u0 = uvp[j] & 1u, u1 = (uvp[j] >> 1) & 1u;
                f = (m0 ? u1 : u0) | ((mL ? u1 : u0) << 1);
            }
            // inclusive scan: F = f_lane o f_lane-1 o ... o f_x0
            uint32_t F = f;
#pragma unroll
            for (int d = 1; d < 32; d <<= 1) {
                const uint32_t o = __shfl_up_sync(0xffffffffu, F, d);
                if (lane >= d) F = ((F >> (o & 1u)) & 1u) | (((F >> ((o >> 1) & 1u)) & 1u) << 1);
            }
            const uint32_t u = (F >> carry) & 1u;
            uint32_t prevU = __shfl_up_sync(0xffffffffu, u, 1);
            if (lane == 0) prevU = carry;
            if (x < D.W) S.uFinal[row + x] = in ? (uint8_t)(u | ((prevU ? mL : m0) ? 2u : 0u)) : (uint8_t)0;
            carry = __shfl_sync(0xffffffffu, u, 31);
        }
    }
}

// ------------------------------------------------------------------------------------------
// global items: a BG pixel's dictionary event or an FG pixel's consultation. The first matching
// word in the pixel's sort table decides; only the replaceable word (last dictionary slot) changes
// features during a frame, so an item whose first non-replaceable match precedes the replaceable
// word is settled here, and the others go to the ordered scan. Run at the end of the pixel's local
// pass: it depends on nothing else that changes during the frame, so a pixel that does not rerun
// keeps its item.
// ------------------------------------------------------------------------------------------
__device__ void pw_item_pixel(const PawcsDev& S, int p, const PwRec& R, uint32_t col) {
    const StreamDev& D = S.sd;
    const PwOut O = S.out[p];
    O.gflags = 0;
    O.epoch = 0;
    O.gword = kPwNone;
    if (!(R.flags & kRfItem)) return;
    const PawcsCtl* pc = S.pc;
    const int G = S.G;
    const int wr = pc->gdict[G - 1];
    const float* fm = D.fm + (size_t)(D.ctl->frame_idx & 1ull) * kNumFloatMaps * D.npx;
    const PwThr th = pw_thresholds(fm[FM_R * D.npx + p], S.unstable[p], S.minColor, S.descOff);
    const uint32_t bits = R.bits;
    const uint8_t* lut = S.glut + (size_t)p * kPwGlutStride;
    int fixedPos = G, wrPos = G, fixedWord = -1;
    for (int g = 0; g < G; ++g) {
        const int w = lut[g];
        if (w == wr) {
            wrPos = g;
            continue;
        }
        if (pw_absdiff(pc->gw_color[w], col) <= th.color && pw_absdiff(bits, pc->gw_bits[w]) <= th.desc / 4u) {
            fixedPos = g;  // a replaceable word further on is behind it
            fixedWord = w;
            break;
        }
    }
    const int critical = wrPos < fixedPos;
    if (!critical) O.gword = (uint32_t)fixedWord;
    S.gitem[p] = (uint32_t)(fixedWord < 0 ? 63 : fixedWord) | ((uint32_t)fixedPos << 6) | ((uint32_t)critical << 12);
    if (critical) O.gflags |= 4;
}

// ------------------------------------------------------------------------------------------
// ordered compactions (raster order kept): mode 0 lists the critical global items, mode 1 the word
// weight contributions per word, mode 2 the pixels that update a neighbour. Mode 1 has a list per word, so it
// counts, makes offsets and scatters in three launches, over blocks of kPwCompactBlk pixels.
// ------------------------------------------------------------------------------------------
__device__ __forceinline__ int pw_category(const PawcsDev& S, int p, int mode, int wr, uint32_t nrep) {
    if (!S.sd.roi[p]) return -1;
    const PwOut O = S.out[p];
    if (mode == 0) return ((S.rec[p].flags & kRfItem) && (O.gflags & 4)) ? 0 : -1;
    if (mode == 2) return O.q != kPwNone ? 0 : -1;
    if (S.contrib[p] < 0.0f) return -1;
    // the replaceable word keeps only the contributions after its last replacement of the frame
    if (O.gword >= (uint32_t)S.G) return -1;
    if ((int)O.gword == wr && nrep > 0 && O.epoch != nrep) return -1;
    return (int)O.gword;
}

extern "C" __global__ void __launch_bounds__(256) pw_k_compact_count(PwParams P) {
    PW_ROUND_GUARD(P);
    if (P.gate && *(const volatile unsigned int*)P.gate == 0u) return;
    const PawcsDev& S = P.streams[0];
    const int nb = (S.sd.npx + kPwCompactBlk - 1) / kPwCompactBlk;
    if ((int)blockIdx.x >= nb) return;
    __shared__ uint32_t cnt[kPwCats];
    if (threadIdx.x < kPwCats) cnt[threadIdx.x] = 0;
    __syncthreads();
    const int wr = S.pc->gdict[S.G - 1];
    const uint32_t nrep = S.pc->n_repl;
    for (int k = 0; k < kPwCompactBlk / 256; ++k) {
        const int p = blockIdx.x * kPwCompactBlk + k * 256 + threadIdx.x;
        if (p < S.sd.npx) {
            const int c = pw_category(S, p, 1, wr, nrep);
            if (c >= 0) atomicAdd(&cnt[c], 1u);
        }
    }
    __syncthreads();
    if (threadIdx.x < kPwCats) S.blkCounts[(size_t)blockIdx.x * kPwCats + threadIdx.x] = cnt[threadIdx.x];
}

// per category (one warp each): exclusive offsets over the blocks (in place), totals and the category
// bases of the word-major list; the compaction uses categories [0, ncat), the others are left empty
extern "C" __global__ void __launch_bounds__(1024) pw_k_compact_offsets(PwParams P, int ncat) {
    PW_ROUND_GUARD(P);
    if (P.gate && *(const volatile unsigned int*)P.gate == 0u) return;
    const PawcsDev& S = P.streams[0];
    const int nb = (S.sd.npx + kPwCompactBlk - 1) / kPwCompactBlk;
    __shared__ uint32_t tot[kPwCats];
    const int lane = threadIdx.x & 31;
    for (int i = threadIdx.x; i < kPwCats; i += blockDim.x) tot[i] = 0;
    __syncthreads();
    for (int c = threadIdx.x >> 5; c < ncat; c += blockDim.x >> 5) {
        uint32_t run = 0;
        for (int b0 = 0; b0 < nb; b0 += 32) {
            const int b = b0 + lane;
            uint32_t* e = &S.blkCounts[(size_t)b * kPwCats + c];
            const uint32_t v = b < nb ? *e : 0u;
            uint32_t inc = v;
#pragma unroll
            for (int d = 1; d < 32; d <<= 1) {
                const uint32_t o = __shfl_up_sync(0xffffffffu, inc, d);
                if (lane >= d) inc += o;
            }
            if (b < nb) *e = run + inc - v;
            run += __shfl_sync(0xffffffffu, inc, 31);
        }
        if (lane == 0) tot[c] = run;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        uint32_t base = 0;
        for (int k = 0; k < kPwCats; ++k) {
            S.catInfo[k] = tot[k];
            S.catInfo[kPwCatBase + k] = base;
            base += tot[k];
        }
    }
}

extern "C" __global__ void __launch_bounds__(256) pw_k_compact_scatter(PwParams P) {
    PW_ROUND_GUARD(P);
    if (P.gate && *(const volatile unsigned int*)P.gate == 0u) return;
    const PawcsDev& S = P.streams[0];
    const StreamDev& D = S.sd;
    const int nb = (D.npx + kPwCompactBlk - 1) / kPwCompactBlk;
    if ((int)blockIdx.x >= nb) return;
    __shared__ uint32_t warpCnt[8][kPwCats];
    __shared__ uint32_t run[kPwCats], passTot[kPwCats];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const int wr = S.pc->gdict[S.G - 1];
    const uint32_t nrep = S.pc->n_repl;
    if (threadIdx.x < kPwCats)
        run[threadIdx.x] = S.catInfo[kPwCatBase + threadIdx.x] + S.blkCounts[(size_t)blockIdx.x * kPwCats + threadIdx.x];
    for (int k = 0; k < kPwCompactBlk / 256; ++k) {
        const int p = blockIdx.x * kPwCompactBlk + k * 256 + threadIdx.x;
        const int c = p < D.npx ? pw_category(S, p, 1, wr, nrep) : -1;
        uint32_t rank = 0;
        const int ncat = S.G;
        for (int j = 0; j < ncat; ++j) {
            const unsigned m = __ballot_sync(0xffffffffu, c == j);
            if (c == j) rank = __popc(m & ((1u << lane) - 1u));
            if (lane == 0) warpCnt[w][j] = __popc(m);
        }
        __syncthreads();
        if (threadIdx.x < ncat) {
            // exclusive offsets of the warps within this pass, then the pass total
            uint32_t r = 0;
            for (int i = 0; i < 8; ++i) {
                const uint32_t v = warpCnt[i][threadIdx.x];
                warpCnt[i][threadIdx.x] = r;
                r += v;
            }
            passTot[threadIdx.x] = r;
        }
        __syncthreads();
        if (c >= 0) {
            const uint32_t pos = run[c] + warpCnt[w][c] + rank;
            S.contribList[pos] = S.contrib[p];
        }
        __syncthreads();
        if (threadIdx.x < ncat) run[threadIdx.x] += passTot[threadIdx.x];
        __syncthreads();
    }
}

// The ordered compactions of one category (modes 0 and 2) in one pass: a block takes the next kPwOneBlk
// pixels (by ticket, so that the blocks before it are running or done), counts its members, publishes the
// count, and finds its offset by looking back over the blocks before it, a warp's width at a time, until one
// that has published its total. Count, offsets and scatter were three launches (7 + 8 + 9 us of a 640x480
// frame, up to eleven times a frame). The wait is bounded (ERR_BARRIER_TIMEOUT). The generation tells this launch's entries from
// the last one's; the block with the last ticket advances it.
__device__ __forceinline__ void pw_list_item(const PawcsDev& S, int mode, int p, uint32_t pos) {
    if (mode == 2) {
        S.updList[pos] = (uint32_t)p;
        return;
    }
    const StreamDev& D = S.sd;
    const float* fm = D.fm + (size_t)(D.ctl->frame_idx & 1ull) * kNumFloatMaps * D.npx;
    // two records per item (pixel, colour|bits, thresholds, descriptors 0-1; descriptor 2|event
    // flags, fixed position|word, and the global scan's speculative outcome)
    const PwRec R = S.rec[p];
    const bool c3 = D.C == 3;
    const PwThr th = c3 ? pw3_thresholds(fm[FM_R * D.npx + p], S.unstable[p], S.minColor, S.descOff)
                        : pw_thresholds(fm[FM_R * D.npx + p], S.unstable[p], S.minColor, S.descOff);
    const uint32_t g = S.gitem[p];
    const uint16_t* dt = S.descT + (size_t)p * (c3 ? 3 : 1);
    const uint32_t a = (c3 ? pw3_color(D.frame, p) : (uint32_t)D.frame[p]) | ((uint32_t)R.bits << 24);
    const uint32_t b = min(th.color, 65535u) | (min(th.desc / 4u, 65535u) << 16);
    const uint32_t d01 = c3 ? (uint32_t)dt[0] | ((uint32_t)dt[1] << 16) : (uint32_t)dt[0];
    const uint32_t d2 = c3 ? (uint32_t)dt[2] : 0u;
    S.itemList[2 * pos] = make_uint4((uint32_t)p, a, b, d01);
    S.itemList[2 * pos + 1] = make_uint4(d2 | ((uint32_t)(R.flags & (kRfEvent | kRfRepDraw)) << 16),
                                         ((g >> 6) & 63u) | ((g & 63u) << 8), 0u, 0u);
}
extern "C" __global__ void __launch_bounds__(kPwOneThreads) pw_k_compact(PwParams P, int mode) {
    PW_ROUND_GUARD(P);
    const PawcsDev& S = P.streams[0];
    const int npx = S.sd.npx, nb = (npx + kPwOneBlk - 1) / kPwOneBlk;
    constexpr int K = kPwOneBlk / kPwOneThreads, WARPS = kPwOneThreads / 32, PER = K * WARPS / 32;
    __shared__ uint32_t sBid, sGen, sCnt[K * WARPS], sBase;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    if (threadIdx.x == 0) {
        sBid = atomicAdd(&S.ticket[0], 1u);
        sGen = *(volatile unsigned int*)&S.ticket[1] & 0x3fffffffu;
    }
    __syncthreads();
    const int bid = (int)sBid;
    bool in[K];
    uint32_t rank[K];
#pragma unroll
    for (int k = 0; k < K; ++k) {
        const int p = bid * kPwOneBlk + k * kPwOneThreads + (int)threadIdx.x;
        in[k] = p < npx && pw_category(S, p, mode, 0, 0u) == 0;
    }
#pragma unroll
    for (int k = 0; k < K; ++k) {
        const unsigned m = __ballot_sync(0xffffffffu, in[k]);
        rank[k] = (uint32_t)__popc(m & ((1u << lane) - 1u));
        if (lane == 0) sCnt[k * WARPS + warp] = (uint32_t)__popc(m);
    }
    __syncthreads();
    if (warp == 0) {
        static_assert(PER * 32 == K * WARPS, "whole lanes");
        // offsets of the warps in raster order and the block's total
        uint32_t v[PER], sum = 0;
#pragma unroll
        for (int i = 0; i < PER; ++i) {
            v[i] = sum;
            sum += sCnt[lane * PER + i];
        }
        uint32_t inc = sum;
#pragma unroll
        for (int d = 1; d < 32; d <<= 1) {
            const uint32_t o = __shfl_up_sync(0xffffffffu, inc, d);
            if (lane >= d) inc += o;
        }
#pragma unroll
        for (int i = 0; i < PER; ++i) sCnt[lane * PER + i] = inc - sum + v[i];
        const uint32_t total = __shfl_sync(0xffffffffu, inc, 31);
        const unsigned long long tag = (unsigned long long)sGen << 34, kCount = 1ull << 32, kTotal = 2ull << 32;
        volatile unsigned long long* chain = S.chain;
        uint32_t base = 0;
        if (bid > 0) {
            if (lane == 0) chain[bid] = tag | kCount | total;
            for (int at = bid - 1; at >= 0;) {
                const int b = at - lane;
                unsigned long long e = tag | kTotal;  // before the first block: a total of 0
                for (int spin = 0; b >= 0; ++spin) {
                    e = chain[b];
                    if ((e >> 34) == (unsigned long long)sGen && ((e >> 32) & 3ull) != 0ull) break;
                    if (spin > (1 << 22)) {
                        atomicOr(P.err, ERR_BARRIER_TIMEOUT);
                        e = tag | kTotal;
                        break;
                    }
                    __nanosleep(20);
                }
                __syncwarp();
                const unsigned done = __ballot_sync(0xffffffffu, ((e >> 32) & 3ull) == 2ull);
                const int stop = done ? __ffs(done) - 1 : 31;  // the nearest block with a total
                base += __reduce_add_sync(0xffffffffu, lane <= stop ? (uint32_t)e : 0u);
                if (done) break;
                at -= 32;
            }
        }
        if (lane == 0) {
            __threadfence();
            chain[bid] = tag | kTotal | (base + total);
            sBase = base;
            if (bid == nb - 1) {
                S.catInfo[0] = base + total;
                S.catInfo[kPwCatBase] = 0u;
                S.ticket[0] = 0u;
                *(volatile unsigned int*)&S.ticket[1] = (sGen + 1u) & 0x3fffffffu;
            }
        }
    }
    __syncthreads();
    const uint32_t base = sBase;
#pragma unroll
    for (int k = 0; k < K; ++k)
        if (in[k])
            pw_list_item(S, mode, bid * kPwOneBlk + k * kPwOneThreads + (int)threadIdx.x, base + sCnt[k * WARPS + warp] + rank[k]);
}

// per 2x2 cell of the spatial maps: the cell's (at most four) items in raster order (:786-791,
// :805-812); final = 1 also writes the frame's map values and word contributions
extern "C" __global__ void pw_k_cells(PwParams P, int final) {
    PW_ROUND_GUARD(P);
    if (P.gate && *(const volatile unsigned int*)P.gate == 0u) return;
    int c = blockIdx.x * blockDim.x + threadIdx.x;
    if (c >= P.totalCells) return;
    int si = 0;
    while (si + 1 < P.nStreams && c >= P.streams[si].gwW * P.streams[si].gwH) {
        c -= P.streams[si].gwW * P.streams[si].gwH;
        ++si;
    }
    const PawcsDev& S = P.streams[si];
    const StreamDev& D = S.sd;
    const PawcsCtl* pc = S.pc;
    const int cx = c % S.gwW, cy = c / S.gwW;
    const size_t ncell = (size_t)S.gwW * S.gwH;
    const int G = S.G;
    const int wr = pc->gdict[G - 1];
    int ws[4];
    float vs[4];
    int nw = 0;
    uint32_t wrE = 0;
    float wrV = S.gmap[(size_t)wr * ncell + c];
    int wrTouched = 0;
    for (int k = 0; k < 4; ++k) {
        const int x = 2 * cx + (k & 1), y = 2 * cy + (k >> 1);
        if (x >= D.W || y >= D.H) continue;
        const int p = y * D.W + x;
        if (!D.roi[p]) continue;
        const PwRec R = S.rec[p];
        if (!(R.flags & kRfItem)) {
            if (final) S.contrib[p] = -1.0f;
            continue;
        }
        const PwOut O = S.out[p];
        const uint32_t w = O.gword;
        float contrib = -1.0f;
        if (w == kPwNone) {
            if (!(R.flags & kRfBG)) O.segm = 255;
        } else {
            float* v;
            if ((int)w == wr) {
                if (O.epoch != wrE) {
                    wrV = 0.0f;  // the word was replaced (its map zeroed) since the cell's last look
                    wrE = O.epoch;
                }
                v = &wrV;
                wrTouched = 1;
            } else {
                int j = 0;
                while (j < nw && ws[j] != (int)w) ++j;
                if (j == nw) {
                    ws[nw] = (int)w;
                    vs[nw] = S.gmap[(size_t)w * ncell + c];
                    ++nw;
                }
                v = &vs[j];
            }
            if (R.flags & kRfBG) {
                if (*v < R.sumW) {
                    *v = *v + R.sumW;
                    contrib = R.sumW;
                }
            } else {
                const float div = (R.flags & kRfFlat) ? 2.0f : 4.0f;
                O.segm = (R.sumW + *v / div < R.thrW) ? 255 : 0;
            }
        }
        if (final) S.contrib[p] = contrib;
    }
    if (!final) return;
    for (int j = 0; j < nw; ++j) S.gmap[(size_t)ws[j] * ncell + c] = vs[j];
    // the replaceable word: values after the frame's last replacement; zero elsewhere when replaced
    const uint32_t nrep = pc->n_repl;
    if (nrep == 0) {
        if (wrTouched) S.gmap[(size_t)wr * ncell + c] = wrV;
    } else {
        S.gmap[(size_t)wr * ncell + c] = (wrTouched && wrE == nrep) ? wrV : 0.0f;
    }
}

// neighbour-update gate and target (:839-848): the draws before it depend on the global outcome
extern "C" __global__ void __launch_bounds__(256) pw_k_nbr(PwParams P) {
    PW_ROUND_GUARD(P);
    const int t0 = blockIdx.x;
    if (t0 >= P.totalTiles) return;
    const PawcsDev& S = P.streams[pw_stream_by_tile(P, t0)];
    const StreamDev& D = S.sd;
    const int lt = t0 - D.tileBase;
    const int x = (lt % D.tilesX) * kTileW + (int)threadIdx.x % kTileW;
    const int y = (lt / D.tilesX) * kTileH + (int)threadIdx.x / kTileW;
    if (x >= D.W || y >= D.H) return;
    const int p = y * D.W + x;
    if (!D.roi[p]) return;
    const PwRec R = S.rec[p];
    const PwOut O = S.out[p];
    const uint32_t t = (uint32_t)(D.ctl->frame_idx + 1ull);
    uint32_t k = R.kScan;
    uint8_t segm;
    if (R.flags & kRfBG) {
        segm = 0;
        ++k;  // the event draw (:774), taken whatever its outcome
        if (R.flags & kRfEvent) {
            const bool noMatch = O.gword == kPwNone || (O.gflags & 1);
            if (noMatch) ++k;  // the replacement draw (:785), taken when no word matched
        }
    } else {
        if (!(R.flags & kRfFlat)) ++k;  // the consultation gate draw
        if (!(R.flags & kRfItem)) O.segm = 255;
        segm = O.segm;
    }
    if (R.flags & kRfBG) O.segm = 0;
    const int border = (R.flags & kRfBorder) != 0, flat = (R.flags & kRfFlat) != 0;
    const int moving = S.pc->moving_cam;
    bool upd = false;
    if (!segm) upd = pw_mod(pw_draw(D.seed, t, (uint32_t)p, k++), R.rate) == 0u;
    upd = upd || border || moving;
    // the previous round's loop inputs (round 0: no update known to the targets' local passes)
    const uint32_t oldQ = P.round == 0 ? kPwNone : O.q;
    const uint16_t oldK = O.kLoop;
    const float oldThr = O.thrW;
    O.q = kPwNone;
    if (upd) {
        const uint32_t r = pw_draw(D.seed, t, (uint32_t)p, k++);
        int nx, ny;
        if (flat || border || moving) nb5_offset((int)(r % 24u), nx, ny);
        else nb3_offset((int)(r % 8u), nx, ny);
        nx += x;
        ny += y;
        nx = nx < 2 ? 2 : nx >= D.W - 2 ? D.W - 3 : nx;
        ny = ny < 2 ? 2 : ny >= D.H - 2 ? D.H - 3 : ny;
        const int q = ny * D.W + nx;
        if (D.roi[q]) O.q = (uint32_t)q;
    }
    O.kLoop = (uint16_t)k;
    O.thrW = R.thrW;
    O.qPrev = oldQ;
    O.chg = (uint8_t)(O.q != oldQ || (O.q != kPwNone && (O.kLoop != oldK || O.thrW != oldThr)));
}

// the neighbour-update loop of updater p on target q (:847-880; one channel: the reference updates a
// copy of each word, so only the weight sum and the draws count). p sees q's dictionary before q's own
// scan (p < q: frame-start words, the last one replaced by the earlier updater rs, if any) or after it
// (p >= q: the scanned words with their illumination marks). Returns the weight sum; k advances by
// the loop's draws; reachedLast tells whether the loop looked at the last word (the only one rs changes).
__device__ float pw_nbr_loop(const PawcsDev& S, uint32_t t, int cur, int nxt, int boot, unsigned long long off, int p,
                             int q, uint32_t rs, uint32_t& k, bool& reachedLast) {
    const StreamDev& D = S.sd;
    const float* fm = D.fm + (size_t)cur * kNumFloatMaps * D.npx;
    const PwRec R = S.rec[p];
    const uint32_t col = D.frame[p], desc = S.descT[p];
    const PwThr th = pw_thresholds(fm[FM_R * D.npx + p], S.unstable[p], S.minColor, S.descOff);
    const int flat = (R.flags & kRfFlat) != 0;
    PwWordSrc ws;
    ws.S = &S;
    ws.q = q;
    ws.L = S.L;
    ws.t = t;
    ws.qcol = D.frame[q];
    ws.qdesc = S.descT[q];
    uint8_t segmQ;
    uint32_t lastDescQ;
    if (p < q) {
        ws.buf = cur;
        ws.m = 0;
        segmQ = 0;
        lastDescQ = D.lastDesc[q];
    } else {
        const PwRec Rq = S.rec[q];
        ws.buf = nxt;
        ws.m = (S.uFinal[q] & 2) ? Rq.m1 : Rq.m0;
        segmQ = S.out[q].segm;
        // the pixel's last descriptor is updated at the end of its own processing (:925-926)
        lastDescQ = p == q ? D.lastDesc[q] : S.descT[q];
    }
    ws.repl = rs != kPwNone;
    if (ws.repl) {
        ws.rcol = D.frame[rs];
        ws.rdesc = S.descT[rs];
        ws.rincr = S.rec[rs].incr;
    }
    float nsum = 0.0f;
    reachedLast = false;
    for (int j = 0; j < S.L && nsum < R.thrW; ++j) {
        if (j == S.L - 1) reachedLast = true;
        const PwWord w = pw_word(ws, j);
        const uint32_t cd = pw_absdiff(col, w.col);
        if (cd <= th.color && (uint32_t)__popc(desc ^ w.desc) <= th.desc) {
            nsum += pw_weight(w.occ, w.first, w.last, t, off);
        } else if (!segmQ && flat && (boot || pw_mod(pw_draw(D.seed, t, (uint32_t)p, k++), R.rate) == 0u)) {
            if (cd <= th.color && (uint32_t)__popc(desc ^ lastDescQ) <= th.desc / 2u)
                nsum += pw_weight(w.occ, w.first, w.last, t, off);
        }
    }
    return nsum;
}

// neighbour updates, pass 1: every updater's loop (one thread each, over the compacted list), as if no
// earlier updater of its target had replaced the target's last word
extern "C" __global__ void __launch_bounds__(256) pw_k_nbr_loops(PwParams P) {
    PW_ROUND_GUARD(P);
    const PawcsDev& S = P.streams[0];
    const StreamDev& D = S.sd;
    const uint32_t n = S.catInfo[0];
    const uint32_t t = (uint32_t)(D.ctl->frame_idx + 1ull);
    const int cur = (int)(D.ctl->frame_idx & 1ull), nxt = cur ^ 1;
    const int boot = t <= (uint32_t)kBootWin;
    const unsigned long long off = S.pc->lword_offset;
    const float initW = 1.0f / (float)off;
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        const int p = (int)S.updList[i];
        const PwOut O = S.out[p];
        uint32_t k = O.kLoop;
        bool reachedLast;
        const float nsum = pw_nbr_loop(S, t, cur, nxt, boot, off, p, (int)O.q, kPwNone, k, reachedLast);
        O.kEnd = (uint16_t)k;
        O.rflags = (uint8_t)((nsum < initW ? 1 : 0) | (reachedLast ? 2 : 0));
    }
}

// neighbour updates, pass 2 (per target, raster order over its <= 25 updaters): the latest updater of
// each group that replaces the last word is the replacement source the next ones see; a later updater
// whose loop reached that word is redone with it (the earlier words are the same either way)
extern "C" __global__ void __launch_bounds__(256) pw_k_replace(PwParams P) {
    PW_ROUND_GUARD(P);
    const int t0 = blockIdx.x;
    if (t0 >= P.totalTiles) return;
    const PawcsDev& S = P.streams[pw_stream_by_tile(P, t0)];
    const StreamDev& D = S.sd;
    const int lt = t0 - D.tileBase;
    const int qx = (lt % D.tilesX) * kTileW + (int)threadIdx.x % kTileW;
    const int qy = (lt / D.tilesX) * kTileH + (int)threadIdx.x / kTileW;
    if (qx >= D.W || qy >= D.H) return;
    const int q = qy * D.W + qx;
    if (!D.roi[q]) return;
    const StreamCtl* ctl = D.ctl;
    const uint32_t t = (uint32_t)(ctl->frame_idx + 1ull);
    const int cur = (int)(ctl->frame_idx & 1ull), nxt = cur ^ 1;
    const int boot = t <= (uint32_t)kBootWin;
    const unsigned long long off = S.pc->lword_offset;
    const float initW = 1.0f / (float)off;
    uint32_t before = kPwNone, after = kPwNone;
    uint32_t hits = 0;  // window slots whose pixel updates q
#pragma unroll
    for (int j = 0; j < 25; ++j) {
        const int px = qx + j % 5 - 2, py = qy + j / 5 - 2;
        if (px >= 0 && py >= 0 && px < D.W && py < D.H && S.out[py * D.W + px].q == (uint32_t)q) hits |= 1u << j;
    }
    for (; hits; hits &= hits - 1u) {
        const int j = __ffs(hits) - 1;
        const int p = (qy + j / 5 - 2) * D.W + qx + j % 5 - 2;
        // p == q happens when the clamped neighbour position falls back onto the pixel itself (at
        // the ROI's outer rows and columns): the update then follows the pixel's own processing
        const PwOut O = S.out[p];
        const uint32_t rs = p < q ? before : after;
        uint8_t rf = O.rflags;
        if (rs != kPwNone && (rf & 2)) {
            uint32_t k = O.kLoop;
            bool reachedLast;
            const float nsum = pw_nbr_loop(S, t, cur, nxt, boot, off, p, q, rs, k, reachedLast);
            rf = (uint8_t)((nsum < initW ? 1 : 0) | (reachedLast ? 2 : 0));
            O.kEnd = (uint16_t)k;
            O.rflags = rf;
        }
        if (rf & 1) {
            if (p < q) before = (uint32_t)p;
            else after = (uint32_t)p;
        }
    }
    S.repBefore[q] = before;
    S.repAfter[q] = after;
}

// pixels whose replacement source changed since their local pass are redone next round
extern "C" __global__ void __launch_bounds__(256) pw_k_dirty(PwParams P) {
    PW_ROUND_GUARD(P);
    const int t0 = blockIdx.x;
    if (t0 >= P.totalTiles) return;
    const PawcsDev& S = P.streams[pw_stream_by_tile(P, t0)];
    const StreamDev& D = S.sd;
    const int lt = t0 - D.tileBase;
    const int x = (lt % D.tilesX) * kTileW + (int)threadIdx.x % kTileW;
    const int y = (lt / D.tilesX) * kTileH + (int)threadIdx.x / kTileW;
    bool dirty = false;
    if (x < D.W && y < D.H) {
        const int p = y * D.W + x;
        dirty = D.roi[p] && S.repBefore[p] != S.rec[p].rsrc;
    }
    pw_round_end(P, dirty);
}

// ------------------------------------------------------------------------------------------
// commit of the frame's pixel loop: final dictionaries (illumination updates, later neighbour
// replacements), feedback maps (:764-771, :800-806, :895-914), illumination mask, last colour and
// descriptor, raw mask (as the post-processing "intent" word) and draw counters
// ------------------------------------------------------------------------------------------
extern "C" __global__ void __launch_bounds__(256) pw_k_commit(PwParams P) {
    PW_TAIL_GATE(P);
    const int t0 = blockIdx.x;
    if (t0 >= P.totalTiles) return;
    const PawcsDev& S = P.streams[pw_stream_by_tile(P, t0)];
    const StreamDev& D = S.sd;
    const int lt = t0 - D.tileBase;
    const int x = (lt % D.tilesX) * kTileW + (int)threadIdx.x % kTileW;
    const int y = (lt / D.tilesX) * kTileH + (int)threadIdx.x / kTileW;
    const bool in = x < D.W && y < D.H;
    const int p = in ? y * D.W + x : 0;
    const bool act = in && D.roi[p];
    int flat = 0;
    if (act) {
        const StreamCtl* ctl = D.ctl;
        const uint32_t t = (uint32_t)(ctl->frame_idx + 1ull);
        const int cur = (int)(ctl->frame_idx & 1ull), nxt = cur ^ 1;
        const int boot = t <= (uint32_t)kBootWin;
        const PwRec R = S.rec[p];
        const PwOut O = S.out[p];
        const uint32_t col = D.frame[p], desc = S.descT[p];
        flat = (R.flags & kRfFlat) != 0;
        // dictionary: illumination updates, then a later neighbour's replacement of the last slot
        const uint8_t u = S.uFinal[p];
        const uint32_t m = (u & 2) ? R.m1 : R.m0;
        for (uint32_t rest = m; rest; rest &= rest - 1u)
            S.wA[pw_slot(S, nxt, __ffs(rest) - 1, p)].w = desc | (col << 16);
        const uint32_t ra = S.repAfter[p];
        if (ra != kPwNone)
            pw_store(S, pw_slot(S, nxt, S.L - 1, p), {S.rec[ra].incr, t, t, S.descT[ra], D.frame[ra]});
        // illumination mask at the end of the frame (:686-690, :889-890): the right neighbour's
        // update sets 1 & ROI; else the own update leaves 2-1 = 1; else the start value (1 & ROI
        // after the left neighbour's update) minus one
        const int roiBit = D.roi[p] & 1;
        const int uRight = (x + 1 < D.W && D.roi[p + 1]) ? (S.uFinal[p + 1] & 1) : 0;
        const int mStart = (x > 0 && D.roi[p - 1] && (S.uFinal[p - 1] & 1)) ? roiBit : (int)S.illum[p];
        int mEnd;
        if (uRight) mEnd = roiBit;
        else if (u & 1) mEnd = 1;
        else mEnd = mStart > 0 ? mStart - 1 : 0;
        S.illum[p] = (uint8_t)mEnd;
        // feedback
        float fLT, fST;
        pw_factors(t, (int)S.nmv, &fLT, &fST);
        const float* fc = D.fm + (size_t)cur * kNumFloatMaps * D.npx;
        float* fn = D.fm + (size_t)nxt * kNumFloatMaps * D.npx;
        const int npx = D.npx;
        float dLT = fc[FM_DMIN_LT * npx + p], dST = fc[FM_DMIN_ST * npx + p];
        float rLT = fc[FM_RAW_LT * npx + p], rST = fc[FM_RAW_ST * npx + p];
        const float nmc = (float)R.minColor / 255.0f, nmd = (float)R.minDesc / 16.0f;
        const float nd0 = (nmc < nmd) ? nmd : nmc;  // std::max
        if (R.flags & kRfBG) {
            dLT = dLT * (1.0f - fLT) + nd0 * fLT;
            dST = dST * (1.0f - fST) + nd0 * fST;
            rLT = rLT * (1.0f - fLT);
            rST = rST * (1.0f - fST);
        } else {
            const float q = (R.thrW - R.sumW) / R.thrW;
            const float nd = (nd0 < q) ? q : nd0;
            dLT = dLT * (1.0f - fLT) + nd * fLT;
            dST = dST * (1.0f - fST) + nd * fST;
            rLT = rLT * (1.0f - fLT) + fLT;
            rST = rST * (1.0f - fST) + fST;
        }
        float Rr = fc[FM_R * npx + p], V = fc[FM_V * npx + p], T = fc[FM_T * npx + p];
        const float finLT = fc[FM_FIN_LT * npx + p], finST = fc[FM_FIN_ST * npx + p];
        S.unstable[p] = (Rr > kUnstR || (rLT - finLT) > kUnstRatio || (rST - finST) > kUnstRatio) ? 1 : 0;
        const uint32_t lastFG = D.lastFG[p];
        const float dmin = (dST < dLT) ? dST : dLT, dmax = (dLT < dST) ? dST : dLT;
        if (lastFG || (dmin < kUnstRatio && O.segm)) {
            const float a = T + kTIncr / (dmax * V);
            T = (kTUpper < a) ? kTUpper : a;
        } else {
            const float a = T - kTDecr * V / dmax;
            T = (a < kTLower) ? kTLower : a;
        }
        if (dmax > kUnstRatio && D.blinks[p]) {
            V += boot ? kVIncr * 2 : kVIncr;
        } else {
            const float a = V - kVDecr * ((boot || flat) ? 2.0f : lastFG ? 0.5f : 1.0f);
            V = (a < kVDecr) ? kVDecr : a;
        }
        // R < std::pow(1+2*dmin, 2) in double: exact via the split x*x = hi + lo
        const float xb = 1.0f + dmin * 2.0f;
        const float hi = xb * xb, lo = __fmaf_rn(xb, xb, -hi);
        if (Rr < hi || (Rr == hi && lo > 0.0f)) {
            Rr += kRVar * (V - kVDecr);
        } else {
            const float a = Rr - kRVar / V;
            Rr = (a < 1.0f) ? 1.0f : a;
        }
        fn[FM_R * npx + p] = Rr;
        fn[FM_V * npx + p] = V;
        fn[FM_T * npx + p] = T;
        fn[FM_DMIN_LT * npx + p] = dLT;
        fn[FM_DMIN_ST * npx + p] = dST;
        fn[FM_RAW_LT * npx + p] = rLT;
        fn[FM_RAW_ST * npx + p] = rST;
        D.lastCol[p] = (uint8_t)col;
        D.lastDesc[p] = (uint16_t)desc;
        D.intent[p] = O.segm ? (kInValid | kInFG) : kInValid;
        D.kctr[p] = O.q != kPwNone ? O.kEnd : O.kLoop;  // the draw count after the pixel's updates
    } else if (in) {
        D.intent[p] = 0u;
    }
    const unsigned b = __ballot_sync(0xffffffffu, act && flat);
    if ((threadIdx.x & 31) == 0 && b) atomicAdd(&S.pc->nflat_acc, (unsigned long long)__popc(b));
}

// global word weights (:789-790): ordered float sums of the frame's contributions, one block per
// (stream, word) over the word's compacted list; the replaceable word restarts from zero at the
// frame's last replacement (its list holds only the contributions after it)
extern "C" __global__ void __launch_bounds__(256) pw_k_weights(PwParams P) {
    PW_TAIL_GATE(P);
    const int si = blockIdx.x / kPwMaxGlobal, w = blockIdx.x % kPwMaxGlobal;
    if (si >= P.nStreams) return;
    const PawcsDev& S = P.streams[si];
    if (w >= S.G) return;
    PawcsCtl* pc = S.pc;
    const int wr = pc->gdict[S.G - 1];
    const uint32_t nrep = pc->n_repl;
    const bool isWr = w == wr;
    const uint32_t n = S.catInfo[w], base = S.catInfo[kPwCatBase + w];
    __shared__ float buf[1024];
    float acc = (isWr && nrep > 0) ? 0.0f : pc->gw_weight[w];
    for (uint32_t c0 = 0; c0 < n; c0 += 1024) {
        const uint32_t cnt = min(1024u, n - c0);
        for (uint32_t i = threadIdx.x; i < cnt; i += blockDim.x) buf[i] = S.contribList[base + c0 + i];
        __syncthreads();
        if (threadIdx.x == 0)
            for (uint32_t i = 0; i < cnt; ++i) acc = acc + buf[i];
        __syncthreads();
    }
    if (threadIdx.x == 0) {
        pc->gw_weight[w] = acc;
        if (isWr && nrep > 0) {
            pc->gw_color[w] = pc->wr_color;
            pc->gw_desc[w] = pc->wr_desc;
            pc->gw_desc2[w] = pc->wr_desc2;
            pc->gw_bits[w] = pc->wr_bits;
        }
    }
}

// ------------------------------------------------------------------------------------------
// end-of-frame global words (:1300-1334)
// ------------------------------------------------------------------------------------------
// per word: every 256/512 frames the weight becomes the map sum (double, raster order); every
// 8/16 frames the map decays where the previous dilated mask was background, then a 3x3 blur
__device__ __forceinline__ void pw_gw_rates(uint32_t t, int* recalc, int* update) {
    const uint32_t rate = t <= (uint32_t)kBootWin ? 8u : 16u;
    *recalc = (t % (rate << 5)) == 0u;
    *update = (t % rate) == 0u;
}

extern "C" __global__ void pw_k_gw_recalc(PwParams P) {
    PW_TAIL_GATE(P);
    const int si = blockIdx.x / kPwMaxGlobal, w = blockIdx.x % kPwMaxGlobal;
    if (si >= P.nStreams) return;
    const PawcsDev& S = P.streams[si];
    if (w >= S.G) return;
    PawcsCtl* pc = S.pc;
    int recalc, update;
    pw_gw_rates((uint32_t)(S.sd.ctl->frame_idx + 1ull), &recalc, &update);
    if (!recalc || !(pc->gw_weight[w] > 0.0f)) return;
    const size_t n = (size_t)S.gwW * S.gwH;
    float* m = S.gmap + (size_t)w * n;
    __shared__ float wsum;
    if (threadIdx.x == 0) {
        double s = 0.0;
        for (size_t i = 0; i < n; ++i) s += (double)m[i];
        wsum = (float)s;
        pc->gw_weight[w] = wsum < 1.0f ? 0.0f : wsum;
    }
    __syncthreads();
    if (wsum < 1.0f)
        for (size_t i = threadIdx.x; i < n; i += blockDim.x) m[i] = 0.0f;
}

// decay (accumulateProduct with the INTER_NEAREST down-scaled previous inverted dilated mask) and the
// first half of the blur (row sums, double); one block row per map row
extern "C" __global__ void pw_k_gw_decay(PwParams P, double* rowsum) {
    PW_TAIL_GATE(P);
    const int si = blockIdx.y / kPwMaxGlobal, w = blockIdx.y % kPwMaxGlobal;
    if (si >= P.nStreams) return;
    const PawcsDev& S = P.streams[si];
    if (w >= S.G) return;
    int recalc, update;
    pw_gw_rates((uint32_t)(S.sd.ctl->frame_idx + 1ull), &recalc, &update);
    if (!update || !(S.pc->gw_weight[w] > 0.0f)) return;
    const int gw = S.gwW, gh = S.gwH, W = S.sd.W, H = S.sd.H;
    const size_t n = (size_t)gw * gh;
    float* m = S.gmap + (size_t)w * n;
    double* rs = rowsum + ((size_t)si * kPwMaxGlobal + w) * n;
    const double ifx = 1.0 / ((double)gw / W), ify = 1.0 / ((double)gh / H);
    for (int yy = blockIdx.x; yy < gh; yy += gridDim.x) {
        int sy = (int)floor(yy * ify);
        sy = sy < H - 1 ? sy : H - 1;
        for (int xx = threadIdx.x; xx < gw; xx += blockDim.x) {
            int sx = (int)floor(xx * ifx);
            sx = sx < W - 1 ? sx : W - 1;
            const size_t i = (size_t)yy * gw + xx;
            if (S.sd.dilInv[(size_t)sy * W + sx]) {
                const float prod = m[i] * -0.1f;
                m[i] = m[i] + prod;
            }
        }
        __syncthreads();
        for (int xx = threadIdx.x; xx < gw; xx += blockDim.x) {
            const int x0 = xx > 0 ? xx - 1 : 0, x1 = xx < gw - 1 ? xx + 1 : gw - 1;
            const size_t r = (size_t)yy * gw;
            rs[r + xx] = ((double)m[r + x0] + (double)m[r + xx]) + (double)m[r + x1];
        }
    }
}

// second half of the blur (column sums * 1/9, to float), the weight decay and, in the last block,
// the one-pass dictionary sort by weight
extern "C" __global__ void pw_k_gw_blur(PwParams P, const double* rowsum) {
    PW_TAIL_GATE(P);
    const int si = blockIdx.y / kPwMaxGlobal, w = blockIdx.y % kPwMaxGlobal;
    if (si >= P.nStreams) return;
    const PawcsDev& S = P.streams[si];
    if (w >= S.G) return;
    int recalc, update;
    pw_gw_rates((uint32_t)(S.sd.ctl->frame_idx + 1ull), &recalc, &update);
    if (!update || !(S.pc->gw_weight[w] > 0.0f)) return;
    const int gw = S.gwW, gh = S.gwH;
    const size_t n = (size_t)gw * gh;
    float* m = S.gmap + (size_t)w * n;
    const double* rs = rowsum + ((size_t)si * kPwMaxGlobal + w) * n;
    for (int yy = blockIdx.x; yy < gh; yy += gridDim.x) {
        const int y0 = yy > 0 ? yy - 1 : 0, y1 = yy < gh - 1 ? yy + 1 : gh - 1;
        for (int xx = threadIdx.x; xx < gw; xx += blockDim.x) {
            const double tsum = (rs[(size_t)y0 * gw + xx] + rs[(size_t)yy * gw + xx]) + rs[(size_t)y1 * gw + xx];
            m[(size_t)yy * gw + xx] = (float)(tsum * (1.0 / 9.0));
        }
    }
}

// weight decay and the dictionary's bubble step (after all maps are final)
extern "C" __global__ void pw_k_gw_sort(PwParams P) {
    PW_TAIL_GATE(P);
    const int si = blockIdx.x * blockDim.x + threadIdx.x;
    if (si >= P.nStreams) return;
    const PawcsDev& S = P.streams[si];
    PawcsCtl* pc = S.pc;
    int recalc, update;
    pw_gw_rates((uint32_t)(S.sd.ctl->frame_idx + 1ull), &recalc, &update);
    for (int g = 0; g < S.G; ++g) {
        const int w = pc->gdict[g];
        if (update && pc->gw_weight[w] > 0.0f) pc->gw_weight[w] *= 0.9f;
        if (g > 0 && pc->gw_weight[pc->gdict[g]] > pc->gw_weight[pc->gdict[g - 1]]) {
            const int tmp = pc->gdict[g];
            pc->gdict[g] = pc->gdict[g - 1];
            pc->gdict[g - 1] = tmp;
        }
    }
}

// per-pixel global word order: one bubble pass on the local map weights (:1318-1330, :415-427);
// mode 0: only on update frames (apply), 1: always (refreshModel), 2: when an automatic reset is pending
extern "C" __global__ void __launch_bounds__(256) pw_k_lut_sort(PwParams P, int mode) {
    PW_TAIL_GATE(P);
    const int t0 = blockIdx.x;
    if (t0 >= P.totalTiles) return;
    const PawcsDev& S = P.streams[pw_stream_by_tile(P, t0)];
    const StreamDev& D = S.sd;
    if (mode == 0) {
        int recalc, update;
        pw_gw_rates((uint32_t)(D.ctl->frame_idx + 1ull), &recalc, &update);
        if (!update) return;
    } else if (mode == 2 && S.pc->reset_pending == 0) {
        return;
    }
    const int lt = t0 - D.tileBase;
    const int x = (lt % D.tilesX) * kTileW + (int)threadIdx.x % kTileW;
    const int y = (lt / D.tilesX) * kTileH + (int)threadIdx.x / kTileW;
    if (x >= D.W || y >= D.H) return;
    const int p = y * D.W + x;
    if (!D.roi[p]) return;
    const size_t n = (size_t)S.gwW * S.gwH;
    const size_t cidx = (size_t)(y / 2) * S.gwW + (x / 2);
    uint8_t* lut = S.glut + (size_t)p * kPwGlutStride;
    uint8_t o[kPwMaxGlobal];
    for (int g = 0; g < S.G; ++g) o[g] = lut[g];
    float last = S.gmap[(size_t)o[0] * n + cidx];
    for (int g = 1; g < S.G; ++g) {
        const float c = S.gmap[(size_t)o[g] * n + cidx];
        if (c > last) {
            const uint8_t tmp = o[g];
            o[g] = o[g - 1];
            o[g - 1] = tmp;
        } else {
            last = c;
        }
    }
    for (int g = 0; g < S.G; ++g) lut[g] = o[g];
}

// blinks (:1443-1446) and the 3x3 closing of the raw mask (:1447)
extern "C" __global__ void __launch_bounds__(256) pw_k_blink_close(PwParams P) {
    PW_TAIL_GATE(P);
    const int t0 = blockIdx.x;
    if (t0 >= P.totalTiles) return;
    const PawcsDev& S = P.streams[pw_stream_by_tile(P, t0)];
    const StreamDev& D = S.sd;
    const int lt = t0 - D.tileBase;
    const int x0 = (lt % D.tilesX) * kTileW, y0 = (lt / D.tilesX) * kTileH;
    constexpr int IW = kTileW + 4, IH = kTileH + 4, DW = kTileW + 2, DH = kTileH + 2;
    __shared__ uint8_t raw[IW * IH];
    __shared__ uint8_t dil[DW * DH];
    const int W = D.W, H = D.H;
    for (int i = threadIdx.x; i < IW * IH; i += blockDim.x) {
        const int gy = y0 - 2 + i / IW, gx = x0 - 2 + i % IW;
        raw[i] = (gy >= 0 && gy < H && gx >= 0 && gx < W && (D.intent[gy * W + gx] & kInFG)) ? 255 : 0;
    }
    __syncthreads();
    // dilation over the clipped 3x3 window (out-of-image pixels never win)
    for (int i = threadIdx.x; i < DW * DH; i += blockDim.x) {
        const int ry = i / DW, rx = i % DW;
        uint8_t v = 0;
        for (int dy = 0; dy < 3; ++dy)
            for (int dx = 0; dx < 3; ++dx) v |= raw[(ry + dy) * IW + rx + dx];
        dil[i] = v;
    }
    __syncthreads();
    const int lx = threadIdx.x % kTileW, ly = threadIdx.x / kTileW;
    const int x = x0 + lx, y = y0 + ly;
    bool rawBit = false, closedBit = false;
    if (x < W && y < H) {
        const int q = y * W + x;
        const uint8_t r = raw[(ly + 2) * IW + lx + 2];
        const uint8_t cb = r ^ D.lastRawFG[q];
        D.blinks[q] = cb | D.lastRawBlink[q];
        D.lastRawBlink[q] = cb;
        D.lastRawFG[q] = r;
        // erosion of the dilated mask over the clipped window
        uint8_t v = 255;
        for (int dy = -1; dy <= 1; ++dy)
            for (int dx = -1; dx <= 1; ++dx) {
                const int gx = x + dx, gy = y + dy;
                if (gx < 0 || gx >= W || gy < 0 || gy >= H) continue;
                v &= dil[(ly + 1 + dy) * DW + lx + 1 + dx];
            }
        rawBit = r != 0;
        closedBit = v != 0;
    }
    // each warp is one 32-pixel tile row: its ballots are the row's words of the raw and closed masks
    const unsigned rawW = __ballot_sync(0xffffffffu, rawBit), closedW = __ballot_sync(0xffffffffu, closedBit);
    if (lx == 0 && y < H) {
        const size_t o = (size_t)y * D.rowWords + x0 / 32;
        bit_plane(D, BP_RAW)[o] = rawW;
        bit_plane(D, BP_CLOSED)[o] = closedW;
    }
    // the nodes of the hole filling: the run starts of the row's 0-pixels (a word's first pixel counts)
    if (x < W && y < H && ((~closedW & ~(~closedW << 1)) >> lx) & 1u) D.label[y * W + x] = y * W + x;
}

// down-sampled frame (INTER_AREA, integral scale), its rolling averages (accumulateWeighted) and the
// per-pixel |LT - ST| of the motion analysis (:1475-1478); one thread per down-sampled pixel
extern "C" __global__ void pw_k_ds(PwParams P) {
    PW_TAIL_GATE(P);
    const PawcsDev& S = P.streams[0];
    const StreamDev& D = S.sd;
    const int nds = D.dsW * D.dsH;
    const int i = (blockIdx.x * blockDim.x + threadIdx.x) >> 3;  // eight lanes per output
    if (i >= nds) return;
    uint32_t v[1];
    area_resample_group<1>(D.frame, D.W, D.H, D.dsW, D.dsH, i % D.dsW, i / D.dsW, v);
    if (threadIdx.x & 7) return;
    const uint32_t t = (uint32_t)(D.ctl->frame_idx + 1ull);
    float fLT, fST;
    pw_factors(t, (int)S.nmv, &fLT, &fST);
    const uint8_t vb = (uint8_t)v[0];
    const float lt = (float)vb * fLT + D.dsLT[i] * (1.0f - fLT);
    const float st = (float)vb * fST + D.dsST[i] * (1.0f - fST);
    D.dsLT[i] = lt;
    D.dsST[i] = st;
    S.dsFrame[i] = vb;
    S.dsAbs[i] = S.dsRoi[i] ? fabsf(lt - st) : 0.0f;
}

// ------------------------------------------------------------------------------------------
// frame level (:1462-1516): LBSP threshold LUT, camera-motion analysis, automatic model reset
// decision; one block per stream
// ------------------------------------------------------------------------------------------
// acc + v[0] + v[1] + ... in that order, from shared memory at a 16-byte boundary. The chain of additions is
// the bound (four cycles each); four vector loads are in flight ahead of it.
__device__ float pw_ordered_sum(const float* v, int n, float acc) {
    const float4* q = (const float4*)v;
    int i = 0;
    for (; i + 16 <= n; i += 16) {
        const float4 a = q[i / 4], b = q[i / 4 + 1], c = q[i / 4 + 2], d = q[i / 4 + 3];
        acc = acc + a.x; acc = acc + a.y; acc = acc + a.z; acc = acc + a.w;
        acc = acc + b.x; acc = acc + b.y; acc = acc + b.z; acc = acc + b.w;
        acc = acc + c.x; acc = acc + c.y; acc = acc + c.z; acc = acc + c.w;
        acc = acc + d.x; acc = acc + d.y; acc = acc + d.z; acc = acc + d.w;
    }
    for (; i < n; ++i) acc = acc + v[i];
    return acc;
}

// the ordered sum of n floats by the block: the block stages the terms in shared memory, one thread (of the
// warp `warp`) adds them in order; the sum is valid on that thread
__device__ float pw_block_ordered_sum(const float* v, int n, float* terms, int warp) {
    float acc = 0.0f;
    for (int c0 = 0; c0 < n; c0 += 2048) {
        const int cnt = min(2048, n - c0);
        for (int i = threadIdx.x; i < cnt; i += blockDim.x) terms[i] = v[c0 + i];
        __syncthreads();
        if (threadIdx.x == 32 * warp) acc = pw_ordered_sum(terms, cnt, acc);
        __syncthreads();
    }
    return acc;
}

// reset decision of the frame-level block (:1509-1513)
__device__ void pw_reset_decide(const PawcsDev& S) {
    StreamCtl* ctl = S.sd.ctl;
    PawcsCtl* pc = S.pc;
    const uint32_t t = (uint32_t)(ctl->frame_idx + 1ull);
    const int boot = t <= (uint32_t)kBootWin;
    const float ratio = pc->frame_ratio;
    if (pc->reset_block) {
        if (ctl->frames_since_reset > (unsigned long long)kBootWin * 2) {
            ctl->auto_reset = 0;
        } else if (ratio >= 45.0f && ctl->cooldown == 0) {
            ctl->frames_since_reset = 0;
            pc->reset_pending = 1;
        } else if (!boot) {
            ++ctl->frames_since_reset;
        }
    }
}

// the frame level; decide: the reset decision too (frames without a camera-motion comparison before it)
extern "C" __global__ void __launch_bounds__(256) pw_k_epilogue(PwParams P, int decide) {
    PW_TAIL_GATE(P);
    const int si = blockIdx.x;
    if (si >= P.nStreams) return;
    const PawcsDev& S = P.streams[si];
    const StreamDev& D = S.sd;
    StreamCtl* ctl = D.ctl;
    PawcsCtl* pc = S.pc;
    // LBSP threshold LUT (:1462-1473), an entry per thread
    const float nonflat = (float)(ctl->n_rel - pc->nflat_acc) / (float)ctl->n_rel;
    const float lastNonflat = pc->last_nonflat_ratio;
    const float rel = S.relThr;
    const float offs = (float)S.lbspOff;
    const int k = threadIdx.x;
    if (nonflat < 0.1f && lastNonflat < 0.1f) {
        const float v = (offs + (float)k * rel) / 4;
        const int r = __float2int_rn(v);
        const int lim = r < 0 ? 0 : r > 255 ? 255 : r;
        if ((int)ctl->lut[k] > lim) --ctl->lut[k];
    } else if (nonflat > 0.5f && lastNonflat > 0.5f) {
        const float v = offs + 255 * rel;
        const int r = __float2int_rn(v);
        const int lim = r < 0 ? 0 : r > 255 ? 255 : r;
        if ((int)ctl->lut[k] < lim) ++ctl->lut[k];
    }
    // ordered float sum of |LT - ST| over the down-sampled ROI (lv::L1dist, math.hpp:255-268)
    __shared__ __align__(16) float terms[2048];
    const float l1 = pw_block_ordered_sum(S.dsAbs, D.dsW * D.dsH, terms, 0);
    __syncthreads();  // every thread has read the ratios
    if (threadIdx.x != 0) return;
    const float ratio = l1 / (float)pc->ds_roi_count;
    pc->frame_ratio = ratio;
    pc->last_nonflat_ratio = nonflat;
    pc->nflat_acc = 0;
    pc->reset_pending = 0;
    // automatic model reset (:1479-1513): the block is entered when the reset is enabled or the camera
    // moves; the camera-motion comparison of frames 500, 1000, ... (pw_k_motion_*) and the reset decision
    // (pw_reset_decide) follow
    if (!ctl->auto_reset && ratio >= 45.0f * 2) ctl->auto_reset = 1;
    pc->reset_block = ctl->auto_reset || pc->moving_cam;
    if (decide) pw_reset_decide(S);
}

// closes the frame: frame index, cooldown, factors of the next frame's final-segmentation averages
// and, for the host, the error flags. resetDone 0: a pending automatic reset leaves the frame open, and the host
// runs it and closes the frame after it.
extern "C" __global__ void pw_k_close(PwParams P, int resetDone) {
    PW_TAIL_GATE(P);
    const int si = blockIdx.x * blockDim.x + threadIdx.x;
    if (si >= P.nStreams) return;
    const PawcsDev& S = P.streams[si];
    StreamCtl* ctl = S.sd.ctl;
    PawcsCtl* pc = S.pc;
    if (!resetDone && pc->reset_pending) {
        P.hflags[PWF_RESET] = 1u;
        return;
    }
    P.hflags[PWF_STATUS] = *(const volatile unsigned int*)P.err;
    P.hflags[PWF_CLOSED] = 1u;
    const uint32_t t = (uint32_t)(ctl->frame_idx + 1ull);
    if (pc->reset_pending == 1) {
        float fLT, fST;
        pw_factors(t, (int)S.nmv, &fLT, &fST);
        const int boot = t <= (uint32_t)kBootWin;
        const unsigned long long nlt = boot ? (unsigned long long)(S.nmv / 2) : (unsigned long long)S.nmv;
        ctl->cooldown = nlt / 4;
    }
    if (ctl->cooldown > 0) --ctl->cooldown;
    ctl->frame_idx = t;
    // factors of the next frame (used by the median kernel's final-segmentation averages)
    float fLT, fST;
    pw_factors((unsigned long long)t + 1ull, (int)S.nmv, &fLT, &fST);
    ctl->fLT = fLT;
    ctl->fST = fST;
    ctl->bLT = (float)((1.0 / 255) * (double)fLT);
    ctl->bST = (float)((1.0 / 255) * (double)fST);
}

// ------------------------------------------------------------------------------------------
// refreshModel (:107-429), one channel
// ------------------------------------------------------------------------------------------
// local resampling: 98 draws from the 7x7 neighbourhood per pixel, then (initialization) the
// random fill of empty slots; one thread per pixel
extern "C" __global__ void __launch_bounds__(128) pw_k_refresh_local(PawcsDev S, uint32_t t, int buf, int baseOcc,
                                                                      float decr, int force, int onlyPending,
                                                                      int useDil) {
    pdl_entry();
    const int p = blockIdx.x * blockDim.x + threadIdx.x;
    const StreamDev& D = S.sd;
    if (p >= D.npx) return;
    if (onlyPending && S.pc->reset_pending == 0) return;
    if (!D.roi[p]) return;
    // m_oLastFGMask_dilated: the complement of the stored inverted mask (all clear at initialization)
    if (!(force || !useDil || D.dilInv[p] != 0)) return;
    const int L = S.L;
    const int x0 = p % D.W, y0 = p / D.W;
    const unsigned long long off = S.pc->lword_offset;
    const float* fm = D.fm + (size_t)buf * kNumFloatMaps * D.npx;
    const PwThr th = pw_thresholds(fm[FM_R * D.npx + p], S.unstable[p], S.minColor, S.descOff);
    uint8_t wc[kPwMaxLocal];
    uint16_t wd[kPwMaxLocal];
    uint32_t wo[kPwMaxLocal], wf[kPwMaxLocal], wl[kPwMaxLocal];
    for (int j = 0; j < L; ++j) {
        const PwWord w = pw_load(S, pw_slot(S, buf, j, p));
        wc[j] = (uint8_t)w.col;
        wd[j] = (uint16_t)w.desc;
        wo[j] = w.occ;
        wf[j] = w.first;
        wl[j] = w.last;
    }
    // empty slots carry first == kPwNone (initialization only)
    if (decr > 0.0f)
        for (int j = 0; j < L; ++j)
            if (wf[j] != kPwNone) wo[j] -= (uint32_t)(decr * (float)wo[j]);
    uint32_t k = D.kctr[p];
    for (int it = 0; it < 98; ++it) {
        const uint32_t r = pw_draw(D.seed, t, (uint32_t)p, k++);
        int rr = 1 + (int)(r % 512u), xx = 0, yy = 0;
        for (int c = 0; c < 49; ++c) {
            rr -= pw_pat7[c];
            if (rr <= 0) {
                xx = c % 7;
                yy = c / 7;
                break;
            }
        }
        int sx = x0 + xx - 3, sy = y0 + yy - 3;
        sx = sx < 2 ? 2 : sx >= D.W - 2 ? D.W - 3 : sx;
        sy = sy < 2 ? 2 : sy >= D.H - 2 ? D.H - 3 : sy;
        const int sp = sy * D.W + sx;
        if (!(force || !useDil || D.dilInv[sp] != 0)) continue;
        const uint32_t scol = D.lastCol[sp], sdesc = D.lastDesc[sp];
        int i;
        for (i = 0; i < L; ++i) {
            if (wf[i] == kPwNone) continue;
            if (pw_absdiff(scol, wc[i]) <= th.color && (uint32_t)__popc(sdesc ^ wd[i]) <= th.desc) {
                wo[i] += 1;
                wl[i] = t;
                break;
            }
        }
        if (i == L) {
            i = L - 1;
            wc[i] = (uint8_t)scol;
            wd[i] = (uint16_t)sdesc;
            wo[i] = (uint32_t)baseOcc;
            wf[i] = t;
            wl[i] = t;
        }
        while (i > 0 && (wf[i - 1] == kPwNone ||
                         pw_weight(wo[i], wf[i], wl[i], t, off) > pw_weight(wo[i - 1], wf[i - 1], wl[i - 1], t, off))) {
            uint8_t c8 = wc[i]; wc[i] = wc[i - 1]; wc[i - 1] = c8;
            uint16_t d16 = wd[i]; wd[i] = wd[i - 1]; wd[i - 1] = d16;
            uint32_t a = wo[i]; wo[i] = wo[i - 1]; wo[i - 1] = a;
            a = wf[i]; wf[i] = wf[i - 1]; wf[i - 1] = a;
            a = wl[i]; wl[i] = wl[i - 1]; wl[i - 1] = a;
            --i;
        }
    }
    for (int i = 1; i < L; ++i) {
        if (wf[i] != kPwNone) continue;
        const int ri = (int)(pw_draw(D.seed, t, (uint32_t)p, k++) % (uint32_t)i);
        const int offc = (int)(pw_draw(D.seed, t, (uint32_t)p, k++) % (th.color + 1u)) - (int)th.color / 2;
        const int v = (int)wc[ri] + offc;
        wc[i] = (uint8_t)(v < 0 ? 0 : v > 255 ? 255 : v);
        wd[i] = wd[ri];
        const uint32_t occ = (uint32_t)((float)wo[ri] * ((float)(L - i) / (float)L));
        wo[i] = occ > 1u ? occ : 1u;
        wf[i] = t;
        wl[i] = t;
    }
    for (int j = 0; j < L; ++j) pw_store(S, pw_slot(S, buf, j, p), {wo[j], wf[j], wl[j], wd[j], wc[j]});
    D.kctr[p] = (uint16_t)k;
}

// global resampling from equally spaced pixels (two passes) and the fill of empty dictionary
// slots; one thread per stream (it visits about 4 G pixels)
extern "C" __global__ void pw_k_refresh_global(PawcsDev S, uint32_t t, int buf, int force, int onlyPending,
                                               int useDil) {
    pdl_entry();
    if (threadIdx.x != 0 || blockIdx.x != 0) return;
    PawcsCtl* pc = S.pc;
    if (onlyPending && pc->reset_pending == 0) return;
    const StreamDev& D = S.sd;
    const int G = S.G, L = S.L;
    const size_t n = (size_t)S.gwW * S.gwH;
    const unsigned long long off = pc->lword_offset;
    const float* fm = D.fm + (size_t)buf * kNumFloatMaps * D.npx;
    size_t incr = (size_t)D.npx / (size_t)G > 1 ? (size_t)D.npx / (size_t)G : 1;
    for (int pass = 0; pass < 2; ++pass) {
        for (size_t p = 0; p < (size_t)D.npx; p += incr) {
            if (!D.roi[p]) continue;
            if (!(force || !useDil || D.dilInv[p] != 0)) continue;
            const int x = (int)(p % D.W), y = (int)(p / D.W);
            const size_t cidx = (size_t)(y / 2) * S.gwW + (x / 2);
            const PwThr th = pw_thresholds(fm[FM_R * D.npx + p], S.unstable[p], S.minColor, S.descOff);
            const PwWord best = pw_load(S, pw_slot(S, buf, 0, (int)p));
            const uint32_t bc = best.col, bd = best.desc;
            const float bw = pw_weight(best.occ, best.first, best.last, t, off);
            const uint32_t bb = __popc(bd);
            int uninit = 0, g;
            for (g = 0; g < G; ++g) {
                const int w = pc->gdict[g];
                if (w < 0) {
                    uninit = 1;
                    continue;
                }
                if (pw_absdiff(pc->gw_color[w], bc) <= th.color && pw_absdiff(bb, pc->gw_bits[w]) <= th.desc / 4u) break;
            }
            if (g == G) {
                g = G - 1;
                const int w = uninit ? pc->gnext++ : pc->gdict[g];
                pc->gw_color[w] = bc;
                pc->gw_desc[w] = bd;
                pc->gw_bits[w] = bb;
                for (size_t i = 0; i < n; ++i) S.gmap[(size_t)w * n + i] = 0.0f;
                pc->gw_weight[w] = 0.0f;
                pc->gdict[g] = w;
            }
            const int w = pc->gdict[g];
            float* lw = S.gmap + (size_t)w * n + cidx;
            if (*lw < bw) {
                pc->gw_weight[w] = pc->gw_weight[w] + bw;
                *lw = *lw + bw;
            }
            while (g > 0 && (pc->gdict[g - 1] < 0 || pc->gw_weight[pc->gdict[g]] > pc->gw_weight[pc->gdict[g - 1]])) {
                const int tmp = pc->gdict[g];
                pc->gdict[g] = pc->gdict[g - 1];
                pc->gdict[g - 1] = tmp;
                --g;
            }
        }
        incr = incr / 3 > 1 ? incr / 3 : 1;
    }
    for (int g = 0; g < G; ++g) {
        if (pc->gdict[g] >= 0) continue;
        const int w = pc->gnext++;
        pc->gw_color[w] = 0;
        pc->gw_desc[w] = 0;
        pc->gw_bits[w] = 0;
        for (size_t i = 0; i < n; ++i) S.gmap[(size_t)w * n + i] = 0.0f;
        pc->gw_weight[w] = 0.0f;
        pc->gdict[g] = w;
    }
    (void)L;
}

// the automatic reset's T(x) := 1 (:1508)
extern "C" __global__ void pw_k_reset_T(PawcsDev S, int buf) {
    pdl_entry();
    if (S.pc->reset_pending == 0) return;
    const StreamDev& D = S.sd;
    float* T = D.fm + (size_t)buf * kNumFloatMaps * D.npx + FM_T * D.npx;
    for (int p = blockIdx.x * blockDim.x + threadIdx.x; p < D.npx; p += gridDim.x * blockDim.x) T[p] = 1.0f;
}

// initial state of a stream's maps (:472-520) and dictionaries
extern "C" __global__ void pw_k_init(PawcsDev S) {
    const StreamDev& D = S.sd;
    for (int p = blockIdx.x * blockDim.x + threadIdx.x; p < D.npx; p += gridDim.x * blockDim.x) {
        for (int b = 0; b < 2; ++b) {
            float* f = D.fm + (size_t)b * kNumFloatMaps * D.npx;
            for (int m = 0; m < kNumFloatMaps; ++m) f[m * D.npx + p] = 0.0f;
            f[FM_T * D.npx + p] = kTLower;
            f[FM_R * D.npx + p] = 2.0f;
            f[FM_V * D.npx + p] = kVIncr * 10;
            for (int j = 0; j < S.L; ++j) pw_store(S, pw_slot(S, b, j, p), {0u, kPwNone, 0u, 0u, 0u});
        }
        S.illum[p] = 0;
        S.unstable[p] = 0;
        D.blinks[p] = 0;
        D.lastRawFG[p] = 0;
        D.lastFG[p] = 0;
        D.dilInv[p] = 0;
        D.lastRawBlink[p] = 0;
        D.kctr[p] = 0;
        for (int g = 0; g < kPwGlutStride; ++g) S.glut[(size_t)p * kPwGlutStride + g] = (uint8_t)g;
    }
}

// last colour and LBSP descriptor of the initialization frame (BackgroundSubtractionUtils.cpp:115-150,
// BackgroundSubtractorLBSP.cpp:26-38: descriptors strictly inside the 2-pixel border)
extern "C" __global__ void pw_k_init_last(PawcsDev S, const uint8_t* img) {
    const StreamDev& D = S.sd;
    for (int p = blockIdx.x * blockDim.x + threadIdx.x; p < D.npx; p += gridDim.x * blockDim.x) {
        const int x = p % D.W, y = p / D.W;
        uint8_t c = 0;
        uint16_t d = 0;
        if (D.roi[p]) {
            c = img[p];
            if (x > 2 && y > 2 && x < D.W - 2 && y < D.H - 2) {
                uint32_t taps[4];
                pw_taps<1>(img, D.W, x, y, 0, taps);
                d = (uint16_t)lbsp_thr(taps, c, D.ctl->lut[c]);
            }
        }
        D.lastCol[p] = c;
        D.lastDesc[p] = d;
    }
}

// camera-motion comparison (:1480-1501), frames t with t % 500 == 0: the background image (left in the label
// buffer by the background kernel), area-down-sampled like the frame, against the long-term mean of the
// down-sampled frames: |LT - BG| per down-sampled pixel (0 outside the fully covered blocks)
extern "C" __global__ void pw_k_motion_bg(PwParams P) {
    PW_TAIL_GATE(P);
    const PawcsDev& S = P.streams[0];
    const StreamDev& D = S.sd;
    const int nds = D.dsW * D.dsH;
    const int i = (blockIdx.x * blockDim.x + threadIdx.x) >> 3;  // eight lanes per output
    if (i >= nds) return;
    if (S.dsRoi[i] != 255) {
        S.dsAbs[i] = 0.0f;
        return;
    }
    uint32_t v[1];
    area_resample_group<1>((const uint8_t*)D.label, D.W, D.H, D.dsW, D.dsH, i % D.dsW, i / D.dsW, v);
    if (threadIdx.x & 7) return;
    S.dsAbs[i] = fabsf(D.dsLT[i] - (float)v[0]);
}

// camera-motion decision: ordered L1 sum, then switch the mode on (during the bootstrap window, ratio
// >= 45) or off (ratio < 45/4) with the local word weight offset (5 / 1000); PWF_MOTION tells the
// host to run refreshModel(1, 1, true), PWF_OFFSET carries the new offset. One grayscale channel: the colour
// distance ratio is 0; three channels: the mean colour distortion of pw3_k_motion_bg.
extern "C" __global__ void __launch_bounds__(256) pw_k_motion_decide(PwParams P) {
    PW_TAIL_GATE(P);
    const PawcsDev& S = P.streams[0];
    const StreamDev& D = S.sd;
    PawcsCtl* pc = S.pc;
    __shared__ __align__(16) float terms[2048];
    float l1 = 0.0f, cs = 0.0f;
    if (pc->reset_block) {
        const int nds = D.dsW * D.dsH;
        l1 = pw_block_ordered_sum(S.dsAbs, nds, terms, 0);
        // three channels: the ordered sum of the colour distortions (written beside the L1 terms)
        if (D.C == 3) cs = pw_block_ordered_sum(S.contrib, nds, terms, 0);
    }
    __syncthreads();  // reset_block has been read
    if (threadIdx.x != 0) return;
    pc->motion_pending = 0;
    if (pc->reset_block) {
        const uint32_t t = (uint32_t)(D.ctl->frame_idx + 1ull);
        const int boot = t <= (uint32_t)kBootWin;
        const float mr = l1 / (float)pc->ds_roi_count;
        const float cr = D.C == 3 ? cs / (float)pc->ds_roi_count : 0.0f;
        if (pc->moving_cam && mr < (float)(45 / 4) && cr < (float)(45 / 10 / 4)) {
            pc->lword_offset = (unsigned long long)kBootWin * 2;
            pc->moving_cam = 0;
            pc->motion_pending = 1;
        } else if (boot && !pc->moving_cam && (mr >= 45.0f || cr >= (float)(45 / 10))) {
            pc->lword_offset = 5;
            pc->moving_cam = 1;
            pc->motion_pending = 1;
        }
    }
    pw_reset_decide(S);
    P.hflags[PWF_OFFSET] = (unsigned int)pc->lword_offset;
    P.hflags[PWF_MOTION] = (unsigned int)pc->motion_pending;
}

// background image (:1518-1545) / descriptors (:1547-1594) from the words of buffer buf; ahead: 1 inside the
// frame step, before the frame index advances
extern "C" __global__ void pw_k_background(PawcsDev S, int buf, uint8_t* outCol, uint16_t* outDesc, int ahead) {
    const StreamDev& D = S.sd;
    const uint32_t t = (uint32_t)D.ctl->frame_idx + (uint32_t)ahead;
    const unsigned long long off = S.pc->lword_offset;
    for (int p = blockIdx.x * blockDim.x + threadIdx.x; p < D.npx; p += gridDim.x * blockDim.x) {
        if (!D.roi[p]) {
            if (outCol) outCol[p] = 0;
            if (outDesc) outDesc[p] = 0;
            continue;
        }
        float tw = 0.0f, tc = 0.0f, td = 0.0f;
        for (int j = 0; j < S.L; ++j) {
            const PwWord wj = pw_load(S, pw_slot(S, buf, j, p));
            const float w = pw_weight(wj.occ, wj.first, wj.last, t, off);
            tc = tc + (float)wj.col * w;
            td = td + (float)wj.desc * w;
            tw = tw + w;
        }
        if (outCol) {
            const int r = __float2int_rn(tc / tw);
            outCol[p] = (uint8_t)(r < 0 ? 0 : r > 255 ? 255 : r);
        }
        if (outDesc) {
            const int r = __float2int_rn(td / tw);
            outDesc[p] = (uint16_t)(r < 0 ? 0 : r > 65535 ? 65535 : r);
        }
    }
}

}  // namespace lvbgs
