// Change-detection evaluation on the device: the pixel classification counters of
// lv::BinClassif::accumulate (modules/datasets/src/metrics.cpp:21-61) and the metrics of
// lv::BinClassifMetrics (modules/datasets/include/litiv/datasets/metrics.hpp:203-256), so that a
// foreground mask already on the device is scored against ground truth without a host round trip.
//
// Ground-truth codes (CDnet, metrics.hpp:23-27): 255 positive, 0 negative, 85 out of scope,
// 170 unknown, 50 shadow. A pixel is "don't care" when its ground truth is out of scope or unknown,
// or when a ROI is given and is 0 there; otherwise it is TP / FP / FN / TN by the mask (255 =
// positive, anything else negative) and the ground truth (255 = positive, anything else negative),
// and additionally a shadow error when the ground truth is shadow and the mask positive.
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <mutex>

#include "../../include/lvbgs.h"
#include "lvbgs_internal.h"
#include "slots.h"
#include "staging.h"

namespace lvbgs {

enum { CL_TP = 0, CL_TN, CL_FP, CL_FN, CL_SE, CL_DC, CL_COUNT };

// the counters of the calls in flight, one place each (zero between calls), and their arrival counts
constexpr int kClassifSlots = 64;
__device__ unsigned long long g_classif[kClassifSlots][8];

// bytes of w that equal the byte b, as 0xff
__device__ __forceinline__ uint32_t bytes_eq(uint32_t w, uint32_t b) { return __vcmpeq4(w, b * 0x01010101u); }

// four pixels (bytes) of mask, ground truth and ROI into the counters; keep: 0xff for the bytes that count
__device__ __forceinline__ void classify4(uint32_t m, uint32_t g, uint32_t r, uint32_t keep, unsigned int (&c)[CL_COUNT]) {
    const uint32_t dc = (bytes_eq(g, 85) | bytes_eq(g, 170) | bytes_eq(r, 0)) & keep;
    const uint32_t in = keep & ~dc, mp = bytes_eq(m, 255), gp = bytes_eq(g, 255);
    c[CL_DC] += __popc(dc);
    c[CL_TP] += __popc(in & mp & gp);
    c[CL_FP] += __popc(in & mp & ~gp);
    c[CL_FN] += __popc(in & ~mp & gp);
    c[CL_TN] += __popc(in & ~mp & ~gp);
    c[CL_SE] += __popc(in & mp & bytes_eq(g, 50));
}

// Sixteen pixels per thread per step, compared four at a time as packed bytes (vec: all three images start at
// 16-byte boundaries; otherwise bytes are gathered). Per-warp and per-block sums, one 64-bit atomic per counter
// per block into the call's place; the block that finishes last writes the totals to page-locked memory and
// leaves the place zero for its next call. Bound by its 3 B/px and the launch: 1920x1080, 6.9 us a byte at a
// time before.
extern "C" __global__ void __launch_bounds__(256) lvbgs_k_classif(const uint8_t* __restrict__ mask,
                                                                  const uint8_t* __restrict__ gt,
                                                                  const uint8_t* __restrict__ roi, size_t n, int vec,
                                                                  int slot, unsigned long long* out) {
    unsigned int c[CL_COUNT] = {0, 0, 0, 0, 0, 0};  // in bits: eight per pixel
    const size_t stride = (size_t)gridDim.x * blockDim.x * 16;
    for (size_t i = ((size_t)blockIdx.x * blockDim.x + threadIdx.x) * 16; i < n; i += stride) {
        uint32_t m[4], g[4], r[4], keep[4];
        if (vec && i + 16 <= n) {
            const uint4 vm = __ldg((const uint4*)(mask + i)), vg = __ldg((const uint4*)(gt + i));
            const uint4 vr = roi ? __ldg((const uint4*)(roi + i)) : make_uint4(~0u, ~0u, ~0u, ~0u);
            m[0] = vm.x, m[1] = vm.y, m[2] = vm.z, m[3] = vm.w;
            g[0] = vg.x, g[1] = vg.y, g[2] = vg.z, g[3] = vg.w;
            r[0] = vr.x, r[1] = vr.y, r[2] = vr.z, r[3] = vr.w;
            keep[0] = keep[1] = keep[2] = keep[3] = ~0u;
        } else {
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                m[j] = g[j] = r[j] = keep[j] = 0u;
                for (int k = 0; k < 4; ++k) {
                    const size_t p = i + 4 * j + k;
                    if (p >= n) break;
                    m[j] |= (uint32_t)__ldg(mask + p) << (8 * k);
                    g[j] |= (uint32_t)__ldg(gt + p) << (8 * k);
                    r[j] |= (roi ? (uint32_t)__ldg(roi + p) : 255u) << (8 * k);
                    keep[j] |= 255u << (8 * k);
                }
            }
        }
#pragma unroll
        for (int j = 0; j < 4; ++j) classify4(m[j], g[j], r[j], keep[j], c);
    }
    __shared__ unsigned int s[CL_COUNT][8];
    __shared__ int sLast;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
    for (int j = 0; j < CL_COUNT; ++j) {
        const unsigned int v = __reduce_add_sync(0xffffffffu, c[j] >> 3);
        if (lane == 0) s[j][warp] = v;
    }
    __syncthreads();
    unsigned long long* acc = g_classif[slot];
    if (threadIdx.x < CL_COUNT) {
        unsigned long long t = 0;
        for (int w = 0; w < (int)(blockDim.x >> 5); ++w) t += s[threadIdx.x][w];
        if (t) atomicAdd(&acc[threadIdx.x], t);
        __threadfence();
    }
    __syncthreads();
    if (threadIdx.x == 0) sLast = atomicAdd(&acc[7], 1ull) == (unsigned long long)gridDim.x - 1ull;
    __syncthreads();
    if (!sLast) return;
    if (threadIdx.x < CL_COUNT) out[threadIdx.x] = atomicExch(&acc[threadIdx.x], 0ull);
    if (threadIdx.x == CL_COUNT) acc[7] = 0ull;
}

}  // namespace lvbgs

namespace {

bool on_device(const void* p) {
    cudaPointerAttributes a;
    if (cudaPointerGetAttributes(&a, p) != cudaSuccess) {
        cudaGetLastError();
        return false;
    }
    return a.type == cudaMemoryTypeDevice || a.type == cudaMemoryTypeManaged;
}

// The places of the calls in flight: an index into g_classif and a page-locked result of 64 bytes.
struct ClassifSlots {
    std::mutex mu;
    lvbgs::SlotPool pool{lvbgs::kClassifSlots};
    unsigned long long* host = nullptr;  // kClassifSlots * 8 words, page-locked, allocated once
    cudaError_t ready() {
        std::lock_guard<std::mutex> lk(mu);
        if (host) return cudaSuccess;
        const cudaError_t e = cudaHostAlloc((void**)&host, lvbgs::kClassifSlots * 64, cudaHostAllocPortable | cudaHostAllocMapped);
        if (e != cudaSuccess) host = nullptr;
        return e;
    }
};
constexpr unsigned long long kNoCounts = ~0ull;  // in a result that the kernel has not written
ClassifSlots& classif_slots() {
    static ClassifSlots s;
    return s;
}

}  // namespace

extern "C" lvbgs_status lvbgs_classif_accumulate(const uint8_t* fgmask, const uint8_t* gt, const uint8_t* roi,
                                                 int width, int height, uint64_t counts[6], int device_id,
                                                 void* cuda_stream) {
    using lvbgs::report_error;
    if (!fgmask || !counts || width <= 0 || height <= 0)
        return report_error(LVBGS_BAD_ARG, "classification: mask, counters and a non-empty size are required");
    const size_t n = (size_t)width * height;
    if (!gt) {
        // metrics.cpp:26-29: without ground truth every pixel is a "don't care"
        counts[lvbgs::CL_DC] += n;
        return LVBGS_OK;
    }
    if (cudaSetDevice(device_id) != cudaSuccess) {
        cudaGetLastError();
        return report_error(LVBGS_DEVICE_ERROR, "cannot select the CUDA device");
    }
    cudaStream_t st = (cudaStream_t)cuda_stream;
    cudaStreamCaptureStatus capture = cudaStreamCaptureStatusNone;
    if (cudaStreamIsCapturing(st, &capture) != cudaSuccess || capture != cudaStreamCaptureStatusNone) {
        cudaGetLastError();
        return report_error(LVBGS_DEVICE_ERROR, "classification waits for its result and cannot be captured");
    }
    // device inputs are read in place, host inputs copied to a stream-ordered staging buffer
    const uint8_t* src[3] = {fgmask, gt, roi};
    const uint8_t* dptr[3] = {nullptr, nullptr, nullptr};
    bool host[3];
    uint8_t* tmp = nullptr;
    const size_t padded = (n + 255) & ~(size_t)255;
    size_t need = 0;
    for (int i = 0; i < 3; ++i) {
        host[i] = src[i] && !on_device(src[i]);
        if (host[i]) need += padded;
    }
    cudaError_t e = cudaSuccess;
    if (need) e = lvbgs::staging_alloc(device_id, (void**)&tmp, need, st);
    size_t off = 0;
    for (int i = 0; i < 3 && e == cudaSuccess; ++i) {
        dptr[i] = src[i];
        if (!host[i]) continue;
        e = cudaMemcpyAsync(tmp + off, src[i], n, cudaMemcpyHostToDevice, st);
        dptr[i] = tmp + off;
        off += padded;
    }
    unsigned long long h[6] = {0, 0, 0, 0, 0, 0};
    if (e == cudaSuccess) e = classif_slots().ready();
    if (e == cudaSuccess) {
        lvbgs::SlotLease place(classif_slots().pool);
        if (place.slot() >= 0) {
            volatile unsigned long long* out = classif_slots().host + 8 * place.slot();
            out[0] = kNoCounts;
            int sms = 0;
            cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device_id);
            const int vec = (((uintptr_t)dptr[0] | (uintptr_t)dptr[1] | (uintptr_t)dptr[2]) & 15) == 0;
            const int blocks = (int)std::max<size_t>(1, std::min<size_t>((size_t)std::max(sms, 1) * 8, (n + 4095) / 4096));
            lvbgs::lvbgs_k_classif<<<blocks, 256, 0, st>>>(dptr[0], dptr[1], dptr[2], n, vec, place.slot(), (unsigned long long*)out);
            e = cudaGetLastError();
            if (tmp) cudaFreeAsync(tmp, st);
            tmp = nullptr;
            // waited for also after an error, which may be an older one: the kernel may be running. The place is given
            // back when the kernel has run to its end or was refused.
            const cudaError_t waited = cudaStreamSynchronize(st);
            const bool written = waited == cudaSuccess && out[0] != kNoCounts;
            if (written || (waited == cudaSuccess && e != cudaSuccess)) place.done();
            if (e == cudaSuccess) e = waited;
            if (e == cudaSuccess && !written) e = cudaErrorUnknown;
            if (e == cudaSuccess)
                for (int i = 0; i < 6; ++i) h[i] = out[i];
        } else {
            e = cudaErrorUnknown;
        }
    }
    if (tmp) cudaFreeAsync(tmp, st);
    if (e != cudaSuccess) {
        cudaGetLastError();
        return report_error(LVBGS_DEVICE_ERROR, cudaGetErrorString(e));
    }
    for (int i = 0; i < 6; ++i) counts[i] += h[i];
    return LVBGS_OK;
}

extern "C" lvbgs_status lvbgs_classif_metrics(const uint64_t counts[6], double out[8]) {
    if (!counts || !out) return lvbgs::report_error(LVBGS_BAD_ARG, "null argument");
    const double tp = (double)counts[0], tn = (double)counts[1], fp = (double)counts[2], fn = (double)counts[3];
    const uint64_t TP = counts[0], TN = counts[1], FP = counts[2], FN = counts[3];
    const uint64_t total = TP + TN + FP + FN;  // "don't care" excluded (metrics.hpp:46-48)
    const double recall = (TP + FN) > 0 ? tp / (double)(TP + FN) : 0.0;
    const double precision = (TP + FP) > 0 ? tp / (double)(TP + FP) : 0.0;
    out[0] = recall;
    out[1] = (TN + FP) > 0 ? tn / (double)(TN + FP) : 0.0;                   // specificity
    out[2] = (FP + TN) > 0 ? fp / (double)(FP + TN) : 0.0;                   // false positive rate
    out[3] = (TP + FN) > 0 ? fn / (double)(TP + FN) : 0.0;                   // false negative rate
    out[4] = total > 0 ? 100.0 * (double)(FN + FP) / (double)total : 0.0;    // percentage of bad classifications
    out[5] = precision;
    out[6] = (recall + precision) > 0 ? 2.0 * (recall * precision) / (recall + precision) : 0.0;  // F-measure
    // Matthews correlation coefficient: 0 when a marginal is empty
    const bool ok = (TP + FP) > 0 && (TP + FN) > 0 && (TN + FP) > 0 && (TN + FN) > 0;
    out[7] = ok ? ((tp * tn) - (double)(FP * FN)) / std::sqrt((tp + fp) * (double)(TP + FN) * (double)(TN + FP) *
                                                              (double)(TN + FN))
                : 0.0;
    return LVBGS_OK;
}
