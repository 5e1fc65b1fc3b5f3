// reconcile.cu -- the reconcile pass (src/cert/reconcile.cpp:4-21) on the GPU: error map
// plus the FP64-grade sum of squares, max and count, in one HBM-bound sweep.
//
// Traffic per pixel: approx 4 B + truth 4 B + mask 1 B read, error 4 B written (13 B).
// Each thread moves 4 pixels per step with 16-byte loads and stores when the buffers allow.
#include "rn_internal.h"
#include "rn_device.cuh"
#include "rn_reduce.cuh"

namespace rn {
namespace {

constexpr int kThreads = 256;

__device__ __forceinline__ float rec_px(float a, float t, uint8_t m, RecAcc& acc) {
    if (!m) return 0.0f;
    const float e = fabsf(__fsub_rn(a, t));
    acc.add(e);
    return e;
}

template <bool kVec>
__global__ void __launch_bounds__(kThreads) reconcile_kernel(const float* __restrict__ approx, const float* __restrict__ truth,
                                                             const uint8_t* __restrict__ mask, size_t npx,
                                                             float* __restrict__ err, RecPartial* parts, RecOut* out,
                                                             RecOut* host_out) {
    RecAcc acc;
    const size_t stride = (size_t)gridDim.x * kThreads;
    size_t tail0 = 0;
    if (kVec) {
        const size_t nq = npx / 4;
        const float4* a4 = reinterpret_cast<const float4*>(approx);
        const float4* t4 = reinterpret_cast<const float4*>(truth);
        const uchar4* m4 = reinterpret_cast<const uchar4*>(mask);
        float4* e4 = reinterpret_cast<float4*>(err);
        // four steps' loads at a time: few blocks run (a block takes eight steps of a thread), so
        // one step after the other is a chain of memory latencies (512 x 512: 12.1 us one at a time, 9.5 now)
        constexpr int kSteps = 4;
        for (size_t q0 = (size_t)blockIdx.x * kThreads + threadIdx.x; q0 < nq; q0 += stride * kSteps) {
            float4 a[kSteps], t[kSteps];
            uchar4 m[kSteps];
#pragma unroll
            for (int k = 0; k < kSteps; ++k) {
                const size_t q = q0 + stride * k;
                if (q < nq) {
                    a[k] = __ldcs(a4 + q);
                    t[k] = __ldcs(t4 + q);
                    m[k] = __ldcs(m4 + q);
                }
            }
#pragma unroll
            for (int k = 0; k < kSteps; ++k) {
                const size_t q = q0 + stride * k;
                if (q >= nq) break;
                float4 e;
                e.x = rec_px(a[k].x, t[k].x, m[k].x, acc);
                e.y = rec_px(a[k].y, t[k].y, m[k].y, acc);
                e.z = rec_px(a[k].z, t[k].z, m[k].z, acc);
                e.w = rec_px(a[k].w, t[k].w, m[k].w, acc);
                if (err) __stcs(e4 + q, e);
            }
        }
        tail0 = nq * 4;
    }
    for (size_t i = tail0 + (size_t)blockIdx.x * kThreads + threadIdx.x; i < npx; i += stride) {
        const float e = rec_px(approx[i], truth[i], mask[i], acc);
        if (err) err[i] = e;
    }
    rec_block_finish<kThreads>(acc, parts, out, blockIdx.x, gridDim.x, host_out);
}

}  // namespace

// The block count depends on the pixel count alone, so the reduction order, and with it
// every bit of the result, is the same on every run and every GPU.
int reconcile_blocks(size_t npx) {
    const size_t per_block = (size_t)kThreads * 4 * 8;
    size_t nb = (npx + per_block - 1) / per_block;
    if (nb < 1) nb = 1;
    if (nb > 2048) nb = 2048;
    return (int)nb;
}

cudaError_t launch_reconcile(const float* approx, const float* truth, const uint8_t* mask, size_t npx, float* err,
                             RecPartial* partials, int nblocks, RecOut* out, cudaStream_t s, RecOut* host_out) {
    const bool vec = ((uintptr_t)approx % 16 == 0) && ((uintptr_t)truth % 16 == 0) && ((uintptr_t)mask % 4 == 0) &&
                     (err == nullptr || (uintptr_t)err % 16 == 0);
    if (vec)
        reconcile_kernel<true><<<nblocks, kThreads, 0, s>>>(approx, truth, mask, npx, err, partials, out, host_out);
    else
        reconcile_kernel<false><<<nblocks, kThreads, 0, s>>>(approx, truth, mask, npx, err, partials, out, host_out);
    return cudaGetLastError();
}

}  // namespace rn
