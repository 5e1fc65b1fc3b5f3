// ssao_device.cuh -- one 32 x 8 tile of the SSAO pass with the reconcile's per-thread share,
// shared by the single-frame kernel (ssao.cu) and the batched multi-view kernel (batch.cu).
// See ssao.cu for the design.
#pragma once
#include "rn_internal.h"
#include "rn_device.cuh"
#include "rn_reduce.cuh"

namespace rn {
namespace ssao_dev {

// A tile is kTX x TY pixels, one thread each (TY = 8 by default; 4 and 16 are the
// autotuner's alternatives), with a window of (TY + 2R) x (kTX + 2R) positions.
constexpr int kTX = 32, kTY = 8, kR = 6;
constexpr int kSW = kTX + 2 * kR, kSH = kTY + 2 * kR;
constexpr int kThreads = kTX * kTY;
template <int TY> struct Tile {
    static constexpr int kH = TY + 2 * kR;
    static constexpr int kThreads = kTX * TY;
};

// std::lround(v) for |v| < 2^21 whose fraction is not within kHalf of a half: the addition of
// 1.5 x 2^23 rounds v to an integer in the sum's low bits. `off` receives v's distance to it.
constexpr float kMagic = 12582912.0f, kHalf = 4e-5f;
__device__ __forceinline__ int round_fast(float v, float& off) {
    const float t = __fadd_rn(v, kMagic);
    off = fabsf(__fsub_rn(v, __fsub_rn(t, kMagic)));
    return __float_as_int(t) - __float_as_int(kMagic);
}
// Sample s's tap offset (ssao.cpp:18-23): lround(cos(a) rad), lround(sin(a) rad) with
// a = 6.2831853 u, rad = (0.3 + 0.7 u') 6, from the pixel's hash sum `base` + s. An integer that
// only changes where the product crosses a half, so it is formed from the hardware's sine and
// cosine of the angle less pi (2^-21.4 on [-pi, pi]; with the angle's and the radius's own
// rounding below 8e-6 of a pixel in all) and formed again by the exact operations, with the host
// libm's bits where `corr` is set, when a product lies within 4e-5 of a half (3 taps in 10,000).
__device__ __forceinline__ void tap_offset(uint32_t base, int s, const uint8_t* __restrict__ corr, int& dx, int& dy) {
    auto mix = [](uint32_t h) { h = (h ^ (h >> 13)) * 1274126177u; return h ^ (h >> 16); };
    const uint32_t p = base + (uint32_t)s * 2246822519u;
    const uint32_t h1 = mix(p), h2 = mix(p + 97u * 2246822519u);
    // cos and sin of a = -cos and -sin of a - pi; a - pi = 2 pi (u - 1/2)
    const float ang = (one_plus(h1) - 1.5f) * 6.2831853f;
    const float rad = __fmaf_rn(one_plus(h2), -4.2f, 2.4f);            // -(1.8 + 4.2 u')
    float ox, oy;
    dx = round_fast(__cosf(ang) * rad, ox);
    dy = round_fast(__sinf(ang) * rad, oy);
    if (fmaxf(ox, oy) > 0.5f - kHalf) {
        const float r = fmul(fadd(0.3f, fmul(0.7f, unit24(h2 & 0xFFFFFFu))), 6.0f);
        float c, sn;
        sample_sincos(h1 & 0xFFFFFFu, corr, c, sn);
        dx = (int)lroundf(fmul(c, r));
        dy = (int)lroundf(fmul(sn, r));
    }
}

// Tile (bx, by) of a w x h frame: SSAO into ao, and with kFused the error against `truth`
// into err (may be null) with this thread's share of the reconcile in `acc`. `win` is the
// block's shared window. Every thread of the block must call it.
template <bool kFused, int TY = kTY>
__device__ __forceinline__ void ssao_tile(float4 (&win)[Tile<TY>::kH][kSW], int bx, int by, int w, int h,
                                          const float* __restrict__ pos, const float* __restrict__ nrm,
                                          const uint8_t* __restrict__ mask, int samples, float radius,
                                          const uint8_t* __restrict__ corr, float* __restrict__ ao,
                                          const float* __restrict__ truth, float* __restrict__ err, RecAcc& acc) {
    const int x0 = bx * kTX, y0 = by * TY;
    for (int q = threadIdx.x; q < Tile<TY>::kH * kSW; q += Tile<TY>::kThreads) {
        const int wy = q / kSW, wx = q % kSW;
        const int gx = x0 - kR + wx, gy = y0 - kR + wy;
        float4 v = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
        if (gx >= 0 && gy >= 0 && gx < w && gy < h) {
            const size_t j = (size_t)gy * w + gx;
            if (mask[j]) v = make_float4(pos[3 * j], pos[3 * j + 1], pos[3 * j + 2], 1.0f);
        }
        win[wy][wx] = v;
    }
    __syncthreads();
    const int tx = threadIdx.x % kTX, ty = threadIdx.x / kTX;
    const int x = x0 + tx, y = y0 + ty;
    if (x < w && y < h) {
        const size_t i = (size_t)y * w + x;
        const bool covered = mask[i] != 0;
        float a = 1.0f;
        if (covered) {
            const float4 Pw = win[ty + kR][tx + kR];
            const v3 P = mk(Pw.x, Pw.y, Pw.z);
            const v3 n = load3(nrm + 3 * i);
            int occ = 0, used = 0;
            // A tap occludes when 1e-4 <= |d| <= radius and n . (d / |d|) > 0.15, each side of the
            // rule a float rounded in the reference's order. Away from its thresholds the squares
            // decide without the root and the division (fused, a few ulps off; the margins are
            // 1e-5 of |d|^2 and 1e-4 of (n . d)^2, which holds them for |n| < 2); near one, or for
            // other normals and radii, the exact operations do.
            const bool plain = n.x * n.x + n.y * n.y + n.z * n.z < 4.0f && radius > 0.0f;
            const float r2 = radius * radius, r2lo = plain ? r2 * 0.99999f : -1.0f, r2hi = plain ? r2 * 1.00001f : __int_as_float(0x7f800000);
            const uint32_t base = (uint32_t)x * 374761393u + (uint32_t)y * 668265263u;
#pragma unroll 2
            for (int s = 0; s < samples; ++s) {
                int dx, dy;
                tap_offset(base, s, corr, dx, dy);
                const float4 Q = win[ty + kR + dy][tx + kR + dx];
                if (Q.w == 0.0f) continue;            // out of the frame or not covered
                ++used;
                const v3 d = sub(mk(Q.x, Q.y, Q.z), P);
                const float d2 = __fmaf_rn(d.x, d.x, __fmaf_rn(d.y, d.y, d.z * d.z));
                const float nd = __fmaf_rn(n.x, d.x, __fmaf_rn(n.y, d.y, n.z * d.z));
                const float q = nd * nd, lim = 0.0225f * d2;
                const bool in = d2 < r2lo && d2 > 1.00001e-8f;
                const bool yes = nd > 0.0f && q > lim * 1.0001f, no = nd <= 0.0f || q < lim * 0.9999f;
                if (in && yes) ++occ;
                else if (!((in && no) || (plain && (d2 > r2hi || d2 < 0.99999e-8f)))) {
                    const float dist = length(d);
                    if (dist < 1e-4f || dist > radius) continue;
                    const float ndl = dot(n, normalize(d));
                    if (ndl > 0.15f) ++occ;
                }
            }
            a = used > 0 ? fsub(1.0f, fdiv((float)occ, (float)used)) : 1.0f;
            a = a < 0.0f ? 0.0f : a;
        }
        ao[i] = a;
        if (kFused) {
            float e = 0.0f;
            if (covered) {
                e = fabsf(fsub(a, truth[i]));
                acc.add(e);
            }
            if (err) err[i] = e;
        }
    }
}

}  // namespace ssao_dev
}  // namespace rn
