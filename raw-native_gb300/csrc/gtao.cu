// gtao.cu -- ground-truth-based ambient occlusion (Jimenez, Wu, Pesce, Jarabo 2016) on the
// GPU: raw::post's GTAO pass (src/renderer/post_gtao.cpp:64-135) over the view-space
// G-buffer (:36-53), the screen-space approximation that the ray-traced oracle judges
// with the same reconcile.
//
// The view-space G-buffer is computed as the reference computes it, in float with one
// rounding per operation (bit-identical). GTAO itself runs in FP32 where the reference
// uses FP64; each slice's screen direction, in the reference the difference of two
// projections 1e-3 of the depth apart, is formed in closed form in pairs of floats (about 2^-44
// relative) and rounded once, and the march positions are kept relative to the pixel, so
// their floor (which pixel a sample falls in) is exact. The parity contract is the
// reference's own for its GPU pass: |gpu - cpu| <= 1e-3 on all but 0.1 % of pixels
// (raw/renderer/post_parity.hpp:15-19).
//
// Bound by instruction issue. What a sample needs discretely (its pixel, its bilinear taps, the
// radius test) keeps its exact float operations; the rest may differ in the last place:
// - depths and their reciprocals lie in one padded plane, so a tap is one 8-byte load without
//   a division or a bounds check (the two-pixel border is empty), and the nearest pixel is one
//   of the four taps;
// - divisions by the frame size and the step count are a multiplication and a residual step;
// - the horizon integral's cosines come from the horizons' cosines by the addition theorem: of
//   nine trigonometric calls a slice the three arc cosines are left;
// - no FP64 (two projections with four divisions and a hypot a slice).
// Over 44 shapes and 88 G-buffers the mean error against 64 bits is 0.947 to 1.008 times, 0.979 on
// average, what it was with FP64 projections and IEEE roots and quotients.
// 2561 x 1441, 16 slices of 16 steps: 12.0 -> 6.2 ms (issue 87 % of cycles, 293.8 M -> 174.9 M warp
// instructions at 1281 x 721).
#include "rn_internal.h"
#include "rn_device.cuh"
#include <algorithm>
#include <cmath>

namespace rn {
namespace {

struct View16 { float m[16]; };

__device__ __forceinline__ float row4(const float* r, float x, float y, float z, float w) {
    return fadd(fadd(fadd(fmul(r[0], x), fmul(r[1], y)), fmul(r[2], z)), fmul(r[3], w));
}

constexpr int kPad = 2;      // border cells of the depth plane: a clamped tap pair lies in it wholly

__global__ void view_gbuffer_kernel(int w, int h, const float* __restrict__ pos, const float* __restrict__ nrm,
                                    const uint8_t* __restrict__ mask, const View16 V, float* __restrict__ vpos,
                                    float* __restrict__ vnrm, float2* __restrict__ vdepth) {
    // the padded depth plane's cells; an empty one (and the border) has depth -1
    const int pw = w + 2 * kPad;
    const size_t n = (size_t)pw * (h + 2 * kPad);
    for (size_t c = (size_t)blockIdx.x * blockDim.x + threadIdx.x; c < n; c += (size_t)gridDim.x * blockDim.x) {
        const int x0 = (int)(c % pw) - kPad, y0 = (int)(c / pw) - kPad;
        if (x0 < 0 || y0 < 0 || x0 >= w || y0 >= h) { vdepth[c] = make_float2(-1.0f, 0.0f); continue; }
        const size_t i = (size_t)y0 * w + x0;
        float px = 0.0f, py = 0.0f, pz = 0.0f, nx = 0.0f, ny = 0.0f, nz = 0.0f, d = -1.0f;
        if (mask[i]) {
            const float x = pos[3 * i], y = pos[3 * i + 1], z = pos[3 * i + 2];
            const float a = nrm[3 * i], b = nrm[3 * i + 1], c = nrm[3 * i + 2];
            px = row4(V.m + 0, x, y, z, 1.0f);
            py = row4(V.m + 4, x, y, z, 1.0f);
            pz = row4(V.m + 8, x, y, z, 1.0f);
            const v3 nv = normalize(mk(row4(V.m + 0, a, b, c, 0.0f), row4(V.m + 4, a, b, c, 0.0f), row4(V.m + 8, a, b, c, 0.0f)));
            nx = nv.x; ny = nv.y; nz = nv.z;
            d = -pz;
        }
        vpos[3 * i] = px; vpos[3 * i + 1] = py; vpos[3 * i + 2] = pz;
        vnrm[3 * i] = nx; vnrm[3 * i + 1] = ny; vnrm[3 * i + 2] = nz;
        // a depth that is not a number is no tap either, and marked so that its own pixel keeps it
        vdepth[c] = make_float2(d >= 0.0f ? d : d < 0.0f ? -1.0f : -2.0f, 1.0f / d);
    }
}

struct GtaoArgs {
    int w, h;
    const float* pos;
    const float* nrm;
    const float2* depth;         // (depth, 1 / depth), padded
    float tan_half, aspect;
    float kx;                    // w / (aspect h) - 1
    float radius;
    int slices, steps;
    float rw, rh, rsteps;        // 1 / w, 1 / h, 1 / steps, rounded to nearest
    float* out;
};

// a / b rounded to nearest, from y = 1 / b rounded to nearest: the product and one residual step
// (Markstein 1990, theorem on division from a correctly rounded reciprocal).
__device__ __forceinline__ float div_by(float a, float b, float y) {
    const float q = a * y;
    return __fmaf_rn(__fmaf_rn(-b, q, a), y, q);
}

// Sums and products as unevaluated pairs hi + lo (Dekker 1971, Knuth's two-sum).
struct Pair { float hi, lo; };
__device__ __forceinline__ Pair two_prod(float a, float b) {
    const float p = a * b;
    return Pair{p, __fmaf_rn(a, b, -p)};
}
__device__ __forceinline__ Pair two_sum(float a, float b) {
    const float s = a + b, t = s - a;
    return Pair{s, (a - (s - t)) + (b - t)};
}
// a b + c d
__device__ __forceinline__ Pair dot2(float a, float b, float c, float d) {
    const Pair p = two_prod(a, b), q = two_prod(c, d), s = two_sum(p.hi, q.hi);
    const float lo = s.lo + (p.lo + q.lo), hi = s.hi + lo;
    return Pair{hi, lo - (hi - s.hi)};
}
__device__ __forceinline__ Pair square(const Pair& x) {
    const Pair p = two_prod(x.hi, x.hi);
    return Pair{p.hi, p.lo + 2.0f * x.hi * x.lo};
}

__global__ void __launch_bounds__(256) gtao_kernel(const GtaoArgs a) {
    const float kPi = 3.14159265358979f;
    __shared__ float2 s_dir[1024];               // (sin, cos) of every slice's angle
    for (int s = threadIdx.x; s < a.slices; s += 256) {
        float sp, cp;
        sincospif((s + 0.5f) / a.slices, &sp, &cp);
        s_dir[s] = make_float2(sp, cp);
    }
    __syncthreads();
    const int x = blockIdx.x * 16 + (threadIdx.x & 15), y = blockIdx.y * 16 + (threadIdx.x >> 4);
    if (x >= a.w || y >= a.h) return;
    const size_t i = (size_t)y * a.w + x;
    const int pw = a.w + 2 * kPad;
    const float2* const plane = a.depth + (size_t)kPad * pw + kPad;      // cell (0, 0)
    float depth = plane[(ptrdiff_t)y * pw + x].x;
    if (depth == -2.0f) depth = __int_as_float(0x7fffffff);
    if (depth < 0.0f) { a.out[i] = 1.0f; return; }
    const float P[3] = {a.pos[3 * i], a.pos[3 * i + 1], a.pos[3 * i + 2]};
    const float N[3] = {a.nrm[3 * i], a.nrm[3 * i + 1], a.nrm[3 * i + 2]};
    const float pl = sqrtf(P[0] * P[0] + P[1] * P[1] + P[2] * P[2]);
    const float V[3] = {-P[0] / pl, -P[1] / pl, -P[2] / pl};
    const float tan_half = a.tan_half, aspect = a.aspect;
    const float rpx = a.radius * a.h / (2.0f * tan_half * depth);
    float T[3] = {1.0f - V[0] * V[0], -V[0] * V[1], -V[0] * V[2]};
    const float tl = sqrtf(T[0] * T[0] + T[1] * T[1] + T[2] * T[2]);
    T[0] /= tl; T[1] /= tl; T[2] /= tl;
    const float B[3] = {V[1] * T[2] - V[2] * T[1], V[2] * T[0] - V[0] * T[2], V[0] * T[1] - V[1] * T[0]};
    // the position scaled by a power of two to a depth in [1, 2): the directions below do not
    // depend on the scale, and their squares cannot leave float's range
    const float up = __uint_as_float((254u - min(253u, max(1u, __float_as_uint(depth) >> 23))) << 23);
    const float Wd = depth * up, Px = P[0] * up, Py = P[1] * up;
    const float fxx = (float)x, fyy = (float)y, fw = (float)a.w, fh = (float)a.h, fsteps = (float)a.steps;
    float sum = 0.0f;
    for (int s = 0; s < a.slices; ++s) {
        const float2 sc = s_dir[s];
        const float dir[3] = {sc.y * T[0] + sc.x * B[0], sc.y * T[1] + sc.x * B[1], sc.y * T[2] + sc.x * B[2]};
        // the screen direction of P + e dir: the two projections' difference is a positive factor
        // times (w / aspect (dir.x depth + P.x dir.z), -h (dir.y depth + P.y dir.z))
        Pair X = dot2(dir[0], Wd, Px, dir[2]);
        const Pair Y = dot2(dir[1], Wd, Py, dir[2]);
        X.lo += X.hi * a.kx;
        const Pair xx = square(X), yy = square(Y), q = two_sum(xx.hi, yy.hi);
        const float ql = q.lo + (xx.lo + yy.lo);
        if (q.hi < 1e-18f) continue;
        // 1 / sqrt(q + ql) = r0 + r1: one Newton step from the hardware's value
        const float r0 = rsqrtf(q.hi);
        const Pair g = two_prod(r0, r0), hp = two_prod(q.hi, g.hi);
        const float res = (1.0f - hp.hi) - (hp.lo + (q.hi * g.lo + ql * g.hi));
        const float r1 = 0.5f * r0 * res;
        const Pair cx = two_prod(X.hi, r0), cy = two_prod(Y.hi, r0);
        const float c = cx.hi + (cx.lo + (X.hi * r1 + X.lo * r0));
        const float sn = -(cy.hi + (cy.lo + (Y.hi * r1 + Y.lo * r0)));
        const float dv = dir[0] * V[0] + dir[1] * V[1] + dir[2] * V[2];
        const float od[3] = {dir[0] - dv * V[0], dir[1] - dv * V[1], dir[2] - dv * V[2]};
        float ax[3] = {od[1] * V[2] - od[2] * V[1], od[2] * V[0] - od[0] * V[2], od[0] * V[1] - od[1] * V[0]};
        const float ral = rsqrtf(ax[0] * ax[0] + ax[1] * ax[1] + ax[2] * ax[2]);
        ax[0] *= ral; ax[1] *= ral; ax[2] *= ral;
        const float na = N[0] * ax[0] + N[1] * ax[1] + N[2] * ax[2];
        const float pn[3] = {N[0] - ax[0] * na, N[1] - ax[1] * na, N[2] - ax[2] * na};
        const float pnl = sqrtf(pn[0] * pn[0] + pn[1] * pn[1] + pn[2] * pn[2]);
        if (pnl < 1e-9f) continue;
        const float sgn = (od[0] * pn[0] + od[1] * pn[1] + od[2] * pn[2]) >= 0.0f ? 1.0f : -1.0f;
        const float cn = fminf(fmaxf((pn[0] * V[0] + pn[1] * V[1] + pn[2] * V[2]) / pnl, 0.0f), 1.0f);
        const float nang = sgn * acosf(cn);
        const float snn = sgn * sqrtf((1.0f - cn) * (1.0f + cn));       // sin(nang)
        // the horizons' cosines; the hemisphere's own at nang +- pi / 2 to begin with
        float hc[2] = {-snn, snn};
#pragma unroll 1
        for (int side = 0; side < 2; ++side) {
            const float step = side == 0 ? rpx : -rpx;
            float best = side == 0 ? hc[0] : hc[1];
#pragma unroll 1
            for (int k = 1; k <= a.steps; ++k) {
                const float off = div_by(step * k, fsteps, a.rsteps);
                // the sample relative to the pixel's corner: fx = x + rx
                const float rx = 0.5f + off * c, ry = 0.5f + off * sn;
                const float gx = rx - 0.5f, gy = ry - 0.5f;
                const float flx = floorf(gx), fly = floorf(gy);
                const int ix = (int)floorf(rx), iy = (int)floorf(ry);
                const int tx = (int)flx, ty = (int)fly;
                // the four nearest pixel centres; clamped into the empty border
                const int x0 = min(max(x + tx, -kPad), a.w), y0 = min(max(y + ty, -kPad), a.h);
                const float2* t = plane + (ptrdiff_t)y0 * pw + x0;
                const float2 t00 = t[0], t01 = t[1], t10 = t[pw], t11 = t[pw + 1];
                // the sample's own pixel is one of them
                const float n0 = ix == tx ? t00.x : t01.x, n1 = ix == tx ? t10.x : t11.x;
                const float nearest = iy == ty ? n0 : n1;
                if (nearest < 0.0f || (ix == 0 && iy == 0)) continue;
                // 1 / depth interpolated between them, or the nearest pixel's depth when one of
                // them is empty or they differ by more than 10 % (post_gtao.cpp:14-33)
                const float lo = fminf(fminf(t00.x, t01.x), fminf(t10.x, t11.x));
                const float hi = fmaxf(fmaxf(t00.x, t01.x), fmaxf(t10.x, t11.x));
                float D = nearest;
                if (lo >= 0.0f && !(hi > 1.1f * lo)) {
                    const float bx = gx - flx, by = gy - fly;
                    const float inv = (t00.y * (1.0f - bx) + t01.y * bx) * (1.0f - by) + (t10.y * (1.0f - bx) + t11.y * bx) * by;
                    D = frcp(inv);
                }
                const float fx = fxx + rx, fy = fyy + ry;
                const float S[3] = {(div_by(fx, fw, a.rw) * 2.0f - 1.0f) * D * tan_half * aspect,
                                    (1.0f - div_by(fy, fh, a.rh) * 2.0f) * D * tan_half, -D};
                const float d[3] = {S[0] - P[0], S[1] - P[1], S[2] - P[2]};
                const float dl = sqrtf(d[0] * d[0] + d[1] * d[1] + d[2] * d[2]);
                if (dl < 1e-9f || dl > a.radius) continue;
                best = fmaxf(best, __fdividef(d[0] * V[0] + d[1] * V[1] + d[2] * V[2], dl));
            }
            if (side == 0) hc[0] = best; else hc[1] = best;
        }
        // a horizon h = +-acos(hc), limited to nang +- pi / 2, where cos(2 h - nang) is -cn;
        // else (2 hc^2 - 1) cn +- 2 hc sqrt(1 - hc^2) sin(nang)
        const float c1 = fminf(fmaxf(hc[0], -1.0f), 1.0f), c0 = fminf(fmaxf(hc[1], -1.0f), 1.0f);
        const float A1 = acosf(c1) - nang, A0 = -acosf(c0) - nang;
        const float h1 = nang + fminf(A1, kPi / 2), h0 = nang + fmaxf(A0, -kPi / 2);
        const float k1 = A1 < kPi / 2 ? (2.0f * c1 * c1 - 1.0f) * cn + 2.0f * c1 * sqrtf((1.0f - c1) * (1.0f + c1)) * snn : -cn;
        const float k0 = A0 > -kPi / 2 ? (2.0f * c0 * c0 - 1.0f) * cn - 2.0f * c0 * sqrtf((1.0f - c0) * (1.0f + c0)) * snn : -cn;
        const float a0 = (cn + 2.0f * h0 * snn - k0) * 0.25f;
        const float a1 = (cn + 2.0f * h1 * snn - k1) * 0.25f;
        sum += pnl * (a0 + a1);
    }
    a.out[i] = sum / a.slices;
}

}  // namespace

size_t gtao_depth_cells(int w, int h) { return (size_t)(w + 2 * kPad) * (size_t)(h + 2 * kPad); }

int launch_gtao(int w, int h, const float* pos, const float* nrm, const uint8_t* mask, const float* view16,
                float fovy, float radius, int slices, int steps, float* vpos, float* vnrm, float2* vdepth, float* out,
                cudaStream_t s) {
    View16 V;
    for (int k = 0; k < 16; ++k) V.m[k] = view16[k];
    const size_t n = gtao_depth_cells(w, h);
    const unsigned blocks = (unsigned)std::min<size_t>((n + 255) / 256, 65535u * 8);
    view_gbuffer_kernel<<<blocks, 256, 0, s>>>(w, h, pos, nrm, mask, V, vpos, vnrm, vdepth);
    const double aspect = (double)((float)w / (float)h);
    GtaoArgs a{w, h, vpos, vnrm, vdepth, (float)std::tan(0.5 * (double)fovy), (float)aspect,
               (float)((double)w / (aspect * (double)h) - 1.0), radius, slices, steps, 1.0f / (float)w, 1.0f / (float)h,
               1.0f / (float)steps, out};
    gtao_kernel<<<dim3((w + 15) / 16, (h + 15) / 16), 256, 0, s>>>(a);
    return cudaGetLastError() == cudaSuccess ? RN_OK : RN_ERR_CUDA;
}

}  // namespace rn
