// ssao.cu -- the screen-space AO pass (src/renderer/ssao.cpp:11-39) on the GPU, with the
// reconcile against the ray-traced truth optionally fused into its epilogue.
//
// Every sample lands within R = 6 pixels of its pixel (radius (0.3 + 0.7 u) * 6, rounded), so
// a 32 x 8 tile needs a 44 x 20 window of positions and coverage. The block stages that window
// in shared memory once (position.xyz and a validity flag: in the frame and covered), and the
// 24 taps of each pixel read it from there: per pixel the pass moves 12 B of position, 12 B
// of normal, 1 B of mask and 4 B of output through HBM, the halo's re-reads hit L2.
//
// Bound by instruction issue (95 % of cycles), so each tap's offset and its occlusion are
// decided by the cheapest arithmetic that can be trusted away from their thresholds, and by the
// reference's exact operations near them (tap_offset, ssao_tile): 2560 x 1440, 24 taps:
// 409 -> 195 us, 480 M -> 206 M warp instructions; the image is the same bits.
#include "ssao_device.cuh"

namespace rn {
namespace {

using namespace ssao_dev;

template <bool kFused, int TY>
__global__ void __launch_bounds__(Tile<TY>::kThreads) ssao_kernel(int w, int h, const float* __restrict__ pos,
                                                                  const float* __restrict__ nrm,
                                                                  const uint8_t* __restrict__ mask, int samples,
                                                                  float radius, const uint8_t* __restrict__ corr,
                                                                  float* __restrict__ ao, const float* __restrict__ truth,
                                                                  float* __restrict__ err, RecPartial* parts, RecOut* out,
                                                                  RecOut* host_out) {
    __shared__ float4 win[Tile<TY>::kH][kSW];
    RecAcc acc;
    ssao_tile<kFused, TY>(win, blockIdx.x, blockIdx.y, w, h, pos, nrm, mask, samples, radius, corr, ao, truth, err, acc);
    if (kFused)
        rec_block_finish<Tile<TY>::kThreads>(acc, parts, out, blockIdx.y * gridDim.x + blockIdx.x, gridDim.x * gridDim.y,
                                             host_out);
}

template <int TY>
void launch_tile(int w, int h, const float* pos, const float* nrm, const uint8_t* mask, int samples, float radius,
                 const uint8_t* corr, float* ao, const float* truth, float* err, RecPartial* partials, RecOut* out,
                 cudaStream_t s, RecOut* host_out) {
    const dim3 grid((w + kTX - 1) / kTX, (h + TY - 1) / TY);
    if (truth)
        ssao_kernel<true, TY><<<grid, Tile<TY>::kThreads, 0, s>>>(w, h, pos, nrm, mask, samples, radius, corr, ao, truth,
                                                                   err, partials, out, host_out);
    else
        ssao_kernel<false, TY><<<grid, Tile<TY>::kThreads, 0, s>>>(w, h, pos, nrm, mask, samples, radius, corr, ao,
                                                                    nullptr, nullptr, nullptr, nullptr, nullptr);
}

// The tuned tile height; 8 rows at most where 16 would leave fewer than eight blocks an SM: the
// blocks all run at once then, and an SM with four of them makes the others wait (512 x 512, 24
// taps: 25.0 us with 16 rows, 22.3 with 8, 22.6 with 4; 1920 x 1080: 114.9, 115.2, 119.7).
int tile_h(int w, int h) {
    const int t = ctx().tune.ssao_tile_h;
    const long blocks = (long)((w + kTX - 1) / kTX) * ((h + 15) / 16);
    return t == 4 ? 4 : t == 16 && blocks >= 8L * ctx().sm_count ? 16 : 8;
}

}  // namespace

// Blocks of one SSAO launch (the fused reconcile keeps one partial per block).
int ssao_blocks(int w, int h) { return ((w + kTX - 1) / kTX) * ((h + tile_h(w, h) - 1) / tile_h(w, h)); }

int launch_ssao(int w, int h, const float* pos, const float* nrm, const uint8_t* mask, int samples, float radius,
                const uint8_t* corr, float* ao, const float* truth, float* err, RecPartial* partials, RecOut* out,
                cudaStream_t s, RecOut* host_out) {
    switch (tile_h(w, h)) {
        case 4: launch_tile<4>(w, h, pos, nrm, mask, samples, radius, corr, ao, truth, err, partials, out, s, host_out); break;
        case 16: launch_tile<16>(w, h, pos, nrm, mask, samples, radius, corr, ao, truth, err, partials, out, s, host_out); break;
        default: launch_tile<8>(w, h, pos, nrm, mask, samples, radius, corr, ao, truth, err, partials, out, s, host_out); break;
    }
    return cudaGetLastError() == cudaSuccess ? RN_OK : RN_ERR_CUDA;
}

}  // namespace rn
