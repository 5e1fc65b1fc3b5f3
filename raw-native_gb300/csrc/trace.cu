// trace.cu -- ray-traced AO and lighting model 2's visibility on the GPU: the hot loop of
// raw-native's CPU oracle (src/renderer/ray_ao.cpp:20-51) as one persistent kernel.
//
// Work: the frame is cut into packets of 32 pixels (8 x 4 by default; 4 x 8 and 16 x 2 are
// the autotuner's alternatives); each warp takes the next packet from a global counter, one
// pixel per lane, and walks its `spp` hemisphere rays, then the sun ray, through the 4-wide BVH.
// Small frames are cut into packets of 16 or 8 pixels, two or four lanes sharing each pixel's
// samples (lanes_log2). Neighbouring lanes trace neighbouring pixels, so the warp's rays
// start close together and visit similar nodes.
//
// One walk per hemisphere ray answers both of the reference's questions about it: a hit
// with t < radius (AO, ray_ao.cpp:39) and, for an open ray, a hit at any distance (sky,
// :41). The walk starts with the far limit and, once it has found a hit beyond the radius,
// keeps looking only for hits nearer than the radius; every box either query could need is
// visited, so both answers are the reference's. The sun ray is the last slot of the same
// loop, so the kernel holds one copy of the walk.
//
// Exactness: ray generation (basis, origin, cosine-weighted direction) and the triangle test
// use one IEEE rounding per operation in the reference's order; the sample angle's cos/sin
// carry the host libm's bits (rn_device.cuh). The box test is only required to be
// conservative, and is: padded boxes, the robust slab exit of Ize (2013) widened by
// 1.0000008, and NaN-safe min/max, so the any-hit answers are exactly the
// scan-every-triangle answers the reference's own BVH reproduces.
#include "trace_device.cuh"

namespace rn {
namespace {

using namespace trace_dev;

// kCount: trace only every `stride`-th tile and add the rays, node fetches and triangle
// fetches to counts[0..3] (hemisphere rays, nodes, tris, sky continuations); the outputs of
// the other tiles are left unwritten. "Sky continuations" are the open hemisphere rays whose
// walk went on past the radius: the same walk serves both queries.
template <bool kCount, int kMinBlocks, int kStackN, bool kLeafPass, int kP, bool kFew = false>
__global__ void __launch_bounds__(256, kMinBlocks) trace_kernel(const __grid_constant__ TraceParams p, uint32_t* tile_ctr,
                                                                unsigned long long* counts, uint32_t stride) {
    const int pl = kP == 0 ? p.packet_log2 : min(p.packet_log2, 5 - kP), tw = 1 << pl, th = (32 >> kP) >> pl;
    const int tiles_x = (p.w + tw - 1) >> pl, tiles_y = (p.h + th - 1) / th;
    const uint32_t ntiles = (uint32_t)tiles_x * tiles_y;
    const unsigned lane = threadIdx.x & 31u;
    __shared__ Node4 frontier[8][kFrontierNodes];
    Node4* F = frontier[threadIdx.x >> 5];
    Counts cn;
    int skip = 0;                                  // packets to walk without the sieve (trace_packet)
    // lighting model 2's sun direction, normalized on the device as computeRTVisibility does
    const v3 toLight = normalize(mk(p.lx, p.ly, p.lz));
    while (true) {
        uint32_t tile = 0;
        if (lane == 0) tile = atomicAdd(tile_ctr, 1u);
        tile = __shfl_sync(0xffffffffu, tile, 0);
        if (tile >= ntiles) break;
        const unsigned px = kP == 0 ? lane : lane & ((32u >> kP) - 1u);
        const int x = ((int)(tile % tiles_x) << pl) + (int)(px & (tw - 1));
        const int y = (int)(tile / tiles_x) * th + (int)(px >> pl);
        // no lane leaves the loop body early: the next tile fetch is a full-warp shuffle
        if (kCount && tile % stride != 0) continue;
        trace_packet<kCount, kStackN, kLeafPass, kP, kFew>(p, p.short_dir, x, y, x < p.w && y < p.h, toLight, cn, skip, F, (int)(lane >> (5 - kP)));
        __syncwarp();                              // the frontier is rebuilt for the next tile
    }
    if (kCount) {
        atomicAdd(counts, cn.rays);
        atomicAdd(counts + 1, cn.nodes);
        atomicAdd(counts + 2, cn.tris);
        atomicAdd(counts + 3, cn.sky);
    }
}

// AO-only walks with warp-level compaction. A warp takes a packet of 32 pixels and puts all
// of its walks (every covered pixel's spp samples) in one queue: each lane runs one walk
// (pixel, sample) at a time, a node per loop step, and whenever fewer than `refill` lanes are
// still walking, the idle lanes take the next walks of the queue, whichever pixel they
// belong to. A lane is therefore not held by the slowest walk of its own pixel's sample
// round, as in trace_kernel's one-pixel-per-lane loop; only the queue's last walks leave
// lanes idle. A walk's rays, box tests and hit test are trace_packet's (sample_direction,
// slab, hit_leaf, the frontier start), and a pixel's AO is its count of open walks over spp:
// an integer count, so the order the walks finish in changes no bit.
// With `sort` (at most kSortSpp samples a pixel) the queue is ordered by the walks' direction
// octant first (a counting sort of the packet's walks in shared memory), so the lanes that
// walk together point into one or two octants: nearby origins, the same signs of the
// direction, similar child orders and node sequences.
constexpr int kSortSpp = 16;
template <int kMinBlocks, int kStackN>
__global__ void __launch_bounds__(256, kMinBlocks) trace_ao_pool_kernel(const __grid_constant__ TraceParams p,
                                                                        uint32_t* tile_ctr, int refill, int sort) {
    const int pl = p.packet_log2, tw = 1 << pl, th = 32 >> pl;
    const int tiles_x = (p.w + tw - 1) >> pl, tiles_y = (p.h + th - 1) / th;
    const uint32_t ntiles = (uint32_t)tiles_x * tiles_y;
    const unsigned lane = threadIdx.x & 31u;
    const unsigned below = (1u << lane) - 1u;
    __shared__ Node4 frontier[8][kFrontierNodes];
    __shared__ int open_sh[8][32];
    __shared__ uint8_t lane_sh[8][32];
    __shared__ uint16_t perm_sh[8][32 * kSortSpp];
    __shared__ uint32_t oct_sh[8][8];
    uint16_t* perm = perm_sh[threadIdx.x >> 5];
    uint32_t* octs = oct_sh[threadIdx.x >> 5];
    Node4* F = frontier[threadIdx.x >> 5];
    int* opens = open_sh[threadIdx.x >> 5];
    uint8_t* lane_of = lane_sh[threadIdx.x >> 5];   // the covered lanes in lane order
    const size_t np = (size_t)p.w * p.h;
    int32_t stack[kStackN];
    while (true) {
        uint32_t tile = 0;
        if (lane == 0) tile = atomicAdd(tile_ctr, 1u);
        tile = __shfl_sync(0xffffffffu, tile, 0);
        if (tile >= ntiles) break;
        const int x = ((int)(tile % tiles_x) << pl) + (int)(lane & (tw - 1));
        const int y = (int)(tile / tiles_x) * th + (int)(lane >> pl);
        const bool valid = x < p.w && y < p.h;
        const size_t i = valid ? (size_t)y * p.w + x : 0;
        uint8_t m = 0;
        v3 P = mk(0.0f, 0.0f, 0.0f), n = P;
        if (valid) {
            m = p.mask[i];
            P = load3(p.pos + 3 * i);
            n = load3(p.nrm + 3 * i);
            if (p.mirror) {
                store3(mirror_pos(p.mirror, np) + 3 * i, P);
                store3(mirror_nrm(p.mirror, np) + 3 * i, n);
                mirror_mask(p.mirror, np)[i] = m;
            }
            if (!m) {
                p.ao[i] = 1.0f;
                if (p.mirror) mirror_ao(p.mirror, np)[i] = 1.0f;
            }
        }
        const bool covered = valid && m;
        // basis (ray_ao.cpp:14-17) of the lane's own pixel; other lanes read it by shuffle
        const v3 a = fabsf(n.x) > 0.9f ? mk(0.0f, 1.0f, 0.0f) : mk(1.0f, 0.0f, 0.0f);
        v3 T = mk(0.0f, 0.0f, 0.0f), B = T, O = T;
        if (covered) {
            T = normalize(cross(a, n));
            B = cross(n, T);
            O = add(P, scale(n, 1e-3f));
        }
        // no plane: an empty frontier is left to the walk's own test
        const int fn = (p.has_geometry && p.frontier == FRONTIER_NEAR)
                           ? max(0, tile_frontier(p, tile_box(O, covered), TilePlane{0.0f, 0.0f, 0.0f, 0.0f, 0.0f}, F)) : 0;
        const unsigned cov = __ballot_sync(0xffffffffu, covered);
        const int nc = __popc(cov);
        opens[lane] = 0;
        if (covered) lane_of[__popc(cov & below)] = (uint8_t)lane;
        __syncwarp();
        const uint32_t total = (uint32_t)nc * (uint32_t)p.spp;
        const bool sorted = sort && p.spp <= kSortSpp && total > 0;
        if (sorted) {
            // the octant of every walk (wi: pixel lane_of[wi % nc], sample wi / nc), counted,
            // then placed: perm[] lists the walks octant by octant
            if (lane < 8) octs[lane] = 0;
            __syncwarp();
            uint64_t mine = 0;                       // 4 bits a walk of this lane's share
            for (uint32_t k = 0; k < (uint32_t)kSortSpp; ++k) {
                const uint32_t wi = lane + 32u * k;
                const bool has = wi < total;
                const int src = (int)lane_of[has ? wi % (uint32_t)nc : 0u];
                const v3 pt = mk(__shfl_sync(0xffffffffu, T.x, src), __shfl_sync(0xffffffffu, T.y, src),
                                 __shfl_sync(0xffffffffu, T.z, src));
                const v3 pb = mk(__shfl_sync(0xffffffffu, B.x, src), __shfl_sync(0xffffffffu, B.y, src),
                                 __shfl_sync(0xffffffffu, B.z, src));
                const v3 pn = mk(__shfl_sync(0xffffffffu, n.x, src), __shfl_sync(0xffffffffu, n.y, src),
                                 __shfl_sync(0xffffffffu, n.z, src));
                const int qx = __shfl_sync(0xffffffffu, x, src), qy = __shfl_sync(0xffffffffu, y, src);
                if (has) {
                    const v3 dd = sample_direction(pt, pb, pn, (uint32_t)qx, (uint32_t)qy, wi / (uint32_t)nc, p.corr);
                    const uint32_t o8 = (dd.x < 0.0f ? 1u : 0u) | (dd.y < 0.0f ? 2u : 0u) | (dd.z < 0.0f ? 4u : 0u);
                    mine |= (uint64_t)o8 << (4 * k);
                    atomicAdd(&octs[o8], 1u);
                }
            }
            __syncwarp();
            if (lane == 0) {
                uint32_t run = 0;
                for (int o8 = 0; o8 < 8; ++o8) { const uint32_t c = octs[o8]; octs[o8] = run; run += c; }
            }
            __syncwarp();
            for (uint32_t k = 0; k < (uint32_t)kSortSpp; ++k) {
                const uint32_t wi = lane + 32u * k;
                if (wi < total) perm[atomicAdd(&octs[(mine >> (4 * k)) & 7u], 1u)] = (uint16_t)wi;
            }
            __syncwarp();
        }
        uint32_t next = 0;
        bool active = false;
        int q = 0;                    // the lane whose pixel the current walk belongs to
        v3 o = O, d = O;
        Inv iv;
        LeafRay wr;
        bool wr_ready = false;
        int32_t cur = 0;
        int sp = 0;
        uint32_t guard = 0;
        const float tmax = p.radius;
        while (p.has_geometry && total > 0) {
            const unsigned busy = __ballot_sync(0xffffffffu, active);
            if (__popc(busy) < refill && next < total) {
                // the idle lanes take the next walks of the queue, in lane order
                const unsigned idle = ~busy;
                const uint32_t my = next + (uint32_t)__popc(idle & below);
                next = min(total, next + (uint32_t)__popc(idle));
                const bool take = !active && my < total;
                const uint32_t wi = take ? (sorted ? (uint32_t)perm[my] : my) : 0u;
                const int src = (int)lane_of[wi % (uint32_t)nc];
                const v3 pt = mk(__shfl_sync(0xffffffffu, T.x, src), __shfl_sync(0xffffffffu, T.y, src),
                                 __shfl_sync(0xffffffffu, T.z, src));
                const v3 pb = mk(__shfl_sync(0xffffffffu, B.x, src), __shfl_sync(0xffffffffu, B.y, src),
                                 __shfl_sync(0xffffffffu, B.z, src));
                const v3 pn = mk(__shfl_sync(0xffffffffu, n.x, src), __shfl_sync(0xffffffffu, n.y, src),
                                 __shfl_sync(0xffffffffu, n.z, src));
                const v3 po = mk(__shfl_sync(0xffffffffu, O.x, src), __shfl_sync(0xffffffffu, O.y, src),
                                 __shfl_sync(0xffffffffu, O.z, src));
                const int qx = __shfl_sync(0xffffffffu, x, src), qy = __shfl_sync(0xffffffffu, y, src);
                if (take) {
                    q = src;
                    o = po;
                    d = sample_direction(pt, pb, pn, (uint32_t)qx, (uint32_t)qy, wi / (uint32_t)nc, p.corr);
                    iv = make_inv<true>(o, d, kShortDir);
                    wr_ready = false;
                    sp = 0;
                    guard = 0;
                    active = true;
                    // start: the frontier's entries stand in for the root (walk(), trace_device.cuh)
                    cur = 0;
                    if (fn > 0) {
                        int32_t nearest = -1;
                        float tbest = 3.0e38f;
                        bool hit = false;
                        for (int e = 0; e < fn && !hit; ++e) {
                            float tn;
                            const FrontierBox fb = frontier_get(F, e);
                            if (!slab(fb.lo[0], fb.hi[0], fb.lo[1], fb.hi[1], fb.lo[2], fb.hi[2], iv, tmax, tn)) continue;
                            const int32_t c = fb.word;
                            if (c < 0) {
                                if (!wr_ready) { wr = make_leaf_ray(o, d); wr_ready = true; }
                                const uint32_t w = (uint32_t)~c;
                                const uint32_t first = w >> 3, count = (w & 7u) + 1u;
                                for (uint32_t k = 0; k < count && !hit; ++k) {
                                    float t, id;
                                    if (hit_leaf(wr, o, d, p.tris + first + k, t, id) && t < tmax) hit = true;
                                }
                                continue;
                            }
                            if (nearest < 0) { nearest = c; tbest = tn; continue; }
                            int32_t push = c;
                            if (tn < tbest) { push = nearest; nearest = c; tbest = tn; }
                            stack[sp++] = push;                  // fn <= kFrontier < kStackN
                        }
                        if (hit) active = false;                 // occluded: not open
                        else if (nearest >= 0) cur = nearest;
                        else if (sp > 0) cur = stack[--sp];
                        else { active = false; atomicAdd(&opens[q], 1); }
                    }
                }
            }
            if (!__any_sync(0xffffffffu, active)) {
                if (next >= total) break;
                continue;
            }
            if (!active) continue;
            // one node of the lane's walk
            const float4* nq = reinterpret_cast<const float4*>(p.nodes + cur);
            const float4 lx = __ldg(nq + 0), hx = __ldg(nq + 1), ly = __ldg(nq + 2), hy = __ldg(nq + 3);
            const float4 lz = __ldg(nq + 4), hz = __ldg(nq + 5);
            const int4 ch = __ldg(reinterpret_cast<const int4*>(nq + 6));
            const int cnt = __ldg(reinterpret_cast<const int*>(nq + 7));
            const float LX[4] = {lx.x, lx.y, lx.z, lx.w}, HX[4] = {hx.x, hx.y, hx.z, hx.w};
            const float LY[4] = {ly.x, ly.y, ly.z, ly.w}, HY[4] = {hy.x, hy.y, hy.z, hy.w};
            const float LZ[4] = {lz.x, lz.y, lz.z, lz.w}, HZ[4] = {hz.x, hz.y, hz.z, hz.w};
            const int32_t CH[4] = {ch.x, ch.y, ch.z, ch.w};
            int32_t nearest = -1;
            float tbest = 3.0e38f;
            bool hit = false, overflow = false;
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                float tn;
                if (hit || k >= cnt || !slab(LX[k], HX[k], LY[k], HY[k], LZ[k], HZ[k], iv, tmax, tn)) continue;
                const int32_t c = CH[k];
                if (c < 0) {
                    if (!wr_ready) { wr = make_leaf_ray(o, d); wr_ready = true; }
                    const uint32_t w = (uint32_t)~c;
                    const uint32_t first = w >> 3, count = (w & 7u) + 1u;
                    for (uint32_t j = 0; j < count; ++j) {
                        float t, id;
                        if (hit_leaf(wr, o, d, p.tris + first + j, t, id) && t < tmax) {
                            hit = true;
                            break;
                        }
                    }
                    continue;
                }
                if (nearest < 0) { nearest = c; tbest = tn; continue; }
                int32_t push = c;
                if (tn < tbest) { push = nearest; nearest = c; tbest = tn; }
                if (sp >= kStackN) { overflow = true; continue; }
                stack[sp++] = push;
            }
            if (overflow) { atomicOr(p.err_word, DEV_STACK_OVERFLOW); active = false; continue; }
            if (hit) { active = false; continue; }
            if (++guard >= kGuard) { atomicOr(p.err_word, DEV_GUARD); active = false; continue; }
            if (nearest >= 0) { cur = nearest; continue; }
            if (sp > 0) { cur = stack[--sp]; continue; }
            active = false;                              // nothing within the radius: open
            atomicAdd(&opens[q], 1);
        }
        __syncwarp();
        if (covered) {
            // no geometry: every ray is open
            const int open = p.has_geometry ? opens[lane] : p.spp;
            p.ao[i] = fdiv((float)open, (float)p.spp);
            if (p.mirror) mirror_ao(p.mirror, np)[i] = p.ao[i];
        }
        __syncwarp();                              // the frontier and counts are reused by the next packet
    }
}

__global__ void occluded_kernel(const Node4* __restrict__ nodes, const LeafTri* __restrict__ tris, int has_geometry,
                                float short_dir,
                                const float* __restrict__ rays, const float* __restrict__ tmax, uint32_t n,
                                uint8_t* __restrict__ hit, uint32_t* err) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const v3 o = load3(rays + (size_t)i * 6), d = load3(rays + (size_t)i * 6 + 3);
    Counts cn;
    const float tm = tmax[i];
    hit[i] = (has_geometry && walk<false>(nodes, tris, short_dir, o, d, tm, tm, err, cn) != 0) ? 1 : 0;
}

// AO of listed pixels with one thread per (pixel, sample): the same rays and hit rule as
// trace_packet (AO only), for pixel sets too small or too uneven to keep packets of pixels
// busy (the surrogate's fallback tiles). open[list[i]] receives pixel list[i]'s open rays,
// added by one atomic per warp and pixel.
__global__ void __launch_bounds__(256) ao_samples_kernel(const __grid_constant__ TraceParams p,
                                                         const uint32_t* __restrict__ list,
                                                         const uint32_t* __restrict__ count,
                                                         uint32_t* __restrict__ open) {
    const uint64_t total = (uint64_t)(*count) * (uint32_t)p.spp;
    const uint64_t stride = (uint64_t)gridDim.x * blockDim.x;
    const uint64_t base = (uint64_t)blockIdx.x * blockDim.x;
    Counts cn;
    // whole warps step together, so the per-warp vote below sees every lane
    for (uint64_t w0 = base; w0 < total; w0 += stride) {
        const uint64_t w = w0 + threadIdx.x;
        const bool valid = w < total;
        uint32_t px = 0xFFFFFFFFu;
        int o = 0;
        if (valid) {
            px = list[w / (uint32_t)p.spp];
            const uint32_t s = (uint32_t)(w % (uint32_t)p.spp);
            const uint32_t x = px % (uint32_t)p.w, y = px / (uint32_t)p.w;
            const v3 P = load3(p.pos + 3 * (size_t)px), n = load3(p.nrm + 3 * (size_t)px);
            const v3 a = fabsf(n.x) > 0.9f ? mk(0.0f, 1.0f, 0.0f) : mk(1.0f, 0.0f, 0.0f);
            const v3 t = normalize(cross(a, n)), b = cross(n, t);
            const v3 origin = add(P, scale(n, 1e-3f));
            const v3 dir = sample_direction(t, b, n, x, y, s, p.corr);
            const int h = p.has_geometry ? walk<false>(p.nodes, p.tris, p.short_dir, origin, dir, p.radius, p.radius, p.err_word, cn) : 0;
            o = (h & HIT_NEAR) ? 0 : 1;
        }
        const unsigned peers = __match_any_sync(0xffffffffu, px);
        const int sum = __popc(__ballot_sync(0xffffffffu, o) & peers);
        if (valid && (__ffs(peers) - 1) == (int)(threadIdx.x & 31u) && sum) atomicAdd(open + px, (uint32_t)sum);
    }
}

}  // namespace

int launch_ao_samples(const TraceParams& p, const uint32_t* list, const uint32_t* count, uint32_t* open,
                      int sm_count, cudaStream_t s) {
    ao_samples_kernel<<<sm_count * 8, 256, 0, s>>>(p, list, count, open);
    return cudaGetLastError() == cudaSuccess ? RN_OK : RN_ERR_CUDA;
}

// Lanes a pixel's samples are shared by (log2). A frame of few packets a warp leaves the last
// packets' samples, a pixel's one after the other, on few warps; with two or four lanes a pixel
// the packets are smaller and as many times more. A packet's own work (its frontier, its pixels'
// frames) is then done more often, which counts where walks are short: a small tree with the sky,
// where most rays end in the sieve, or few samples a lane. Measured one / two / four lanes, us:
// 512 x 512 x 64 (2.2 packets a warp) built-in scene with sky 199 / 168 / 184, without 157 / 107 /
// 87, 146k triangles 3336 / 2693 / 2394 and 1542 / 932 / 782; 256 x 256 x 64 (0.6) 143 / 102 / 75
// and 2581 / 1461 / 862; 1024 x 768 x 32 (6.7) 212 / 248 / 306, without sky 105 / 100 / 137, 146k
// 3539 / 3379 / 3360 and 1095 / 937 / 1022; 1283 x 723 x 16 (8) 135 / 169, without 71 / 78, 146k
// 2046 / 1942 and 633 / 652; 1920 x 1080 x 16 (18) 275 / 355, 146k 4060 / 4068 and 1087 / 1179.
// The small tree with the sky, one / two lanes by packets a warp: 16 samples 70.0 / 68.1 at 2.8, 73.2 /
// 75.5 at 3.2, 83.0 / 93.8 at 4.2; 32 samples 128 / 126 at 3.8, 134 / 138 at 4.2; 64 samples 236 / 220 at
// 4.2, 253 / 249 at 4.8. Up to nine packets two lanes are the faster on deeper trees and from 32
// samples without the sky (8.8 packets: 106 / 105, 146k triangles 1038 / 923 and with sky 4241 / 4100).
int lanes_log2(const TraceParams& p, long warps) {
    const long tw = 1L << p.packet_log2, th = 32 >> p.packet_log2;
    const double r = (double)(((p.w + tw - 1) / tw) * ((p.h + th - 1) / th)) / (double)warps;
    const bool deep = p.stack_need >= stack_need(6);           // a tree of six levels and more
    if (p.spp >= 32 && r < (p.want_sky && !deep ? 1.5 : 3.0)) return 2;
    const double sky = deep ? 9.0 : p.spp >= 64 ? 4.5 : p.spp >= 32 ? 4.0 : 3.0;
    return p.spp >= 16 && r < (p.want_sky ? sky : p.spp >= 32 ? 9.0 : 4.0) ? 1 : 0;
}

// The samples up to which a packet runs in the form for few (trace_packet). AO from the frontier
// gains by it for longer than frames with the sky, and most in deep trees, whose rays mostly go on
// past the sieve (radius 1 at 1920 x 1080, 4 and 8 samples: 744k triangles 773 -> 692 and 1306 ->
// 1219 us, 7.88M 1135 -> 1039 and 1995 -> 1890; 14 triangles, radius 3, 4 samples 125 -> 120, but 6
// and 8: 141 -> 149, 156 -> 176).
int few_spp(const TraceParams& p) {
    if (p.frontier != FRONTIER_NEAR || p.want_sky) return 2;
    return p.stack_need >= stack_need(6) ? 8 : 4;              // a tree of six levels and more
}

// Residency variants: the register budget decides how many 256-thread blocks share an SM
// (2: up to 128 registers, 3: 80, 4: 64, with spills to L1). The launch uses enough
// blocks to fill every SM at that residency; ctx().tune.trace_min_blocks picks the variant.
// Stack variants: 48 entries where the tree's bound (17 + 3 x wide depth) fits, else 96.
// The counting build (traversal statistics) always uses the 96-entry stack and tests each leaf as
// its child is met; the others test a node's leaves after its four slab tests (a kernel that tests
// them as they are met took 0.98 to 1.9 times as long with one lane a pixel, 14 to 744k triangles,
// and up to 4 times where lanes would share one).
template <int kMB, int kStackN>
void launch_variant(const TraceParams& p, int sm_count, cudaStream_t s, uint32_t* tile_ctr, unsigned long long* counts,
                    uint32_t stride) {
    const int blocks = sm_count * kMB;
    const int pool = ctx().tune.trace_pool;
    if (counts)
        trace_kernel<true, kMB, kStack, false, 0><<<blocks, 256, 0, s>>>(p, tile_ctr, counts, stride < 1 ? 1 : stride);
    else if (pool > 0 && !p.want_sky && p.short_dir == kShortDir)      // no far scene (its make_inv)
        trace_ao_pool_kernel<kMB, kStackN><<<blocks, 256, 0, s>>>(p, tile_ctr, pool, ctx().tune.trace_pool_sort);
    else if (p.spp <= few_spp(p))
        trace_kernel<false, kMB, kStackN, true, 0, true><<<blocks, 256, 0, s>>>(p, tile_ctr, nullptr, 1);
    else
        switch (lanes_log2(p, 8L * blocks)) {
            case 2: trace_kernel<false, kMB, kStackN, true, 2><<<blocks, 256, 0, s>>>(p, tile_ctr, nullptr, 1); break;
            case 1: trace_kernel<false, kMB, kStackN, true, 1><<<blocks, 256, 0, s>>>(p, tile_ctr, nullptr, 1); break;
            default: trace_kernel<false, kMB, kStackN, true, 0><<<blocks, 256, 0, s>>>(p, tile_ctr, nullptr, 1);
        }
}

template <int kStackN>
void launch_stack(const TraceParams& p, int sm_count, cudaStream_t s, uint32_t* tile_ctr, unsigned long long* counts,
                  uint32_t stride) {
    switch (ctx().tune.trace_min_blocks) {
        case 2: launch_variant<2, kStackN>(p, sm_count, s, tile_ctr, counts, stride); break;
        case 4: launch_variant<4, kStackN>(p, sm_count, s, tile_ctr, counts, stride); break;
        default: launch_variant<3, kStackN>(p, sm_count, s, tile_ctr, counts, stride); break;
    }
}

int launch_trace(const TraceParams& p, int sm_count, cudaStream_t s, unsigned long long* counts, uint32_t stride) {
    // the tile counter sits in the word after the error word
    uint32_t* tile_ctr = p.err_word + 1;
    cudaMemsetAsync(tile_ctr, 0, 4, s);
    if (ctx().tune.trace_stack <= 48 && p.stack_need <= 48)
        launch_stack<48>(p, sm_count, s, tile_ctr, counts, stride);
    else
        launch_stack<kStack>(p, sm_count, s, tile_ctr, counts, stride);
    return cudaGetLastError() == cudaSuccess ? RN_OK : RN_ERR_CUDA;
}

int launch_occluded(const rn_accel& accel, const float* rays, const float* tmax, uint32_t n,
                    uint8_t* hit, uint32_t* err_word, cudaStream_t s) {
    if (n == 0) return RN_OK;
    occluded_kernel<<<(n + 255) / 256, 256, 0, s>>>(accel.d_nodes, accel.d_tris, accel.ntri > 0, short_dir(accel), rays, tmax, n, hit,
                                                       err_word);
    return cudaGetLastError() == cudaSuccess ? RN_OK : RN_ERR_CUDA;
}

}  // namespace rn
