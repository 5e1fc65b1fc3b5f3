// trace_device.cuh -- the AO walk and the per-pixel loop of the ray-traced pass, shared by
// the single-frame kernel (trace.cu) and the batched multi-view kernel (batch.cu). See
// trace.cu for the design and the exactness argument.
#pragma once
#include "rn_internal.h"
#include "rn_device.cuh"

namespace rn {
namespace trace_dev {


constexpr int kStack = 96;
constexpr uint32_t kGuard = 1u << 24;       // node visits per ray before giving up
constexpr int kTileW = 8, kTileH = 4;

// inverse(d) of src/renderer/bvh.cpp:29-33: 1/x, a signed infinity for a zero component.
// The slab tests only prune, so 1/x need not be correctly rounded: the hardware reciprocal
// (rcp.approx, at most 1 ulp off) scales each axis's plane distances by at most 1 +- 2^-23, and a
// box the ray truly enters then still passes t0 <= t1 x (1 + 2^-22 or so), inside the test's exit
// widening of 1.0000008 (about 1 + 2^-20.2).
__device__ __forceinline__ float rcp_approx(float x) {
    float r;
    asm("rcp.approx.f32 %0, %1;" : "=f"(r) : "f"(x));
    return r;
}
// For directions with a component of 1e-3 or more: reciprocals within +-1e27. An infinite one
// makes plane * inv - o * inv NaN on both planes of most boxes: the axis constrains nothing, and a
// ray straight along an axis visits every node (a sample whose u is exactly zero is the normal
// itself, one in 2^24: 12 ms of one warp over 146k triangles, 800 x 600 x 64 samples 14.9 -> 4.2 ms,
// 1280 x 720 x 64 16.8 -> 7.3). At 1e27 a plane's distance says on which side of it the origin
// lies, its rounding 2^-24 |o| of position, inside the boxes' padding; a component below 1e-27 moves
// the ray by less than that over any distance the others leave in the scene. From |o| = 3.4e11 on
// o * inv is infinite, and such a ray stays beyond that coordinate: its boxes are culled, rightly
// where the scene lies within kFarCoord (else see careful_inv).
constexpr float kInvMax = 1e27f;
static_assert(kFarCoord * kInvMax < 3.4e38f, "o * inv is finite within kFarCoord");
__device__ __forceinline__ float inv_clamped(float x) { return fminf(fmaxf(rcp_approx(x), -kInvMax), kInvMax); }
// For any direction: a component below 1e-28 that is not zero gives NaN, so that its axis
// constrains nothing: with its reciprocal one of plane * inv and o * inv could overflow alone
// and cull a box that the ray enters.
__device__ __forceinline__ float safe_inv(float x) {
    return fabsf(x) < 1e-28f && x != 0.0f ? __int_as_float(0x7fffffff) : rcp_approx(x);
}

// Three-input maximum and minimum (one instruction each on sm_100 and later); a NaN operand
// is left out, as fmaxf and fminf leave it out.
__device__ __forceinline__ float max3(float a, float b, float c) {
    float r;
    asm("max.f32 %0, %1, %2, %3;" : "=f"(r) : "f"(a), "f"(b), "f"(c));
    return r;
}
__device__ __forceinline__ float min3(float a, float b, float c) {
    float r;
    asm("min.f32 %0, %1, %2, %3;" : "=f"(r) : "f"(a), "f"(b), "f"(c));
    return r;
}

// The ray's inverse direction, origin x inverse direction, and the byte offset of each axis's
// near plane in a node (nx, ny, nz: the lo plane for a direction that is not negative, else
// the hi plane 16 bytes further; the far plane sits at the other of the two), formed once
// per walk.
struct Inv { float x, y, z, ox, oy, oz; uint32_t nx, ny, nz; };
// One axis of a ray with a short direction or in a far scene: the reciprocal, a finite one kept
// where its product with the origin is finite too (else both planes of every box lie at the same
// infinity and the boxes that the ray enters are culled). At that limit a plane of a box around the
// origin is still more than 5e32 away: its padding, 2^-19 of the coordinate, times the reciprocal.
__device__ __forceinline__ float careful_inv(float o, float d, float inv, bool is_short) {
    if (is_short) inv = safe_inv(d);
    const float lim = 3e38f * rcp_approx(fabsf(o));
    return fabsf(inv) > lim && !isinf(inv) ? copysignf(lim, inv) : inv;
}
// short_dir: the tree's (rn::short_dir), so a scene with far coordinates costs the others nothing
// (a test of each origin's size: 0.5 to 1 % of every frame). kUnit: the direction is about of unit
// length and the origin within kFarCoord.
template <bool kUnit = false>
__device__ __forceinline__ Inv make_inv(const v3& o, const v3& d, float short_dir) {
    Inv r;
    r.x = inv_clamped(d.x); r.y = inv_clamped(d.y); r.z = inv_clamped(d.z);
    if (!kUnit) {
        const float longest = max3(fabsf(d.x), fabsf(d.y), fabsf(d.z));
        if (!(longest >= short_dir)) {
            const bool is_short = !(longest >= kShortDir);
            r.x = careful_inv(o.x, d.x, r.x, is_short);
            r.y = careful_inv(o.y, d.y, r.y, is_short);
            r.z = careful_inv(o.z, d.z, r.z, is_short);
        }
    }
    r.ox = o.x * r.x; r.oy = o.y * r.y; r.oz = o.z * r.z;
    r.nx = (__float_as_uint(r.x) >> 31) * 16u;
    r.ny = 32u + (__float_as_uint(r.y) >> 31) * 16u;
    r.nz = 64u + (__float_as_uint(r.z) >> 31) * 16u;
    return r;
}

// Slab test of one box from its near and far planes along the ray (near = lo where the
// direction is positive, hi where it is negative), each plane distance as one fused
// multiply-add, plane * inv - o * inv. The BVH only prunes, so the test has to be
// conservative, not exact: against (plane - o) * inv the fused form is off by at most about
// 2^-24 |o| in position, far inside the child boxes' outward padding (2^-19 of the coordinate
// plus 1e-6 of the extent), so no box a triangle hit lies in is culled. A rounded product is
// monotonic in the plane, so picking the planes by the direction's sign gives the values that
// the smaller and larger of the two distances had. A plane whose distance is NaN (a
// vanishing component of a short direction, products that overflow) constrains nothing.
__device__ __forceinline__ bool slab_nf(float nx, float fx, float ny, float fy, float nz, float fz, const Inv& iv,
                                        float tmax, float& tnear) {
    const float ax = __fmaf_rn(nx, iv.x, -iv.ox), bx = __fmaf_rn(fx, iv.x, -iv.ox);
    const float ay = __fmaf_rn(ny, iv.y, -iv.oy), by = __fmaf_rn(fy, iv.y, -iv.oy);
    const float az = __fmaf_rn(nz, iv.z, -iv.oz), bz = __fmaf_rn(fz, iv.z, -iv.oz);
    const float t0 = max3(ax, ay, fmaxf(az, 0.0f)), t1 = min3(bx, by, fminf(bz, tmax));
    tnear = t0;
    return t0 <= t1 * 1.0000008f;
}
__device__ __forceinline__ bool slab(float lox, float hix, float loy, float hiy, float loz, float hiz, const Inv& iv,
                                     float tmax, float& tnear) {
    return slab_nf(iv.nx & 16u ? hix : lox, iv.nx & 16u ? lox : hix, iv.ny & 16u ? hiy : loy, iv.ny & 16u ? loy : hiy,
                   iv.nz & 16u ? hiz : loz, iv.nz & 16u ? loz : hiz, iv, tmax, tnear);
}

// The four slab tests of a node: its planes are read near and far by address (no select, no
// minimum or maximum of a plane pair), so a child costs six multiply-adds, four three-input
// minima and maxima, one multiply and one compare. hit[k] also says that child k exists: an
// unused slot holds an inverted box, which only a ray without a finite direction component
// can pass, and the child word kNoChild. Every traversal is bound by instruction issue: six
// batched views of 744k triangles 36.8 -> 33.5 ms against selects and pairwise minima, the path
// tracer's room 38.8 -> 33.2; two planes per packed multiply-add: 27.3 -> 26.4 ms later on.
__device__ __forceinline__ uint64_t pack2(float a, float b) {
    uint64_t r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b));
    return r;
}
__device__ __forceinline__ void fma2(float& a, float& b, float x, float y, uint64_t m, uint64_t c) {
    asm("{\n.reg .b64 t;\nmov.b64 t, {%2, %3};\nfma.rn.f32x2 t, t, %4, %5;\nmov.b64 {%0, %1}, t;\n}\n"
        : "=f"(a), "=f"(b) : "f"(x), "f"(y), "l"(m), "l"(c));
}
template <typename L>
__device__ __forceinline__ void node_test(const char* node, L ld, const Inv& iv, float tmax, int32_t (&CH)[4],
                                          float (&tn)[4], bool (&hit)[4]) {
    const float4 nx = ld(node + iv.nx), fx = ld(node + (iv.nx ^ 16u));
    const float4 ny = ld(node + iv.ny), fy = ld(node + (iv.ny ^ 16u));
    const float4 nz = ld(node + iv.nz), fz = ld(node + (iv.nz ^ 16u));
    const float4 ch = ld(node + 96);
    const uint64_t ix = pack2(iv.x, iv.x), iy = pack2(iv.y, iv.y), iz = pack2(iv.z, iv.z);
    const uint64_t ox = pack2(-iv.ox, -iv.ox), oy = pack2(-iv.oy, -iv.oy), oz = pack2(-iv.oz, -iv.oz);
    float ax[4], bx[4], ay[4], by[4], az[4], bz[4];
    fma2(ax[0], ax[1], nx.x, nx.y, ix, ox); fma2(ax[2], ax[3], nx.z, nx.w, ix, ox);
    fma2(bx[0], bx[1], fx.x, fx.y, ix, ox); fma2(bx[2], bx[3], fx.z, fx.w, ix, ox);
    fma2(ay[0], ay[1], ny.x, ny.y, iy, oy); fma2(ay[2], ay[3], ny.z, ny.w, iy, oy);
    fma2(by[0], by[1], fy.x, fy.y, iy, oy); fma2(by[2], by[3], fy.z, fy.w, iy, oy);
    fma2(az[0], az[1], nz.x, nz.y, iz, oz); fma2(az[2], az[3], nz.z, nz.w, iz, oz);
    fma2(bz[0], bz[1], fz.x, fz.y, iz, oz); fma2(bz[2], bz[3], fz.z, fz.w, iz, oz);
#pragma unroll
    for (int k = 0; k < 4; ++k) {
        const float t0 = max3(ax[k], ay[k], fmaxf(az[k], 0.0f)), t1 = min3(bx[k], by[k], fminf(bz[k], tmax));
        tn[k] = t0;
        hit[k] = t0 <= t1 * 1.0000008f;
    }
    CH[0] = __float_as_int(ch.x); CH[1] = __float_as_int(ch.y); CH[2] = __float_as_int(ch.z); CH[3] = __float_as_int(ch.w);
}
struct LdGlobal {
    __device__ __forceinline__ float4 operator()(const char* p) const { return __ldg(reinterpret_cast<const float4*>(p)); }
};
struct LdShared {
    __device__ __forceinline__ float4 operator()(const char* p) const { return *reinterpret_cast<const float4*>(p); }
};

// Per-thread traversal counters (the measurement build; compiled out otherwise).
struct Counts { unsigned long long rays = 0, nodes = 0, tris = 0, sky = 0; };

enum : int { HIT_NEAR = 1, HIT_FAR = 2 };

// A warp's frontier: BVH entries (a child word and its padded box) that together hold every
// triangle a short ray of the warp's tile can reach. A triangle hit at t < radius lies within
// radius of its ray's origin, so its leaf box, and every ancestor's, overlaps the box Q of
// the tile's origins grown by the radius; the frontier is the set of Q-overlapping nodes
// reached by expanding Q-overlapping nodes from the root, level by level, while at most
// kFrontier entries result. AO walks start from it instead of re-descending from the root.
// The entries are kept in the node layout, four to a group: a walk tests a group exactly as
// it tests a node.
constexpr int kFrontierNodes = kFrontier / 4;
struct FrontierBox { float lo[3], hi[3]; int32_t word; };
__device__ __forceinline__ void frontier_put(Node4* F, int e, const FrontierBox& b) {
    Node4& n = F[e >> 2];
    const int k = e & 3;
    n.lox[k] = b.lo[0]; n.loy[k] = b.lo[1]; n.loz[k] = b.lo[2];
    n.hix[k] = b.hi[0]; n.hiy[k] = b.hi[1]; n.hiz[k] = b.hi[2];
    n.child[k] = b.word;
}
__device__ __forceinline__ FrontierBox frontier_get(const Node4* F, int e) {
    const Node4& n = F[e >> 2];
    const int k = e & 3;
    return FrontierBox{{n.lox[k], n.loy[k], n.loz[k]}, {n.hix[k], n.hiy[k], n.hiz[k]}, n.child[k]};
}
__device__ __forceinline__ FrontierBox frontier_child(const Node4* N, int k) {
    return FrontierBox{{N->lox[k], N->loy[k], N->loz[k]}, {N->hix[k], N->hiy[k], N->hiz[k]}, N->child[k]};
}

__device__ __forceinline__ bool box_overlaps(float lx, float ly, float lz, float hx, float hy, float hz,
                                             const float* qlo, const float* qhi) {
    return lx <= qhi[0] && hx >= qlo[0] && ly <= qhi[1] && hy >= qlo[1] && lz <= qhi[2] && hz >= qlo[2];
}

// The tangent plane of a warp's packet where its covered pixels share one normal (flat
// surfaces): every hemisphere ray leaves its origin o with direction . n > 0 (the sampler's lz
// is sqrt(1 - u) >= 2.4e-4, far above the rounding of the frame and the direction), so a box
// that lies wholly below the lowest origin's plane holds no triangle that a ray of the packet
// can reach. `below` asks for 2e-6 of the coordinates more than that (16 units in the last
// place: the rounding of the support point's product, and of the triangle test, which may be
// off by a few ulps of the coordinates). Off (n all zero) when the normals differ or are far
// from unit length: nothing is then below. Six views of 744k triangles 31.2 -> 30.3 ms.
struct TilePlane { float nx, ny, nz, low, mag; };
__device__ __forceinline__ TilePlane tile_plane(const v3& n, const v3& o, bool covered, unsigned any) {
    const int first = __ffs(any) - 1;
    const v3 f = mk(__shfl_sync(0xffffffffu, n.x, first), __shfl_sync(0xffffffffu, n.y, first),
                    __shfl_sync(0xffffffffu, n.z, first));
    const float d2 = f.x * f.x + f.y * f.y + f.z * f.z;
    const bool alike = !covered || (fabsf(n.x - f.x) <= 1e-5f && fabsf(n.y - f.y) <= 1e-5f && fabsf(n.z - f.z) <= 1e-5f);
    if (!(__all_sync(0xffffffffu, alike) && d2 > 0.9f && d2 < 1.1f)) return TilePlane{0.0f, 0.0f, 0.0f, 0.0f, 0.0f};
    float low = covered ? f.x * o.x + f.y * o.y + f.z * o.z : 3.0e38f;
    float mag = covered ? fabsf(o.x) + fabsf(o.y) + fabsf(o.z) : 0.0f;
    for (int off = 16; off > 0; off >>= 1) {
        low = fminf(low, __shfl_xor_sync(0xffffffffu, low, off));
        mag = fmaxf(mag, __shfl_xor_sync(0xffffffffu, mag, off));
    }
    return TilePlane{f.x, f.y, f.z, low, mag};
}
__device__ __forceinline__ bool below(const TilePlane& t, float lx, float ly, float lz, float hx, float hy, float hz) {
    const float cx = t.nx > 0.0f ? hx : lx, cy = t.ny > 0.0f ? hy : ly, cz = t.nz > 0.0f ? hz : lz;
    const float m = 2e-6f * (fabsf(cx) + fabsf(cy) + fabsf(cz) + t.mag);
    return (t.nx != 0.0f || t.ny != 0.0f || t.nz != 0.0f) && t.nx * cx + t.ny * cy + t.nz * cz < t.low - m;
}

// A node's children in registers, a load for each plane: seven in flight.
struct NodeChildren {
    float4 lx, hx, ly, hy, lz, hz;
    int4 word;
    __device__ __forceinline__ explicit NodeChildren(const Node4* N) {
        const float4* q = reinterpret_cast<const float4*>(N);
        lx = __ldg(q); hx = __ldg(q + 1); ly = __ldg(q + 2); hy = __ldg(q + 3); lz = __ldg(q + 4); hz = __ldg(q + 5);
        word = __ldg(reinterpret_cast<const int4*>(q + 6));
    }
    static __device__ __forceinline__ float at(const float4& v, int k) { return k == 0 ? v.x : k == 1 ? v.y : k == 2 ? v.z : v.w; }
    __device__ __forceinline__ FrontierBox box(int k) const {
        return FrontierBox{{at(lx, k), at(ly, k), at(lz, k)}, {at(hx, k), at(hy, k), at(hz, k)},
                           k == 0 ? word.x : k == 1 ? word.y : k == 2 ? word.z : word.w};
    }
};
// The children of N (a bit each) that overlap Q and are not below the packet's plane. kWide: its
// planes are fetched together, and an unused slot tells by its word; else each value is fetched
// when it is needed, in fewer registers. Few samples are bound by these fetches, a dependent chain
// for each round: their kernel takes the wide form (AO of radius 0.02 at 1920 x 1080, 1 sample, 744k
// triangles 233 -> 202 us, 7.88M 275 -> 240), and so do batches (2560 x 1440 and 1281 x 723, 4
// samples, 744k triangles 2162 -> 2042 us). In the others it cost registers that the walks miss (14
// triangles, 3840 x 2160, 256 samples with sky 12.9 -> 13.2 ms).
template <bool kWide>
__device__ __forceinline__ unsigned frontier_hits(const Node4* N, const float* qlo, const float* qhi, const TilePlane& pl) {
    unsigned hit = 0;
    if (kWide) {
        const NodeChildren ch(N);
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            const FrontierBox b = ch.box(k);
            if (b.word != kNoChild && box_overlaps(b.lo[0], b.lo[1], b.lo[2], b.hi[0], b.hi[1], b.hi[2], qlo, qhi) &&
                !below(pl, b.lo[0], b.lo[1], b.lo[2], b.hi[0], b.hi[1], b.hi[2]))
                hit |= 1u << k;
        }
    } else {
        for (int k = 0; k < N->meta[0]; ++k)
            if (box_overlaps(N->lox[k], N->loy[k], N->loz[k], N->hix[k], N->hiy[k], N->hiz[k], qlo, qhi) &&
                !below(pl, N->lox[k], N->loy[k], N->loz[k], N->hix[k], N->hiy[k], N->hiz[k]))
                hit |= 1u << k;
    }
    return hit;
}
// The warp builds the frontier of box [qlo, qhi] into F (all 32 lanes call it); returns its
// size (0: start at the root; -1: nothing within reach). Breadth first: each round every entry
// that is an interior node is replaced by its children that overlap Q and are not below the
// packet's plane, the lanes expanding their entries in
// parallel (one node fetch per lane, a prefix sum over the lanes for the output slots),
// while the result stays within `cap` entries (kFrontier at most). A round costs one dependent node fetch,
// so the build takes about the tree's depth in fetch latencies. Up to `tail` greedy steps
// follow, each replacing the largest interior entry by its children while the frontier fits.
template <bool kWide>
__device__ inline int build_frontier(const Node4* __restrict__ nodes, const float* qlo, const float* qhi,
                                     const TilePlane& pl, Node4* F, int cap, int tail) {
    const int lane = (int)(threadIdx.x & 31u);
    int32_t word = 0;                       // lane 0 starts with the root node
    float lo[3] = {0.0f, 0.0f, 0.0f}, hi[3] = {0.0f, 0.0f, 0.0f};
    int n = 1, built = 0;
    for (int round = 0; round < 64; ++round) {
        const bool mine = lane < n;
        const bool inner = mine && word >= 0;
        const Node4* N = nodes + (inner ? word : 0);
        const unsigned hit = inner ? frontier_hits<kWide>(N, qlo, qhi, pl) : 0u;
        const int c = inner ? __popc(hit) : (mine ? 1 : 0);
        int incl = c;
        for (int off = 1; off < 32; off <<= 1) {
            const int v = __shfl_up_sync(0xffffffffu, incl, off);
            if (lane >= off) incl += v;
        }
        const int total = __shfl_sync(0xffffffffu, incl, 31);
        if (!__any_sync(0xffffffffu, inner) || total > cap) break;
        __syncwarp();                       // every lane has read its entry of the last round
        int pos = incl - c;
        if (inner) {
            if constexpr (kWide) {
                const NodeChildren ch(N);
#pragma unroll
                for (int k = 0; k < 4; ++k)
                    if (hit & (1u << k)) frontier_put(F, pos++, ch.box(k));
            } else {
                for (int k = 0; k < 4; ++k)
                    if (hit & (1u << k)) frontier_put(F, pos++, frontier_child(N, k));
            }
        } else if (mine) {
            frontier_put(F, pos, FrontierBox{{lo[0], lo[1], lo[2]}, {hi[0], hi[1], hi[2]}, word});
        }
        __syncwarp();
        n = total;
        built = 1;
        if (lane < n) {
            const FrontierBox e = frontier_get(F, lane);
            lo[0] = e.lo[0]; lo[1] = e.lo[1]; lo[2] = e.lo[2];
            hi[0] = e.hi[0]; hi[1] = e.hi[1]; hi[2] = e.hi[2];
            word = e.word;
        }
    }
    // then up to `tail` single steps, largest interior entry first, while the result fits
    for (int step = 0; built && step < tail; ++step) {
        const bool inner = lane < n && word >= 0;
        float best = inner ? fmaxf(fmaxf(hi[0] - lo[0], hi[1] - lo[1]), hi[2] - lo[2]) : -1.0f;
        int bl = lane;
        for (int off = 16; off > 0; off >>= 1) {
            const float ob = __shfl_xor_sync(0xffffffffu, best, off);
            const int ol = __shfl_xor_sync(0xffffffffu, bl, off);
            if (ob > best || (ob == best && ol < bl)) { best = ob; bl = ol; }
        }
        if (best < 0.0f) break;
        const Node4* N = nodes + (lane == bl ? word : 0);
        const unsigned hit = lane == bl ? frontier_hits<kWide>(N, qlo, qhi, pl) : 0u;
        const int c = __popc(__shfl_sync(0xffffffffu, hit, bl));
        if (n - 1 + c > cap) break;
        __syncwarp();
        if (lane == bl) {
            // the children replace entry bl and append after the last entry; none: the last
            // entry moves into slot bl
            int pos = bl;
            if (c == 0 && bl != n - 1) frontier_put(F, bl, frontier_get(F, n - 1));
            for (int k = 0; k < 4; ++k)
                if (hit & (1u << k)) {
                    frontier_put(F, pos, frontier_child(N, k));
                    pos = pos == bl ? n : pos + 1;
                }
        }
        __syncwarp();
        n = n - 1 + c;
        if (lane < n) {
            const FrontierBox e = frontier_get(F, lane);
            lo[0] = e.lo[0]; lo[1] = e.lo[1]; lo[2] = e.lo[2];
            hi[0] = e.hi[0]; hi[1] = e.hi[1]; hi[2] = e.hi[2];
            word = e.word;
        }
    }
    // the last group's unused slots: boxes no ray passes
    if (built && lane >= n && lane < ((n + 3) & ~3))
        frontier_put(F, lane, FrontierBox{{1e30f, 1e30f, 1e30f}, {-1e30f, -1e30f, -1e30f}, kNoChild});
    return built ? (n > 0 ? n : -1) : 0;
}

// One walk, two limits (tnear <= tfar): HIT_NEAR | HIT_FAR when some triangle is hit at
// 1e-4 < t < tnear; HIT_FAR alone when the nearest hit it needed to find lies in
// [tnear, tfar); 0 when nothing is hit before tfar. The any-hit query of raw::Bvh::occluded
// (src/renderer/bvh.cpp:119-138) is tnear == tfar.
// kLeafPass: a node's leaf children are tested after all four slab tests, in one loop over
// the leaves that passed (lanes whose leaves sit at different child positions test them
// together, and the triangle test exists once in the code instead of once per position).
// Either order finds the same answers: boxes are only culled against tmax >= tnear, and a
// far hit only lowers tmax to tnear.
// kNearest: of a node's interior children the nearest is descended into and the others stacked;
// else the first, without a comparison per child (any order finds the same answers). Short AO
// rays meet an occluder sooner in the nearest child, the path tracer's shadow rays do not gain
// what the comparisons cost (1080p room, 4 samples: 24.8 ms with them, 24.1 without).
template <bool kCount, int kStackN = kStack, bool kLeafPass = true, bool kNearest = true>
__device__ int walk(const Node4* __restrict__ nodes, const LeafTri* __restrict__ tris, float short_dir, const v3& o,
                    const v3& d, float tnear, float tfar, uint32_t* err, Counts& cn, const Node4* F = nullptr, int fn = 0) {
    const Inv iv = make_inv(o, d, short_dir);
    LeafRay wr;                          // the watertight set-up: formed at the first leaf
    bool wr_ready = false;
    float tmax = tfar;
    int far_hit = 0;
    int32_t stack[kStackN + 3];          // past kStackN: what the node that passes it pushes
    int sp = 0;
    int32_t cur = 0;                     // the root is always node 0
    // the triangles of leaf word c: true when one is hit nearer than tnear (the walk ends)
    auto leaf = [&](int32_t c) -> bool {
        if (c == kNoChild) return false;
        if (!wr_ready) { wr = make_leaf_ray(o, d); wr_ready = true; }
        const uint32_t w = (uint32_t)~c;
        const uint32_t first = w >> 3, count = (w & 7u) + 1u;
        for (uint32_t i = 0; i < count; ++i) {
            if (kCount) ++cn.tris;
            float t, id;
            if (!hit_leaf(wr, o, d, tris + first + i, t, id)) continue;
            if (t < tnear) return true;
            if (t < tmax) { far_hit = HIT_FAR; tmax = tnear; }
        }
        return false;
    };
    // The children that passed node_test: leaves are tested (true: one is hit nearer than tnear,
    // the walk ends), the nearest interior child so far stays in `nearest`, the others are
    // stacked. Written without branches up to the leaves, so a warp's lanes stay together
    // whatever mix of children each of them hit.
    int32_t nearest;
    float tbest;
    auto visit = [&](const int32_t (&CH)[4], const float (&tn)[4], const bool (&hit)[4]) -> bool {
        unsigned leaves = 0;
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            const int32_t c = CH[k];
            const bool in = hit[k] && c >= 0;
            if (hit[k] && c < 0) {
                if (kLeafPass) leaves |= 1u << k;
                else if (leaf(c)) return true;
            }
            const bool closer = in && (kNearest ? tn[k] < tbest : nearest < 0);
            const int32_t push = closer ? nearest : c;
            if (in && nearest >= 0) stack[sp++] = push;
            nearest = closer ? c : nearest;
            tbest = closer ? tn[k] : tbest;
        }
        if (kLeafPass)
            while (leaves) {
                const int k = __ffs(leaves) - 1;
                leaves &= leaves - 1u;
                if (leaf(k == 0 ? CH[0] : k == 1 ? CH[1] : k == 2 ? CH[2] : CH[3])) return true;
            }
        return false;
    };
    if (fn > 0) {
        // start from the frontier: its entries are the root's stand-ins
        nearest = -1;
        tbest = 3.0e38f;
        for (int g = 0; 4 * g < fn; ++g) {            // at most kFrontier - 1 < kStackN entries stacked
            float tn[4];
            bool hit[4];
            int32_t CH[4];
            node_test(reinterpret_cast<const char*>(F + g), LdShared(), iv, tmax, CH, tn, hit);
            if (visit(CH, tn, hit)) return HIT_NEAR | HIT_FAR;
        }
        if (nearest >= 0) cur = nearest;
        else if (sp > 0) cur = stack[--sp];
        else return far_hit;
    }
    for (uint32_t guard = 0; guard < kGuard; ++guard) {
        if (kCount) ++cn.nodes;
        float tn[4];
        bool hit[4];
        int32_t CH[4];
        node_test(reinterpret_cast<const char*>(nodes + cur), LdGlobal(), iv, tmax, CH, tn, hit);
        // a node stacks at most three of its children, one of the last level none: a walk within
        // stack_need may visit a node with the stack full (the build refuses trees whose depth
        // could need more)
        if (sp > kStackN) { atomicOr(err, DEV_STACK_OVERFLOW); return far_hit; }
        nearest = -1;
        tbest = 3.0e38f;
        if (visit(CH, tn, hit)) return HIT_NEAR | HIT_FAR;
        if (nearest >= 0) { cur = nearest; continue; }
        if (sp == 0) return far_hit;
        cur = stack[--sp];
    }
    atomicOr(err, DEV_GUARD);
    return far_hit;
}

// The nearest hit of raw::rt::closest (src/renderer/rt_bvh.cpp:125-152): the smallest t of the
// watertight test with 1e-4 < t < tmax, ties to the lowest triangle index (leaf triangles carry
// their input index). Children are visited nearest entry first; a box is culled only when its
// (padded, exit-widened) slab entry passes the best t so far, so the answer is the scan's.
__device__ inline int walk_closest(const Node4* __restrict__ nodes, const LeafTri* __restrict__ tris, float short_dir,
                            const v3& o, const v3& d, float tmax, float& t_hit, uint32_t* err) {
    const Inv iv = make_inv(o, d, short_dir);
    const LeafRay wr = make_leaf_ray(o, d);
    float best = tmax;
    int best_tri = -1;
    int32_t stack[kStack];
    int sp = 0;
    int32_t cur = 0;
    for (uint32_t guard = 0; guard < kGuard; ++guard) {
        float tn[4];
        bool hit[4];
        int32_t CH[4];
        node_test(reinterpret_cast<const char*>(nodes + cur), LdGlobal(), iv, best, CH, tn, hit);
        // the leaves among them, tested in one loop
        unsigned leaves = 0;
#pragma unroll
        for (int k = 0; k < 4; ++k)
            if (hit[k] && CH[k] < 0) leaves |= 1u << k;
        while (leaves) {
            const int k = __ffs(leaves) - 1;
            leaves &= leaves - 1u;
            const int32_t c = k == 0 ? CH[0] : k == 1 ? CH[1] : k == 2 ? CH[2] : CH[3];
            if (c == kNoChild) continue;
            const uint32_t u = (uint32_t)~c;
            const uint32_t first = u >> 3, count = (u & 7u) + 1u;
            for (uint32_t i = 0; i < count; ++i) {
                float t, fid;
                if (!hit_leaf(wr, o, d, tris + first + i, t, fid)) continue;
                const int id = __float_as_int(fid);
                if (t < best || (best_tri >= 0 && t == best && id < best_tri)) {
                    best = t;
                    best_tri = id;
                }
            }
        }
        // the interior children that the ray still enters before `best`, sorted in registers
        // farthest first by five compare-exchanges (the others sort to the front as -1)
        const float lim = best * 1.0000008f;
#pragma unroll
        for (int k = 0; k < 4; ++k)
            if (!(hit[k] && CH[k] >= 0 && tn[k] <= lim)) { CH[k] = -1; tn[k] = 3.0e38f; }
        auto cx = [&](int a, int b) {
            const bool s = tn[a] < tn[b];
            const float ta = s ? tn[b] : tn[a], tb = s ? tn[a] : tn[b];
            const int32_t ca = s ? CH[b] : CH[a], cb = s ? CH[a] : CH[b];
            tn[a] = ta; tn[b] = tb; CH[a] = ca; CH[b] = cb;
        };
        cx(0, 1); cx(2, 3); cx(0, 2); cx(1, 3); cx(1, 2);
        // push the farther children, descend into the nearest
        if (sp + 3 > kStack) { atomicOr(err, DEV_STACK_OVERFLOW); t_hit = best; return best_tri; }
#pragma unroll
        for (int k = 0; k < 3; ++k)
            if (CH[k] >= 0) stack[sp++] = CH[k];
        if (CH[3] >= 0) { cur = CH[3]; continue; }
        // pop the next pushed node: its children meet the best hit found since
        if (sp == 0) { t_hit = best; return best_tri; }
        cur = stack[--sp];
    }
    atomicOr(err, DEV_GUARD);
    t_hit = best;
    return best_tri;
}

// The bounds of the packet's ray origins (o: the lane's, where `covered`; all 32 lanes call it).
struct TileBox { float lo[3], hi[3], mag; };
__device__ __forceinline__ TileBox tile_box(const v3& o, bool covered) {
    TileBox t{{3.0e38f, 3.0e38f, 3.0e38f}, {-3.0e38f, -3.0e38f, -3.0e38f}, 0.0f};
    if (covered) {
        t.lo[0] = t.hi[0] = o.x; t.lo[1] = t.hi[1] = o.y; t.lo[2] = t.hi[2] = o.z;
        t.mag = fmaxf(fmaxf(fabsf(o.x), fabsf(o.y)), fabsf(o.z));
    }
    for (int off = 16; off > 0; off >>= 1) {
        for (int a = 0; a < 3; ++a) {
            t.lo[a] = fminf(t.lo[a], __shfl_xor_sync(0xffffffffu, t.lo[a], off));
            t.hi[a] = fmaxf(t.hi[a], __shfl_xor_sync(0xffffffffu, t.hi[a], off));
        }
        t.mag = fmaxf(t.mag, __shfl_xor_sync(0xffffffffu, t.mag, off));
    }
    return t;
}
// The frontier of the warp's packet for AO walks of `radius` (all 32 lanes call it and build
// it together). Returns its size, 0: the walks start at the root, -1: no triangle is within
// reach. Below four samples, four entries for each: a round more costs a dependent fetch whatever
// the samples that start from it (213k triangles, 1920 x 1080, radius 3: 1 sample 271 us with 8
// entries, 264 with 4, 3 samples 562 with 24 and 546 with 12; 7.88M triangles, radius 1, 3 samples
// the other way, 821 and 852; 4 samples 1040 with 24, 1085 with 12).
template <bool kWide = false>
__device__ __forceinline__ int tile_frontier(const TraceParams& p, const TileBox& t, const TilePlane& pl, Node4* F) {
    float lo[3] = {t.lo[0], t.lo[1], t.lo[2]}, hi[3] = {t.hi[0], t.hi[1], t.hi[2]};
    if (lo[0] > hi[0]) return 0;
    // grow by the radius with margin for the rounding of t, |d| and the hit point
    const float g = p.radius * 1.0001f + 1e-5f * (t.mag + 1.0f);
    for (int a = 0; a < 3; ++a) { lo[a] -= g; hi[a] += g; }
    const int n = build_frontier<kWide>(p.nodes, lo, hi, pl, F, p.spp < 4 ? 4 * p.spp : kFrontier, p.frontier_tail);
    __syncwarp();
    return n;
}
// For walks that start at the root: its children that are not below the packet's plane, put
// into F as frontier entries (all 32 lanes call it). Returns their number, -1: none.
__device__ __forceinline__ int root_frontier(const Node4* __restrict__ nodes, const TilePlane& pl, Node4* F) {
    const int lane = (int)(threadIdx.x & 31u);
    bool live = false;
    if (lane < nodes->meta[0])
        live = !below(pl, nodes->lox[lane], nodes->loy[lane], nodes->loz[lane], nodes->hix[lane], nodes->hiy[lane],
                      nodes->hiz[lane]);
    const unsigned m = __ballot_sync(0xffffffffu, live);
    const int n = __popc(m);
    if (live) frontier_put(F, __popc(m & ((1u << lane) - 1u)), frontier_child(nodes, lane));
    if (lane >= n && lane < 4)
        frontier_put(F, lane, FrontierBox{{1e30f, 1e30f, 1e30f}, {-1e30f, -1e30f, -1e30f}, kNoChild});
    __syncwarp();
    return n > 0 ? n : -1;
}

// Hemisphere direction of sample s of pixel (ux, uy) with frame (t, b, n): the arithmetic of
// trace_packet's below (src/renderer/ray_ao.cpp:30-37), for callers that trace one
// sample per thread.
__device__ __forceinline__ v3 sample_direction(const v3& t, const v3& b, const v3& n, uint32_t ux, uint32_t uy,
                                               uint32_t s, const uint8_t* __restrict__ corr) {
    const uint32_t k2 = hash24(ux, uy, 2u * s + 1u);
    const float u1 = unit24(hash24(ux, uy, 2u * s));
    float c, sn;
    angle_sincos(sample_angle(k2), sn, c);
    if (corr) apply_corr(__ldg(corr + k2), c, sn);
    const float r = fsqrt(u1);
    const float lx = fmul(r, c), ly = fmul(r, sn);
    const float lz = fsqrt(smax(0.0f, fsub(1.0f, u1)));
    return normalize(add(add(scale(t, lx), scale(b, ly)), scale(n, lz)));
}

// The sieve's rays are rough: the direction to 1e-5 (hardware sine, cosine and roots, no table
// byte, not normalized: |n| is within a few percent of one), and the entries of F grown by 2e-5
// of the distance to their farthest corner from any origin of the packet, so that the rough ray
// enters the grown box wherever the exact ray enters the box.
__device__ __forceinline__ void grow_entries(Node4* F, int n, const TileBox& t) {
    const int lane = (int)(threadIdx.x & 31u);
    if (lane < n) {
        FrontierBox b = frontier_get(F, lane);
        float d = 0.0f;
        for (int a = 0; a < 3; ++a) d += fmaxf(b.hi[a] - t.lo[a], t.hi[a] - b.lo[a]);
        const float g = 2e-5f * d;
        for (int a = 0; a < 3; ++a) { b.lo[a] -= g; b.hi[a] += g; }
        frontier_put(F, lane, b);
    }
    __syncwarp();
}
__device__ __forceinline__ float sqrt_rough(float x) {
    float r;
    asm("sqrt.approx.f32 %0, %1;" : "=f"(r) : "f"(x));
    return r;
}
// sample_direction to 1e-5, of about unit length. The radius keeps its exact u (the root of a
// small one would feel its last bit); the angle is taken less pi, where the hardware's sine and
// cosine are good to 2^-21.
__device__ __forceinline__ v3 rough_direction(const v3& t, const v3& b, const v3& n, uint32_t ux, uint32_t uy, uint32_t s) {
    const float u1 = unit24(hash24(ux, uy, 2u * s));
    const float ang = (one_plus(hash24(ux, uy, 2u * s + 1u)) - 1.5f) * 6.2831853f;
    const float r = -sqrt_rough(u1), lz = sqrt_rough(1.0f - u1);
    const float lx = r * __cosf(ang), ly = r * __sinf(ang);
    return mk(__fmaf_rn(t.x, lx, __fmaf_rn(b.x, ly, n.x * lz)), __fmaf_rn(t.y, lx, __fmaf_rn(b.y, ly, n.y * lz)),
              __fmaf_rn(t.z, lx, __fmaf_rn(b.z, ly, n.z * lz)));
}
// Whether a walk along the rough direction d has anything to descend into: any of the fn grown
// entries of F is entered before tmax.
__device__ __forceinline__ bool walk_starts(const v3& o, const v3& d, float tmax, const Node4* F, int fn) {
    const Inv iv = make_inv<true>(o, d, kShortDir);
    bool any;
    int g = 0;
    do {
        float tn[4];
        bool hit[4];
        int32_t CH[4];
        node_test(reinterpret_cast<const char*>(F + g), LdShared(), iv, tmax, CH, tn, hit);
        any = hit[0] || hit[1] || hit[2] || hit[3];
    } while (4 * ++g < fn && !any);
    return any;
}

// A packet of 32 pixels, one per lane (`valid`: the lane's pixel is in the frame; all 32 lanes
// call it): the spp cosine-weighted rays of each (AO and, when asked, the sky), then the sun
// ray.
//
// The sieve. Where most rays miss everything at the root (open scenes: 0.18 triangle tests a
// ray on the built-in scene), the few lanes whose rays go on hold the others of their warp, in
// every sample round. So the samples run in chunks of 64: first every lane tests its chunk's
// rays against the root (or the frontier) alone, all lanes together, and keeps a bit for each
// that enters a box; then each lane walks its own remaining samples one after the other,
// whatever their numbers, and the rounds left are the longest lane's count of them. The
// open and free counts are integers, so the order changes no bit. Where more than kSieveNum /
// kSieveDen of the rays go on, the first pass only costs: the warp then walks every sample
// directly, and looks again after kSieveSkip packets (`skip`, kept by the warp). Measured: the
// built-in scene at 3840 x 2160, 256 spp with sky 25.4 -> 18.9 ms with exact rays in the sieve,
// 18.0 -> 13.2 with rough ones; views of 744k triangles within 1 % either way (thresholds of
// 3/8, 5/8, 8/8: 22.0, 19.2 ms, and views 33.6 ms against 33.1).
// Few samples (kFew) take none of this: what the packet's rays share then costs
// more than it saves (built-in scene with sky, 2561 x 1441, 1 sample 155 -> 136 us; from 3 samples
// on the sieve is the faster one there). AO walks still start from the frontier.
// With kP > 0 a packet is 32 >> kP pixels and 1 << kP lanes share each (`part`, the lane's high
// bits): a part takes a run of the pixel's samples, part 0 the sun as well, and the counts are
// added up at the end; integers, so the split changes no bit.
constexpr int kChunk = 64, kSieveNum = 7, kSieveDen = 8, kSieveSkip = 15;
template <bool kCount, int kStackN = kStack, bool kLeafPass = true, int kP = 0, bool kFew = false, bool kWide = kFew>
__device__ __forceinline__ void trace_packet(const TraceParams& p, float short_dir, int x, int y, bool valid,
                                             const v3& toLight, Counts& cn, int& skip, Node4* F, int part = 0) {
    const bool lead = kP == 0 || part == 0;        // writes the pixel
    const int span = kP == 0 ? p.spp : (p.spp + (1 << kP) - 1) >> kP;      // a part's samples: first .. first + mine
    const int sbase = kP == 0 ? 0 : part * span, mine = kP == 0 ? p.spp : max(0, min(span, p.spp - sbase));
    const float kFar = 1e30f;
    const size_t i = valid ? (size_t)y * p.w + x : 0;
    const uint8_t m = valid ? p.mask[i] : 0;
    v3 P = mk(0.0f, 0.0f, 0.0f), n = P;
    if (valid) { P = load3(p.pos + 3 * i); n = load3(p.nrm + 3 * i); }
    if (valid && p.mirror && lead) {
        const size_t np = (size_t)p.w * p.h;
        store3(mirror_pos(p.mirror, np) + 3 * i, P);
        store3(mirror_nrm(p.mirror, np) + 3 * i, n);
        mirror_mask(p.mirror, np)[i] = m;
        if (!m) mirror_ao(p.mirror, np)[i] = 1.0f;
    }
    if (valid && !m && lead) {
        p.ao[i] = 1.0f;
        if (p.want_sky) { p.sky[i] = 1.0f; p.sun[i] = 1.0f; }
    }
    const unsigned covered = __ballot_sync(0xffffffffu, m != 0);
    if (covered == 0) return;
    // basis (ray_ao.cpp:14-17)
    const v3 a = fabsf(n.x) > 0.9f ? mk(0.0f, 1.0f, 0.0f) : mk(1.0f, 0.0f, 0.0f);
    const v3 t = normalize(cross(a, n)), b = cross(n, t);
    const v3 origin = add(P, scale(n, 1e-3f));
    const uint32_t ux = (uint32_t)x, uy = (uint32_t)y;
    const float tfar_h = p.want_sky ? kFar : p.radius;
    const bool sun = p.want_sky && !p.sun_forced;
    const int slots = span + (sun ? 1 : 0);
    // what the packet's rays can reach: AO-only walks start from the entries within the radius, or
    // from the root's live children; the sky's start at the root, whose live children serve the
    // sieve (rebuilt for every packet)
    int fn = 0;
    bool sieve = false;
    const bool near = p.frontier == FRONTIER_NEAR && !p.want_sky;
    if (p.has_geometry && (near || (!kFew && (p.want_sky || (p.frontier && !kCount))))) {
        const TilePlane pl = tile_plane(n, origin, m != 0, covered);
        const TileBox tb = tile_box(origin, m != 0);
        fn = near ? tile_frontier<kWide>(p, tb, pl, F) : root_frontier(p.nodes, pl, F);
        // the sieve needs normals of about unit length (its rough rays are not normalized) and
        // origins whose products with a reciprocal stay finite (a rough ray off by 1e-5 that stays
        // beyond kFarCoord says nothing of the exact one)
        const float n2 = n.x * n.x + n.y * n.y + n.z * n.z;
        sieve = !kCount && !kFew && fn > 0 && skip == 0 && tb.mag <= kFarCoord && __all_sync(0xffffffffu, !m || (n2 > 0.9f && n2 < 1.1f));
        if (!kCount && fn > 0 && skip > 0) --skip;
        if (sieve) grow_entries(F, fn, tb);
    }
    int open = 0, freec = 0;
    bool lit = true;
    // sample s's direction from its angle's index k2 and correction byte (both fetched ahead)
    auto direction = [&](int s, uint32_t k2, int cb) -> v3 {
        const float u1 = unit24(hash24(ux, uy, (uint32_t)(2 * s)));
        float c, sn;
        angle_sincos(sample_angle(k2), sn, c);
        if (p.corr) apply_corr(cb, c, sn);
        const float r = fsqrt(u1);
        const float lx = fmul(r, c), ly = fmul(r, sn);
        const float lz = fsqrt(smax(0.0f, fsub(1.0f, u1)));
        return normalize(add(add(scale(t, lx), scale(b, ly)), scale(n, lz)));
    };
    uint32_t k2n = 0;
    int cbn = 0;
    auto fetch = [&](int s) {                      // the next sample's angle index and correction byte
        k2n = hash24(ux, uy, (uint32_t)(2 * s + 1));
        cbn = p.corr ? __ldg(p.corr + k2n) : 0;
    };
    // nothing within reach: every hemisphere ray is open and free, only the sun ray is left
    const bool walks = p.has_geometry && fn >= 0;
    const int first = walks ? 0 : span;
    if (!walks) {
        open = freec = mine;
        if (kCount && m) { cn.rays += mine; if (p.want_sky) cn.sky += mine; }
    }
    // slot s of the part's: a sample's walk, or the sun's; `next`: the sample whose angle to fetch
    // ahead (-1: none)
    auto slot = [&](int s, int next) {
        v3 dir;
        float tn, tf;
        if (s < span) {
            const uint32_t k2 = k2n;
            const int cb = cbn;
            if (next >= 0) fetch(next);
            dir = direction(sbase + s, k2, cb);
            tn = p.radius;
            tf = tfar_h;
        } else {
            dir = toLight;
            tn = tf = kFar;
        }
        // AO-only walks may start from the warp's frontier; the sky and the sun need the root
        const bool local = s < span && tf == p.radius;
        const int h = p.has_geometry
                          ? walk<kCount, kStackN, kLeafPass>(p.nodes, p.tris, short_dir, origin, dir, tn, tf, p.err_word, cn,
                                                             local ? F : nullptr, local ? fn : 0)
                          : 0;
        if (s < span) {
            if (kCount) { ++cn.rays; if (p.want_sky && !(h & HIT_NEAR)) ++cn.sky; }
            if (!(h & HIT_NEAR)) {
                ++open;
                if (!(h & HIT_FAR)) ++freec;
            }
        } else {
            lit = h == 0;
        }
    };
    if (kFew) {
        if (m && first < slots) {
            fetch(first);
            for (int s = first; s < slots; ++s) slot(s, s + 1);
        }
        __syncwarp();
    }
    for (int s0 = first; !kFew && s0 < slots; s0 += kChunk) {
        const int nslot = min(kChunk, slots - s0), nsamp = min(kChunk, span - s0);
        uint64_t todo = 0;
        if (kP == 0) {
            todo = m ? (nslot == 64 ? ~0ull : (1ull << nslot) - 1ull) : 0ull;
        } else if (m) {
            const int nb = min(kChunk, max(0, mine - s0));
            todo = nb == 64 ? ~0ull : (1ull << nb) - 1ull;
            if (lead && sun && span - s0 < kChunk) todo |= 1ull << (span - s0);
        }
        if (sieve && nsamp > 0) {
            uint64_t keep = todo;
            if (m)
                for (int k = 0; k < nsamp; ++k)
                    if ((kP == 0 || s0 + k < mine) &&
                        !walk_starts(origin, rough_direction(t, b, n, ux, uy, (uint32_t)(sbase + s0 + k)), 1.1f * tfar_h, F, fn)) {
                        keep &= ~(1ull << k);
                        ++open;
                        ++freec;
                    }
            todo = keep;
            const unsigned left = __reduce_add_sync(0xffffffffu, (unsigned)__popcll(keep));
            if (left * kSieveDen > (unsigned)(nsamp * __popc(covered)) * kSieveNum) {
                sieve = false;
                skip = kSieveSkip;
            }
        }
        if (todo) fetch(sbase + s0 + __ffsll((long long)todo) - 1);
        while (todo) {
            const int s = s0 + __ffsll((long long)todo) - 1;
            todo &= todo - 1ull;
            slot(s, todo ? sbase + s0 + __ffsll((long long)todo) - 1 : -1);
        }
        __syncwarp();
    }
#pragma unroll
    for (int o = 16; o >= 32 >> kP; o >>= 1) {     // the parts' counts
        open += __shfl_xor_sync(0xffffffffu, open, o);
        freec += __shfl_xor_sync(0xffffffffu, freec, o);
    }
    if (!m || !lead) return;
    p.ao[i] = fdiv((float)open, (float)p.spp);
    if (p.mirror) mirror_ao(p.mirror, (size_t)p.w * p.h)[i] = p.ao[i];
    if (p.want_sky) {
        p.sky[i] = fdiv((float)freec, (float)p.spp);
        p.sun[i] = lit ? 1.0f : 0.0f;
    }
}


}  // namespace trace_dev
}  // namespace rn
