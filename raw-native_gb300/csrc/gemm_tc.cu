// gemm_tc.cu -- the tensor-core GEMM of the learned AO surrogate: C = P * Q^T with P (M x K)
// and Q (N x K) in BF16, both K-major, accumulated in FP32 on sm_103a's fifth-generation
// tensor cores.
//
// One CTA of 128 threads computes one 128 x BN tile of C (BN = 32..256):
//   - warp 0, lane 0: TMA producer. Each 64-wide K step loads a 128 x 64 tile of P and a
//     BN x 64 tile of Q (cp.async.bulk.tensor, 128-byte swizzle) into one of 4 shared-memory
//     stages and signals the stage's "full" mbarrier with the byte count;
//   - warp 1: MMA issuer (convergent, an elected lane executing). Per stage, four tcgen05.mma.kind::f16 (M 128, N BN, K 16)
//     accumulate into a BN-column TMEM accumulator; tcgen05.commit releases the stage
//     ("empty" mbarrier) when its MMAs have read it, and a final commit signals "done";
//   - all four warps: epilogue. Each thread owns one row (its warp's TMEM lane quarter),
//     reads it with tcgen05.ld 16 columns at a time, adds the bias, applies ReLU, and stores
//     BF16 or FP32 (or adds FP32 atomically for split K).
// Every mbarrier wait is bounded; on a timeout the kernel sets the error word, waits
// (bounded) for its own copies in flight, frees its TMEM and returns.
#include "gemm_tc.h"
#include <cuda.h>
#include <cudaTypedefs.h>
#include <cuda_bf16.h>
#include <algorithm>
#include <mutex>
#include <type_traits>

namespace rn {
namespace tc {

constexpr int kStages = 4, kThreads = 128;
constexpr uint32_t kSpin = 1u << 24;      // try_wait rounds before a wait gives up

__device__ __forceinline__ uint32_t smem_u32(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }

// The thread's warp in its block, known to be the same for the whole warp.
__device__ __forceinline__ int warp_index() { return __shfl_sync(0xffffffffu, (int)(threadIdx.x >> 5), 0); }

__device__ __forceinline__ float2 add2(float2 a, float2 b) {
    uint64_t r;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(*reinterpret_cast<uint64_t*>(&a)), "l"(*reinterpret_cast<uint64_t*>(&b)));
    return *reinterpret_cast<float2*>(&r);
}

__device__ __forceinline__ void mbar_init(uint32_t bar, uint32_t count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bar), "r"(count) : "memory");
}
__device__ __forceinline__ void mbar_expect_tx(uint32_t bar, uint32_t bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
}
__device__ __forceinline__ bool mbar_wait(uint32_t bar, uint32_t parity, uint32_t limit = kSpin) {
    for (uint32_t i = 0; i < limit; ++i) {
        uint32_t ok;
        asm volatile(
            "{\n.reg .pred p;\nmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\nselp.u32 %0, 1, 0, p;\n}\n"
            : "=r"(ok)
            : "r"(bar), "r"(parity)
            : "memory");
        if (ok) return true;
    }
    return false;
}
__device__ __forceinline__ void tma_load_2d(uint32_t dst, const CUtensorMap* map, int x, int y, uint32_t bar) {
    asm volatile(
        "cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];" ::"r"(dst),
        "l"(reinterpret_cast<uint64_t>(map)), "r"(x), "r"(y), "r"(bar)
        : "memory");
}
// Shared-memory matrix descriptor: K-major, 128-byte swizzle, 8-row atoms 1024 bytes apart.
__device__ __forceinline__ uint64_t smem_desc(uint32_t addr) {
    uint64_t d = (uint64_t)((addr >> 4) & 0x3FFFu);          // start address
    d |= (uint64_t)((1024u >> 4) & 0x3FFFu) << 32;            // stride byte offset
    d |= (uint64_t)1 << 46;                                   // descriptor version
    d |= (uint64_t)2 << 61;                                   // 128-byte swizzle
    return d;
}
// The same for rows of 64 bytes (32 BF16): 64-byte swizzle, 8-row atoms 512 bytes apart.
__device__ __forceinline__ uint64_t smem_desc64(uint32_t addr) {
    uint64_t d = (uint64_t)((addr >> 4) & 0x3FFFu);
    d |= (uint64_t)((512u >> 4) & 0x3FFFu) << 32;
    d |= (uint64_t)1 << 46;
    d |= (uint64_t)4 << 61;                                   // 64-byte swizzle
    return d;
}
__device__ __forceinline__ void tma_load_4d(uint32_t dst, const CUtensorMap* map, int c, int x, int y, int b,
                                            uint32_t bar) {
    asm volatile(
        "cp.async.bulk.tensor.4d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4, %5}], [%6];" ::"r"(dst),
        "l"(reinterpret_cast<uint64_t>(map)), "r"(c), "r"(x), "r"(y), "r"(b), "r"(bar)
        : "memory");
}
// Instruction descriptor of tcgen05.mma.kind::f16: FP32 accumulator, BF16 A and B, both
// K-major, M = 128, N = n.
__host__ __device__ constexpr uint32_t instr_desc(int n) {
    return (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(n >> 3) << 17) | ((uint32_t)(kBM >> 4) << 24);
}
// Issued by a whole warp, one elected lane executing (the same lane each time): the warp stays
// convergent, so the operands can be formed in the uniform registers that the instruction
// reads. From a branch of one lane a row-ring MMA cost 84 to 130 cycles where the tensor pipe
// needs 35 to 60 (64 + 128 -> 64 channels at 1088 x 1920: 643 us so, 362 convergent).
__device__ __forceinline__ void tc_mma(uint32_t tmem, uint64_t a, uint64_t b, uint32_t idesc, uint32_t accumulate) {
    asm volatile(
        "{\n.reg .pred p, e;\nelect.sync _|e, 0xffffffff;\nsetp.ne.b32 p, %4, 0;\n@e tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n}\n" ::"r"(tmem),
        "l"(a), "l"(b), "r"(idesc), "r"(accumulate)
        : "memory");
}
__device__ __forceinline__ void tc_commit(uint32_t bar) {
    asm volatile(
        "{\n.reg .pred e;\nelect.sync _|e, 0xffffffff;\n@e tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];\n}\n" ::"r"(bar)
        : "memory");
}
__device__ __forceinline__ void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tmem_ld16(uint32_t taddr, uint32_t (&v)[16]) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];"
        : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]), "=r"(v[8]),
          "=r"(v[9]), "=r"(v[10]), "=r"(v[11]), "=r"(v[12]), "=r"(v[13]), "=r"(v[14]), "=r"(v[15])
        : "r"(taddr));
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
}

// Zeros into 32 consecutive TMEM columns of this warp's 32 lanes (its wait is separate:
// tcgen05.wait::st before the columns are handed to the MMAs).
__device__ __forceinline__ void tmem_zero32(uint32_t taddr) {
    asm volatile(
        "tcgen05.st.sync.aligned.32x32b.x32.b32 [%0], {%1, %1, %1, %1, %1, %1, %1, %1, %1, %1, %1, %1, %1, %1, %1, %1, "
        "%1, %1, %1, %1, %1, %1, %1, %1, %1, %1, %1, %1, %1, %1, %1, %1};" ::"r"(taddr), "r"(0u)
        : "memory");
}
__device__ __forceinline__ void tmem_wait_st() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }

// 32 consecutive TMEM columns of this warp's 32 lanes, the load and its wait in one
// statement (the registers are defined only once the wait has returned).
__device__ __forceinline__ void tmem_ld32(uint32_t taddr, uint32_t (&v)[32]) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x32.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, "
        "%16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%32];\n"
        "tcgen05.wait::ld.sync.aligned;"
        : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]), "=r"(v[8]),
          "=r"(v[9]), "=r"(v[10]), "=r"(v[11]), "=r"(v[12]), "=r"(v[13]), "=r"(v[14]), "=r"(v[15]), "=r"(v[16]),
          "=r"(v[17]), "=r"(v[18]), "=r"(v[19]), "=r"(v[20]), "=r"(v[21]), "=r"(v[22]), "=r"(v[23]), "=r"(v[24]),
          "=r"(v[25]), "=r"(v[26]), "=r"(v[27]), "=r"(v[28]), "=r"(v[29]), "=r"(v[30]), "=r"(v[31])
        : "r"(taddr)
        : "memory");
}

template <int BN>
__global__ void __launch_bounds__(kThreads, 1) tc_gemm_kernel(const __grid_constant__ CUtensorMap mapP,
                                                              const __grid_constant__ CUtensorMap mapQ,
                                                              const Epilogue e) {
    extern __shared__ uint8_t smem_raw[];
    uint8_t* smem = (uint8_t*)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
    constexpr uint32_t kABytes = kBM * kBK * 2, kBBytes = BN * kBK * 2;
    constexpr uint32_t kCols = BN < 32 ? 32 : BN;
    uint8_t* sA = smem;
    uint8_t* sB = smem + kStages * kABytes;
    uint64_t* bars = reinterpret_cast<uint64_t*>(sB + kStages * kBBytes);
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 2 * kStages + 1);
    __shared__ int s_abort;
    const int warp = warp_index(), lane = threadIdx.x & 31;
    const int m0 = blockIdx.x * kBM, n0 = blockIdx.y * BN;
    const int kbeg = blockIdx.z * e.k_per_split, nkb = e.k_per_split / kBK;
    auto full = [&](int s) { return smem_u32(&bars[s]); };
    auto empty = [&](int s) { return smem_u32(&bars[kStages + s]); };
    const uint32_t done = smem_u32(&bars[2 * kStages]);

    if (threadIdx.x == 0) {
        for (int s = 0; s < kStages; ++s) { mbar_init(full(s), 1); mbar_init(empty(s), 1); }
        mbar_init(done, 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        s_abort = 0;
    }
    if (warp == 1) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)),
                     "r"(kCols)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = __shfl_sync(0xffffffffu, *tmem_slot, 0);

    const uint32_t spin = e.spin ? e.spin : kSpin;
    if (warp == 0 && lane == 0) {
        // producer
        int issued = 0;
        for (int kb = 0; kb < nkb; ++kb) {
            const int s = kb % kStages;
            const uint32_t ph = (uint32_t)(kb / kStages) & 1u;
            if (!mbar_wait(empty(s), ph ^ 1u, spin)) { atomicOr(e.err, DEV_GUARD); s_abort = 1; break; }
            mbar_expect_tx(full(s), kABytes + kBBytes);
            if (e.withhold && kb == 0) continue;      // the self-test's missing copy: its stage never fills
            tma_load_2d(smem_u32(sA + s * kABytes), &mapP, kbeg + kb * kBK, m0, full(s));
            tma_load_2d(smem_u32(sB + s * kBBytes), &mapQ, kbeg + kb * kBK, n0, full(s));
            ++issued;
        }
        // the copies this thread issued must land before the CTA can leave
        for (int kb = issued > kStages ? issued - kStages : 0; kb < issued; ++kb)
            mbar_wait(full(kb % kStages), (uint32_t)(kb / kStages) & 1u, spin);
    } else if (warp == 1) {
        // MMA issuer
        const uint32_t idesc = instr_desc(BN);
        for (int kb = 0; kb < nkb; ++kb) {
            const int s = kb % kStages;
            const uint32_t ph = (uint32_t)(kb / kStages) & 1u;
            if (!__all_sync(0xffffffffu, mbar_wait(full(s), ph, spin))) {
                if (lane == 0) { atomicOr(e.err, DEV_GUARD); s_abort = 1; }
                break;
            }
            tc_fence_after();
            const uint32_t a0 = smem_u32(sA + s * kABytes), b0 = smem_u32(sB + s * kBBytes);
#pragma unroll
            for (int k = 0; k < kBK / 16; ++k)
                tc_mma(tmem, smem_desc(a0 + k * 32), smem_desc(b0 + k * 32), idesc, (kb | k) != 0 ? 1u : 0u);
            tc_commit(empty(s));
        }
        tc_commit(done);
    }
    // epilogue: thread t owns row m0 + t, TMEM lane t
    const bool ok = __all_sync(0xffffffffu, mbar_wait(done, 0, spin));    // warp-uniform: the loads below are .sync.aligned
    tc_fence_after();
    if (!ok && lane == 0) atomicOr(e.err, DEV_GUARD);
    const int abort_warp = __shfl_sync(0xffffffffu, *(volatile int*)&s_abort, 0);
    if (ok && !abort_warp) {
        const int row = m0 + warp * 32 + lane;
        const uint32_t tbase = tmem + ((uint32_t)(warp * 32) << 16);
#pragma unroll 1
        for (int c0 = 0; c0 < BN; c0 += 16) {
            uint32_t v[16];
            tmem_ld16(tbase + (uint32_t)c0, v);
            float f[16];
            const int col = n0 + c0;
#pragma unroll
            for (int j = 0; j < 16; ++j) {
                float x = __uint_as_float(v[j]);
                if (e.bias) x += e.bias[col + j];
                if (e.relu) x = fmaxf(x, 0.0f);
                f[j] = x;
            }
            const size_t o = (size_t)row * e.ldc + col;
            if (e.c16) {
                uint4 out[2];
                __nv_bfloat16* ob = reinterpret_cast<__nv_bfloat16*>(out);
#pragma unroll
                for (int j = 0; j < 16; ++j) ob[j] = __float2bfloat16_rn(f[j]);
                uint4* d4 = reinterpret_cast<uint4*>(e.c16 + o);
                d4[0] = out[0];
                d4[1] = out[1];
            }
            if (e.c32) {
                float4* d4 = reinterpret_cast<float4*>(e.c32 + o);
#pragma unroll
                for (int h = 0; h < 4; ++h) {
                    const float4 q = make_float4(f[4 * h], f[4 * h + 1], f[4 * h + 2], f[4 * h + 3]);
                    if (e.atomic) atomicAdd(d4 + h, q);
                    else d4[h] = q;
                }
            }
        }
    }
    tc_fence_before();
    __syncthreads();
    if (warp == 1)
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(kCols) : "memory");
}


// ------------------------------------------------------------------ implicit 3x3 convolution
// A persistent kernel: each CTA walks work items (128-pixel tile, BN-column slice) with a
// stride of the grid, keeping its barriers and TMEM across items. CB is the channel block of
// one K step (64: 128-byte rows and swizzle; 32: 64-byte rows and swizzle); a K step is
// (tap, source, channel block), taps outermost, matching the weights' column order
// tap * Cin + ci. Roles (10 warps):
//   - warp 0: TMA producer over all items' K steps, through a ring of kSt stages;
//   - warp 1: MMA issuer (an elected lane); item i accumulates into TMEM buffer i & 1 (2 x BN columns),
//     so the MMAs of item i + 1 run while the epilogue drains item i;
//   - warps 2..9: epilogue, two sets of four; warp w reads TMEM lanes 32 (w % 4) .. +31 (its row
//     quarter) of its set's columns, then releases the buffer.
// Every wait is bounded and also gives up when another role has aborted.
constexpr int kConvThreads = 192;

struct ConvArgs {
    int nsrc;
    int C0, C1;                 // channels of the sources
    int B, H, W, tw_log2;       // output (= input) geometry and tiling
    int tiles_x, tiles_y;       // tiles per image row / column
    int cin;                    // C0 + C1
    int n_slices;               // N / BN
    int items;                  // tiles x slices
    __nv_bfloat16* up16;        // optional 2x nearest-upsampled copy of the BF16 output
};

__device__ __forceinline__ bool mbar_wait_or_abort(uint32_t bar, uint32_t parity, volatile int* abort_flag) {
    for (uint32_t i = 0; i < kSpin; ++i) {
        uint32_t ok;
        asm volatile(
            "{\n.reg .pred p;\nmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\nselp.u32 %0, 1, 0, p;\n}\n"
            : "=r"(ok)
            : "r"(bar), "r"(parity)
            : "memory");
        if (ok) return true;
        if ((i & 255u) == 255u && *abort_flag) return false;
    }
    return false;
}
__device__ __forceinline__ void mbar_arrive(uint32_t bar) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory");
}

// kT tiles per work item (1 or 2): with 2, every weight box feeds two 128-pixel tiles (two
// A boxes per stage, two TMEM accumulators per buffer), halving the weights' L2 traffic;
// each tile's MMAs are the same in the same order.
// Pipeline stages of tc_conv_kernel: 8 of 32 channels or 4 of 64; pairs of tiles with a
// 64-column or narrower slice take half as many and single tiles with 64 columns one less, so that
// two CTAs still share an SM beside the epilogue's stage (96 -> 64 at 136 x 976, single tiles of 32
// channels: 8 stages and one CTA 49.6 us, 7 and two 31.2).
__host__ __device__ constexpr int conv_stages(int bn, int cb, int kt) {
    const int full = cb == 32 ? 8 : 4;
    return kt == 2 && bn <= 64 ? full / 2 : bn == 64 ? full - 1 : full;
}

constexpr int kTapThreads = 320;                // two sets of four epilogue warps
constexpr size_t kTapStage = 8 * 128 * 16;      // their stages
constexpr size_t kTapStatic = 2048 + 64;        // static shared memory: the bias, the abort flag
__host__ __device__ constexpr size_t conv_smem(int bn, int cb, int kt) {
    const int n = conv_stages(bn, cb, kt);
    return 1024 + (size_t)n * (kt * kBM * cb * 2 + bn * cb * 2) + kTapStage + (2 * n + 4) * 8 + 16;
}

template <int BN, int CB, int kT>
__global__ void __launch_bounds__(kTapThreads, 2) tc_conv_kernel(const __grid_constant__ CUtensorMap map0,
                                                                  const __grid_constant__ CUtensorMap map1,
                                                                  const __grid_constant__ CUtensorMap mapW,
                                                                  const ConvArgs a, const Epilogue e) {
    constexpr int kSt = conv_stages(BN, CB, kT);
    extern __shared__ uint8_t smem_raw[];
    uint8_t* smem = (uint8_t*)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
    constexpr uint32_t kABytes = kBM * CB * 2, kBBytes = BN * CB * 2;
    constexpr uint32_t kCols = 2 * kT * BN;                  // two buffers of kT accumulators
    uint8_t* sA = smem;                                      // kSt stages of kT A boxes
    uint8_t* sB = smem + kSt * kT * kABytes;
    uint4* s_stage = reinterpret_cast<uint4*>(sB + kSt * kBBytes);
    uint64_t* bars = reinterpret_cast<uint64_t*>(sB + kSt * kBBytes + kTapStage);
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 2 * kSt + 4);
    __shared__ int s_abort;
    __shared__ __align__(16) float s_bias[512];       // the bias of every output channel, staged once
    volatile int* abort_flag = &s_abort;
    const int warp = warp_index(), lane = threadIdx.x & 31;
    const int tw = 1 << a.tw_log2, th = kBM >> a.tw_log2;
    const int nb0 = a.C0 / CB, nb1 = a.nsrc > 1 ? a.C1 / CB : 0, per_tap = nb0 + nb1;
    const int nkb = 9 * per_tap;
    auto full = [&](int s) { return smem_u32(&bars[s]); };
    auto empty = [&](int s) { return smem_u32(&bars[kSt + s]); };
    auto acc_full = [&](int b) { return smem_u32(&bars[2 * kSt + b]); };
    auto acc_empty = [&](int b) { return smem_u32(&bars[2 * kSt + 2 + b]); };

    if (threadIdx.x == 0) {
        for (int s = 0; s < kSt; ++s) { mbar_init(full(s), 1); mbar_init(empty(s), 1); }
        for (int b = 0; b < 2; ++b) { mbar_init(acc_full(b), 1); mbar_init(acc_empty(b), 8); }
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        s_abort = 0;
    }
    if (e.bias)
        for (int i = threadIdx.x; i < a.n_slices * BN; i += blockDim.x) s_bias[i] = e.bias[i];
    if (warp == 1) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)),
                     "r"(kCols)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = __shfl_sync(0xffffffffu, *tmem_slot, 0);

    if (warp == 0) {
        // The warp fills the stages in order, all lanes waiting for the same one: lane 0 arms its
        // barrier, lanes 0 .. kT - 1 issue a tile's box each, lane kT the weights'. (A lane per
        // stage, each waiting for its own, held one another up: a lane suspended in try_wait
        // keeps the warp from the lane whose stage is free.) Stage, phase, tap and channel block
        // are kept by increment.
        uint32_t issued = 0, ph = 0;
        int s = 0;
        bool ok = true;
        for (int item = blockIdx.x; ok && item < a.items; item += gridDim.x) {
            const int group = item / a.n_slices, n0 = (item % a.n_slices) * BN;
            const int tile = group * kT + (lane < kT ? lane : 0);
            const int tx = tile % a.tiles_x, ty = (tile / a.tiles_x) % a.tiles_y, b = tile / (a.tiles_x * a.tiles_y);
            for (int tap = 0; ok && tap < 9; ++tap) {
                const int x = tx * tw + tap % 3 - 1, y = ty * th + tap / 3 - 1;
                for (int r = 0; r < per_tap; ++r) {
                    ok = __all_sync(0xffffffffu, mbar_wait_or_abort(empty(s), ph ^ 1u, abort_flag));
                    if (!ok) break;
                    if (lane == 0) mbar_expect_tx(full(s), kT * kABytes + kBBytes);
                    __syncwarp();
                    const bool second = r >= nb0;
                    const int cb = second ? r - nb0 : r;
                    if (lane < kT)
                        tma_load_4d(smem_u32(sA + (s * kT + lane) * kABytes), second ? &map1 : &map0, cb * CB, x, y, b, full(s));
                    else if (lane == kT)
                        tma_load_2d(smem_u32(sB + s * kBBytes), &mapW, tap * a.cin + (second ? a.C0 : 0) + cb * CB, n0, full(s));
                    ++issued;
                    if (++s == kSt) { s = 0; ph ^= 1u; }
                }
            }
        }
        if (!ok && lane == 0) { atomicOr(e.err, DEV_GUARD); s_abort = 1; }
        // the copies issued must land before the CTA can leave
        if (lane == 0)
            for (uint32_t k = issued > (uint32_t)kSt ? issued - kSt : 0; k < issued; ++k) mbar_wait(full((int)(k % kSt)), (k / kSt) & 1u);
    } else if (warp == 1) {
        const uint32_t idesc = instr_desc(BN);
        uint32_t ph = 0, i = 0;
        int s = 0;
        bool ok = true;
        for (int item = blockIdx.x; item < a.items; item += gridDim.x, ++i) {
            const uint32_t buf = i & 1u, use = i >> 1;
            ok = __all_sync(0xffffffffu, mbar_wait_or_abort(acc_empty(buf), (use & 1u) ^ 1u, abort_flag));
            if (!ok) break;
            tc_fence_after();
            const uint32_t acc = tmem + buf * kT * BN;
            for (int kb = 0; kb < nkb; ++kb) {
                ok = __all_sync(0xffffffffu, mbar_wait_or_abort(full(s), ph, abort_flag));
                if (!ok) break;
                tc_fence_after();
                const uint32_t b0 = smem_u32(sB + s * kBBytes);
#pragma unroll
                for (int k = 0; k < CB / 16; ++k) {
                    const uint64_t db = CB == 64 ? smem_desc(b0 + k * 32) : smem_desc64(b0 + k * 32);
#pragma unroll
                    for (int t = 0; t < kT; ++t) {
                        const uint32_t a0 = smem_u32(sA + (s * kT + t) * kABytes);
                        const uint64_t da = CB == 64 ? smem_desc(a0 + k * 32) : smem_desc64(a0 + k * 32);
                        tc_mma(acc + (uint32_t)(t * BN), da, db, idesc, (kb | k) != 0 ? 1u : 0u);
                    }
                }
                tc_commit(empty(s));
                if (++s == kSt) { s = 0; ph ^= 1u; }
            }
            if (!ok) break;
            tc_commit(acc_full(buf));
        }
        if (!ok && lane == 0) {
            atomicOr(e.err, DEV_GUARD);
            s_abort = 1;
        }
    } else {
        // epilogue warps 2..9: TMEM lane quarter q = warp % 4 holds rows 32 q .. 32 q + 31. An
        // item's accumulators are units of 32 columns of a tile, the two sets of four warps taking
        // them in turn. One set, 16 columns at a time and stored from there in 32-byte pieces, took
        // longer than the MMAs: 128 -> 128 with its upsampled copy at 544 x 960 309 -> 170 us, 256 ->
        // 256 at 272 x 480 177 -> 120, 64 -> 128 at 544 x 960 82 -> 68. A BF16
        // output passes through the warp's stage, 32 pixels of 32 channels, and is stored in
        // whole sectors: chunk c of pixel p at 4 p + (c ^ (p >> 1) % 4), clear of bank conflicts
        // both ways.
        const int q = warp & 3, set = (warp - 2) >> 2;
        constexpr int kUnits = kT * BN / 32;
        uint4* stage = s_stage + (warp - 2) * 128;
        auto slot = [](int p, int c) { return p * 4 + (c ^ ((p >> 1) & 3)); };
        uint32_t i = 0;
        for (int item = blockIdx.x; item < a.items; item += gridDim.x, ++i) {
            const uint32_t buf = i & 1u, use = i >> 1;
            const bool ok = __all_sync(0xffffffffu, mbar_wait_or_abort(acc_full(buf), use & 1u, abort_flag));
            if (!ok) {
                if (lane == 0) { atomicOr(e.err, DEV_GUARD); s_abort = 1; }
                break;
            }
            tc_fence_after();
            const int group = item / a.n_slices, n0 = (item % a.n_slices) * BN;
#pragma unroll 1
            for (int u = set; u < kUnits; u += 2) {
                const int t = u / (BN / 32), col = n0 + u % (BN / 32) * 32;
                const int tile = group * kT + t;
                const int tx = tile % a.tiles_x, ty = (tile / a.tiles_x) % a.tiles_y, b = tile / (a.tiles_x * a.tiles_y);
                uint32_t v[32];
                tmem_ld32(tmem + buf * kT * BN + (uint32_t)(u * 32) + ((uint32_t)(q * 32) << 16), v);
                if (u + 2 >= kUnits) {                        // this warp's last read of the buffer
                    tc_fence_before();
                    __syncwarp();
                    if (lane == 0) mbar_arrive(acc_empty(buf));
                }
                float f[32];
#pragma unroll
                for (int j = 0; j < 32; j += 4) {
                    float4 bv = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
                    if (e.bias) bv = *reinterpret_cast<const float4*>(s_bias + col + j);
                    const float bb[4] = {bv.x, bv.y, bv.z, bv.w};
#pragma unroll
                    for (int k = 0; k < 4; ++k) {
                        float x = __uint_as_float(v[j + k]);
                        if (e.bias) x += bb[k];
                        if (e.relu) x = fmaxf(x, 0.0f);
                        f[j + k] = x;
                    }
                }
                // pixel p of the warp's quarter
                auto at = [&](int p, int& y, int& x) {
                    const int r = q * 32 + p;
                    y = ty * th + (r >> a.tw_log2);
                    x = tx * tw + (r & (tw - 1));
                };
                if (e.c32 || e.head_out) {
                    int y, x;
                    at(lane, y, x);
                    const size_t pix = ((size_t)b * a.H + y) * a.W + x;
                    if (e.head_out) {                         // N 32: the unit has every channel
                        float hz = e.head_b[0];
#pragma unroll
                        for (int j = 0; j < 32; ++j) hz += __bfloat162float(__float2bfloat16_rn(f[j])) * e.head_w[j];
                        e.head_out[pix] = 1.0f / (1.0f + __expf(-hz));
                    }
                    if (e.c32) {
                        float4* d4 = reinterpret_cast<float4*>(e.c32 + pix * e.ldc + col);
#pragma unroll
                        for (int h = 0; h < 8; ++h) d4[h] = make_float4(f[4 * h], f[4 * h + 1], f[4 * h + 2], f[4 * h + 3]);
                    }
                }
                if (e.c16) {
#pragma unroll
                    for (int c = 0; c < 4; ++c) {
                        uint4 o;
                        uint32_t* ob = reinterpret_cast<uint32_t*>(&o);
#pragma unroll
                        for (int h = 0; h < 4; ++h) {
                            const __nv_bfloat162 o2 = __floats2bfloat162_rn(f[c * 8 + 2 * h], f[c * 8 + 2 * h + 1]);
                            ob[h] = *reinterpret_cast<const uint32_t*>(&o2);
                        }
                        stage[slot(lane, c)] = o;
                    }
                    __syncwarp();
                    const int c = lane & 3;
#pragma unroll
                    for (int k = 0; k < 4; ++k) {
                        const int p = k * 8 + (lane >> 2);
                        int y, x;
                        at(p, y, x);
                        uint4 o = stage[slot(p, c)];
                        const size_t off = (((size_t)b * a.H + y) * a.W + x) * e.ldc + col + c * 8;
                        if (e.gate) {                          // zero where the gate is not positive
                            const uint4 gv = *reinterpret_cast<const uint4*>(e.gate + off);
                            const uint32_t* g = reinterpret_cast<const uint32_t*>(&gv);
                            uint32_t* ob = reinterpret_cast<uint32_t*>(&o);
#pragma unroll
                            for (int h = 0; h < 4; ++h)
                                ob[h] &= __hgt2_mask(*reinterpret_cast<const __nv_bfloat162*>(g + h), __floats2bfloat162_rn(0.0f, 0.0f));
                        }
                        *reinterpret_cast<uint4*>(e.c16 + off) = o;
                        if (a.up16) {                          // nearest 2x: four copies
                            __nv_bfloat16* d = a.up16 + (((size_t)b * 2 * a.H + 2 * y) * (2 * a.W) + 2 * x) * e.ldc + col + c * 8;
                            const size_t row = (size_t)2 * a.W * e.ldc;
                            *reinterpret_cast<uint4*>(d) = o;
                            *reinterpret_cast<uint4*>(d + e.ldc) = o;
                            *reinterpret_cast<uint4*>(d + row) = o;
                            *reinterpret_cast<uint4*>(d + row + e.ldc) = o;
                        }
                    }
                    __syncwarp();                              // the stage is free again
                }
            }
            if (set >= kUnits) {                               // one unit: the second set has none
                __syncwarp();
                if (lane == 0) mbar_arrive(acc_empty(buf));
            }
        }
    }
    tc_fence_before();
    __syncthreads();
    if (warp == 1)
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(kCols) : "memory");
}


// ------------------------------------------------------------------ implicit 3x3, row ring
// For 128-pixel tiles of one image row (W % 128 == 0) and a layer whose whole weight matrix
// fits in shared memory. A work item is a strip of 128 pixels (x0 .. x0 + 127) over a chunk
// of output rows [y0, y1); the CTA loads the chunk's input rows y0 - 1 .. y1 one at a time,
// each as ONE TMA box per source holding 136 pixels (x0 - 1 .. x0 + 134) of every input
// channel, into a ring of row slots. Output row y reads the slots of rows y - 1, y, y + 1
// in place, each tap's A operand starting one pixel further along its row: every input row
// crosses from L2 once per chunk instead of three times. A row in its slot:
// - fan-out form: a source lies as chunks of 64, 32 or 16 channels (the widest that divides its
//   channel count), each a K-major tile of 136 pixel rows of 128, 64 or 32 bytes with the swizzle
//   of that width: one box per chunk, and a tap's shift moves the operand's start by one pixel
//   row, the swizzle following the address;
// - row by row: without swizzle, a 136 x 16-byte group per 8 channels, the groups of all sources one
//   after the other (one box per source), so that one loop takes any channel count: a tap's shift is
//   16 bytes and a K16 step two groups (48 -> 32 at 272 x 1920 50 us, on swizzled chunks 114).
// The weights are loaded once per CTA, in the no-swizzle K-major canonical form: 8 rows x 16
// bytes per core matrix, core matrices 128 bytes apart along N and one channel group (N x 16
// bytes) apart along K. K order (tap outermost, then channel) and the K16 steps are
// tc_conv_kernel's, so the two kernels give identical results.
constexpr int kHaloW = 136;                        // box width: 128 + 2 halo, rounded for alignment
constexpr uint32_t kHaloGroup = kHaloW * 16;       // bytes of one 8-channel group of a row slot

__device__ __forceinline__ uint64_t desc_plain(uint32_t addr, uint32_t lbo, uint32_t sbo) {
    uint64_t d = (uint64_t)((addr >> 4) & 0x3FFFu);
    d |= (uint64_t)((lbo >> 4) & 0x3FFFu) << 16;      // leading byte offset: next core matrix along K
    d |= (uint64_t)((sbo >> 4) & 0x3FFFu) << 32;      // stride byte offset: next 8 rows along M / N
    d |= (uint64_t)1 << 46;                           // descriptor version; layout 0: no swizzle
    return d;
}
// Pixel rows of cb channels (64, 32 or 16) with the swizzle of that width, 8-row atoms one
// after the other. The start may be any pixel row or 32-byte step of a tile: the swizzle
// is a function of the address.
__device__ __forceinline__ uint64_t desc_rows(uint32_t addr, int cb) {
    uint64_t d = (uint64_t)((addr >> 4) & 0x3FFFu);
    d |= (uint64_t)cb << 32;                          // stride byte offset: 8 rows x 2 cb bytes, in 16-byte units
    d |= (uint64_t)1 << 46;
    d |= (uint64_t)(cb == 64 ? 2 : cb == 32 ? 4 : 6) << 61;
    return d;
}
__device__ __forceinline__ void tma_load_5d(uint32_t dst, const CUtensorMap* map, int c0, int c1, int c2, int c3, int c4,
                                            uint32_t bar) {
    asm volatile(
        "cp.async.bulk.tensor.5d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4, %5, %6}], [%7];" ::"r"(dst),
        "l"(reinterpret_cast<uint64_t>(map)), "r"(c0), "r"(c1), "r"(c2), "r"(c3), "r"(c4), "r"(bar)
        : "memory");
}
__device__ __forceinline__ void tma_load_3d(uint32_t dst, const CUtensorMap* map, int c0, int c1, int c2, uint32_t bar) {
    asm volatile(
        "cp.async.bulk.tensor.3d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4}], [%5];" ::"r"(dst),
        "l"(reinterpret_cast<uint64_t>(map)), "r"(c0), "r"(c1), "r"(c2), "r"(bar)
        : "memory");
}

// tcgen05.cp of a 128-row x 256-bit matrix (128 pixels x 16 BF16 channels, K-major, the
// descriptor's canonical layout) from shared memory into TMEM columns [taddr, taddr + 8).
__device__ __forceinline__ void tc_cp_128x256b(uint32_t taddr, uint64_t sdesc) {
    asm volatile("{\n.reg .pred e;\nelect.sync _|e, 0xffffffff;\n@e tcgen05.cp.cta_group::1.128x256b [%0], %1;\n}\n" ::"r"(taddr), "l"(sdesc)
                 : "memory");
}
// tcgen05.mma.kind::f16 with the A operand read from TMEM (128 lanes = M rows, K in columns).
__device__ __forceinline__ void tc_mma_ta(uint32_t tmem_d, uint32_t tmem_a, uint64_t b, uint32_t idesc,
                                          uint32_t accumulate) {
    asm volatile(
        "{\n.reg .pred p, e;\nelect.sync _|e, 0xffffffff;\nsetp.ne.b32 p, %4, 0;\n@e tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n}\n" ::"r"(tmem_d),
        "r"(tmem_a), "l"(b), "r"(idesc), "r"(accumulate)
        : "memory");
}
// The A operands of one input row kept in TMEM (kTA): its three horizontal taps (the row
// shifted by -1, 0, +1 pixel) x the K steps of its channels, 8 columns each, in a ring of
// kTaSlots rows after the two accumulators. Each input row is copied from its shared-memory
// slot once and read by the three output rows that need it, so shared memory serves the A
// operand once per input row instead of once per tap of every output row; the MMAs then
// read only the weights (B) from shared memory.
constexpr int kTaSlots = 4;
constexpr uint32_t kTaRowCols = 3 * 2 * 8;         // taps x K steps (at most 32 channels) x 8 columns

struct HaloArgs {
    int nsrc, C0, C1, cin;
    int cb0, cb1;               // fan-out: the width of the sources' channel chunks in a row slot (64, 32 or 16)
    int nch0, nch1;             // and their number (nch1: 0 with one source)
    int q16;                    // K16 steps of a tap
    int B, H, W;
    int chunk, chunks_y;        // output rows per work item; items per strip column
    int items;                  // n_slices x slice_items
    int n_slices, slice_items;  // output-channel slices of BN (fan-out; else 1) and items per slice,
                                // (W / 128) x chunks_y x B
    int stages;                 // row slots in the ring (>= 4; fan-out >= 2)
    int sets;                   // sets of four epilogue warps, taking the output rows in turn (1 or 2)
    uint32_t a_bytes, b_bytes;  // one row slot (all sources), the resident weights
    __nv_bfloat16* up16;
};

// Work item -> (output-channel slice, image, strip, first row, rows). The slices of one strip
// chunk are consecutive items: with a grid that is a multiple of the slice count every CTA
// keeps one slice (its weights load once), and the CTAs that hold a chunk's slices read its
// input rows at about the same time, so the second read finds them in L2.
struct HaloItem { int slice, b, tx, y0, rows; };
__device__ __forceinline__ HaloItem halo_item(const HaloArgs& a, int item) {
    const int tiles_x = a.W >> 7;
    HaloItem it;
    it.slice = item % a.n_slices;
    item /= a.n_slices;
    it.tx = item % tiles_x;
    const int c = (item / tiles_x) % a.chunks_y;
    it.b = item / (tiles_x * a.chunks_y);
    it.y0 = c * a.chunk;
    it.rows = min(a.chunk, a.H - it.y0);
    return it;
}

// Fan-out (kFan): the MMAs follow the input rows instead of the output rows. Input row r is
// read by output rows r + 1, r and r - 1 (vertical taps 0, 1, 2), so one MMA of N = 3 x BN
// (A: the row shifted by dx, K16 channels; B: the three vertical taps' weights stacked along
// N) adds its products to all three rows' accumulators at once. An output row's accumulator
// lives in a ring of kAcc = 256 / BN TMEM slots, ring index i at columns (kAcc - 1 - i % kAcc)
// x BN: ascending columns hold descending rows, so the three rows r + 1, r, r - 1 sit in
// ascending columns and their taps 0, 1, 2 in ascending B rows (where the ring wraps, the MMA
// splits in two). The weights are staged as [dx][channel group][dy][n][8 channels] by a 5-D
// box. Per output row the K16 steps still run tap by tap (dy, then dx) and channel by channel
// within a tap, as in the row-by-row MMAs; the accumulators start at zero (the epilogue warps
// clear each one after reading it, and the whole ring at the start) and every MMA adds, so
// both forms give the same values (0 + x = x; at most the sign of an all-zero sum differs).
// Each row slot in shared memory is read by the MMAs of its own input row only; the row's A
// operand crosses from shared memory three times (dx) instead of nine.
// Accumulator ring and residency: 256 TMEM columns (eight rows' accumulators at BN 32, four at
// BN 64) and two CTAs per SM where shared memory allows two; else all 512 columns (kWide), which
// halves the loads whose MMAs split at the ring's wrap (64 -> 64 at 1088 x 1920 131 -> 112 us,
// 64 + 128 -> 64 354 -> 338, 32 + 64 -> 32 at 2176 x 3840 408 -> 393; but one wide CTA where
// two would fit: 32 -> 32 at 2176 x 3840 173 -> 221).
constexpr int kFanMaxAcc = 16;
__host__ __device__ constexpr int fan_cols(bool wide) { return wide ? 512 : 256; }
// Static shared memory of tc_conv_halo_kernel, rounded up: the bias (512 floats) and the abort
// flag; and the epilogue's stage (a set's four warps x 32 pixels x BN BF16 channels).
constexpr size_t kHaloStatic = 2048 + 64;
__host__ __device__ constexpr size_t halo_stage(int bn, int sets) { return (size_t)sets * 4 * 32 * bn * 2; }
constexpr int kFanThreads = 320;    // two sets of epilogue warps

// One load's MMAs in fan-out form for sources of C0 and C1 channels (C1: 0 with one source),
// every operand a base descriptor plus a constant. The row ring's pace is the MMA warp's: its
// instructions come cold from the cache at each row, beside eight epilogue warps, and a loop's
// branch costs as much as an MMA, so a tap's steps are straight line and the three shifts loop
// around them. Measured at 2176 x 3840, 16 -> 32 channels / 32 + 64 -> 32, and at 1088 x 1920,
// 64 + 128 -> 64: loops over chunks and steps 184 / 615 / 446 us, all shifts unrolled
// 145 / 422 / 375, this 144 / 408 / 354. They take the channel counts of the U-Net's layers whose
// weights fit; any other runs loops over its chunks, straight line within one (fan_chunks).
struct FanRow {
    uint64_t a0, a1;            // the sources' descriptors at the row's first pixel
    uint64_t b0, b1;            // B at each piece's first row
    uint32_t acc0, acc1, id0, id1;
    bool split;                 // a second piece
};
__device__ __forceinline__ uint64_t desc_add(uint64_t d, uint32_t n) {      // the address field is in the low word
    return (d & 0xFFFFFFFF00000000ull) | ((uint32_t)d + n);
}
__host__ __device__ constexpr int chunk_channels(int C) { return C % 64 == 0 ? 64 : C % 32 == 0 ? 32 : 16; }
template <int BN, int C0, int C1>
__device__ __forceinline__ void fan_row(const FanRow& f) {
    constexpr uint32_t b_grp = 3u * BN;                                     // 16-byte units, as all here
    auto step = [&](bool split, uint32_t xa0, uint32_t xa1, uint32_t xb) {
#pragma unroll
        for (int q = 0; q < (C0 + C1) / 16; ++q) {
            const bool first = q * 16 < C0;
            const int ch = first ? q * 16 : q * 16 - C0, cb = first ? chunk_channels(C0) : chunk_channels(C1 ? C1 : 16);
            const uint32_t oa = (uint32_t)(ch / cb * kHaloW * (cb >> 3) + ch % cb / 8), ob = (uint32_t)(2 * q) * b_grp + xb;
            const uint64_t da = first ? desc_add(f.a0, oa + xa0) : desc_add(f.a1, oa + xa1);
            tc_mma(f.acc0, da, desc_add(f.b0, ob), f.id0, 1u);
            if (split) tc_mma(f.acc1, da, desc_add(f.b1, ob), f.id1, 1u);
        }
    };
    auto run = [&](bool split) {
        constexpr uint32_t p0 = chunk_channels(C0) >> 3, p1 = chunk_channels(C1 ? C1 : 16) >> 3, pb = (C0 + C1) / 8 * b_grp;
#pragma unroll 1
        for (uint32_t dx = 0; dx < 3; ++dx) step(split, dx * p0, dx * p1, dx * pb);
    };
    if (f.split) run(true);
    else run(false);
}

// The same for any channel counts: one source's chunks of one tap, the chunk's width fixed in each
// of three loops (at 272 x 1920 48 -> 32 channels 36.2 us with one loop of a run-time width, 29.1 so, 112
// -> 64 94.9 and 67.3, 16 + 112 -> 32 101.7 and 62.6). Moves b0 and b1 past the source's steps.
template <int BN>
__device__ __forceinline__ void fan_chunks(const FanRow& f, uint64_t a, int cb, int chunks, bool split, uint64_t& b0,
                                           uint64_t& b1) {
    constexpr uint32_t kStepB = 2u * 3u * BN;                               // the next 16 channels of B
    auto steps = [&](auto width) {
        constexpr int kW = decltype(width)::value;
#pragma unroll
        for (int k = 0; k < kW / 16; ++k) {
            tc_mma(f.acc0, desc_add(a, 2u * k), desc_add(b0, k * kStepB), f.id0, 1u);
            if (split) tc_mma(f.acc1, desc_add(a, 2u * k), desc_add(b1, k * kStepB), f.id1, 1u);
        }
        a = desc_add(a, kHaloW * (kW >> 3));
        b0 = desc_add(b0, kW / 16 * kStepB);
        b1 = desc_add(b1, kW / 16 * kStepB);
    };
    if (cb == 64) {
#pragma unroll 1
        for (int c = 0; c < chunks; ++c) steps(std::integral_constant<int, 64>());
    } else if (cb == 32) {
#pragma unroll 2
        for (int c = 0; c < chunks; ++c) steps(std::integral_constant<int, 32>());
    } else {
#pragma unroll 4
        for (int c = 0; c < chunks; ++c) steps(std::integral_constant<int, 16>());
    }
}

// Bytes of one row slot (C1: 0 with one source).
__host__ __device__ constexpr uint32_t halo_slot(int C0, int C1, bool fan) {
    return !fan ? ((uint32_t)(C0 + C1) * 2u * kHaloW + 1023u) & ~1023u
              : (((uint32_t)C0 * 2u * kHaloW + 1023u) & ~1023u) + (((uint32_t)C1 * 2u * kHaloW + 1023u) & ~1023u);
}

template <int BN, bool kTA, bool kFan, bool kWide>
__global__ void __launch_bounds__(kFan ? kFanThreads : kConvThreads, kFan && !kWide ? 2 : 1) tc_conv_halo_kernel(const __grid_constant__ CUtensorMap map0,
                                                                       const __grid_constant__ CUtensorMap map1,
                                                                       const __grid_constant__ CUtensorMap mapW,
                                                                       const HaloArgs a, const Epilogue e) {
    extern __shared__ uint8_t smem_raw[];
    uint8_t* smem = (uint8_t*)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
    // TMEM: kAcc accumulators (the MMAs of a row run while the previous row is in the
    // epilogue; four measured no faster), then (kTA) the ring of input rows' A operands; a
    // power of two. Fan-out: a ring of 256 / BN accumulators.
    static_assert(!(kTA && kFan), "one form at a time");
    static_assert(!kFan || (3 * BN <= 256 && 512 / BN <= kFanMaxAcc), "three rows' accumulators in one MMA");
    constexpr uint32_t kAcc = kFan ? (uint32_t)(fan_cols(kWide) / BN) : 2u;
    constexpr uint32_t kCols = kTA ? 256u : kAcc * BN;
    static_assert(!kTA || 2 * BN + kTaSlots * kTaRowCols <= 256, "the TMEM ring fits");
    const int kSt = a.stages;
    uint8_t* sB = smem;
    uint8_t* sA = smem + ((a.b_bytes + 1023) & ~1023u);
    const uint32_t a_stride = halo_slot(a.C0, a.C1, kFan);
    // full[kSt], empty[kSt], acc_full[kFanMaxAcc], acc_empty[kFanMaxAcc], w (weights landed), wfree
    // (the weights' last MMAs done: a slice's weights may be replaced)
    uint4* s_stage = reinterpret_cast<uint4*>(sA + kSt * a_stride);
    uint64_t* bars = reinterpret_cast<uint64_t*>(sA + kSt * a_stride + halo_stage(BN, a.sets));
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 2 * kSt + 2 * kFanMaxAcc + 2);
    __shared__ int s_abort;
    __shared__ __align__(16) float s_bias[512];       // the bias of every output channel, staged once
    volatile int* abort_flag = &s_abort;
    const int warp = warp_index(), lane = threadIdx.x & 31;
    auto full = [&](int s) { return smem_u32(&bars[s]); };
    auto empty = [&](int s) { return smem_u32(&bars[kSt + s]); };
    auto acc_full = [&](int b) { return smem_u32(&bars[2 * kSt + b]); };
    auto acc_empty = [&](int b) { return smem_u32(&bars[2 * kSt + kFanMaxAcc + b]); };
    const uint32_t wbar = smem_u32(&bars[2 * kSt + 2 * kFanMaxAcc]);
    const uint32_t wfree = smem_u32(&bars[2 * kSt + 2 * kFanMaxAcc + 1]);
    // first TMEM column of the accumulator of output row i (counted over the CTA's items)
    auto acc_col = [&](uint32_t i) -> uint32_t { return kFan ? (kAcc - 1u - i % kAcc) * BN : (i % kAcc) * BN; };

    if (threadIdx.x == 0) {
        for (int s = 0; s < kSt; ++s) { mbar_init(full(s), 1); mbar_init(empty(s), 1); }
        for (int b = 0; b < (int)kAcc; ++b) { mbar_init(acc_full(b), 1); mbar_init(acc_empty(b), 4); }
        mbar_init(wbar, 1);
        mbar_init(wfree, 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        s_abort = 0;
    }
    if (e.bias)
        for (int i = threadIdx.x; i < a.n_slices * BN; i += blockDim.x) s_bias[i] = e.bias[i];
    if (warp == 1) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)),
                     "r"(kCols)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = __shfl_sync(0xffffffffu, *tmem_slot, 0);
    // the second source's place in a row slot (the swizzled tiles start on 1024 bytes)
    const uint32_t src1_off = !kFan ? (uint32_t)(a.C0 / 8) * kHaloGroup : ((uint32_t)a.C0 * 2u * kHaloW + 1023u) & ~1023u;
    constexpr uint32_t kStepA = (2u * kHaloGroup) >> 4;               // row by row: the next 16 channels of A
    if (kFan) {
        // fan-out accumulators start at zero and every MMA adds to them: each epilogue warp
        // clears its lane quarter of the ring now and of each row again once it has read it
        if (warp >= 2)
            for (uint32_t c = 0; c < kCols; c += 32) tmem_zero32(tmem + c + ((uint32_t)((warp & 3) * 32) << 16));
        tmem_wait_st();
        tc_fence_before();
        __syncthreads();
        tc_fence_after();
    }

    if (warp == 0) {
        if (lane == 0) {
            // loads in ring order: item by item, input rows y0 - 1 .. y0 + rows
            // the weights of the first item's slice; a later slice's replace them once the MMA
            // thread reports the last MMAs that read them done (wfree)
            int wslice = (int)blockIdx.x % a.n_slices;
            uint32_t wfree_ph = 0;
            mbar_expect_tx(wbar, a.b_bytes);
            if (kFan) tma_load_5d(smem_u32(sB), &mapW, 0, wslice * BN, 0, 0, 0, wbar);
            else tma_load_3d(smem_u32(sB), &mapW, 0, 0, 0, wbar);
            // kc counts loads; s and ph are its ring slot and the slot's phase (kc % kSt and
            // kc / kSt mod 2, kept by increment: kSt is a launch argument, and a division per
            // load would sit on this thread's path)
            uint32_t kc = 0, ph = 0;
            int s = 0;
            for (int item = blockIdx.x; item < a.items && !*abort_flag; item += gridDim.x) {
                const HaloItem it = halo_item(a, item);
                if (kFan && it.slice != wslice) {
                    if (!mbar_wait_or_abort(wfree, wfree_ph, abort_flag)) {
                        atomicOr(e.err, DEV_GUARD);
                        s_abort = 1;
                        break;
                    }
                    wfree_ph ^= 1u;
                    wslice = it.slice;
                    mbar_expect_tx(wbar, a.b_bytes);
                    tma_load_5d(smem_u32(sB), &mapW, 0, wslice * BN, 0, 0, 0, wbar);
                }
                for (int r = -1; r <= it.rows && !*abort_flag; ++r, ++kc) {
                    if (!mbar_wait_or_abort(empty(s), ph ^ 1u, abort_flag)) {
                        atomicOr(e.err, DEV_GUARD);
                        s_abort = 1;
                        break;
                    }
                    mbar_expect_tx(full(s), a.a_bytes);
                    const uint32_t dst = smem_u32(sA + s * a_stride);
                    if (!kFan) {
                        tma_load_5d(dst, &map0, 0, it.tx * 128 - 1, it.y0 + r, it.b, 0, full(s));
                        if (a.nsrc > 1) tma_load_5d(dst + src1_off, &map1, 0, it.tx * 128 - 1, it.y0 + r, it.b, 0, full(s));
                    } else {
                        for (int c = 0; c < a.nch0; ++c)
                            tma_load_4d(dst + (uint32_t)(c * a.cb0 * 2 * kHaloW), &map0, c * a.cb0, it.tx * 128 - 1, it.y0 + r,
                                        it.b, full(s));
                        for (int c = 0; c < a.nch1; ++c)
                            tma_load_4d(dst + src1_off + (uint32_t)(c * a.cb1 * 2 * kHaloW), &map1, c * a.cb1,
                                        it.tx * 128 - 1, it.y0 + r, it.b, full(s));
                    }
                    if (++s == kSt) { s = 0; ph ^= 1u; }
                }
            }
            // the copies this lane issued must land before the CTA can leave
            for (uint32_t k = kc > (uint32_t)kSt ? kc - kSt : 0; k < kc; ++k) mbar_wait(full(k % kSt), (k / kSt) & 1u);
            mbar_wait(wbar, wfree_ph);      // the last weights load (one more than the reloads)
        }
    } else if (warp == 1 && kFan) {
        const uint32_t b_grp = 3u * BN * 16u;                         // next channel group of B (LBO)
        const uint64_t db0 = desc_plain(smem_u32(sB), b_grp, 128);
        bool ok = __all_sync(0xffffffffu, mbar_wait_or_abort(wbar, 0, abort_flag));
        int wslice = (int)blockIdx.x % a.n_slices;
        uint32_t w_ph = 0;
        uint32_t i0 = 0;            // output rows of earlier items
        // the current load's ring slot, its phase and its shared-memory row (kept by increment)
        int slot = 0;
        uint32_t phase = 0, row_smem = smem_u32(sA);
        // Descriptors are affine in their address (the 14-bit field holds address / 16, and
        // no offset here carries out of it): every MMA is a base descriptor plus a constant.
        for (int item = blockIdx.x; ok && item < a.items; item += gridDim.x) {
            const HaloItem it = halo_item(a, item);
            if (it.slice != wslice) {
                // the next slice's weights: once this slice's MMAs have read theirs
                tc_commit(wfree);
                w_ph ^= 1u;
                ok = __all_sync(0xffffffffu, mbar_wait_or_abort(wbar, w_ph, abort_flag));
                if (!ok) break;
                wslice = it.slice;
            }
            // load k is input row y0 - 1 + k; it feeds output rows k - 2 .. k of the item
            for (int k = 0; k <= it.rows + 1; ++k) {
                // the output rows that exist, lo .. hi of them: one piece with the top row first
                // and, where the ring wraps below it, a second; each an accumulator address, N
                // and the offset of its first B row (vertical tap k - h for its top row h)
                const int lo = max(0, k - 2), hi = min(it.rows - 1, k);
                const uint32_t ih = (i0 + (uint32_t)hi) % kAcc;
                const int n = hi - lo + 1, n0 = min(n, (int)ih + 1), n1 = n - n0;
                const uint32_t acc0 = tmem + (kAcc - 1u - ih) * BN, acc1 = tmem;   // the wrapped piece: ring index kAcc - 1
                const uint32_t id0 = instr_desc(n0 * BN), id1 = instr_desc(n1 * BN);
                const uint64_t b0 = db0 + (uint64_t)((k - hi) * BN), b1 = b0 + (uint64_t)(n0 * BN);
                if (hi == k) {
                    // output row k's first load: its accumulator must be free
                    const uint32_t i = i0 + (uint32_t)k;
                    ok = __all_sync(0xffffffffu, mbar_wait_or_abort(acc_empty(i % kAcc), ((i / kAcc) & 1u) ^ 1u, abort_flag));
                    if (!ok) break;
                }
                ok = __all_sync(0xffffffffu, mbar_wait_or_abort(full(slot), phase, abort_flag));
                if (!ok) break;
                tc_fence_after();
                const FanRow fr{desc_rows(row_smem, a.cb0), desc_rows(row_smem + src1_off, a.cb1), b0, b1, acc0, acc1, id0, id1, n1 != 0};
                if (a.C0 == 32 && a.C1 == 0) fan_row<BN, 32, 0>(fr);
                else if (a.C0 == 16 && a.C1 == 0) fan_row<BN, 16, 0>(fr);
                else if (a.C0 == 64 && a.C1 == 0) fan_row<BN, 64, 0>(fr);
                else if (a.C0 == 128 && a.C1 == 0) fan_row<BN, 128, 0>(fr);
                else if (a.C0 == 32 && a.C1 == 64) fan_row<BN, 32, 64>(fr);
                else if (a.C0 == 64 && a.C1 == 128) fan_row<BN, 64, 128>(fr);
                else {
                    auto run = [&](bool split) {
                        uint64_t d0 = b0, d1 = b1;                    // the taps lie one after the other
#pragma unroll 1
                        for (uint32_t dx = 0; dx < 3; ++dx) {
                            fan_chunks<BN>(fr, desc_add(fr.a0, dx * (uint32_t)(a.cb0 >> 3)), a.cb0, a.nch0, split, d0, d1);
                            if (a.nch1) fan_chunks<BN>(fr, desc_add(fr.a1, dx * (uint32_t)(a.cb1 >> 3)), a.cb1, a.nch1, split, d0, d1);
                        }
                    };
                    if (n1) run(true);
                    else run(false);
                }
                // the row slot is free once its MMAs have read it; output row k - 2 is complete
                tc_commit(empty(slot));
                if (k >= 2) tc_commit(acc_full((i0 + (uint32_t)(k - 2)) % kAcc));
                if (++slot == kSt) {
                    slot = 0;
                    phase ^= 1u;
                    row_smem = smem_u32(sA);
                } else {
                    row_smem += a_stride;
                }
            }
            if (!ok) break;
            i0 += (uint32_t)it.rows;
        }
        if (!ok && lane == 0) {
            atomicOr(e.err, DEV_GUARD);
            s_abort = 1;
        }
    } else if (warp == 1 && kTA) {
        const uint32_t idesc = instr_desc(BN);
        const uint32_t b0 = smem_u32(sB);
        const int g_tap = a.cin / 8;
        const uint32_t ta0 = tmem + 2u * BN;
        bool ok = __all_sync(0xffffffffu, mbar_wait_or_abort(wbar, 0, abort_flag));
        uint32_t base = 0, i = 0;   // ring index of the item's first load; output rows so far
        for (int item = blockIdx.x; ok && item < a.items; item += gridDim.x) {
            const HaloItem it = halo_item(a, item);
            for (int j = 0; ok && j < it.rows; ++j, ++i) {
                // output row y0 + j reads loads j, j + 1, j + 2 of the item
                const uint32_t buf = i % kAcc, use = i / kAcc;
                // row i - 2's MMAs are done once its accumulator is free again: the TMEM
                // slots they read may be overwritten
                if (!__all_sync(0xffffffffu, mbar_wait_or_abort(acc_empty(buf), (use & 1u) ^ 1u, abort_flag))) { ok = false; break; }
                if (j == 0 && i > 0) {
                    // a new item reloads three rows: the previous row's MMAs must be done too
                    const uint32_t pi = i - 1;
                    if (!__all_sync(0xffffffffu, mbar_wait_or_abort(acc_full(pi % kAcc), (pi / kAcc) & 1u, abort_flag))) { ok = false; break; }
                }
                for (int d = (j == 0 ? 0 : 2); d < 3 && ok; ++d) {
                    const uint32_t k = base + (uint32_t)(j + d);
                    ok = __all_sync(0xffffffffu, mbar_wait_or_abort(full(k % kSt), (k / kSt) & 1u, abort_flag));
                    if (!ok) break;
                    tc_fence_after();
                    const uint32_t row = smem_u32(sA + (k % kSt) * a_stride);
                    const uint32_t slot = ta0 + (k % kTaSlots) * kTaRowCols;
                    for (int dx = 0; dx < 3; ++dx)
                        for (int q = 0; q < a.q16; ++q)
                            tc_cp_128x256b(slot + (uint32_t)(dx * a.q16 + q) * 8u,
                                           desc_plain(row + (uint32_t)dx * 16u + (uint32_t)(2 * q) * kHaloGroup,
                                                      kHaloGroup, 128));
                    // the shared-memory slot is free once its copies have run
                    tc_commit(empty(k % kSt));
                }
                if (!ok) break;
                const uint32_t acc = tmem + buf * BN;
                for (int t = 0; t < 9; ++t) {
                    const uint32_t k = base + (uint32_t)(j + t / 3);
                    const uint32_t slot = ta0 + (k % kTaSlots) * kTaRowCols + (uint32_t)((t % 3) * a.q16) * 8u;
                    for (int q = 0; q < a.q16; ++q) {
                        const uint64_t db = desc_plain(b0 + (uint32_t)(t * g_tap + 2 * q) * (BN * 16), BN * 16, 128);
                        tc_mma_ta(acc, slot + (uint32_t)q * 8u, db, idesc, (t | q) != 0 ? 1u : 0u);
                    }
                }
                tc_commit(acc_full(buf));
            }
            if (!ok) break;
            base += (uint32_t)it.rows + 2;
        }
        if (!ok && lane == 0) {
            atomicOr(e.err, DEV_GUARD);
            s_abort = 1;
        }
    } else if (warp == 1) {
        const uint32_t idesc = instr_desc(BN);
        const int g_tap = a.cin / 8;
        const uint64_t db0 = desc_plain(smem_u32(sB), BN * 16, 128);
        const uint32_t dq_b = (2u * BN * 16u) >> 4;                   // the next 16 channels of B
        const uint32_t dtap_b = ((uint32_t)g_tap * BN * 16u) >> 4;    // the next tap of B
        bool ok = __all_sync(0xffffffffu, mbar_wait_or_abort(wbar, 0, abort_flag));
        uint32_t base = 0, i = 0;   // ring index of the item's first load; output rows so far
        for (int item = blockIdx.x; ok && item < a.items; item += gridDim.x) {
            const HaloItem it = halo_item(a, item);
            for (int j = 0; ok && j < it.rows; ++j, ++i) {
                // output row y0 + j reads loads j, j + 1, j + 2 of the item
                const uint32_t buf = i % kAcc, use = i / kAcc;
                if (!__all_sync(0xffffffffu, mbar_wait_or_abort(acc_empty(buf), (use & 1u) ^ 1u, abort_flag))) { ok = false; break; }
                uint32_t row_addr[3];
                for (int d = 0; d < 3 && ok; ++d) {
                    const uint32_t k = base + (uint32_t)(j + d);
                    ok = __all_sync(0xffffffffu, mbar_wait_or_abort(full(k % kSt), (k / kSt) & 1u, abort_flag));
                    row_addr[d] = smem_u32(sA + (k % kSt) * a_stride);
                }
                if (!ok) break;
                tc_fence_after();
                const uint32_t acc = tmem + buf * BN;
                // a descriptor is affine in its address (the 14-bit field holds address / 16
                // and no offset here carries out of it): each MMA's operands are the row's or
                // the weights' base descriptor plus a constant, so the issuing thread spends
                // a few instructions per MMA instead of forming two descriptors
                uint64_t db_tap = db0;
                uint32_t add = 0;
#pragma unroll
                for (int t = 0; t < 9; ++t) {
                    uint64_t da = desc_plain(row_addr[t / 3] + (uint32_t)(t % 3) * 16u, kHaloGroup, 128), db = db_tap;
#pragma unroll 4
                    for (int q = 0; q < a.q16; ++q) {
                        tc_mma(acc, da, db, idesc, add);
                        add = 1u;
                        da = desc_add(da, kStepA);
                        db = desc_add(db, dq_b);
                    }
                    db_tap = desc_add(db_tap, dtap_b);
                }
                tc_commit(acc_full(buf));
                // load j (input row y0 + j - 1) has no later reader
                tc_commit(empty((base + (uint32_t)j) % kSt));
            }
            if (!ok) break;
            // the item's last two loads
            tc_commit(empty((base + (uint32_t)it.rows) % kSt));
            tc_commit(empty((base + (uint32_t)it.rows + 1) % kSt));
            base += (uint32_t)it.rows + 2;
        }
        if (!ok && lane == 0) {
            atomicOr(e.err, DEV_GUARD);
            s_abort = 1;
        }
    } else {
        const int q = warp & 3;
        const int r = q * 32 + lane;
        // BF16 outputs pass through shared memory: a lane converts its pixel's BN channels
        // into 16-byte chunks of its warp's stage, then the warp stores the stage's 32 pixels
        // as whole 512-byte runs (16 contiguous bytes a lane) instead of one 16-byte piece a
        // lane 2 x BN bytes apart. Chunk c of pixel p sits at slot p kCh + (c ^ swz(p)): a
        // quarter-warp's eight 16-byte accesses then fall in eight different bank groups
        // both when lanes write their own pixels and when they read consecutive chunks.
        constexpr int kCh = BN / 8;
        uint4* stage = s_stage + (warp - 2) * 32 * kCh;
        // One set's row takes it 1,300 cycles from the accumulator to the last store, all of it
        // latency: two sets in turn (16 -> 32 at 2176 x 3840 173 -> 144 us with the second, 32 ->
        // 32 202 -> 174, 32 -> 64 at 1088 x 1920 111 -> 88).
        const int set = (warp - 2) >> 2;
        auto slot = [](int p, int c) { return p * kCh + (c ^ ((kCh == 4 ? (p >> 1) : p) & (kCh - 1))); };
        uint32_t i = 0;
        bool ok = true;
        for (int item = blockIdx.x; ok && item < a.items; item += gridDim.x) {
            const HaloItem it = halo_item(a, item);
            for (int j = 0; j < it.rows; ++j, ++i) {
                if (a.sets == 2 && (int)(i & 1u) != set) continue;
                const uint32_t buf = i % kAcc, use = i / kAcc;
                ok = __all_sync(0xffffffffu, mbar_wait_or_abort(acc_full(buf), use & 1u, abort_flag));
                if (!ok) {
                    if (lane == 0) { atomicOr(e.err, DEV_GUARD); s_abort = 1; }
                    break;
                }
                tc_fence_after();
                const int y = it.y0 + j, x = it.tx * 128 + r;
                const size_t pix = ((size_t)it.b * a.H + y) * a.W + x;
                const uint32_t tbase = tmem + acc_col(i) + ((uint32_t)(q * 32) << 16);
                const int n0 = it.slice * BN;                  // the item's first output channel
                float hz = e.head_out ? e.head_b[0] : 0.0f;
                const bool plain = !e.head_out && !e.c32;
                const __nv_bfloat16* gate = e.gate ? e.gate + pix * e.ldc + n0 : nullptr;
#pragma unroll
                for (int c32 = 0; c32 < BN; c32 += 32) {
                    // 32 columns in one TMEM load and one wait
                    uint32_t vv[32];
                    tmem_ld32(tbase + (uint32_t)c32, vv);
                    if (kFan) tmem_zero32(tbase + (uint32_t)c32);      // the row's next use starts from zero
                    if (plain) {
                        // two channels an instruction: bias added in FP32, then rounded, then
                        // ReLU and gate on the rounded pair (the same values: rounding keeps the
                        // sign, and a gated value is zero either way)
#pragma unroll
                        for (int c8 = 0; c8 < 32; c8 += 8) {
                            uint4 out, gv;
                            uint32_t* ob = reinterpret_cast<uint32_t*>(&out);
                            if (gate) gv = *reinterpret_cast<const uint4*>(gate + c32 + c8);
#pragma unroll
                            for (int h = 0; h < 4; ++h) {
                                float2 t = make_float2(__uint_as_float(vv[c8 + 2 * h]), __uint_as_float(vv[c8 + 2 * h + 1]));
                                if (e.bias) t = add2(t, *reinterpret_cast<const float2*>(s_bias + n0 + c32 + c8 + 2 * h));
                                __nv_bfloat162 o2 = __floats2bfloat162_rn(t.x, t.y);
                                if (e.relu) o2 = __hmax2(o2, __floats2bfloat162_rn(0.0f, 0.0f));
                                ob[h] = *reinterpret_cast<uint32_t*>(&o2);
                            }
                            if (gate) {
                                const uint32_t* g = reinterpret_cast<const uint32_t*>(&gv);
#pragma unroll
                                for (int h = 0; h < 4; ++h)
                                    ob[h] &= __hgt2_mask(*reinterpret_cast<const __nv_bfloat162*>(g + h), __floats2bfloat162_rn(0.0f, 0.0f));
                            }
                            stage[slot(lane, (c32 + c8) / 8)] = out;
                        }
                        continue;
                    }
#pragma unroll
                    for (int c0 = c32; c0 < c32 + 32; c0 += 16) {
                        const uint32_t* v = vv + (c0 - c32);
                        float f[16];
#pragma unroll
                        for (int jj = 0; jj < 16; ++jj) {
                            float t = __uint_as_float(v[jj]);
                            if (e.bias) t += s_bias[n0 + c0 + jj];
                            if (e.relu) t = fmaxf(t, 0.0f);
                            f[jj] = t;
                        }
                        if (e.head_out)
#pragma unroll
                            for (int jj = 0; jj < 16; ++jj)
                                hz += __bfloat162float(__float2bfloat16_rn(f[jj])) * e.head_w[c0 + jj];
                        if (e.c16) {
                            uint4 out[2];
                            __nv_bfloat16* ob = reinterpret_cast<__nv_bfloat16*>(out);
#pragma unroll
                            for (int jj = 0; jj < 16; ++jj) ob[jj] = __float2bfloat16_rn(f[jj]);
                            stage[slot(lane, c0 / 8)] = out[0];
                            stage[slot(lane, c0 / 8 + 1)] = out[1];
                        }
                        if (e.c32) {
                            float4* d4 = reinterpret_cast<float4*>(e.c32 + pix * e.ldc + n0 + c0);
#pragma unroll
                            for (int h = 0; h < 4; ++h) d4[h] = make_float4(f[4 * h], f[4 * h + 1], f[4 * h + 2], f[4 * h + 3]);
                        }
                    }
                }
                if (e.head_out) e.head_out[pix] = 1.0f / (1.0f + __expf(-hz));
                if (kFan) tmem_wait_st();
                tc_fence_before();
                __syncwarp();
                // the accumulator is read (and, fan-out, cleared): the MMAs may refill it while
                // the warp stores
                if (lane == 0) mbar_arrive(acc_empty(buf));
                if (e.c16) {
                    const size_t pix0 = pix - lane;                       // the warp's first pixel
                    __nv_bfloat16* d = e.c16 + (pix0 + lane / kCh) * e.ldc + n0 + lane % kCh * 8;
                    const size_t dk = (size_t)(32 / kCh) * e.ldc;
#pragma unroll
                    for (int k = 0; k < kCh; ++k, d += dk)
                        *reinterpret_cast<uint4*>(d) = stage[slot(k * (32 / kCh) + lane / kCh, lane % kCh)];
                    if (a.up16) {
                        // rows 2y and 2y + 1 of the 2x copy: 64 pixels, each source pixel twice
                        const size_t up0 = ((size_t)it.b * 2 * a.H + 2 * y) * (2 * a.W) + 2 * (x - lane);
#pragma unroll 1
                        for (int k = 0; k < 2 * kCh; ++k) {
                            const int idx = k * 32 + lane, P = idx / kCh, c = idx % kCh;
                            const uint4 v = stage[slot(P >> 1, c)];
                            *reinterpret_cast<uint4*>(a.up16 + (up0 + P) * e.ldc + n0 + c * 8) = v;
                            *reinterpret_cast<uint4*>(a.up16 + (up0 + 2 * a.W + P) * e.ldc + n0 + c * 8) = v;
                        }
                    }
                    __syncwarp();                                         // the stage is free again
                }
            }
        }
    }
    tc_fence_before();
    __syncthreads();
    if (warp == 1)
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(kCols) : "memory");
}

// ------------------------------------------------------------------ weight gradient
// dW[(tap, ci)][n] = sum over pixels of x[pixel + tap][ci] * dz[pixel][n]: a contraction over
// pixels whose operands both lie channel-contiguous in memory, so both are read MN-major
// (tcgen05's transposed operands): a TMA box of 64 pixels x CA channels at a tap's offset lands
// in shared memory as rows of CA channels, which is the canonical MN-major tile (CA 64, 32 or 16
// channels: 128-, 64- or 32-byte swizzle; 8 pixels per swizzle atom, the atoms of a tile one
// after the other along the channels). The border reads TMA's zero fill, the convolution's
// padding. No im2col rows are formed and nothing is transposed in memory: at batch 64 of
// 128 x 128 the 14 layers took 12.2 ms as im2col, two transposes and a GEMM, 0.80 ms so.
//
// An "atom" is one (tap, CA-channel chunk); 128 / CA atoms make an M tile of 128 weight rows. A
// CTA takes a group of up to 256 / N M tiles (256 TMEM columns, two CTAs per SM) and a slice of
// the pixel boxes: per box it loads dz once and each M tile's atoms through a ring, so dz is
// read once per group, and every x element nine times, from L2. At the end it adds its tiles
// to gw with FP32 atomics. The bias gradient, dz's column sums, comes from the same boxes: in the
// first group's CTAs the epilogue warps, idle until the end, add up each dz box in shared memory
// before its slot is released (a pass of its own read dz again: 14 passes, 250 us). Roles: warp 0
// loads (its lanes issue a tile's atoms together), warp 1 issues the MMAs (convergent, an elected
// lane executing), warps 2..5 read the accumulators. Waits are bounded and give up when another
// role has aborted.
struct WgradArgs {
    int nb0, nb1;               // CA-channel chunks of the sources
    int tiles_x, tiles_y;       // 64-pixel boxes per image row / column
    int tw, th;
    int boxes;                  // all images' boxes
    int natoms, mtiles;         // 9 (nb0 + nb1); M tiles over them
    int per_group, groups, slices;
    int cin_out, ch_valid;
    float* gw;
    float* gb;                  // column sums of dz, or null
    uint32_t* err;
};
constexpr int kWgPix = 64;
__host__ __device__ constexpr int wg_a_stages(int n) { return n == 32 ? 6 : n == 64 ? 5 : n == 128 ? 4 : 2; }
__host__ __device__ constexpr int wg_b_stages(int n) { return n <= 64 ? 3 : 2; }

// MN-major descriptor: atoms of CA channels (CA * 2 bytes a pixel row) one box apart along M or
// N (the leading offset), 8-pixel groups 8 rows apart along K (the stride offset).
template <int CA>
__device__ __forceinline__ uint64_t desc_mn(uint32_t addr) {
    constexpr uint32_t row = CA * 2;
    uint64_t d = (uint64_t)((addr >> 4) & 0x3FFFu);
    d |= (uint64_t)(((kWgPix * row) >> 4) & 0x3FFFu) << 16;
    d |= (uint64_t)(((8 * row) >> 4) & 0x3FFFu) << 32;
    d |= (uint64_t)1 << 46;
    d |= (uint64_t)(CA == 64 ? 2 : CA == 32 ? 4 : 6) << 61;
    return d;
}

template <int N, int CA>
__global__ void __launch_bounds__(kConvThreads, 2) tc_wgrad_kernel(const __grid_constant__ CUtensorMap map0,
                                                                   const __grid_constant__ CUtensorMap map1,
                                                                   const __grid_constant__ CUtensorMap mapZ,
                                                                   const WgradArgs a) {
    constexpr int kA = wg_a_stages(N), kB = wg_b_stages(N), kApt = 128 / CA, CB = N >= 64 ? 64 : 32;
    constexpr uint32_t kAtom = kWgPix * CA * 2, kABytes = kWgPix * 128 * 2, kBBytes = kWgPix * N * 2;
    constexpr uint32_t kCols = 256;
    extern __shared__ uint8_t smem_raw[];
    uint8_t* smem = (uint8_t*)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
    uint8_t* sA = smem;
    uint8_t* sB = smem + kA * kABytes;
    uint64_t* bars = reinterpret_cast<uint64_t*>(sB + kB * kBBytes);
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 2 * (kA + kB) + 1);
    __shared__ int s_abort;
    volatile int* abort_flag = &s_abort;
    const int warp = warp_index(), lane = threadIdx.x & 31;
    auto a_full = [&](int s) { return smem_u32(&bars[s]); };
    auto a_empty = [&](int s) { return smem_u32(&bars[kA + s]); };
    auto b_full = [&](int s) { return smem_u32(&bars[2 * kA + s]); };
    auto b_empty = [&](int s) { return smem_u32(&bars[2 * kA + kB + s]); };
    const uint32_t done = smem_u32(&bars[2 * (kA + kB)]);
    // this CTA's M tiles [m0, m0 + nm) and boxes [k0, k1)
    const int group = (int)blockIdx.x % a.groups, slice = (int)blockIdx.x / a.groups;
    const bool sums = a.gb && group == 0;
    const int m0 = group * a.per_group, nm = min(a.per_group, a.mtiles - m0);
    const int k0 = (int)((long long)a.boxes * slice / a.slices), k1 = (int)((long long)a.boxes * (slice + 1) / a.slices);

    if (threadIdx.x == 0) {
        for (int s = 0; s < kA; ++s) { mbar_init(a_full(s), 1); mbar_init(a_empty(s), 1); }
        for (int s = 0; s < kB; ++s) { mbar_init(b_full(s), 1); mbar_init(b_empty(s), sums ? 5 : 1); }
        mbar_init(done, 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        s_abort = 0;
    }
    if (warp == 1) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)),
                     "r"(kCols)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = __shfl_sync(0xffffffffu, *tmem_slot, 0);

    if (warp == 0) {
        // every lane waits for the slot; lane 0 arms its barrier before the lanes issue the copies
        const int nchunk = a.nb0 + a.nb1;
        uint32_t ia = 0, ib = 0;
        bool ok = true;
        for (int k = k0; ok && k < k1; ++k, ++ib) {
            const int x = (k % a.tiles_x) * a.tw, y = ((k / a.tiles_x) % a.tiles_y) * a.th, b = k / (a.tiles_x * a.tiles_y);
            const int sb = (int)(ib % kB);
            ok = __all_sync(0xffffffffu, mbar_wait_or_abort(b_empty(sb), ((ib / kB) & 1u) ^ 1u, abort_flag));
            if (!ok) break;
            if (lane == 0) mbar_expect_tx(b_full(sb), kBBytes);
            __syncwarp();
            if (lane < N / CB) tma_load_4d(smem_u32(sB + sb * kBBytes) + lane * kWgPix * CB * 2, &mapZ, lane * CB, x, y, b, b_full(sb));
            for (int m = 0; m < nm; ++m, ++ia) {
                const int sa = (int)(ia % kA);
                ok = __all_sync(0xffffffffu, mbar_wait_or_abort(a_empty(sa), ((ia / kA) & 1u) ^ 1u, abort_flag));
                if (!ok) break;
                const int j0 = (m0 + m) * kApt, nat = min(kApt, a.natoms - j0);
                if (lane == 0) mbar_expect_tx(a_full(sa), (uint32_t)nat * kAtom);
                __syncwarp();
                if (lane < nat) {
                    const int j = j0 + lane, tap = j / nchunk, c = j % nchunk;
                    const bool second = c >= a.nb0;
                    tma_load_4d(smem_u32(sA + sa * kABytes) + lane * kAtom, second ? &map1 : &map0,
                                (second ? c - a.nb0 : c) * CA, x + tap % 3 - 1, y + tap / 3 - 1, b, a_full(sa));
                }
            }
        }
        if (!ok && lane == 0) { atomicOr(a.err, DEV_GUARD); s_abort = 1; }
        // the copies issued must land before the CTA can leave
        if (lane == 0) {
            for (uint32_t i = ia > (uint32_t)kA ? ia - kA : 0; i < ia; ++i) mbar_wait(a_full((int)(i % kA)), (i / kA) & 1u);
            for (uint32_t i = ib > (uint32_t)kB ? ib - kB : 0; i < ib; ++i) mbar_wait(b_full((int)(i % kB)), (i / kB) & 1u);
        }
    } else if (warp == 1) {
        constexpr uint32_t idesc = instr_desc(N) | (1u << 15) | (1u << 16);      // A and B MN-major
        uint32_t ia = 0, ib = 0;
        bool ok = true;
        for (int k = k0; ok && k < k1; ++k, ++ib) {
            const int sb = (int)(ib % kB);
            ok = __all_sync(0xffffffffu, mbar_wait_or_abort(b_full(sb), (ib / kB) & 1u, abort_flag));
            const uint64_t db = desc_mn<CB>(smem_u32(sB + sb * kBBytes));
            for (int m = 0; ok && m < nm; ++m, ++ia) {
                const int sa = (int)(ia % kA);
                ok = __all_sync(0xffffffffu, mbar_wait_or_abort(a_full(sa), (ia / kA) & 1u, abort_flag));
                if (!ok) break;
                tc_fence_after();
                const uint64_t da = desc_mn<CA>(smem_u32(sA + sa * kABytes));
#pragma unroll
                for (int q = 0; q < kWgPix / 16; ++q)       // 16 pixels: two 8-row groups further
                    tc_mma(tmem + (uint32_t)(m * N), da + (uint64_t)(q * ((16 * CA * 2) >> 4)),
                           db + (uint64_t)(q * ((16 * CB * 2) >> 4)), idesc, (k > k0 || q > 0) ? 1u : 0u);
                tc_commit(a_empty(sa));
            }
            tc_commit(b_empty(sb));
        }
        if (!ok && lane == 0) { atomicOr(a.err, DEV_GUARD); s_abort = 1; }
        tc_commit(done);
    } else {
        const int q = warp & 3, r = q * 32 + lane;
        if (sums) {
            // a thread keeps eight channels (one 16-byte chunk, found by its tile's swizzle) of
            // every (1024 / N)-th pixel
            constexpr int kChunks = N / 8, kRows = 128 / kChunks;
            const int ch = r % kChunks, sub = ch / (CB / 8), j = ch % (CB / 8);
            float t[8] = {0.0f, 0.0f, 0.0f, 0.0f, 0.0f, 0.0f, 0.0f, 0.0f};
            uint32_t ib = 0;
            bool more = true;
            for (int k = k0; more && k < k1; ++k, ++ib) {
                const int sb = (int)(ib % kB);
                more = __all_sync(0xffffffffu, mbar_wait_or_abort(b_full(sb), (ib / kB) & 1u, abort_flag));
                if (!more) break;
                const uint8_t* tile = sB + sb * kBBytes + sub * (kWgPix * CB * 2);
#pragma unroll
                for (int p0 = 0; p0 < kWgPix; p0 += kRows) {
                    const int px = p0 + r / kChunks;
                    const int at = j ^ (CB == 64 ? px & 7 : (px >> 1) & 3);
                    const uint4 v = *reinterpret_cast<const uint4*>(tile + px * (CB * 2) + at * 16);
                    const __nv_bfloat16* h = reinterpret_cast<const __nv_bfloat16*>(&v);
#pragma unroll
                    for (int c = 0; c < 8; ++c) t[c] += __bfloat162float(h[c]);
                }
                // the loads must have returned before the slot's next copy may write it: the copy
                // is the async proxy's, and without the fence a load queued behind the MMAs'
                // operand reads can still be under way when the arrival is seen
                asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
                __syncwarp();
                if (lane == 0) mbar_arrive(b_empty(sb));
            }
            // lanes a multiple of kChunks apart hold the same channels
#pragma unroll
            for (int o = kChunks; o < 32; o <<= 1)
#pragma unroll
                for (int c = 0; c < 8; ++c) t[c] += __shfl_xor_sync(0xffffffffu, t[c], o);
            if (more && lane < kChunks)
#pragma unroll
                for (int c = 0; c < 8; ++c) atomicAdd(a.gb + ch * 8 + c, t[c]);
        }
        const bool ok = __all_sync(0xffffffffu, mbar_wait_or_abort(done, 0, abort_flag)) && !*abort_flag;
        tc_fence_after();
        if (__all_sync(0xffffffffu, ok) && k1 > k0) {
            const int nchunk = a.nb0 + a.nb1;
            for (int m = 0; m < nm; ++m) {
                const int j = (m0 + m) * kApt + r / CA, ch = r % CA, tap = j / nchunk, c = j % nchunk;
                const bool real = j < a.natoms && (a.ch_valid == 0 || ch < a.ch_valid);
                float* row = a.gw + (size_t)(tap * a.cin_out + c * CA + ch) * N;
#pragma unroll 1
                for (int c0 = 0; c0 < N; c0 += 32) {
                    uint32_t v[32];
                    tmem_ld32(tmem + (uint32_t)(m * N + c0) + ((uint32_t)(q * 32) << 16), v);
                    if (real)
#pragma unroll
                        for (int h = 0; h < 8; ++h)
                            atomicAdd(reinterpret_cast<float4*>(row + c0) + h,
                                      make_float4(__uint_as_float(v[4 * h]), __uint_as_float(v[4 * h + 1]),
                                                  __uint_as_float(v[4 * h + 2]), __uint_as_float(v[4 * h + 3])));
                }
            }
        } else if (!ok && lane == 0) {
            atomicOr(a.err, DEV_GUARD);
        }
    }
    tc_fence_before();
    __syncthreads();
    if (warp == 1)
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(kCols) : "memory");
}

// ------------------------------------------------------------------ host side
PFN_cuTensorMapEncodeTiled_v12000 encoder() {
    static PFN_cuTensorMapEncodeTiled_v12000 fn = nullptr;
    static std::once_flag once;
    std::call_once(once, [] {
        void* p = nullptr;
        cudaDriverEntryPointQueryResult q;
        if (cudaGetDriverEntryPointByVersion("cuTensorMapEncodeTiled", &p, 12000, cudaEnableDefault, &q) == cudaSuccess &&
            q == cudaDriverEntryPointSuccess)
            fn = reinterpret_cast<PFN_cuTensorMapEncodeTiled_v12000>(p);
    });
    return fn;
}

// A 2-D map of a row-major BF16 matrix [rows][ld] (ld elements, K-major rows of `cols`), read
// in boxes of 64 x box_rows with the 128-byte swizzle.
bool make_map(CUtensorMap* m, const void* base, uint64_t rows, uint64_t cols, uint64_t ld, uint32_t box_rows) {
    auto fn = encoder();
    if (!fn) return false;
    const cuuint64_t dims[2] = {cols, rows};
    const cuuint64_t strides[1] = {ld * 2};
    const cuuint32_t box[2] = {(cuuint32_t)kBK, box_rows};
    const cuuint32_t elem[2] = {1, 1};
    return fn(m, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<void*>(base), dims, strides, box, elem,
              CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
              CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}


// A 2-D weight map [rows][ld] read in boxes of cb x box_rows (128- or 64-byte swizzle).
bool make_map_cb(CUtensorMap* m, const void* base, uint64_t rows, uint64_t cols, uint64_t ld, uint32_t box_rows, int cb) {
    auto fn = encoder();
    if (!fn) return false;
    const cuuint64_t dims[2] = {cols, rows};
    const cuuint64_t strides[1] = {ld * 2};
    const cuuint32_t box[2] = {(cuuint32_t)cb, box_rows};
    const cuuint32_t elem[2] = {1, 1};
    return fn(m, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<void*>(base), dims, strides, box, elem,
              CU_TENSOR_MAP_INTERLEAVE_NONE, cb == 64 ? CU_TENSOR_MAP_SWIZZLE_128B : CU_TENSOR_MAP_SWIZZLE_64B,
              CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

// A 4-D map of an NHWC BF16 tensor [B][H][W][C], boxes of cb x tw x th x 1; coordinates
// outside the tensor read zeros (the convolution's padding).
bool make_map_nhwc(CUtensorMap* m, const void* base, int B, int H, int W, int C, int tw, int th, int cb) {
    auto fn = encoder();
    if (!fn) return false;
    const cuuint64_t dims[4] = {(cuuint64_t)C, (cuuint64_t)W, (cuuint64_t)H, (cuuint64_t)B};
    const cuuint64_t strides[3] = {(cuuint64_t)C * 2, (cuuint64_t)W * C * 2, (cuuint64_t)H * W * C * 2};
    const cuuint32_t box[4] = {(cuuint32_t)cb, (cuuint32_t)tw, (cuuint32_t)th, 1};
    const cuuint32_t elem[4] = {1, 1, 1, 1};
    return fn(m, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 4, const_cast<void*>(base), dims, strides, box, elem,
              CU_TENSOR_MAP_INTERLEAVE_NONE,
              cb == 64 ? CU_TENSOR_MAP_SWIZZLE_128B : cb == 32 ? CU_TENSOR_MAP_SWIZZLE_64B : CU_TENSOR_MAP_SWIZZLE_32B,
              CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

template <int N, int CA>
int launch_wgrad(const CUtensorMap& m0, const CUtensorMap& m1, const CUtensorMap& mz, const WgradArgs& a, cudaStream_t s) {
    const size_t smem = 1024 + wg_a_stages(N) * kWgPix * 128 * 2 + wg_b_stages(N) * kWgPix * N * 2 +
                        (2 * (wg_a_stages(N) + wg_b_stages(N)) + 1) * 8 + 16;
    static bool attr = false;
    if (!attr) {
        if (cudaFuncSetAttribute(tc_wgrad_kernel<N, CA>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem) !=
                cudaSuccess ||
            cudaFuncSetAttribute(tc_wgrad_kernel<N, CA>, cudaFuncAttributePreferredSharedMemoryCarveout,
                                 cudaSharedmemCarveoutMaxShared) != cudaSuccess)
            return RN_ERR_CUDA;
        attr = true;
    }
    tc_wgrad_kernel<N, CA><<<a.groups * a.slices, kConvThreads, smem, s>>>(m0, m1, mz, a);
    return cudaGetLastError() == cudaSuccess ? RN_OK : RN_ERR_CUDA;
}

template <int BN, int CB, int kT>
int launch_conv(const CUtensorMap& m0, const CUtensorMap& m1, const CUtensorMap& mw, const ConvArgs& a,
                const Epilogue& e, cudaStream_t s) {
    constexpr size_t smem = conv_smem(BN, CB, kT);
    static int per_sm = 0;
    if (!per_sm) {
        if (cudaFuncSetAttribute(tc_conv_kernel<BN, CB, kT>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem) !=
                cudaSuccess ||
            cudaFuncSetAttribute(tc_conv_kernel<BN, CB, kT>, cudaFuncAttributePreferredSharedMemoryCarveout,
                                 cudaSharedmemCarveoutMaxShared) != cudaSuccess)
            return RN_ERR_CUDA;
        // residency: shared memory (228 KB per SM, 1 KB reserved per CTA), TMEM (512 columns per
        // SM, 2 x BN per CTA) and at most 2 CTAs of 320 threads and 96 registers
        int smem_sm = 0;
        cudaDeviceGetAttribute(&smem_sm, cudaDevAttrMaxSharedMemoryPerMultiprocessor, ctx().device);
        const int by_smem = smem_sm / (int)(smem + kTapStatic + 1024);
        per_sm = std::max(1, std::min(std::min(by_smem, 512 / (2 * kT * BN)), 2));
    }
    const int ctas = std::min(a.items, per_sm * ctx().sm_count);
    tc_conv_kernel<BN, CB, kT><<<ctas, kTapThreads, smem, s>>>(m0, m1, mw, a, e);
    return cudaGetLastError() == cudaSuccess ? RN_OK : RN_ERR_CUDA;
}


// The row box of one source without swizzle: a 5-D view of the NHWC tensor, (8 channels, W, H, B, C / 8
// groups), read in boxes of 8 x 136 x 1 x 1 x C/8 without swizzle (the channel groups
// outermost in shared memory).
bool make_map_halo(CUtensorMap* m, const void* base, int B, int H, int W, int C) {
    auto fn = encoder();
    if (!fn) return false;
    const cuuint64_t dims[5] = {8, (cuuint64_t)W, (cuuint64_t)H, (cuuint64_t)B, (cuuint64_t)(C / 8)};
    const cuuint64_t strides[4] = {(cuuint64_t)C * 2, (cuuint64_t)W * C * 2, (cuuint64_t)H * W * C * 2, 16};
    const cuuint32_t box[5] = {8, (cuuint32_t)kHaloW, 1, 1, (cuuint32_t)(C / 8)};
    const cuuint32_t elem[5] = {1, 1, 1, 1, 1};
    return fn(m, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 5, const_cast<void*>(base), dims, strides, box, elem,
              CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
              CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}
// The resident weights: (8 columns, N rows, K / 8 groups), one box of 8 x N x kgroups.
bool make_map_wgroups(CUtensorMap* m, const void* base, int N, int ldw, int kgroups) {
    auto fn = encoder();
    if (!fn) return false;
    const cuuint64_t dims[3] = {8, (cuuint64_t)N, (cuuint64_t)(ldw / 8)};
    const cuuint64_t strides[2] = {(cuuint64_t)ldw * 2, 16};
    const cuuint32_t box[3] = {8, (cuuint32_t)N, (cuuint32_t)kgroups};
    const cuuint32_t elem[3] = {1, 1, 1};
    return fn(m, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 3, const_cast<void*>(base), dims, strides, box, elem,
              CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
              CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

// The resident weights in the fan-out order: a 5-D view (8 columns, N rows, vertical tap dy,
// channel group, horizontal tap dx) of the [N][ldw] matrix whose column is
// (3 dy + dx) cin + channel, one box of a slice of bn rows: shared memory [dx][group][dy][n][8].
bool make_map_wfan(CUtensorMap* m, const void* base, int N, int ldw, int cin, int bn) {
    auto fn = encoder();
    if (!fn) return false;
    const cuuint64_t dims[5] = {8, (cuuint64_t)N, 3, (cuuint64_t)(cin / 8), 3};
    const cuuint64_t strides[4] = {(cuuint64_t)ldw * 2, (cuuint64_t)cin * 6, 16, (cuuint64_t)cin * 2};
    const cuuint32_t box[5] = {8, (cuuint32_t)bn, 3, (cuuint32_t)(cin / 8), 3};
    const cuuint32_t elem[5] = {1, 1, 1, 1, 1};
    return fn(m, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 5, const_cast<void*>(base), dims, strides, box, elem,
              CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
              CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

template <int BN, bool kTA, bool kFan, bool kWide>
int launch_conv_halo(const CUtensorMap& m0, const CUtensorMap& m1, const CUtensorMap& mw, const HaloArgs& a,
                     const Epilogue& e, size_t smem, cudaStream_t s) {
    static size_t attr = 0;
    if (attr < smem) {
        if (cudaFuncSetAttribute(tc_conv_halo_kernel<BN, kTA, kFan, kWide>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 (int)smem) != cudaSuccess ||
            cudaFuncSetAttribute(tc_conv_halo_kernel<BN, kTA, kFan, kWide>, cudaFuncAttributePreferredSharedMemoryCarveout,
                                 cudaSharedmemCarveoutMaxShared) != cudaSuccess)
            return RN_ERR_CUDA;
        attr = smem;
    }
    int smem_sm = 0;
    cudaDeviceGetAttribute(&smem_sm, cudaDevAttrMaxSharedMemoryPerMultiprocessor, ctx().device);
    // co-resident CTAs: shared memory (dynamic, static and 1 KB reserved) and TMEM (512
    // columns an SM) both have to fit
    const int tmem_cols = kTA ? 256 : kFan ? fan_cols(kWide) : 2 * BN;
    const int per_cta = (int)(smem + kHaloStatic + 1024);
    const int per_sm = std::max(1, std::min(std::min(smem_sm / per_cta, 512 / tmem_cols), 3));
    const int ctas = std::min(a.items, per_sm * ctx().sm_count);
    tc_conv_halo_kernel<BN, kTA, kFan, kWide><<<ctas, 64 + 128 * a.sets, smem, s>>>(m0, m1, mw, a, e);
    return cudaGetLastError() == cudaSuccess ? RN_OK : RN_ERR_CUDA;
}

ConvTiling conv_tiling(int H, int W) {
    ConvTiling t{0, false};
    if (H <= 0 || W <= 0) return t;
    int lg = 0;
    while (lg < 7 && (W % (2 << lg)) == 0) ++lg;            // TW = 2^lg <= 128 divides W
    const int th = kBM >> lg;
    t.tw_log2 = lg;
    t.ok = (H % th) == 0;
    return t;
}

template <int BN>
int launch_bn(const CUtensorMap& mp, const CUtensorMap& mq, const Epilogue& e, int M, int N, int splits,
              cudaStream_t s) {
    const size_t smem = 1024 + kStages * (kBM * kBK * 2 + BN * kBK * 2) + (2 * kStages + 1) * 8 + 16;
    static bool attr = false;
    if (!attr) {
        if (cudaFuncSetAttribute(tc_gemm_kernel<BN>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem) != cudaSuccess)
            return RN_ERR_CUDA;
        attr = true;
    }
    const dim3 grid(M / kBM, N / BN, splits);
    tc_gemm_kernel<BN><<<grid, kThreads, smem, s>>>(mp, mq, e);
    return cudaGetLastError() == cudaSuccess ? RN_OK : RN_ERR_CUDA;
}

}  // namespace tc

// C (M x N, row stride ldc) = P (M x K, row stride ldp) * Q (N x K, row stride ldq)^T.
// M % 128 == 0, N in {32, 64, 128, 256} or a multiple of 128, K % (64 * splits) == 0;
// P, Q 16-byte aligned with ldp, ldq multiples of 8. splits > 1 requires c32 with atomic.
int tc_gemm(const __nv_bfloat16* P, int ldp, const __nv_bfloat16* Q, int ldq, int M, int N, int K, int splits,
            const tc::Epilogue& epi, cudaStream_t s, rn_status* st) {
    if (M <= 0 || N <= 0 || K <= 0 || M % tc::kBM || splits < 1 || K % (tc::kBK * splits))
        return fail(st, RN_ERR_INVALID, "tc_gemm shape M %d N %d K %d splits %d", M, N, K, splits);
    if ((ldp % 8) || (ldq % 8) || ((uintptr_t)P % 16) || ((uintptr_t)Q % 16))
        return fail(st, RN_ERR_INVALID, "tc_gemm operands must be 16-byte aligned rows");
    if (epi.gate) return fail(st, RN_ERR_INVALID, "tc_gemm: no gated epilogue");
    if (splits > 1 && !(epi.c32 && epi.atomic)) return fail(st, RN_ERR_INVALID, "split K needs an atomic FP32 output");
    int bn = (N == 32 || N == 64 || N == 128 || N == 256) ? N : 128;
    if (N % bn) return fail(st, RN_ERR_INVALID, "tc_gemm N %d", N);
    while (bn > ctx().tune.conv_bn_max && bn > 32) bn /= 2;     // the tuned tile width (divides N)
    tc::Epilogue e = epi;
    e.k_per_split = K / splits;
    CUtensorMap mp, mq;
    if (!tc::make_map(&mp, P, (uint64_t)M, (uint64_t)K, (uint64_t)ldp, tc::kBM) ||
        !tc::make_map(&mq, Q, (uint64_t)N, (uint64_t)K, (uint64_t)ldq, (uint32_t)bn))
        return fail(st, RN_ERR_CUDA, "cuTensorMapEncodeTiled failed");
    int rc;
    switch (bn) {
        case 32: rc = tc::launch_bn<32>(mp, mq, e, M, N, splits, s); break;
        case 64: rc = tc::launch_bn<64>(mp, mq, e, M, N, splits, s); break;
        case 256: rc = tc::launch_bn<256>(mp, mq, e, M, N, splits, s); break;
        default: rc = tc::launch_bn<128>(mp, mq, e, M, N, splits, s); break;
    }
    if (rc != RN_OK) return cuda_fail(st, cudaGetLastError(), "tc_gemm_kernel");
    return RN_OK;
}


int tc_conv3x3(const tc::ConvSrc* src, int nsrc, int B, int H, int W, const __nv_bfloat16* w, int ldw, int N,
               const tc::Epilogue& epi, __nv_bfloat16* up16, cudaStream_t s, rn_status* st) {
    if (nsrc < 1 || nsrc > 2 || !src) return fail(st, RN_ERR_INVALID, "tc_conv3x3: %d sources", nsrc);
    const tc::ConvTiling t = tc::conv_tiling(H, W);
    if (!t.ok || B <= 0) return fail(st, RN_ERR_INVALID, "tc_conv3x3: %dx%d cannot be tiled", H, W);
    int cin = 0;
    bool all64 = true, all32 = true;
    for (int i = 0; i < nsrc; ++i) {
        if (!src[i].ptr || src[i].C <= 0 || src[i].C % 16 || ((uintptr_t)src[i].ptr % 16))
            return fail(st, RN_ERR_INVALID, "tc_conv3x3: source %d (C %d)", i, src[i].C);
        all64 = all64 && src[i].C % 64 == 0;
        all32 = all32 && src[i].C % 32 == 0;
        cin += src[i].C;
    }
    if (ldw < 9 * cin || ldw % 8 || ((uintptr_t)w % 16)) return fail(st, RN_ERR_INVALID, "tc_conv3x3: weight stride %d", ldw);
    if (epi.atomic || (epi.gate && (!epi.c16 || epi.c32 || up16 || epi.head_out)))
        return fail(st, RN_ERR_INVALID, "tc_conv3x3: no atomic epilogue, and a gated one has a BF16 output alone");
    if (epi.head_out && (N != 32 || !epi.head_w || !epi.head_b || up16))
        return fail(st, RN_ERR_INVALID, "tc_conv3x3: the fused head needs N 32, its weights and no upsampled copy");
    int bn = (N == 32 || N == 64 || N == 128 || N == 256) ? N : 128;
    if (N % bn || N > 512) return fail(st, RN_ERR_INVALID, "tc_conv3x3 N %d", N);
    while (bn > ctx().tune.conv_bn_max && bn > 32) bn /= 2;
    if (up16 && !epi.c16) return fail(st, RN_ERR_INVALID, "tc_conv3x3: the upsampled copy needs a BF16 output");
    // row-ring tiles: rows of 128 pixels, channels in groups of 16, the weights resident in
    // shared memory. Row by row (conv_fan 0, conv_tmem_a): N 32 or 64 in one slice and a ring of
    // at least four row slots. Fan-out (conv_fan 1): N 32 or 64 in one slice where that fits,
    // else slices of 32 output channels (N a multiple of 32 up to 512), at least two slots, and
    // two CTAs per SM where shared memory allows, one otherwise. Sources of 16 channels have
    // only this kernel (the per-tap boxes take 32 or 64 channels).
    const bool ta = ctx().tune.conv_tmem_a && N == 32 && cin <= 32;
    const bool fan = !ta && ctx().tune.conv_fan;
    const bool ring_shape = t.tw_log2 == 7 && (9 * cin) / 8 <= 256 && cin % 16 == 0;
    const bool one_slice = N == 32 || N == 64;
    if ((ctx().tune.conv_halo || !all32) && ring_shape && (one_slice || (fan && N % 32 == 0 && N <= 512))) {
        const uint32_t a_bytes = (uint32_t)cin / 8 * tc::kHaloGroup;
        // a row slot; two swizzled sources each start on 1024 bytes
        const uint32_t a_stride = tc::halo_slot(src[0].C, nsrc > 1 ? src[1].C : 0, fan);
        auto chunk = [](int C) { return tc::chunk_channels(C); };
        const size_t bars = (size_t)(2 * 8 + 2 * tc::kFanMaxAcc + 2) * 8 + 16;
        int bn = one_slice && (N == 32 || !fan || ctx().tune.conv_fan_bn == 64) ? N : 32, stages = 0;
        uint32_t b_bytes = 0, b_pad = 0;
        int sets = 1;
        auto fit = [&](int bnf) {
            b_bytes = (uint32_t)bnf * 9 * cin * 2;
            b_pad = (b_bytes + 1023) & ~1023u;
            const size_t stat = tc::kHaloStatic + tc::halo_stage(bnf, 1);
            if (!fan) {
                // dynamic shared memory: 227 KB a block less the kernel's static arrays (the
                // bias, the abort flag and the epilogue's BF16 stage of 4 x 32 pixels x N)
                const size_t budget = 220 * 1024 - stat;
                return (int)std::min<size_t>(8, (budget - std::min<size_t>(budget, b_pad + 2048)) / a_stride);
            }
            // fan-out: a slot is busy only until its own MMAs have run: four at most (4, 6 and 8
            // measured alike); two CTAs per SM (228 KB less 1 KB reserved each) where two slots
            // fit, else one CTA with the whole 227 KB of a block
            for (const size_t cta : {(size_t)228 * 1024 / 2 - 1024, (size_t)227 * 1024})
                for (sets = 2; sets >= 1; --sets) {
                    const size_t fixed = tc::kHaloStatic + tc::halo_stage(bnf, sets) + 1024 + bars + b_pad;
                    const size_t room = cta > fixed ? (cta - fixed) / a_stride : 0;
                    if (room >= 2) return (int)std::min<size_t>(4, room);
                }
            sets = 1;
            return 0;
        };
        stages = fit(bn);
        if (fan && bn == 64 && stages < 2) {
            bn = 32;
            stages = fit(bn);
        }
        CUtensorMap hm[2], hw;
        bool maps = stages >= (fan ? 2 : 4) && (fan || one_slice);
        for (int i = 0; maps && i < nsrc; ++i)
            maps = fan ? tc::make_map_nhwc(&hm[i], src[i].ptr, B, H, W, src[i].C, tc::kHaloW, 1, chunk(src[i].C))
                       : tc::make_map_halo(&hm[i], src[i].ptr, B, H, W, src[i].C);
        if (maps && nsrc == 1) hm[1] = hm[0];
        maps = maps && (fan ? tc::make_map_wfan(&hw, w, N, ldw, cin, bn) : tc::make_map_wgroups(&hw, w, N, ldw, 9 * cin / 8));
        if (maps) {
            tc::HaloArgs h{};
            h.nsrc = nsrc; h.C0 = src[0].C; h.C1 = nsrc > 1 ? src[1].C : 0; h.cin = cin;
            h.cb0 = chunk(src[0].C); h.cb1 = nsrc > 1 ? chunk(src[1].C) : 16;
            h.nch0 = src[0].C / h.cb0; h.nch1 = nsrc > 1 ? src[1].C / h.cb1 : 0;
            h.q16 = cin / 16;
            h.B = B; h.H = H; h.W = W;
            // chunks of 16 output rows (2 halo rows re-read per chunk), fewer where that leaves
            // less than two items per SM
            h.chunk = 16;
            while (h.chunk > 4 && (long)(W / 128) * B * ((H + h.chunk - 1) / h.chunk) < 2L * ctx().sm_count) h.chunk /= 2;
            h.chunks_y = (H + h.chunk - 1) / h.chunk;
            h.n_slices = N / bn;
            h.slice_items = (W / 128) * h.chunks_y * B;
            h.items = h.n_slices * h.slice_items;
            h.stages = stages;
            h.sets = sets;
            h.a_bytes = a_bytes; h.b_bytes = b_bytes;
            h.up16 = up16;
            const size_t smem = 1024 + b_pad + (size_t)stages * a_stride + tc::halo_stage(bn, sets) + bars;
            const bool wide = smem + tc::kHaloStatic + 1024 > (size_t)228 * 1024 / 2;      // one CTA per SM
            const int rc = ta    ? tc::launch_conv_halo<32, true, false, false>(hm[0], hm[1], hw, h, epi, smem, s)
                         : fan && wide ? (bn == 32 ? tc::launch_conv_halo<32, false, true, true>(hm[0], hm[1], hw, h, epi, smem, s)
                                                   : tc::launch_conv_halo<64, false, true, true>(hm[0], hm[1], hw, h, epi, smem, s))
                         : fan   ? (bn == 32 ? tc::launch_conv_halo<32, false, true, false>(hm[0], hm[1], hw, h, epi, smem, s)
                                             : tc::launch_conv_halo<64, false, true, false>(hm[0], hm[1], hw, h, epi, smem, s))
                         : N == 32 ? tc::launch_conv_halo<32, false, false, false>(hm[0], hm[1], hw, h, epi, smem, s)
                                   : tc::launch_conv_halo<64, false, false, false>(hm[0], hm[1], hw, h, epi, smem, s);
            if (rc != RN_OK) return cuda_fail(st, cudaGetLastError(), "tc_conv_halo_kernel");
            return RN_OK;
        }
    }
    if (!all32)
        return fail(st, RN_ERR_INVALID, "tc_conv3x3: 16-channel sources need 128-pixel rows, N 32 or 64 and resident weights");
    const int cb = all64 ? 64 : 32;
    const int tw = 1 << t.tw_log2, th = tc::kBM >> t.tw_log2;
    CUtensorMap m[2], mw;
    for (int i = 0; i < nsrc; ++i)
        if (!tc::make_map_nhwc(&m[i], src[i].ptr, B, H, W, src[i].C, tw, th, cb))
            return fail(st, RN_ERR_CUDA, "cuTensorMapEncodeTiled (activation) failed");
    if (nsrc == 1) m[1] = m[0];
    if (!tc::make_map_cb(&mw, w, (uint64_t)N, (uint64_t)ldw, (uint64_t)ldw, (uint32_t)bn, cb))
        return fail(st, RN_ERR_CUDA, "cuTensorMapEncodeTiled (weights) failed");
    tc::ConvArgs a{};
    a.nsrc = nsrc;
    a.C0 = src[0].C;
    a.C1 = nsrc > 1 ? src[1].C : 0;
    a.B = B; a.H = H; a.W = W; a.tw_log2 = t.tw_log2;
    a.tiles_x = W / tw; a.tiles_y = H / th;
    a.cin = cin;
    a.n_slices = N / bn;
    // two tiles per item where the tile count is even, both accumulator pairs fit in TMEM and
    // the doubled A stages keep as many CTAs per SM as single tiles do
    const long tiles = (long)a.tiles_x * a.tiles_y * B;
    auto resident = [&](int kt) {
        int smem_sm = 0;
        cudaDeviceGetAttribute(&smem_sm, cudaDevAttrMaxSharedMemoryPerMultiprocessor, ctx().device);
        return std::min(std::min(smem_sm / (int)(tc::conv_smem(bn, cb, kt) + tc::kTapStatic + 1024), 512 / (2 * kt * bn)), 2);
    };
    const bool pair = ctx().tune.conv_pair && tiles % 2 == 0 && bn <= 128 && resident(2) >= std::max(1, resident(1));
    a.items = (int)(tiles / (pair ? 2 : 1)) * a.n_slices;
    a.up16 = up16;
    int rc;
#define RN_CONV_CASE(BNV, KT)                                                                         \
    case BNV:                                                                                         \
        rc = cb == 64 ? tc::launch_conv<BNV, 64, KT>(m[0], m[1], mw, a, epi, s)                       \
                      : tc::launch_conv<BNV, 32, KT>(m[0], m[1], mw, a, epi, s);                      \
        break;
    if (pair) {
        switch (bn) {
            RN_CONV_CASE(32, 2)
            RN_CONV_CASE(64, 2)
            default: RN_CONV_CASE(128, 2)
        }
    } else {
        switch (bn) {
            RN_CONV_CASE(32, 1)
            RN_CONV_CASE(64, 1)
            RN_CONV_CASE(256, 1)
            default: RN_CONV_CASE(128, 1)
        }
    }
#undef RN_CONV_CASE
    if (rc != RN_OK) return cuda_fail(st, cudaGetLastError(), "tc_conv_kernel");
    return RN_OK;
}

int tc_wgrad3x3(const tc::ConvSrc* src, int nsrc, int B, int H, int W, const __nv_bfloat16* dz, int N, float* gw,
                int cin_out, int ch_valid, float* gb, uint32_t* err, cudaStream_t s, rn_status* st) {
    const tc::ConvTiling t = tc::conv_tiling(H, W);
    if (nsrc < 1 || nsrc > 2 || !src || !dz || !gw || B <= 0 || !t.ok)
        return fail(st, RN_ERR_INVALID, "tc_wgrad3x3: %dx%dx%d, %d sources", B, H, W, nsrc);
    if (N != 32 && N != 64 && N != 128 && N != 256) return fail(st, RN_ERR_INVALID, "tc_wgrad3x3 N %d", N);
    int ca = 64;
    for (int i = 0; i < nsrc; ++i)
        while (ca >= 16 && src[i].C % ca) ca /= 2;
    if (ca < 16) return fail(st, RN_ERR_INVALID, "tc_wgrad3x3: source channels");
    // 64-pixel boxes: tw x th with tw a power of two dividing W, th dividing H
    const int tw = std::min(1 << t.tw_log2, tc::kWgPix), th = tc::kWgPix / tw;
    CUtensorMap m[2], mz;
    for (int i = 0; i < nsrc; ++i)
        if (!tc::make_map_nhwc(&m[i], src[i].ptr, B, H, W, src[i].C, tw, th, ca))
            return fail(st, RN_ERR_CUDA, "cuTensorMapEncodeTiled (activation) failed");
    if (nsrc == 1) m[1] = m[0];
    if (!tc::make_map_nhwc(&mz, dz, B, H, W, N, tw, th, N >= 64 ? 64 : 32))
        return fail(st, RN_ERR_CUDA, "cuTensorMapEncodeTiled (gradient) failed");
    tc::WgradArgs a{};
    a.nb0 = src[0].C / ca;
    a.nb1 = nsrc > 1 ? src[1].C / ca : 0;
    a.tw = tw; a.th = th;
    a.tiles_x = W / tw; a.tiles_y = H / th;
    a.boxes = B * a.tiles_x * a.tiles_y;
    a.natoms = 9 * (a.nb0 + a.nb1);
    a.mtiles = (a.natoms * ca + 127) / 128;
    // groups of equal size, at most 256 TMEM columns; pixel slices so that the items fill two
    // CTAs an SM once
    a.groups = (a.mtiles + 256 / N - 1) / (256 / N);
    a.per_group = (a.mtiles + a.groups - 1) / a.groups;
    a.groups = (a.mtiles + a.per_group - 1) / a.per_group;
    a.slices = std::max(1, std::min(a.boxes, 2 * ctx().sm_count / a.groups));
    a.cin_out = cin_out;
    a.ch_valid = ch_valid;
    a.gw = gw;
    a.gb = gb;
    a.err = err;
    int rc = RN_ERR_INVALID;
#define RN_WGRAD_CASE(NV)                                                            \
    case NV:                                                                         \
        rc = ca == 64   ? tc::launch_wgrad<NV, 64>(m[0], m[1], mz, a, s)             \
             : ca == 32 ? tc::launch_wgrad<NV, 32>(m[0], m[1], mz, a, s)             \
                        : tc::launch_wgrad<NV, 16>(m[0], m[1], mz, a, s);            \
        break;
    switch (N) {
        RN_WGRAD_CASE(32)
        RN_WGRAD_CASE(64)
        RN_WGRAD_CASE(128)
        RN_WGRAD_CASE(256)
    }
#undef RN_WGRAD_CASE
    if (rc != RN_OK) return cuda_fail(st, cudaGetLastError(), "tc_wgrad_kernel");
    return RN_OK;
}

}  // namespace rn

using namespace rn;

// Test and measurement entry of the GEMM (device pointers, the library's stream).
extern "C" int rn_tc_gemm(const void* P, int ldp, const void* Q, int ldq, int M, int N, int K, int splits, float* c32,
                          void* c16, int ldc, const float* bias, int relu, rn_status* st) {
    RN_TRY(ensure_ctx(st));
    tc::Epilogue e{};
    e.ldc = ldc;
    e.c32 = c32;
    e.c16 = (__nv_bfloat16*)c16;
    e.bias = bias;
    e.relu = relu;
    e.atomic = splits > 1;
    e.err = ctx().dev_error;
    RN_TRY(tc_gemm((const __nv_bfloat16*)P, ldp, (const __nv_bfloat16*)Q, ldq, M, N, K, splits, e, ctx().stream, st));
    return ok(st);
}

// Test and measurement entry of the implicit 3x3 convolution (device pointers, NHWC BF16
// sources, the library's stream).
extern "C" int rn_tc_conv3x3(const void* src0, int c0, const void* src1, int c1, int B, int H, int W, const void* w,
                             int ldw, int N, float* c32, void* c16, void* up16, const float* bias, int relu,
                             rn_status* st) {
    RN_TRY(ensure_ctx(st));
    tc::ConvSrc src[2] = {{(const __nv_bfloat16*)src0, c0}, {(const __nv_bfloat16*)src1, c1}};
    tc::Epilogue e{};
    e.ldc = N;
    e.c32 = c32;
    e.c16 = (__nv_bfloat16*)c16;
    e.bias = bias;
    e.relu = relu;
    e.err = ctx().dev_error;
    RN_TRY(tc_conv3x3(src, src1 ? 2 : 1, B, H, W, (const __nv_bfloat16*)w, ldw, N, e, (__nv_bfloat16*)up16,
                      ctx().stream, st));
    return ok(st);
}

// Self-test of the device-side wait budget (no counterpart in the reference): a 128 x 32 x 64
// GEMM whose only K block's copies are withheld, so its stage never fills. The MMA thread's
// bounded wait gives up after `spin_limit` rounds, sets the error word and the CTA frees its
// TMEM and returns: the call must come back with RN_ERR_BUDGET and leave the context usable.
extern "C" int rn_selftest_wait_budget(uint32_t spin_limit, rn_status* st) {
    RN_TRY(ensure_ctx(st));
    if (spin_limit == 0 || spin_limit > (1u << 24)) return fail(st, RN_ERR_INVALID, "spin limit %u", spin_limit);
    ScopedDev pb, qb, cb;
    RN_CUDA(cudaMalloc(&pb.p, 128 * 64 * 2), st);
    RN_CUDA(cudaMalloc(&qb.p, 32 * 64 * 2), st);
    RN_CUDA(cudaMalloc(&cb.p, 128 * 32 * 4), st);
    void *p = pb.p, *q = qb.p, *c = cb.p;
    RN_CUDA(cudaMemsetAsync(p, 0, 128 * 64 * 2, ctx().stream), st);
    RN_CUDA(cudaMemsetAsync(q, 0, 32 * 64 * 2, ctx().stream), st);
    tc::Epilogue e{};
    e.ldc = 32;
    e.c32 = (float*)c;
    e.err = ctx().dev_error;
    e.spin = spin_limit;
    e.withhold = 1;
    int rc = tc_gemm((const __nv_bfloat16*)p, 64, (const __nv_bfloat16*)q, 64, 128, 32, 64, 1, e, ctx().stream, st);
    if (rc == RN_OK) rc = check_device_error(st, "rn_selftest_wait_budget");
    cudaStreamSynchronize(ctx().stream);
    return rc;
}
