// 3x3x3 convolutions (padding 1, stride 1 or 2) of the warm-start network
// on the fifth-generation tensor cores: tcgen05.mma with the accumulators in
// tensor memory; and the weight gradients.  No reference counterpart (the
// reference always starts from rest).
//
// A CTA computes output blocks of 8 (x) x 16 (y) x TZ (z) voxels (TZ = 4 at
// stride 1, 1 at stride 2) and all co output channels.  Per 16-channel chunk
// of the input it stages the input voxels the block reads (the block plus
// its one-voxel halo, 10 x 18 x 6 at stride 1; 17 x 33 x 3 at stride 2),
// zero outside the grid (the padding), and the chunk of all 27 taps'
// weights, in the canonical no-swizzle K-major layout of the MMA operands:
// core matrices of 8 rows x 16 bytes (8 channels), rows 16 bytes apart.
//   input:   [channel half k (2)][x parity p (S)][z][y][x / S][8 channels]
//   weights: [tap block][co / 8][channel half k][co % 8][8 channels]
//            (stride 1: blocks in weight_block's order)
// The 128 output voxels of one z plane (8 x by 16 y) are the M = 128 rows
// of one MMA: row m = 8 y + x.  Output x reads input x = S x + tx - 1, so
// with the input's x split by parity (stride 2: even and odd columns in
// separate runs) rows m..m+7 are 8 consecutive staged voxels -- one core
// matrix -- and the 16 groups of 8 rows are 16 output rows, S input rows
// apart: the stride-dimension offset.  The two channel halves of the K = 16
// slice are one staged half apart: the leading-dimension offset.  A tap
// (tx, ty, tz) is just the descriptor's start address (parity tx mod S,
// column tx / S, row ty, plane S z + tz): the 27 taps reuse the staged block
// with no copies.  One thread issues the MMAs of a chunk (M = 128, K = 16,
// BF16 x BF16 -> FP32) into TZ accumulators of co tensor-memory columns each
// and commits them to an mbarrier; every wait is bounded.  At stride 2: 27
// MMAs of N = co.  At stride 1 the accumulators of the TZ planes are adjacent
// column ranges and one staged plane feeds up to three output planes (through
// taps tz = 2, 1, 0), so each (ty, tx) takes one MMA per staged plane with
// N = 1-3 co: 9 x 6 = 54 MMAs instead of 4 x 27, each reading its A operand
// once.  The epilogue reads the accumulators with tcgen05.ld (warp w owns
// tensor-memory lanes 32 w .. 32 w + 31, i.e. rows y = 4 w .. 4 w + 3), adds
// the bias, applies ReLU and stores BF16 (and FP32 when asked) channels-last.
#include <cuda.h>
#include <cuda_bf16.h>

#include <atomic>
#include <cstdint>
#include <type_traits>

#include "lbm_internal.cuh"

namespace {

using bf16 = __nv_bfloat16;

constexpr int TX = 8, TY = 16;
constexpr int kThreads = 128;
constexpr long kWaitLimit = 1L << 20;  // mbarrier polls (each bounded by the hardware's own time limit)

// Staged geometry at stride 2: planes, rows, and voxels per x parity run
// (input x = 2 xh + p).
struct Geo2 {
    static constexpr int ZB = 3, YB = 2 * (TY - 1) + 3, XH = TX + 1;
    static constexpr int PLANE_RAW = ZB * YB * XH * 16;          // bytes one copy writes
    static constexpr int PLANE = (PLANE_RAW + 127) / 128 * 128;  // copy destinations 128-byte aligned
    static constexpr int HALF = 2 * PLANE;                       // bytes of one channel half
    static constexpr int TILE = 2 * HALF;
    static constexpr int TX_BYTES = 4 * PLANE_RAW;               // bytes the copies of a chunk deliver
};

// Set when a bounded wait gave up (read and cleared by conv_tc_status).
__device__ unsigned g_conv_tc_flags;

__device__ __forceinline__ uint32_t saddr(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }

// Shared-memory matrix descriptor, no swizzle: start address, leading-
// dimension (K-direction core matrix) byte offset, stride-dimension (next 8
// rows) byte offset, descriptor version 1.
__device__ __forceinline__ uint64_t smem_desc(uint32_t addr, uint32_t lbo, uint32_t sbo) {
    return (uint64_t)((addr >> 4) & 0x3FFFu) | ((uint64_t)((lbo >> 4) & 0x3FFFu) << 16) |
           ((uint64_t)((sbo >> 4) & 0x3FFFu) << 32) | ((uint64_t)1 << 46);
}

// Instruction descriptor of kind::f16: FP32 accumulator, BF16 A and B, both
// K-major, N >> 3 at bit 17, M >> 4 at bit 24.
__host__ __device__ constexpr uint32_t idesc_bf16(int m, int n) {
    return (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(n >> 3) << 17) | ((uint32_t)(m >> 4) << 24);
}

__device__ __forceinline__ void cp_async16(uint32_t dst, const void* src, bool valid) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(valid ? 16 : 0)
                 : "memory");
}

__device__ __forceinline__ void mbar_init(uint32_t bar, uint32_t count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bar), "r"(count) : "memory");
}

__device__ __forceinline__ bool mbar_try(uint32_t bar, uint32_t parity) {
    uint32_t done;
    asm volatile(
        "{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\tselp.u32 %0, 1, 0, p;\n\t}\n"
        : "=r"(done)
        : "r"(bar), "r"(parity)
        : "memory");
    return done != 0;
}

__device__ __forceinline__ bool mbar_wait(uint32_t bar, uint32_t parity) {
    for (long k = 0; k < kWaitLimit; ++k)
        if (mbar_try(bar, parity)) return true;
    return false;
}

__device__ __forceinline__ void mbar_expect_tx(uint32_t bar, uint32_t bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
}

// 4-D tiled tensor copy global -> shared completing on an mbarrier;
// coordinates innermost first (channel, x, y, z).
__device__ __forceinline__ void tma_load4(uint32_t dst, const CUtensorMap* map, int c0, int c1, int c2, int c3,
                                          uint32_t bar) {
    asm volatile(
        "cp.async.bulk.tensor.4d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4, "
        "%5}], [%6];" ::"r"(dst),
        "l"(reinterpret_cast<uint64_t>(map)), "r"(c0), "r"(c1), "r"(c2), "r"(c3), "r"(bar)
        : "memory");
}

__device__ __forceinline__ void mma_bf16(uint32_t dtmem, uint64_t adesc, uint64_t bdesc, uint32_t idesc,
                                         uint32_t accumulate) {
    asm volatile(
        "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}\n" ::"r"(dtmem),
        "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate)
        : "memory");
}

// 16 columns of this warp's 32 lanes, without waiting; tc_ld_wait waits for
// every load issued and orders the registers' use behind it.
__device__ __forceinline__ void tc_ld16_issue(uint32_t taddr, uint32_t (&r)[16]) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
          "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
        : "r"(taddr));
}

__device__ __forceinline__ void tc_ld_wait(uint32_t (&r)[4][16]) {
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
    for (int k = 0; k < 4; ++k)
#pragma unroll
        for (int e = 0; e < 16; ++e) asm volatile("" : "+r"(r[k][e]));
}

__device__ __forceinline__ void tc_ld16(uint32_t taddr, float (&v)[16]) {
    uint32_t r[16];
    tc_ld16_issue(taddr, r);
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
    for (int k = 0; k < 16; ++k) {
        asm volatile("" : "+r"(r[k]));
        v[k] = __uint_as_float(r[k]);
    }
}

// 16 channels at element `at` of the output from their FP32 sums: bias (of those channels), ReLU, BF16 (and FP32) store.
__device__ __forceinline__ void store16(float (&v)[16], const float* __restrict__ bias, int relu, bf16* __restrict__ y,
                                        float* __restrict__ y32, int64_t at) {
#pragma unroll
    for (int k = 0; k < 16; ++k) {
        v[k] += bias ? bias[k] : 0.f;
        if (relu) v[k] = fmaxf(v[k], 0.f);
    }
    uint4 p[2];
    __nv_bfloat162* h = reinterpret_cast<__nv_bfloat162*>(p);
#pragma unroll
    for (int k = 0; k < 8; ++k) h[k] = __floats2bfloat162_rn(v[2 * k], v[2 * k + 1]);
    uint4* dst = reinterpret_cast<uint4*>(y + at);
    dst[0] = p[0];
    dst[1] = p[1];
    if (y32) {
        float4* d32 = reinterpret_cast<float4*>(y32 + at);
#pragma unroll
        for (int k = 0; k < 4; ++k) d32[k] = make_float4(v[4 * k], v[4 * k + 1], v[4 * k + 2], v[4 * k + 3]);
    }
}

// Shared-memory block of tap t = 9 tz + 3 ty + tx in the weights staged at
// stride 1: the three z taps of each (ty, tx) in the order tz = 2, 1, 0, so
// that one MMA of N = 3 co takes all three: staged plane zz feeds output
// planes zz - 2, zz - 1, zz through taps tz = 2, 1, 0, and the accumulators
// of those planes are the adjacent tensor-memory column ranges (z co .. z co
// + co - 1 for plane z).
__host__ __device__ constexpr int weight_block(int t) { return ((t / 3) % 3 * 3 + t % 3) * 3 + (2 - t / 9); }

// One lane of a converged warp.
__device__ __forceinline__ bool elect_one() {
    uint32_t p;
    asm volatile("{\n\t.reg .pred p;\n\telect.sync _|p, 0xffffffff;\n\tselp.u32 %0, 1, 0, p;\n\t}\n" : "=r"(p));
    return p != 0;
}

__device__ __forceinline__ void mbar_arrive(uint32_t bar) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory");
}

__device__ __forceinline__ void tc_commit(uint32_t bar) {
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar) : "memory");
}

template <int CO>
__host__ __device__ constexpr int smem_bytes() {
    return Geo2::TILE + 27 * CO * 32 + 32;  // input, weights, two mbarriers + tensor-memory address
}

template <int CO>
__host__ __device__ constexpr uint32_t tmem_cols() {
    return CO < 32 ? 32u : (uint32_t)CO;  // a power of two for CO in {16, 32, 64}
}

// Stride 2.  x [Di][Hi][Wi][ci] (read through `map`: the 4-D tensor map of x,
// box 8 channels x 2 XH with element stride 2 x YB x ZB), w [co][27][ci],
// y [Do][Ho][Wo][co] with Do = Di / 2 etc.; Ho % 16 == 0, Wo % 8 == 0 (the
// launcher checks).  The input by tensor copies (one per channel half and x
// parity, element stride 2 along x), the weights by cp.async.
template <int CO>
__global__ void __launch_bounds__(kThreads) k_conv3_s2_tc(const __grid_constant__ CUtensorMap map,
                                                          const bf16* __restrict__ w, const float* __restrict__ bias,
                                                          bf16* __restrict__ y, float* __restrict__ y32, int Do, int Ho,
                                                          int Wo, int ci, int relu) {
    using G = Geo2;
    extern __shared__ __align__(128) unsigned char smem[];
    unsigned char* tile = smem;
    unsigned char* wsm = smem + G::TILE;
    uint64_t* bar = reinterpret_cast<uint64_t*>(wsm + 27 * CO * 32);  // [0] MMAs done, [1] input copies done
    uint32_t* tslot = reinterpret_cast<uint32_t*>(bar + 2);
    volatile int& copy_failed = *reinterpret_cast<volatile int*>(tslot + 1);
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int nbx = Wo / TX, nby = Ho / TY;
    const int bx = blockIdx.x % nbx, by = (blockIdx.x / nbx) % nby, z0 = blockIdx.x / (nbx * nby);
    const int x0 = bx * TX, y0 = by * TY;
    constexpr uint32_t NCOL = tmem_cols<CO>();

    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(saddr(tslot)),
                     "r"(NCOL)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    if (tid == 0) {
        mbar_init(saddr(bar), 1);
        mbar_init(saddr(bar + 1), 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        copy_failed = 0;
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem = *tslot;

    const uint32_t tile_a = saddr(tile), w_a = saddr(wsm);
    constexpr uint32_t IDESC = idesc_bf16(128, CO);
    constexpr uint32_t SBO = 2 * G::XH * 16;  // two input rows per output row
    bool ok = true;
    const int chunks = ci / 16;
    int c = 0;
    for (; c < chunks && ok; ++c) {
        // the input voxels of this chunk by tensor copies (zero outside the grid: the padding)
        if (tid == 0) {
            mbar_expect_tx(saddr(bar + 1), (uint32_t)G::TX_BYTES);
            for (int k = 0; k < 2; ++k)
                for (int p = 0; p < 2; ++p)
                    tma_load4(tile_a + k * G::HALF + p * G::PLANE, &map, c * 16 + k * 8, 2 * x0 - 1 + p, 2 * y0 - 1,
                              2 * z0 - 1, saddr(bar + 1));
        }
        // the weights of this chunk
        for (int i = tid; i < 27 * CO * 2; i += kThreads) {
            const int k = i & 1, n = (i >> 1) % CO, t = (i >> 1) / CO;
            cp_async16(w_a + t * (CO * 32) + (n >> 3) * 256 + k * 128 + (n & 7) * 16,
                       w + ((int64_t)n * 27 + t) * ci + c * 16 + k * 8, true);
        }
        asm volatile("cp.async.commit_group;\n\tcp.async.wait_group 0;" ::: "memory");
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        __syncthreads();
        if (tid == 0) {
            if (mbar_wait(saddr(bar + 1), (uint32_t)(c & 1))) {
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                for (int t = 0; t < 27; ++t) {
                    const int tz = t / 9, ty = (t / 3) % 3, tx = t % 3;
                    const uint32_t a = tile_a + (tx & 1) * G::PLANE + ((tz * G::YB + ty) * G::XH + tx / 2) * 16;
                    mma_bf16(tmem, smem_desc(a, G::HALF, SBO), smem_desc(w_a + t * (CO * 32), 128, 256), IDESC,
                             (c > 0 || t > 0) ? 1u : 0u);
                }
                tc_commit(saddr(bar));
            } else {
                copy_failed = 1;
            }
        }
        __syncthreads();
        if (copy_failed) {
            // the copies did not complete in time: record it and wait
            // (bounded) once more before the shared memory is released
            if (tid == 0) {
                atomicOr(&g_conv_tc_flags, 2u);
                mbar_wait(saddr(bar + 1), (uint32_t)(c & 1));
            }
            ok = false;
            c = -1;  // no MMAs of this chunk to wait for; those of earlier chunks are done
            break;
        }
        // every thread: the MMAs of this chunk are done (they read the staged block)
        ok = mbar_wait(saddr(bar), (uint32_t)(c & 1));
        ok = __syncthreads_and(ok);
    }
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    if (ok) {
        // epilogue: warp w reads lanes 32 w .. 32 w + 31 = rows y = 4 w + lane / 8, x = lane % 8
        const int m = 32 * warp + lane;
        const int64_t vox = ((int64_t)z0 * Ho + y0 + (m >> 3)) * Wo + x0 + (m & 7);
#pragma unroll
        for (int c16 = 0; c16 < CO / 16; ++c16) {
            float v[16];
            tc_ld16(tmem + ((uint32_t)(32 * warp) << 16) + (uint32_t)(c16 * 16), v);
            store16(v, bias ? bias + c16 * 16 : nullptr, relu, y, y32, vox * CO + c16 * 16);
        }
    } else if (c > 0) {
        // the wait of chunk c - 1 gave up: record it, wait (bounded) once
        // more for that chunk's MMAs, then release the tensor memory
        if (tid == 0) atomicOr(&g_conv_tc_flags, 1u);
        mbar_wait(saddr(bar), (uint32_t)((c - 1) & 1));
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    if (warp == 0)
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(NCOL) : "memory");
}

// ---------------------------------------------------------------------------
// Stride 1 (forward, and the input gradient with flipped weights): any grid,
// of which conv3_tc_applies gives it those of 16 rows or more.
// The same block (8 x 16 x 4 outputs), staged layout and MMAs as described
// at the top, in one persistent CTA an SM whose warps each do one thing:
//   warps 0-3  epilogue: tensor memory -> bias, ReLU -> global memory
//   warp 4     one thread issues the MMAs
//   warps 5-12 producers: the block's input voxels (16 channels) into the
//              next of NS stages by cp.async, zero outside the grid
// so the copies of later blocks and the stores of the previous one run
// beside the current one's MMAs (two sets of accumulators), and the weights
// of CO output channels (16, or 32 of 32 or 64: grid.y) are staged once per
// CTA.  mbarriers hand over the stages (full / empty) and accumulators
// (tfull / tempty); every wait is bounded, and a role that gives up raises
// the flag and leaves, whereupon the others' waits run out.
//
// What bounds it: the MMAs, at 77 to 83 SM cycles each whatever their N up to
// 192 (ncu: 4364 a SM in 335k cycles at N = 64 to 192, 1091 in 90k at N = 16 to
// 48; each reads a 4 KB A operand from shared memory), 54 a chunk.  Neighbours
// that add to the same accumulators are not the reason: two blocks' MMAs
// issued in turn ran the same 117 us at 16 -> 16 channels.  The kernel before
// staged with tensor copies, whose 8-channel layout is boxes of 16-byte
// rows: 2160 a chunk at about 3 cycles each, 7.2k cycles a chunk whatever
// its MMAs.  The same bytes by cp.async are 68 warp instructions.  256 x 128
// x 128: 16 -> 16 196 -> 117 us, 32 -> 16 278 -> 186 us; 128 x 64 x 64:
// 64 -> 32 82 -> 64 us (906 TFLOP/s), 64 -> 64 123 us (167 with all 64
// output channels in one CTA, whose weights do not fit beside the stages).
constexpr int kPipeZ = 4;                                  // output planes of a block
constexpr int kPipeVox = (kPipeZ + 2) * 18 * 10;           // staged voxels of a block
constexpr int kPipeHalf = kPipeVox * 16 + 64;              // bytes of an 8-channel half (+64: the halves in different banks)
constexpr int kPipeTile = 2 * kPipeHalf;
constexpr int kProducers = 256;
constexpr int kPipeThreads = 32 * (4 + 1) + kProducers;
constexpr int kPipeBars = 256;                             // bytes for barriers and the tensor-memory address

// The weights [co][27][ci] of 16-channel chunk c into dst: tap blocks of CO
// rows in weight_block's order, canonical K-major core matrices.
template <int CO>
__device__ __forceinline__ void stage_weights(uint32_t dst, const bf16* __restrict__ w, int ci, int c, int tid, int n) {
    for (int i = tid; i < 27 * CO * 2; i += n) {
        const int k = i & 1, o = (i >> 1) % CO, t = (i >> 1) / CO;
        cp_async16(dst + weight_block(t) * (CO * 32) + (o >> 3) * 256 + k * 128 + (o & 7) * 16,
                   w + ((int64_t)o * 27 + t) * ci + c * 16 + k * 8, true);
    }
}

// The five other warps' weight copies are done and visible to the MMAs.
__device__ __forceinline__ void weights_staged() {
    asm volatile("cp.async.commit_group;\n\tcp.async.wait_group 0;" ::: "memory");
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    asm volatile("bar.sync 1, %0;" ::"n"(kPipeThreads - kProducers) : "memory");
}

template <int CO>
__global__ void __launch_bounds__(kPipeThreads, 1) k_conv3_pipe(const bf16* __restrict__ x, const bf16* __restrict__ w,
                                                              const float* __restrict__ bias, bf16* __restrict__ y,
                                                              float* __restrict__ y32, int D, int H, int W, int ci,
                                                              int co, int relu, int ntiles, int NS) {
    constexpr int STAGE = kPipeTile;
    constexpr uint32_t ACC = kPipeZ * CO, NCOL = 2 * ACC;  // tensor-memory columns of one / both accumulator sets
    extern __shared__ __align__(128) unsigned char smem[];
    const int chunks = ci / 16;
    const int o0 = blockIdx.y * CO;  // first output channel
    w += (int64_t)o0 * 27 * ci;
    if (bias) bias += o0;
    // [barriers][weights of all chunks][stages]
    uint64_t* full = reinterpret_cast<uint64_t*>(smem);
    uint64_t* empty = full + 8;
    uint64_t* tfull = empty + 8;
    uint64_t* tempty = tfull + 2;
    uint32_t* tslot = reinterpret_cast<uint32_t*>(tempty + 2);
    const uint32_t wres = saddr(smem) + kPipeBars, stages = wres + 27 * CO * 32 * chunks;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int nbx = (W + TX - 1) / TX, nby = (H + TY - 1) / TY;

    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(saddr(tslot)),
                     "r"(NCOL)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    if (tid == 0) {
        for (int s = 0; s < NS; ++s) {
            mbar_init(saddr(full + s), kProducers / 32);
            mbar_init(saddr(empty + s), 1);
        }
        for (int b = 0; b < 2; ++b) {
            mbar_init(saddr(tfull + b), 1);
            mbar_init(saddr(tempty + b), 4);
        }
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem = *tslot;
    bool ok = true;
    if (warp < 5) {
        // the weights, while the producers' first copies are under way
        for (int c = 0; c < chunks; ++c) stage_weights<CO>(wres + c * 27 * CO * 32, w, ci, c, tid, kPipeThreads - kProducers);
        weights_staged();
    }

    if (warp >= 5) {
        // ---- producers: item = (voxel, 8-channel half); a thread's voxels lie 128 apart
        const int p = tid - 160;
        static_assert(kProducers == 256, "a thread's next voxel: 128 on");
        const int64_t next = (int64_t)(12 * W + 8) * ci, next_x = (int64_t)(W - 10) * ci,
                      next_y = (int64_t)(H - 18) * W * ci;
        int g = 0;          // chunk count over all blocks
        int pend = -1;      // the stage written but not yet announced
        auto announce = [&](int newer, int s) {
            if (newer) asm volatile("cp.async.wait_group 1;" ::: "memory");
            else asm volatile("cp.async.wait_group 0;" ::: "memory");
            asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
            __syncwarp();
            if (lane == 0) mbar_arrive(saddr(full + s));
        };
        for (int tile = blockIdx.x; tile < ntiles && ok; tile += gridDim.x) {
            const int bx = tile % nbx, by = (tile / nbx) % nby, bz = tile / (nbx * nby);
            for (int c = 0; c < chunks && ok; ++c, ++g) {
                const int s = g % NS;
                if (g >= NS && !__all_sync(0xffffffffu, mbar_try(saddr(empty + s), (uint32_t)((g / NS - 1) & 1)))) {
                    // the stage is not free yet: announce the one before first
                    if (pend >= 0) announce(0, pend);
                    pend = -1;
                    ok = mbar_wait(saddr(empty + s), (uint32_t)((g / NS - 1) & 1));
                    ok = __all_sync(0xffffffffu, ok);
                    if (!ok) break;
                }
                const uint32_t dst = stages + s * STAGE + (p & 1) * kPipeHalf;
                int v = p >> 1, vx = v % 10, gy = by * TY - 1 + v / 10, gz = bz * kPipeZ - 1;  // the first plane
                int gx = bx * TX - 1 + vx;
                const int yend = by * TY + 17;
                int64_t at = (((int64_t)gz * H + gy) * W + gx) * ci + c * 16 + (p & 1) * 8;
                while (v < kPipeVox) {
                    const bool in = (unsigned)gx < (unsigned)W && (unsigned)gy < (unsigned)H && (unsigned)gz < (unsigned)D;
                    cp_async16(dst + v * 16, x + (in ? at : 0), in);
                    // 128 voxels on: 12 rows and 8, wrapped into 10 x 18
                    v += kProducers / 2;
                    vx += 8; gx += 8; gy += 12; at += next;
                    if (vx >= 10) { vx -= 10; gx -= 10; ++gy; at += next_x; }
                    if (gy >= yend) { gy -= 18; ++gz; at += next_y; }
                }
                asm volatile("cp.async.commit_group;" ::: "memory");
                if (pend >= 0) announce(1, pend);
                pend = s;
            }
        }
        if (pend >= 0) announce(0, pend);
    } else if (warp == 4) {
        // ---- MMAs.  The whole warp runs the loop and one elected lane
        // issues, so that descriptors are warp-uniform values (uniform
        // registers, as the instruction takes them).
        // Per (ty, tx): one MMA per staged plane zz, into output planes lo ..
        // hi - 1 (N = (hi - lo) co) with the taps tz = zz - lo .. zz - hi + 1
        // (weight_block); 54 MMAs, each reading its A operand once.  The
        // first (ty, tx) of the first chunk starts with planes 2 and 5, whose
        // output ranges (0..2 and 3) cover every accumulator once: they
        // initialise it.
        static_assert(kPipeZ == 4, "merged z taps: 4 output planes, 6 staged");
        constexpr uint32_t ID[4] = {0, idesc_bf16(128, CO), idesc_bf16(128, 2 * CO), idesc_bf16(128, 3 * CO)};
        const bool leader = elect_one();
        const uint32_t tm = __shfl_sync(0xffffffffu, tmem, 0), st0 = __shfl_sync(0xffffffffu, stages, 0),
                       w0 = __shfl_sync(0xffffffffu, wres, 0);
        int g = 0, it = 0, s = 0, ph = 0;  // chunk and block counts; stage of chunk g and its phase
        for (int tile = blockIdx.x; tile < ntiles && ok; tile += gridDim.x, ++it) {
            const int b = it & 1;
            if (it >= 2) ok = __all_sync(0xffffffffu, mbar_wait(saddr(tempty + b), (uint32_t)((it / 2 - 1) & 1)));
            const uint32_t acc = tm + b * ACC;
            for (int c = 0; c < chunks && ok; ++c, ++g) {
                ok = __all_sync(0xffffffffu, mbar_wait(saddr(full + s), (uint32_t)ph));
                if (!ok) break;
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                const uint32_t ta = st0 + s * STAGE, wa = w0 + c * 27 * CO * 32;
                const uint64_t ad0 = smem_desc(ta, kPipeHalf, 160), bd0 = smem_desc(wa, 128, 256);
                if (leader) {
#pragma unroll
                    for (int u = 0; u < 9; ++u) {
                        const int ty = u / 3, tx = u % 3;
#pragma unroll
                        for (int j = 0; j < 6; ++j) {
                            constexpr int kOrder[6] = {2, 5, 0, 1, 3, 4};
                            const int zz = kOrder[j];
                            const int lo = zz > 2 ? zz - 2 : 0, hi = zz + 1 < kPipeZ ? zz + 1 : kPipeZ;
                            const int b0 = 2 - (zz - lo);
                            // addresses below 256 KB: the offsets never carry out of the descriptor's address field
                            const uint64_t ad = ad0 + (uint64_t)((zz * 18 + ty) * 10 + tx);
                            const uint64_t bd = bd0 + (uint64_t)((u * 3 + b0) * (CO * 2));
                            if (u > 0 || j >= 2) mma_bf16(acc + (uint32_t)(lo * CO), ad, bd, ID[hi - lo], 1u);
                            else mma_bf16(acc + (uint32_t)(lo * CO), ad, bd, ID[hi - lo], c > 0 ? 1u : 0u);
                        }
                    }
                    tc_commit(saddr(empty + s));
                    if (c == chunks - 1) tc_commit(saddr(tfull + b));
                }
                __syncwarp();
                if (++s == NS) { s = 0; ph ^= 1; }
            }
        }
        // the MMAs issued are done before the shared and tensor memory go
        if (g > 0) mbar_wait(saddr(empty + (g - 1) % NS), (uint32_t)(((g - 1) / NS) & 1));
        __syncwarp();
    } else {
        // ---- epilogue: warp w reads lanes 32 w .. 32 w + 31 = rows y = 4 w + lane / 8, x = lane % 8
        const int m = 32 * warp + lane;
        int it = 0;
        for (int tile = blockIdx.x; tile < ntiles && ok; tile += gridDim.x, ++it) {
            const int bx = tile % nbx, by = (tile / nbx) % nby, bz = tile / (nbx * nby), b = it & 1;
            ok = mbar_wait(saddr(tfull + b), (uint32_t)((it / 2) & 1));
            ok = __all_sync(0xffffffffu, ok);
            if (!ok) break;
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            const int gx = bx * TX + (m & 7), gy = by * TY + (m >> 3);
            const bool in = gx < W && gy < H;
            // 64 accumulator columns a pass, their loads in flight together;
            // the set is handed back once the last pass has been read
#pragma unroll
            for (int pass = 0; pass < (int)ACC / 64; ++pass) {
                uint32_t r[4][16];
#pragma unroll
                for (int k = 0; k < 4; ++k)
                    tc_ld16_issue(tmem + ((uint32_t)(32 * warp) << 16) + b * ACC + (uint32_t)(pass * 64 + k * 16), r[k]);
                tc_ld_wait(r);
                if (pass == (int)ACC / 64 - 1) {
                    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
                    __syncwarp();
                    if (lane == 0) mbar_arrive(saddr(tempty + b));
                }
#pragma unroll
                for (int k = 0; k < 4; ++k) {
                    const int col = pass * 64 + k * 16, z = col / CO, c16 = col % CO / 16;
                    const int gz = bz * kPipeZ + z;
                    if (in && gz < D) {
                        float v[16];
#pragma unroll
                        for (int e = 0; e < 16; ++e) v[e] = __uint_as_float(r[k][e]);
                        store16(v, bias ? bias + c16 * 16 : nullptr, relu, y, y32,
                                (((int64_t)gz * H + gy) * W + gx) * co + o0 + c16 * 16);
                    }
                }
                __syncwarp();
            }
        }
    }
    if (!ok && lane == 0) atomicOr(&g_conv_tc_flags, 1u);
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    if (warp == 0)
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(NCOL) : "memory");
}

// ---------------------------------------------------------------------------
// Input gradient at stride 2, any grid (conv3_dx2_applies: planes of more than 8
// output voxels): dx[i] = sum over taps t of
// dY[(i + 1 - t) / 2] W[t] where i + 1 - t is even (per axis).  With i =
// 2 j + p, an even i (p = 0) has one tap, t = 1 at dY[j]; an odd one two,
// t = 2 at dY[j] and t = 0 at dY[j + 1].  So the 8 parity classes of an 8 x
// 16 block of j share one staged block of dY (9 x 17 x 2 voxels, all co
// channels), and each of its 8 offsets in {0, 1}^3 is one view (as the taps
// above) that feeds the classes with p = 1 wherever the offset is 1: 8, 4, 2
// or 1 of them, 27 (offset, class) blocks of CI columns.  The classes'
// accumulators lie side by side in tensor memory (class 4 pz + 2 py + px), so
// neighbouring classes take one MMA: 14 MMAs per 16 channels of dY, N = CI to
// 8 CI.  Offsets run from (1, 1, 1) down, all channels of one before the next:
// a class's taps ascend, as in the mma.sync kernel, and the sums are its sums
// bit for bit.  Roles and barriers as in k_conv3_pipe; a stage holds all co
// channels of a block.
// (The fallback read dY once per tap, 7/8 of them for nothing: 2293 us for
// 32 -> 16 channels onto 256 x 128 x 128, 57 us here; 64 -> 32 onto 128 x 64 x
// 64 489 -> 38 us; bound by the MMAs, as k_conv3_pipe.)
constexpr int kD2Vox = 2 * 17 * 9;
constexpr int kD2Half = kD2Vox * 16 + 64;

// First block (of the 27) of offset 4 z + 2 y + x.
__host__ __device__ constexpr int d2_first(int o) {
    return o < 4 ? (o < 2 ? 8 * o : 4 * o + 4) : (o < 6 ? 4 * o + 2 : 2 * o + 12);
}
static_assert(d2_first(0) == 0 && d2_first(1) == 8 && d2_first(2) == 12 && d2_first(3) == 16 && d2_first(4) == 18 &&
                  d2_first(5) == 22 && d2_first(6) == 24 && d2_first(7) == 26,
              "8, 4, 4, 2, 4, 2, 2, 1 classes");
// Tap of class bit p at offset o along one axis.
__host__ __device__ constexpr int d2_tap(int p, int o) { return p == 0 ? 1 : (o == 0 ? 2 : 0); }

template <int CI>
__global__ void __launch_bounds__(kPipeThreads, 1) k_conv3_dx2(const bf16* __restrict__ dy, const bf16* __restrict__ wt,
                                                             bf16* __restrict__ dx, int D, int H, int W, int ci,
                                                             int Do, int Ho, int Wo, int co, int ntiles, int NS) {
    constexpr uint32_t ACC = 8 * CI, NCOL = 2 * ACC;
    extern __shared__ __align__(128) unsigned char smem[];
    const int groups = co / 8, chunks = co / 16, stage_bytes = groups * kD2Half;
    const int c0 = blockIdx.y * CI;  // first input channel
    uint64_t* full = reinterpret_cast<uint64_t*>(smem);
    uint64_t* empty = full + 8;
    uint64_t* tfull = empty + 8;
    uint64_t* tempty = tfull + 2;
    uint32_t* tslot = reinterpret_cast<uint32_t*>(tempty + 2);
    const uint32_t wres = saddr(smem) + kPipeBars, stages = wres + 27 * CI * 2 * co;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int nbx = (Wo + TX - 1) / TX, nby = (Ho + TY - 1) / TY;

    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(saddr(tslot)),
                     "r"(NCOL)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    if (tid == 0) {
        for (int s = 0; s < NS; ++s) {
            mbar_init(saddr(full + s), kProducers / 32);
            mbar_init(saddr(empty + s), 1);
        }
        for (int b = 0; b < 2; ++b) {
            mbar_init(saddr(tfull + b), 1);
            mbar_init(saddr(tempty + b), 4);
        }
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem = *tslot;
    bool ok = true;
    if (warp < 5) {
        // wt [ci][27][co]: rows c of the block of (offset, class), 16-byte pieces of 8 co
        for (int i = tid; i < 27 * CI * groups; i += kPipeThreads - kProducers) {
            const int k8 = i % groups, n = (i / groups) % CI, blk = i / (groups * CI);
            int o = 0;
            while (o < 7 && blk >= d2_first(o + 1)) ++o;
            int cls = 0;  // the (blk - first)-th class with p = 1 where the offset is 1
            for (int m = blk - d2_first(o); (cls & o) != o || m-- > 0; ++cls) {}
            const int t = (d2_tap(cls >> 2, o >> 2) * 3 + d2_tap((cls >> 1) & 1, (o >> 1) & 1)) * 3 + d2_tap(cls & 1, o & 1);
            cp_async16(wres + ((k8 >> 1) * 27 + blk) * (CI * 32) + (n >> 3) * 256 + (k8 & 1) * 128 + (n & 7) * 16,
                       wt + ((int64_t)(c0 + n) * 27 + t) * co + k8 * 8, true);
        }
        weights_staged();
    }

    if (warp >= 5) {
        // ---- producers: item = (voxel, 8-channel group), groups fastest
        const int p = tid - 160, gsh = 31 - __clz(groups);
        int it = 0, pend = -1;
        auto announce = [&](int newer, int s) {
            if (newer) asm volatile("cp.async.wait_group 1;" ::: "memory");
            else asm volatile("cp.async.wait_group 0;" ::: "memory");
            asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
            __syncwarp();
            if (lane == 0) mbar_arrive(saddr(full + s));
        };
        for (int tile = blockIdx.x; tile < ntiles && ok; tile += gridDim.x, ++it) {
            const int bx = tile % nbx, by = (tile / nbx) % nby, bz = tile / (nbx * nby);
            const int s = it % NS;
            if (it >= NS && !__all_sync(0xffffffffu, mbar_try(saddr(empty + s), (uint32_t)((it / NS - 1) & 1)))) {
                if (pend >= 0) announce(0, pend);
                pend = -1;
                ok = mbar_wait(saddr(empty + s), (uint32_t)((it / NS - 1) & 1));
                ok = __all_sync(0xffffffffu, ok);
                if (!ok) break;
            }
            const uint32_t dst = stages + s * stage_bytes;
            for (int i = p; i < kD2Vox << gsh; i += kProducers) {
                const int v = i >> gsh, k8 = i & (groups - 1);
                const int vx = v % 9, vy = (v / 9) % 17, vz = v / 153;
                const int gx = bx * TX + vx, gy = by * TY + vy, gz = bz + vz;
                const bool in = gx < Wo && gy < Ho && gz < Do;
                cp_async16(dst + k8 * kD2Half + v * 16,
                           dy + (in ? (((int64_t)gz * Ho + gy) * Wo + gx) * co + k8 * 8 : 0), in);
            }
            asm volatile("cp.async.commit_group;" ::: "memory");
            if (pend >= 0) announce(1, pend);
            pend = s;
        }
        if (pend >= 0) announce(0, pend);
    } else if (warp == 4) {
        // ---- MMAs (whole warp, one elected lane issues)
        const bool leader = elect_one();
        const uint32_t tm = __shfl_sync(0xffffffffu, tmem, 0), st0 = __shfl_sync(0xffffffffu, stages, 0),
                       w0 = __shfl_sync(0xffffffffu, wres, 0);
        int it = 0;
        for (int tile = blockIdx.x; tile < ntiles && ok; tile += gridDim.x, ++it) {
            const int b = it & 1, s = it % NS;
            if (it >= 2) ok = __all_sync(0xffffffffu, mbar_wait(saddr(tempty + b), (uint32_t)((it / 2 - 1) & 1)));
            if (ok) ok = __all_sync(0xffffffffu, mbar_wait(saddr(full + s), (uint32_t)((it / NS) & 1)));
            if (!ok) break;
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            const uint32_t acc = tm + b * ACC;
            if (leader) {
                // A class's first offset is its own number: it alone starts
                // from zero there.
#pragma unroll
                for (int k = 0; k < 8; ++k) {
                    const int need = 7 - k, oz = need >> 2, oy = need >> 1 & 1, ox = need & 1;
                    for (int c = 0; c < chunks; ++c) {
                        const uint64_t ad = smem_desc(st0 + s * stage_bytes + 2 * c * kD2Half, kD2Half, 144) +
                                            (uint64_t)((oz * 17 + oy) * 9 + ox);
                        const uint64_t bd0 = smem_desc(w0 + c * 27 * CI * 32, 128, 256);
                        // runs of neighbouring classes
                        int blk = d2_first(need);
#pragma unroll
                        for (int cls = 0; cls < 8; ++cls) {
                            if ((cls & need) != need || (cls > 0 && ((cls - 1) & need) == need)) continue;
                            int run = 1;
#pragma unroll
                            for (int e = 1; e < 8; ++e)
                                if (run == e && cls + e < 8 && ((cls + e) & need) == need) run = e + 1;
                            const uint64_t bd = bd0 + (uint64_t)(blk * (CI * 2));
                            if (cls == need && c == 0) {
                                mma_bf16(acc + (uint32_t)(cls * CI), ad, bd, idesc_bf16(128, CI), 0u);
                                if (run > 1)
                                    mma_bf16(acc + (uint32_t)((cls + 1) * CI), ad, bd + (uint64_t)(CI * 2),
                                             idesc_bf16(128, (run - 1) * CI), 1u);
                            } else {
                                mma_bf16(acc + (uint32_t)(cls * CI), ad, bd, idesc_bf16(128, run * CI), 1u);
                            }
                            blk += run;
                        }
                    }
                }
                tc_commit(saddr(empty + s));
                tc_commit(saddr(tfull + b));
            }
            __syncwarp();
        }
        // the MMAs issued are done before the shared and tensor memory go
        if (it > 0) mbar_wait(saddr(empty + (it - 1) % NS), (uint32_t)(((it - 1) / NS) & 1));
        __syncwarp();
    } else {
        // ---- epilogue: lane = coarse voxel (rows y = 4 w + lane / 8, x = lane % 8), columns = (class, channel)
        const int m = 32 * warp + lane;
        int it = 0;
        for (int tile = blockIdx.x; tile < ntiles && ok; tile += gridDim.x, ++it) {
            const int bx = tile % nbx, by = (tile / nbx) % nby, bz = tile / (nbx * nby), b = it & 1;
            ok = mbar_wait(saddr(tfull + b), (uint32_t)((it / 2) & 1));
            ok = __all_sync(0xffffffffu, ok);
            if (!ok) break;
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            const int gx = 2 * (bx * TX + (m & 7)), gy = 2 * (by * TY + (m >> 3)), gz = 2 * bz;
#pragma unroll
            for (int pass = 0; pass < (int)ACC / 64; ++pass) {
                uint32_t r[4][16];
#pragma unroll
                for (int k = 0; k < 4; ++k)
                    tc_ld16_issue(tmem + ((uint32_t)(32 * warp) << 16) + b * ACC + (uint32_t)(pass * 64 + k * 16), r[k]);
                tc_ld_wait(r);
                if (pass == (int)ACC / 64 - 1) {
                    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
                    __syncwarp();
                    if (lane == 0) mbar_arrive(saddr(tempty + b));
                }
#pragma unroll
                for (int k = 0; k < 4; ++k) {
                    const int col = pass * 64 + k * 16, cls = col / CI, c16 = col % CI / 16;
                    const int x = gx + (cls & 1), y = gy + ((cls >> 1) & 1), z = gz + (cls >> 2);
                    if (x < W && y < H && z < D) {
                        float v[16];
#pragma unroll
                        for (int e = 0; e < 16; ++e) v[e] = __uint_as_float(r[k][e]);
                        store16(v, nullptr, 0, dx, nullptr, (((int64_t)z * H + y) * W + x) * ci + c0 + c16 * 16);
                    }
                }
                __syncwarp();
            }
        }
    }
    if (!ok && lane == 0) atomicOr(&g_conv_tc_flags, 1u);
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    if (warp == 0)
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(NCOL) : "memory");
}

// ---------------------------------------------------------------------------
// Weight gradient dW[o][t][c] += sum over output voxels m of
// dY[m][o] X[src(m, t)][c] (kernel size 3, stride 1 or 2, or kernel size 1).
// A contraction over the voxels with few rows and columns (co x ci of 16 to
// 64) for each of 27 taps.  On tcgen05 it needs either an im2col operand --
// 27 copies of X through shared memory, which is what bounded the kernel
// before this one (864 16-byte cp.async per 16 voxels: 1.46 ms on the
// 16-channel layer at 256 x 128 x 128) -- or shifted views of one staged
// tile as 128 matrix rows a constant stride apart, of which 30% are
// products that count, in more accumulators than tensor memory has columns.
// Warp-level MMAs take any 8 voxel rows as an operand, so all taps read one
// staged tile: per 16 voxels one ldmatrix of dY and one per tap of X, the
// sums in registers.
//
// A CTA walks output tiles of TZ x TY x TX voxels, NS of them in flight:
// per tile a tensor copy of dY (COB channels) and of the input voxels its
// taps read (16 channels), zero-filled outside the grids (the padding),
// swizzled so that the 8 rows of an ldmatrix phase lie in different banks at
// stride 1 for any tap.  Warps are NG tap groups (TPW taps each) x KG groups
// of voxel rows; D = dY^T X with m16n8k16 (M = 16 output channels, N = 8 input
// channels, K = 16 voxels of an x-run).  Bound by the MMAs and shared memory
// together: an ldmatrix.x4 (4 cycles) per four MMAs of 2 cycles at 32 channels.
// At 16, a view of an input row serves one output row's MMAs per tap, two per
// ldmatrix.x4; so a warp with all 9 taps of a tz goes down the rows and uses a
// view for the three output rows that it meets (ROLL): 4 ldmatrix.x4 for 18
// MMAs, 16 -> 16 channels 162 -> 142 us.  256 x 128 x 128: 16 -> 16 142 us (1122
// with the tcgen05 im2col), 32 -> 16 275 us (2493), stride-2 16 -> 32 63 us
// (153), 1x1x1 61 us (411); 128 x 64 x 64, 32 -> 32: 92 us (327).
// A tile at the grid's end leaves out the output voxels outside it: their dY
// is zero, but X beside them need not be finite, and 0 x Inf would reach taps
// that no Inf belongs to.
// grid.y walks the (co / COB) x (ci / 16) channel blocks.  Every
// FLUSH tiles the KG groups add their sums in turn to the CTA's in shared
// memory: an MMA drops bits of its accumulator, so that chains of 216 MMAs
// left dW 2.4e-6 from the kernel before, further off FP64 than it (7e-7);
// with chains of 64 it is not.
// Each CTA adds its block to dW with FP32 atomics.
template <int KS_, int S_, int COB_>
struct WGeo {
    static constexpr int KS = KS_, S = S_, COB = COB_;
    static constexpr int TAPS = KS * KS * KS;
    // tile and warps: the input tile (with its halo) of NS stages fills the
    // shared memory; 9 taps a warp at COB 16 (72 sums a thread), 3 at COB 32
    static constexpr int TZ = S == 2 ? 2 : 4, TY = S == 2 ? 4 : 8, TX = (S == 1 && COB == 16) ? 32 : 16;
    static constexpr int XD = S * (TZ - 1) + KS, XH = S * (TY - 1) + KS, XW = S * (TX - 1) + KS;
    static constexpr int TPW = KS == 1 ? 1 : (COB == 16 ? 9 : 3);
    static constexpr int NG = TAPS / TPW;
    static constexpr bool ROLL = KS == 3 && S == 1 && TPW == 9;  // rows in turn, views kept for three ty
    static constexpr int KG = KS == 1 ? 12 : (COB == 16 ? 4 : 2);
    static constexpr int THREADS = 32 * NG * KG;
    static constexpr int KSTEPS = TZ * TY * TX / 16;
    static constexpr int XBYTES = XD * XH * XW * 32, YBYTES = TZ * TY * TX * COB * 2;
    static constexpr int XPAD = (XBYTES + 1023) / 1024 * 1024, STAGE = XPAD + (YBYTES + 1023) / 1024 * 1024;
    // tiles between flushes of a thread's sums: chains of at most 64 MMAs
    static constexpr int FLUSH = 64 * KG / KSTEPS > 1 ? 64 * KG / KSTEPS : 1;
    // sums [o][tap][16], rows 8 floats apart modulo the 32 banks
    static constexpr int ROW = TAPS * 16 % 32 == 16 ? TAPS * 16 + 8 : TAPS * 16 + 24;
    static constexpr int SUMS = COB * ROW * 4;
    static constexpr int NS = 3 * STAGE + SUMS <= 220 * 1024 ? 3 : 2;
    // voxels of zeros, read in place of what no sum may meet: all views of one voxel (ROLL: one row, by itself)
    static constexpr int ZROWS = ROLL ? 1 : (TPW == 9 ? 2 * XW + 3 : 3);
    static constexpr int SMEM = NS * STAGE + SUMS + ZROWS * 32 + 1024;  // stages from a 1024-byte boundary
    static_assert(SMEM <= 227 * 1024, "shared memory");
};

__device__ __forceinline__ void ldmatrix4_trans(uint32_t (&r)[4], uint32_t addr) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
                 : "r"(addr)
                 : "memory");
}

__device__ __forceinline__ void mma_m16n8k16(float (&c)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
    asm volatile(
        "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
        : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
        : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}

// Byte offset of 16-byte chunk k of voxel v in a staged tile of 16 / 32
// channels: the tensor copy's 32- / 64-byte swizzle.
__device__ __forceinline__ uint32_t chunk16(uint32_t v, uint32_t k) { return (v << 5) | ((k << 4) ^ ((v & 4u) << 2)); }
__device__ __forceinline__ uint32_t chunk32(uint32_t v, uint32_t k) { return (v << 6) | ((k << 4) ^ ((v & 6u) << 3)); }

// RAGGED: some tiles reach past the grid (the others take the plain sums; a kernel
// of its own, whose test alone costs whole grids 1.5%).  Without a halo, X is zero
// wherever dY is: never RAGGED.
template <class G, bool RAGGED>
__global__ void __launch_bounds__(G::THREADS, 1) k_conv_wgrad_tiles(const __grid_constant__ CUtensorMap xmap,
                                                                   const __grid_constant__ CUtensorMap ymap,
                                                                   float* __restrict__ dw, int Do, int Ho, int Wo,
                                                                   int ci, int ntiles, uint32_t copied) {
    constexpr int S = G::S, KS = G::KS, COB = G::COB, NS = G::NS, MT = COB / 16;
    extern __shared__ unsigned char smem_raw[];
    __shared__ __align__(8) uint64_t full[NS];
    __shared__ int inside[NS];  // of the tile in a stage: its output voxels inside the grid per axis, x | y << 8 | z << 16
    unsigned char* smem = smem_raw + ((1024u - (saddr(smem_raw) & 1023u)) & 1023u);
    const uint32_t base = saddr(smem);
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int tg = warp % G::NG, kg = warp / G::NG;
    const int cb = ci / 16, c0 = (blockIdx.y % cb) * 16, o0 = (blockIdx.y / cb) * COB;
    const int nbx = (Wo + G::TX - 1) / G::TX, nby = (Ho + G::TY - 1) / G::TY;

    auto issue = [&](int tile, int s) {
        const int bx = tile % nbx, by = (tile / nbx) % nby, bz = tile / (nbx * nby);
        const uint32_t bar = saddr(full + s), dst = base + s * G::STAGE;
        if constexpr (RAGGED)
            inside[s] = min(Wo - bx * G::TX, G::TX) | min(Ho - by * G::TY, G::TY) << 8 | min(Do - bz * G::TZ, G::TZ) << 16;
        mbar_expect_tx(bar, copied);
        tma_load4(dst, &xmap, c0, S * bx * G::TX - KS / 2, S * by * G::TY - KS / 2, S * bz * G::TZ - KS / 2, bar);
        tma_load4(dst + G::XPAD, &ymap, o0, bx * G::TX, by * G::TY, bz * G::TZ, bar);
    };

    if (tid == 0) {
        for (int s = 0; s < NS; ++s) mbar_init(saddr(full + s), 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    const uint32_t zero = base + NS * G::STAGE + G::SUMS;
    if constexpr (RAGGED)
        for (int e = tid; e < G::ZROWS * 2; e += G::THREADS)
            reinterpret_cast<uint4*>(smem + NS * G::STAGE + G::SUMS)[e] = make_uint4(0u, 0u, 0u, 0u);
    __syncthreads();
    const int first = blockIdx.x, step = gridDim.x;
    int issued = 0;  // thread 0: tiles issued
    if (tid == 0)
        for (; issued < NS - 1 && first + issued * step < ntiles; ++issued) issue(first + issued * step, issued);

    float acc[G::TPW][MT][2][4];
#pragma unroll
    for (int t = 0; t < G::TPW; ++t)
#pragma unroll
        for (int m = 0; m < MT; ++m)
#pragma unroll
            for (int k = 0; k < 4; ++k) acc[t][m][0][k] = acc[t][m][1][k] = 0.f;

    // this lane's voxel of the K = 16 and its 16-byte chunk in an ldmatrix.x4:
    // (voxels 0-7, 0-7, 8-15, 8-15) x (channels 0-7, 8-15, 0-7, 8-15)
    const uint32_t lv = ((lane >> 4) << 3) | (lane & 7), lc = (lane >> 3) & 1;
    const int tz = KS == 1 ? 0 : (G::TPW == 9 ? tg : tg / 3), ty0 = G::TPW == 3 ? tg % 3 : 0;
    const uint32_t tapv = (uint32_t)((tz * G::XH + ty0) * G::XW);
    float* sum = reinterpret_cast<float*>(smem + NS * G::STAGE);
    const int g = lane >> 2, q = lane & 3;
    bool summed = false;
    auto flush = [&]() {
        for (int r = 0; r < G::KG; ++r) {
            if (kg == r) {
#pragma unroll
                for (int t = 0; t < G::TPW; ++t)
#pragma unroll
                    for (int m = 0; m < MT; ++m)
#pragma unroll
                        for (int n = 0; n < 2; ++n)
#pragma unroll
                            for (int h = 0; h < 2; ++h) {
                                float2* p = reinterpret_cast<float2*>(sum + (16 * m + g + 8 * h) * G::ROW +
                                                                      (tg * G::TPW + t) * 16 + 8 * n + 2 * q);
                                float2 v = make_float2(acc[t][m][n][2 * h], acc[t][m][n][2 * h + 1]);
                                if (summed || r > 0) {
                                    const float2 w = *p;
                                    v.x += w.x;
                                    v.y += w.y;
                                }
                                *p = v;
                                acc[t][m][n][2 * h] = acc[t][m][n][2 * h + 1] = 0.f;
                            }
            }
            __syncthreads();
        }
        summed = true;
    };
    bool ok = true;
    int it = 0;
    for (int tile = first; tile < ntiles; tile += step, ++it) {
        const int s = it % NS;
        if (tid == 0 && first + issued * step < ntiles) {
            // the stage's previous tile was read before the barrier that ended its pass
            asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
            issue(first + issued * step, issued % NS);
            ++issued;
        }
        ok = mbar_wait(saddr(full + s), (uint32_t)((it / NS) & 1));
        ok = __syncthreads_and(ok);
        if (!ok) break;
        const uint32_t xs = base + s * G::STAGE, ys = xs + G::XPAD;
        constexpr int kWhole = G::TX | G::TY << 8 | G::TZ << 16;
        const int part = RAGGED ? inside[s] : kWhole, ex = part & 0xff, ey = (part >> 8) & 0xff, ez = part >> 16;
        auto sums = [&](auto whole) {
            constexpr bool WHOLE = decltype(whole)::value;
            constexpr int RUNS = G::TX / 16;
            if constexpr (G::ROLL) {
                // x-runs of 16 voxels down the rows: an input row's three views
                // (tx) meet the output rows of all three ty while they are at hand
                for (int run = kg; run < G::TZ * RUNS; run += G::KG) {
                    const int z = run / RUNS, x = run % RUNS * 16;
                    if (!WHOLE && (z >= ez || x >= ex)) continue;
                    const bool in = WHOLE || x + (int)lv < ex;
                    const uint32_t dv = (uint32_t)(z * G::TY * G::TX + x) + lv,
                                   xv = (uint32_t)(z * G::XH * G::XW + x) + lv + tapv;
                    uint32_t a[3][4];
#pragma unroll
                    for (int r = 0; r < G::XH; ++r) {
                        if (r < G::TY) ldmatrix4_trans(a[r % 3], ys + chunk16(dv + (uint32_t)(r * G::TX), lc));
#pragma unroll
                        for (int tx = 0; tx < 3; ++tx) {
                            uint32_t b[4];
                            const uint32_t at = xs + chunk16(xv + (uint32_t)(r * G::XW + tx), lc);
                            ldmatrix4_trans(b, in ? at : zero);
#pragma unroll
                            for (int ty = 0; ty < 3; ++ty) {
                                const int y = r - ty;
                                if (y < 0 || y >= G::TY || (!WHOLE && y >= ey)) continue;
                                mma_m16n8k16(acc[ty * 3 + tx][0][0], a[y % 3], b[0], b[2]);
                                mma_m16n8k16(acc[ty * 3 + tx][0][1], a[y % 3], b[1], b[3]);
                            }
                        }
                    }
                }
            } else {
                for (int ks = kg; ks < G::KSTEPS; ks += G::KG) {
                    const int row = ks / RUNS, x = (ks % RUNS) * 16, z = row / G::TY, y = row % G::TY;
                    if (!WHOLE && (z >= ez || y >= ey || x >= ex)) continue;
                    const bool in = WHOLE || x + (int)lv < ex;
                    const uint32_t dv = (uint32_t)(row * G::TX + x) + lv;
                    uint32_t a[MT][4];
#pragma unroll
                    for (int m = 0; m < MT; ++m)
                        ldmatrix4_trans(a[m], ys + (COB == 16 ? chunk16(dv, lc) : chunk32(dv, 2 * m + lc)));
                    const uint32_t xv = in ? (uint32_t)((S * z * G::XH + S * y) * G::XW + S * x) + S * lv + tapv : (zero - xs) >> 5;
#pragma unroll
                    for (int t = 0; t < G::TPW; ++t) {
                        uint32_t b[4];
                        ldmatrix4_trans(b, xs + chunk16(xv + (uint32_t)((t / 3) * G::XW + t % 3), lc));
#pragma unroll
                        for (int m = 0; m < MT; ++m) {
                            mma_m16n8k16(acc[t][m][0], a[m], b[0], b[2]);
                            mma_m16n8k16(acc[t][m][1], a[m], b[1], b[3]);
                        }
                    }
                }
            }
        };
        if (!RAGGED || part == kWhole) sums(std::integral_constant<bool, true>());
        else if constexpr (RAGGED) sums(std::integral_constant<bool, false>());
        __syncthreads();
        if ((it + 1) % G::FLUSH == 0) flush();
    }
    if (!ok) {
        // a copy did not land in time: record it and wait (bounded) for those in flight
        if (tid == 0) {
            atomicOr(&g_conv_tc_flags, 2u);
            for (int k = it; k < issued; ++k) mbar_wait(saddr(full + k % NS), (uint32_t)((k / NS) & 1));
        }
        __syncthreads();
        return;
    }
    flush();
    for (int e = tid; e < G::TAPS * COB * 16; e += G::THREADS) {
        const int c = e & 15, t = (e >> 4) % G::TAPS, o = (e >> 4) / G::TAPS;
        atomicAdd(dw + ((int64_t)(o0 + o) * G::TAPS + t) * ci + c0 + c, sum[o * G::ROW + t * 16 + c]);
    }
}

// Wt [ci][t][co] = W [co][26 - t][ci]: the input gradient of a stride-1
// convolution is the forward convolution of dy with these weights.
__global__ void k_flip_transpose(const bf16* __restrict__ w, bf16* __restrict__ wt, int co, int ci) {
    const int64_t e = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (e >= (int64_t)co * 27 * ci) return;
    const int c = (int)(e % ci), t = (int)((e / ci) % 27), o = (int)(e / ((int64_t)ci * 27));
    wt[((int64_t)c * 27 + (26 - t)) * co + o] = w[e];
}

// cuTensorMapEncodeTiled through the runtime's driver entry point (no link
// against the driver library), looked up once.
using EncodeTiled = CUresult (*)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                                 const cuuint64_t*, const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave,
                                 CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

EncodeTiled encode_tiled() {
    static std::atomic<EncodeTiled> fn{nullptr};
    EncodeTiled f = fn.load(std::memory_order_acquire);
    if (!f) {
        void* p = nullptr;
        cudaDriverEntryPointQueryResult q{};
        if (cudaGetDriverEntryPointByVersion("cuTensorMapEncodeTiled", &p, 12000, cudaEnableDefault, &q) !=
                cudaSuccess ||
            q != cudaDriverEntryPointSuccess)
            return nullptr;
        f = reinterpret_cast<EncodeTiled>(p);
        fn.store(f, std::memory_order_release);
    }
    return f;
}

// The tensor map of x [Di][Hi][Wi][ci] BF16 at stride 2: box 8 channels x
// 2 XH voxels along x with element stride 2 (one parity) x YB x ZB, zero fill
// outside the tensor.
cudaError_t input_map_s2(CUtensorMap* map, const bf16* x, int Di, int Hi, int Wi, int ci) {
    using G = Geo2;
    EncodeTiled f = encode_tiled();
    if (!f) return cudaErrorNotSupported;
    const cuuint64_t dims[4] = {(cuuint64_t)ci, (cuuint64_t)Wi, (cuuint64_t)Hi, (cuuint64_t)Di};
    const cuuint64_t strides[3] = {(cuuint64_t)ci * 2, (cuuint64_t)Wi * ci * 2, (cuuint64_t)Hi * Wi * ci * 2};
    const cuuint32_t box[4] = {8, (cuuint32_t)(2 * G::XH), (cuuint32_t)G::YB, (cuuint32_t)G::ZB};
    const cuuint32_t estride[4] = {1, 2, 1, 1};
    const CUresult r = f(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 4, const_cast<bf16*>(x), dims, strides, box, estride,
                         CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
                         CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    return r == CUDA_SUCCESS ? cudaSuccess : cudaErrorInvalidValue;
}

// Tensor map of a channels-last BF16 tensor [D][H][W][C] with box
// (bd, bh, bw, bc), bc = 16 or 32 channels, its 32- / 64-byte rows swizzled,
// zero fill outside.
cudaError_t tile_map(CUtensorMap* map, const bf16* x, int D, int H, int W, int C, int bd, int bh, int bw, int bc) {
    EncodeTiled f = encode_tiled();
    if (!f) return cudaErrorNotSupported;
    const cuuint64_t dims[4] = {(cuuint64_t)C, (cuuint64_t)W, (cuuint64_t)H, (cuuint64_t)D};
    const cuuint64_t strides[3] = {(cuuint64_t)C * 2, (cuuint64_t)W * C * 2, (cuuint64_t)H * W * C * 2};
    const cuuint32_t box[4] = {(cuuint32_t)bc, (cuuint32_t)bw, (cuuint32_t)bh, (cuuint32_t)bd};
    const cuuint32_t estride[4] = {1, 1, 1, 1};
    const CUresult r = f(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 4, const_cast<bf16*>(x), dims, strides, box, estride,
                         CU_TENSOR_MAP_INTERLEAVE_NONE, bc == 16 ? CU_TENSOR_MAP_SWIZZLE_32B : CU_TENSOR_MAP_SWIZZLE_64B,
                         CU_TENSOR_MAP_L2_PROMOTION_L2_128B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    return r == CUDA_SUCCESS ? cudaSuccess : cudaErrorInvalidValue;
}

template <class G>
cudaError_t launch_wgrad(const bf16* x, const bf16* dy, float* dw, int Di, int Hi, int Wi, int ci, int co,
                         cudaStream_t st) {
    const int Do = (Di - 1) / G::S + 1, Ho = (Hi - 1) / G::S + 1, Wo = (Wi - 1) / G::S + 1;
    CUtensorMap xm, ym;
    // a grid of fewer planes than a tile's copies no more of them (they are not read)
    const int tz = G::KS == 3 && Do < G::TZ ? Do : G::TZ, xd = G::S * (tz - 1) + G::KS;
    cudaError_t e = tile_map(&xm, x, Di, Hi, Wi, ci, xd, G::XH, G::XW, 16);
    if (e == cudaSuccess) e = tile_map(&ym, dy, Do, Ho, Wo, co, tz, G::TY, G::TX, G::COB);
    bool ragged = false;
    if constexpr (G::KS == 3) ragged = Do % G::TZ || Ho % G::TY || Wo % G::TX;
    auto kern = k_conv_wgrad_tiles<G, false>;
    if constexpr (G::KS == 3)
        if (ragged) kern = k_conv_wgrad_tiles<G, true>;
    if (e == cudaSuccess) e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, G::SMEM);
    if (e != cudaSuccess) return e;
    const int64_t tiles = lbm::ceil_div(Do, G::TZ) * lbm::ceil_div(Ho, G::TY) * lbm::ceil_div(Wo, G::TX);
    const int roles = co / G::COB * (ci / 16);
    // one CTA an SM over all channel blocks, each with about the same number of tiles
    const int64_t want = lbm::sm_count() / roles > 1 ? lbm::sm_count() / roles : 1;
    const int64_t per = lbm::ceil_div(tiles, want);
    kern<<<dim3((unsigned)lbm::ceil_div(tiles, per), (unsigned)roles), G::THREADS, G::SMEM, st>>>(
        xm, ym, dw, Do, Ho, Wo, ci, (int)tiles, (uint32_t)(G::XBYTES / G::XD * xd + G::YBYTES / G::TZ * tz));
    return cudaGetLastError();
}

template <int CO>
cudaError_t launch_s2(const bf16* x, const bf16* w, const float* bias, bf16* y, float* y32, int Di, int Hi, int Wi,
                      int ci, int relu, cudaStream_t st) {
    constexpr int bytes = smem_bytes<CO>();
    // Resident CTAs per SM times their tensor-memory columns must fit the 512
    // columns of an SM (an allocation that cannot be met waits for another
    // CTA's release): shared memory bounds the residency below that here.
    static_assert(bytes <= 227 * 1024 && (227 * 1024 / bytes) * tmem_cols<CO>() <= 512, "shared and tensor memory");
    CUtensorMap map;
    cudaError_t e = input_map_s2(&map, x, Di, Hi, Wi, ci);
    if (e != cudaSuccess) return e;
    e = cudaFuncSetAttribute(k_conv3_s2_tc<CO>, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
    if (e != cudaSuccess) return e;
    const int Do = Di / 2, Ho = Hi / 2, Wo = Wi / 2;
    const int64_t blocks = (int64_t)(Wo / TX) * (Ho / TY) * Do;
    k_conv3_s2_tc<CO><<<(unsigned)blocks, kThreads, bytes, st>>>(map, w, bias, y, y32, Do, Ho, Wo, ci, relu);
    return cudaGetLastError();
}

// Shared memory of a persistent CTA: `fixed` bytes and as many stages as fit
// (2 to 6; the kernels have room for 8 barriers); more than half of an SM's,
// so that a CTA's tensor memory is alone on its SM.
struct PipeShape {
    int stages, bytes;
};
PipeShape pipe_shape(int fixed, int stage) {
    constexpr int kMost = 227 * 1024, kLeast = 116 * 1024;
    int ns = (kMost - fixed) / stage;
    ns = ns < 6 ? ns : 6;
    const int bytes = fixed + ns * stage;
    return {ns, bytes > kLeast ? bytes : kLeast};
}

// Stride 1: one CTA an SM over all blocks and channel parts, every CTA about
// the same number of blocks.
template <int CO>
cudaError_t launch_pipe(const bf16* x, const bf16* w, const float* bias, bf16* y, float* y32, int D, int H, int W,
                        int ci, int co, int relu, cudaStream_t st) {
    const int64_t tiles = lbm::ceil_div(D, kPipeZ) * lbm::ceil_div(H, TY) * lbm::ceil_div(W, TX);
    if (tiles > 0x7fffffffLL) return cudaErrorInvalidConfiguration;
    static_assert(kPipeBars + 27 * 32 * 2 * 64 + 2 * kPipeTile <= 227 * 1024, "32 of 64 -> 64 channels");
    const PipeShape p = pipe_shape(kPipeBars + 27 * CO * 2 * ci, kPipeTile);
    cudaError_t e = cudaFuncSetAttribute(k_conv3_pipe<CO>, cudaFuncAttributeMaxDynamicSharedMemorySize, 227 * 1024);
    if (e != cudaSuccess) return e;
    const int parts = co / CO;
    const int64_t per = lbm::ceil_div(tiles, lbm::sm_count() / parts > 1 ? lbm::sm_count() / parts : 1);
    k_conv3_pipe<CO><<<dim3((unsigned)lbm::ceil_div(tiles, per), (unsigned)parts), kPipeThreads, p.bytes, st>>>(
        x, w, bias, y, y32, D, H, W, ci, co, relu, (int)tiles, p.stages);
    return cudaGetLastError();
}

template <int CI>
cudaError_t launch_dx2(const bf16* dy, const bf16* wt, bf16* dx, int D, int H, int W, int ci, int co, cudaStream_t st) {
    const int Do = (D - 1) / 2 + 1, Ho = (H - 1) / 2 + 1, Wo = (W - 1) / 2 + 1;
    const int64_t tiles = (int64_t)Do * lbm::ceil_div(Ho, TY) * lbm::ceil_div(Wo, TX);
    static_assert(kPipeBars + 27 * 32 * 2 * 64 + 2 * 8 * kD2Half <= 227 * 1024, "64 channels of dY, 32 of dx");
    const PipeShape p = pipe_shape(kPipeBars + 27 * CI * 2 * co, co / 8 * kD2Half);
    cudaError_t e = cudaFuncSetAttribute(k_conv3_dx2<CI>, cudaFuncAttributeMaxDynamicSharedMemorySize, 227 * 1024);
    if (e != cudaSuccess) return e;
    const int parts = ci / CI;
    const int64_t per = lbm::ceil_div(tiles, lbm::sm_count() / parts > 1 ? lbm::sm_count() / parts : 1);
    k_conv3_dx2<CI><<<dim3((unsigned)lbm::ceil_div(tiles, per), (unsigned)parts), kPipeThreads, p.bytes, st>>>(
        dy, wt, dx, D, H, W, ci, Do, Ho, Wo, co, (int)tiles, p.stages);
    return cudaGetLastError();
}

}  // namespace

namespace lbm {

bool conv3_tc_applies(int D, int H, int W, int ci, int co, int stride) {
    const bool ch = (ci == 16 || ci == 32 || ci == 64) && (co == 16 || co == 32 || co == 64);
    if (!ch || D <= 0 || H <= 0 || W <= 0) return false;
    // Lower than a block's 16 rows, as a network's lowest level is: the mma.sync
    // kernel, whose order of summation such levels have always had (a network's
    // gradients move by 4e-4 with the order here; 16 x 8 x 8, 64 -> 64 channels
    // take 12 us there, 9 here).  A line drawn for values: the kernel here takes
    // such grids too.
    if (stride == 1) return H >= TY && ceil_div(D, kPipeZ) * ceil_div(H, TY) * ceil_div(W, TX) <= 0x7fffffffLL;
    if (stride == 2) return D % 2 == 0 && H % (2 * TY) == 0 && W % (2 * TX) == 0;
    return false;
}

cudaError_t conv3_tc(const void* x, int D, int H, int W, int ci, const void* w, const float* bias, int co, int relu,
                     void* y, float* y32, int stride, cudaStream_t st) {
    const bf16* xb = static_cast<const bf16*>(x);
    const bf16* wb = static_cast<const bf16*>(w);
    bf16* yb = static_cast<bf16*>(y);
    if (stride == 2) {
        switch (co) {
            case 16: return launch_s2<16>(xb, wb, bias, yb, y32, D, H, W, ci, relu, st);
            case 32: return launch_s2<32>(xb, wb, bias, yb, y32, D, H, W, ci, relu, st);
            default: return launch_s2<64>(xb, wb, bias, yb, y32, D, H, W, ci, relu, st);
        }
    }
    return co == 16 ? launch_pipe<16>(xb, wb, bias, yb, y32, D, H, W, ci, co, relu, st)
                    : launch_pipe<32>(xb, wb, bias, yb, y32, D, H, W, ci, co, relu, st);
}

bool conv3_dx2_applies(int D, int H, int W, int ci, int co) {
    const bool ch = (ci == 16 || ci == 32 || ci == 64) && (co == 16 || co == 32 || co == 64);
    // Columns of a few voxels a plane leave nearly all of a block's 8 x 16 rows
    // empty: the mma.sync kernel, the same sums bit for bit (64 -> 64 channels, us
    // here / there: 4096 x 1 x 1 92.6 / 18.7, 2048 x 2 x 2 61.8 / 24.5, 1024 x 4 x 4
    // 45.3 / 26.9, but 1024 x 8 x 8 44.7 / 73.0).
    if ((int64_t)((H + 1) / 2) * ((W + 1) / 2) <= 8) return false;
    return ch && D > 0 && H > 0 && W > 0 &&
           ((int64_t)(D + 1) / 2) * ceil_div((H + 1) / 2, TY) * ceil_div((W + 1) / 2, TX) <= 0x7fffffffLL;
}

cudaError_t conv3_dx2(const void* dy, const void* wt, void* dx, int D, int H, int W, int ci, int co, cudaStream_t st) {
    const bf16* db = static_cast<const bf16*>(dy);
    const bf16* wb = static_cast<const bf16*>(wt);
    return ci == 16 ? launch_dx2<16>(db, wb, static_cast<bf16*>(dx), D, H, W, ci, co, st)
                    : launch_dx2<32>(db, wb, static_cast<bf16*>(dx), D, H, W, ci, co, st);
}

bool conv_wgrad_tiles_applies(int D, int H, int W, int ci, int co, int ks, int stride) {
    const bool ch = (ci == 16 || ci == 32 || ci == 64) && (co == 16 || co == 32 || co == 64);
    if (!ch || D <= 0 || H <= 0 || W <= 0 || !((ks == 3 && (stride == 1 || stride == 2)) || (ks == 1 && stride == 1)))
        return false;
    // Of a few voxels a sum costs less than a tile's way through shared memory and
    // the block's sums: the plain mma.sync kernel, a block a tap (us here / there, 3x3x3
    // stride 1, 16 -> 16 and 64 -> 64 channels: 1 voxel 8.6 / 4.3 and 10.5 / 4.4, 64 10.8 / 6.5
    // and 12.6 / 8.3, 93 10.6 / 8.4 and 14.6 / 10.3, 128 9.2 / 10.4 and 12.5 / 12.4, 512
    // 11.5 / 32.0; stride 2, 64: 8.4 / 6.5, 125 8.6 / 10.4; 1x1x1, 16: 6.1 / 4.2, 51 5.7 / 6.4).
    const int64_t out = (int64_t)((D - 1) / stride + 1) * ((H - 1) / stride + 1) * ((W - 1) / stride + 1);
    return out > (ks == 3 ? 96 : 24) && (int64_t)D * H * W < ((int64_t)1 << 31);
}

cudaError_t conv_wgrad_tiles(const void* x, int D, int H, int W, int ci, const void* dy, int co, int ks, int stride,
                             float* dw, cudaStream_t st) {
    const bf16* xb = static_cast<const bf16*>(x);
    const bf16* db = static_cast<const bf16*>(dy);
    if (ks == 1)
        return co == 16 ? launch_wgrad<WGeo<1, 1, 16>>(xb, db, dw, D, H, W, ci, co, st)
                        : launch_wgrad<WGeo<1, 1, 32>>(xb, db, dw, D, H, W, ci, co, st);
    if (stride == 1)
        return co == 16 ? launch_wgrad<WGeo<3, 1, 16>>(xb, db, dw, D, H, W, ci, co, st)
                        : launch_wgrad<WGeo<3, 1, 32>>(xb, db, dw, D, H, W, ci, co, st);
    return co == 16 ? launch_wgrad<WGeo<3, 2, 16>>(xb, db, dw, D, H, W, ci, co, st)
                    : launch_wgrad<WGeo<3, 2, 32>>(xb, db, dw, D, H, W, ci, co, st);
}

cudaError_t conv3_flip_transpose(const void* w, void* wt, int co, int ci, cudaStream_t st) {
    const int64_t n = (int64_t)co * 27 * ci;
    k_flip_transpose<<<(unsigned)ceil_div(n, 256), 256, 0, st>>>(static_cast<const bf16*>(w), static_cast<bf16*>(wt),
                                                               co, ci);
    return cudaGetLastError();
}

cudaError_t conv_tc_status(unsigned* flags) {
    cudaError_t e = cudaMemcpyFromSymbol(flags, g_conv_tc_flags, sizeof(unsigned));
    if (e != cudaSuccess) return e;
    const unsigned zero = 0;
    return cudaMemcpyToSymbol(g_conv_tc_flags, &zero, sizeof(unsigned));
}

}  // namespace lbm
