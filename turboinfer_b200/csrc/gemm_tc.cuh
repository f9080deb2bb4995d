// gemm_tc.cuh -- tcgen05 tensor-core GEMM for the batched side of the hot path (prefill / batched decode), where the
// work really is a dense contraction:  Y[M,N] = X[M,K] . dequant(Wq[K,N]).
//
// Replaces simd_gemm_float (src/core/tensor_engine.cpp:191-255, the M,N,K >= 32 branch of TensorEngine::matmul) on
// quantized weights.  Same arithmetic contract as the streaming GEMV (gemv.cuh), so a row of the GEMM is bit-identical
// to the GEMV of that row: each activation row is converted to 24-bit block fixed point and split into three signed
// 8-bit digit planes; the tensor cores multiply the INT8 planes with the INT8 / unpacked-INT4 weights (kind::i8, exact
// int32 accumulation in TMEM, one accumulator per digit); the epilogue recombines the digits in int64 and scales once.
//
// A pair of neighbouring SMs (cta_group::2) owns a tile of 256 weight columns x T tokens.  The MMA's M side is the weight columns (128 a
// CTA), its N side the tokens, whose digit rows are split between the two CTAs; D[256 x T] per digit plane, 3 T <= 480 TMEM columns.  A k-step
// brings 16 KiB of weights and 3 T / 2 digit rows into each CTA for 6 T clocks of tensor work: 48 bytes a clock and SM at T = 160, against
// 85 for one-CTA tiles of 128 x 128 (L2 gives an SM about 64).  Clusters walk the tiles, tokens fastest.
//   warp 0        producer: one box of the weights' tile images, one 3-D box of the digit planes (128 B x T / 2 rows x 3 planes,
//                 SWIZZLE_128B) a stage; both CTAs' copies complete on the even CTA's barrier; 4 stages of 46 KiB
//   warp 1        TMEM allocation; even CTA: tcgen05.mma (M 256, N T, K 32), 4 k-steps x 3 digits a stage, issued warp-uniformly (elect_one)
//   warps 2..9    epilogue: tcgen05.ld 32x32b (lane = weight column), digit recombination, scale, residual, stores of 32 neighbouring columns
// Measured (kernel alone, INT8 weights, B200; before = one-CTA tiles of 128 x 128 with one-lane issue): M 2048, K 4096, N 22016 525 -> 385 us
// (2.88 POP/s of INT8 work issued), K 4096, N 12288 292 -> 220, K 11008, N 4096 248 -> 184 (3.0 POP/s); M 256, K 4096, N 4096 16 us.  Bound by
// the tensor pipe at the power cap plus an exposed epilogue of about 3 us a tile.
// Operands are K-major in shared memory; descriptors follow the sm_100 layout (start address, SBO = 1024 B between 8-row
// groups, version 1, layout type SWIZZLE_128B); the k-step inside the 128-byte swizzle atom advances the start address.
#pragma once
#include <cuda.h>

#include <algorithm>

#include "gemv.cuh"

namespace tib {

constexpr int kGemmBM = 128, kGemmBN = 128, kGemmBK = 128;   // row padding of the planes; weight columns of a CTA; BK in bytes = int8 elements
constexpr int kGemmMaxTokens = 160;
constexpr int kGemmStages = 4, kGemmEpiWarps = 8;
constexpr int kGemmThreads = 64 + 32 * kGemmEpiWarps;
constexpr int kGemmTileBytes = kGemmBN * kGemmBK;              // 16 KiB of weights
constexpr int kGemmStageBytes = kGemmTileBytes + 3 * (kGemmMaxTokens / 2) * kGemmBK;   // + three digit planes of half the tile's tokens: 46 KiB
constexpr size_t kGemmSmemBytes = (size_t)kGemmStages * kGemmStageBytes + 1024 /*align*/ + 256 /*barriers*/ + kGemmMaxTokens * 16 /*the tokens' numbers*/;

struct GemmArgs {
    int M, N, K;            // logical sizes
    int m_pad, k_pad;       // padded to 128
    int a_signed_b;         // 1: weights are signed bytes (INT8), 0: unsigned (INT4 nibbles stored as q + woff)
    int woff;
    const float* sx;        // [M] s_x of each row
    const long long* sxf;   // [M] sum of xf of each row
    const float* colscale;  // [N]
    const float* colzterm;  // [N] or nullptr
    float* y;               // [M][N]
    const float* resid;     // optional [M][N] added to the result (may alias y): the residual connections of the decoder
    const uint8_t* wt;      // weights, tile-major pre-swizzled (wtile_offset)
};

// ---- activations -> digit planes [3][m_pad][k_pad] (K-major rows), one block per row ------------------------
__global__ void gemm_digits_kernel(const float* x, int M, int K, int m_pad, int k_pad, int8_t* planes, float* sx_out, long long* sxf_out) {
    __shared__ float red[32];
    __shared__ long long redl[32];
    const int row = blockIdx.x;
    const float* xr = x + (size_t)row * K;
    float amax = 0.f;
    for (int k = threadIdx.x; k < K; k += blockDim.x) amax = fmaxf(amax, fabsf(xr[k]));
    amax = warp_max(amax);
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = amax;
    __syncthreads();
    amax = 0.f;
    for (int i = 0; i < (int)(blockDim.x >> 5); ++i) amax = fmaxf(amax, red[i]);
    const bool finite = amax > 0.f && amax < INFINITY;
    const float inv_s = finite ? kXQMax / amax : 0.f;   // the expressions of gemv_stage_x, so rows match the GEMV bit for bit
    const float s_x = finite ? amax / kXQMax : 0.f;
    long long sxf = 0;
    for (int k = threadIdx.x; k < k_pad; k += blockDim.x) {
        const int f = k < K ? __float2int_rn(xr[k] * inv_s) : 0;
        sxf += f;
        // signed digits, f = d2*65536 + d1*256 + d0 with every digit in [-128, 127]: the bytes of f + 0x808080, xor 0x80
        const int u = f + 0x808080;
        planes[((size_t)0 * m_pad + row) * k_pad + k] = (int8_t)((u & 0xFF) ^ 0x80);
        planes[((size_t)1 * m_pad + row) * k_pad + k] = (int8_t)(((u >> 8) & 0xFF) ^ 0x80);
        planes[((size_t)2 * m_pad + row) * k_pad + k] = (int8_t)(((u >> 16) & 0xFF) ^ 0x80);
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) sxf += __shfl_xor_sync(0xffffffffu, sxf, o);
    if ((threadIdx.x & 31) == 0) redl[threadIdx.x >> 5] = sxf;
    __syncthreads();
    if (threadIdx.x == 0) {
        long long t = 0;
        for (int i = 0; i < (int)(blockDim.x >> 5); ++i) t += redl[i];
        sx_out[row] = s_x;
        sxf_out[row] = t;
    }
}

// ---- the B operand in HBM: tile-major, pre-swizzled ---------------------------------------------------------------
// A weight tile of a k-step (128 columns x 128 B of k) is stored as the exact 16 KiB SWIZZLE_128B image the MMA reads from
// shared memory, tiles ordered [column tile][k-step]: one 1-D bulk copy per tile and k-step.  (A TMA box over a row-major
// [N][K] copy fetches 128 separate 128-byte rows 4 KiB apart; streamed once from HBM that was bound by the TMA request
// rate at ~30 GB/s per SM -- measured, ~1 us per k-step whatever the pipeline depth.)
// SWIZZLE_128B: inside every 8-row x 128-byte atom the 16-byte chunk c of row r sits at chunk position c ^ (r & 7).
TIB_HD size_t sw128_offset(int row, int byte) {   // inside a tile whose rows are 128 B
    return (size_t)(row >> 3) * 1024 + (size_t)(row & 7) * 128 + (size_t)(((byte >> 4) ^ (row & 7)) << 4) + (byte & 15);
}
TIB_HD size_t wtile_offset(int n, int k, int k_pad) {
    return ((size_t)(n / kGemmBN) * (k_pad / kGemmBK) + k / kGemmBK) * kGemmTileBytes + sw128_offset(n % kGemmBN, k % kGemmBK);
}
// packed streaming layout -> tile-major bytes, grid (slabs, parts), thread mapping of unpack_kernel.  A word of the packed layout is four
// consecutive k of one column (INT8), or two such fours 32 k apart (INT4, low and high nibbles): whole words are stored (with byte stores the
// first prompt of a model behind 0.8 GB of INT8 weights took 16 ms longer than the next one, now 7)
__global__ void unpack_kmajor_kernel(const uint8_t* packed, QLayout L, int k_pad, uint8_t* wk) {
    const Slab slab = make_slab(L, blockIdx.x);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int kik = kitem_k(L.bits);
    for_each_quad_word(L, slab, warp, lane, [&](size_t off, int nl, int grp, int chunk, int ki, int widx) {
        const uint32_t word = *reinterpret_cast<const uint32_t*>(packed + off);
        int row, kk;
        kitem_word_elem(L.bits, nl, widx, 0, row, kk);
        const int n = slab.col0 + 16 * grp + row, k = chunk * L.kc + ki * kik + kk;   // (k and k_pad are multiples of four)
        if (L.bits == 8) {   // two's complement q
            if (k < k_pad) *reinterpret_cast<uint32_t*>(wk + wtile_offset(n, k, k_pad)) = word;
        } else {             // u = q + woff (0..15)
            if (k < k_pad) *reinterpret_cast<uint32_t*>(wk + wtile_offset(n, k, k_pad)) = word & 0x0F0F0F0Fu;
            if (k + 32 < k_pad) *reinterpret_cast<uint32_t*>(wk + wtile_offset(n, k + 32, k_pad)) = (word >> 4) & 0x0F0F0F0Fu;
        }
    }, blockIdx.y, gridDim.y);
}

// ---- PTX wrappers ---------------------------------------------------------------------------------------
__device__ __forceinline__ void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }
__device__ __forceinline__ bool mbar_wait_bounded(uint64_t* bar, uint32_t parity, int* err) {
    if (mbar_try_wait(bar, parity)) return true;
    const long long t0 = clock64();
    while (!mbar_try_wait(bar, parity)) {
        if (clock64() - t0 > 2000000000LL) {   // about a second
            *reinterpret_cast<volatile int*>(err) = 1;   // (device or mapped host memory)
            return false;
        }
    }
    return true;
}
// The last thing a producer does: wait (again with a limit) until the copies it asked for have landed, also when it or another role gave up, so that
// none arrives in shared memory that the block has left.  Stage i was filled uses + 1 times for i < st, uses times otherwise.  (Copies of both blocks of a
// pair complete on the even one's barriers; the cluster barrier at the exit holds the odd one.)
__device__ __forceinline__ void drain_copies(uint64_t* full, int stages, int st, int uses, int* err) {
    for (int i = 0; i < stages; ++i) {
        const int n = uses + (i < st ? 1 : 0);
        if (n > 0) mbar_wait_bounded(&full[i], (n - 1) & 1, err);
    }
}
__device__ __forceinline__ uint32_t cluster_ctarank() {
    uint32_t r;
    asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
    return r;
}
__device__ __forceinline__ void cluster_sync_all() {
    asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
// the shared-memory address of the even CTA's copy of a barrier (bit 24 of a shared::cluster address is the CTA's place in its pair)
__device__ __forceinline__ uint32_t pair_leader(uint32_t saddr) { return saddr & 0xFEFFFFFFu; }
__device__ __forceinline__ void tma_load_2d_pair(uint32_t dst, const CUtensorMap* map, int c0, int c1, uint32_t bar, uint32_t lead) {
    asm volatile(
        "{\n\t.reg .pred e;\n\tsetp.ne.b32 e, %5, 0;\n\t"
        "@e cp.async.bulk.tensor.2d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];\n\t}" ::"r"(dst),
        "l"(reinterpret_cast<uint64_t>(map)), "r"(c0), "r"(c1), "r"(bar), "r"(lead)
        : "memory");
}
__device__ __forceinline__ void mbar_expect_tx_if(uint32_t bar, uint32_t bytes, uint32_t lead) {
    asm volatile("{\n\t.reg .pred e;\n\tsetp.ne.b32 e, %2, 0;\n\t@e mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;\n\t}" ::"r"(bar), "r"(bytes), "r"(lead) : "memory");
}
// One lane of the warp, the same one every time.  The warps that drive the copy engine and the tensor cores run their loops with all lanes
// and let `lead` predicate the single-thread instructions: inside a branch that one lane takes, the operands of those instructions live
// in per-thread registers and every issue pays for moving them to uniform ones (measured: 80 clocks a tcgen05.mma, 630 a k-step of any
// width; without the branch the k-step runs at the tensor rate).
__device__ __forceinline__ uint32_t elect_one() {
    uint32_t lead;
    asm volatile("{\n\t.reg .pred e;\n\telect.sync _|e, 0xffffffff;\n\tselp.u32 %0, 1, 0, e;\n\t}" : "=r"(lead));
    return lead;
}
__device__ __forceinline__ void tc_commit_pair(uint32_t bar, uint32_t lead) {   // arrives at the barrier of that offset in both CTAs
    asm volatile(
        "{\n\t.reg .pred e;\n\tsetp.ne.b32 e, %2, 0;\n\t"
        "@e tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;\n\t}" ::"r"(bar), "h"((uint16_t)3), "r"(lead)
        : "memory");
}
__device__ __forceinline__ void mbar_arrive_cluster(uint32_t bar) {
    asm volatile("mbarrier.arrive.release.cluster.shared::cluster.b64 _, [%0];" ::"r"(bar) : "memory");
}
__device__ __forceinline__ void tmem_ld32(uint32_t (&a)[32], uint32_t taddr) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x32.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16, %17, %18, %19, %20, %21, %22, %23, %24, "
        "%25, %26, %27, %28, %29, %30, %31}, [%32];"
        : "=r"(a[0]), "=r"(a[1]), "=r"(a[2]), "=r"(a[3]), "=r"(a[4]), "=r"(a[5]), "=r"(a[6]), "=r"(a[7]), "=r"(a[8]), "=r"(a[9]), "=r"(a[10]), "=r"(a[11]),
          "=r"(a[12]), "=r"(a[13]), "=r"(a[14]), "=r"(a[15]), "=r"(a[16]), "=r"(a[17]), "=r"(a[18]), "=r"(a[19]), "=r"(a[20]), "=r"(a[21]), "=r"(a[22]), "=r"(a[23]),
          "=r"(a[24]), "=r"(a[25]), "=r"(a[26]), "=r"(a[27]), "=r"(a[28]), "=r"(a[29]), "=r"(a[30]), "=r"(a[31])
        : "r"(taddr));
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
}

__device__ __forceinline__ void tc_commit_if(uint32_t bar, uint32_t lead) {
    asm volatile(
        "{\n\t.reg .pred e;\n\tsetp.ne.b32 e, %1, 0;\n\t"
        "@e tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];\n\t}" ::"r"(bar), "r"(lead)
        : "memory");
}
__device__ __forceinline__ void bulk_g2s_if(uint32_t dst, const void* src, uint32_t bytes, uint32_t bar, uint32_t lead) {
    asm volatile(
        "{\n\t.reg .pred e;\n\tsetp.ne.b32 e, %4, 0;\n\t"
        "@e cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];\n\t}" ::"r"(dst),
        "l"(src), "r"(bytes), "r"(bar), "r"(lead)
        : "memory");
}

__device__ __forceinline__ void tc_mma_i8_if(uint32_t tmem_d, uint64_t adesc, uint64_t bdesc, uint32_t idesc, uint32_t accumulate, uint32_t lead) {
    asm volatile(
        "{\n\t.reg .pred p, e;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "setp.ne.b32 e, %5, 0;\n\t"
        "@e tcgen05.mma.cta_group::1.kind::i8 [%0], %1, %2, %3, p;\n\t}"
        ::"r"(tmem_d), "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate), "r"(lead)
        : "memory");
}
// K-major, SWIZZLE_128B, tile rows 128 B apart inside 1024-byte 8-row groups
__device__ __forceinline__ uint64_t umma_desc_sw128(uint32_t smem_addr) {
    uint64_t d = 0;
    d |= (uint64_t)((smem_addr >> 4) & 0x3FFF);        // start address
    d |= (uint64_t)1 << 16;                             // leading byte offset (unused for swizzled K-major)
    d |= (uint64_t)(1024 >> 4) << 32;                   // stride byte offset: 8 rows x 128 B
    d |= (uint64_t)1 << 46;                             // descriptor version (Blackwell)
    d |= (uint64_t)2 << 61;                             // SWIZZLE_128B
    return d;
}
// One tile of the pair kernel: 256 weight columns (128 a CTA) x T tokens, T a multiple of 32 up to 160 chosen by i8_tile_tokens()
struct PairGemmArgs {
    GemmArgs g;
    int T;             // tokens of a tile
    int tiles_t, tiles;
    int* err;          // set to 1 when a wait ran out
};
__device__ __forceinline__ void tma_load_3d_pair(uint32_t dst, const CUtensorMap* map, int c0, int c1, int c2, uint32_t bar, uint32_t lead) {
    asm volatile(
        "{\n\t.reg .pred e;\n\tsetp.ne.b32 e, %6, 0;\n\t"
        "@e cp.async.bulk.tensor.3d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4}], [%5];\n\t}" ::"r"(dst),
        "l"(reinterpret_cast<uint64_t>(map)), "r"(c0), "r"(c1), "r"(c2), "r"(bar), "r"(lead)
        : "memory");
}
__device__ __forceinline__ void tc_mma_i8_pair(uint32_t tmem_d, uint64_t adesc, uint64_t bdesc, uint32_t idesc, uint32_t accumulate, uint32_t lead) {
    asm volatile(
        "{\n\t.reg .pred p, e;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "setp.ne.b32 e, %5, 0;\n\t"
        "@e tcgen05.mma.cta_group::2.kind::i8 [%0], %1, %2, %3, p;\n\t}"
        ::"r"(tmem_d), "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate), "r"(lead)
        : "memory");
}
__host__ __device__ constexpr uint32_t umma_idesc_i8_mn(int a_signed, int b_signed, int m, int n) {
    return (2u << 4) | ((uint32_t)a_signed << 7) | ((uint32_t)b_signed << 10) | ((uint32_t)(n >> 3) << 17) | ((uint32_t)(m >> 4) << 24);   // D format S32
}
// the integer sum of a (column, token), and it as fp32: exact in 64 bits, then one rounding (the GEMV epilogue's expression)
__device__ __forceinline__ long long digits_sum(int a2, int a1, int a0) { return ((long long)a2 << 16) + ((long long)a1 << 8) + (long long)a0; }
__device__ __forceinline__ float int_to_float(long long t) {
    const int hi = (int)(t >> 23), lo = (int)(t & 0x7FFFFF);
    return fmaf((float)hi, 8388608.0f, (float)lo);
}
// tokens of a tile: waves of the pairs times what they cost in clocks -- a k-step takes 6 a token at the tensor rate or its bytes at
// 60 a clock, a tile its epilogue on top (the accumulators of a wide tile fill TMEM, so the next tile starts behind it)
inline int i8_tile_tokens(int M, int n_tiles, int ksteps, int pairs) {
    int best = 160;
    float best_t = 1e30f;
    for (int T = 160; T >= 32; T -= 32) {
        const int waves = (((M + T - 1) / T) * n_tiles + pairs - 1) / pairs;
        const float step = std::max(6.f * T, (kGemmTileBytes + 192.f * T) / 60.f);
        const float t = waves * (ksteps * step + 1500.f + 20.f * T);
        if (t < best_t) { best_t = t; best = T; }
    }
    return best;
}

__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(kGemmThreads, 1)
gemm_i8_tc_kernel(const __grid_constant__ CUtensorMap map_x, const __grid_constant__ CUtensorMap map_w, const PairGemmArgs pg) {
    extern __shared__ uint8_t gsm_raw[];
    const GemmArgs& g = pg.g;
    const uint32_t base = (smem_u32(gsm_raw) + 1023u) & ~1023u;
    uint8_t* tiles = gsm_raw + (base - smem_u32(gsm_raw));
    uint64_t* full = reinterpret_cast<uint64_t*>(tiles + (size_t)kGemmStages * kGemmStageBytes);
    uint64_t* empty = full + kGemmStages;
    uint64_t* acc_full = empty + kGemmStages;
    uint64_t* acc_empty = acc_full + 1;       // the even CTA's: both CTAs' epilogue warps
    uint32_t* tmem_ptr = reinterpret_cast<uint32_t*>(acc_empty + 1);
    // [160] of the tile's tokens: woff * sum(xf), then {s_x, sum(xf)}
    long long* s_off = reinterpret_cast<long long*>(tiles + (size_t)kGemmStages * kGemmStageBytes + 256);
    float2* s_x = reinterpret_cast<float2*>(s_off + kGemmMaxTokens);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const uint32_t rank = cluster_ctarank();
    const int pair = blockIdx.x >> 1, pairs = gridDim.x >> 1;
    const int KB = g.k_pad / kGemmBK, T = pg.T;

    if (threadIdx.x == 0) {
        for (int i = 0; i < kGemmStages; ++i) { mbar_init(&full[i], 1); mbar_init(&empty[i], 1); }
        mbar_init(acc_full, 1);
        mbar_init(acc_empty, 2 * kGemmEpiWarps);
        fence_mbar_init();
    }
    if (warp == 1) {
        asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], 512;" ::"r"(smem_u32(tmem_ptr)) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
    }
    pdl_wait_prior_grid();   // (everything above touches only this CTA: it runs under the tail of the kernel before)
    tc_fence_before();
    __syncthreads();
    cluster_sync_all();      // the peer's barriers are initialised before anything is signalled across
    tc_fence_after();
    const uint32_t tmem = *tmem_ptr;

    if (warp == 0) {
        const uint32_t lead = elect_one();
        const uint32_t bytes = 2u * (uint32_t)(kGemmTileBytes + 3 * (T / 2) * kGemmBK);   // both CTAs' boxes (rows beyond the tensors arrive as zeros and count)
        const uint32_t full_s = smem_u32(full);
        bool ok = true;
        int st = 0, use = 0;
        for (int tile = pair; tile < pg.tiles && ok; tile += pairs) {
            const int tb = tile % pg.tiles_t, nb = tile / pg.tiles_t;
            const int tok = tb * T + (int)rank * (T / 2), wrow = (2 * nb + (int)rank) * KB * kGemmBN;
            for (int kb = 0; kb < KB; ++kb) {
                if (use > 0 && !(ok = mbar_wait_bounded(&empty[st], (use - 1) & 1, pg.err))) break;
                const uint32_t sbase = base + st * kGemmStageBytes, bar = pair_leader(full_s + 8 * st);
                if (rank == 0) mbar_expect_tx_if(full_s + 8 * st, bytes, lead);
                tma_load_2d_pair(sbase, &map_w, 0, wrow + kb * kGemmBN, bar, lead);
                tma_load_3d_pair(sbase + kGemmTileBytes, &map_x, kb * kGemmBK, tok, 0, bar, lead);
                if (++st == kGemmStages) { st = 0; ++use; }
            }
        }
        if (rank == 0) drain_copies(full, kGemmStages, st, use, pg.err);
    } else if (warp == 1) {
        if (rank == 0) {
            const uint32_t lead = elect_one();
            const uint32_t idesc = umma_idesc_i8_mn(g.a_signed_b, 1, 256, T);   // A = weights (unsigned nibbles in bytes or signed bytes), B = signed digits
            const uint64_t desc0 = umma_desc_sw128(base);   // (addresses stay below 2^18: adding to the address field never carries out of it)
            const uint32_t empty_s = smem_u32(empty), plane = (uint32_t)(T / 2) * kGemmBK >> 4;
            bool ok = true;
            int st = 0, use = 0, n_tile = 0;
            for (int tile = pair; tile < pg.tiles && ok; tile += pairs, ++n_tile) {
                if (n_tile > 0) ok = mbar_wait_bounded(acc_empty, (n_tile - 1) & 1, pg.err);
                tc_fence_after();
                for (int kb = 0; kb < KB && ok; ++kb) {
                    ok = mbar_wait_bounded(&full[st], use & 1, pg.err);
                    if (!ok) break;
                    tc_fence_after();
                    const uint64_t wd = desc0 + (uint64_t)(st * (kGemmStageBytes >> 4)), xd = wd + (kGemmTileBytes >> 4);
#pragma unroll
                    for (int k4 = 0; k4 < kGemmBK / 32; ++k4)
#pragma unroll
                        for (int d = 0; d < 3; ++d)
                            tc_mma_i8_pair(tmem + d * T, wd + 2 * k4, xd + d * plane + 2 * k4, idesc, (kb | k4) != 0 ? 1u : 0u, lead);
                    tc_commit_pair(empty_s + 8 * st, lead);
                    if (++st == kGemmStages) { st = 0; ++use; }
                }
                tc_commit_pair(smem_u32(acc_full), lead);   // also on the failure path: the epilogue warps must not wait for ever
            }
        }
    } else {
        // TMEM lane = weight column, TMEM column = token: a store of a warp is 32 neighbouring columns of one token
        const int q = warp & 3, half = (warp - 2) >> 2, et = threadIdx.x - 64;
        bool ok = true;
        int n_tile = 0;
        // (after a failed wait the loop goes on without waiting or storing: the warps meet at the same barriers to the end)
        for (int tile = pair; tile < pg.tiles; tile += pairs, ++n_tile) {
            const int tb = tile % pg.tiles_t, nb = tile / pg.tiles_t;
            const int tok0 = tb * T;
            bar_sync(1, 32 * kGemmEpiWarps);   // the previous tile's token numbers are no longer read
            if (et < T) {
                const bool in = tok0 + et < g.M;
                const long long sxf = in ? g.sxf[tok0 + et] : 0;
                s_off[et] = g.woff * sxf;
                s_x[et] = make_float2(in ? g.sx[tok0 + et] : 0.f, (float)sxf);
            }
            bar_sync(1, 32 * kGemmEpiWarps);
            const int n = (2 * nb + (int)rank) * kGemmBN + q * 32 + lane;
            const bool n_ok = n < g.N;
            const float cs = n_ok ? g.colscale[n] : 0.f;
            const float zt = (n_ok && g.colzterm) ? g.colzterm[n] : 0.f;
            if (ok) ok = mbar_wait_bounded(acc_full, n_tile & 1, pg.err);
            ok = __all_sync(0xffffffffu, ok);
            tc_fence_after();
            const int c1 = min((half + 1) * (T / 2), g.M - tok0);
            for (int c0 = half * (T / 2); ok && c0 < c1; c0 += 16) {
                uint32_t a[3][16];
#pragma unroll
                for (int d = 0; d < 3; ++d) {
                    const uint32_t taddr = tmem + ((uint32_t)(q * 32) << 16) + (uint32_t)(d * T + c0);
                    asm volatile(
                        "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];"
                        : "=r"(a[d][0]), "=r"(a[d][1]), "=r"(a[d][2]), "=r"(a[d][3]), "=r"(a[d][4]), "=r"(a[d][5]), "=r"(a[d][6]), "=r"(a[d][7]),
                          "=r"(a[d][8]), "=r"(a[d][9]), "=r"(a[d][10]), "=r"(a[d][11]), "=r"(a[d][12]), "=r"(a[d][13]), "=r"(a[d][14]), "=r"(a[d][15])
                        : "r"(taddr));
                }
                float r[16];
                const size_t at = (size_t)(tok0 + c0) * g.N + n;
#pragma unroll
                for (int i = 0; i < 16; ++i) r[i] = (g.resid && n_ok && c0 + i < c1) ? g.resid[at + (size_t)i * g.N] : 0.f;
                asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
                float v[16];
#pragma unroll
                for (int i = 0; i < 16; ++i) {
                    const float2 x = s_x[c0 + i];
                    const float tf = int_to_float(digits_sum((int)a[2][i], (int)a[1][i], (int)a[0][i]) - s_off[c0 + i]);
                    v[i] = (fmaf(zt, x.y, tf) * x.x) * cs;   // (zt = 0 without a zero point: the sum itself)
                }
#pragma unroll
                for (int i = 0; i < 16; ++i)
                    if (n_ok && c0 + i < c1) g.y[at + (size_t)i * g.N] = g.resid ? r[i] + v[i] : v[i];
            }
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive_cluster(pair_leader(smem_u32(acc_empty)));
        }
    }
    tc_fence_before();
    __syncthreads();
    cluster_sync_all();   // nothing of the peer's is in flight towards this CTA's shared memory or TMEM any more
    if (warp == 1) {
        tc_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, 512;" ::"r"(tmem) : "memory");
    }
}

// ---- the same GEMM for M <= 32 rows (batched decode), operands swapped, dealt evenly to the SMs ------------------------
// With a handful of rows the work is a stream of weights.  The MMA's M side (128 rows) are 128 WEIGHT COLUMNS, its N side R batch rows
// (16 or 32) of all three digit planes at once, D[128 x 3 R].  The (column tile, k-step) units of the whole matrix are numbered tile by
// tile and every CTA takes one contiguous run of them, so that all SMs stream the same number of bytes whatever the number of
// column tiles (172 tiles of a 4096 x 22016 matrix on 148 SMs would otherwise be two waves); a run covers the end of a tile, whole tiles, the
// beginning of another.
//   * per k-step a CTA loads 16 KiB of weights and 3 R digit rows (6 or 12 KiB -- the same bytes for every CTA, an L2 broadcast), both stored
//     as ready-made swizzled tile images and fetched with 1-D bulk copies into a ring of 196 KiB; under programmatic dependent launch
//     the first ring of WEIGHTS is requested while the kernel before (which makes the digits) still runs;
//   * a tile that several CTAs share: each leaves its partial sums (exact integers) in its own place of a workspace and counts itself in;
//     the CTA that arrives last adds them (order-independent: bit-identical to an unshared tile), applies offset, scales and residual, and
//     leaves the counter zeroed for the next GEMM;
//   * two accumulators: the epilogue of a tile runs under the k-steps of the next.
// warps 0..7: epilogue (warp w: weight columns 32 (w % 4) .., rows 16 (w / 4) ..), warp 8: TMEM allocation + MMA issue, warp 9: producer.
// Measured (4096 x 22016, 32 rows, us a launch in a chain of launches on a B200): 31 with whole column tiles and K split into at most eight,
// 22 now; the four products of a 4096-wide layer on average 29 -> 20.7, against 3 to 14 for their weight bytes.
constexpr int kSmallRows = 32, kSmallEpiWarps = 8, kSmallThreads = 64 + 32 * kSmallEpiWarps;
constexpr int kSmallRing = 196 * 1024;
constexpr int kSmallTmemCols = 256;                                          // two accumulators of up to 96 columns
constexpr size_t kSmallSmemBytes = (size_t)kSmallRing + 1024 /*align*/ + 256 /*barriers*/ + kSmallRows * 16 /*the rows' numbers*/;
__host__ __device__ constexpr int small_stage_bytes(int R) { return kGemmTileBytes + 3 * R * kGemmBK; }   // 28 KiB (7 stages) or 22 KiB (8 of 9)
__host__ __device__ constexpr int small_stages(int R) { return R == 32 ? 7 : 8; }
// the digit planes of a step's rows are laid out for 16 or for 32 rows
TIB_HD int small_rows(int M) { return M <= 16 ? 16 : 32; }

// The digit planes for this kernel: [k-step][3 R rows = R d + m][128 B], each k-step's rows the exact SWIZZLE_128B image (one bulk copy)
TIB_HD size_t xtile_offset(int d, int m, int k, int R) {
    return (size_t)(k / kGemmBK) * 3 * R * kGemmBK + sw128_offset(d * R + m, k % kGemmBK);
}
struct SmallArgs {
    const uint8_t* xt;        // digit planes in xtile_offset order
    long long* ws;            // [2 CTAs][32][128] partial sums: a CTA's first and last tile when they are shared
    unsigned int* cnt;        // [column tiles] arrivals, zero between GEMMs
    int tiles, KB;            // column tiles, k-steps
    int* err;                 // set to 1 when a wait ran out
};
// first unit of CTA c (units * CTAs fits 32 bits: at most 2^22 units on 148 SMs)
TIB_HD int small_unit(int units, int c, int ctas) { return (int)((uint32_t)units * (uint32_t)c / (uint32_t)ctas); }
// CTAs of a launch: all SMs as long as each has at least four k-steps, a shorter run would be mostly the fix-up of its shared tiles.  Only matrices below 592
// units (9.7 M weights) are concerned.  A whole step of 4 rows through eight layers, us, at 1 / 2 / 4 / 8 / 16 k-steps: 256 wide 315 / 233 / 304 / 351 / 386, 512 wide
// 355 / 332 / 272 / 297 / 382, 768 wide 433 / 360 / 412 / 388 / 363, 1024 wide 510 / 413 / 349 / 302 / 336 (best where a run is a whole tile)
inline int small_gemm_ctas(int units, int sms) { return std::max(1, std::min(sms, units / 4)); }

template <int R>
__global__ void __launch_bounds__(kSmallThreads, 1)
gemm_i8_tc_small_kernel(const GemmArgs g, const SmallArgs sk) {
    constexpr int kStages = small_stages(R), kStageBytes = small_stage_bytes(R), kCols = 3 * R;
    static_assert(kStages * kStageBytes <= kSmallRing, "ring");
    extern __shared__ uint8_t gsm_raw[];
    const uint32_t base = (smem_u32(gsm_raw) + 1023u) & ~1023u;
    uint8_t* tiles = gsm_raw + (base - smem_u32(gsm_raw));
    uint64_t* full = reinterpret_cast<uint64_t*>(tiles + kSmallRing);
    uint64_t* empty = full + kStages;
    uint64_t* acc_full = empty + kStages;     // [2]
    uint64_t* acc_empty = acc_full + 2;       // [2]
    uint32_t* tmem_ptr = reinterpret_cast<uint32_t*>(acc_empty + 2);
    int* flag = reinterpret_cast<int*>(tmem_ptr + 1);
    long long* s_off = reinterpret_cast<long long*>(tiles + kSmallRing + 256);   // [32]: woff * sum(xf) per row, then {s_x, sum(xf)}
    float2* s_x = reinterpret_cast<float2*>(s_off + kSmallRows);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int KB = sk.KB, units = sk.tiles * KB, ctas = gridDim.x;
    const int u0 = small_unit(units, blockIdx.x, ctas), u1 = small_unit(units, blockIdx.x + 1, ctas);

    if (threadIdx.x == 0) {
        for (int i = 0; i < kStages; ++i) { mbar_init(&full[i], 1); mbar_init(&empty[i], 1); }
        for (int i = 0; i < 2; ++i) { mbar_init(&acc_full[i], 1); mbar_init(&acc_empty[i], kSmallEpiWarps); }
        fence_mbar_init();
    }
    if (warp == 8) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_ptr)), "n"(kSmallTmemCols) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = *tmem_ptr;
    pdl_launch_dependents();

    if (warp == 9) {
        const uint32_t lead = elect_one();
        const uint32_t full_s = smem_u32(full);
        auto weights = [&](int u, int st) {
            mbar_expect_tx_if(full_s + 8 * st, (uint32_t)kStageBytes, lead);
            bulk_g2s_if(base + st * kStageBytes, g.wt + (size_t)u * kGemmTileBytes, kGemmTileBytes, full_s + 8 * st, lead);   // (units are in the images' order)
        };
        auto digits = [&](int u, int st) {
            bulk_g2s_if(base + st * kStageBytes + kGemmTileBytes, sk.xt + (size_t)(u % KB) * kCols * kGemmBK, kCols * kGemmBK, full_s + 8 * st, lead);
        };
        const int ahead = min(kStages, u1 - u0);
        for (int i = 0; i < ahead; ++i) weights(u0 + i, i);
        pdl_wait_prior_grid();
        for (int i = 0; i < ahead; ++i) digits(u0 + i, i);
        int st = ahead % kStages, use = ahead / kStages;
        for (int u = u0 + ahead; u < u1; ++u) {
            if (!mbar_wait_bounded(&empty[st], (use - 1) & 1, sk.err)) break;
            weights(u, st);
            digits(u, st);
            if (++st == kStages) { st = 0; ++use; }
        }
        drain_copies(full, kStages, st, use, sk.err);
    } else if (warp == 8) {
        // A = weights (unsigned nibbles-in-bytes for INT4, signed for INT8); B = all three signed digit planes at once: their rows are
        // contiguous in the stage, so one MMA with N = 3 R fills the three accumulators (columns R d + m)
        const uint32_t lead = elect_one();
        const uint32_t id = umma_idesc_i8_mn(g.a_signed_b, 1, kGemmBN, kCols);
        const uint64_t desc0 = umma_desc_sw128(base);
        const uint32_t empty_s = smem_u32(empty);
        bool ok = true;
        int st = 0, use = 0, n_seg = 0;
        for (int u = u0; u < u1 && ok; ++n_seg) {
            const int buf = n_seg & 1, end = min(u1, (u / KB + 1) * KB), begin = u;
            if (n_seg > 1) ok = mbar_wait_bounded(&acc_empty[buf], ((n_seg >> 1) - 1) & 1, sk.err);
            tc_fence_after();
            for (; u < end && ok; ++u) {
                ok = mbar_wait_bounded(&full[st], use & 1, sk.err);
                if (!ok) break;
                tc_fence_after();
                const uint64_t wd = desc0 + (uint64_t)(st * (kStageBytes >> 4)), xd = wd + (kGemmTileBytes >> 4);
#pragma unroll
                for (int k4 = 0; k4 < kGemmBK / 32; ++k4) tc_mma_i8_if(tmem + buf * 128, wd + 2 * k4, xd + 2 * k4, id, (u != begin || k4 != 0) ? 1u : 0u, lead);
                tc_commit_if(empty_s + 8 * st, lead);
                if (++st == kStages) { st = 0; ++use; }
            }
            tc_commit_if(smem_u32(&acc_full[buf]), lead);   // also on the failure path: the epilogue warps must not wait for ever
        }
    } else {
        // epilogue: TMEM lane = weight column of the tile, TMEM column = batch row (per digit plane)
        pdl_wait_prior_grid();
        if (threadIdx.x < R) {
            const bool in = (int)threadIdx.x < g.M;
            const long long sxf = in ? g.sxf[threadIdx.x] : 0;
            s_off[threadIdx.x] = g.woff * sxf;
            s_x[threadIdx.x] = make_float2(in ? g.sx[threadIdx.x] : 0.f, (float)sxf);
        }
        bar_sync(1, 32 * kSmallEpiWarps);
        bool ok = true;
        int n_seg = 0;
        const int tile0 = u0 / KB, q = warp & 3, col = q * 32 + lane, m0 = 16 * (warp >> 2);
        const bool active = m0 < g.M;
        // (after a failed wait the loop goes on without storing: the warps meet at the same barriers to the end)
        for (int u = u0; u < u1; ++n_seg) {
            const int buf = n_seg & 1, tile = u / KB, end = min(u1, (tile + 1) * KB);
            const bool whole = u == tile * KB && end == (tile + 1) * KB;
            u = end;
            const int n = tile * kGemmBN + col;
            const bool n_ok = n < g.N;
            const float cs = n_ok ? g.colscale[n] : 0.f;
            const float zt = (n_ok && g.colzterm) ? g.colzterm[n] : 0.f;
            // a shared tile: the CTAs c0 .. c1 whose runs touch it
            int c0 = 0, c1 = 0;
            if (!whole) {
                const int first = tile * KB, last = first + KB - 1;
                c0 = (int)((uint32_t)first * (uint32_t)ctas / (uint32_t)units);
                while (small_unit(units, c0 + 1, ctas) <= first) ++c0;
                c1 = (int)((uint32_t)last * (uint32_t)ctas / (uint32_t)units);
                while (c1 + 1 < ctas && small_unit(units, c1 + 1, ctas) <= last) ++c1;
            }
            if (ok) ok = mbar_wait_bounded(&acc_full[buf], (n_seg >> 1) & 1, sk.err);
            ok = __all_sync(0xffffffffu, ok);
            tc_fence_after();
            auto finish = [&](const long long (&t)[16]) {   // t[i] = sum over all k of u * xf for (row m0 + i, column n)
                float r[16], y[16];
                const size_t at = (size_t)m0 * g.N + n;
#pragma unroll
                for (int i = 0; i < 16; ++i) r[i] = (g.resid && n_ok && m0 + i < g.M) ? g.resid[at + (size_t)i * g.N] : 0.f;
#pragma unroll
                for (int i = 0; i < 16; ++i) {
                    const float2 x = s_x[m0 + i];
                    y[i] = (fmaf(zt, x.y, int_to_float(t[i] - s_off[m0 + i])) * x.x) * cs;   // the GEMV epilogue's expression
                }
#pragma unroll
                for (int i = 0; i < 16; ++i)
                    if (n_ok && m0 + i < g.M) g.y[at + (size_t)i * g.N] = g.resid ? r[i] + y[i] : y[i];
            };
            constexpr int kPlace = kSmallRows * kGemmBN;
            if (active && ok) {
                uint32_t a[3][16];
#pragma unroll
                for (int d = 0; d < 3; ++d) {
                    const uint32_t taddr = tmem + ((uint32_t)(q * 32) << 16) + (uint32_t)(buf * 128 + d * R + m0);
                    asm volatile(
                        "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];"
                        : "=r"(a[d][0]), "=r"(a[d][1]), "=r"(a[d][2]), "=r"(a[d][3]), "=r"(a[d][4]), "=r"(a[d][5]), "=r"(a[d][6]), "=r"(a[d][7]),
                          "=r"(a[d][8]), "=r"(a[d][9]), "=r"(a[d][10]), "=r"(a[d][11]), "=r"(a[d][12]), "=r"(a[d][13]), "=r"(a[d][14]), "=r"(a[d][15])
                        : "r"(taddr));
                }
                asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
                long long t[16];
#pragma unroll
                for (int i = 0; i < 16; ++i) t[i] = digits_sum((int)a[2][i], (int)a[1][i], (int)a[0][i]);
                if (whole) {
                    finish(t);
                } else {   // (all 16 rows of the place: the ones beyond M are never read into a result)
                    long long* mine = sk.ws + ((size_t)blockIdx.x * 2 + (tile == tile0 ? 0 : 1)) * kPlace + (size_t)m0 * kGemmBN + col;
#pragma unroll
                    for (int i = 0; i < 16; ++i) __stcg(mine + (size_t)i * kGemmBN, t[i]);
                }
            }
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(&acc_empty[buf]);
            if (whole) continue;
            bar_sync(1, 32 * kSmallEpiWarps);
            if (threadIdx.x == 0) {
                fence_acq_rel_gpu();   // (the other warps' partial sums are ordered before this by the barrier)
                const unsigned int prev = atomicAdd(sk.cnt + tile, 1u);
                *flag = prev == (unsigned int)(c1 - c0) ? 1 : 0;
                if (*flag) sk.cnt[tile] = 0u;
                fence_acq_rel_gpu();
            }
            bar_sync(1, 32 * kSmallEpiWarps);
            if (*flag && ok && active) {
                long long t[16];
#pragma unroll
                for (int i = 0; i < 16; ++i) t[i] = 0;
                for (int c = c0; c <= c1; ++c) {
                    const long long* p = sk.ws + ((size_t)c * 2 + (small_unit(units, c, ctas) / KB == tile ? 0 : 1)) * kPlace + (size_t)m0 * kGemmBN + col;
                    long long v[16];   // (all requested before the first is added)
#pragma unroll
                    for (int i = 0; i < 16; ++i) v[i] = __ldcg(p + (size_t)i * kGemmBN);
#pragma unroll
                    for (int i = 0; i < 16; ++i) t[i] += v[i];
                }
                finish(t);
            }
        }
        tc_fence_before();
    }
    __syncthreads();
    if (warp == 8) {
        tc_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "n"(kSmallTmemCols) : "memory");
    }
}

}  // namespace tib
