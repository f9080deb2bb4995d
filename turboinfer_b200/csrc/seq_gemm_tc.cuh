// seq_gemm_tc.cuh -- bf16 x bf16 -> fp32 GEMM on the 5th-generation tensor cores for the prompt side of the layered sequence
// engine:  C[M, N] = epi(A[M, K] . W[N, K]^T), A = bf16 activations (row-major), W = bf16 weights as stored ([out, in]).
// Both operands are K-major, so both are fetched with plain 2-D TMA boxes (64 elements = 128 bytes a row, SWIZZLE_128B; rows and k
// beyond the tensor are zero-filled by the copy engine, so no operand is padded in memory).
//
// A pair of neighbouring SMs (cta_group::2) owns a tile of 256 rows x BN columns, BN a multiple of 32 from 64 to 256 chosen by
// pair_tile_columns(): each CTA loads its own 128 rows of A and HALF of the tile's weight rows, the even CTA issues one MMA (M 256) that
// reads both halves out of both shared memories, and each CTA holds its 128 rows of the result in its own TMEM.  An operand byte brought in
// from L2 serves twice the products it serves in a 128 x 128 tile of one CTA, whose 64 bytes a clock and SM were all that L2 gives.
// Clusters walk the tiles (rows fastest: neighbours share the weight tile in L2); two accumulators of up to 256 columns let the epilogue of a
// tile run under the main loop of the next.
//   warp 0   producer: TMA boxes of A (64 x 128) and W (64 x BN / 2), 6 stages of 32 KiB; both CTAs' copies complete on the even CTA's barrier
//   warp 1   TMEM allocation; even CTA: four MMAs of K 16 a stage; commits go to both CTAs
//   warps 2..5 epilogue: 32 x 32 blocks through a padded corner of shared memory, so that a store (and the read of C for EPI_ADD) covers
//            whole 128-byte lines instead of 16 bytes of 32 rows
// Measured (back-to-back launches on a B200, us, before = 128 x 128 tiles of one CTA with one-lane issue branches): 2048 x 2048 x 2048 28.4 -> 18.7,
// 2048 x 11264 x 2048 129 -> 74 (1.28 PFLOP/s), 1999 x 16896 x 4096 362 -> 204 (1.36 PFLOP/s, the 1000 W cap), 800 x 1024 x 1024 24.7 -> 12.0,
// 41 x 4096 x 4096 32.9 -> 16.5.  Large products are bound by the tensor cores at the power cap, small ones by set-up, the first copies
// and the last epilogue (about 8 us of the 12).
// Every wait is bounded: a wait that runs out sets *err and the roles fall through to the common exit (a cluster barrier, then TMEM is freed).
#pragma once
#include "gemm_tc.cuh"
#include "seq_kernels.cuh"

namespace tib {
namespace seq {

constexpr int kSgBM = 128, kSgBK = 64;                      // rows of a CTA; BK in bf16 elements (128 bytes)
constexpr int kSgTileBytes = kSgBM * kSgBK * 2;             // 16 KiB
constexpr int kSgStages = 6, kSgThreads = 192;
constexpr int kSgStageBytes = 2 * kSgTileBytes;
constexpr int kSgLd = 36;                                   // floats between rows of an epilogue block: 16-byte accesses without conflicts
constexpr int kSgEpiBytes = 32 * kSgLd * 4;                 // one block a warp
constexpr size_t kSgSmemBytes = (size_t)kSgStages * kSgStageBytes + 4 * kSgEpiBytes + 1024 /*align*/ + 256 /*barriers*/;

struct TcArgs {
    int M, N, K;
    float* C;
    int ldc;
    int epi;
    float alpha, beta;
    GluCols cols;   // cols.single with cols.ff > 0: columns cols.first .. N - 1 end as act(v) in cols.out instead of C
    int* err;   // set to 1 when a wait ran out
};

// D fp32, A and B bf16, both K-major
__host__ __device__ constexpr uint32_t umma_idesc_bf16(int m, int n) {
    return (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(n >> 3) << 17) | ((uint32_t)(m >> 4) << 24);
}

struct PairArgs {
    TcArgs t;
    int bn;          // columns of a tile
    int tiles_m, tiles;
};
// The tile width: waves of the pairs times what a k-step of that width costs, plus a wave's change of tile and the last epilogue (us;
// measured: a k-step takes 0.15 us at 64 columns, 0.18 at 128, 0.25 at 256).  A width that saves a wave wins over a wider one:
// 1530 x 2048 x 5632 in 66 tiles of 192 takes 35.0 us, in 48 of 256 43.2, in 96 of 128 45.2.
inline int pair_tile_columns(int M, int N, int K, int pairs) {
    int best = 256;
    float best_t = 1e30f;
    const int kb = (K + kSgBK - 1) / kSgBK, tm = (M + 255) / 256;
    for (int bn = 256; bn >= 64; bn -= 32) {
        const int waves = (tm * ((N + bn - 1) / bn) + pairs - 1) / pairs;
        const float t = waves * (kb * (0.12f + 0.0005f * bn) + 0.5f) + 0.01f * bn;
        if (t < best_t) { best_t = t; best = bn; }
    }
    return best;
}

__device__ __forceinline__ void tc_mma_bf16_pair(uint32_t tmem_d, uint64_t adesc, uint64_t bdesc, uint32_t idesc, uint32_t accumulate, uint32_t lead) {
    asm volatile(
        "{\n\t.reg .pred p, e;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "setp.ne.b32 e, %5, 0;\n\t"
        "@e tcgen05.mma.cta_group::2.kind::f16 [%0], %1, %2, %3, p;\n\t}"
        ::"r"(tmem_d), "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate), "r"(lead)
        : "memory");
}
// four neighbouring results of one row to where they belong: C through the epilogue, or the activated columns
__device__ __forceinline__ void pair_put4(const TcArgs& g, int row, int n, float4 v) {
    const GluCols& u = g.cols;
    if (u.ff > 0 && n + 4 > u.first) {
        if (n >= u.first && n + 4 <= g.N && u.out16) {
            __nv_bfloat16* h = u.out16 + (size_t)row * u.ld + (n - u.first);
            if ((reinterpret_cast<uintptr_t>(h) & 7) == 0) {
                const __nv_bfloat162 a = __floats2bfloat162_rn(ff_act(v.x, u.act), ff_act(v.y, u.act)), b = __floats2bfloat162_rn(ff_act(v.z, u.act), ff_act(v.w, u.act));
                *reinterpret_cast<uint2*>(h) = make_uint2(*reinterpret_cast<const uint32_t*>(&a), *reinterpret_cast<const uint32_t*>(&b));
                return;
            }
        } else if (n >= u.first && n + 4 <= g.N) {
            float* o = u.out + (size_t)row * u.ld + (n - u.first);
            if ((reinterpret_cast<uintptr_t>(o) & 15) == 0) {
                *reinterpret_cast<float4*>(o) = make_float4(ff_act(v.x, u.act), ff_act(v.y, u.act), ff_act(v.z, u.act), ff_act(v.w, u.act));
                return;
            }
        }
    } else if (n + 4 <= g.N && (g.ldc & 3) == 0 && (reinterpret_cast<uintptr_t>(g.C) & 15) == 0) {
        float4* cp = reinterpret_cast<float4*>(g.C + (size_t)row * g.ldc + n);
        if (g.epi == EPI_ADD) {
            const float4 c = *cp;
            *cp = make_float4(c.x + v.x, c.y + v.y, c.z + v.z, c.w + v.w);
        } else if (g.epi == EPI_NONE) {
            *cp = v;
        } else {
            *cp = make_float4(epi_apply(v.x, g.epi, g.alpha, g.beta), epi_apply(v.y, g.epi, g.alpha, g.beta), epi_apply(v.z, g.epi, g.alpha, g.beta),
                              epi_apply(v.w, g.epi, g.alpha, g.beta));
        }
        return;
    }
    const float e[4] = {v.x, v.y, v.z, v.w};   // edges, and columns on both sides of `first`
    for (int i = 0; i < 4 && n + i < g.N; ++i) {
        if (u.ff > 0 && n + i >= u.first) {
            const size_t at = (size_t)row * u.ld + (n + i - u.first);
            if (u.out16) u.out16[at] = __float2bfloat16_rn(ff_act(e[i], u.act));
            else u.out[at] = ff_act(e[i], u.act);
        } else {
            epi_put(g.C + (size_t)row * g.ldc + n + i, e[i], g.epi, g.alpha, g.beta);
        }
    }
}

__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(kSgThreads, 1)
gemm_bf16_tc_kernel(const __grid_constant__ CUtensorMap map_a, const __grid_constant__ CUtensorMap map_w, const PairArgs pg) {
    extern __shared__ uint8_t psm_raw[];
    const TcArgs& g = pg.t;
    const uint32_t base = (smem_u32(psm_raw) + 1023u) & ~1023u;
    uint8_t* tiles = psm_raw + (base - smem_u32(psm_raw));
    float* epi_smem = reinterpret_cast<float*>(tiles + (size_t)kSgStages * kSgStageBytes);
    uint64_t* full = reinterpret_cast<uint64_t*>(tiles + (size_t)kSgStages * kSgStageBytes + 4 * kSgEpiBytes);
    uint64_t* empty = full + kSgStages;
    uint64_t* acc_full = empty + kSgStages;    // [2]
    uint64_t* acc_empty = acc_full + 2;        // [2], the even CTA's: both CTAs' epilogue warps
    uint32_t* tmem_ptr = reinterpret_cast<uint32_t*>(acc_empty + 2);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const uint32_t rank = cluster_ctarank();
    const int pair = blockIdx.x >> 1, pairs = gridDim.x >> 1;
    const int KB = (g.K + kSgBK - 1) / kSgBK, bn = pg.bn;

    if (threadIdx.x == 0) {
        for (int i = 0; i < kSgStages; ++i) { mbar_init(&full[i], 1); mbar_init(&empty[i], 1); }
        for (int i = 0; i < 2; ++i) { mbar_init(&acc_full[i], 1); mbar_init(&acc_empty[i], 8); }
        fence_mbar_init();
    }
    if (warp == 1) {
        asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], 512;" ::"r"(smem_u32(tmem_ptr)) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
    }
    pdl_wait_prior_grid();   // (everything above touches only this CTA: it runs under the tail of the kernel before)
    tc_fence_before();
    __syncthreads();
    cluster_sync_all();   // the peer's barriers are initialised before anything is signalled across
    tc_fence_after();
    const uint32_t tmem = *tmem_ptr;

    if (warp == 0) {
        const uint32_t lead = elect_one();
        const uint32_t bytes = 2u * (uint32_t)(kSgTileBytes + (bn / 2) * kSgBK * 2);   // both CTAs' boxes (rows and k beyond the tensor arrive as zeros and count)
        const uint32_t full_s = smem_u32(full);
        bool ok = true;
        int st = 0, use = 0;
        for (int tile = pair; tile < pg.tiles && ok; tile += pairs) {
            const int mb = tile % pg.tiles_m, nb = tile / pg.tiles_m;
            const int row = mb * 256 + (int)rank * 128, col = nb * bn + (int)rank * (bn / 2);
            for (int kb = 0; kb < KB; ++kb) {
                if (use > 0 && !(ok = mbar_wait_bounded(&empty[st], (use - 1) & 1, g.err))) break;
                const uint32_t sbase = base + st * kSgStageBytes, bar = pair_leader(full_s + 8 * st);
                if (rank == 0) mbar_expect_tx_if(full_s + 8 * st, bytes, lead);
                tma_load_2d_pair(sbase, &map_a, kb * kSgBK, row, bar, lead);
                tma_load_2d_pair(sbase + kSgTileBytes, &map_w, kb * kSgBK, col, bar, lead);
                if (++st == kSgStages) { st = 0; ++use; }
            }
        }
        if (rank == 0) drain_copies(full, kSgStages, st, use, g.err);
    } else if (warp == 1) {
        if (rank == 0) {
            const uint32_t lead = elect_one();
            const uint32_t idesc = umma_idesc_bf16(256, bn);
            const uint64_t desc0 = umma_desc_sw128(base);   // (addresses stay below 2^18: adding to the address field never carries out of it)
            const uint32_t empty_s = smem_u32(empty), accf_s = smem_u32(acc_full);
            bool ok = true;
            int st = 0, use = 0, n_tile = 0;
            for (int tile = pair; tile < pg.tiles && ok; tile += pairs, ++n_tile) {
                const int buf = n_tile & 1, use_t = n_tile >> 1;
                if (use_t > 0) ok = mbar_wait_bounded(&acc_empty[buf], (use_t - 1) & 1, g.err);
                tc_fence_after();
                for (int kb = 0; kb < KB && ok; ++kb) {
                    ok = mbar_wait_bounded(&full[st], use & 1, g.err);
                    if (!ok) break;
                    tc_fence_after();
                    const uint64_t ad = desc0 + (uint64_t)(st * (kSgStageBytes >> 4)), bd = ad + (kSgTileBytes >> 4);
#pragma unroll
                    for (int k4 = 0; k4 < kSgBK / 16; ++k4)
                        tc_mma_bf16_pair(tmem + buf * 256, ad + 2 * k4, bd + 2 * k4, idesc, (kb | k4) != 0 ? 1u : 0u, lead);
                    tc_commit_pair(empty_s + 8 * st, lead);
                    if (++st == kSgStages) { st = 0; ++use; }
                }
                tc_commit_pair(accf_s + 8 * buf, lead);   // also on the failure path: the epilogue warps must not wait for ever
            }
        }
    } else {
        const int q = warp & 3;
        float* blk = epi_smem + (warp - 2) * (kSgEpiBytes / 4);
        const bool plain_cols = (g.epi == EPI_NONE || g.epi == EPI_ADD) && (g.ldc & 3) == 0 && (reinterpret_cast<uintptr_t>(g.C) & 15) == 0;
        bool ok = true;
        int n_tile = 0;
        for (int tile = pair; tile < pg.tiles && ok; tile += pairs, ++n_tile) {
            const int buf = n_tile & 1, use_t = n_tile >> 1;
            ok = mbar_wait_bounded(&acc_full[buf], use_t & 1, g.err);
            ok = __all_sync(0xffffffffu, ok && *reinterpret_cast<volatile int*>(g.err) == 0);
            if (!ok) break;
            tc_fence_after();
            const int mb = tile % pg.tiles_m, nb = tile / pg.tiles_m;
            const int row0 = mb * 256 + (int)rank * 128 + q * 32;
            for (int c0 = 0; c0 < bn && nb * bn + c0 < g.N; c0 += 32) {
                uint32_t a[32];
                tmem_ld32(a, tmem + ((uint32_t)(q * 32) << 16) + (uint32_t)(buf * 256 + c0));
#pragma unroll
                for (int i = 0; i < 32; i += 4)
                    *reinterpret_cast<uint4*>(blk + lane * kSgLd + i) = make_uint4(a[i], a[i + 1], a[i + 2], a[i + 3]);
                __syncwarp();
                const int n = nb * bn + c0 + 4 * (lane & 7), row = row0 + (lane >> 3);
                float4 v[8];
#pragma unroll
                for (int r = 0; r < 8; ++r) v[r] = *reinterpret_cast<const float4*>(blk + (4 * r + (lane >> 3)) * kSgLd + 4 * (lane & 7));
                __syncwarp();
                if (plain_cols && (g.cols.ff == 0 || nb * bn + c0 + 32 <= g.cols.first) && nb * bn + c0 + 32 <= g.N) {   // whole 16-byte groups of C
                    float* cp = g.C + (size_t)row * g.ldc + n;
                    if (g.epi == EPI_ADD) {
#pragma unroll
                        for (int h = 0; h < 8; h += 4) {
                            float4 c[4];
#pragma unroll
                            for (int r = 0; r < 4; ++r) c[r] = row + 4 * (h + r) < g.M ? *reinterpret_cast<const float4*>(cp + (size_t)(4 * (h + r)) * g.ldc) : make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
                            for (int r = 0; r < 4; ++r)
                                if (row + 4 * (h + r) < g.M)
                                    *reinterpret_cast<float4*>(cp + (size_t)(4 * (h + r)) * g.ldc) = make_float4(c[r].x + v[h + r].x, c[r].y + v[h + r].y, c[r].z + v[h + r].z, c[r].w + v[h + r].w);
                        }
                    } else {
#pragma unroll
                        for (int r = 0; r < 8; ++r)
                            if (row + 4 * r < g.M) *reinterpret_cast<float4*>(cp + (size_t)(4 * r) * g.ldc) = v[r];
                    }
                } else {
#pragma unroll 1
                    for (int r = 0; r < 8; ++r) {
                        const float4 w = *reinterpret_cast<const float4*>(blk + (4 * r + (lane >> 3)) * kSgLd + 4 * (lane & 7));
                        if (row + 4 * r < g.M && n < g.N) pair_put4(g, row + 4 * r, n, w);
                    }
                    __syncwarp();
                }
            }
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive_cluster(pair_leader(smem_u32(&acc_empty[buf])));
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


}  // namespace seq
}  // namespace tib
