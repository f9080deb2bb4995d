// attn_tc.cuh -- softmax attention of prompt rows on the 5th-generation tensor cores from split 16-bit operands, shared by the prefill of the
// quantized decoder and the prompt portions of the layered sequence engine.
//
// Every fp32 operand is split into two fp16 halves, x = hi + lo (hi = fp16(x), lo = fp16(x - hi)): 22 mantissa bits from magnitudes of about 2^-3 up, below
// them an absolute error of about 2^-25 (the low half meets fp16's smallest step), infinite above 65504.  Rows that must not lose range or
// bits against the decode kernels do not come here (capi.cu prefill_gemm).  Each product is
// lo hi + hi lo + hi hi with fp32 accumulation, the arithmetic of the warp-level kernels in prefill.cuh / seq_attn_tc.cuh that this replaces
// for head sizes of 64 and 128 (and smaller ones padded with zeros).  Scores, softmax and the running output stay fp32.
//
// Keys and values are split ONCE a layer by kv_images_kernel into tile images of 64 keys (the 16 query tiles of a 2048-token prompt used to
// repeat that work): one record per (key tile, key/value head), [K hi | K lo | V hi | V lo], each a row of 128-byte blocks of 64 coordinates
// with the 128-byte swizzle, so that a tile is two bulk copies.  K is read K-major (coordinates), V by the same image MN-major (the
// k index of P V is the key).
//
// attn_tc_kernel: a CTA owns up to 128 query rows of one sequence and one head.
//   warps 0, 2   producers: bulk copies of the key and the value halves of a tile into two stages each
//   warp 1       tcgen05.mma: S(i + 1) = Q K^T is issued before P(i) V, so that the scores of the next tile are made while the softmax of
//                this one runs; S and the tile outputs P V have two TMEM buffers each (2 x 64 + 2 x DV columns)
//   warps 4..11  softmax, two threads a row with 32 keys each (they exchange their maxima through shared memory): scores from TMEM, masks, running
//                maximum, expf, halves of P to shared memory
//   warps 12..15 running output in registers, one thread a row: o = o * factor(i) + (P V)(i); then the finish (denominator, gates) and
//                stores of whole 128-byte lines; they take the registers that the others give back (80 + 112 + 112 + 208 = 4 x 128)
// What bounds it: a tile of 64 keys takes about 2450 clocks against 1920 for its 36 MMAs (the scores' operand reads limit them); the rest is the chain
// copy -> scores -> softmax -> P V -> output where neighbouring tiles do not cover one another, and each block has about 6400 clocks of set-up and
// 4200 of finish.  Measured, a layer of 2048 tokens x 32 heads of 128: 664 us with warp-level MMAs, 145 with one softmax thread a row (four
// warps), about 130 now.
// Waits are bounded; a wait that runs out sets *err and nothing is stored.
#pragma once
#include <cuda_fp16.h>

#include "gemm_tc.cuh"

namespace tib {

constexpr int kAtQ = 128, kAtKT = 64, kAtHalf = kAtKT / 2, kAtThreads = 512;
__host__ __device__ constexpr int at_pad(int d) { return d <= 64 ? 64 : 128; }
__host__ __device__ constexpr size_t at_record_bytes(int dk, int dv) { return (size_t)kAtKT * (dk + dv) * 4; }   // hi and lo of 64 rows
template <int DK, int DV> constexpr size_t attn_tc_smem_bytes5() {
    return (size_t)kAtQ * DK * 4 + 2 * at_record_bytes(DK, DV) + (size_t)kAtQ * kAtKT * 4 + 5 * kAtQ * sizeof(float) + 256;
}

__device__ __forceinline__ void split_half(float x, float y, uint32_t& hi, uint32_t& lo) {   // two neighbours, packed
    const __half2 h = __floats2half2_rn(x, y);
    const float2 f = __half22float2(h);
    const __half2 l = __floats2half2_rn(x - f.x, y - f.y);
    hi = *reinterpret_cast<const uint32_t*>(&h);
    lo = *reinterpret_cast<const uint32_t*>(&l);
}
// byte offset of coordinate d (in eights) of row r inside an image of `rows` rows: blocks of 64 coordinates, 128 bytes a row, swizzled
__device__ __forceinline__ uint32_t at_offset(int rows, int r, int d) {
    return (uint32_t)((d >> 6) * rows * 128 + r * 128 + ((((d >> 3) & 7) ^ (r & 7)) << 4));
}

// A source of keys and values: where key t of the sequence of key tile `kt` lies.  grid (key tiles, key/value heads), 256 threads
template <int DK, int DV, typename Src>
__global__ void __launch_bounds__(256) kv_images_kernel(const Src src, uint8_t* images) {
    const int g = src.g0 + blockIdx.y;
    typename Src::Tile tile;
    src.tile(blockIdx.x, tile);
    uint8_t* rec = images + ((size_t)blockIdx.x * gridDim.y + blockIdx.y) * at_record_bytes(DK, DV);
    // a thread takes eight coordinates of a key: two 16-byte loads, one 16-byte store into each half
    for (int i = threadIdx.x; i < kAtKT * (DK + DV) / 8; i += 256) {
        const int r = i / ((DK + DV) / 8), c = (i % ((DK + DV) / 8)) * 8;
        const bool is_v = c >= DK;
        const int d = is_v ? c - DK : c, size = is_v ? src.dv : src.d;
        float x[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
        const float* row = src.row(tile, r, g, is_v);
        if (row) {   // (sizes are multiples of four)
            if (d < size) *reinterpret_cast<float4*>(x) = *reinterpret_cast<const float4*>(row + d);
            if (d + 4 < size) *reinterpret_cast<float4*>(x + 4) = *reinterpret_cast<const float4*>(row + d + 4);
        }
        uint4 hi, lo;
        split_half(x[0], x[1], hi.x, lo.x);
        split_half(x[2], x[3], hi.y, lo.y);
        split_half(x[4], x[5], hi.z, lo.z);
        split_half(x[6], x[7], hi.w, lo.w);
        uint8_t* im = rec + (is_v ? (size_t)kAtKT * DK * 4 : 0) + at_offset(kAtKT, r, d);
        *reinterpret_cast<uint4*>(im) = hi;
        *reinterpret_cast<uint4*>(im + (size_t)kAtKT * (is_v ? DV : DK) * 2) = lo;
    }
}

// D fp32, A and B fp16; b_mn: B is MN-major
__host__ __device__ constexpr uint32_t umma_idesc_f16(int m, int n, int b_mn) {
    return (1u << 4) | ((uint32_t)b_mn << 16) | ((uint32_t)(n >> 3) << 17) | ((uint32_t)(m >> 4) << 24);
}
__device__ __forceinline__ void tc_mma_f16_if(uint32_t tmem_d, uint64_t adesc, uint64_t bdesc, uint32_t idesc, uint32_t accumulate, uint32_t lead) {
    asm volatile(
        "{\n\t.reg .pred p, e;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "setp.ne.b32 e, %5, 0;\n\t"
        "@e tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}"
        ::"r"(tmem_d), "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate), "r"(lead)
        : "memory");
}
// Shape: tile(y, row0, count, pos0, image0) -- the rows of the block, the position of the first, the record of the sequence's key tile 0;
// d, dv (multiples of four), h0 (first query head of the launch), group (query heads a key/value head); q(row, h); first_key(pos), never
// later for an earlier row; scores(): scales (and caps) 32 raw products; sigmoid(): weights sigmoid_weight(score, pb(h)) instead of a softmax;
// finish(row, h, m, l): factor on the output; store4(row, h, c, v)
template <int DK, int DV, typename Shape>
__global__ void __launch_bounds__(kAtThreads, 1) attn_tc_kernel(const Shape s, const uint8_t* images, int* err) {
    extern __shared__ __align__(1024) uint8_t at_smem[];
    constexpr uint32_t kQ = kAtQ * DK * 2;                       // one half of the query image
    constexpr uint32_t kK = kAtKT * DK * 2, kV = kAtKT * DV * 2; // one half of a key / value tile
    uint8_t* Q = at_smem;                                        // [hi | lo]
    uint8_t* Ks = Q + 2 * kQ;                                    // [2 stages][hi | lo]
    uint8_t* Vs = Ks + 4 * kK;
    uint8_t* P = Vs + 4 * kV;                                    // [hi | lo], 128 rows of 64 keys
    float* factor = reinterpret_cast<float*>(P + kAtQ * kAtKT * 4);   // [3][128]: what the running output is multiplied by in front of tile i
    float* pmax = factor + 3 * kAtQ;                             // [2][128]: the maxima of the two halves of a row's keys
    uint64_t* bars = reinterpret_cast<uint64_t*>(pmax + 2 * kAtQ);
    uint64_t *k_full = bars, *k_empty = bars + 2, *v_full = bars + 4, *v_empty = bars + 6, *s_full = bars + 8, *s_empty = bars + 10, *o_full = bars + 12,
             *o_empty = bars + 14, *p_full = bars + 16, *p_empty = bars + 17, *fin_full = bars + 18;
    uint32_t* tmem_ptr = reinterpret_cast<uint32_t*>(bars + 19);
    // behind the last tile the key stages hold what the rows end with, and the blocks of the store
    float* fin = reinterpret_cast<float*>(Ks);                   // [m: 128][l of either half: 2 x 128]
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int h = s.h0 + blockIdx.x;
    int row0, M, pos0, image0;
    s.tile(blockIdx.y, row0, M, pos0, image0);
    const int last_pos = pos0 + M - 1, first = s.first_key(pos0) / kAtKT, n_tiles = last_pos / kAtKT - first + 1;

    const int groups = gridDim.x / s.group;   // (the launch covers whole key/value heads from h0 on)
    const uint8_t* rec0 = images + ((size_t)(image0 + first) * groups + blockIdx.x / s.group) * at_record_bytes(DK, DV);
    const size_t step = (size_t)groups * at_record_bytes(DK, DV);
    const uint32_t lead = elect_one();

    if (warp == 0) {
        if (lead) {
        for (int i = 0; i < 2; ++i) {
            mbar_init(&k_full[i], 1); mbar_init(&k_empty[i], 1); mbar_init(&v_full[i], 1); mbar_init(&v_empty[i], 1);
            mbar_init(&s_full[i], 1); mbar_init(&s_empty[i], 8); mbar_init(&o_full[i], 1); mbar_init(&o_empty[i], 4);
        }
        mbar_init(p_full, 8); mbar_init(p_empty, 1); mbar_init(fin_full, 8);
        fence_mbar_init();
        if (smem_u32(at_smem) & 1023u) *reinterpret_cast<volatile int*>(err) = 1;   // (the swizzle needs 1024-byte blocks)
        }
        __syncwarp();
        // the first two key and value tiles are on their way while the query tile is split
        for (int i = 0; i < 2 && i < n_tiles; ++i) {
            mbar_expect_tx_if(smem_u32(&k_full[i]), 2 * kK, lead);
            bulk_g2s_if(smem_u32(Ks) + i * 2 * kK, rec0 + i * step, 2 * kK, smem_u32(&k_full[i]), lead);
            mbar_expect_tx_if(smem_u32(&v_full[i]), 2 * kV, lead);
            bulk_g2s_if(smem_u32(Vs) + i * 2 * kV, rec0 + i * step + 2 * kK, 2 * kV, smem_u32(&v_full[i]), lead);
        }
    }
    if (warp == 1) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], 512;" ::"r"(smem_u32(tmem_ptr)) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    // the query tile's halves, a thread's loads all in flight together
    constexpr int kQVecs = kAtQ * DK / 8 / kAtThreads;
    float x[kQVecs][8];
#pragma unroll
    for (int i = 0; i < kQVecs; ++i) {
        const int c = threadIdx.x + i * kAtThreads, r = c / (DK / 8), d = (c % (DK / 8)) * 8;
#pragma unroll
        for (int e = 0; e < 8; ++e) x[i][e] = 0.f;
        if (r < M) {
            const float* q = s.q(row0 + r, h) + d;   // (the row pitch need not be a multiple of 4)
            if ((reinterpret_cast<uintptr_t>(q) & 15) == 0) {
                if (d < s.d) *reinterpret_cast<float4*>(x[i]) = *reinterpret_cast<const float4*>(q);
                if (d + 4 < s.d) *reinterpret_cast<float4*>(x[i] + 4) = *reinterpret_cast<const float4*>(q + 4);
            } else {
#pragma unroll
                for (int e = 0; e < 8; ++e)
                    if (d + e < s.d) x[i][e] = q[e];
            }
        }
    }
#pragma unroll
    for (int i = 0; i < kQVecs; ++i) {
        const int c = threadIdx.x + i * kAtThreads, r = c / (DK / 8), d = (c % (DK / 8)) * 8;
        uint4 hi, lo;
        split_half(x[i][0], x[i][1], hi.x, lo.x);
        split_half(x[i][2], x[i][3], hi.y, lo.y);
        split_half(x[i][4], x[i][5], hi.z, lo.z);
        split_half(x[i][6], x[i][7], hi.w, lo.w);
        const uint32_t at = at_offset(kAtQ, r, d);
        *reinterpret_cast<uint4*>(Q + at) = hi;
        *reinterpret_cast<uint4*>(Q + kQ + at) = lo;
    }
    fence_proxy_async();
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = *tmem_ptr;
    constexpr uint32_t kSCol = 0, kOCol = 2 * kAtKT;             // TMEM columns: two score buffers, two output buffers

    // (the registers move inside the roles' own branches: the compiler allots each branch by it)
    if (warp == 0 || warp == 2) {   // keys, values
        reg_dealloc<80>();
        const bool is_v = warp == 2;
        const uint32_t bytes = 2 * (is_v ? kV : kK), full = smem_u32(is_v ? v_full : k_full), dst = smem_u32(is_v ? Vs : Ks);
        uint64_t* empty = is_v ? v_empty : k_empty;
        const uint8_t* src = rec0 + (is_v ? 2 * kK : 0) + 2 * step;
        int i = min(2, n_tiles);   // (the first two tiles were asked for in front of the query tile)
        for (; i < n_tiles; ++i, src += step) {
            const int st = i & 1;
            if (!mbar_wait_bounded(&empty[st], ((i >> 1) - 1) & 1, err)) break;
            mbar_expect_tx_if(full + 8 * st, bytes, lead);
            bulk_g2s_if(dst + st * bytes, src, bytes, full + 8 * st, lead);
        }
        drain_copies(is_v ? v_full : k_full, 2, i & 1, i >> 1, err);
    } else if (warp == 1) {
        reg_dealloc<80>();
        constexpr uint32_t id_s = umma_idesc_f16(kAtQ, kAtKT, 0), id_o = umma_idesc_f16(kAtQ, DV, 1);
        const uint64_t qd = umma_desc_sw128(smem_u32(Q)), kd0 = umma_desc_sw128(smem_u32(Ks)), pd = umma_desc_sw128(smem_u32(P));
        // values, MN-major: 64 coordinates a block (leading offset: the next block), 8 keys apart 1024 bytes
        const uint64_t vd0 = (umma_desc_sw128(smem_u32(Vs)) & ~((uint64_t)0x3FFF << 16)) | ((uint64_t)(kAtKT * 128 >> 4) << 16);
        bool ok = true;
        auto scores = [&](int i) {   // S(i): small products first
            const int b = i & 1, use = i >> 1;
            if (ok) ok = mbar_wait_bounded(&k_full[b], use & 1, err);
            if (ok && use > 0) ok = mbar_wait_bounded(&s_empty[b], (use - 1) & 1, err);
            if (!ok) return;
            tc_fence_after();
            const uint64_t kd = kd0 + (uint64_t)(b * (2 * kK >> 4));
#pragma unroll
            for (int p = 0; p < 3; ++p) {
                const uint64_t a = qd + (p == 0 ? (uint64_t)(kQ >> 4) : 0), k = kd + (p == 1 ? (uint64_t)(kK >> 4) : 0);
#pragma unroll
                for (int ks = 0; ks < DK / 16; ++ks)
                    tc_mma_f16_if(tmem + kSCol + b * kAtKT, a + (ks >> 2) * (kAtQ * 128 >> 4) + (ks & 3) * 2, k + (ks >> 2) * (kAtKT * 128 >> 4) + (ks & 3) * 2, id_s,
                                  (p | ks) != 0 ? 1u : 0u, lead);
            }
            tc_commit_if(smem_u32(&k_empty[b]), lead);
            tc_commit_if(smem_u32(&s_full[b]), lead);
        };
        scores(0);
        for (int i = 0; i < n_tiles && ok; ++i) {
            if (i + 1 < n_tiles) scores(i + 1);
            const int b = i & 1, use = i >> 1;
            if (ok) ok = mbar_wait_bounded(&v_full[b], use & 1, err);
            if (ok) ok = mbar_wait_bounded(p_full, i & 1, err);
            if (ok && use > 0) ok = mbar_wait_bounded(&o_empty[b], (use - 1) & 1, err);
            if (!ok) break;
            tc_fence_after();
            const uint64_t vd = vd0 + (uint64_t)(b * (2 * kV >> 4));
#pragma unroll
            for (int p = 0; p < 3; ++p) {
                const uint64_t a = pd + (p == 0 ? (uint64_t)(kAtQ * kAtKT * 2 >> 4) : 0), v = vd + (p == 1 ? (uint64_t)(kV >> 4) : 0);
#pragma unroll
                for (int ks = 0; ks < kAtKT / 16; ++ks)
                    tc_mma_f16_if(tmem + kOCol + b * DV, a + ks * 2, v + ks * (16 * 128 >> 4), id_o, (p | ks) != 0 ? 1u : 0u, lead);
            }
            tc_commit_if(smem_u32(p_empty), lead);
            tc_commit_if(smem_u32(&v_empty[b]), lead);
            tc_commit_if(smem_u32(&o_full[b]), lead);
        }
    } else if (warp == 3) {
        reg_dealloc<80>();
    } else if (warp < 12) {
        reg_dealloc<112>();
        const int q = warp & 3, r = q * 32 + lane, half = (warp - 4) >> 2, k0 = half * kAtHalf;   // TMEM lane = row of the tile
        const int qp = r < M ? pos0 + r : -1, lo = r < M ? s.first_key(pos0 + r) : 0;
        const int all_hi = M == kAtQ ? pos0 : -1, all_lo = s.first_key(last_pos);   // keys in [all_lo, all_hi] are visible to every row of the tile
        const float pb = s.sigmoid() ? s.pb(h) : 0.f;
        float m = -INFINITY, l = 0.f;
        bool ok = true;
        // (after a failed wait the loop goes on without waiting: the two warps of a row meet at the same barriers to the end)
        for (int i = 0, slot = 0; i < n_tiles; ++i, slot = slot == 2 ? 0 : slot + 1) {
            const int b = i & 1, use = i >> 1;
            if (ok) ok = mbar_wait_bounded(&s_full[b], use & 1, err);
            ok = __all_sync(0xffffffffu, ok);
            tc_fence_after();
            uint32_t raw[kAtHalf];
            tmem_ld32(raw, tmem + ((uint32_t)(q * 32) << 16) + kSCol + b * kAtKT + k0);
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(&s_empty[b]);
            float sc[kAtHalf];
#pragma unroll
            for (int j = 0; j < kAtHalf; ++j) sc[j] = __uint_as_float(raw[j]);
            s.scores(sc);
            const int t0 = (first + i) * kAtKT;
            if (!(t0 >= all_lo && t0 + kAtKT - 1 <= all_hi)) {
#pragma unroll
                for (int j = 0; j < kAtHalf; ++j) sc[j] = (t0 + k0 + j <= qp && t0 + k0 + j >= lo) ? sc[j] : -INFINITY;
            }
            float f = 1.f;
            if (s.sigmoid()) {   // no softmax: a visible key's weight is sigmoid(score + pb)
#pragma unroll
                for (int j = 0; j < kAtHalf; ++j) sc[j] = sc[j] == -INFINITY ? 0.f : s.sigmoid_weight(sc[j], pb);
            } else {
                float mx[4] = {sc[0], sc[1], sc[2], sc[3]};
#pragma unroll
                for (int j = 4; j < kAtHalf; ++j) mx[j & 3] = fmaxf(mx[j & 3], sc[j]);
                const float mine = fmaxf(fmaxf(mx[0], mx[1]), fmaxf(mx[2], mx[3]));
                pmax[half * kAtQ + r] = mine;
                bar_sync(2 + q, 64);
                const float mn = fmaxf(m, fmaxf(mine, pmax[(half ^ 1) * kAtQ + r]));
                bar_sync(2 + q, 64);   // (both have read: the place is free for the next tile)
                const float base = mn == -INFINITY ? 0.f : mn;   // (nothing visible so far: exp(-inf) = 0 everywhere)
                float sum[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
                for (int j = 0; j < kAtHalf; ++j) {
                    sc[j] = expf(sc[j] - base);   // (in base 2 with a rounded maximum, neighbouring tiles of large scores would not agree on it)
                    sum[j & 3] += sc[j];
                }
                f = mn == -INFINITY ? 1.f : expf(m - mn);
                l = l * f + ((sum[0] + sum[1]) + (sum[2] + sum[3]));
                m = mn;
            }
            if (ok && i > 0) ok = mbar_wait_bounded(p_empty, (i - 1) & 1, err);   // the previous tile's P V has read the halves
            ok = __all_sync(0xffffffffu, ok);
#pragma unroll
            for (int c = 0; c < kAtHalf / 8; ++c) {
                uint4 hi, lo4;
                split_half(sc[8 * c], sc[8 * c + 1], hi.x, lo4.x);
                split_half(sc[8 * c + 2], sc[8 * c + 3], hi.y, lo4.y);
                split_half(sc[8 * c + 4], sc[8 * c + 5], hi.z, lo4.z);
                split_half(sc[8 * c + 6], sc[8 * c + 7], hi.w, lo4.w);
                const uint32_t at = at_offset(kAtQ, r, k0 + 8 * c);
                *reinterpret_cast<uint4*>(P + at) = hi;
                *reinterpret_cast<uint4*>(P + kAtQ * kAtKT * 2 + at) = lo4;
            }
            if (half == 0) factor[slot * kAtQ + r] = f;   // (three slots: the output warps are at most two tiles behind)
            fence_proxy_async();
            __syncwarp();
            if (lane == 0) mbar_arrive(p_full);
        }
        if (ok) {   // (every S has been made: the key stages are free)
            if (half == 0) fin[r] = m;
            fin[(1 + half) * kAtQ + r] = l;
            __syncwarp();
            if (lane == 0) mbar_arrive(fin_full);
        }
    } else {
        reg_alloc<208>();
        const int q = warp & 3, r = q * 32 + lane;
        const int qp = r < M ? pos0 + r : -1, lo = r < M ? s.first_key(pos0 + r) : 0;
        float o[DV];
#pragma unroll
        for (int c = 0; c < DV; ++c) o[c] = 0.f;
        bool ok = true;
        for (int i = 0, slot = 0; i < n_tiles; ++i, slot = slot == 2 ? 0 : slot + 1) {
            const int b = i & 1, use = i >> 1;
            ok = mbar_wait_bounded(&o_full[b], use & 1, err);
            ok = __all_sync(0xffffffffu, ok);
            if (!ok) break;
            tc_fence_after();
            const float f = factor[slot * kAtQ + r];
            // (a tile without a key the row sees is left out, not added as zeros: its values may be infinite, and zero times infinity is not zero)
            const int t0 = (first + i) * kAtKT;
            const bool seen = t0 <= qp && t0 + kAtKT > lo;
#pragma unroll
            for (int c = 0; c < DV; c += 32) {
                uint32_t v[32];
                tmem_ld32(v, tmem + ((uint32_t)(q * 32) << 16) + kOCol + b * DV + c);
                if (seen) {
#pragma unroll
                    for (int e = 0; e < 32; ++e) o[c + e] = fmaf(o[c + e], f, __uint_as_float(v[e]));
                }
            }
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(&o_empty[b]);
        }
        if (ok) ok = mbar_wait_bounded(fin_full, 0, err);
        ok = __all_sync(0xffffffffu, ok);
        if (ok) {
            const float fac = r < M ? s.finish(row0 + r, h, fin[r], fin[kAtQ + r] + fin[2 * kAtQ + r]) : 0.f;
            float* blk = reinterpret_cast<float*>(Ks + 2048) + (warp - 12) * (32 * 36);
            const int rr = lane >> 3, cc = 4 * (lane & 7);
#pragma unroll
            for (int c = 0; c < DV; c += 32) {
                if (c < s.dv) {
#pragma unroll
                    for (int e = 0; e < 32; e += 4)
                        *reinterpret_cast<float4*>(blk + lane * 36 + e) = make_float4(o[c + e] * fac, o[c + e + 1] * fac, o[c + e + 2] * fac, o[c + e + 3] * fac);
                    __syncwarp();
                    float4 v[8];
#pragma unroll
                    for (int e = 0; e < 8; ++e) v[e] = *reinterpret_cast<const float4*>(blk + (4 * e + rr) * 36 + cc);
                    __syncwarp();
                    if (c + cc < s.dv) {   // (sizes in fours)
#pragma unroll
                        for (int e = 0; e < 8; ++e) {
                            const int row = q * 32 + 4 * e + rr;
                            if (row < M) s.store4(row0 + row, h, c + cc, v[e]);
                        }
                    }
                }
            }
        }
        tc_fence_before();
    }
    __syncthreads();
    if (warp == 1) {
        tc_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, 512;" ::"r"(tmem) : "memory");
    }
}

// key/value heads of a launch: their images fit `budget` bytes (at least one head)
inline int at_heads_per_launch(int kv_heads, size_t key_tiles, int dk, int dv, size_t budget) {
    const size_t one = std::max<size_t>(1, key_tiles * at_record_bytes(dk, dv));
    return (int)std::max<size_t>(1, std::min<size_t>(kv_heads, budget / one));
}
constexpr size_t kAtImageBudget = (size_t)256 << 20;
// ... and the buffer that holds them, a power of two of bytes while that is within the budget: contexts that grow by a page a step must not ask for a new one
// each time.  One that cannot be had is asked for in halves, down to one head (0: no room for that either).  `refused`: the smallest size that
// was not to be had in this pass over the layers, which is not asked for again
template <typename Buf>
int at_heads_with_room(Buf& images, int kv_heads, size_t key_tiles, int dk, int dv, size_t& refused) {
    const size_t one = key_tiles * at_record_bytes(dk, dv);
    for (int per = at_heads_per_launch(kv_heads, key_tiles, dk, dv, kAtImageBudget);; per = (per + 1) / 2) {
        if (images.n >= per * one) return per;
        size_t whole = 1;
        while (whole < per * one) whole *= 2;
        for (size_t size : {whole, per * one}) {
            if (size >= refused || (size == whole && whole > kAtImageBudget)) continue;
            if (images.alloc(size) == 0) return per;
            refused = size;
        }
        if (per == 1) return 0;
    }
}

}  // namespace tib
