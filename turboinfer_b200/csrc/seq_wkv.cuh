// seq_wkv.cuh -- the token-shifted linear recurrence ("wkv") of prompt portions in chunks of 16 tokens.
//
//   o_t = (S_{t-1} + diag(u) k_t v_t^T)^T r_t,   S_t = diag(w_t) S_{t-1} + k_t v_t^T,   w = exp(-exp(z + w0)) in (0, 1) per channel
//
// Inside a chunk (t, s = 0 .. 15, S the state in front of it, D(s, t) = w_{s+1} .. w_{t-1} per channel):
//   o_t = (r_t w_0 .. w_{t-1})^T S + sum_{s <= t} M[t][s] v_s,     M[t][s] = sum_c r_t k_s D(s, t) for s < t,  sum_c r_t u k_t for s = t
//   S  <- diag(w_0 .. w_15) S + sum_s (k_s w_{s+1} .. w_15) v_s^T
// so that only two small products a chunk wait for one another instead of 16 tokens.  The decays are multiplied up step by step, as the
// token-by-token form does (quotients of running products, or differences of summed logarithms, would lose what strong decays leave behind): every
// factor is at most one and nothing is divided.
//   wkv_chunk_prepare_kernel   all chunks and heads at once: M, the chunk's whole decay, and r and k with their decays, in place
//   wkv_chunk_scan_kernel      a block walks the chunks of one sequence, one head and 16 value columns
// Measured, 2048 tokens and 32 heads of 64, us: wkv_scan_split_kernel 256 (token by token, shared-memory latency on 64 blocks); here 37 + 133, the
// preparation three times its memory traffic's time, the walk bound by the latency between its two barriers a chunk (eight warps an SM).
#pragma once
#include "seq_kernels.cuh"

namespace tib {
namespace seq {

constexpr int kWkvChunk = 16, kWkvCols = 16;
// rows of a portion from which the chunked form is taken (a step through two layers of 2048, us, in chunks | token by token: 48 rows 234 | 230, 64 rows
// 236 | 236, 96 rows 244 | 245, 128 rows 251 | 255, 256 rows 279 | 296)
constexpr int kWkvChunkedMinRows = 64;

struct WkvChunkArgs {
    WkvArgs w;        // w.r and w.k are rewritten by the preparation
    float* M;         // [chunks][heads][16][16]
    float* decay;     // [chunks][heads][d]
};
// chunk number b of the step -> its entry, first row and rows
__device__ __forceinline__ void wkv_chunk_rows(const StepMeta& m, int b, int& row0, int& rows) {
    for (int e = 0; e < m.E; ++e) {
        const int r0 = m.ent_row0[e], n = m.ent_row0[e + 1] - r0, nc = (n + kWkvChunk - 1) / kWkvChunk;
        if (b < nc) {
            row0 = r0 + b * kWkvChunk;
            rows = min(kWkvChunk, n - b * kWkvChunk);
            return;
        }
        b -= nc;
    }
    row0 = rows = 0;
}

// grid (chunks, heads), 4 D threads: thread (s, channels 4 c ..) carries key s through the tokens behind it
template <int D>
__global__ void __launch_bounds__(4 * D) wkv_chunk_prepare_kernel(WkvChunkArgs a, StepMeta m) {
    // (no early start for the walk behind this: its few long blocks would crowd on the SMs that empty first, 400 us a prompt)
    pdl_wait_prior_grid();
    constexpr int G = D / 4;   // threads a token
    __shared__ __align__(16) float r[kWkvChunk][D], w[kWkvChunk][D];
    const int hd = blockIdx.y, s = threadIdx.x / G, c = 4 * (threadIdx.x % G);
    int row0, rows;
    wkv_chunk_rows(m, blockIdx.x, row0, rows);
    if (rows == 0) return;
    const size_t C = (size_t)a.w.heads * D, at = (size_t)(row0 + min(s, rows - 1)) * C + (size_t)hd * D + c;
    const float4 zero = make_float4(0.f, 0.f, 0.f, 0.f);
    const float4 r4 = s < rows ? *reinterpret_cast<const float4*>(a.w.r + at) : zero;
    float4 k4 = s < rows ? *reinterpret_cast<const float4*>(a.w.k + at) : zero;
    const float4 z4 = *reinterpret_cast<const float4*>(a.w.z + at);
    const float *w0 = a.w.w0 + hd * D + c, *u = a.w.u + hd * D + c;
    const float4 one = make_float4(1.f, 1.f, 1.f, 1.f);
    const float4 w4 = s < rows ? make_float4(expf(-expf(z4.x + w0[0])), expf(-expf(z4.y + w0[1])), expf(-expf(z4.z + w0[2])), expf(-expf(z4.w + w0[3]))) : one;
    *reinterpret_cast<float4*>(&r[s][c]) = r4;
    *reinterpret_cast<float4*>(&w[s][c]) = w4;
    __syncthreads();
    auto group_sum = [](float v) {   // over the token's threads (neighbouring lanes)
#pragma unroll
        for (int o = G / 2; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
        return v;
    };
    float* M = a.M + ((size_t)blockIdx.x * a.w.heads + hd) * (kWkvChunk * kWkvChunk);
    const float own = group_sum(r4.x * (u[0] * k4.x) + r4.y * (u[1] * k4.y) + r4.z * (u[2] * k4.z) + r4.w * (u[3] * k4.w));
    float4 front = one;   // the decays in front of token s
    // every thread runs all tokens (the sums are over lanes of tokens of the same warp, which start at different places)
#pragma unroll 1
    for (int t = 0; t < kWkvChunk; ++t) {
        const float4 wt = *reinterpret_cast<const float4*>(&w[t][c]);
        float part = 0.f;
        if (t > s) {
            const float4 rt = *reinterpret_cast<const float4*>(&r[t][c]);
            part = rt.x * k4.x + rt.y * k4.y + rt.z * k4.z + rt.w * k4.w;
            k4.x *= wt.x; k4.y *= wt.y; k4.z *= wt.z; k4.w *= wt.w;
        } else if (t < s) {
            front.x *= wt.x; front.y *= wt.y; front.z *= wt.z; front.w *= wt.w;
        }
        part = group_sum(part);
        if (c == 0) M[t * kWkvChunk + s] = t > s ? part : t == s ? own : 0.f;
    }
    if (s < rows) {
        *reinterpret_cast<float4*>(const_cast<float*>(a.w.r) + at) = make_float4(r4.x * front.x, r4.y * front.y, r4.z * front.z, r4.w * front.w);
        *reinterpret_cast<float4*>(const_cast<float*>(a.w.k) + at) = k4;
    }
    if (s == kWkvChunk - 1)
        *reinterpret_cast<float4*>(a.decay + ((size_t)blockIdx.x * a.w.heads + hd) * D + c) = make_float4(front.x * w4.x, front.y * w4.y, front.z * w4.z, front.w * w4.w);
}

// grid (entries, heads, D / 16), 4 D threads: thread (channels 4 c .. , column j) holds four entries of the state.  The operands of the next three
// chunks are on their way (cp.async): a chunk takes less than a round trip to memory.
constexpr int kWkvStages = 4;
constexpr int wkv_stage_floats(int D) { return 2 * kWkvChunk * D + kWkvChunk * kWkvCols + kWkvChunk * kWkvChunk + D; }
constexpr size_t wkv_chunk_smem_bytes(int D) { return sizeof(float) * ((size_t)kWkvStages * wkv_stage_floats(D) + (size_t)(D / 8) * kWkvChunk * kWkvCols); }
template <int D>
__global__ void __launch_bounds__(4 * D) wkv_chunk_scan_kernel(WkvChunkArgs a, StepMeta m) {
    pdl_launch_dependents();
    pdl_wait_prior_grid();
    constexpr int NT = 4 * D, NW = NT / 32, L = kWkvChunk, F = (L * kWkvCols + NT - 1) / NT;
    extern __shared__ __align__(16) float wkv_smem[];
    float* part = wkv_smem + kWkvStages * wkv_stage_floats(D);   // [NW][L][cols]
    const int e = blockIdx.x, hd = blockIdx.y, col0 = blockIdx.z * kWkvCols, tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int c = 4 * (tid / kWkvCols), j = tid % kWkvCols;
    const size_t C = (size_t)a.w.heads * D;
    float* Sg = a.w.state + ((size_t)m.ent_slot[e] * a.w.heads + hd) * (size_t)D * D;
    const bool fresh = m.ent_pos0[e] == 0;
    float S[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) S[i] = fresh ? 0.f : Sg[(size_t)(c + i) * D + col0 + j];
    const int t0 = m.ent_row0[e], n = m.ent_row0[e + 1] - t0, chunks = (n + L - 1) / L;
    int chunk0 = 0;
    for (int i = 0; i < e; ++i) chunk0 += (m.ent_row0[i + 1] - m.ent_row0[i] + L - 1) / L;
    // a stage: r [L][D], k [L][D], v [L][cols], M [L][L], decay [D]; rows behind the entry's last are zero
    auto fetch = [&](int q) {
        if (q < chunks) {
            float* st = wkv_smem + (q % kWkvStages) * wkv_stage_floats(D);
            const size_t ch = (size_t)(chunk0 + q) * a.w.heads + hd;
            const int rows = n - q * L;
            constexpr int kRow = L * D / 4, kV = L * kWkvCols / 4, kM = L * L / 4, kAll = 2 * kRow + kV + kM + D / 4;
            for (int x = tid; x < kAll; x += NT) {
                const float* src;
                bool in = true;
                if (x < 2 * kRow) {
                    const int y = x % kRow, t = y / (D / 4);
                    in = t < rows;
                    src = (x < kRow ? a.w.r : a.w.k) + (size_t)(t0 + q * L + (in ? t : 0)) * C + (size_t)hd * D + 4 * (y % (D / 4));
                } else if (x < 2 * kRow + kV) {
                    const int y = x - 2 * kRow, t = y / (kWkvCols / 4);
                    in = t < rows;
                    src = a.w.v + (size_t)(t0 + q * L + (in ? t : 0)) * C + (size_t)hd * D + col0 + 4 * (y % (kWkvCols / 4));
                } else if (x < 2 * kRow + kV + kM) {
                    src = a.M + ch * (L * L) + 4 * (x - 2 * kRow - kV);
                } else {
                    src = a.decay + ch * D + 4 * (x - 2 * kRow - kV - kM);
                }
                cp_async16(st + 4 * x, src, in);
            }
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
    for (int q = 0; q < kWkvStages - 1; ++q) fetch(q);
    for (int q = 0; q < chunks; ++q) {
        asm volatile("cp.async.wait_group %0;" ::"n"(kWkvStages - 2) : "memory");
        __syncthreads();   // this chunk's operands are there; the previous chunk's, and its partial outputs, are no longer read
        fetch(q + kWkvStages - 1);
        const float* r = wkv_smem + (q % kWkvStages) * wkv_stage_floats(D);
        const float *k = r + L * D, *v = k + L * D, *M = v + L * kWkvCols, *decay = M + L * L;
        // r_t^T S over the warp's channels (two groups of four): all loads, all sums, then all stores (a store between them would hold the loads behind it back)
        float o[L];
#pragma unroll
        for (int t = 0; t < L; ++t) {
            const float4 x = *reinterpret_cast<const float4*>(r + t * D + c);
            o[t] = fmaf(x.x, S[0], x.y * S[1]) + fmaf(x.z, S[2], x.w * S[3]);
        }
#pragma unroll
        for (int t = 0; t < L; ++t) o[t] += __shfl_xor_sync(0xffffffffu, o[t], 16);
        const float4 d4 = *reinterpret_cast<const float4*>(decay + c);
        S[0] *= d4.x; S[1] *= d4.y; S[2] *= d4.z; S[3] *= d4.w;
#pragma unroll
        for (int t = 0; t < L; ++t) {
            const float4 x = *reinterpret_cast<const float4*>(k + t * D + c);
            const float y = v[t * kWkvCols + j];
            S[0] = fmaf(x.x, y, S[0]); S[1] = fmaf(x.y, y, S[1]); S[2] = fmaf(x.z, y, S[2]); S[3] = fmaf(x.w, y, S[3]);
        }
        // (the two halves of the warp hold the same sums: each stores half of the tokens)
#pragma unroll
        for (int t = 0; t < L / 2; ++t) part[(warp * L + 2 * t + (lane >> 4)) * kWkvCols + j] = lane < 16 ? o[2 * t] : o[2 * t + 1];
        __syncthreads();
#pragma unroll
        for (int p = 0; p < F; ++p) {
            const int x = tid + p * NT, t = x / kWkvCols, col = x % kWkvCols;
            if (x < L * kWkvCols && q * L + t < n) {
                float s4[4] = {0.f, 0.f, 0.f, 0.f};   // four chains
#pragma unroll
                for (int i = 0; i < NW; ++i) s4[i & 3] += part[(i * L + t) * kWkvCols + col];
#pragma unroll
                for (int i = 0; i < L; ++i) s4[i & 3] = fmaf(M[t * L + i], i <= t ? v[i * kWkvCols + col] : 0.f, s4[i & 3]);   // (M is zero behind t, but a later token's v may be infinite)
                a.w.out[(size_t)(t0 + q * L + t) * C + (size_t)hd * D + col0 + col] = (s4[0] + s4[1]) + (s4[2] + s4[3]);
            }
        }
    }
    asm volatile("cp.async.wait_group 0;" ::: "memory");
#pragma unroll
    for (int i = 0; i < 4; ++i) Sg[(size_t)(c + i) * D + col0 + j] = S[i];
}

}  // namespace seq
}  // namespace tib
