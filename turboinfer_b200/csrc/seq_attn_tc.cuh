// seq_attn_tc.cuh -- attention of the layered sequence engine.  Prompt portions: the tcgen05 kernel of attn_tc.cuh over
//   - ragged steps: a block owns up to 128 consecutive rows of ONE sequence (tiles[2 i] = first row, tiles[2 i + 1] = count),
//   - grouped key/value heads, a sliding window or chunks of positions (only the pages the tile's rows can see are visited),
//   - capped scores, sigmoid weights, the per-head and per-coordinate output gates and the sink term of the softmax denominator,
// for query/key and value sizes up to 128 in fours; other shapes use the fp32 tiled kernel.
// Also here: the split-key attention of decode rows (flash-decoding: key chunks in parallel, then a merge).
#pragma once
#include "prefill.cuh"
#include "seq_kernels.cuh"

namespace tib {
namespace seq {

constexpr int kAttnTcTile = kAtQ;   // 128 rows a block

struct SeqKeys {   // kv_images_kernel: the pages (64 tokens) that the step's portions see, one after another
    StepMeta m;
    AttnShape s;
    const int* pages;   // [2 x] = entry, [2 x + 1] = page of its sequence
    const float *k_pool, *v_pool;
    int d, dv, g0;
    struct Tile { size_t tok0; int t0, lo, last; };
    __device__ void tile(int x, Tile& t) const {
        const int e = pages[2 * x], p = pages[2 * x + 1], pos0 = m.ent_pos0[e];
        t.t0 = p * kPageTokens;
        t.lo = attn_first_key(s, pos0);
        t.last = pos0 + m.ent_row0[e + 1] - m.ent_row0[e] - 1;
        t.tok0 = (size_t)m.page_table[(size_t)m.ent_slot[e] * m.table_stride + p] * kPageTokens;
    }
    __device__ const float* row(const Tile& t, int r, int g, bool is_v) const {
        if (t.t0 + r < t.lo || t.t0 + r > t.last) return nullptr;
        return is_v ? v_pool + ((t.tok0 + r) * s.kv_heads + g) * dv : k_pool + ((t.tok0 + r) * s.kv_heads + g) * d;
    }
};
struct SeqAttn {
    StepMeta m;
    AttnShape s;
    const int* tiles;
    const int* image0;   // [entries]: where the record of an entry's page 0 would lie (negative when its first pages have none)
    const float* qkvg;
    float* out;
    int d, dv, group, h0;
    __device__ void tile(int y, int& row0, int& count, int& pos0, int& img0) const {
        row0 = tiles[2 * y];
        count = tiles[2 * y + 1];
        pos0 = m.row_pos[row0];
        img0 = image0[m.row_ent[row0]];
    }
    __device__ const float* q(int row, int h) const { return qkvg + (size_t)row * s.ld + (size_t)h * d; }
    __device__ int first_key(int pos) const { return attn_first_key(s, pos); }
    __device__ void scores(float (&v)[kAtHalf]) const {
        if (s.softcap > 0.f) {
            const float pre = s.scale / s.softcap;
#pragma unroll
            for (int j = 0; j < kAtHalf; ++j) v[j] = s.softcap * tanhf(v[j] * pre);
        } else {
#pragma unroll
            for (int j = 0; j < kAtHalf; ++j) v[j] *= s.scale;
        }
    }
    __device__ bool sigmoid() const { return s.pb != nullptr; }
    __device__ float pb(int h) const { return s.pb[h]; }
    __device__ float sigmoid_weight(float score, float pb) const { return attn_sigmoid(score, pb); }
    __device__ float finish(int row, int h, float mx, float l) const { return attn_gate(s, qkvg, row, h) * attn_finish_factor(s, h, mx, l); }
    __device__ void store4(int row, int h, int c, float4 v) const {
        if (s.egate) {
            const float* eg = s.egate + (size_t)row * s.egate_ld + (size_t)h * dv + c;
            v.x *= sigmoid_f32(eg[0]); v.y *= sigmoid_f32(eg[1]); v.z *= sigmoid_f32(eg[2]); v.w *= sigmoid_f32(eg[3]);
        }
        float* o = out + (size_t)row * attn_out_stride(s) + (size_t)h * dv + c;
        if ((reinterpret_cast<uintptr_t>(o) & 15) == 0) *reinterpret_cast<float4*>(o) = v;
        else { o[0] = v.x; o[1] = v.y; o[2] = v.z; o[3] = v.w; }
    }
};

// ---- decode rows with long windows: key chunks in parallel -----------------------------------------------------------------
// grid (rows, heads, splits): split z of a (row, head) takes keys lo + z * chunk .. and leaves its partial (max, sum, o[dv]) in
// `part`; the block that finishes last (counted in `arrived` [rows][heads], zero between launches) combines the splits in ascending
// order, whichever block that is, and applies the gate.  chunk = ceil(visible keys / splits); at most 32 splits.
template <int PL>
__global__ void __launch_bounds__(kAttnWarps * 32) window_attention_split_kernel(const float* qkvg, StepMeta m, AttnShape s, const int* rows, int splits,
                                                                                  const float* k_pool, const float* v_pool, float* part, int* arrived, float* out) {
    pdl_launch_dependents();   // the kernel behind this one may be scheduled (and a few-row product may fetch its weights) ...
    pdl_wait_prior_grid();     // ... while this one waits here for the kernel before it, when it was launched ahead of its end
    extern __shared__ float sm[];
    const int bx = blockIdx.x, t = rows ? rows[bx] : bx, h = blockIdx.y, z = blockIdx.z;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int pos = m.row_pos[t];
    const int* table = m.page_table + (size_t)m.ent_slot[m.row_ent[t]] * m.table_stride;
    const int g = h / (s.heads / s.kv_heads);
    const float* q = qkvg + (size_t)t * s.ld + (size_t)h * s.dim;
    float qr[PL], o[PL];
#pragma unroll
    for (int i = 0; i < PL; ++i) {
        const int d = lane + 32 * i;
        qr[i] = d < s.dim ? q[d] : 0.f;
        o[i] = 0.f;
    }
    const int lo = attn_first_key(s, pos);
    const int chunk = (pos - lo + 1 + splits - 1) / splits;
    const int j0 = lo + z * chunk, j1 = min(pos, j0 + chunk - 1);
    float mx = s.pb ? 0.f : -INFINITY, l = 0.f;   // (weights without a softmax: the running maximum stays 0)
    const float pb = s.pb ? s.pb[h] : 0.f;
    const size_t kstride = (size_t)s.kv_heads * s.dim, vstride = attn_vstride(s);
    // a warp takes its keys four at a time: the four K rows (and then the four V rows) are requested together
    for (int jb = j0 + 4 * warp; jb <= j1; jb += 4 * kAttnWarps) {
        size_t off[4];
        float sc[4];
#pragma unroll
        for (int u = 0; u < 4; ++u) {
            const int j = min(jb + u, j1);
            off[u] = (size_t)table[j / kPageTokens] * kPageTokens + j % kPageTokens;
            sc[u] = 0.f;
        }
#pragma unroll
        for (int i = 0; i < PL; ++i) {
            const int d = lane + 32 * i;
            if (d < s.dim) {
#pragma unroll
                for (int u = 0; u < 4; ++u) sc[u] = fmaf(qr[i], k_pool[off[u] * kstride + (size_t)g * s.dim + d], sc[u]);
            }
        }
        float vv[4][PL];
#pragma unroll
        for (int i = 0; i < PL; ++i) {
            const int d = lane + 32 * i;
#pragma unroll
            for (int u = 0; u < 4; ++u) vv[u][i] = d < s.vdim ? v_pool[off[u] * vstride + (size_t)g * s.vdim + d] : 0.f;
        }
#pragma unroll
        for (int u = 0; u < 4; ++u) {
            const float su = attn_score(s, warp_sum(sc[u]));
            if (jb + u <= j1) {
                const float nm = s.pb ? 0.f : fmaxf(mx, su);
                const float corr = expf(mx - nm), p = s.pb ? attn_sigmoid(su, pb) : expf(su - nm);
                l = l * corr + p;
#pragma unroll
                for (int i = 0; i < PL; ++i) o[i] = fmaf(p, vv[u][i], o[i] * corr);
                mx = nm;
            }
        }
    }
    float* po = sm;
    float* pm = sm + kAttnWarps * s.vdim;
    float* pl = pm + kAttnWarps;
#pragma unroll
    for (int i = 0; i < PL; ++i) {
        const int d = lane + 32 * i;
        if (d < s.vdim) po[warp * s.vdim + d] = o[i];
    }
    if (lane == 0) {
        pm[warp] = mx;
        pl[warp] = l;
    }
    __syncthreads();
    float Mx = -INFINITY;
    for (int w = 0; w < kAttnWarps; ++w) Mx = fmaxf(Mx, pm[w]);
    float L = 0.f, f[kAttnWarps];
    for (int w = 0; w < kAttnWarps; ++w) {
        f[w] = (pm[w] == -INFINITY) ? 0.f : expf(pm[w] - Mx);
        L += pl[w] * f[w];
    }
    float* dst = part + (((size_t)bx * s.heads + h) * splits + z) * (size_t)(s.vdim + 2);
    for (int d = threadIdx.x; d < s.vdim; d += blockDim.x) {
        float acc = 0.f;
        for (int w = 0; w < kAttnWarps; ++w) acc += po[w * s.vdim + d] * f[w];
        dst[2 + d] = acc;
    }
    if (threadIdx.x == 0) {
        dst[0] = Mx;
        dst[1] = L;
    }
    __shared__ int last;
    __threadfence();
    __syncthreads();
    if (threadIdx.x == 0) {
        int* cnt = arrived + (size_t)bx * s.heads + h;
        last = atomicAdd(cnt, 1) == splits - 1;
        if (last) *cnt = 0;
    }
    __syncthreads();
    if (!last) return;
    __threadfence();
    // lane z holds split z's (max, sum); every warp works out the factors, the coordinates are spread over the block
    const size_t ps = (size_t)(s.vdim + 2);
    const float* p = part + ((size_t)bx * s.heads + h) * splits * ps;
    const float mz = lane < splits ? __ldcg(p + (size_t)lane * ps) : -INFINITY;
    const float lz = lane < splits ? __ldcg(p + (size_t)lane * ps + 1) : 0.f;
    const float Mt = warp_max(mz);
    const float fz = mz == -INFINITY ? 0.f : expf(mz - Mt);
    const float fin = attn_finish_factor(s, h, Mt, warp_sum(lz * fz)) * attn_gate(s, qkvg, t, h);
    constexpr int kMaxSplits = 32;
    float fs[kMaxSplits];   // every split's factor in registers first, so that the loads of a coordinate's partials do not wait on one another
#pragma unroll
    for (int q = 0; q < kMaxSplits; ++q) fs[q] = __shfl_sync(0xFFFFFFFFu, fz, q);
    for (int d = threadIdx.x; d < s.vdim; d += blockDim.x) {
        float acc = 0.f;
#pragma unroll
        for (int q = 0; q < kMaxSplits; ++q)
            if (q < splits) acc = fmaf(__ldcg(p + (size_t)q * ps + 2 + d), fs[q], acc);
        out[(size_t)t * attn_out_stride(s) + (size_t)h * s.vdim + d] = acc * fin;
    }
}

}  // namespace seq
}  // namespace tib
