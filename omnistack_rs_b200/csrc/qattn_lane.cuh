// The fp32 lane-per-key attention of one warp: the lane-per-key kernel (qattn.cu) and, for codebooks that the fp16 tables
// cannot hold, the warp-level tensor-core kernel (qattn_mma.cu) run it over their share of the work units.
//
// Work unit: one warp per (user, query head, query token, key split), 32 keys at a time.  Scores: lane = key, its K row
// dequantised in registers by a 16-entry codebook lookup in shared memory (16 words occupy 16 distinct banks, so any access
// pattern is conflict-free) and multiplied with the query row from shared memory.  Output: lane = 8 dims of one key of each of
// the 16 pairs of the pair layout, so a V row is read as consecutive words and eight accumulators suffice.  The QJL part of K is
// applied as a score correction  norm * c * sum_i s_i (q . g_i)  with the 64 values
// (q . g_i) computed once per work unit -- the same algebra as the reference kernel
// (kernels/fused_attention.py:198-213, 260-276) but with G seeded per (user, kv head)
// exactly as the codec does (kernels/quantize.py:583), which is what the reference's
// CPU path (kernels/fused_attention.py:435-466) computes.
//
// What bounds it: the shared-memory pipe (256 codebook lookups per 32 keys).  The same lane = key for the output took 128
// accumulators per lane, 168 registers and a butterfly over 128 values per work unit: 64 users x 8 heads x 2,048 keys 112.6 us
// against 104.5, 32 x 32 x 300 41.2 against 37.9, and called from the warp-level kernel it cost that kernel spills.  Error against
// fp64 (relative 2-norm, 4 users x 32 heads x 32,768 keys, centroids to 11): 7.3e-7, with per-lane maxima and one serial sum
// per dot product 1.9e-6.
#pragma once
#include "qattn.cuh"

namespace omni {

struct LaneScratch {                 // one warp's shared memory
    __align__(16) float q[kHeadDim];
    __align__(16) float qg[kQjlDim];
    float cb[16];
};

__device__ __forceinline__ void prefetch_l2(const void* p) { asm volatile("prefetch.global.L2 [%0];\n" :: "l"(p)); }

// Key pairs of the pair layout, in order: (0,3), (1,2), (4,7), (5,6) of every group of eight; the second key is the first ^ 3.
__device__ __forceinline__ constexpr int pair_first(int j) { return 8 * (j >> 2) + (j & 1) + 2 * (j & 2); }

// Work units first, first + stride, ... of B * Hq * T * n_splits.
template <int DT, bool LORA>
__device__ __forceinline__ void lane_per_key_rows(const AttnArgs& a, LaneScratch& sc, int64_t first, int64_t stride) {
    const int lane = threadIdx.x & 31;
    const int64_t n_work = a.B * a.Hq * a.T * a.n_splits;
    for (int64_t work = first; work < n_work; work += stride) {
    const int split = (int)(work % a.n_splits);
    int64_t rest = work / a.n_splits;
    const int64_t qrow = rest;                       // index into q / out: ((b*Hq + hq)*T + tq)
    rest /= a.T;
    const int hq = (int)(rest % a.Hq);
    const int64_t b = rest / a.Hq;
    const int hkv = hq / (a.Hq / a.Hkv);

    // ---- prologue: query, codebook, q . g_i ------------------------------------
    float qv[4];
    Elem<DT>::load4(a.q, qrow * kHeadDim + 4 * lane, qv);
    if (LORA && a.lora.x)                             // per-user low-rank update of the query row
        lora_fold_row(a.lora, b, a.T, (int)(qrow % a.T), a.Hq * kHeadDim, hq * kHeadDim + 4 * lane, lane, a.status, qv);
    if (a.rotate_q) wht128_warp(qv, lane);
    *reinterpret_cast<float4*>(&sc.q[4 * lane]) = make_float4(qv[0], qv[1], qv[2], qv[3]);
    {
        const float c = __ldg(a.codebooks + (a.cb_per_head ? hkv * 16 : 0) + (lane & 15));
        if (lane < 16) sc.cb[lane] = c;
        // an infinite or NaN centroid has no meaningful attention result: say so through the status word
        if (__any_sync(kFullMask, !isfinite(c)) && lane == 0 && a.status) atomicExch(a.status, OMNI_STATUS_BAD_CODEBOOK);
    }
    __syncwarp();
    if (a.with_qjl) {
        const int32_t uid = a.user_ids ? a.user_ids[b] : a.user_id;
        const uint4* grow = reinterpret_cast<const uint4*>(a.g_rows) + (size_t)seed_of(uid, hkv) * kQjlDim;
        const uint4 g0 = __ldg(grow + lane), g1 = __ldg(grow + lane + 32);
        const uint32_t w0[4] = {g0.x, g0.y, g0.z, g0.w};
        const uint32_t w1[4] = {g1.x, g1.y, g1.z, g1.w};
        float acc0 = 0.f, acc1 = 0.f;
#pragma unroll
        for (int w = 0; w < 4; ++w) {
#pragma unroll 8
            for (int j = 0; j < 32; ++j) {
                const float qd = sc.q[w * 32 + j];
                acc0 += ((w0[w] >> j) & 1u) ? qd : -qd;
                acc1 += ((w1[w] >> j) & 1u) ? qd : -qd;
            }
        }
        const float cs = kQjlCoef * a.scale;
        sc.qg[lane] = acc0 * cs;
        sc.qg[lane + 32] = acc1 * cs;
    }
    __syncwarp();

    // ---- key range of this split -----------------------------------------------
    int64_t len = a.seq_lens ? (int64_t)a.seq_lens[b] : a.S;
    len = len < 0 ? 0 : (len > a.S ? a.S : len);
    int64_t per = (len + a.n_splits - 1) / a.n_splits;
    per = (per + 31) / 32 * 32;
    const int64_t s0 = (int64_t)split * per;
    const int64_t s1 = (s0 + per < len) ? s0 + per : len;
    const int64_t slot = a.cache_slots ? (int64_t)a.cache_slots[b] : b;
    const int64_t base_row = slot * a.ks_b + (int64_t)hkv * a.ks_h;

    const int64_t paired = a.v_paired ? (len & ~(int64_t)7) : 0;       // keys below this are stored pair-wise
    const float* qs = sc.q;
    const float* cbs = sc.cb;
    const int half = lane >> 4, w = lane & 15;
    float m = -INFINITY, l = 0.f, O[8];                // m: the same in every lane; l: of this lane's keys
#pragma unroll
    for (int n = 0; n < 8; ++n) O[n] = 0.f;

    // the K row, sign bytes and norm of this lane's key among 32 (the last key where there are fewer); the next 32 keys' are
    // fetched as soon as the scores no longer need these
    uint4 kw[4];
    uint2 sb = make_uint2(0u, 0u);
    float nrm = 0.f;
    auto fetch_k = [&](int64_t k0) {
        const int64_t row = base_row + (k0 + lane < s1 ? k0 + lane : s1 - 1);
        const uint4* kp = reinterpret_cast<const uint4*>(a.k_nib + row * kNibBytes);
#pragma unroll
        for (int c = 0; c < 4; ++c) kw[c] = __ldg(kp + c);
        if (a.with_qjl) {
            sb = __ldg(reinterpret_cast<const uint2*>(a.k_qjl + row * kQjlBytes));
            nrm = __ldg(a.k_norms + row);
        }
    };
    if (s0 < s1) fetch_k(s0);

    for (int64_t k0 = s0; k0 < s1; k0 += 32) {
        // ---- the lane's word of one key of every pair, used after the scores ----
        const int n_keys = s1 - k0 < 32 ? (int)(s1 - k0) : 32;
        uint32_t vw[16];
#pragma unroll
        for (int j = 0; j < 16; ++j) {
            const int key = pair_first(j) ^ (3 * half);
            vw[j] = __ldg(reinterpret_cast<const uint32_t*>(a.v_nib + (base_row + k0 + (key < n_keys ? key : n_keys - 1)) * kNibBytes) + w);
        }
        if (k0 + 32 + lane < s1) prefetch_l2(a.v_nib + (base_row + k0 + 32 + lane) * kNibBytes);
        // ---- scores: lane = key ----
        float dot[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
        for (int c = 0; c < 4; ++c) {
            const uint32_t ww[4] = {kw[c].x, kw[c].y, kw[c].z, kw[c].w};
#pragma unroll
            for (int i = 0; i < 4; ++i) {
#pragma unroll
                for (int h = 0; h < 2; ++h) {
                    const float4 q4 = *reinterpret_cast<const float4*>(qs + c * 32 + i * 8 + 4 * h);
                    dot[0] = fmaf(q4.x, cbs[(ww[i] >> (16 * h)) & 15u], dot[0]);
                    dot[1] = fmaf(q4.y, cbs[(ww[i] >> (16 * h + 4)) & 15u], dot[1]);
                    dot[2] = fmaf(q4.z, cbs[(ww[i] >> (16 * h + 8)) & 15u], dot[2]);
                    dot[3] = fmaf(q4.w, cbs[(ww[i] >> (16 * h + 12)) & 15u], dot[3]);
                }
            }
        }
        float score = ((dot[0] + dot[1]) + (dot[2] + dot[3])) * a.scale;
        if (a.with_qjl) {
            float corr[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
            for (int i = 0; i < 32; i += 4) {
                const float4 ga = *reinterpret_cast<const float4*>(&sc.qg[i]), gb = *reinterpret_cast<const float4*>(&sc.qg[i + 32]);
                const float g0[4] = {ga.x, ga.y, ga.z, ga.w}, g1[4] = {gb.x, gb.y, gb.z, gb.w};
#pragma unroll
                for (int e = 0; e < 4; ++e) {
                    corr[e & 1] += ((sb.x >> (i + e)) & 1u) ? g0[e] : -g0[e];
                    corr[2 + (e & 1)] += ((sb.y >> (i + e)) & 1u) ? g1[e] : -g1[e];
                }
            }
            score = fmaf(nrm, (corr[0] + corr[1]) + (corr[2] + corr[3]), score);
        }
        if (k0 + 32 < s1) fetch_k(k0 + 32);
        if (lane >= n_keys) score = -INFINITY;
        const float m_new = fmaxf(m, warp_max(score));
        const float p = expf(score - m_new), alpha = expf(m - m_new);
        m = m_new;
        l = fmaf(l, alpha, p);
        // ---- output: lane = 8 dims of one key of a pair; summed over the 32 keys first, then added to the running sums ----
        float acc[8];
#pragma unroll
        for (int n = 0; n < 8; ++n) acc[n] = 0.f;
#pragma unroll
        for (int j = 0; j < 16; ++j) {
            if (8 * (j >> 2) >= n_keys) break;
            const float pj = __shfl_sync(kFullMask, p, pair_first(j) ^ (3 * half));
            uint32_t x = vw[j];
            if (k0 + 8 * (j >> 2) < paired) {          // (X: even dims of both keys, Y: odd dims) -> this key's word
                const uint32_t o = __shfl_xor_sync(kFullMask, x, 16);
                x = half ? ((o >> 4) & 0x0F0F0F0Fu) | (x & 0xF0F0F0F0u) : (x & 0x0F0F0F0Fu) | ((o & 0x0F0F0F0Fu) << 4);
            }
#pragma unroll
            for (int n = 0; n < 8; ++n) acc[n] = fmaf(pj, cbs[(x >> (4 * n)) & 15u], acc[n]);
        }
#pragma unroll
        for (int n = 0; n < 8; ++n) O[n] = fmaf(O[n], alpha, acc[n]);
    }

    // ---- add up the two halves; lane = dims 4 lane .. 4 lane + 3 ------------------------------------------------
    const float l_w = warp_sum(l);
#pragma unroll
    for (int n = 0; n < 8; ++n) O[n] += __shfl_xor_sync(kFullMask, O[n], 16);
    float o[4];
#pragma unroll
    for (int k = 0; k < 4; ++k) {
        const float lo = __shfl_sync(kFullMask, O[k], lane >> 1), hi = __shfl_sync(kFullMask, O[k + 4], lane >> 1);
        o[k] = (lane & 1) ? hi : lo;
    }
    if (a.n_splits == 1) {
        const float inv = l_w > 0.f ? 1.f / l_w : 0.f;
#pragma unroll
        for (int k = 0; k < 4; ++k) o[k] *= inv;
        if (a.unrotate_out) wht128_warp(o, lane);
        *reinterpret_cast<float4*>(a.out + qrow * kHeadDim + 4 * lane) = make_float4(o[0], o[1], o[2], o[3]);
    } else {
        float* ws = a.ws + work * kWsStride;
        *reinterpret_cast<float4*>(ws + 4 * lane) = make_float4(o[0], o[1], o[2], o[3]);
        if (lane == 0) { ws[128] = m; ws[129] = l_w; }
    }
    __syncwarp();                      // the next unit overwrites this warp's query row in shared memory
    }
}

}  // namespace omni
