// The fp32 lane-per-key attention of one warp: the lane-per-key kernel (qattn.cu) and, for codebooks that the fp16 tables
// cannot hold, the warp-level tensor-core kernel (qattn_mma.cu) run it over their share of the work units.
//
// Work unit: one warp per (user, query head, query token, key split).  Lane l walks
// keys l, l+32, ... of its split with a private online-softmax state (max, sum, 128
// accumulators); nothing crosses lanes until the final merge.  K and V are dequantised
// in registers by a 16-entry codebook lookup in shared memory (16 words occupy 16
// distinct banks, so any access pattern is conflict-free).  The QJL part of K is
// applied as a score correction  norm * c * sum_i s_i (q . g_i)  with the 64 values
// (q . g_i) computed once per work unit -- the same algebra as the reference kernel
// (kernels/fused_attention.py:198-213, 260-276) but with G seeded per (user, kv head)
// exactly as the codec does (kernels/quantize.py:583), which is what the reference's
// CPU path (kernels/fused_attention.py:435-466) computes.
#pragma once
#include "qattn.cuh"

namespace omni {

struct LaneScratch {                 // one warp's shared memory
    __align__(16) float q[kHeadDim];
    __align__(16) float qg[kQjlDim];
    float cb[16];
};

__device__ __forceinline__ void prefetch_l2(const void* p) { asm volatile("prefetch.global.L2 [%0];\n" :: "l"(p)); }

// Work units first, first + stride, ... of B * Hq * T * n_splits.
template <int DT>
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
    if (a.lora.x) {                                   // per-user low-rank update of the query row
        lora_fold_row(a.lora, b, a.T, (int)(qrow % a.T), a.Hq * kHeadDim, hq * kHeadDim + 4 * lane, lane, a.status, qv);
    }
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

    float m = -INFINITY, l = 0.f;
    float O[kHeadDim];
#pragma unroll
    for (int d = 0; d < kHeadDim; ++d) O[d] = 0.f;
    const float* qs = sc.q;
    const float* cbs = sc.cb;

    for (int64_t k = s0 + lane; k < s1; k += 32) {
        const int64_t row = base_row + k;
        const uint4* kp = reinterpret_cast<const uint4*>(a.k_nib + row * kNibBytes);
        // This key's sign bytes, norm and V row are needed one after the other further down: on a cold cache that is
        // three memory latencies in a row, so they are requested now, together with the K and V rows of the lane's
        // next key (a V row in the pair layout lies in this key's row and its partner's: the same 512-byte group).
        prefetch_l2(a.v_nib + row * kNibBytes);
        if (a.v_paired && k < (len & ~(int64_t)7)) prefetch_l2(a.v_nib + (base_row + (k ^ 3)) * kNibBytes);
        if (a.with_qjl) { prefetch_l2(a.k_qjl + row * kQjlBytes); prefetch_l2(a.k_norms + row); }
        if (k + 32 < s1) { prefetch_l2(a.k_nib + (row + 32) * kNibBytes); prefetch_l2(a.v_nib + (row + 32) * kNibBytes); }
        float dot = 0.f;
#pragma unroll
        for (int c4 = 0; c4 < 4; ++c4) {
            const uint4 wv = __ldg(kp + c4);
            const uint32_t ww[4] = {wv.x, wv.y, wv.z, wv.w};
#pragma unroll
            for (int wi = 0; wi < 4; ++wi) {
                const float4 qa = *reinterpret_cast<const float4*>(qs + c4 * 32 + wi * 8);
                const float4 qb = *reinterpret_cast<const float4*>(qs + c4 * 32 + wi * 8 + 4);
                const uint32_t w = ww[wi];
                dot = fmaf(qa.x, cbs[w & 15], dot);
                dot = fmaf(qa.y, cbs[(w >> 4) & 15], dot);
                dot = fmaf(qa.z, cbs[(w >> 8) & 15], dot);
                dot = fmaf(qa.w, cbs[(w >> 12) & 15], dot);
                dot = fmaf(qb.x, cbs[(w >> 16) & 15], dot);
                dot = fmaf(qb.y, cbs[(w >> 20) & 15], dot);
                dot = fmaf(qb.z, cbs[(w >> 24) & 15], dot);
                dot = fmaf(qb.w, cbs[(w >> 28) & 15], dot);
            }
        }
        float score = dot * a.scale;
        if (a.with_qjl) {
            const uint2 sb = __ldg(reinterpret_cast<const uint2*>(a.k_qjl + row * kQjlBytes));
            const float nrm = __ldg(a.k_norms + row);
            float corr = 0.f;
#pragma unroll
            for (int i = 0; i < 32; ++i) {
                const float g0 = sc.qg[i], g1 = sc.qg[i + 32];
                corr += ((sb.x >> i) & 1u) ? g0 : -g0;
                corr += ((sb.y >> i) & 1u) ? g1 : -g1;
            }
            score = fmaf(nrm, corr, score);
        }
        const float m_new = fmaxf(m, score);
        const float p = expf(score - m_new);
        if (m_new > m) {
            const float alpha = expf(m - m_new);
            l *= alpha;
#pragma unroll
            for (int d = 0; d < kHeadDim; ++d) O[d] *= alpha;
            m = m_new;
        }
        l += p;
        if (a.v_paired && k < (len & ~(int64_t)7)) {
            // pair layout: this key's even-d nibbles sit in the row of the pair's first key, its odd-d nibbles in
            // the row of the second (pairs (0,3), (1,2), (4,7), (5,6) of a group of eight: partner = key ^ 3), in
            // the low nibbles when this key is the first of the pair, else in the high ones
            const int64_t first = (k & 2) ? (k ^ 3) : k;
            const int sh = (k & 2) ? 4 : 0;
            const uint4* xp = reinterpret_cast<const uint4*>(a.v_nib + (base_row + first) * kNibBytes);
            const uint4* yp = reinterpret_cast<const uint4*>(a.v_nib + (base_row + (first ^ 3)) * kNibBytes);
#pragma unroll
            for (int c4 = 0; c4 < 4; ++c4) {
                const uint4 xv = __ldg(xp + c4), yv = __ldg(yp + c4);
                const uint32_t xw[4] = {xv.x, xv.y, xv.z, xv.w}, yw[4] = {yv.x, yv.y, yv.z, yv.w};
#pragma unroll
                for (int wi = 0; wi < 4; ++wi) {
#pragma unroll
                    for (int i = 0; i < 4; ++i) {
                        const int d = c4 * 32 + wi * 8 + 2 * i;
                        O[d] = fmaf(p, cbs[(xw[wi] >> (8 * i + sh)) & 15], O[d]);
                        O[d + 1] = fmaf(p, cbs[(yw[wi] >> (8 * i + sh)) & 15], O[d + 1]);
                    }
                }
            }
        } else {
            const uint4* vp = reinterpret_cast<const uint4*>(a.v_nib + row * kNibBytes);
#pragma unroll
            for (int c4 = 0; c4 < 4; ++c4) {
                const uint4 wv = __ldg(vp + c4);
                const uint32_t ww[4] = {wv.x, wv.y, wv.z, wv.w};
#pragma unroll
                for (int wi = 0; wi < 4; ++wi) {
                    const uint32_t w = ww[wi];
#pragma unroll
                    for (int n = 0; n < 8; ++n)
                        O[c4 * 32 + wi * 8 + n] = fmaf(p, cbs[(w >> (4 * n)) & 15], O[c4 * 32 + wi * 8 + n]);
                }
            }
        }
    }

    // ---- merge the 32 lane states ------------------------------------------------
    const float m_w = warp_max(m);
    const float f = (m == -INFINITY) ? 0.f : expf(m - m_w);
    const float l_w = warp_sum(l * f);
#pragma unroll
    for (int d = 0; d < kHeadDim; ++d) O[d] *= f;
    // butterfly reduce-scatter: afterwards O[0..3] hold dims 4*lane .. 4*lane+3
#pragma unroll
    for (int half = 64, mk = 16; half >= 4; half >>= 1, mk >>= 1) {
        const bool upper = (lane & mk) != 0;
#pragma unroll
        for (int j = 0; j < half; ++j) {
            const float send = upper ? O[j] : O[j + half];
            const float keep = upper ? O[j + half] : O[j];
            O[j] = keep + __shfl_xor_sync(kFullMask, send, mk);
        }
    }
    if (a.n_splits == 1) {
        float o[4];
        const float inv = l_w > 0.f ? 1.f / l_w : 0.f;
#pragma unroll
        for (int k = 0; k < 4; ++k) o[k] = O[k] * inv;
        if (a.unrotate_out) wht128_warp(o, lane);
        *reinterpret_cast<float4*>(a.out + qrow * kHeadDim + 4 * lane) = make_float4(o[0], o[1], o[2], o[3]);
    } else {
        float* w = a.ws + work * kWsStride;
        *reinterpret_cast<float4*>(w + 4 * lane) = make_float4(O[0], O[1], O[2], O[3]);
        if (lane == 0) { w[128] = m_w; w[129] = l_w; }
    }
    __syncwarp();                      // the next unit overwrites this warp's query row in shared memory
    }
}

}  // namespace omni
