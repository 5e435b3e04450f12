// Attention over short caches (up to a few hundred keys per user) in fp32 on the CUDA cores: the calls whose time is
// latency, where neither a tensor-core work item (table build, operand build, one warp walking all keys) nor one warp per
// query row can spread a user's few keys over enough threads.
//
// One CTA of 128 threads serves one (user, kv head, tile of C query columns) and takes the keys 64 at a time:
//   scores   two threads per key, 64 dims and 32 sign projections each; the K row is dequantised once into registers and
//            multiplied with every column of the tile (queries and q.g projections broadcast from shared memory);
//   output   thread (word w, key group g): dims 8w .. 8w+7 of four key pairs, so a V row is read as consecutive words;
//            the eight key groups are added up once at the end.
// The packed bytes of the first 64 keys are requested before anything else, so their latency runs beside the loads of the
// query, the codebook and G.  What bounds it: the chain launch -> loads -> q.g -> scores -> softmax -> output of one chunk
// of keys: 3.5 us for up to 16 users x 8 heads x 50 keys, 6.0 us for 64 x 8 x 50, where one warp per query row took 12 and 13.5 us.
//
// Same numerics as the lane-per-key kernel: fp32 throughout, centroids of any finite size.
#include "qattn.cuh"

namespace omni {

constexpr int kShortThreads = 128;
constexpr int kShortKeys = 64;                       // keys per pass
constexpr int kHalfStride = 68;                      // a query row's two halves, 4 words further apart than they are long: the two
                                                     // broadcast addresses of a warp fall into different banks

__device__ __forceinline__ float sum_of_four(const float (&s)[4]) { return (s[0] + s[1]) + (s[2] + s[3]); }

// The common small case of lora_update below with its extents known at compile time: the rows of A and B that a warp needs are
// all requested before the first is used (64 users x 32 / 8 heads x 50 keys, rank 16: 16.8 us with the general form, 14.9 us).
template <int RANK, int C>
__device__ __forceinline__ void lora_update_small(const AttnArgs& a, int li, int64_t b, int hkv, int Gq, int col0, int ncols, float (&down)[kHeadDim],
                                                  int warp, int lane, float (&qv)[4]) {
    const LoraFold& L = a.lora;
    const float4 xv = __ldg(reinterpret_cast<const float4*>(L.x + b * 128) + lane);
    // words of a B row requested at a time, and those of them requested before the rows of A are used (with rank 32 these hold
    // 32 registers themselves)
    constexpr int kR4 = RANK / 4, kAhead = kR4 < 4 ? kR4 : 4, kEarly = RANK <= 16 ? kAhead : 1;
    float4 av[kR4], wv[4][kAhead];
    const float4* br = reinterpret_cast<const float4*>(L.b + (((int64_t)li * a.Hq + hkv * Gq + col0 + warp) * kHeadDim + 4 * lane) * RANK);
    auto fetch_b = [&](int r4, int from, int to) {
#pragma unroll
        for (int i = 0; i < 4; ++i) {
#pragma unroll
            for (int k = from; k < to; ++k) wv[i][k] = __ldg(br + i * kR4 + r4 + k);
        }
    };
#pragma unroll
    for (int j = 0; j < kR4; ++j) av[j] = __ldg(reinterpret_cast<const float4*>(L.a + ((int64_t)li * RANK + warp + 4 * j) * 128) + lane);
    if (warp < ncols) fetch_b(0, 0, kEarly);
#pragma unroll
    for (int j = 0; j < kR4; ++j) {
        float v = 0.f;
        v = fmaf(xv.x, av[j].x, v); v = fmaf(xv.y, av[j].y, v); v = fmaf(xv.z, av[j].z, v); v = fmaf(xv.w, av[j].w, v);
        v = warp_sum(v);
        if (lane == 0) down[warp + 4 * j] = v;
    }
    if (warp < ncols) fetch_b(0, kEarly, kAhead);
    __syncthreads();
    if (warp >= ncols) return;
    float up[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll 1
    for (int r4 = 0; r4 < kR4; r4 += kAhead) {
        if (r4 > 0) fetch_b(r4, 0, kAhead);
#pragma unroll
        for (int k = 0; k < kAhead; ++k) {
            const float4 dv = *reinterpret_cast<const float4*>(&down[4 * (r4 + k)]);
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                up[i] = fmaf(dv.x, wv[i][k].x, up[i]); up[i] = fmaf(dv.y, wv[i][k].y, up[i]);
                up[i] = fmaf(dv.z, wv[i][k].z, up[i]); up[i] = fmaf(dv.w, wv[i][k].w, up[i]);
            }
        }
    }
#pragma unroll
    for (int i = 0; i < 4; ++i) qv[i] = fmaf(up[i], L.alpha, qv[i]);
}

// The user's adapter, or -1 when the query stays as it is; the same for every thread of the CTA.
__device__ __forceinline__ int32_t adapter_of(const AttnArgs& a, int64_t b, int tid) {
    const int32_t li = __ldg(a.lora.idx + b);
    if (li < a.lora.n_adapters) return li;
    if (a.status && tid == 0) atomicMax(a.status, OMNI_STATUS_BAD_INDEX);
    return -1;
}

// Per-user low-rank query update of the tile's columns by the whole CTA: the warps share the rows of the down projection
// (once per CTA, or once per column when the columns are different tokens), then warp c adds the up projection to its own
// column.  Operations and order per element are those of the separate launch (lora_q.cu), hence the same bits.
template <int C>
__device__ __forceinline__ void lora_update(const AttnArgs& a, int64_t b, int hkv, int Gq, int col0, int ncols, float (&down)[C][kHeadDim],
                                            int tid, int warp, int lane, float (&qv)[4]) {
    const LoraFold& L = a.lora;
    const int32_t li = adapter_of(a, b, tid);
    if (li < 0) return;
    if (a.T == 1 && L.hidden == 128 && (L.rank == 8 || L.rank == 16) &&
        ((reinterpret_cast<uintptr_t>(L.x) | reinterpret_cast<uintptr_t>(L.a) | reinterpret_cast<uintptr_t>(L.b)) & 15) == 0) {
        if (L.rank == 16) lora_update_small<16, C>(a, li, b, hkv, Gq, col0, ncols, down[0], warp, lane, qv);
        else              lora_update_small<8, C>(a, li, b, hkv, Gq, col0, ncols, down[0], warp, lane, qv);
        return;
    }
    const float* am = L.a + (int64_t)li * L.rank * L.hidden;
    const int n_down = a.T == 1 ? 1 : ncols;
    for (int c = 0; c < n_down; ++c) {
        const float* xr = L.x + (b * a.T + (col0 + c) % a.T) * (int64_t)L.hidden;
#pragma unroll 4
        for (int r = warp; r < L.rank; r += 4) {
            const float v = lora_down_row(xr, am + (int64_t)r * L.hidden, L.hidden, lane);
            if (lane == 0) down[c][r] = v;
        }
    }
    __syncthreads();
    if (warp < ncols) {
        const float* d = down[a.T == 1 ? 0 : warp];
        const int cg = col0 + warp;
        const float* br = L.b + ((int64_t)li * a.Hq * kHeadDim + (int64_t)(hkv * Gq + cg / a.T) * kHeadDim + 4 * lane) * L.rank;
        float up[4] = {0.f, 0.f, 0.f, 0.f};
        if (L.rank % 4 == 0 && (reinterpret_cast<uintptr_t>(L.b) & 15) == 0) {
#pragma unroll 2
            for (int r = 0; r < L.rank; r += 4) {
                const float4 dv = *reinterpret_cast<const float4*>(d + r);
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    const float4 wv = __ldg(reinterpret_cast<const float4*>(br + (int64_t)i * L.rank + r));
                    up[i] = fmaf(dv.x, wv.x, up[i]); up[i] = fmaf(dv.y, wv.y, up[i]);
                    up[i] = fmaf(dv.z, wv.z, up[i]); up[i] = fmaf(dv.w, wv.w, up[i]);
                }
            }
        } else {
            for (int r = 0; r < L.rank; ++r)
#pragma unroll
                for (int i = 0; i < 4; ++i) up[i] = fmaf(d[r], __ldg(br + (int64_t)i * L.rank + r), up[i]);
        }
#pragma unroll
        for (int i = 0; i < 4; ++i) qv[i] = fmaf(up[i], L.alpha, qv[i]);
    }
}

// Builds of the kernel.  The query update's registers set its occupancy (128 of them, four CTAs per SM), so
//   kAnyUpdate  serves calls without an update and with any;
//   kRank32     the update of rank 32 with all rows requested ahead, whose registers the others would pay for (16 users x 8 heads x
//               50 keys 5.5 us against 9.8 with the general form, 128 x 8 x 50 16.0 against 21.3);
//   kNoUpdate   eight CTAs per SM, for one column and more CTAs than four per SM hold: 127 users x 8 heads x 17 keys 8.2 us against
//               9.5 (the lane-per-key kernel 9.2); with fewer CTAs its 64 registers are too few (8 CTAs x 256 keys 7.6 against 6.4).
enum ShortBuild { kAnyUpdate, kRank32, kNoUpdate };
constexpr int64_t kFourPerSm = 4 * 148;

template <int DT, int C, ShortBuild BUILD>
__global__ void __launch_bounds__(kShortThreads, BUILD == kNoUpdate ? 8 : 4) qattn_short_kernel(AttnArgs a, int n_ctiles) {
    __shared__ __align__(16) float q_s[C][2 * kHalfStride];
    __shared__ __align__(16) float qg_s[C][2 * 36];
    __shared__ __align__(16) float red_s[4][C][kHeadDim];       // prologue: down projections of the query update; end: the warps' sums
    __shared__ float p_s[C][kShortKeys];
    __shared__ float cb_s[16];
    __shared__ float max_s[2][4][C], sum_s[4][C];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int Gq = a.Hq / a.Hkv, ncols_all = Gq * a.T;
    int64_t rest = blockIdx.x;
    const int col0 = C * (int)(rest % n_ctiles);
    rest /= n_ctiles;
    const int hkv = (int)(rest % a.Hkv);
    const int64_t b = rest / a.Hkv;
    const int ncols = ncols_all - col0 < C ? ncols_all - col0 : C;

    const int64_t len64 = a.seq_lens ? (int64_t)a.seq_lens[b] : a.S;
    const int len = (int)(len64 < 0 ? 0 : (len64 > a.S ? a.S : len64));
    const int paired = a.v_paired ? (len & ~7) : 0;              // keys below this are stored pair-wise
    const int64_t slot = a.cache_slots ? (int64_t)a.cache_slots[b] : b;
    const int64_t row0 = slot * a.ks_b + (int64_t)hkv * a.ks_h;

    // ---- packed bytes of a pass -------------------------------------------------------------------------------------
    const int ks = tid >> 1, hf = tid & 1;                       // scores: key of the pass, half of its row
    const int w = tid & 15, kg = tid >> 4;                       // output: word of the row, key group
    uint4 kn0, kn1;
    uint32_t sw = 0u;
    float nrm = 0.f;
    uint32_t va[4], vb[4];                                       // words of the key pairs kg + 8 j (keys: pair_first, ^ 3)
    auto pair_first = [&](int j) { const int p = kg + 8 * j; return (p >> 2) * 8 + (p & 1) + 2 * (p & 2); };
    auto fetch = [&](int k0) {
        const int last = len - 1;
        const int64_t r = row0 + (k0 + ks < len ? k0 + ks : last);
        const uint4* kp = reinterpret_cast<const uint4*>(a.k_nib + r * kNibBytes + 32 * hf);
        kn0 = __ldg(kp);
        kn1 = __ldg(kp + 1);
        if (a.with_qjl) {
            sw = __ldg(reinterpret_cast<const uint32_t*>(a.k_qjl + r * kQjlBytes) + hf);
            nrm = __ldg(a.k_norms + r);
        }
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const int ka = k0 + pair_first(j), kb = ka ^ 3;
            va[j] = __ldg(reinterpret_cast<const uint32_t*>(a.v_nib + (row0 + (ka < len ? ka : last)) * kNibBytes) + w);
            vb[j] = __ldg(reinterpret_cast<const uint32_t*>(a.v_nib + (row0 + (kb < len ? kb : last)) * kNibBytes) + w);
        }
    };
    if (len > 0) fetch(0);

    // ---- prologue: query rows (with the per-user update and the rotation), codebook, q.g ------------------------------
    uint2 gw = make_uint2(0u, 0u);                               // signs of projection tid >> 1, dims 64 hf ..
    if (a.with_qjl) {
        const int32_t uid = a.user_ids ? a.user_ids[b] : a.user_id;
        gw = __ldg(reinterpret_cast<const uint2*>(a.g_rows + ((size_t)seed_of(uid, hkv) * kQjlDim + ks) * 4) + hf);
    }
    float qv[4] = {0.f, 0.f, 0.f, 0.f};                          // warp c: column c, dims 4 lane ..
    if (warp < ncols) {
        const int cg = col0 + warp;
        const int64_t qrow = (b * a.Hq + (int64_t)hkv * Gq + cg / a.T) * a.T + (cg % a.T);
        Elem<DT>::load4(a.q, qrow * kHeadDim + 4 * lane, qv);
    }
    if (tid < 16) {
        const float cv = __ldg(a.codebooks + (a.cb_per_head ? hkv * 16 : 0) + tid);
        cb_s[tid] = cv;
        // an infinite or NaN centroid has no meaningful attention result: say so through the status word
        if (!isfinite(cv) && a.status) atomicExch(a.status, OMNI_STATUS_BAD_CODEBOOK);
    }
    if (BUILD == kRank32) {
        const int32_t li = adapter_of(a, b, tid);
        if (li >= 0) lora_update_small<32, C>(a, li, b, hkv, Gq, col0, ncols, red_s[0][0], warp, lane, qv);
    } else if (BUILD == kAnyUpdate && a.lora.x) {
        lora_update<C>(a, b, hkv, Gq, col0, ncols, red_s[0], tid, warp, lane, qv);
    }
    if (a.rotate_q) wht128_warp(qv, lane);
    if (warp < C) *reinterpret_cast<float4*>(&q_s[warp][(lane >> 4) * kHalfStride + 4 * (lane & 15)]) = make_float4(qv[0], qv[1], qv[2], qv[3]);
    __syncthreads();
    if (a.with_qjl) {
        float acc[C][4];
#pragma unroll
        for (int c = 0; c < C; ++c) { acc[c][0] = 0.f; acc[c][1] = 0.f; acc[c][2] = 0.f; acc[c][3] = 0.f; }
        const uint32_t gword[2] = {gw.x, gw.y};
#pragma unroll
        for (int wd = 0; wd < 2; ++wd) {
#pragma unroll
            for (int j = 0; j < 32; j += 4) {
                float s[4];
#pragma unroll
                for (int i = 0; i < 4; ++i) s[i] = ((gword[wd] >> (j + i)) & 1u) ? 1.f : -1.f;
#pragma unroll
                for (int c = 0; c < C; ++c) {
                    const float4 q4 = *reinterpret_cast<const float4*>(&q_s[c][hf * kHalfStride + 32 * wd + j]);
                    acc[c][0] = fmaf(s[0], q4.x, acc[c][0]); acc[c][1] = fmaf(s[1], q4.y, acc[c][1]);
                    acc[c][2] = fmaf(s[2], q4.z, acc[c][2]); acc[c][3] = fmaf(s[3], q4.w, acc[c][3]);
                }
            }
        }
        const float cs = kQjlCoef * a.scale;
#pragma unroll
        for (int c = 0; c < C; ++c) {
            float v = sum_of_four(acc[c]);
            v += __shfl_xor_sync(kFullMask, v, 1);
            if (hf == 0) qg_s[c][(ks >> 5) * 36 + (ks & 31)] = v * cs;
        }
        __syncthreads();
    }

    // ---- passes over 64 keys ------------------------------------------------------------------------------------------
    float m_run[C], l_run[C], O[C][8];
#pragma unroll
    for (int c = 0; c < C; ++c) {
        m_run[c] = -INFINITY; l_run[c] = 0.f;
#pragma unroll
        for (int n = 0; n < 8; ++n) O[c][n] = 0.f;
    }
    for (int k0 = 0; k0 < len; k0 += kShortKeys) {
        float s[C];
        {
            float acc[C][4];
#pragma unroll
            for (int c = 0; c < C; ++c) { acc[c][0] = 0.f; acc[c][1] = 0.f; acc[c][2] = 0.f; acc[c][3] = 0.f; }
            const uint32_t kw[8] = {kn0.x, kn0.y, kn0.z, kn0.w, kn1.x, kn1.y, kn1.z, kn1.w};
#pragma unroll
            for (int e = 0; e < 8; ++e) {
#pragma unroll
                for (int h = 0; h < 2; ++h) {
                    float kd[4];
#pragma unroll
                    for (int i = 0; i < 4; ++i) kd[i] = cb_s[(kw[e] >> (16 * h + 4 * i)) & 15u];
#pragma unroll
                    for (int c = 0; c < C; ++c) {
                        const float4 q4 = *reinterpret_cast<const float4*>(&q_s[c][hf * kHalfStride + 8 * e + 4 * h]);
                        acc[c][0] = fmaf(kd[0], q4.x, acc[c][0]); acc[c][1] = fmaf(kd[1], q4.y, acc[c][1]);
                        acc[c][2] = fmaf(kd[2], q4.z, acc[c][2]); acc[c][3] = fmaf(kd[3], q4.w, acc[c][3]);
                    }
                }
            }
#pragma unroll
            for (int c = 0; c < C; ++c) s[c] = sum_of_four(acc[c]) * a.scale;
        }
        if (a.with_qjl) {
            float acc[C][4];
#pragma unroll
            for (int c = 0; c < C; ++c) { acc[c][0] = 0.f; acc[c][1] = 0.f; acc[c][2] = 0.f; acc[c][3] = 0.f; }
#pragma unroll
            for (int j = 0; j < 32; j += 4) {
                float sg[4];
#pragma unroll
                for (int i = 0; i < 4; ++i) sg[i] = ((sw >> (j + i)) & 1u) ? 1.f : -1.f;
#pragma unroll
                for (int c = 0; c < C; ++c) {
                    const float4 g4 = *reinterpret_cast<const float4*>(&qg_s[c][hf * 36 + j]);
                    acc[c][0] = fmaf(sg[0], g4.x, acc[c][0]); acc[c][1] = fmaf(sg[1], g4.y, acc[c][1]);
                    acc[c][2] = fmaf(sg[2], g4.z, acc[c][2]); acc[c][3] = fmaf(sg[3], g4.w, acc[c][3]);
                }
            }
#pragma unroll
            for (int c = 0; c < C; ++c) s[c] = fmaf(nrm, sum_of_four(acc[c]), s[c]);
        }
        const int buf = (k0 / kShortKeys) & 1;                   // two buffers: a pass's maxima outlive the next barrier
#pragma unroll
        for (int c = 0; c < C; ++c) {
            s[c] += __shfl_xor_sync(kFullMask, s[c], 1);
            if (k0 + ks >= len) s[c] = -INFINITY;
            const float m = warp_max(s[c]);
            if (lane == 0) max_s[buf][warp][c] = m;
        }
        __syncthreads();                                         // also: the previous pass has read p_s
#pragma unroll
        for (int c = 0; c < C; ++c) {
            const float mx = fmaxf(fmaxf(max_s[buf][0][c], max_s[buf][1][c]), fmaxf(max_s[buf][2][c], max_s[buf][3][c]));
            const float m_new = fmaxf(m_run[c], mx);
            const float alpha = m_run[c] == -INFINITY ? 0.f : expf(m_run[c] - m_new);
            const float p = expf(s[c] - m_new);
            l_run[c] = fmaf(l_run[c], alpha, p);                 // counted twice (both halves of a key): halved at the end
#pragma unroll
            for (int n = 0; n < 8; ++n) O[c][n] *= alpha;
            m_run[c] = m_new;
            if (hf == 0) p_s[c][ks] = p;
        }
        uint32_t xa[4], xb[4];
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            xa[j] = va[j]; xb[j] = vb[j];
            if (k0 + pair_first(j) < paired) {                   // (X: even dims of both keys, Y: odd dims) -> the two keys' words
                const uint32_t X = va[j], Y = vb[j];
                xa[j] = (X & 0x0F0F0F0Fu) | ((Y & 0x0F0F0F0Fu) << 4);
                xb[j] = ((X >> 4) & 0x0F0F0F0Fu) | (Y & 0xF0F0F0F0u);
            }
        }
        if (k0 + kShortKeys < len) fetch(k0 + kShortKeys);
        __syncthreads();
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const int ka = pair_first(j);
            float pa[C], pb[C];
#pragma unroll
            for (int c = 0; c < C; ++c) { pa[c] = p_s[c][ka]; pb[c] = p_s[c][ka ^ 3]; }
#pragma unroll
            for (int n = 0; n < 8; ++n) {
                const float fa = cb_s[(xa[j] >> (4 * n)) & 15u], fb = cb_s[(xb[j] >> (4 * n)) & 15u];
#pragma unroll
                for (int c = 0; c < C; ++c) O[c][n] = fmaf(pb[c], fb, fmaf(pa[c], fa, O[c][n]));
            }
        }
    }

    // ---- add up: key groups and sums of weights, then one warp per column normalises (and rotates back) ------------------
    __syncthreads();
#pragma unroll
    for (int c = 0; c < C; ++c) {
        const float l = warp_sum(l_run[c]);
        if (lane == 0) sum_s[warp][c] = l;
#pragma unroll
        for (int n = 0; n < 8; ++n) O[c][n] += __shfl_xor_sync(kFullMask, O[c][n], 16);
        if (lane < 16) {
            *reinterpret_cast<float4*>(&red_s[warp][c][8 * w]) = make_float4(O[c][0], O[c][1], O[c][2], O[c][3]);
            *reinterpret_cast<float4*>(&red_s[warp][c][8 * w + 4]) = make_float4(O[c][4], O[c][5], O[c][6], O[c][7]);
        }
    }
    __syncthreads();
    if (warp < ncols) {
        const int c = warp;
        const float l = 0.5f * ((sum_s[0][c] + sum_s[1][c]) + (sum_s[2][c] + sum_s[3][c]));
        const float inv = l > 0.f ? 1.f / l : 0.f;
        float4 r[4];
#pragma unroll
        for (int k = 0; k < 4; ++k) r[k] = *reinterpret_cast<const float4*>(&red_s[k][c][4 * lane]);
        float o[4] = {((r[0].x + r[1].x) + (r[2].x + r[3].x)) * inv, ((r[0].y + r[1].y) + (r[2].y + r[3].y)) * inv,
                      ((r[0].z + r[1].z) + (r[2].z + r[3].z)) * inv, ((r[0].w + r[1].w) + (r[2].w + r[3].w)) * inv};
        if (a.unrotate_out) wht128_warp(o, lane);
        const int cg = col0 + c;
        const int64_t qrow = (b * a.Hq + (int64_t)hkv * Gq + cg / a.T) * a.T + (cg % a.T);
        *reinterpret_cast<float4*>(a.out + qrow * kHeadDim + 4 * lane) = make_float4(o[0], o[1], o[2], o[3]);
    }
}

bool short_eligible(const AttnArgs& a) {
    const int64_t cols = (int64_t)(a.Hq / a.Hkv) * a.T;
    // any split count: the kernel splits a user's keys over its threads and writes finished rows
    return a.S <= 4096 && a.B * a.Hkv * cols <= 0x7fffffffLL;
}

// Fewer than 128 keys and 1,024 rows: always (calls that were never given to fp16 operands; the lane-per-key kernel takes
// 8 to 20 us on them, this one 3.3 to 12.6, the most with 127 users x 8 heads x 127 keys, where the tensor-core kernel takes
// 12.5).  Otherwise it competes with the warp-level tensor-core kernel,
// which costs 8 to 10 us before its first key but less per key: measured (device time, one column per kv head) 8 CTAs x 4 passes of
// 64 keys 6.0 us against 12, x 8 passes 9.4 against 14, 512 x 2 passes 8.4 against 9.5, 512 x 4 13.3 against 13, 2,048 x 2 23.7
// against 20.5; four columns: 32 CTAs x 4 passes 11.8 against 14, x 8 20 against 16, 512 x 1 9.7 against 10, 512 x 2 14.4 against 11.
bool short_preferred(const AttnArgs& a) {
    if (a.S < 128 && a.B * a.Hq * a.T < 1024) return true;
    const int64_t cols = (int64_t)(a.Hq / a.Hkv) * a.T, tile = cols == 1 ? 1 : (cols == 2 ? 2 : 4);
    const int64_t ctas = a.B * a.Hkv * ((cols + tile - 1) / tile), passes = (a.S + kShortKeys - 1) / kShortKeys;
    if (tile == 1) return passes <= 8 && ctas * passes <= 1024;
    if (tile == 2) return passes <= 6 && ctas * passes <= 768;
    return passes <= 4 && ctas * passes <= 512;
}

template <int DT, int C, ShortBuild BUILD>
static int32_t launch_short_build(const AttnArgs& a, cudaStream_t st) {
    const int64_t n_ctiles = ((int64_t)(a.Hq / a.Hkv) * a.T + C - 1) / C;
    qattn_short_kernel<DT, C, BUILD><<<(unsigned)(a.B * a.Hkv * n_ctiles), kShortThreads, 0, st>>>(a, (int)n_ctiles);
    return check_cuda(cudaGetLastError(), "qattn_short_kernel launch");
}

template <int DT, int C>
static int32_t launch_short_c(const AttnArgs& a, cudaStream_t st) {
    const LoraFold& L = a.lora;
    if (L.x && a.T == 1 && L.hidden == 128 && L.rank == 32 &&
        ((reinterpret_cast<uintptr_t>(L.x) | reinterpret_cast<uintptr_t>(L.a) | reinterpret_cast<uintptr_t>(L.b)) & 15) == 0)
        return launch_short_build<DT, C, kRank32>(a, st);
    if constexpr (C == 1)
        if (!L.x && a.B * a.Hkv > kFourPerSm) return launch_short_build<DT, 1, kNoUpdate>(a, st);
    return launch_short_build<DT, C, kAnyUpdate>(a, st);
}

template <int DT>
static int32_t launch_short_t(const AttnArgs& a, cudaStream_t st) {
    const int64_t cols = (int64_t)(a.Hq / a.Hkv) * a.T;
    if (cols == 1) return launch_short_c<DT, 1>(a, st);
    if (cols == 2) return launch_short_c<DT, 2>(a, st);
    return launch_short_c<DT, 4>(a, st);
}

int32_t launch_short(const AttnArgs& a, cudaStream_t st) {
    switch (a.q_dtype) {
        case OMNI_F32:  return launch_short_t<OMNI_F32>(a, st);
        case OMNI_BF16: return launch_short_t<OMNI_BF16>(a, st);
        case OMNI_F16:  return launch_short_t<OMNI_F16>(a, st);
    }
    return set_error(OMNI_ERR_ARG, "qattn: unknown q dtype code %d", a.q_dtype);
}

}  // namespace omni
