// Lloyd-Max fit of the 16-level codebooks on the GPU (the reference's offline calibration,
// quantization/codebook.py:64-108 `LloydMaxCalibrator.fit`, :148-172 `calibrate_per_group`).
//
// The reference assigns every sample to its nearest centroid (first-index argmin of |x - c| in fp32) and
// replaces each centroid by the mean of its samples, up to 300 times.  With the samples SORTED the cell of
// centroid c is a contiguous range of the array, so one iteration needs only the 15 cell boundaries (a search
// each, with the reference's own fp32 comparison as the predicate) and the range sums, which come from
// an fp64 prefix-sum array as a difference.  An iteration therefore costs a few loads per boundary instead of a pass
// over n x 16 distances, and the whole loop (initialisation, iterations, convergence test, final sort) runs in
// one launch with one CTA per group, without a host round trip.
//
// Means are formed in fp64 from the prefix sums and rounded to fp32 once; the reference sums in fp32 in an
// order its tensor library chooses, so codebooks agree with it to a few fp32 ulps, not bit for bit.
#include "common.cuh"

namespace omni {

constexpr int kScanThreads = 256;
constexpr int kScanPerThread = 32;
constexpr int kScanChunk = kScanThreads * kScanPerThread;   // samples per CTA of the prefix-sum kernels
constexpr int kLevels = 16;

__device__ __forceinline__ double warp_inclusive_scan(double v, int lane) {
#pragma unroll
    for (int m = 1; m < 32; m <<= 1) {
        const double o = __shfl_up_sync(kFullMask, v, m);
        if (lane >= m) v += o;
    }
    return v;
}

// Inclusive scan of one value per thread over a CTA of kScanThreads; returns the CTA total through *total.
__device__ __forceinline__ double block_inclusive_scan(double v, double* total) {
    __shared__ double warp_tot[kScanThreads / 32];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    v = warp_inclusive_scan(v, lane);
    if (lane == 31) warp_tot[warp] = v;
    __syncthreads();
    double before = 0.0, all = 0.0;
#pragma unroll
    for (int w = 0; w < kScanThreads / 32; ++w) {
        if (w < warp) before += warp_tot[w];
        all += warp_tot[w];
    }
    __syncthreads();
    *total = all;
    return v + before;
}

// Pass 1: the fp64 sum of every chunk of kScanChunk samples.
__global__ void __launch_bounds__(kScanThreads) chunk_sums_kernel(const float* x, int64_t n, double* chunk_sum) {
    const int64_t base = (int64_t)blockIdx.x * kScanChunk;
    double s = 0.0;
    for (int j = 0; j < kScanPerThread; ++j) {
        const int64_t i = base + (int64_t)j * kScanThreads + threadIdx.x;     // coalesced
        if (i < n) s += (double)x[i];
    }
    double total;
    block_inclusive_scan(s, &total);
    if (threadIdx.x == 0) chunk_sum[blockIdx.x] = total;
}

// Pass 2: exclusive scan of the chunk sums in place (one CTA; each thread owns a contiguous run).
__global__ void __launch_bounds__(kScanThreads) scan_chunk_sums_kernel(double* chunk_sum, int64_t n_chunks) {
    const int64_t per = (n_chunks + kScanThreads - 1) / kScanThreads;
    const int64_t lo = (int64_t)threadIdx.x * per;
    const int64_t hi = lo + per < n_chunks ? lo + per : n_chunks;
    double s = 0.0;
    for (int64_t i = lo; i < hi; ++i) s += chunk_sum[i];
    double total;
    const double incl = block_inclusive_scan(s, &total);
    double run = incl - s;
    for (int64_t i = lo; i < hi; ++i) {
        const double v = chunk_sum[i];
        chunk_sum[i] = run;
        run += v;
    }
}

// Pass 3: prefix[i] = sum of x[0..i) for i in [0, n].  A warp owns 1,024 consecutive samples and takes them 32 at a time,
// so every load and store of a warp is one contiguous run (a thread with 32 consecutive samples of its own touched 32
// separate lines per instruction).
__global__ void __launch_bounds__(kScanThreads) write_prefix_kernel(const float* x, int64_t n, const double* chunk_off,
                                                                   double* prefix) {
    __shared__ double warp_tot[kScanThreads / 32];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int64_t first = (int64_t)blockIdx.x * kScanChunk + (int64_t)warp * (32 * kScanPerThread) + lane;
    float v[kScanPerThread];
    double s = 0.0;
#pragma unroll
    for (int j = 0; j < kScanPerThread; ++j) {
        v[j] = first + 32 * j < n ? x[first + 32 * j] : 0.f;
        s += (double)v[j];
    }
#pragma unroll
    for (int m = 16; m >= 1; m >>= 1) s += __shfl_xor_sync(kFullMask, s, m);
    if (lane == 0) warp_tot[warp] = s;
    __syncthreads();
    double run = chunk_off[blockIdx.x];
    for (int w = 0; w < warp; ++w) run += warp_tot[w];
#pragma unroll
    for (int j = 0; j < kScanPerThread; ++j) {
        const double incl = warp_inclusive_scan((double)v[j], lane);
        if (first + 32 * j <= n) prefix[first + 32 * j] = run + (incl - (double)v[j]);
        run += __shfl_sync(kFullMask, incl, 31);
    }
}

// The reference's assignment: index of the first smallest |x - c| over the 16 centroids, in fp32.
__device__ __forceinline__ int nearest_level(float x, const float* cent) {
    float best = fabsf(x - cent[0]);
    int idx = 0;
#pragma unroll
    for (int k = 1; k < kLevels; ++k) {
        const float d = fabsf(x - cent[k]);
        if (d < best) { best = d; idx = k; }
    }
    return idx;
}

// Boundary search.  Cell boundary c (between levels c and c + 1) is the first position of the sorted group whose sample is
// assigned to a level above c.  While the samples are finite the centroids stay in ascending order (each is the mean of a
// range of the sorted array, and an empty cell's centroid lies between its neighbours' midpoints), so for x >= cent[c]
// the closest of the levels 0..c is c itself (rounding is monotone), and below cent[c] no higher level can be strictly closer:
//     level(x) > c   <=>   x >= cent[c]  and  min_{k > c} |x - cent[k]| < |x - cent[c]|
// with the reference's own fp32 distances.  For x <= cent[c+1] the minimum is the distance to c + 1; farther levels are
// looked at only by samples beyond it that tie with c (equal or nearly equal centroids).
__device__ __forceinline__ bool above_level(float x, int c, float cl, float cr, const float* cent) {
    const float dl = fabsf(x - cl);
    bool above = x >= cl && fabsf(x - cr) < dl;
    if (__any_sync(kFullMask, !above && x > cr)) {
        for (int k = c + 2; k < kLevels; ++k) above = above || (x > cr && fabsf(x - cent[k]) < dl);
    }
    return above;
}

constexpr int kLloydWarps = kLevels;      // one warp per boundary (the last one only takes part in the updates)

// One CTA per group.  Warp c searches the boundary above level c, 32 probes at a time: first the 32 positions around its
// place in the previous iteration (centroids move by a few samples per iteration once they have settled, and those lines are
// in L1), then 32 positions 32 apart, then a 32-way search of what is left.  The prefix sums of the window are fetched
// together with its samples, so an iteration is one load latency, one exchange through shared memory and one division.  Every
// warp then updates all centroids redundantly (same operations, same bits), which saves a second barrier.
// What bounds it: that chain, 300 times.  `calibrate_per_group` of 8 groups x 409,600 samples, sorts included: 1,937 us with
// one warp per group whose lanes each ran a binary search (19 dependent loads and 16-level scans per iteration), 1,176 us now.
__global__ void __launch_bounds__(kLloydWarps * 32) lloyd_max_kernel(const float* sorted, const double* prefix, const int64_t* group_off,
                                                                    int max_iters, double tol, float* codebooks, int32_t* iters_out) {
    __shared__ __align__(16) float cent_s[kLloydWarps][kLevels];      // every warp's own copy
    __shared__ long long bound_s[2][kLevels + 1];                     // two buffers: one barrier per iteration
    __shared__ double pre_s[2][kLevels + 1];
    const int g = blockIdx.x, lane = threadIdx.x & 31, c = threadIdx.x >> 5;
    const int64_t lo = group_off[g], hi = group_off[g + 1], n = hi - lo;
    const int64_t per = n / kLevels;
    float* const cent = cent_s[c];
    // equal-mass initialisation: the mean of each sixteenth of the sorted sample
    float mine = 0.f;
    if (lane < kLevels) {
        const int64_t a = lo + lane * per, b = a + per;
        mine = (float)((prefix[b] - prefix[a]) / (double)per);
        cent[lane] = mine;
    }
    if (threadIdx.x < 2) {
        bound_s[threadIdx.x][0] = lo; pre_s[threadIdx.x][0] = prefix[lo];
        bound_s[threadIdx.x][kLevels] = hi; pre_s[threadIdx.x][kLevels] = prefix[hi];
    }
    __syncthreads();
    // sorted in ascending order, NaN last: the ends tell whether every sample is finite
    const bool finite = isfinite(sorted[lo]) && isfinite(sorted[hi - 1]);
    int64_t at = lo + (c + 1) * per;                                 // this warp's boundary
    int steps = 0;
    for (int64_t span = n; span > 0; span >>= 1) ++steps;            // enough halvings for a range of n + 1 positions
    int it = 0;
    for (; it < max_iters; ++it) {
        const int buf = it & 1;
        if (c < kLevels - 1) {
            double pre;
            if (finite) {
                const float cl = cent[c], cr = cent[c + 1];
                // probes lane 0..31 at from + stride * lane; a position before lo counts as below, one from hi on as above
                auto probe = [&](int64_t from, int64_t stride) -> unsigned {
                    const int64_t pos = from + stride * lane;
                    const bool in = pos >= lo && pos < hi;
                    const float x = sorted[in ? pos : lo];
                    const bool above = above_level(x, c, cl, cr, cent);
                    return __ballot_sync(kFullMask, pos >= lo && (pos >= hi || above));
                };
                const int64_t base = at - 16, near = base + lane;
                const double pre_near = prefix[near < lo ? lo : (near > hi ? hi : near)];
                const unsigned m = probe(base, 1);
                if (m != 0u && !(m & 1u)) {
                    const int j = __ffs(m) - 1;
                    at = base + j;
                    pre = __shfl_sync(kFullMask, pre_near, j);
                } else {
                    // answer in [a, b]: everything before a is below, b is above (or hi)
                    int64_t a = m == 0u ? base + 32 : lo, b = m == 0u ? hi : (base < hi ? base : hi);
                    {
                        const int64_t from = m == 0u ? a : b - 32 * 31;
                        const unsigned w = probe(from, 32);          // clear below the answer, set from it on
                        if (w != 0u) { const int64_t q = from + 32 * (int64_t)(__ffs(w) - 1); b = q < b ? q : b; }
                        if (!(w & 1u)) {
                            const int64_t q = from + 32 * (int64_t)(w == 0u ? 31 : __ffs(w) - 2);
                            a = q + 1 > a ? q + 1 : a;
                        }
                    }
                    while (b > a) {
                        const int64_t stride = (b - a + 31) >> 5;
                        const unsigned w = probe(a, stride);
                        if (w == 0u) { const int64_t q = a + 31 * stride + 1; a = q < b ? q : b; }
                        else {
                            const int j = __ffs(w) - 1;
                            const int64_t q = a + stride * j;
                            b = q < b ? q : b;
                            if (j > 0) a = q - stride + 1; else a = b;
                        }
                    }
                    at = a < b ? a : b;
                    pre = prefix[at];
                }
            } else {
                // infinite or NaN samples: a plain binary search with the reference's scan (nothing is known about order)
                int64_t a = lo, b = hi;
                for (int s = 0; s < steps && a < b; ++s) {
                    const int64_t mid = a + ((b - a) >> 1);
                    if (nearest_level(sorted[mid], cent) > c) b = mid; else a = mid + 1;
                }
                at = a;
                pre = prefix[at];
            }
            if (lane == 0) { bound_s[buf][c + 1] = at; pre_s[buf][c + 1] = pre; }
        }
        __syncthreads();
        float moved = 0.f;
        if (lane < kLevels) {
            const int64_t a = bound_s[buf][lane], b = bound_s[buf][lane + 1];
            if (b > a) {                                             // an empty cell keeps its centroid
                const float fresh = (float)((pre_s[buf][lane + 1] - pre_s[buf][lane]) / (double)(b - a));
                moved = fabsf(fresh - mine);
                mine = fresh;
            }
            cent[lane] = mine;
        }
#pragma unroll
        for (int m = 16; m >= 1; m >>= 1) moved = fmaxf(moved, __shfl_xor_sync(kFullMask, moved, m));
        __syncwarp();
        if ((double)moved < tol) { ++it; break; }                    // the same in every warp
    }
    if (c != 0) return;
    if (lane == 0) {
        for (int i = 1; i < kLevels; ++i) {                          // ascending order for the codec's search
            const float v = cent[i];
            int j = i - 1;
            while (j >= 0 && cent[j] > v) { cent[j + 1] = cent[j]; --j; }
            cent[j + 1] = v;
        }
        if (iters_out) iters_out[g] = it;
    }
    __syncwarp();
    if (lane < kLevels) codebooks[(int64_t)g * kLevels + lane] = cent[lane];
}

static int64_t n_chunks_of(int64_t n) { return (n + 1 + kScanChunk - 1) / kScanChunk; }
static size_t prefix_bytes(int64_t n) { return (((size_t)(n + 1) * sizeof(double)) + 255) & ~(size_t)255; }

}  // namespace omni

using namespace omni;

extern "C" size_t omni_lloyd_max_workspace_bytes(int64_t n_total) {
    if (n_total <= 0) return 0;
    return prefix_bytes(n_total) + (size_t)n_chunks_of(n_total) * sizeof(double);
}

extern "C" int32_t omni_lloyd_max_fit(const float* sorted, int64_t n_total, const int64_t* group_offsets, int32_t n_groups,
                                      int32_t max_iters, double tol, void* workspace, size_t workspace_bytes,
                                      float* codebooks, int32_t* iters_out, void* stream) {
    OMNI_REQUIRE(n_groups >= 0 && n_total >= 0 && max_iters >= 0, OMNI_ERR_ARG, "omni_lloyd_max_fit: bad extent");
    if (n_groups == 0) return OMNI_OK;
    OMNI_REQUIRE(sorted && group_offsets && codebooks && workspace, OMNI_ERR_ARG, "omni_lloyd_max_fit: NULL buffer");
    OMNI_REQUIRE(n_total >= (int64_t)n_groups * kLevels, OMNI_ERR_ARG,
                 "omni_lloyd_max_fit: every group needs at least %d samples", kLevels);
    OMNI_REQUIRE(workspace_bytes >= omni_lloyd_max_workspace_bytes(n_total) && reinterpret_cast<uintptr_t>(workspace) % 8 == 0, OMNI_ERR_ARG,
                 "omni_lloyd_max_fit: workspace of %zu bytes needed, got %zu", omni_lloyd_max_workspace_bytes(n_total),
                 workspace_bytes);
    const int64_t chunks = n_chunks_of(n_total);
    OMNI_REQUIRE(chunks <= 0x7fffffffLL, OMNI_ERR_UNSUPPORTED, "omni_lloyd_max_fit: too many samples for one grid");
    cudaStream_t st = (cudaStream_t)stream;
    double* prefix = (double*)workspace;
    double* chunk_sum = (double*)((char*)workspace + prefix_bytes(n_total));
    chunk_sums_kernel<<<(unsigned)chunks, kScanThreads, 0, st>>>(sorted, n_total, chunk_sum);
    scan_chunk_sums_kernel<<<1, kScanThreads, 0, st>>>(chunk_sum, chunks);
    write_prefix_kernel<<<(unsigned)chunks, kScanThreads, 0, st>>>(sorted, n_total, chunk_sum, prefix);
    lloyd_max_kernel<<<(unsigned)n_groups, kLloydWarps * 32, 0, st>>>(sorted, prefix, group_offsets, max_iters, tol, codebooks, iters_out);
    return check_cuda(cudaGetLastError(), "lloyd_max kernels launch");
}
