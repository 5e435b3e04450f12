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

// ---- ascending order within every group ---------------------------------------------------------------------------------
// Least-significant-digit radix sort of the fp32 samples of all groups at once, keys only, four passes of eight bits.  Each
// pass counts the digits of every chunk of kSortChunk samples, scans the counts of each (group, digit) over the group's
// chunks, and scatters the chunk stably: a warp takes 512 consecutive samples 32 at a time and ranks equal digits with eight
// ballots.  A library sort per group moves an 8-byte index with every key and costs 13 launches per group: 8 groups x 409,600
// samples 530 us of kernels behind 1.1 ms of host work, against 210 us here.
constexpr int kSortThreads = 256;
constexpr int kSortRounds = 16;
constexpr int kSortChunk = OMNI_SORT_CHUNK;
static_assert(kSortChunk == kSortThreads * kSortRounds, "a chunk is 16 rounds of every thread");

// fp32 order as unsigned order: -inf .. -0, +0 .. +inf, NaN (any sign) last.
__device__ __forceinline__ uint32_t sort_key(float x) {
    const uint32_t b = __float_as_uint(x);
    return x != x ? 0xFFFFFFFFu : (b >> 31 ? ~b : b | 0x80000000u);
}
__device__ __forceinline__ float sort_value(uint32_t k) { return __uint_as_float(k >> 31 ? k & 0x7FFFFFFFu : ~k); }

// Which group a chunk belongs to: the last g with chunk_base[g] <= chunk (groups are not empty).
__device__ __forceinline__ int group_of_chunk(const int64_t* chunk_base, int n_groups, int64_t chunk) {
    int lo = 0, hi = n_groups - 1;
    while (lo < hi) {
        const int mid = (lo + hi + 1) >> 1;
        if (chunk_base[mid] <= chunk) lo = mid; else hi = mid - 1;
    }
    return lo;
}

struct SortChunk { int group; int64_t first, end, counts; int n_chunks, index; };   // `counts`: first counter of the group
__device__ __forceinline__ SortChunk sort_chunk(const int64_t* group_off, const int64_t* chunk_base, int n_groups) {
    SortChunk c;
    c.group = group_of_chunk(chunk_base, n_groups, blockIdx.x);
    c.index = (int)(blockIdx.x - chunk_base[c.group]);
    c.n_chunks = (int)(chunk_base[c.group + 1] - chunk_base[c.group]);
    c.first = group_off[c.group] + (int64_t)c.index * kSortChunk;
    c.end = group_off[c.group + 1];
    c.counts = chunk_base[c.group] * 256;
    return c;
}
// lanes of the warp with the same digit as this one (lanes without a sample never match those with one)
__device__ __forceinline__ unsigned same_digit(uint32_t digit, bool have) {
    unsigned m = __ballot_sync(kFullMask, have);
    m = have ? m : ~m;
#pragma unroll
    for (int b = 0; b < 8; ++b) {
        const bool bit = (digit >> b) & 1u;
        const unsigned v = __ballot_sync(kFullMask, bit);
        m &= bit ? v : ~v;
    }
    return m;
}
template <bool FIRST>
__device__ __forceinline__ uint32_t load_key(const void* in, int64_t i) {
    return FIRST ? sort_key(__ldg(reinterpret_cast<const float*>(in) + i)) : __ldg(reinterpret_cast<const uint32_t*>(in) + i);
}

template <bool FIRST>
__global__ void __launch_bounds__(kSortThreads) sort_count_kernel(const void* in, const int64_t* group_off, const int64_t* chunk_base,
                                                                 int n_groups, int shift, uint32_t* counts) {
    __shared__ uint32_t hist[256];
    const SortChunk c = sort_chunk(group_off, chunk_base, n_groups);
    const int lane = threadIdx.x & 31;
    hist[threadIdx.x] = 0u;
    __syncthreads();
#pragma unroll 4
    for (int r = 0; r < kSortRounds; ++r) {
        const int64_t i = c.first + r * kSortThreads + threadIdx.x;
        const bool have = i < c.end;
        const uint32_t d = have ? (load_key<FIRST>(in, i) >> shift) & 255u : 0u;
        const unsigned m = same_digit(d, have);
        if (have && __ffs(m) - 1 == lane) atomicAdd(&hist[d], (uint32_t)__popc(m));
    }
    __syncthreads();
    counts[c.counts + (int64_t)threadIdx.x * c.n_chunks + c.index] = hist[threadIdx.x];
}

// One CTA per (group, digit): exclusive scan of the digit's counts over the group's chunks, in place; the total to `totals`.
__global__ void __launch_bounds__(kSortThreads) sort_scan_kernel(const int64_t* chunk_base, uint32_t* counts, uint32_t* totals) {
    __shared__ uint32_t warp_tot[kSortThreads / 32];
    const int g = blockIdx.x >> 8, digit = blockIdx.x & 255, lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int n = (int)(chunk_base[g + 1] - chunk_base[g]);
    uint32_t* p = counts + chunk_base[g] * 256 + (int64_t)digit * n;
    uint32_t run = 0u;
    for (int i0 = 0; i0 < n; i0 += kSortThreads) {
        const int i = i0 + threadIdx.x;
        const uint32_t v = i < n ? p[i] : 0u;
        uint32_t incl = v;
#pragma unroll
        for (int m = 1; m < 32; m <<= 1) {
            const uint32_t o = __shfl_up_sync(kFullMask, incl, m);
            if (lane >= m) incl += o;
        }
        if (lane == 31) warp_tot[warp] = incl;
        __syncthreads();
        uint32_t before = run;
        for (int w = 0; w < kSortThreads / 32; ++w) {
            if (w < warp) before += warp_tot[w];
            run += warp_tot[w];
        }
        if (i < n) p[i] = before + incl - v;
        __syncthreads();
    }
    if (threadIdx.x == 0) totals[blockIdx.x] = run;
}

template <bool FIRST, bool LAST>
__global__ void __launch_bounds__(kSortThreads) sort_scatter_kernel(const void* in, void* out, const int64_t* group_off,
                                                                   const int64_t* chunk_base, int n_groups, int shift,
                                                                   const uint32_t* counts, const uint32_t* totals) {
    __shared__ uint32_t place[kSortThreads / 32][256];       // per warp and digit: samples so far, then their first position
    __shared__ uint32_t warp_tot[kSortThreads / 32];
    const SortChunk c = sort_chunk(group_off, chunk_base, n_groups);
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    for (int i = threadIdx.x; i < kSortThreads / 32 * 256; i += kSortThreads) place[0][i] = 0u;
    // thread = digit: where the digit starts in the group
    const uint32_t total = totals[c.group * 256 + threadIdx.x];
    uint32_t incl = total;
#pragma unroll
    for (int m = 1; m < 32; m <<= 1) {
        const uint32_t o = __shfl_up_sync(kFullMask, incl, m);
        if (lane >= m) incl += o;
    }
    if (lane == 31) warp_tot[warp] = incl;
    __syncthreads();
    uint32_t start = incl - total + counts[c.counts + (int64_t)threadIdx.x * c.n_chunks + c.index];
    for (int w = 0; w < warp; ++w) start += warp_tot[w];
    // stable ranks within the warp's 512 consecutive samples
    uint32_t key[kSortRounds], rank[kSortRounds];
    const int64_t first = c.first + warp * (32 * kSortRounds) + lane;
#pragma unroll
    for (int r = 0; r < kSortRounds; ++r) key[r] = first + 32 * r < c.end ? load_key<FIRST>(in, first + 32 * r) : 0u;
#pragma unroll
    for (int r = 0; r < kSortRounds; ++r) {
        const bool have = first + 32 * r < c.end;
        const uint32_t d = (key[r] >> shift) & 255u;
        const unsigned m = same_digit(d, have);
        const uint32_t before = have ? place[warp][d] : 0u;
        __syncwarp();
        rank[r] = before + (uint32_t)__popc(m & ((1u << lane) - 1u));
        if (have && __ffs(m) - 1 == lane) place[warp][d] = before + (uint32_t)__popc(m);
        __syncwarp();
    }
    __syncthreads();
#pragma unroll
    for (int w = 0; w < kSortThreads / 32; ++w) {
        const uint32_t n = place[w][threadIdx.x];
        place[w][threadIdx.x] = start;
        start += n;
    }
    __syncthreads();
    const int64_t base = group_off[c.group];
#pragma unroll
    for (int r = 0; r < kSortRounds; ++r) {
        if (first + 32 * r < c.end) {
            const int64_t to = base + place[warp][(key[r] >> shift) & 255u] + rank[r];
            if (LAST) reinterpret_cast<float*>(out)[to] = sort_value(key[r]);
            else reinterpret_cast<uint32_t*>(out)[to] = key[r];
        }
    }
}

static size_t aligned256(size_t n) { return (n + 255) & ~(size_t)255; }

// The prefix sums run over all groups back to back, so they leave infinite and NaN samples out: in the sums they would turn
// every later group's means into NaN.  The group that holds them adds them to the cells they fall into.
__device__ __forceinline__ double finite_or_zero(float x) { return isfinite(x) ? (double)x : 0.0; }
__device__ __forceinline__ double if_not_finite(float x) { return isfinite(x) ? 0.0 : (double)x; }

// Pass 1: the fp64 sum of every chunk of kScanChunk samples.
__global__ void __launch_bounds__(kScanThreads) chunk_sums_kernel(const float* x, int64_t n, double* chunk_sum) {
    const int64_t base = (int64_t)blockIdx.x * kScanChunk;
    double s = 0.0;
    for (int j = 0; j < kScanPerThread; ++j) {
        const int64_t i = base + (int64_t)j * kScanThreads + threadIdx.x;     // coalesced
        if (i < n) s += finite_or_zero(x[i]);
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
        const float xj = first + 32 * j < n ? x[first + 32 * j] : 0.f;
        v[j] = isfinite(xj) ? xj : 0.f;
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

// One CTA per group.  Warp c searches the boundary above level c, 32 probes at a time: first the 32 positions around
// where its last move, repeated, would take it (moves shrink by a few per cent per iteration, so that is nearly always
// enough, and those lines are in L1 once the centroids have settled), then 32 positions 32 apart, then a 32-way search of what is left.  The prefix sums of the window are fetched
// together with its samples, so an iteration is one load latency, one exchange through shared memory and one division.  Every
// warp then updates all centroids redundantly (same operations, same bits), which saves a second barrier.
// What bounds it: that chain, 300 times (1.1 us each).  8 groups x 409,600 samples: 1,200 us with one warp per group whose lanes
// each ran a binary search (19 dependent loads and 16-level scans per iteration), 435 us with windows around the last place,
// 342 us with windows where the last move leads.  `calibrate_per_group` as a whole: 1,937 us, 1,176 us, 641 us with the sort
// above.
__global__ void __launch_bounds__(kLloydWarps * 32) lloyd_max_kernel(const float* sorted, const double* prefix, const int64_t* group_off,
                                                                    int max_iters, double tol, float* codebooks, int32_t* iters_out) {
    __shared__ __align__(16) float cent_s[kLloydWarps][kLevels];      // every warp's own copy
    __shared__ long long bound_s[2][kLevels + 1];                     // two buffers: one barrier per iteration
    __shared__ double pre_s[2][kLevels + 1];
    const int g = blockIdx.x, lane = threadIdx.x & 31, c = threadIdx.x >> 5;
    const int64_t lo = group_off[g], hi = group_off[g + 1], n = hi - lo;
    const int64_t per = n / kLevels;
    float* const cent = cent_s[c];
    // sorted in ascending order, NaN last: the ends tell whether every sample is finite
    const bool finite = isfinite(sorted[lo]) && isfinite(sorted[hi - 1]);
    // a range's mean; its infinite or NaN samples lie at its ends
    auto mean = [&](double sum, int64_t a, int64_t b) {
        if (!finite) sum += if_not_finite(sorted[a]) + if_not_finite(sorted[b - 1]);
        return (float)(sum / (double)(b - a));
    };
    // equal-mass initialisation: the mean of each sixteenth of the sorted sample
    float mine = 0.f;
    if (lane < kLevels) {
        const int64_t a = lo + lane * per, b = a + per;
        mine = mean(prefix[b] - prefix[a], a, b);
        cent[lane] = mine;
    }
    if (threadIdx.x < 2) {
        bound_s[threadIdx.x][0] = lo; pre_s[threadIdx.x][0] = prefix[lo];
        bound_s[threadIdx.x][kLevels] = hi; pre_s[threadIdx.x][kLevels] = prefix[hi];
    }
    __syncthreads();
    int64_t at = lo + (c + 1) * per, step = 0;                       // this warp's boundary and its last move
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
                const int64_t was = at;
                int64_t base = at + step - 16;                       // moves shrink by a few per cent per iteration
                base = base < lo - 16 ? lo - 16 : (base > hi - 16 ? hi - 16 : base);
                const int64_t near = base + lane;
                const double pre_near = prefix[near < lo ? lo : (near > hi ? hi : near)];
                const unsigned m = probe(base, 1);
                if (m != 0u && !(m & 1u)) {
                    const int j = __ffs(m) - 1;
                    at = base + j;
                    pre = __shfl_sync(kFullMask, pre_near, j);
                } else {
                    // answer in [a, b]: everything before a is below, b is above (or hi)
                    int64_t a = m == 0u ? base + 32 : lo, b = m == 0u ? hi : (base < hi ? (base > lo ? base : lo) : hi);
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
                step = at - was;
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
                const float fresh = mean(pre_s[buf][lane + 1] - pre_s[buf][lane], a, b);
                moved = fabsf(fresh - mine);
                mine = fresh;
            }
            cent[lane] = mine;
        }
        // moves are not negative, so they order like their bits (a NaN, from infinite samples, does not count as a move)
        moved = __uint_as_float(__reduce_max_sync(kFullMask, moved == moved ? __float_as_uint(moved) : 0u));
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

extern "C" size_t omni_sort_groups_workspace_bytes(int64_t n_total, int32_t n_groups, int64_t n_chunks) {
    if (n_total <= 0 || n_groups <= 0 || n_chunks <= 0) return 0;
    return aligned256((size_t)n_total * 4) + aligned256((size_t)n_chunks * 1024) + (size_t)n_groups * 1024;
}

extern "C" int32_t omni_sort_groups(const float* samples, int64_t n_total, const int64_t* group_offsets, const int64_t* chunk_base,
                                    int32_t n_groups, int64_t n_chunks, void* workspace, size_t workspace_bytes, float* sorted, void* stream) {
    OMNI_REQUIRE(n_groups >= 0 && n_total >= 0 && n_chunks >= 0, OMNI_ERR_ARG, "omni_sort_groups: negative extent");
    if (n_groups == 0 || n_total == 0) return OMNI_OK;
    OMNI_REQUIRE(samples && group_offsets && chunk_base && workspace && sorted && sorted != samples, OMNI_ERR_ARG, "omni_sort_groups: NULL or aliased buffer");
    OMNI_REQUIRE(n_total <= 0x7fffffffLL && n_groups <= 0x7fffff, OMNI_ERR_UNSUPPORTED, "omni_sort_groups: %lld samples in %d groups exceed 32-bit positions",
                 (long long)n_total, n_groups);
    OMNI_REQUIRE(n_chunks >= n_groups && n_chunks <= n_total, OMNI_ERR_ARG, "omni_sort_groups: %lld chunks for %d groups of %lld samples", (long long)n_chunks,
                 n_groups, (long long)n_total);
    const size_t need = omni_sort_groups_workspace_bytes(n_total, n_groups, n_chunks);
    OMNI_REQUIRE(workspace_bytes >= need && reinterpret_cast<uintptr_t>(workspace) % 8 == 0, OMNI_ERR_ARG,
                 "omni_sort_groups: workspace of %zu bytes needed, got %zu", need, workspace_bytes);
    cudaStream_t st = (cudaStream_t)stream;
    uint32_t* spare = (uint32_t*)workspace;
    uint32_t* counts = (uint32_t*)((char*)workspace + aligned256((size_t)n_total * 4));
    uint32_t* totals = (uint32_t*)((char*)counts + aligned256((size_t)n_chunks * 1024));
    const void* from[4] = {samples, spare, sorted, spare};
    void* to[4] = {spare, sorted, spare, sorted};
    const unsigned grid = (unsigned)n_chunks;
    for (int pass = 0; pass < 4; ++pass) {
        const int shift = 8 * pass;
        if (pass == 0) sort_count_kernel<true><<<grid, kSortThreads, 0, st>>>(from[pass], group_offsets, chunk_base, n_groups, shift, counts);
        else           sort_count_kernel<false><<<grid, kSortThreads, 0, st>>>(from[pass], group_offsets, chunk_base, n_groups, shift, counts);
        sort_scan_kernel<<<(unsigned)n_groups * 256u, kSortThreads, 0, st>>>(chunk_base, counts, totals);
        if (pass == 0)      sort_scatter_kernel<true, false><<<grid, kSortThreads, 0, st>>>(from[pass], to[pass], group_offsets, chunk_base, n_groups, shift, counts, totals);
        else if (pass == 3) sort_scatter_kernel<false, true><<<grid, kSortThreads, 0, st>>>(from[pass], to[pass], group_offsets, chunk_base, n_groups, shift, counts, totals);
        else                sort_scatter_kernel<false, false><<<grid, kSortThreads, 0, st>>>(from[pass], to[pass], group_offsets, chunk_base, n_groups, shift, counts, totals);
    }
    return check_cuda(cudaGetLastError(), "sort kernels launch");
}
