// Fast rotate + quantize kernel of the KV-cache codec (sm_100a).
//
// Layout: a warp takes 8 consecutive tokens of one (user, head) at a time; row r of the group is
// owned by lanes 4r..4r+3 and lane t of those holds the 32 contiguous elements d = 32t..32t+31.
//   * rotation: five butterfly stages inside the thread, two across lanes (xor 1, xor 2), in the
//     reference's stage order h = 1..64 with one rounding per add/subtract (the cross-lane stages use
//     fma(+-1, mine, partner), which rounds exactly like the add or subtract it replaces);
//   * INT4 code: a 32-cell uniform grid over the threshold range gives a base code, one exact fp32
//     threshold compare settles base / base+1.  Thresholds and cell bases are derived per codebook at
//     kernel start by bisection against the defining first-index argmin of |y - c|, so the result is
//     the reference's code bit for bit; inputs outside the range where that shortcut is proven
//     (|y| beyond `guard`, or a codebook the grid cannot resolve) take the defining scan instead;
//   * QJL sign bits: the residual row is scaled by a power of two to 15-bit integers and split into a
//     signed high and an unsigned low byte; the 64 x 128 +-1 projection runs on the int8 tensor cores
//     (mma.sync m16n8k32, G as the A operand, the 8 rows as the 8 columns of B).  The integer sum
//     differs from the exact scaled sum by at most 64, so |sum| > 64 decides the sign rigorously; the
//     few projections inside that band are recomputed exactly in fp64;
//   * packed outputs: 16-byte nibble stores per lane (64 contiguous bytes per row), 2-byte sign stores.
#include "codec_fast.cuh"
#include <mutex>
#include <utility>
#include <vector>
#include <cstdlib>

namespace omni {

constexpr int kFqWarps = 8;
constexpr int kFqMaxHeads = 32;

// Per-head quantiser tables in shared memory.  The cell records come first and the struct is 256-byte aligned, so
// that (byte offset of a cell) | (address of the table) addresses a record without an add.
struct alignas(256) HeadTables {
    float2 cell2[32];       // per grid cell: x = threshold between the cell's two codes, y = the lower code (int bits)
    float thr[20];          // thr[c], c = 1..15: smallest fp32 y whose code is >= c; thr[16] = +inf
    float cb[16];
    float inv32, off32;     // cell(y): see cell_offset
    float guard;            // |y| <= guard: the threshold shortcut is valid
    int valid;              // 0: this codebook always takes the defining scan; 1: grid cell + one compare;
                            // 2: binary search over the 15 exact thresholds (the grid cannot resolve them)
};
static_assert(sizeof(HeadTables) % 16 == 0, "HeadTables must keep 16-byte alignment in an array");

__device__ __forceinline__ int order_key(float x) {           // monotone float -> int
    const int b = __float_as_int(x);
    return b >= 0 ? b : (int)(0x80000000u - (uint32_t)b);
}
__device__ __forceinline__ float order_unkey(int k) {
    return __int_as_float(k >= 0 ? k : (int)(0x80000000u - (uint32_t)k));
}
// the reference's code: first index minimising |y - c| in fp32
__device__ __forceinline__ int code_by_scan(float y, const float* cb) {
    float best = fabsf(__fsub_rn(y, cb[0]));
    int code = 0;
#pragma unroll
    for (int c = 1; c < 16; ++c) {
        const float d = fabsf(__fsub_rn(y, cb[c]));
        if (d < best) { best = d; code = c; }
    }
    return code;
}
// Grid cell of y as the byte offset of its 8-byte record: with u = sat(y * inv32 + off32) in [0, 1], the low mantissa
// bits of fma(u, 248, 1.5 * 2^23) hold j = rn(248 u) in [0, 248]; j & 0xF8 = 8 * (j >> 3), cell j >> 3 in [0, 31].
// Any monotone cell function serves: the records are derived from the function itself (build_head_tables).
__device__ __forceinline__ uint32_t cell_offset(float y, float inv32, float off32) {
    const float u = __saturatef(fmaf(y, inv32, off32));
    return __float_as_uint(fmaf(u, 248.f, 12582912.f)) & 0xF8u;
}
__device__ __forceinline__ int cell_of(float y, float inv32, float off32) { return (int)(cell_offset(y, inv32, off32) >> 3); }

// One warp derives the tables of one codebook (lane = grid cell, lanes 1..15 also own a threshold).
__device__ void build_head_tables(HeadTables& ht, const float* cb_global, int lane) {
    if (lane < 16) ht.cb[lane] = __ldg(cb_global + lane);
    __syncwarp();
    const float c_me = ht.cb[lane & 15], c_prev = ht.cb[(lane + 15) & 15];
    const bool ordered = (lane == 0 || lane >= 16) ? true : (c_me > c_prev);
    const bool finite = isfinite(c_me);
    float gap = (lane >= 1 && lane < 16) ? c_me - c_prev : INFINITY;
#pragma unroll
    for (int m = 16; m >= 1; m >>= 1) gap = fminf(gap, __shfl_xor_sync(kFullMask, gap, m));
    const float maxabs = fmaxf(fabsf(ht.cb[0]), fabsf(ht.cb[15]));
    const float guard = gap * 1048576.f;
    bool ok = __all_sync(kFullMask, ordered && finite) && gap > 0.f;
    if (!ok) {                                       // uniform: every element of this head is scanned
        if (lane == 0) { ht.valid = 0; ht.guard = -1.f; ht.inv32 = 0.f; ht.off32 = 0.f; }
        __syncwarp();
        return;
    }
    // thresholds: bisection between cb[c-1] (code c-1) and cb[c] (code c).  Inside that bracket the nearest of the levels
    // 0..c-1 is c-1 and the nearest of the levels c..15 is c (fp32 rounding is monotone), so "code >= c" is one strict
    // comparison of two distances instead of the 16-level scan.
    if (lane >= 1 && lane < 16) {
        int lo = order_key(c_prev), hi = order_key(c_me);
        while ((int64_t)hi - lo > 1) {
            const int mid = (int)(((int64_t)lo + hi) >> 1);
            const float y = order_unkey(mid);
            if (fabsf(__fsub_rn(y, c_me)) < fabsf(__fsub_rn(y, c_prev))) hi = mid; else lo = mid;
        }
        ht.thr[lane] = order_unkey(hi);
    }
    if (lane == 16) ht.thr[16] = INFINITY;
    if (lane == 0) ht.thr[0] = -INFINITY;
    __syncwarp();
    if (!(isfinite(guard) && guard >= 4.f * maxabs)) {   // uniform: gaps too small for the grid, thresholds still exact
        if (lane == 0) { ht.valid = 2; ht.guard = 3.0e38f; ht.inv32 = 0.f; ht.off32 = 0.f; }
        __syncwarp();
        return;
    }
    const float t1 = ht.thr[1], t15 = ht.thr[15];
    const float margin = (t15 - t1) * (1.f / 29.f);
    const float lo_y = t1 - margin, hi_y = t15 + margin;
    const float inv32 = 1.f / (hi_y - lo_y), off32 = -lo_y * inv32;
    // cell u: a = smallest y in [-guard, guard] with cell_of(y) >= u; its code is the cell's base
    float a = -guard;
    if (lane > 0) {
        int lo = order_key(-guard), hi = order_key(guard);          // cell(lo) = 0 < lane <= cell(hi) = 31
        while ((int64_t)hi - lo > 1) {                               // the key range spans more than 2^31
            const int mid = (int)(((int64_t)lo + hi) >> 1);
            if (cell_of(order_unkey(mid), inv32, off32) >= lane) hi = mid; else lo = mid;
        }
        a = order_unkey(hi);
    }
    const int base = code_by_scan(a, ht.cb);
    // last y of the cell = predecessor of the next cell's first y (guard for the last cell)
    const float a_next = __shfl_down_sync(kFullMask, a, 1);
    const float b = (lane == 31) ? guard : order_unkey(order_key(a_next) - 1);
    const int top = code_by_scan(b, ht.cb);
    ok = __all_sync(kFullMask, top - base <= 1 && top >= base) &&
         cell_of(-guard, inv32, off32) == 0 && cell_of(guard, inv32, off32) == 31;
    ht.cell2[lane] = make_float2(ht.thr[base + 1], __int_as_float(base));
    // A grid that cannot separate the thresholds (two of them in one cell) leaves the exact thresholds usable
    // by themselves: such codebooks take the four-step binary search, for every finite y.
    if (lane == 0) { ht.valid = ok ? 1 : 2; ht.guard = ok ? guard : 3.0e38f; ht.inv32 = inv32; ht.off32 = off32; }
    __syncwarp();
}

// ---- small PTX helpers ------------------------------------------------------------------------
// Packed fp32 pairs (sm_100): one instruction rounds both halves exactly like the scalar add / fma would, at half
// the issue slots.  (ax, ay) op (bx, by) -> (dx, dy).
__device__ __forceinline__ void add2(float& dx, float& dy, float ax, float ay, float bx, float by) {
    asm("{\n .reg .b64 ra, rb, rd;\n mov.b64 ra, {%2, %3};\n mov.b64 rb, {%4, %5};\n add.rn.f32x2 rd, ra, rb;\n"
        " mov.b64 {%0, %1}, rd;\n}\n" : "=f"(dx), "=f"(dy) : "f"(ax), "f"(ay), "f"(bx), "f"(by));
}
__device__ __forceinline__ void fma2(float& dx, float& dy, float ax, float ay, float bx, float by, float cx, float cy) {
    asm("{\n .reg .b64 ra, rb, rc, rd;\n mov.b64 ra, {%2, %3};\n mov.b64 rb, {%4, %5};\n mov.b64 rc, {%6, %7};\n"
        " fma.rn.f32x2 rd, ra, rb, rc;\n mov.b64 {%0, %1}, rd;\n}\n"
        : "=f"(dx), "=f"(dy) : "f"(ax), "f"(ay), "f"(bx), "f"(by), "f"(cx), "f"(cy));
}
__device__ __forceinline__ void mul2(float& dx, float& dy, float ax, float ay, float bx, float by) {
    asm("{\n .reg .b64 ra, rb, rd;\n mov.b64 ra, {%2, %3};\n mov.b64 rb, {%4, %5};\n mul.rn.f32x2 rd, ra, rb;\n"
        " mov.b64 {%0, %1}, rd;\n}\n" : "=f"(dx), "=f"(dy) : "f"(ax), "f"(ay), "f"(bx), "f"(by));
}
__device__ __forceinline__ uint32_t prmt_sign_bytes(uint32_t x) {     // each byte -> 0xFF if its MSB is set, else 0x00
    uint32_t r;
    asm("prmt.b32 %0, %1, %1, 0xBA98;\n" : "=r"(r) : "r"(x));
    return r;
}
// four int8 of +-1 from 4 bits of a Rademacher row: bit 1 -> +1, bit 0 -> -1 (bits at LOW..LOW+3 of w)
template <int LOW>
__device__ __forceinline__ uint32_t pm1_bytes(uint32_t w) {
    const uint32_t spread = (~w & (0xFu << LOW)) * (LOW == 0 ? 0x10204080u : 0x01020408u);
    return prmt_sign_bytes(spread) | 0x01010101u;
}
__device__ __forceinline__ void imma_s8s8(int (&c)[4], const uint4& a, uint32_t b0, uint32_t b1) {
    asm("mma.sync.aligned.m16n8k32.row.col.s32.s8.s8.s32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};\n"
        : "+r"(c[0]), "+r"(c[1]), "+r"(c[2]), "+r"(c[3]) : "r"(a.x), "r"(a.y), "r"(a.z), "r"(a.w), "r"(b0), "r"(b1));
}
__device__ __forceinline__ void imma_s8u8(int (&c)[4], const uint4& a, uint32_t b0, uint32_t b1) {
    asm("mma.sync.aligned.m16n8k32.row.col.s32.s8.u8.s32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};\n"
        : "+r"(c[0]), "+r"(c[1]), "+r"(c[2]), "+r"(c[3]) : "r"(a.x), "r"(a.y), "r"(a.z), "r"(a.w), "r"(b0), "r"(b1));
}
// gather the bits at positions 4k + s (k = 0..7) of w into one byte
__device__ __forceinline__ uint32_t every_fourth_bit(uint32_t w, int s) {
    uint32_t x = (w >> s) & 0x11111111u;
    x = (x | (x >> 3)) & 0x03030303u;
    x = (x | (x >> 6)) & 0x000F000Fu;
    x = (x | (x >> 12)) & 0xFFu;
    return x;
}

// 32 consecutive elements of a row, staged as 16-byte chunks and unpacked to fp32
template <int DT> struct Row32;
template <> struct Row32<OMNI_F32> {
    static constexpr int kChunks = 8;
    static __device__ __forceinline__ const char* addr(const void* p, int64_t i) { return reinterpret_cast<const char*>(reinterpret_cast<const float*>(p) + i); }
    static __device__ __forceinline__ void unpack(const uint4 (&c)[8], float (&y)[32]) {
#pragma unroll
        for (int k = 0; k < 8; ++k) {
            y[4 * k] = __uint_as_float(c[k].x); y[4 * k + 1] = __uint_as_float(c[k].y);
            y[4 * k + 2] = __uint_as_float(c[k].z); y[4 * k + 3] = __uint_as_float(c[k].w);
        }
    }
    static __device__ __forceinline__ void round_pair(float& a, float& b) {}
    static __device__ __forceinline__ void pack(const float (&y)[32], uint4 (&c)[8]) {
#pragma unroll
        for (int k = 0; k < 8; ++k)
            c[k] = make_uint4(__float_as_uint(y[4 * k]), __float_as_uint(y[4 * k + 1]), __float_as_uint(y[4 * k + 2]), __float_as_uint(y[4 * k + 3]));
    }
};
template <> struct Row32<OMNI_BF16> {
    static constexpr int kChunks = 4;
    static __device__ __forceinline__ const char* addr(const void* p, int64_t i) { return reinterpret_cast<const char*>(reinterpret_cast<const __nv_bfloat16*>(p) + i); }
    static __device__ __forceinline__ void unpack(const uint4 (&c)[4], float (&y)[32]) {
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            const uint32_t w[4] = {c[k].x, c[k].y, c[k].z, c[k].w};
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                y[8 * k + 2 * j] = __uint_as_float(w[j] << 16);
                y[8 * k + 2 * j + 1] = __uint_as_float(w[j] & 0xffff0000u);
            }
        }
    }
    static __device__ __forceinline__ void round_pair(float& a, float& b) {
        const __nv_bfloat162 h = __floats2bfloat162_rn(a, b);
        const uint32_t w = *reinterpret_cast<const uint32_t*>(&h);
        a = __uint_as_float(w << 16); b = __uint_as_float(w & 0xffff0000u);
    }
    static __device__ __forceinline__ void pack(const float (&y)[32], uint4 (&c)[4]) {
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            uint32_t w[4];
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                const __nv_bfloat162 h = __floats2bfloat162_rn(y[8 * k + 2 * j], y[8 * k + 2 * j + 1]);
                w[j] = *reinterpret_cast<const uint32_t*>(&h);
            }
            c[k] = make_uint4(w[0], w[1], w[2], w[3]);
        }
    }
};
template <> struct Row32<OMNI_F16> {
    static constexpr int kChunks = 4;
    static __device__ __forceinline__ const char* addr(const void* p, int64_t i) { return reinterpret_cast<const char*>(reinterpret_cast<const __half*>(p) + i); }
    static __device__ __forceinline__ void unpack(const uint4 (&c)[4], float (&y)[32]) {
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            const uint32_t w[4] = {c[k].x, c[k].y, c[k].z, c[k].w};
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                const float2 f = __half22float2(*reinterpret_cast<const __half2*>(&w[j]));
                y[8 * k + 2 * j] = f.x; y[8 * k + 2 * j + 1] = f.y;
            }
        }
    }
    static __device__ __forceinline__ void round_pair(float& a, float& b) {
        const float2 f = __half22float2(__floats2half2_rn(a, b));
        a = f.x; b = f.y;
    }
    static __device__ __forceinline__ void pack(const float (&y)[32], uint4 (&c)[4]) {
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            uint32_t w[4];
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                const __half2 h = __floats2half2_rn(y[8 * k + 2 * j], y[8 * k + 2 * j + 1]);
                w[j] = *reinterpret_cast<const uint32_t*>(&h);
            }
            c[k] = make_uint4(w[0], w[1], w[2], w[3]);
        }
    }
};

// Normalised 128-point Walsh-Hadamard transform of a row held by four lanes (lane t = elements 32t .. 32t+31),
// in the reference's stage order with one rounding per add / subtract; the result is not yet rounded to the
// element type.
__device__ __forceinline__ void rotate_row32(float (&y)[32], int t) {
    // elements i and i + 16 travel as a packed pair through every stage but h = 16; u - v is fma(v, -1, u),
    // which rounds exactly like the subtraction
#pragma unroll
    for (int hh = 1; hh < 16; hh <<= 1) {
#pragma unroll
        for (int i = 0; i < 16; ++i) {
            if ((i & hh) == 0) {
                const float u0 = y[i], u1 = y[i + 16], v0 = y[i | hh], v1 = y[(i | hh) + 16];
                add2(y[i], y[i + 16], u0, u1, v0, v1);
                fma2(y[i | hh], y[(i | hh) + 16], v0, v1, -1.f, -1.f, u0, u1);
            }
        }
    }
#pragma unroll
    for (int i = 0; i < 16; ++i) {
        const float u = y[i], v = y[i + 16];
        y[i] = __fadd_rn(u, v);
        y[i + 16] = __fsub_rn(u, v);
    }
    // the two stages across the row's four lanes: fma(+-1, mine, partner) rounds like the add / subtract
#pragma unroll
    for (int m = 1; m <= 2; m <<= 1) {
        const float sgn = (t & m) ? -1.f : 1.f;
#pragma unroll
        for (int i = 0; i < 16; ++i) {
            const float o0 = __shfl_xor_sync(kFullMask, y[i], m), o1 = __shfl_xor_sync(kFullMask, y[i + 16], m);
            fma2(y[i], y[i + 16], sgn, sgn, y[i], y[i + 16], o0, o1);
        }
    }
    const float sc = __uint_as_float(OMNI_WHT_SCALE_BITS);
#pragma unroll
    for (int i = 0; i < 16; ++i) mul2(y[i], y[i + 16], y[i], y[i + 16], sc, sc);
}

// Input staging: a lane copies its 32 elements of the NEXT 8-token group into shared memory with cp.async while
// the current group is being processed, so the global-memory latency is off the critical path.  Layout per warp
// and buffer: chunk k of lane l at (k * 32 + l) * 16 bytes (conflict-free 16-byte reads).
constexpr int kStageChunks = 8;                                     // room for the widest element type
constexpr int kStageBytesPerWarp = kStageChunks * 32 * 16;          // one buffer: it is refilled as soon as it is read
constexpr int kBallotBytesPerWarp = 64;                             // the 16 sign ballots of a group, handed from lane 0 to the lanes
__device__ __forceinline__ void cp_async16(uint32_t dst, const void* src) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" :: "r"(dst), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_async_wait_all() { asm volatile("cp.async.wait_all;\n" ::: "memory"); }
__device__ __forceinline__ float2 lds_f2(uint32_t addr) {              // tables that no longer change once built
    float2 v;
    asm("ld.shared.v2.f32 {%0,%1}, [%2];\n" : "=f"(v.x), "=f"(v.y) : "r"(addr));
    return v;
}
__device__ __forceinline__ void sts_u4(uint32_t addr, uint32_t a, uint32_t b, uint32_t c, uint32_t d) {
    asm volatile("st.shared.v4.u32 [%0], {%1,%2,%3,%4};\n" :: "r"(addr), "r"(a), "r"(b), "r"(c), "r"(d) : "memory");
}
__device__ __forceinline__ uint2 lds_u2(uint32_t addr) {
    uint2 v;
    asm volatile("ld.shared.v2.u32 {%0,%1}, [%2];\n" : "=r"(v.x), "=r"(v.y) : "r"(addr) : "memory");
    return v;
}
__device__ __forceinline__ uint4 lds_u4(uint32_t addr) {
    uint4 v;
    asm volatile("ld.shared.v4.u32 {%0,%1,%2,%3}, [%4];\n" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "r"(addr));
    return v;
}
template <int DT>
__device__ __forceinline__ void stage_row(uint32_t buf, const void* x, int64_t i) {
    const char* src = Row32<DT>::addr(x, i);
#pragma unroll
    for (int k = 0; k < Row32<DT>::kChunks; ++k) cp_async16(buf + k * 512, src + 16 * k);
}

// SIGNS = false: only the nibble rows are produced (a.qjl and a.norms are null): V rows of a cache whose attention
// never reads their sign bits or norms skip the projections altogether.
// TWO = false: one job, whose arguments are constants of the launch (indexed by block they cost a large call 1 %).
template <int DT, bool ROTATE, bool SIGNS, bool TWO>
__global__ void __launch_bounds__(kFqWarps * 32, 2) fast_quantize_kernel(const __grid_constant__ FastQuantJobs jobs) {
    extern __shared__ __align__(256) unsigned char fq_smem[];
    const FastQuantArgs& a = jobs.job[TWO ? blockIdx.y : 0];
    const int n_tabs = a.cb_per_head ? a.H : 1;
    HeadTables* tabs = reinterpret_cast<HeadTables*>(fq_smem);
    uint4* gfrag_all = reinterpret_cast<uint4*>(fq_smem + sizeof(HeadTables) * n_tabs);
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int g = lane >> 2, t = lane & 3;
    uint4* gfrag = gfrag_all + (size_t)warp * 16 * 32 + lane;      // this lane's 16 A fragments, 32 uint4 apart
    const uint32_t stage = (uint32_t)__cvta_generic_to_shared(gfrag_all + (size_t)kFqWarps * 16 * 32) +
                           warp * kStageBytesPerWarp + lane * 16;  // this lane's chunk 0 of buffer 0
    // sign ballots of a group: written by lane 0 as [m-tile][column parity][half], read back by lane (g, t) as the
    // pair (m-tile t, parity g & 1, halves 0 and 1)
    const uint32_t ballots = (uint32_t)__cvta_generic_to_shared(gfrag_all + (size_t)kFqWarps * 16 * 32) +
                             kFqWarps * kStageBytesPerWarp + warp * kBallotBytesPerWarp;
    const uint32_t my_ballots = ballots + (uint32_t)(t * 4 + (g & 1) * 2) * 4;

    // The 8-token groups of all (user, head) pairs, in order, are dealt out in equal consecutive shares, one per warp of the
    // grid: a warp's share may begin and end inside a pair.  A whole pair per warp left the last round of a large call
    // mostly empty and all but 8 warps of a one-user call idle: K and V of 1,024 users x 8 heads x 256 tokens (3.46 pairs
    // per warp, so 4 rounds) 989 us against 862 us, 256 x 8 x 203 fp32 rows with their rotation 202 against 187 us.
    const int T = (int)a.T;                                          // fast_quantize_eligible: groups and tokens fit 32 bits
    const uint32_t gpp = (uint32_t)(T + 7) >> 3;                     // groups of one pair
    uint32_t gi, last;
    {
        const uint64_t n_groups = (uint64_t)(a.B * a.H) * gpp, n_warps = (uint64_t)gridDim.x * kFqWarps;
        const uint64_t wid = (uint64_t)blockIdx.x * kFqWarps + warp, w0 = wid - warp;
        gi = (uint32_t)(n_groups * wid / n_warps);
        last = (uint32_t)(n_groups * (wid + 1) / n_warps);
        // the codebooks of the heads this block's shares touch
        const uint64_t p0 = n_groups * w0 / n_warps / gpp, p1 = (n_groups * (w0 + kFqWarps) / n_warps + gpp - 1) / gpp;
        const int need = a.cb_per_head ? (p1 - p0 < (uint64_t)a.H ? (int)(p1 - p0) : a.H) : (p1 > p0);
        for (int i = warp; i < need; i += kFqWarps) {
            const int h = a.cb_per_head ? (int)((p0 + i) % a.H) : 0;
            build_head_tables(tabs[h], a.codebooks + h * 16, lane);
        }
    }
    __syncthreads();

    while (gi < last) {
        const uint32_t p = gi / gpp;
        const int t_begin = (int)(gi - p * gpp) * 8;
        const int t_end = (last - gi) < gpp && (int)(t_begin + (last - gi) * 8) < T ? (int)(t_begin + (last - gi) * 8) : T;
        gi = (p + 1) * gpp;
        const int64_t b = p / (uint32_t)a.H;
        const int h = (int)(p % (uint32_t)a.H);
        const int32_t uid = a.user_ids ? a.user_ids[b] : a.user_id;
        const int seed = seed_of(uid, h);
        const uint32_t* grow = a.g_rows + (size_t)seed * kQjlDim * 4;
        // A fragments of G for this lane: m-tile mt (16 projections), k-step ks (8 of this lane's dims)
#pragma unroll
        for (int mt = 0; SIGNS && mt < 4; ++mt) {
            const uint32_t w0 = __ldg(grow + (16 * mt + g) * 4 + t), w1 = __ldg(grow + (16 * mt + g + 8) * 4 + t);
#pragma unroll
            for (int ks = 0; ks < 4; ++ks) {
                const uint32_t b0 = w0 >> (8 * ks), b1 = w1 >> (8 * ks);
                gfrag[(mt * 4 + ks) * 32] = make_uint4(pm1_bytes<0>(b0), pm1_bytes<0>(b1), pm1_bytes<4>(b0), pm1_bytes<4>(b1));
            }
        }
        const HeadTables& ht = tabs[a.cb_per_head ? h : 0];
        const float inv32 = ht.inv32, off32 = ht.off32, guard = ht.guard;
        const uint32_t cell_base = (uint32_t)__cvta_generic_to_shared(ht.cell2);        // 256-byte aligned
        const int64_t in_base = b * a.xs_b + (int64_t)h * a.xs_h + 32 * t;
        const int64_t out_base = b * a.os_b + (int64_t)h * a.os_h + (a.out_offsets ? a.out_offsets[b] : a.out_offset);

        // rows past the end of a group are clamped to the last token (computed, never stored)
        stage_row<DT>(stage, a.x, in_base + (t_begin + g < T ? t_begin + g : T - 1) * a.xs_t);
        for (int t0 = t_begin; t0 < t_end; t0 += 8) {
            const int tr = t0 + g;
            const bool active = tr < T;
            cp_async_wait_all();
            float y[32];
            {
                uint4 c[Row32<DT>::kChunks];
#pragma unroll
                for (int k = 0; k < Row32<DT>::kChunks; ++k) c[k] = lds_u4(stage + k * 512);
                if (t0 + 8 < t_end) {               // the chunks are in registers: refill the buffer with the next group
                    const int tn = tr + 8;
                    stage_row<DT>(stage, a.x, in_base + (tn < T ? tn : T - 1) * a.xs_t);
                }
                Row32<DT>::unpack(c, y);
            }
            if (ROTATE) {
                rotate_row32(y, t);
#pragma unroll
                for (int i = 0; i < 32; i += 2) Row32<DT>::round_pair(y[i], y[i + 1]);
            }
            // ---- INT4 codes and residual (y becomes the residual) ---------------------------------
            float amax = 0.f;
#pragma unroll
            for (int i = 0; i < 32; ++i) amax = fmaxf(amax, fabsf(y[i]));
            uint32_t codes[4] = {0u, 0u, 0u, 0u};
            if (__any_sync(kFullMask, !(amax <= guard))) {
#pragma unroll
                for (int i = 0; i < 32; ++i) {
                    const int c = code_by_scan(y[i], ht.cb);
                    codes[i >> 3] |= (uint32_t)c << (4 * (i & 7));
                    y[i] = __fsub_rn(y[i], ht.cb[c]);
                }
            } else if (ht.valid == 2) {
#pragma unroll
                for (int i = 0; i < 32; ++i) {                 // code = number of thresholds thr[1..15] that are <= y
                    int c = (y[i] >= ht.thr[8]) ? 8 : 0;
                    c += (y[i] >= ht.thr[c + 4]) ? 4 : 0;
                    c += (y[i] >= ht.thr[c + 2]) ? 2 : 0;
                    c += (y[i] >= ht.thr[c + 1]) ? 1 : 0;
                    codes[i >> 3] |= (uint32_t)c << (4 * (i & 7));
                    y[i] = __fsub_rn(y[i], ht.cb[c]);
                }
            } else {
#pragma unroll
                for (int q = 0; q < 4; ++q) {
                    uint32_t word = 0u;
#pragma unroll
                    for (int k = 7; k >= 0; --k) {                 // last element first: element 8q ends in the low nibble
                        const int i = 8 * q + k;
                        const float2 rec = lds_f2(cell_offset(y[i], inv32, off32) | cell_base);
                        const int c = __float_as_int(rec.y) + (y[i] >= rec.x ? 1 : 0);
                        word = word * 16u + (uint32_t)c;
                        y[i] = __fsub_rn(y[i], ht.cb[c]);
                    }
                    codes[q] = word;
                }
            }
            if (!SIGNS) {
                if (active)
                    *reinterpret_cast<uint4*>(a.nib + (out_base + tr) * kNibBytes + 16 * t) = make_uint4(codes[0], codes[1], codes[2], codes[3]);
                continue;
            }
            // ---- residual norm and fixed-point scale ------------------------------------------------
            float ss = 0.f, emax = 0.f;
            {
                float sa = 0.f, sb = 0.f;
#pragma unroll
                for (int i = 0; i < 16; ++i) {
                    fma2(sa, sb, y[i], y[i + 16], y[i], y[i + 16], sa, sb);
                    emax = fmaxf(emax, fmaxf(fabsf(y[i]), fabsf(y[i + 16])));
                }
                ss = sa + sb;
            }
            ss += __shfl_xor_sync(kFullMask, ss, 1);   ss += __shfl_xor_sync(kFullMask, ss, 2);
            emax = fmaxf(emax, __shfl_xor_sync(kFullMask, emax, 1));
            emax = fmaxf(emax, __shfl_xor_sync(kFullMask, emax, 2));
            const int E = (__float_as_uint(emax) >> 23) & 0xFF;
            // rows whose largest residual is 0 / tiny / inf, or that hold a NaN (then the sum of squares is not
            // finite), cannot be scaled to integers: all their signs are recomputed exactly
            const bool degenerate = (E < 16) || (E == 255) || !(ss < INFINITY);
            // scale = 2^(141-E) * (1 - 2^-9): emax * scale lies in [2^14 - 32, 2^15 - 64), so the rounded integers fit int16.
            // The scale need not be a power of two: the fused multiply-add below rounds e*scale + magic once.
            const float scale = degenerate ? 0.f : __uint_as_float(((uint32_t)(267 - E) << 23) | 0x7F8000u);
            // ---- projections on the int8 tensor cores -------------------------------------------------
            // The low-limb accumulators start at 64, so that sum64 = 256 * hi + lo is the integer sum plus 64: the
            // sign test is sum64 >= 64 and the undecided band |sum| <= 64 is one unsigned compare, sum64 <= 128.
            int chi[4][4], clo[4][4];
#pragma unroll
            for (int mt = 0; mt < 4; ++mt)
#pragma unroll
                for (int j = 0; j < 4; ++j) { chi[mt][j] = 0; clo[mt][j] = 64; }
#pragma unroll
            for (int kp = 0; kp < 2; ++kp) {
                // k-steps kp and kp + 2 together: their elements i and i + 16 are the packed pairs of the rotation
                float va[8], vb[8];
#pragma unroll
                for (int k = 0; k < 8; ++k)                                                // low 16 bits = int16
                    fma2(va[k], vb[k], y[8 * kp + k], y[8 * kp + k + 16], scale, scale, 12582912.f, 12582912.f);
#pragma unroll
                for (int half = 0; half < 2; ++half) {
                    const int ks = kp + 2 * half;
                    uint32_t v[8];
#pragma unroll
                    for (int k = 0; k < 8; ++k) v[k] = __float_as_uint(half ? vb[k] : va[k]);
                    const uint32_t p01 = __byte_perm(v[0], v[1], 0x5140), p23 = __byte_perm(v[2], v[3], 0x5140);
                    const uint32_t p45 = __byte_perm(v[4], v[5], 0x5140), p67 = __byte_perm(v[6], v[7], 0x5140);
                    const uint32_t lo0 = __byte_perm(p01, p23, 0x5410), hi0 = __byte_perm(p01, p23, 0x7632);
                    const uint32_t lo1 = __byte_perm(p45, p67, 0x5410), hi1 = __byte_perm(p45, p67, 0x7632);
#pragma unroll
                    for (int mt = 0; mt < 4; ++mt) {
                        const uint4 af = gfrag[(mt * 4 + ks) * 32];
                        imma_s8s8(chi[mt], af, hi0, hi1);
                        imma_s8u8(clo[mt], af, lo0, lo1);
                    }
                }
            }
            // ---- sign / ambiguity bits: C element (mt, j) = projection 16mt + g + 8(j>>1) of row 2t + (j&1) ----
            // Ballot words are warp-uniform; lane (row g, quarter t) needs those of m-tile t, column parity g & 1,
            // halves 0 and 1, and keeps them as the m-tiles go by.
            // Sign ballots are warp-uniform; lane (row g, quarter t) needs those of m-tile t, column parity g & 1,
            // halves 0 and 1: lane 0 leaves all sixteen in shared memory and every lane reads its pair.  A projection
            // inside the band, or a row that could not be scaled, is rare: one vote tells whether the group has any,
            // and only then are the sixteen ambiguity ballots taken.
            bool undecided = degenerate;
#pragma unroll
            for (int mt = 0; mt < 4; ++mt) {
                uint32_t sgn[4];
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    const int sum64 = chi[mt][j] * 256 + clo[mt][j];
                    sgn[j] = __ballot_sync(kFullMask, sum64 >= 64);
                    undecided = undecided || ((uint32_t)sum64 <= 128u);
                }
                if (lane == 0) sts_u4(ballots + 16 * mt, sgn[0], sgn[2], sgn[1], sgn[3]);
            }
            __syncwarp();
            const uint2 wsp = lds_u2(my_ballots);
            const uint32_t ws0 = wsp.x, ws1 = wsp.y;
            __syncwarp();                                       // the ballots are read before the next group overwrites them
            const int sh = g >> 1;                              // the C owner of this row's columns has t'' = g >> 1
            uint32_t bits16 = every_fourth_bit(ws0, sh) | (every_fourth_bit(ws1, sh) << 8);
            if (__any_sync(kFullMask, undecided)) {
                const bool deg0 = __shfl_sync(kFullMask, (int)degenerate, 8 * t) != 0;         // row 2t   (lanes 8t..)
                const bool deg1 = __shfl_sync(kFullMask, (int)degenerate, 8 * t + 4) != 0;     // row 2t+1
                const bool odd = (g & 1) != 0;
                uint32_t wa0 = 0u, wa1 = 0u;
#pragma unroll
                for (int mt = 0; mt < 4; ++mt) {
                    uint32_t ba[4];
#pragma unroll
                    for (int j = 0; j < 4; ++j) {
                        const int sum64 = chi[mt][j] * 256 + clo[mt][j];
                        ba[j] = __ballot_sync(kFullMask, (uint32_t)sum64 <= 128u || ((j & 1) ? deg1 : deg0));
                    }
                    const bool mine = (t == mt);
                    wa0 = mine ? (odd ? ba[1] : ba[0]) : wa0; wa1 = mine ? (odd ? ba[3] : ba[2]) : wa1;
                }
                uint32_t amb16 = every_fourth_bit(wa0, sh) | (every_fourth_bit(wa1, sh) << 8);
                if (!active) amb16 = 0u;
                // ---- recomputation of the undecided projections, one per row at a time.  First in fp32: four running sums of
                // eight signed residuals each, added up over the row's lanes, are off by at most 12 roundings of partial sums
                // no larger than 128 emax, 12 * 2^-24 * 128 emax < 1e-4 emax, so a larger result has the exact sum's sign; the
                // few that are not (3 in 64 of the undecided), and rows that could not be scaled, go to fp64.  (Every undecided
                // projection in fp64, a chain of 32 conversions and adds: prefill of 1,024 users x 8 heads x 256 tokens 862 us
                // against 842 us.)
                uint64_t pending = (uint64_t)__shfl_sync(kFullMask, amb16, 4 * g) |
                                   ((uint64_t)__shfl_sync(kFullMask, amb16, 4 * g + 1) << 16) |
                                   ((uint64_t)__shfl_sync(kFullMask, amb16, 4 * g + 2) << 32) |
                                   ((uint64_t)__shfl_sync(kFullMask, amb16, 4 * g + 3) << 48);
                const float sure = degenerate ? INFINITY : emax * 1e-4f;
                uint64_t close = 0ull;
                while (__any_sync(kFullMask, pending != 0ull)) {
                    const bool have = pending != 0ull;
                    const int pi = have ? __ffsll((long long)pending) - 1 : 0;
                    if (have) pending &= pending - 1ull;
                    const uint32_t flip = ~__ldg(grow + pi * 4 + t);
                    float p[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
                    for (int i = 0; i < 32; ++i) p[i & 3] += __uint_as_float(__float_as_uint(y[i]) ^ ((flip << (31 - i)) & 0x80000000u));
                    float acc = (p[0] + p[1]) + (p[2] + p[3]);
                    acc += __shfl_xor_sync(kFullMask, acc, 1);
                    acc += __shfl_xor_sync(kFullMask, acc, 2);
                    if (have && !(fabsf(acc) > sure)) close |= 1ull << pi;
                    if (have && t == (pi >> 4)) {
                        const uint32_t m = 1u << (pi & 15);
                        bits16 = (acc >= 0.f) ? (bits16 | m) : (bits16 & ~m);
                    }
                }
                while (__any_sync(kFullMask, close != 0ull)) {
                    const bool have = close != 0ull;
                    const int pi = have ? __ffsll((long long)close) - 1 : 0;
                    if (have) close &= close - 1ull;
                    const uint32_t gw = __ldg(grow + pi * 4 + t);
                    double acc = 0.0;
#pragma unroll
                    for (int i = 0; i < 32; ++i) { const double ev = (double)y[i]; acc += ((gw >> i) & 1u) ? ev : -ev; }
                    acc += __shfl_xor_sync(kFullMask, acc, 1);
                    acc += __shfl_xor_sync(kFullMask, acc, 2);
                    if (have && t == (pi >> 4)) {
                        const uint32_t m = 1u << (pi & 15);
                        bits16 = (acc >= 0.0) ? (bits16 | m) : (bits16 & ~m);
                    }
                }
            }
            // ---- stores ----------------------------------------------------------------------------------
            if (active) {
                const int64_t ro = out_base + tr;
                *reinterpret_cast<uint4*>(a.nib + ro * kNibBytes + 16 * t) = make_uint4(codes[0], codes[1], codes[2], codes[3]);
                *reinterpret_cast<uint16_t*>(a.qjl + ro * kQjlBytes + 2 * t) = (uint16_t)bits16;
                if (t == 0) a.norms[ro] = sqrtf(ss);
            }
        }
    }
}

// The same transform of a row whose 16-byte chunks are dealt to its four lanes in turn: chunk 4 m + t is y[E m .. E m + E - 1]
// of lane t (E elements per chunk), so the stages below E are inside the thread, the next two across lanes and the rest
// inside the thread again -- the reference's order h = 1 .. 64, one rounding per add / subtract.
template <int E>
__device__ __forceinline__ void rotate_row32_chunked(float (&y)[32], int t) {
    auto stage = [&](int hh) {                                    // elements i and i + 16 as packed pairs
#pragma unroll
        for (int i = 0; i < 16; ++i) {
            if ((i & hh) == 0) {
                const float u0 = y[i], u1 = y[i + 16], v0 = y[i | hh], v1 = y[(i | hh) + 16];
                add2(y[i], y[i + 16], u0, u1, v0, v1);
                fma2(y[i | hh], y[(i | hh) + 16], v0, v1, -1.f, -1.f, u0, u1);
            }
        }
    };
#pragma unroll
    for (int hh = 1; hh < E; hh <<= 1) stage(hh);
#pragma unroll
    for (int m = 1; m <= 2; m <<= 1) {
        const float sgn = (t & m) ? -1.f : 1.f;
#pragma unroll
        for (int i = 0; i < 16; ++i) {
            const float o0 = __shfl_xor_sync(kFullMask, y[i], m), o1 = __shfl_xor_sync(kFullMask, y[i + 16], m);
            fma2(y[i], y[i + 16], sgn, sgn, y[i], y[i + 16], o0, o1);
        }
    }
#pragma unroll
    for (int hh = E; hh < 16; hh <<= 1) stage(hh);
    const float sc = __uint_as_float(OMNI_WHT_SCALE_BITS);
#pragma unroll
    for (int i = 0; i < 16; ++i) {
        const float u = y[i], v = y[i + 16];
        mul2(y[i], y[i + 16], __fadd_rn(u, v), __fsub_rn(u, v), sc, sc);
    }
}

// Stand-alone rotation, 8 rows per warp, 4 lanes per row: two cross-lane stages instead of five, which matters for 16-bit
// rows, where the warp-per-row kernel is bound by shuffle throughput.  A row's lanes take its 16-byte chunks in turn, so an
// access of the warp touches 64 consecutive bytes of each row (with 64 consecutive bytes per LANE it touched 16 lines for
// the same 512 bytes and L1 was the limit: 1,048,576 bf16 rows 107 us against 85 us, 94 % of the copy peak).
template <int DT>
__global__ void __launch_bounds__(kFqWarps * 32) fast_rotate_kernel(const void* x, void* y_out, int64_t n_rows) {
    constexpr int kChunks = Row32<DT>::kChunks, E = 32 / kChunks;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int g = lane >> 2, t = lane & 3;
    const int64_t n_groups = (n_rows + 7) / 8;
    for (int64_t grp = (int64_t)blockIdx.x * kFqWarps + warp; grp < n_groups; grp += (int64_t)gridDim.x * kFqWarps) {
        const int64_t row = grp * 8 + g;
        const bool active = row < n_rows;
        const int64_t rc = active ? row : n_rows - 1;
        uint4 c[kChunks];
        const uint4* src = reinterpret_cast<const uint4*>(Row32<DT>::addr(x, rc * kHeadDim)) + t;
#pragma unroll
        for (int k = 0; k < kChunks; ++k) c[k] = __ldg(src + 4 * k);
        float y[32];
        Row32<DT>::unpack(c, y);
        rotate_row32_chunked<E>(y, t);
        Row32<DT>::pack(y, c);
        if (active) {
            uint4* dst = reinterpret_cast<uint4*>(const_cast<char*>(Row32<DT>::addr(y_out, rc * kHeadDim))) + t;
#pragma unroll
            for (int k = 0; k < kChunks; ++k) dst[4 * k] = c[k];
        }
    }
}

int32_t launch_fast_rotate(const void* x, void* y, int64_t n_rows, int dtype, cudaStream_t st) {
    int64_t blocks = ((n_rows + 7) / 8 + kFqWarps - 1) / kFqWarps;
    if (blocks > 148 * 16) blocks = 148 * 16;
    if (blocks < 1) blocks = 1;
    switch (dtype) {
        case OMNI_F32:  fast_rotate_kernel<OMNI_F32><<<(unsigned)blocks, kFqWarps * 32, 0, st>>>(x, y, n_rows); break;
        case OMNI_BF16: fast_rotate_kernel<OMNI_BF16><<<(unsigned)blocks, kFqWarps * 32, 0, st>>>(x, y, n_rows); break;
        case OMNI_F16:  fast_rotate_kernel<OMNI_F16><<<(unsigned)blocks, kFqWarps * 32, 0, st>>>(x, y, n_rows); break;
        default: return set_error(OMNI_ERR_ARG, "omni_rotate: unknown dtype code %d", dtype);
    }
    return check_cuda(cudaGetLastError(), "fast_rotate_kernel launch");
}

}  // namespace omni
#include "codec_tc.cuh"
namespace omni {

// ---- host side ------------------------------------------------------------------------------------
static bool fq_aligned(const void* p, size_t n) { return (reinterpret_cast<uintptr_t>(p) % n) == 0; }

// true when the fast kernel covers this call (shape, alignment); the caller falls back otherwise
bool fast_quantize_eligible(const FastQuantArgs& a, int dtype) {
    const int64_t esz = dtype == OMNI_F32 ? 4 : 2;
    const int64_t vec = 16 / esz;
    if (a.cb_per_head && a.H > kFqMaxHeads) return false;
    if (!fq_aligned(a.x, 16) || a.xs_b % vec || a.xs_h % vec || a.xs_t % vec) return false;
    if (!fq_aligned(a.nib, 16) || !fq_aligned(a.qjl, 2)) return false;
    if ((a.qjl == nullptr) != (a.norms == nullptr)) return false;
    // token and group numbers of the kernel are 32-bit (every row's packed bytes would not fit a GPU's memory sooner)
    return a.T > 0 && a.T <= 0x7ffffff0LL && a.B * a.H * ((a.T + 7) >> 3) < 0xffffffffLL;
}

// One launch for one call, or for two calls of the same extents (keys and values of one append): grid.y = jobs.
template <int DT, bool TWO>
static int32_t launch_fast_t(const FastQuantArgs* jobs, int n_jobs, int rotate, cudaStream_t st) {
    const FastQuantArgs& a = jobs[0];
    int dev = 0, sms = 148;
    OMNI_CUDA(cudaGetDevice(&dev));
    OMNI_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
    const int n_tabs = a.cb_per_head ? a.H : 1;
    const size_t smem = sizeof(HeadTables) * n_tabs + (size_t)kFqWarps * 16 * 32 * sizeof(uint4) +
                        (size_t)kFqWarps * (kStageBytesPerWarp + kBallotBytesPerWarp);
    const int64_t groups = a.B * a.H * ((a.T + 7) >> 3);
    // two resident CTAs per SM, over both jobs while these have no more groups than warps (a second wave would build its
    // tables after the first one's work: K and V of one token for 64 users x 8 heads 20.6 us against 12.0 us); fewer groups than warps are spread over the SMs, one group per warp
    const int64_t most = n_jobs * groups <= 2 * sms * kFqWarps ? 2 * sms / n_jobs : 2 * sms;
    const int64_t blocks = groups < most ? groups : most;
    const bool signs = a.qjl != nullptr;
    auto kern = signs ? (rotate ? fast_quantize_kernel<DT, true, true, TWO> : fast_quantize_kernel<DT, false, true, TWO>)
                      : (rotate ? fast_quantize_kernel<DT, true, false, TWO> : fast_quantize_kernel<DT, false, false, TWO>);
    {   // opt in once per (kernel, device) to the shared memory of the largest table count the kernel accepts
        static std::mutex mu;
        static std::vector<std::pair<const void*, int>> done;
        const void* key = reinterpret_cast<const void*>(kern);
        std::lock_guard<std::mutex> lk(mu);
        bool seen = false;
        for (const auto& p : done) seen = seen || (p.first == key && p.second == dev);
        if (!seen) {
            const size_t smem_max = sizeof(HeadTables) * kFqMaxHeads + (size_t)kFqWarps * 16 * 32 * sizeof(uint4) +
                                    (size_t)kFqWarps * (kStageBytesPerWarp + kBallotBytesPerWarp);
            OMNI_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem_max));
            done.emplace_back(key, dev);
        }
    }
    FastQuantJobs j;
    j.job[0] = jobs[0];
    j.job[1] = jobs[n_jobs - 1];
    kern<<<dim3((unsigned)blocks, (unsigned)n_jobs), kFqWarps * 32, smem, st>>>(j);
    return check_cuda(cudaGetLastError(), "fast_quantize_kernel launch");
}

// Row-per-thread kernel with tensor-memory projections: calls with at least 64 tokens per (user, head), whose
// 128-token tiles are reasonably full.  OMNI_QUANT_KERNEL=warp keeps such calls on the warp-cooperative kernel, =tc
// sends every eligible call here (tests and profiling).
static bool use_tc_kernel(const FastQuantArgs& a) {
    if (!fq_aligned(a.qjl, 8)) return false;
    const char* e = getenv("OMNI_QUANT_KERNEL");
    if (e && e[0] == 't') return true;
    // Measured (1,048,576 bf16 rows): 398 us here against 298 us for the warp-cooperative kernel -- 127 warp
    // instructions per row instead of 172, but a straight-line body of some 4,000 instructions per row that the
    // instruction cache cannot hold (the top stall is "no instruction") on eight warps per SM.  The warp-cooperative
    // kernel therefore stays the default; this one is kept selectable and under the same tests.
    return false;
}

int32_t launch_fast_quantize(const FastQuantArgs& a, int dtype, int rotate, cudaStream_t st) {
    if (use_tc_kernel(a)) {
        switch (dtype) {
            case OMNI_F32:  return launch_tc_t<OMNI_F32>(a, rotate, st);
            case OMNI_BF16: return launch_tc_t<OMNI_BF16>(a, rotate, st);
            case OMNI_F16:  return launch_tc_t<OMNI_F16>(a, rotate, st);
        }
    }
    return launch_fast_quantize_jobs(&a, 1, dtype, rotate, st);
}

int32_t launch_fast_quantize_jobs(const FastQuantArgs* jobs, int n_jobs, int dtype, int rotate, cudaStream_t st) {
    switch (dtype) {
        case OMNI_F32:  return n_jobs == 2 ? launch_fast_t<OMNI_F32, true>(jobs, 2, rotate, st) : launch_fast_t<OMNI_F32, false>(jobs, 1, rotate, st);
        case OMNI_BF16: return n_jobs == 2 ? launch_fast_t<OMNI_BF16, true>(jobs, 2, rotate, st) : launch_fast_t<OMNI_BF16, false>(jobs, 1, rotate, st);
        case OMNI_F16:  return n_jobs == 2 ? launch_fast_t<OMNI_F16, true>(jobs, 2, rotate, st) : launch_fast_t<OMNI_F16, false>(jobs, 1, rotate, st);
    }
    return set_error(OMNI_ERR_ARG, "unknown dtype code %d", dtype);
}

}  // namespace omni
