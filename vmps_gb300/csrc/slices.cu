// FP64 grouped GEMM on the tensor cores by slices (sm_103a).
//
// GB300's FP64 pipe does two FMAs per clock and SM; tcgen05 does 4096 bf16 ones.
// A splitting (the scheme of Ozaki, Ogita, Oishi and Rump, 2012) turns an FP64
// product into sums of bf16 products without rounding: with E the exponent of a
// panel row's largest element, every element is rounded to an integer multiple
// of 2^(E-61) and written as seven signed base-512 digits,
//     x = 2^(E-7) sum_s d_s 512^-s,   |d_0| <= 128, -256 <= d_s <= 255,
// and each digit is a bf16 value exactly.  Elements more than 2^8 below their row's largest lose
// bits that way, so rows are levelled first: one factor of each product, F (L or R, which do not change), is scaled
// along K by powers of two to columns of one magnitude, and the other, V, by their inverses.
// After that no element of V is rounded against one that F would make small.
//
// Error of sum_k F_ik V_kj, with M_j the largest over i of sum_k |F_ik V_kj|: the scaled row maxima multiply to
// at most 4 M_j; rounding the elements costs K 2^-61 of it, the dropped orders (below) K 2^-58.4: K 2^-56
// M_j in all, where FMAs are bounded by K 2^-53 sum_k |F_ik V_kj|.  Exponents along K are shared by blocks
// alike within 3 bits (tasks.cpp), which makes it K 2^-53 M_j at most.  So an entry's error is that of FMAs
// for the largest sum of its column (products with L; with R: of its row), whatever the grading of the
// contracted index, of the rows and of the columns; an entry far below the others there is less precise than by
// FMAs.
//
// The sum over K <= 64 of the products of
// equal order d = i + j,
//     S_d = sum_{i+j=d} sum_k a_i(k) b_j(k),   |S_d| <= 2^24 for d <= 4,
// is an integer an FP32 accumulator holds exactly (a rounding of S_5 or S_6, which
// only digits all near their largest could cause, is below 2^-58 of the row and
// column maxima); orders d <= 6 are kept, 28 of the 49 slice pairs, and the dropped
// products lie below 2^-61 each.  An accumulator is flushed after at most 64 columns of
// K: the multiple of 2^(Ea+Eb-63) nearest to 2^(Ea+Eb-14) sum_d S_d 512^-d is formed
// in integers (fine enough for products with identity-like blocks, whose results lie
// far below the row and column maxima times K); up to three flushes (192 columns) of one
// segment are added as integers, and their sum is rounded to FP64 and added in FP64.  So the
// rounding errors left are two per 64 to 192 columns, against one per product by FMAs.
// Rows with an Inf or NaN give NaN.
//
// slice_columns  : the exponents along K of L's and R's blocks, when a plan is made
// slice_kernel   : FP64 blocks (or sums of blocks) -> digit panels and row exponents
// gg_slice_kernel: the grouped GEMM on digit panels, FP64 output
//
// Panel layout: element (row i, K index k) of slice s at
//     i * pitch + (k / 32) * 224 + s * 32 + k % 32,
// so a K step of 32 of an operand is one 3-d TMA box (32 elements, rows, 7
// slices), 64-byte swizzled in shared memory: slice after slice, K-major.  The
// B slices lie one under another there, so slice i of A times slices 0..6-i of B
// is ONE tcgen05.mma of N = (7 - i) nb whose column groups i..6 are the orders.
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include "kernels.hpp"
#include "pdl.cuh"
#include "umma.cuh"

namespace vmps {

// ===========================================================================
// operand slices
// ===========================================================================
namespace sl {
constexpr int NT = 128, ROWS = 32;   // 32 panel rows per block of threads
constexpr int LD = ROWS + 1;         // values of K index k at k * LD
constexpr int UN = 8;                // loads a thread keeps in flight per term
}

// x 2^s as a signed multiple of 2^(E-61), E = emax - 1022 (emax: the row's largest
// exponent field after the scaling), rounded to nearest; NORMAL: x is a normal number
template <bool NORMAL>
__device__ __forceinline__ int64_t slice_fixed(double x, int s, int emax) {
    const uint64_t bits = (uint64_t)__double_as_longlong(x);
    const int ef = (int)(bits >> 52) & 0x7ff;
    uint64_t q = (bits & 0xfffffffffffffull) << 8;
    if (NORMAL || ef) q |= 1ull << 60;
    const int sh = min(emax - s - (NORMAL ? ef : max(ef, 1)), 63);
    if (NORMAL || sh >= 0) q = (q + ((1ull << sh) >> 1)) >> sh;
    else if (q) q <<= -sh;   // (a subnormal row maximum)
    return (bits >> 63) ? -(int64_t)q : (int64_t)q;
}
// 256 in every base-512 digit: digit s of q is field s of q + kDigitBias, less 256
constexpr uint64_t kDigitBias = 256ull * ((1ull << 54) + (1ull << 45) + (1ull << 36) + (1ull << 27) + (1ull << 18) +
                                          (1ull << 9) + 1ull);

// the exponent field x has or, subnormal, would have; kSliceNone for zero, 0x7ff for Inf and NaN
__device__ __forceinline__ int slice_field(double x) {
    const int f = (__double2hiint(x) >> 20) & 0x7ff;
    if (f) return f;
    const uint64_t m = (uint64_t)__double_as_longlong(x) & 0xfffffffffffffull;
    return m ? 12 - __clzll((long long)m) : kSliceNone;
}

// values of up to 32 panel rows and K indices [k0, k0 + kn) into shared memory; the lanes of a
// warp run along the contiguous dimension.  A first term with coefficient 1 or -1 takes
// no FP64 operation (nor does the look at it), a further one takes one.
__device__ __forceinline__ void slice_load(const SliceArgs& a, const SliceBlock& b, int row0, int rows, int k0, int kn,
                                           double* sh) {
    using namespace sl;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int outer = b.trans ? kn : rows, inner = b.trans ? rows : kn;   // warps take `outer`, lanes `inner`
    const int64_t base = b.trans ? (int64_t)row0 + (int64_t)k0 * b.ld : (int64_t)k0 + (int64_t)row0 * b.ld;
    const int so = b.trans ? LD : 1, si = b.trans ? 1 : LD;
    for (int i = lane; i < inner; i += 32)
        for (int o0 = warp; o0 < outer; o0 += 4 * UN) {
            double x[UN];
            for (int t = 0; t < b.term_count; ++t) {
                const GTerm tm = a.terms[b.term_begin + t];
                const double* p = a.src + tm.off + base + i;
                double v[UN];
#pragma unroll
                for (int u = 0; u < UN; ++u) v[u] = o0 + 4 * u < outer ? p[(int64_t)(o0 + 4 * u) * b.ld] : 0.0;
                const int64_t cb = __double_as_longlong(tm.coef), sign = cb & INT64_MIN;
                if (t == 0 && (cb ^ sign) == 0x3ff0000000000000ll) {
#pragma unroll
                    for (int u = 0; u < UN; ++u) x[u] = __longlong_as_double(__double_as_longlong(v[u]) ^ sign);
                } else {
#pragma unroll
                    for (int u = 0; u < UN; ++u) x[u] = t == 0 ? tm.coef * v[u] : fma(tm.coef, v[u], x[u]);
                }
            }
#pragma unroll
            for (int u = 0; u < UN; ++u)
                if (o0 + 4 * u < outer) sh[(o0 + 4 * u) * so + i * si] = x[u];
        }
}

// digits of eight consecutive K indices of a row (zero where sk is kSliceNone or the row is bad): one
// 16-byte store per slice
template <bool NORMAL>
__device__ __forceinline__ void slice_store8(__nv_bfloat16* o, const double* x, const int* sk, int emax) {
    const int4 s0 = reinterpret_cast<const int4*>(sk)[0], s1 = reinterpret_cast<const int4*>(sk)[1];
    const int s[8] = {s0.x, s0.y, s0.z, s0.w, s1.x, s1.y, s1.z, s1.w};
    uint64_t q8[8];
#pragma unroll
    for (int q = 0; q < 8; ++q)
        q8[q] = (uint64_t)slice_fixed<NORMAL>(x[q * sl::LD], s[q], emax) + kDigitBias;
#pragma unroll
    for (int s = 0; s < kSlices; ++s) {
        uint32_t w[4];
#pragma unroll
        for (int h = 0; h < 4; ++h) {
            const float f0 = __uint_as_float(0x4B000000u | ((uint32_t)(q8[2 * h] >> (54 - 9 * s)) & 0x1ffu));
            const float f1 = __uint_as_float(0x4B000000u | ((uint32_t)(q8[2 * h + 1] >> (54 - 9 * s)) & 0x1ffu));
            const __nv_bfloat162 v = __floats2bfloat162_rn(f0 - 8388864.f, f1 - 8388864.f);
            w[h] = *reinterpret_cast<const uint32_t*>(&v);
        }
        *reinterpret_cast<uint4*>(o + s * 32) = make_uint4(w[0], w[1], w[2], w[3]);
    }
}

// Exponents along K of the blocks of X or Z: 2^e <= |largest finite element at K index k| < 2^(e+1).  Read
// once when a plan's fixed operands are prepared: bound by memory.
__global__ void __launch_bounds__(sl::NT) slice_columns_kernel(SliceArgs a) {
    using namespace sl;
    __shared__ int red[NT / 32][32];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    auto field = [](double x) {
        const int f = slice_field(x);
        return f == 0x7ff ? kSliceNone : f;
    };
    pdl_wait();
    for (int p = blockIdx.x; p < a.npieces; p += gridDim.x) {
        const SlicePiece pc = a.pieces[p];
        const SliceBlock b = a.blocks[pc.block];
        const int k0 = pc.row0, kn = min(32, b.K - k0);
        const double* src = a.src + a.terms[b.term_begin].off;
        if (b.trans) {   // panel rows are contiguous: a warp takes every fourth K index
            for (int k = warp; k < kn; k += NT / 32) {
                int f = kSliceNone;
#pragma unroll 8
                for (int i = lane; i < b.rows; i += 32) f = max(f, field(src[i + (int64_t)(k0 + k) * b.ld]));
                f = __reduce_max_sync(0xffffffffu, f);
                if (lane == 0) red[0][k] = f;
            }
        } else {         // K indices are: a warp takes every fourth panel row
            int f = kSliceNone;
            if (lane < kn)
#pragma unroll 8
                for (int i = warp; i < b.rows; i += NT / 32) f = max(f, field(src[k0 + lane + (int64_t)i * b.ld]));
            red[warp][lane] = f;
        }
        __syncthreads();
        if (warp == 0 && lane < kn) {
            int f = red[0][lane];
            if (!b.trans)
#pragma unroll
                for (int w = 1; w < NT / 32; ++w) f = max(f, red[w][lane]);
            a.kexp[b.koff + k0 + lane] = f == kSliceNone ? kSliceNone : f - 1023;
        }
        __syncthreads();
    }
}

// Bound by memory for large blocks (8 bytes read per term, 14 written per element)
// and by latency for small ones.  The sums of the terms go through shared memory,
// loaded along the contiguous dimension of the block whichever way it lies; then
// four threads share a panel row and take its octets of K in turn.  The digits
// come from integer shifts: in FP64 arithmetic they would cost 21 operations per element on the slow pipe.
// Rows of normal numbers alone take a form without the tests for the others.  Rows longer than the shared
// buffer (a.kcache) are loaded twice, once for the exponent and once for the digits.  Scalings along K add an
// addition and a shared-memory load per element and pass: 31.5 -> 32.3 us for the sums of the D = 1024 two-site
// Hubbard HxV (37.8 us while the last octet of a row had a form of its own, which warps then ran besides the other).
__global__ void __launch_bounds__(sl::NT, 6) slice_kernel(SliceArgs a) {
    using namespace sl;
    extern __shared__ double sh[];
    int* sk = reinterpret_cast<int*>(sh + a.kcache * LD);   // the chunk's exponents along K, as scalings
    constexpr int EMPTY = -(1 << 25), BAD = 1 << 25;
    const int r = threadIdx.x >> 2, g = threadIdx.x & 3;
    pdl_wait();
    for (int p = blockIdx.x; p < a.npieces; p += gridDim.x) {
        const SlicePiece pc = a.pieces[p];
        const SliceBlock b = a.blocks[pc.block];
        const int rows = min(ROWS, b.rows - pc.row0), row = pc.row0 + r;
        const bool on = r < rows;
        __nv_bfloat16* d = (__nv_bfloat16*)a.dst + b.dst_off + (int64_t)row * b.pitch;
        int emax = EMPTY;
        bool bad = false, normal = true, odd = false;   // odd: the thread met a zero, subnormal number, Inf or NaN
        auto row_max = [&] {
            emax = max(emax, __shfl_xor_sync(0xffffffffu, emax, 1));
            emax = max(emax, __shfl_xor_sync(0xffffffffu, emax, 2));
            bad = emax >= BAD / 2;                 // Inf or NaN: digits of zero, the row's products become NaN
            normal = !__any_sync(0xffffffffu, odd);
            if (emax < kSliceNone / 2) emax = 1022;   // nothing but zeros, or opposite zeros of the other operand
        };
        const int passes = b.K <= a.kcache ? 1 : 2;
        for (int pass = 0; pass < passes; ++pass) {
            for (int k0 = 0; k0 < b.K; k0 += a.kcache) {
                const int kn = min(a.kcache, b.K - k0);
                __syncthreads();   // the buffer is free
                // (loaded before the elements, stored after them: one wait for both)
                static_assert(kSliceCacheK == 2 * NT, "two exponents along K per thread");
                const int t0 = threadIdx.x, t1 = t0 + NT;
                const int e0 = t0 < kn ? a.kexp[b.koff + k0 + t0] : 0, e1 = t1 < kn ? a.kexp[b.koff + k0 + t1] : 0;
                slice_load(a, b, pc.row0, rows, k0, kn, sh);
                if (t0 < a.kcache) sk[t0] = t0 < kn ? a.ksign * e0 : kSliceNone;   // (past the row's end: zero digits)
                if (t1 < a.kcache) sk[t1] = t1 < kn ? a.ksign * e1 : kSliceNone;
                __syncthreads();
                if (pass == 0 && on) {
                    int e = emax;
                    bool again = false;
                    for (int k = g; k < kn; k += 4) {
                        const int f = (__double2hiint(sh[k * LD + r]) >> 20) & 0x7ff;
                        again |= (unsigned)(f - 1) >= 0x7feu;
                        e = max(e, f + sk[k]);
                    }
                    odd |= again;
                    if (again)
                        for (int k = g; k < kn; k += 4) {
                            const int f = slice_field(sh[k * LD + r]);
                            emax = max(emax, f == 0x7ff ? BAD : f == kSliceNone ? EMPTY : f + sk[k]);
                        }
                    else
                        emax = e;
                }
                if (pass + 1 == passes) {
                    if (passes == 1) row_max();
                    if (on)
                        for (int k = g * 8; k < kn; k += 32) {
                            __nv_bfloat16* o = d + ((k0 + k) >> 5) * (kSlices * kSliceK) + ((k0 + k) & 31);
                            if (normal) slice_store8<true>(o, sh + k * LD + r, sk + k, emax);
                            else slice_store8<false>(o, sh + k * LD + r, sk + k, emax);
                        }
                }
            }
            if (pass == 0 && passes == 2) row_max();
        }
        if (on && g == 0) a.exps[b.erow + row] = bad ? kSliceBad : emax - 1022;
    }
}

// ===========================================================================
// grouped GEMM on digit panels
// ===========================================================================
namespace sg {
constexpr int EPI = 16, NT = 64 + 32 * EPI;   // flush warps: four per TMEM lane quadrant, 8 columns each
constexpr int MAX_STAGES = 6;
constexpr int B_BYTES = kSlices * kSliceTileN * 64;     // B region of a stage: 14 KB
constexpr int RING_BYTES = 3 * (kSlices * kSliceTileM * 64 + B_BYTES);
constexpr int SMEM_BYTES = RING_BYTES + 1024 + 256;
static_assert(SMEM_BYTES <= 227 * 1024, "shared memory");
constexpr uint32_t ACC_COLS = 256;                     // one accumulator: seven orders x 32 columns
constexpr uint32_t TMEM_COLS = 2 * ACC_COLS;           // two, so that a flush overlaps the next group's products
static_assert((2 * MAX_STAGES + 5) * 8 + 16 <= 256, "barrier area overflow");
}

// shared-memory matrix descriptor: K-major, 64-byte swizzle, 8-row groups 512 B apart
__device__ __forceinline__ uint64_t sw64_desc(uint32_t saddr) {
    uint64_t d = 0;
    d |= (uint64_t)((saddr >> 4) & 0x3FFFu);
    d |= (uint64_t)1 << 16;
    d |= (uint64_t)(512 >> 4) << 32;
    d |= (uint64_t)1 << 46;
    d |= (uint64_t)4 << 61;
    return d;
}
__device__ __forceinline__ void tma_load_3d(uint32_t dst, const void* tmap, int x, int y, int z, uint32_t bar) {
    asm volatile(
        "cp.async.bulk.tensor.3d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4}], "
        "[%5];\n" ::"r"(dst),
        "l"(tmap), "r"(x), "r"(y), "r"(z), "r"(bar)
        : "memory");
}
// 32 lanes x 4 consecutive 32-bit columns of tensor memory (completion: tmem_wait_ld)
__device__ __forceinline__ void tmem_ld4(uint32_t taddr, uint32_t* r) {
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x4.b32 {%0,%1,%2,%3}, [%4];\n"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
                 : "r"(taddr));
}
__device__ __forceinline__ void tmem_ldn(uint32_t taddr, uint32_t (&r)[4]) { tmem_ld4(taddr, r); }
__device__ __forceinline__ void tmem_ldn(uint32_t taddr, uint32_t (&r)[2]) {
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x2.b32 {%0,%1}, [%2];\n" : "=r"(r[0]), "=r"(r[1]) : "r"(taddr));
}
template <int N>
__device__ __forceinline__ void reg_fence(uint32_t (&r)[N]) {
#pragma unroll
    for (int i = 0; i < N; ++i) asm volatile("" : "+r"(r[i]));
}
__device__ __forceinline__ SliceStep load_slice_step(const SliceStep* p) {
    const int4 a = __ldg(reinterpret_cast<const int4*>(p));
    const int4 b = __ldg(reinterpret_cast<const int4*>(p) + 1);
    SliceStep s;
    s.amap = a.x; s.bmap = a.y; s.az = a.z; s.bz = a.w;
    s.ay = b.x; s.by = b.y; s.arows = b.z; s.flags = b.w;
    return s;
}

// A flush has to keep up with the products of 64 columns of K (~3,500 clocks, bound by shared
// memory).  Per warp and SM quadrant an integer operation takes 2 clocks, an FP64 operation or
// 64-bit conversion 64: summing the orders of an element takes ~45 clocks of the integer pipe,
// making a double of it ~65, and 32 such elements fall to a quadrant.  The conversion
// instructions of the rare cases are volatile so that they are not executed speculatively.
__device__ __forceinline__ int slice_cvt(uint32_t v) {
    int r;
    asm volatile("cvt.rni.s32.f32 %0, %1;" : "=r"(r) : "f"(__uint_as_float(v)));
    return r;
}

// A flushed element, the orders S_0..S_6 (FP32, exact integers) summed in units of 2^-49 of
// S_0's: hi 256 + lo, |hi| < 1.1 2^61 and |lo| < 2^29, so that the sums of three fit 64
// and 32 bits
struct SliceSum { int64_t hi; int lo; };
// Integers come from adding 1.5 * 2^23, which holds |S| <= 2^22: S_0 and S_1 always (<= 2^20,
// 2^22), S_2 .. S_6 (<= 2^25) in all but contrived sums, for which `off` becomes nonzero
// (|S_2| >= 2^21, so that S_2 512 + S_3 stays below 2^31).
template <int N>
__device__ __forceinline__ SliceSum slice_sum(const uint32_t (&v)[kSlices][N], int c, uint32_t& off) {
    constexpr uint32_t K = 0x4B400000u;
    uint32_t r[kSlices];
#pragma unroll
    for (int d = 0; d < kSlices; ++d) r[d] = __float_as_uint(__uint_as_float(v[d][c]) + 12582912.f);
    off |= ((r[2] - (K - 0x200000u)) & 0xFFC00000u) |
           (((r[3] ^ 0x4B000000u) | (r[4] ^ 0x4B000000u) | (r[5] ^ 0x4B000000u) | (r[6] ^ 0x4B000000u)) & 0xFF800000u);
    const uint32_t a = r[0] * 512u + r[1] - (K * 512u + K);     // weight 2^32
    const int b = (int)(r[2] * 512u + r[3] - (K * 512u + K));   // weight 2^14
    const int l = (int)(r[4] * 32u - K * 32u);
    return {(int64_t)b * (1 << 14) + l + (int64_t)((uint64_t)a << 32),
            (int)(r[5] * 16u - K * 16u) + ((int)(r[6] - (K - 16u)) >> 5)};
}
template <int N>
__device__ __forceinline__ SliceSum slice_sum_any(const uint32_t (&v)[kSlices][N], int c) {
    int s[kSlices];
#pragma unroll
    for (int d = 0; d < kSlices; ++d) s[d] = slice_cvt(v[d][c]);
    return {(int64_t)(s[0] * 512 + s[1]) * (1ll << 32) + (int64_t)s[2] * (1 << 23) + (int64_t)s[3] * (1 << 14) +
                (int64_t)s[4] * (1 << 5), s[5] * 16 + ((s[6] + 16) >> 5)};
}

// x, one flush or a sum of up to three, in units of 2^(e - 63), as 64 bits in units of 2^(e - 63) or, from
// |hi| = 2^53 on, 2^(e - 55): |result| < 2^61 + 2^31 or < 3.4 2^61
__device__ __forceinline__ int64_t slice_pack(const SliceSum& x, int& e) {
    const bool big = (((uint32_t)(x.hi >> 32) + 0x200000u) & 0xFFC00000u) != 0;   // |hi| >= 2^53
    e -= big ? 55 : 63;
    return big ? x.hi + ((x.lo + 128) >> 8) : x.hi * 256 + x.lo;
}
// x 2^e, rounded to nearest, by integer operations; |e| < 1000 and 2^36 <= |x| < 2^63 (below, `small`
// becomes nonzero)
__device__ __forceinline__ double slice_to_double(int64_t x, int e, uint32_t& small) {
    const uint32_t s = (uint32_t)(x >> 63);
    const uint64_t u = ((uint64_t)x ^ ((uint64_t)s << 32 | s)) - (int64_t)(int)s;
    const uint32_t uhi = (uint32_t)(u >> 32);
    small |= uhi < 16u;
    const int lz = __clz((int)(uhi | 1u));                        // 1 .. 27
    const uint64_t t = u << (lz - 1);
    const uint64_t m = (t + 511u + ((uint32_t)(t >> 10) & 1u)) >> 10;   // 2^52 .. 2^53, ties to even
    return __hiloint2double((int)((uint32_t)(m >> 32) + (uint32_t)(1023 + 63 - 1 + e - lz) * (1u << 20) + (s & 0x80000000u)),
                            (int)(uint32_t)m);
}
// the same by the conversion unit of the FP64 pipe; |e| < 900
__device__ __forceinline__ double slice_to_double_cvt(int64_t x, int e) {
    const double d = (double)x;
    const int hi = __double2hiint(d);
    return __hiloint2double(hi ? hi + e * (1 << 20) : 0, __double2loint(d));
}
__device__ __forceinline__ double slice_to_double_any(int64_t x, int e) {
    double d;
    asm volatile("cvt.rn.f64.s64 %0, %1;" : "=d"(d) : "l"((long long)x));
    if (e >= kSliceBad / 2) return __longlong_as_double(0x7ff8000000000000ll);
    const int k = max(e, -2044), k1 = k / 2;
    const double f1 = __hiloint2double((1023 + k1) << 20, 0), f2 = __hiloint2double((1023 + k - k1) << 20, 0);
    asm volatile("mul.rn.f64 %0, %0, %1;\n\tmul.rn.f64 %0, %0, %2;" : "+d"(d) : "d"(f1), "d"(f2));
    return d;
}

// Persistent, warp-specialised: warp 0 one lane of TMA, warp 1 one lane of MMA
// (seven tcgen05.mma per K16 slice), warps 2..17 flush (four per TMEM lane quadrant,
// 8 columns each).  The tile is 128 x 32: seven orders of 32 columns take half
// the tensor memory, so that a flush overlaps the next group's products.  CTA b
// runs tiles[cta_tiles[b] .. cta_tiles[b+1]), its K steps and flush groups are
// consecutive.  Barrier waits are bounded as in the split engine (umma.cu).
//
// ONE_SUM: every tile is one segment of K <= 192 (phase 1), whose flushes are added as integers
// and stored, the conversions on the otherwise idle FP64 pipe.  ONE_FLUSH: every flush is a sum
// (K <= 64, or hardly any longer segments), so that no open sums are held.  Otherwise the
// flushes of a segment are added as integers, up to kSliceSumEnd.  Conversions that are followed
// by an FP64 addition go one of four to the FP64 pipe, the others to the integer pipe.  18 warps
// leave 96 registers per thread, and a spilled value costs more than anything here: columns are
// taken two at a time (four in the smallest variant), and tile fields are read when needed.
// Clocks per launch, two-site Hubbard D = 1024 / 2048 / 4096: 79 / 239 / 966 thousand, of which the
// products take ~52 / 150 / 650.  Every flush converted by itself 76 / 245 / 1301; four columns at a
// time everywhere, with spills, 72 / 326 / 1390; eight warps of 16 columns 103 / 302 / 1661.
template <bool ONE_SUM, bool ONE_FLUSH>
__global__ void __launch_bounds__(sg::NT, 1) gg_slice_kernel(const SliceGemmArgs g, const __grid_constant__ TmaMaps maps) {
    using namespace sg;
    extern __shared__ __align__(1024) unsigned char smraw[];
    const uint32_t raw = su32(smraw);
    const uint32_t pad = ((raw + 1023u) & ~1023u) - raw;
    const uint32_t ring = raw + pad;
    uint64_t* bars = reinterpret_cast<uint64_t*>(smraw + pad + RING_BYTES);
    // the ring holds as many stages as the phase's largest A box leaves room for
    const int STAGES = g.stages, STAGE_BYTES = g.stage_bytes, A_BYTES = STAGE_BYTES - B_BYTES;
    // bars[0..S) full, [S..2S) empty, [2S..2S+2) accumulator full, [2S+2..2S+4) accumulator empty, [2S+4] drain
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 2 * MAX_STAGES + 5);
    volatile int* s_fail = reinterpret_cast<volatile int*>(tmem_slot + 1);
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    auto bar = [&](int i) { return su32(&bars[i]); };
    if (tid == 0) {
        *s_fail = 0;
        for (int s = 0; s < STAGES; ++s) { mbar_init(bar(s), 1); mbar_init(bar(STAGES + s), 1); }
        for (int b = 0; b < 2; ++b) { mbar_init(bar(2 * STAGES + b), 1); mbar_init(bar(2 * STAGES + 2 + b), EPI); }
        mbar_init(bar(2 * STAGES + 4), 1);
        asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
    }
    if (warp == 1) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;\n" ::"r"(su32(tmem_slot)),
                     "r"(TMEM_COLS));
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;\n" ::);
    }
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = *tmem_slot;
    const int t0 = g.cta_tiles[blockIdx.x], t1 = g.cta_tiles[blockIdx.x + 1];
    const long long wb = g.wait_budget > 0 ? g.wait_budget : um::WAIT_BUDGET;
    int S0 = 0, S1 = 0;
    if (t0 < t1) {
        S0 = g.tiles[t0].step0;
        S1 = g.tiles[t1 - 1].step0 + g.tiles[t1 - 1].nsteps;
    }
    if (tid < 8 && S0 + tid < S1) prefetch_l1(g.steps + S0 + tid);
    pdl_wait();

    if (warp == 0) {
        if (lane == 0) {
            fence_async_global();
            // stage of step `it` and the parity of its use, counted instead of divided
            int it = 0, st = 0, use = 0;
            SliceStep r{};
            if (S0 < S1) r = load_slice_step(g.steps + S0);
            for (int j = S0; j < S1; ++j, ++it) {
                if (j + 8 < S1) prefetch_l1(g.steps + j + 8);
                SliceStep next{};
                if (j + 1 < S1) next = load_slice_step(g.steps + j + 1);
                if (use >= 1 && !mbar_wait(bar(STAGES + st), (uint32_t)((use - 1) & 1), s_fail, wb)) break;
                const uint32_t sb = ring + st * STAGE_BYTES;
                const int nb = (r.flags & kSliceNarrow) ? 16 : 32;
                mbar_expect_tx(bar(st), (uint32_t)((r.arows + nb) * 64 * kSlices));
                tma_load_3d(sb, &maps.a[r.amap], 0, r.ay, r.az, bar(st));
                tma_load_3d(sb + A_BYTES, &maps.b[r.bmap], 0, r.by, r.bz, bar(st));
                r = next;
                if (++st == STAGES) { st = 0; ++use; }
            }
            for (int i = it - 1; i >= 0 && i >= it - STAGES; --i)
                mbar_drain(bar(i % STAGES), (uint32_t)((i / STAGES) & 1), s_fail);
        }
    } else if (warp == 1) {
        if (lane == 0) {
            int grp = 0, st = 0, use = 0;
            uint32_t dacc = tmem;
            SliceStep r{};
            if (S0 < S1) r = load_slice_step(g.steps + S0);
            for (int j = S0; j < S1 && !*s_fail; ++j) {
                SliceStep next{};
                if (j + 1 < S1) next = load_slice_step(g.steps + j + 1);
                if (r.flags & kSliceFirst) {
                    const int buf = grp & 1, gu = grp >> 1;
                    if (gu >= 1 && !mbar_wait(bar(2 * STAGES + 2 + buf), (uint32_t)((gu - 1) & 1), s_fail, wb)) break;
                    tc_fence_after();
                    dacc = tmem + (uint32_t)buf * ACC_COLS;
                }
                if (!mbar_wait(bar(st), (uint32_t)(use & 1), s_fail, wb)) break;
                tc_fence_after();
                const uint32_t sb = ring + st * STAGE_BYTES;
                const uint64_t a0 = sw64_desc(sb), b0 = sw64_desc(sb + A_BYTES);
                const uint64_t as = (uint64_t)(r.arows * 64) >> 4;   // one A slice
                const int nb = (r.flags & kSliceNarrow) ? 16 : 32;
                const int nk = (r.flags & kSliceHalf) ? 1 : 2;
                for (int kk = 0; kk < nk; ++kk) {
                    const uint64_t ko = (uint64_t)(kk * 32) >> 4;
                    const uint32_t acc0 = (r.flags & kSliceFirst) && kk == 0 ? 0u : 1u;
#pragma unroll
                    for (int i = 0; i < kSlices; ++i)
                        umma_bf16(dacc + (uint32_t)(i * nb), a0 + ko + as * i, b0 + ko,
                                  um::IDESC_BASE | ((uint32_t)(((kSlices - i) * nb) >> 3) << 17), i == 0 ? acc0 : 1u);
                }
                umma_commit(bar(STAGES + st));
                if (r.flags & kSliceLast) {
                    umma_commit(bar(2 * STAGES + (grp & 1)));
                    ++grp;
                }
                r = next;
                if (++st == STAGES) { st = 0; ++use; }
            }
            umma_commit(bar(2 * STAGES + 4));
            mbar_drain(bar(2 * STAGES + 4), 0, s_fail);
        }
    } else {
        const int sp = warp & 3, rl = sp * 32 + lane, c0 = ((warp - 2) >> 2) * 8;   // TMEM lanes, tile row, first column
        // the groups of the CTA are consecutive: their exponents (the lane's row; column c0 +
        // lane % 8) come one group ahead, their list two
        const int G0 = t0 < t1 ? g.tiles[t0].group0 : 0;
        const int G1 = t0 < t1 ? g.tiles[t1 - 1].group0 + g.tiles[t1 - 1].ngroups : 0;
        auto group = [&](int q) {
            const int4 r = q < G1 ? __ldg(reinterpret_cast<const int4*>(g.groups + q)) : make_int4(0, 0, 0, 0);
            return make_int3(r.x, r.y, r.z);
        };
        int3 ge = group(G0), ge1 = group(G0 + 1);
        int ea = g.ea[ge.x + rl], eb = g.eb[ge.y + c0 + (lane & 7)];
        int grp = 0;
        bool ok = true;
        for (int t = t0; t < t1 && ok; ++t) {
            if (t + 1 < t1) prefetch_l1(g.tiles + t + 1);
            // fields are read where they are used, to keep registers for the sums
            const volatile SliceTile& tile = g.tiles[t];
            const int tn = tile.tn, tm = tile.tm, ngroups = tile.ngroups;
            constexpr int W = ONE_FLUSH ? 4 : 2, P = ONE_FLUSH && ONE_SUM ? 4 : 2;   // columns per load, columns at a time
            const int nb = tn <= 16 ? 16 : 32;
            const bool cols = c0 < tn && sp * 32 < tm, rows = rl < tm;   // cols is warp-uniform
            double acc[ONE_SUM ? 1 : 8];
            SliceSum part[ONE_FLUSH ? 1 : 8];   // the open sums of flushes of equal exponents
            bool added = false;
            if (!ONE_FLUSH) {
#pragma unroll
                for (int c = 0; c < 8; ++c) part[c] = {0, 0};
            }
            if (!ONE_SUM) {
#pragma unroll
                for (int c = 0; c < 8; ++c) acc[c] = 0.0;
            }
            for (int q = 0; q < ngroups; ++q, ++grp) {
                const int ea1 = g.ea[ge1.x + rl], eb1 = g.eb[ge1.y + c0 + (lane & 7)];
                const int3 ge2 = group(G0 + grp + 2);
                const int buf = grp & 1, use = grp >> 1;
                ok = __all_sync(0xffffffffu, mbar_wait(bar(2 * STAGES + buf), (uint32_t)(use & 1), s_fail, wb));
                if (!ok) break;
                tc_fence_after();
                const bool end = ONE_FLUSH || (ge.z & kSliceSumEnd);
                // an exponent the integer conversion has no room for, or a bad row or column: each row's is
                // known to its own lane, each column's to four lanes, whether or not those have a row
                const bool far = __any_sync(0xffffffffu, (rows && (unsigned)(ea + 440) > 880u) ||
                                                             (c0 + (lane & 7) < tn && (unsigned)(eb + 440) > 880u));
                if (cols) {
#pragma unroll
                    for (int h = 0; h < 8; h += W) {
                        uint32_t v[kSlices][W];
                        const uint32_t ta = tmem + ((uint32_t)(sp * 32) << 16) + (uint32_t)buf * ACC_COLS + (uint32_t)(c0 + h);
#pragma unroll
                        for (int d = 0; d < kSlices; ++d) tmem_ldn(ta + (uint32_t)(d * nb), v[d]);
                        tmem_wait_ld();
#pragma unroll
                        for (int d = 0; d < kSlices; ++d) reg_fence(v[d]);
                        if (h + W == 8) {
                            tc_fence_before();
                            __syncwarp();
                            if (lane == 0) mbar_arrive(bar(2 * STAGES + 2 + buf));
                        }
#pragma unroll
                        for (int i = 0; i < W; i += P) {
                            // columns past the tile and rows of other blocks hold values nobody reads
                            uint32_t rare = 0;
                            SliceSum x[P];
#pragma unroll
                            for (int c = 0; c < P; ++c) x[c] = slice_sum(v, i + c, rare);
                            if (__any_sync(0xffffffffu, rows && rare)) {
#pragma unroll
                                for (int c = 0; c < P; ++c) x[c] = slice_sum_any(v, i + c);
                            }
                            if (!ONE_FLUSH) {
#pragma unroll
                                for (int c = 0; c < P; ++c) {
                                    part[h + i + c].hi += x[c].hi;
                                    part[h + i + c].lo += x[c].lo;
                                }
                            }
                            if (!end) continue;
                            const int64_t ldc = ONE_SUM ? tile.ldc : 0;
                            double* C = ONE_SUM ? g.C + tile.c_off + tile.row0 + rl + (tile.col0 + c0) * ldc : nullptr;
                            rare = 0;
                            double y[P];
#pragma unroll
                            for (int c = 0; c < P; ++c) {
                                const SliceSum z = ONE_FLUSH ? x[c] : part[h + i + c];
                                int e = ea + __shfl_sync(0xffffffffu, eb, h + i + c);
                                const int64_t p = slice_pack(z, e);
                                y[c] = ONE_SUM || (h + i + c) % 4 == 3 ? slice_to_double_cvt(p, e) : slice_to_double(p, e, rare);
                            }
                            if (far || __any_sync(0xffffffffu, rows && rare)) {
#pragma unroll
                                for (int c = 0; c < P; ++c) {
                                    const SliceSum z = ONE_FLUSH ? x[c] : part[h + i + c];
                                    int e = ea + __shfl_sync(0xffffffffu, eb, h + i + c);
                                    const int64_t p = slice_pack(z, e);
                                    y[c] = slice_to_double_any(p, e);
                                    // a sum that has overflowed stays as it is, as one of FMAs does
                                    if (!ONE_SUM && isinf(acc[h + i + c]) && isinf(y[c])) y[c] = 0.0;
                                }
                            }
#pragma unroll
                            for (int c = 0; c < P; ++c) {
                                if (!ONE_FLUSH && !ONE_SUM) part[h + i + c] = {0, 0};
                                if (ONE_SUM) {
                                    if (rows && c0 + h + i + c < tn) C[(h + i + c) * ldc] = y[c];
                                } else if (added) {
                                    asm volatile("add.rn.f64 %0, %0, %1;" : "+d"(acc[h + i + c]) : "d"(y[c]));
                                } else {
                                    acc[h + i + c] = y[c];   // the first sum, without an FP64 addition
                                }
                            }
                        }
                    }
                    added = added || end;
                } else {
                    tc_fence_before();
                    __syncwarp();
                    if (lane == 0) mbar_arrive(bar(2 * STAGES + 2 + buf));
                }
                ea = ea1;
                eb = eb1;
                ge = ge1;
                ge1 = ge2;
            }
            // (a tile without a segment is zero)
            if (ok && rows && cols && (!ONE_SUM || ngroups == 0)) {
                const int64_t ldc = tile.ldc;
                double* C = g.C + tile.c_off + tile.row0 + rl + (tile.col0 + c0) * ldc;
#pragma unroll
                for (int c = 0; c < 8; ++c)
                    if (c0 + c < tn) C[c * ldc] = ONE_SUM ? 0.0 : acc[c];
            }
        }
    }
    __syncthreads();
    if (*s_fail && tid == 0 && g.err) atomicOr_system(g.err, 1);   // (mapped host memory)
    tc_fence_after();
    if (warp == 1) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;\n" ::"r"(tmem), "r"(TMEM_COLS));
}

cudaError_t slices_init() {
    const cudaError_t e = cudaFuncSetAttribute(slice_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                               kSliceCacheK * (sl::LD * 8 + 4));
    if (e != cudaSuccess) return e;
    auto opt = [](auto* k) { return cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, sg::SMEM_BYTES); };
    cudaError_t r;
    if ((r = opt(gg_slice_kernel<true, true>)) != cudaSuccess || (r = opt(gg_slice_kernel<true, false>)) != cudaSuccess)
        return r;
    if ((r = opt(gg_slice_kernel<false, true>)) != cudaSuccess) return r;
    return opt(gg_slice_kernel<false, false>);
}

cudaError_t launch_slice_columns(const SliceArgs& a, cudaStream_t st) {
    if (a.npieces <= 0) return cudaSuccess;
    if (!a.pieces || !a.blocks || !a.terms || !a.src || !a.kexp) return cudaErrorInvalidValue;
    launch_pdl(slice_columns_kernel, a.npieces < 16384 ? a.npieces : 16384, sl::NT, 0, st, a);
    return cudaGetLastError();
}

cudaError_t launch_slices(const SliceArgs& a, cudaStream_t st) {
    if (a.npieces <= 0) return cudaSuccess;
    if (!a.pieces || !a.blocks || !a.terms || !a.src || !a.dst || !a.exps || !a.kexp || (a.ksign != 1 && a.ksign != -1) ||
        a.kcache < 32 || a.kcache % 32 || a.kcache > kSliceCacheK)
        return cudaErrorInvalidValue;
    launch_pdl(slice_kernel, a.npieces < 16384 ? a.npieces : 16384, sl::NT, a.kcache * (sl::LD * 8 + 4), st, a);
    return cudaGetLastError();
}

cudaError_t launch_gg_slices(const SliceGemmArgs& a, const TmaMaps& maps, cudaStream_t st) {
    if (a.ncta <= 0) return cudaSuccess;
    if (!a.tiles || !a.cta_tiles || !a.C || !a.ea || !a.eb || !a.steps || !a.groups) return cudaErrorInvalidValue;
    SliceGemmArgs b = a;
    if (b.max_arows < 16 || b.max_arows > kSliceTileM) return cudaErrorInvalidValue;
    b.stage_bytes = kSlices * b.max_arows * 64 + sg::B_BYTES;
    b.stages = sg::RING_BYTES / b.stage_bytes < sg::MAX_STAGES ? sg::RING_BYTES / b.stage_bytes : sg::MAX_STAGES;
    if (b.one_sum && b.one_flush) launch_pdl(gg_slice_kernel<true, true>, b.ncta, sg::NT, sg::SMEM_BYTES, st, b, maps);
    else if (b.one_sum) launch_pdl(gg_slice_kernel<true, false>, b.ncta, sg::NT, sg::SMEM_BYTES, st, b, maps);
    else if (!b.one_flush) launch_pdl(gg_slice_kernel<false, false>, b.ncta, sg::NT, sg::SMEM_BYTES, st, b, maps);
    else launch_pdl(gg_slice_kernel<false, true>, b.ncta, sg::NT, sg::SMEM_BYTES, st, b, maps);
    return cudaGetLastError();
}

}  // namespace vmps
