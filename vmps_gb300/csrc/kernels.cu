// CUDA kernels of the GB300 effective-Hamiltonian engine (sm_103a).
//
// gg_fp64  : grouped GEMM, FP64 operands, FP64 FMAs -- the plain drop-in form,
//            the arithmetic type of the Eigen path of
//            pivot/DmrgPivotMatrix1.h:236-262; large FP64 plans run on the
//            tensor cores (slices.cu) instead.
// The split-precision (BF16x3) grouped GEMM is the tcgen05 engine in
// umma.cu; this file holds its operand preparation (FP64 -> bf16 hi/lo
// panels) and the vector kernels.
//
// Work layout (planned on the host, engine.hpp): every CTA owns one output tile
// and loops over that tile's segments; a segment is one GEMM of K columns
// whose A operand is a linear combination of up to several same-shape blocks
// (sum_t c_t A_t).  Output tiles are written exactly once, so no atomics are
// needed and results are deterministic.
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include <algorithm>

#include "convert.hpp"
#include "kernels.hpp"
#include "pdl.cuh"

namespace vmps {

// ===========================================================================
// FP64 grouped GEMM: tiles of at most 16 x 16, 128 threads, one output element
// per thread and pass, scalar FMAs.
//
// GB300's FP64 pipe retires half an FMA per clock and SM quadrant whichever
// instruction feeds it (an 8x8x4 DMMA holds its quadrant for 512 clocks), so DMMA
// has no rate to gain and loses what its fragments round up: the blocks of these
// tensors are 5 to 200 wide.  64 x 64 DMMA tiles left an 11 x 11 block to one
// warp of one SM (72 us per launch at D = 64, now ~11); here the elements of a
// tile spread over all four quadrants without rounding, and the tiles over more
// SMs.  Large blocks gain as well: by this kernel, whole D = 1024 and 4096 two-site HxVs went from
// 0.76 to 0.43 ms and from 17.9 to 16.3 ms, the FP64 pipe bounding both (by slices, which plans of
// that size take unless pinned, they run 0.20 and 2.1 ms).  Small
// ones are bound by the latency of the segment chain, so the segments and terms
// of a tile come to shared memory first and each K chunk's loads are issued one
// chunk ahead.  Several right-hand sides share a launch (blockIdx.y): one launch
// of 16 vectors of the two-site Hubbard pivot at D = 256 (5.2 MFLOP each) in place
// of 16 launches, each too short to fill the chip.
// ===========================================================================
namespace f64k {
constexpr int T = kTileMax, NT = 128, BK = 16, LD = T + 1;
constexpr int SEGS = 32;                 // segments (and their terms) staged at a time
constexpr int PER = T * BK / NT;         // operand elements a thread stages per chunk
}

__global__ void __launch_bounds__(f64k::NT) gg_fp64_kernel(GGArgs g) {
    using namespace f64k;
    __shared__ double As[2][BK * LD], Bs[2][BK * LD];   // [k][row], [k][column]
    __shared__ GSeg sseg[SEGS];
    __shared__ GTerm sterm[SEGS * kMaxTerms];
    pdl_wait();
    const GTile tile = g.tiles[blockIdx.x];
    const double* A = pdl_data((const double*)g.A + blockIdx.y * g.strideA);
    const double* B = pdl_data((const double*)g.B + blockIdx.y * g.strideB);
    const int tid = threadIdx.x, tm = tile.tm, tn = tile.tn, ne = tm * tn;
    const bool tA = g.transA, tB = g.transB;
    // the output elements of this thread, column by column; a second one for tiles of more than 128
    const int e1 = tid + NT;
    const bool on0 = tid < ne, on1 = e1 < ne;
    const int j0 = on0 ? tid / tm : 0, i0 = on0 ? tid - j0 * tm : 0;
    const int j1 = on1 ? e1 / tm : 0, i1 = on1 ? e1 - j1 * tm : 0;
    double acc0 = 0.0, acc1 = 0.0;

    for (int sb = tile.seg_begin; sb < tile.seg_end; sb += SEGS) {
        const int ns = min(SEGS, tile.seg_end - sb);
        __syncthreads();   // the staged lists and both chunk buffers are free
        for (int s = tid; s < ns; s += NT) sseg[s] = g.segs[sb + s];
        __syncthreads();
        const int tb = sseg[0].term_begin, nt = sseg[ns - 1].term_begin + sseg[ns - 1].term_count - tb;
        for (int t = tid; t < nt; t += NT) sterm[t] = g.terms[tb + t];
        __syncthreads();
        double ra[PER], rb[PER];
        auto stage = [&](int s, int k0) {
            const GSeg& sg = sseg[s];
            const int krem = sg.K - k0, t0 = sg.term_begin - tb;
#pragma unroll
            for (int r = 0; r < PER; ++r) {
                const int v = tid + NT * r, lo = v & (T - 1), hi = v / T;
                const int i = tA ? hi : lo, k = tA ? lo : hi;   // lanes run along the contiguous dimension
                ra[r] = 0.0;
                if (i < tm && k < krem) {
                    const int64_t e = tA ? (int64_t)(k0 + k) + (int64_t)(tile.row0 + i) * sg.lda
                                         : (int64_t)(tile.row0 + i) + (int64_t)(k0 + k) * sg.lda;
                    // a first term of coefficient 1 (every segment of phase 1) takes no FP64 operation
                    const GTerm first = sterm[t0];
                    const double x = ld_global(A + first.off + e);
                    ra[r] = __double_as_longlong(first.coef) == 0x3ff0000000000000ll ? x : fma(first.coef, x, 0.0);
                    for (int t = 1; t < sg.term_count; ++t) {
                        const GTerm tm_ = sterm[t0 + t];
                        ra[r] = fma(tm_.coef, ld_global(A + tm_.off + e), ra[r]);
                    }
                }
                const int j = tB ? lo : hi, kb = tB ? hi : lo;
                rb[r] = 0.0;
                if (j < tn && kb < krem) {
                    const int64_t e = tB ? (int64_t)(tile.col0 + j) + (int64_t)(k0 + kb) * sg.ldb
                                         : (int64_t)(k0 + kb) + (int64_t)(tile.col0 + j) * sg.ldb;
                    rb[r] = ld_global(B + sg.b_off + e);
                }
            }
        };
        int s = 0, k0 = 0, buf = 0;
        stage(0, 0);
        while (true) {
#pragma unroll
            for (int r = 0; r < PER; ++r) {
                const int v = tid + NT * r, lo = v & (T - 1), hi = v / T;
                As[buf][tA ? lo * LD + hi : hi * LD + lo] = ra[r];
                Bs[buf][tB ? hi * LD + lo : lo * LD + hi] = rb[r];
            }
            __syncthreads();
            const int kc = min(BK, sseg[s].K - k0);
            k0 += BK;
            if (k0 >= sseg[s].K) { k0 = 0; ++s; }
            const bool more = s < ns;
            if (more) stage(s, k0);
            if (on0) {
                const double* a = As[buf];
                const double* b = Bs[buf];
                if (on1) {
#pragma unroll 4
                    for (int k = 0; k < kc; ++k) {
                        acc0 = fma(a[k * LD + i0], b[k * LD + j0], acc0);
                        acc1 = fma(a[k * LD + i1], b[k * LD + j1], acc1);
                    }
                } else {
#pragma unroll 4
                    for (int k = 0; k < kc; ++k) acc0 = fma(a[k * LD + i0], b[k * LD + j0], acc0);
                }
            }
            if (!more) break;
            buf ^= 1;
        }
    }
    double* C = (double*)g.C + blockIdx.y * g.strideC + tile.c_off;
    auto put = [&](int i, int j, double x) {
        const int64_t gr = tile.row0 + i, gc = tile.col0 + j;
        C[g.transC ? gc + gr * tile.ldc : gr + gc * tile.ldc] = x;
    };
    if (on0) put(i0, j0, acc0);
    if (on1) put(i1, j1, acc1);
}

// ---------------------------------------------------------------------------
// split-precision panels (engine.hpp): element k of panel row i at
// i*pitch + (k/32)*64 + k%32 (hi) and + 32 (lo)
// ---------------------------------------------------------------------------
__device__ __forceinline__ int panel_pos(int k) { return ((k >> 5) << 6) | (k & 31); }

// v -> bf16 hi = bf16(v), lo = bf16(v - hi)
__device__ __forceinline__ void split_store(__nv_bfloat16* row, int k, float v) {
    const __nv_bfloat16 h = __float2bfloat16_rn(v);
    const int p = panel_pos(k);
    row[p] = h;
    row[p + 32] = __float2bfloat16_rn(v - __bfloat162float(h));
}

// operand preparation: scale, split into bf16 hi/lo, write the block's panel rows
__global__ void prep_kernel(const PrepBlock* pbs, int nb, const double* src,
                            __nv_bfloat16* dst) {
    pdl_wait();
    for (int b = blockIdx.x; b < nb; b += gridDim.x) {
        const PrepBlock pb = pbs[b];
        const int rows = pb.rows, n = pb.rows * pb.cols;
        const bool unit = pb.scale == 1.0;
        for (int e = threadIdx.x; e < n; e += blockDim.x) {
            const int j = e / rows, i = e - j * rows;   // source (i, j), column-major
            const double x = src[pb.src_off + i + (int64_t)j * pb.src_ld];
            const float v = f64_to_f32_rn(unit ? x : pb.scale * x);
            // trans = 1: panel row i, K index j;  trans = 0: panel row j, K index i
            const int r = pb.trans ? i : j, k = pb.trans ? j : i;
            split_store(dst + pb.dst_off + (int64_t)r * pb.dst_ld, k, v);
        }
    }
}

// column pieces of a column-major FP64 or FP32 source into panels: column c of
// the piece is panel row c, its element r is K index r.  A thread converts four
// consecutive elements of one column (one 16-byte load per four floats, two per
// four doubles) into four hi and four lo values of the same 32-element panel
// group (two 8-byte stores).  Columns start at multiples of 8 elements in the
// padded vector layout, so the group's loads stay inside the column's padded
// extent; pieces whose offsets or strides break that alignment (or the stores')
// take the element-wise path.
__device__ __forceinline__ float piece_value(double x, bool unit, double scale) {
    return f64_to_f32_rn(unit ? x : scale * x);
}
__device__ __forceinline__ float piece_value(float x, bool unit, double scale) {
    return unit ? x : f64_to_f32_rn(scale) * x;
}
__device__ __forceinline__ void piece_load4(const float* p, float (&x)[4]) {
    const float4 v = *reinterpret_cast<const float4*>(p);
    x[0] = v.x; x[1] = v.y; x[2] = v.z; x[3] = v.w;
}
__device__ __forceinline__ void piece_load4(const double* p, double (&x)[4]) {
    const double2 a = reinterpret_cast<const double2*>(p)[0], b = reinterpret_cast<const double2*>(p)[1];
    x[0] = a.x; x[1] = a.y; x[2] = b.x; x[3] = b.y;
}
template <typename T>
__global__ void panel_split_kernel(const PanelPiece* pieces, int np, const T* src,
                                   __nv_bfloat16* dst) {
    pdl_wait();
    for (int b = blockIdx.x; b < np; b += gridDim.x) {
        const PanelPiece pc = pieces[b];
        const int rows = pc.rows, nr4 = (rows + 3) >> 2, ng = nr4 * pc.cols;
        const T* s = src + pc.src_off;
        __nv_bfloat16* d = dst + pc.dst_off;
        const bool unit = pc.scale == 1.0;
        const bool vload = ((reinterpret_cast<uintptr_t>(s) | (uintptr_t)pc.src_ld * sizeof(T)) & 15) == 0 &&
                           pc.src_ld >= 4 * nr4;
        const bool vstore = ((reinterpret_cast<uintptr_t>(d) | (uintptr_t)pc.dst_pitch * 2) & 7) == 0;
        for (int g = threadIdx.x; g < ng; g += blockDim.x) {
            const int c = g / nr4, r0 = (g - c * nr4) << 2;
            const T* sc = s + (int64_t)c * pc.src_ld + r0;
            T x[4];
            if (vload) {
                piece_load4(sc, x);
            } else {
#pragma unroll
                for (int q = 0; q < 4; ++q) x[q] = r0 + q < rows ? sc[q] : T(0);
            }
            __nv_bfloat16* row = d + (int64_t)c * pc.dst_pitch;
            if (vstore && r0 + 4 <= rows) {
                // hi = bf16(v), lo = bf16(v - hi), two elements per conversion
                uint32_t h[2], l[2];
#pragma unroll
                for (int q = 0; q < 2; ++q) {
                    const float v0 = piece_value(x[2 * q], unit, pc.scale);
                    const float v1 = piece_value(x[2 * q + 1], unit, pc.scale);
                    const __nv_bfloat162 hv = __floats2bfloat162_rn(v0, v1);
                    const float2 hf = __bfloat1622float2(hv);
                    const __nv_bfloat162 lv = __floats2bfloat162_rn(v0 - hf.x, v1 - hf.y);
                    h[q] = *reinterpret_cast<const uint32_t*>(&hv);
                    l[q] = *reinterpret_cast<const uint32_t*>(&lv);
                }
                const int p = panel_pos(r0);   // r0 % 4 == 0: the four stay in one 32-group
                *reinterpret_cast<uint2*>(row + p) = make_uint2(h[0], h[1]);
                *reinterpret_cast<uint2*>(row + p + 32) = make_uint2(l[0], l[1]);
            } else {
#pragma unroll
                for (int q = 0; q < 4; ++q)
                    if (r0 + q < rows) split_store(row, r0 + q, piece_value(x[q], unit, pc.scale));
            }
        }
    }
}

// ---------------------------------------------------------------------------
// 3xTF32 panels: FP32 storage, element k of panel row i at i*pitch + (k/16)*32 +
// k%16 (hi) and + 16 (lo); hi = tf32(v), lo = tf32(v - hi), both with their low
// 13 mantissa bits zero (the tensor cores read TF32 from the upper 19 bits)
// ---------------------------------------------------------------------------
__device__ __forceinline__ int panel_pos_tf32(int k) { return ((k >> 4) << 5) | (k & 15); }
__device__ __forceinline__ float to_tf32(float v) {
    uint32_t r;
    asm("cvt.rna.tf32.f32 %0, %1;\n" : "=r"(r) : "f"(v));
    return __uint_as_float(r);
}
__device__ __forceinline__ void split_store_tf32(float* row, int k, float v) {
    const float h = to_tf32(v);
    const int p = panel_pos_tf32(k);
    row[p] = h;
    row[p + 16] = to_tf32(v - h);
}
__global__ void prep_tf32_kernel(const PrepBlock* pbs, int nb, const double* src,
                                 float* dst) {
    pdl_wait();
    for (int b = blockIdx.x; b < nb; b += gridDim.x) {
        const PrepBlock pb = pbs[b];
        const int rows = pb.rows, n = pb.rows * pb.cols;
        const bool unit = pb.scale == 1.0;
        for (int e = threadIdx.x; e < n; e += blockDim.x) {
            const int j = e / rows, i = e - j * rows;
            const double x = src[pb.src_off + i + (int64_t)j * pb.src_ld];
            const float v = f64_to_f32_rn(unit ? x : pb.scale * x);
            const int r = pb.trans ? i : j, k = pb.trans ? j : i;
            split_store_tf32(dst + pb.dst_off + (int64_t)r * pb.dst_ld, k, v);
        }
    }
}
// vector pieces -> 3xTF32 panels: one element per thread (column c of the piece is
// panel row c, its element r is K index r)
template <typename T>
__global__ void panel_split_tf32_kernel(const PanelPiece* pieces, int np, const T* src,
                                        float* dst) {
    pdl_wait();
    for (int b = blockIdx.x; b < np; b += gridDim.x) {
        const PanelPiece pc = pieces[b];
        const int rows = pc.rows, n = rows * pc.cols;
        const bool unit = pc.scale == 1.0;
        for (int e = threadIdx.x; e < n; e += blockDim.x) {
            const int c = e / rows, r = e - c * rows;
            const T x = src[pc.src_off + (int64_t)c * pc.src_ld + r];
            split_store_tf32(dst + pc.dst_off + (int64_t)c * pc.dst_pitch, r, piece_value(x, unit, pc.scale));
        }
    }
}

// ===========================================================================
// layout conversion, vector algebra
// ===========================================================================
// dst (padded) <- scale * src (compact), or the reverse
__global__ void pack_kernel(const PackBlock* blocks, int nb, const double* src, double* dst,
                            int to_padded) {
    pdl_wait();
    for (int b = blockIdx.x; b < nb; b += gridDim.x) {
        const PackBlock pb = blocks[b];
        // pieces hold at most a few thousand elements: 32-bit index arithmetic
        const int rows = (int)pb.rows, n = (int)(pb.rows * pb.cols), ld = (int)pb.ld;
        const double* s = src + (to_padded ? pb.coff : pb.doff);
        double* d = dst + (to_padded ? pb.doff : pb.coff);
        // four independent loads in flight per thread, then the four stores
        const bool unit = pb.scale == 1.0;   // U(1) blocks: a plain copy, no FP64 arithmetic
        for (int e0 = threadIdx.x; e0 < n; e0 += 4 * blockDim.x) {
            double x[4];
            int at[4];
#pragma unroll
            for (int u = 0; u < 4; ++u) {
                const int e = e0 + u * blockDim.x;
                const int c = e / rows, r = e - c * rows;
                const int pe = r + c * ld;
                at[u] = to_padded ? pe : e;
                x[u] = e < n ? s[to_padded ? e : pe] : 0.0;
            }
#pragma unroll
            for (int u = 0; u < 4; ++u) {
                if (e0 + u * blockDim.x >= n) break;
                d[at[u]] = unit ? x[u] : (to_padded ? pb.scale * x[u] : x[u] / pb.scale);
            }
        }
    }
}


// partial dot products: fixed chunking -> deterministic two-pass reduction
constexpr int kDotThreads = 256;
// sum over the block, thread t + w added to thread t for w = 128 .. 1 (valid in thread 0)
__device__ __forceinline__ double block_tree_sum(double s) {
    __shared__ double red[kDotThreads];
    red[threadIdx.x] = s;
    __syncthreads();
#pragma unroll
    for (int w = kDotThreads / 2; w >= 32; w >>= 1) {
        if (threadIdx.x < w) red[threadIdx.x] += red[threadIdx.x + w];
        __syncthreads();
    }
    if (threadIdx.x < 32) {
        s = red[threadIdx.x];
#pragma unroll
        for (int w = 16; w > 0; w >>= 1) s += __shfl_down_sync(0xffffffffu, s, w);
    }
    return s;
}
__global__ void dot_partial_kernel(const double* x, const double* y, int64_t n,
                                   int64_t chunk, double* part) {
    pdl_wait();
    const int64_t b0 = blockIdx.x * chunk, b1 = min(n, b0 + chunk);
    double s = 0;
#pragma unroll 8
    for (int64_t i = b0 + threadIdx.x; i < b1; i += kDotThreads) s = fma(x[i], y[i], s);
    s = block_tree_sum(s);
    if (threadIdx.x == 0) part[blockIdx.x] = s;
}
__global__ void sum_partial_kernel(const double* part, int np, double* out) {
    pdl_wait();
    double s = 0;
    for (int i = threadIdx.x; i < np; i += kDotThreads) s += part[i];
    s = block_tree_sum(s);
    if (threadIdx.x == 0) *out = s;
}

// ---- GMRES of the transfer operator ---------------------------------------------------------
// An Arnoldi step of these short vectors (13,000 elements for 256 multiplets) is a chain of
// launches of a few microseconds each, so the sums of partials and the dot weights are folded into
// the kernels around them: 6 launches in place of 13, with the same roundings.  The weighted vector
// r = wm * w is formed where w is written: formed in the dots, it took two more FP64 operations
// per element and basis row (an operation holds an SM quadrant's pipe for 64 clocks per warp).
//
// part[j][chunk] of <V_j, r>, j < nv (V row-major [nv][n])
__global__ void __launch_bounds__(kDotThreads) arnoldi_dot_kernel(const double* V, int64_t n,
                                                                  const double* r, int64_t chunk,
                                                                  int nchunk, double* part) {
    pdl_wait();
    const int64_t b0 = blockIdx.x * chunk, b1 = min(n, b0 + chunk);
    const double* v = V + (int64_t)blockIdx.y * n;
    double s = 0;
#pragma unroll 16
    for (int64_t i = b0 + threadIdx.x; i < b1; i += kDotThreads) s = fma(v[i], r[i], s);
    s = block_tree_sum(s);
    if (threadIdx.x == 0) part[(int64_t)blockIdx.y * nchunk + blockIdx.x] = s;
}
// the sum of nchunk <= 32 partials in the order of block_tree_sum (which adds zeros to them)
__device__ __forceinline__ double partial_tree_sum(const double* p, int nchunk) {
    double t[32];
#pragma unroll
    for (int c = 0; c < 32; ++c) t[c] = c < nchunk ? 0.0 + p[c] : 0.0;
#pragma unroll
    for (int w = 16; w > 0; w >>= 1)
        if (w < nchunk) {
#pragma unroll
            for (int c = 0; c < w; ++c) t[c] += t[c + w];
        }
    return t[0];
}
__global__ void msum_partial_kernel(const double* part, int nchunk, double* out) {
    pdl_wait();
    double s = 0;
    for (int i = threadIdx.x; i < nchunk; i += kDotThreads) s += part[(int64_t)blockIdx.x * nchunk + i];
    s = block_tree_sum(s);
    if (threadIdx.x == 0) out[blockIdx.x] = s;
}
// w -= sum_j coef[j] V_j, r = wm * w; part set: coef[j] is summed here from nchunk <= 32 partials by every
// block, and stored by the first
__global__ void __launch_bounds__(256) arnoldi_update_kernel(const double* V, int nv, int64_t n,
                                                             const double* part, int nchunk, double* coef,
                                                             const double* wm, double* w,
                                                             double* r) {
    pdl_wait();
    extern __shared__ double c[];
    for (int j = threadIdx.x; j < nv; j += blockDim.x) {
        const double x = part ? partial_tree_sum(part + (int64_t)j * nchunk, nchunk) : coef[j];
        c[j] = -x;
        if (part && blockIdx.x == 0) coef[j] = x;
    }
    __syncthreads();
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
        double s = w[i];
#pragma unroll 8
        for (int j = 0; j < nv; ++j) s = fma(c[j], V[(int64_t)j * n + i], s);
        w[i] = s;
        r[i] = wm[i] * s;
    }
}
// out[0] = <w, r>, the partials summed by the last block (out[4]: its counter, zero between
// launches)
__global__ void __launch_bounds__(kDotThreads) arnoldi_norm_kernel(const double* w,
                                                                   const double* r, int64_t n, int64_t chunk,
                                                                   double* part, double* out) {
    pdl_wait();
    const int64_t b0 = blockIdx.x * chunk, b1 = min(n, b0 + chunk);
    double s = 0;
#pragma unroll 16
    for (int64_t i = b0 + threadIdx.x; i < b1; i += kDotThreads) s = fma(w[i], r[i], s);
    s = block_tree_sum(s);
    unsigned* count = reinterpret_cast<unsigned*>(out + 4);
    __shared__ bool last;
    if (threadIdx.x == 0) {
        part[blockIdx.x] = s;
        __threadfence();
        last = atomicAdd(count, 1u) == gridDim.x - 1;
    }
    __syncthreads();
    if (!last) return;
    __threadfence();
    s = 0;
    for (int i = threadIdx.x; i < (int)gridDim.x; i += kDotThreads) s += __ldcg(part + i);
    s = block_tree_sum(s);
    if (threadIdx.x == 0) {
        out[0] = s;
        *count = 0;
    }
}
__global__ void axpy_kernel(double a, const double* x, double* y, int64_t n) {
    pdl_wait();
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
        y[i] = fma(a, x[i], y[i]);
}
__global__ void hadamard_kernel(const double* a, const double* b, double* out,
                                int64_t n) {
    pdl_wait();
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
        out[i] = a[i] * b[i];
}
// y = a x (y = x allowed)
__global__ void scale_kernel(double a, const double* x, double* y, int64_t n) {
    pdl_wait();
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
        y[i] = x[i] * a;
}
// y = sum_j c[j] V_j  (Ritz vector assembly)
__global__ void combine_kernel(const double* V, int nv, int64_t n, const double* c,
                               double* y) {
    pdl_wait();
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
        double s = 0;
        for (int j = 0; j < nv; ++j) s = fma(c[j], V[(int64_t)j * n + i], s);
        y[i] = s;
    }
}
__global__ void finite_kernel(const double* x, int64_t n, int* bad) {
    pdl_wait();
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
        if (!isfinite(x[i])) { atomicOr(bad, 1); return; }
}

// split-K of the grouped GEMM: out[e] = sum_j part[j * n + e], parts in order
template <typename T>
__global__ void splitk_reduce_kernel(const T* part, int nparts, int64_t n, T* out) {
    pdl_wait();
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
        double s = (double)part[i];
        for (int j = 1; j < nparts; ++j) s += (double)part[(int64_t)j * n + i];
        out[i] = (T)s;
    }
}

// ---------------------------------------------------------------------------
// Excited-state projector of an HxV (pivot/DmrgPivotMatrix1.h:304-331):
// out_r += sum_p E <d_p, y_r> a_p for right-hand sides r < nrhs (stride n) and
// projectors p < npen; d_p and a_p are the projector vector in the padded layout
// with the SU(2) dot weights folded in.  Fixed chunks and a fixed summation
// order: the same bits in every run.
// ---------------------------------------------------------------------------
template <typename TY>
__global__ void pen_dot_kernel(PenaltyArgs a, const TY* y) {
    pdl_wait();
    __shared__ double red[kDotThreads];
    const int pr = blockIdx.y, p = pr / a.nrhs, r = pr - p * a.nrhs;
    const int64_t b0 = blockIdx.x * a.chunk, b1 = min(a.n, b0 + a.chunk);
    const double* d = a.dvec + (int64_t)p * a.n;
    const TY* v = y + (int64_t)r * a.n;
    double s = 0;
    for (int64_t i = b0 + threadIdx.x; i < b1; i += kDotThreads) s = fma(d[i], (double)v[i], s);
    red[threadIdx.x] = s;
    __syncthreads();
    for (int w = kDotThreads / 2; w > 0; w >>= 1) {
        if (threadIdx.x < w) red[threadIdx.x] += red[threadIdx.x + w];
        __syncthreads();
    }
    if (threadIdx.x == 0) a.part[(int64_t)pr * a.nchunk + blockIdx.x] = red[0];
}
// coef[p * nrhs + r] = E * (sum of the chunk partials), one block per (p, r)
__global__ void pen_sum_kernel(PenaltyArgs a) {
    pdl_wait();
    __shared__ double red[kDotThreads];
    const int pr = blockIdx.x;
    double s = 0;
    for (int i = threadIdx.x; i < a.nchunk; i += kDotThreads) s += a.part[(int64_t)pr * a.nchunk + i];
    red[threadIdx.x] = s;
    __syncthreads();
    for (int w = kDotThreads / 2; w > 0; w >>= 1) {
        if (threadIdx.x < w) red[threadIdx.x] += red[threadIdx.x + w];
        __syncthreads();
    }
    if (threadIdx.x == 0) a.coef[pr] = a.E * red[0];
}
template <typename TO>
__global__ void pen_add_kernel(PenaltyArgs a, TO* out) {
    pdl_wait();
    const int r = blockIdx.y;
    TO* o = out + (int64_t)r * a.n;
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < a.n; i += (int64_t)gridDim.x * blockDim.x) {
        double s = (double)o[i];
        for (int p = 0; p < a.npen; ++p) s = fma(a.coef[p * a.nrhs + r], a.avec[(int64_t)p * a.n + i], s);
        o[i] = (TO)s;
    }
}

// ---------------------------------------------------------------------------
// VUMPS transfer operator pieces
// ---------------------------------------------------------------------------
// part[b] = w_b * sum_ij V[i + j*v_ld] * LR[j + i*lr_ld]  (the trace of a block product)
__global__ void __launch_bounds__(kDotThreads) trace_pairs_kernel(const TracePair* tp, int n,
                                                                  const double* V,
                                                                  const double* LR, double* part) {
    pdl_wait();
    for (int b = blockIdx.x; b < n; b += gridDim.x) {
        const TracePair p = tp[b];
        double s = 0;
#pragma unroll 8
        for (int e = threadIdx.x; e < p.rows * p.cols; e += kDotThreads) {
            const int j = e / p.rows, i = e - j * p.rows;
            s = fma(V[p.v_off + i + (int64_t)j * p.v_ld], LR[p.lr_off + j + (int64_t)i * p.lr_ld], s);
        }
        s = block_tree_sum(s);
        if (threadIdx.x == 0) part[b] = p.weight * s;
        __syncthreads();
    }
}

// out[block] = V[block] - T[block] + s * identity, per matched block pair, s the sum of the np trace
// partials (every block sums them: cheaper than a launch); r set: r = wm * out there as well.
// gridDim.y blocks share a pair
__global__ void __launch_bounds__(kDotThreads) transfer_combine_kernel(const CombineBlock* cb, int n,
                                                                       const double* V,
                                                                       const double* T,
                                                                       double* out,
                                                                       const double* part, int np,
                                                                       const double* wm,
                                                                       double* r) {
    pdl_wait();
    __shared__ double sc_;
    double t = 0;
    for (int i = threadIdx.x; i < np; i += kDotThreads) t += part[i];
    t = block_tree_sum(t);
    if (threadIdx.x == 0) sc_ = t;
    __syncthreads();
    const double sc = sc_;
    for (int b = blockIdx.x; b < n; b += gridDim.x) {
        const CombineBlock c = cb[b];
#pragma unroll 4
        for (int e = blockIdx.y * kDotThreads + threadIdx.x; e < c.rows * c.cols; e += gridDim.y * kDotThreads) {
            const int j = e / c.rows, i = e - j * c.rows;
            const int64_t vo = c.v_off + i + (int64_t)j * c.v_ld;
            const double x = V[vo] - T[c.t_off + i + (int64_t)j * c.t_ld] + (i == j ? sc : 0.0);
            out[vo] = x;
            if (r) r[vo] = wm[vo] * x;
        }
    }
}

// ===========================================================================
// launchers
// ===========================================================================
static int grid_for(int64_t n, int threads, int cap) {
    int64_t g = (n + threads - 1) / threads;
    if (g > cap) g = cap;
    if (g < 1) g = 1;
    return (int)g;
}

// opt the split kernels into their dynamic shared memory size (once per process,
// before any launch or stream capture)
cudaError_t kernels_init() {
    cudaError_t e = umma_init();
    if (e == cudaSuccess) e = slices_init();
    return e != cudaSuccess ? e : lz_init();
}

cudaError_t launch_gg64(const GGArgs& a, cudaStream_t st) {
    if (a.ntiles <= 0) return cudaSuccess;
    if (a.nrhs < 1 || a.nrhs > 65535) return cudaErrorInvalidValue;
    launch_pdl(gg_fp64_kernel, dim3(a.ntiles, a.nrhs), f64k::NT, 0, st, a);
    return cudaGetLastError();
}

cudaError_t launch_prep(const PrepBlock* pb, int nb, const double* src, void* dst, cudaStream_t st) {
    if (nb <= 0) return cudaSuccess;
    if (!pb || !src || !dst) return cudaErrorInvalidValue;
    launch_pdl(prep_kernel, min(nb, 8192), 256, 0, st, pb, nb, src, (__nv_bfloat16*)dst);
    return cudaGetLastError();
}

cudaError_t launch_panel_split(const PanelPiece* pieces, int np, const double* src, void* dst, cudaStream_t st) {
    if (np <= 0) return cudaSuccess;
    if (!pieces || !src || !dst) return cudaErrorInvalidValue;
    launch_pdl(panel_split_kernel<double>, min(np, 4096), 256, 0, st, pieces, np, src, (__nv_bfloat16*)dst);
    return cudaGetLastError();
}
cudaError_t launch_prep_tf32(const PrepBlock* pb, int nb, const double* src, void* dst, cudaStream_t st) {
    if (nb <= 0) return cudaSuccess;
    if (!pb || !src || !dst) return cudaErrorInvalidValue;
    launch_pdl(prep_tf32_kernel, min(nb, 8192), 256, 0, st, pb, nb, src, (float*)dst);
    return cudaGetLastError();
}
cudaError_t launch_panel_split_tf32(const PanelPiece* pieces, int np, const double* src, const float* srcf, void* dst,
                                    cudaStream_t st) {
    if (np <= 0) return cudaSuccess;
    if (!pieces || (!src && !srcf) || !dst) return cudaErrorInvalidValue;
    if (srcf) launch_pdl(panel_split_tf32_kernel<float>, min(np, 4096), 256, 0, st, pieces, np, srcf, (float*)dst);
    else launch_pdl(panel_split_tf32_kernel<double>, min(np, 4096), 256, 0, st, pieces, np, src, (float*)dst);
    return cudaGetLastError();
}
cudaError_t launch_panel_split_f32(const PanelPiece* pieces, int np, const float* src, void* dst, cudaStream_t st) {
    if (np <= 0) return cudaSuccess;
    if (!pieces || !src || !dst) return cudaErrorInvalidValue;
    launch_pdl(panel_split_kernel<float>, min(np, 4096), 256, 0, st, pieces, np, src, (__nv_bfloat16*)dst);
    return cudaGetLastError();
}

cudaError_t launch_trace_pairs(const TracePair* tp, int n, const double* V, const double* LR, double* part,
                               cudaStream_t st) {
    if (n <= 0) return cudaSuccess;
    if (!tp || !V || !LR || !part) return cudaErrorInvalidValue;
    launch_pdl(trace_pairs_kernel, min(n, 4096), kDotThreads, 0, st, tp, n, V, LR, part);
    return cudaGetLastError();
}

cudaError_t launch_transfer_combine(const CombineBlock* cb, int n, const double* V, const double* T, double* out,
                                    const double* part, int np, const double* wm, double* r, cudaStream_t st) {
    if (n <= 0) return cudaSuccess;
    if (!cb || !V || !T || !out || (np > 0 && !part) || (r && !wm)) return cudaErrorInvalidValue;
    launch_pdl(transfer_combine_kernel, dim3(min(n, 4096), n < 152 ? 8 : 1), kDotThreads, 0, st, cb, n, V, T, out, part, np, wm, r);
    return cudaGetLastError();
}

cudaError_t launch_pack(const PackBlock* blocks, int nb, const double* src, double* dst, int to_padded, cudaStream_t st) {
    if (nb <= 0) return cudaSuccess;
    if (!blocks || !src || !dst) return cudaErrorInvalidValue;   // never launch on an unallocated buffer
    launch_pdl(pack_kernel, min(nb, 4096), 256, 0, st, blocks, nb, src, dst, to_padded);
    return cudaGetLastError();
}
// chunked dot: part must hold nchunk doubles
int64_t dot_chunk(int64_t n) {
    const int64_t c = (n + 2047) / 2048;
    return c > 8192 ? c : 8192;
}
int dot_nchunk(int64_t n) { return (int)((n + dot_chunk(n) - 1) / dot_chunk(n)); }
cudaError_t launch_dot(const double* x, const double* y, int64_t n, double* part, double* out, cudaStream_t st) {
    const int64_t ch = dot_chunk(n);
    const int nc = dot_nchunk(n);
    launch_pdl(dot_partial_kernel, nc, kDotThreads, 0, st, x, y, n, ch, part);
    launch_pdl(sum_partial_kernel, 1, kDotThreads, 0, st, part, nc, out);
    return cudaGetLastError();
}
cudaError_t launch_arnoldi_pass(const double* V, int nv, int64_t n, const double* wm, double* w, double* r, double* part,
                                double* coef, cudaStream_t st) {
    if (nv < 1 || nv > kArnoldiMax || n <= 0 || !V || !wm || !w || !r || !part || !coef) return cudaErrorInvalidValue;
    const int64_t ch = dot_chunk(n);
    const int nc = dot_nchunk(n);
    launch_pdl(arnoldi_dot_kernel, dim3(nc, nv), kDotThreads, 0, st, V, n, r, ch, nc, part);
    if (nc > 32) launch_pdl(msum_partial_kernel, nv, kDotThreads, 0, st, part, nc, coef);
    launch_pdl(arnoldi_update_kernel, grid_for(n, 256, 152 * 8), 256, nv * 8, st, V, nv, n, nc > 32 ? nullptr : part, nc, coef, wm,
                                                                         w, r);
    return cudaGetLastError();
}
cudaError_t launch_arnoldi_norm(const double* w, const double* r, int64_t n, double* part, double* out, cudaStream_t st) {
    if (n <= 0 || !w || !r || !part || !out) return cudaErrorInvalidValue;
    launch_pdl(arnoldi_norm_kernel, dot_nchunk(n), kDotThreads, 0, st, w, r, n, dot_chunk(n), part, out);
    return cudaGetLastError();
}
cudaError_t launch_axpy(double a, const double* x, double* y, int64_t n, cudaStream_t st) {
    launch_pdl(axpy_kernel, grid_for(n, 256, 152 * 8), 256, 0, st, a, x, y, n);
    return cudaGetLastError();
}
cudaError_t launch_hadamard(const double* a, const double* b, double* out, int64_t n, cudaStream_t st) {
    if (n <= 0) return cudaSuccess;
    if (!a || !b || !out) return cudaErrorInvalidValue;
    launch_pdl(hadamard_kernel, grid_for(n, 256, 152 * 8), 256, 0, st, a, b, out, n);
    return cudaGetLastError();
}
cudaError_t launch_scale(double a, double* x, int64_t n, cudaStream_t st) { return launch_scale_to(a, x, x, n, st); }
cudaError_t launch_scale_to(double a, const double* x, double* y, int64_t n, cudaStream_t st) {
    launch_pdl(scale_kernel, grid_for(n, 256, 152 * 8), 256, 0, st, a, x, y, n);
    return cudaGetLastError();
}
cudaError_t launch_combine(const double* V, int nv, int64_t n, const double* c, double* y, cudaStream_t st) {
    launch_pdl(combine_kernel, grid_for(n, 256, 152 * 8), 256, 0, st, V, nv, n, c, y);
    return cudaGetLastError();
}
cudaError_t launch_splitk_reduce(const void* part, int nparts, int64_t n, void* out, int f32, cudaStream_t st) {
    if (n <= 0) return cudaSuccess;
    if (!part || !out || nparts < 1) return cudaErrorInvalidValue;
    if (f32) launch_pdl(splitk_reduce_kernel<float>, grid_for(n, 256, 152 * 8), 256, 0, st, (const float*)part, nparts, n, (float*)out);
    else launch_pdl(splitk_reduce_kernel<double>, grid_for(n, 256, 152 * 8), 256, 0, st, (const double*)part, nparts, n, (double*)out);
    return cudaGetLastError();
}
cudaError_t launch_penalty(const PenaltyArgs& a, const double* y, const float* yf, double* o, float* of,
                           cudaStream_t st) {
    if (a.npen <= 0 || a.nrhs <= 0) return cudaSuccess;
    if (!a.dvec || !a.avec || !a.part || !a.coef || (!y && !yf) || (!o && !of) || a.chunk <= 0 ||
        (int64_t)a.nchunk * a.chunk < a.n)
        return cudaErrorInvalidValue;
    const dim3 gd(a.nchunk, a.npen * a.nrhs);
    if (yf) launch_pdl(pen_dot_kernel<float>, gd, kDotThreads, 0, st, a, yf);
    else launch_pdl(pen_dot_kernel<double>, gd, kDotThreads, 0, st, a, y);
    launch_pdl(pen_sum_kernel, a.npen * a.nrhs, kDotThreads, 0, st, a);
    const dim3 ga(grid_for(a.n, 256, 152 * 4), a.nrhs);
    if (of) launch_pdl(pen_add_kernel<float>, ga, 256, 0, st, a, of);
    else launch_pdl(pen_add_kernel<double>, ga, 256, 0, st, a, o);
    return cudaGetLastError();
}
cudaError_t launch_finite(const double* x, int64_t n, int* bad, cudaStream_t st) {
    launch_pdl(finite_kernel, grid_for(n, 256, 152 * 8), 256, 0, st, x, n, bad);
    return cudaGetLastError();
}

}  // namespace vmps
