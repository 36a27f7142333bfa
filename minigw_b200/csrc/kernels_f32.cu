// kernels_f32.cu -- the mixed-precision form of the screening (GWB200_MIXED, eta == 0).
//
// Same algorithm as kernels_fp64.cu (tall matrix [eps ; (D^1/2 X)^T], right-looking blocked
// Cholesky, squared row norms), with:
//   * the tall matrices stored in FP32 (eps has eigenvalues >= 1, entries O(1..100)), halving HBM
//     footprint and traffic;
//   * each 64x64 diagonal block factored and inverted in FP64 in shared memory, stored as FP32;
//   * the panel solve and the trailing updates on the tensor cores (mma.sync m16n8k8 TF32; the updates
//     on tcgen05 where kernels_tc.cu takes them) with the 3xTF32 split (a = a_hi + a_lo, each a TF32 value; a*b ~ a_hi b_hi + a_hi b_lo +
//     a_lo b_hi, accumulated in FP32), about 21 significant bits per product;
//   * the squared norms, the G0 frequency contraction, Pade and QP in FP64.
// There is no FP64 refinement: the result carries FP32-level error (stated, not hidden, by
// bench.py and the tests).
#include "panel_common.cuh"
#include "tc_common.cuh"

#include <cmath>

namespace gwb200 {
namespace {

constexpr int kLdf = 68;  // padded shared row stride (floats) of a 64-wide FP32 tile
constexpr int kKcf = 32;  // K slice of the pipelined FP32 update
constexpr int kLdkf = kKcf + 4;

__device__ __forceinline__ unsigned to_tf32(float x) {
    unsigned r;
    asm("cvt.rna.tf32.f32 %0, %1;\n" : "=r"(r) : "f"(x));
    return r;
}
__device__ __forceinline__ void split_tf32(float x, unsigned& hi, unsigned& lo) {
    hi = to_tf32(x);
    lo = to_tf32(x - __uint_as_float(hi));
}
__device__ __forceinline__ void mma_tf32(float (&c)[4], const unsigned (&a)[4], unsigned b0, unsigned b1) {
    asm volatile("mma.sync.aligned.m16n8k8.row.col.f32.tf32.tf32.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, "
                 "{%0,%1,%2,%3};\n"
                 : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
                 : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}

// acc += sgn * As(64 x KD) * Bs(64 x KD)^T, FP32 tiles in shared memory with row stride LD.
// 8 warps as 4 (rows) x 2 (cols): warp tile 16 x 32 = one m16 tile by four n8 tiles.
// Fragments (PTX ISA, mma.m16n8k8 .tf32): A a0..a3 = (g,t) (g+8,t) (g,t+4) (g+8,t+4);
// B b0,b1 = (k=t, n=g) (k=t+4, n=g); C c0..c3 = (g,2t) (g,2t+1) (g+8,2t) (g+8,2t+1).
template <int LD, int KD>
__device__ __forceinline__ void tile_mma_3xtf32(const float* __restrict__ As, const float* __restrict__ Bs,
                                                float (&acc)[4][4], float sgn) {
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const int g = lane >> 2, t = lane & 3;
    const int r0 = 16 * (w >> 1), c0 = 32 * (w & 1);
#pragma unroll 2
    for (int kk = 0; kk < KD; kk += 8) {
        unsigned ah[4], al[4];
        split_tf32(sgn * As[(r0 + g) * LD + kk + t], ah[0], al[0]);
        split_tf32(sgn * As[(r0 + g + 8) * LD + kk + t], ah[1], al[1]);
        split_tf32(sgn * As[(r0 + g) * LD + kk + t + 4], ah[2], al[2]);
        split_tf32(sgn * As[(r0 + g + 8) * LD + kk + t + 4], ah[3], al[3]);
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            unsigned bh0, bl0, bh1, bl1;
            split_tf32(Bs[(c0 + 8 * j + g) * LD + kk + t], bh0, bl0);
            split_tf32(Bs[(c0 + 8 * j + g) * LD + kk + t + 4], bh1, bl1);
            mma_tf32(acc[j], al, bh0, bh1);
            mma_tf32(acc[j], ah, bl0, bl1);
            mma_tf32(acc[j], ah, bh0, bh1);
        }
    }
}

// The C fragments of tile_mma_3xtf32 to a 64 x 64 tile in shared memory (row stride LD).
template <int LD>
__device__ __forceinline__ void store_fragments(float* __restrict__ s, const float (&acc)[4][4], int w) {
    const int lane = threadIdx.x & 31;
    const int g = lane >> 2, t = lane & 3;
    const int r0 = 16 * (w >> 1), c0 = 32 * (w & 1);
#pragma unroll
    for (int j = 0; j < 4; ++j)
#pragma unroll
        for (int h = 0; h < 2; ++h)
            *reinterpret_cast<float2*>(s + (r0 + g + 8 * h) * LD + c0 + 8 * j + 2 * t) =
                make_float2(acc[j][2 * h], acc[j][2 * h + 1]);
}

// 64 x W floats of global (row stride ld) into shared memory (row stride LD), 16-byte pieces.
template <int W, int LD>
__device__ __forceinline__ void load_f32_async(float* __restrict__ s, const float* __restrict__ gsrc, int64_t ld) {
    for (int idx = threadIdx.x; idx < 64 * (W / 4); idx += blockDim.x) {
        const int r = idx / (W / 4), c4 = idx % (W / 4);
        panel::cp_async16(s + r * LD + 4 * c4, gsrc + (size_t)r * ld + 4 * c4);
    }
}

// Tall FP32 matrices: eps lower triangle (computed in FP64, rounded) and (D^1/2 X)^T rows.
__global__ void k_build_tall32(int64_t n, int64_t m, int64_t n_pad, int64_t ld, int64_t stride, int64_t rows,
                               const double* __restrict__ v, const double* __restrict__ xt,
                               const double* __restrict__ dvec, int nf, float* __restrict__ a) {
    const int64_t c = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (c >= n_pad) return;
    for (int64_t r = blockIdx.y; r < rows; r += gridDim.y) {
        if (r < n_pad) {
            if (c > r) continue;
            const double vrc = (r < n && c < n) ? v[r * n + c] : 0.0;
            const double diag = (r == c) ? 1.0 : 0.0;
            for (int f = 0; f < nf; ++f) {
                const double* d = dvec + (size_t)f * n_pad;
                a[(size_t)f * stride + r * ld + c] = (float)fma(d[r] * vrc, d[c], diag);
            }
        } else {
            const int64_t j = r - n_pad;
            const double x = (j < m && c < n) ? xt[j * n + c] : 0.0;
            for (int f = 0; f < nf; ++f) a[(size_t)f * stride + r * ld + c] = (float)(dvec[(size_t)f * n_pad + c] * x);
        }
    }
}

// Diagonal step of outer block [k, k + NB): the 64 x 64 diagonal blocks are factored and inverted
// in FP64 (panel_common.cuh) and their inverses, rounded to FP32, replace them in the tall matrix;
// for NB = 128 the block between them is solved (L21 = A21 L11^{-T}) and the second diagonal block
// updated (A22 -= L21 L21^T) in 3xTF32 first, as for the rows below.  One CTA per matrix.
constexpr size_t kDiag32Smem = panel::DiagShape<kNb>::kSmem + 2 * 64 * kLdf * sizeof(float);

template <int NB>
__global__ void __launch_bounds__(256) k_diag32(float* __restrict__ a, int64_t ld, int64_t stride, int64_t k,
                                                unsigned long long* err_pivot) {
    extern __shared__ __align__(16) double smem[];
    using Sh = panel::DiagShape<kNb>;
    constexpr int LD = Sh::kLd;
    double* S = smem;
    double* work = S + Sh::kBlockDoubles;
    float* Yf = reinterpret_cast<float*>(work + Sh::kWorkDoubles);
    float* Pf = Yf + 64 * kLdf;
    const int tid = threadIdx.x;
    float* A = a + (size_t)blockIdx.x * stride + k * ld + k;
    for (int idx = tid; idx < kNb * LD; idx += 256) {
        const int i = idx / LD, j = idx % LD;
        S[idx] = j <= i ? (double)A[(size_t)i * ld + j] : 0.0;
    }
    if (NB == 128) load_f32_async<64, kLdf>(Pf, A + (size_t)kNb * ld, ld);
    asm volatile("cp.async.commit_group;\n" ::);
    auto inverse_out = [&](float* dst) {
        for (int idx = tid; idx < kNb * kNb; idx += 256) {
            const int i = idx / kNb, j = idx % kNb;
            const float y = j <= i ? (float)S[j * LD + i + 1] : 0.0f;
            Yf[i * kLdf + j] = y;
            dst[(size_t)i * ld + j] = y;
        }
    };
    __syncthreads();
    panel::factor_diag<kNb>(S, work, k, err_pivot);
    inverse_out(A);
    if (NB == 128) {
        const int lane = tid & 31, w = tid >> 5;
        const int g = lane >> 2, t = lane & 3;
        const int rr = 16 * (w >> 1), cc = 32 * (w & 1);
        float* A21 = A + (size_t)kNb * ld;
        float* A22 = A21 + kNb;
        asm volatile("cp.async.wait_group 0;\n" ::);
        __syncthreads();
        float acc[4][4] = {};
        tile_mma_3xtf32<kLdf, 64>(Pf, Yf, acc, 1.0f);
        __syncthreads();
        store_fragments<kLdf>(Pf, acc, w);
        __syncthreads();
        for (int idx = tid; idx < 64 * 16; idx += 256) {
            const int r = idx >> 4, c4 = idx & 15;
            *reinterpret_cast<float4*>(A21 + (size_t)r * ld + 4 * c4) = *reinterpret_cast<const float4*>(Pf + r * kLdf + 4 * c4);
        }
        float upd[4][4] = {};
        tile_mma_3xtf32<kLdf, 64>(Pf, Pf, upd, -1.0f);
#pragma unroll
        for (int j = 0; j < 4; ++j)
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                const int i = rr + g + 8 * (e >> 1), c = cc + 8 * j + 2 * t + (e & 1);
                S[i * LD + c] = c <= i ? (double)(A22[(size_t)i * ld + c] + upd[j][e]) : 0.0;
            }
        if (tid < kNb) S[tid * LD + kNb] = 0.0;  // the last identity column
        __syncthreads();
        panel::factor_diag<kNb>(S, work, k + kNb, err_pivot);
        inverse_out(A22);
    }
}

// The rows below an outer block, from row0 on: P1 = A1 L11^{-T}, A2 -= P1 L21^T, P2 = A2 L22^{-T}
// (3xTF32; a 64-wide block is P1 alone), in one pass with the block's three tiles kept in shared
// memory.  Every warp walks 16-row tiles of its own, all 64 output columns of a product at once, so
// nothing but the warp is ever waited for.  Bound by the mma.sync TF32 rate (470 multiply-adds per
// clock and SM, 5,000 cycles per 64 rows); with 16 x 32 warp tiles that split both operands at every
// use and a barrier between the products it took 14,500.  The block's tiles are split once per CTA,
// the two parts of a lane's two k values together (one 16-byte load per column tile and k step).  2000 pairs, 64 frequencies: 101 -> 74 us a launch.
//   solve_row0  rows before it are finished (the solve-only pass): passed through to `panel` alone
//   rows_end    rows to write to `panel` (beyond `rows` zeros)
//   panel       the solved rows' hi / lo parts for the tcgen05 update (the layout of kernels_tc.cu);
//               null: none
//   keep        write the solved rows back to the tall matrix
//   qacc        squared norms (FP64) of the right-hand-side rows are added; null: none
constexpr int kPanelWarps = 12;
constexpr int kLdy = 144;        // split block row: 64 k as (hi, hi, lo, lo) of k, k + 4; = 16 mod 32 words
constexpr int kBlk = 64 * kLdy;  // one split block
template <int NB>
constexpr int kLdr = NB + 4;  // a warp's row stride
template <int NB>
constexpr size_t kPanel32Smem = sizeof(float) * ((NB == 128 ? 3 : 1) * kBlk + kPanelWarps * 16 * kLdr<NB>);

// acc += sgn * (16 x 64 rows at X, stride LD) * (split block B)^T, the products of a k step in the order
// lo.hi, hi.lo, hi.hi.
template <int LD>
__device__ __forceinline__ void rows_mma(const float* __restrict__ X, const float* __restrict__ B, float (&acc)[8][4],
                                         float sgn) {
    const int lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
    const float* x0 = X + g * LD + t;
    const float* b0 = B + g * kLdy + 4 * t;
#pragma unroll 2
    for (int k8 = 0; k8 < 8; ++k8) {
        unsigned ah[4], al[4];
        split_tf32(sgn * x0[8 * k8], ah[0], al[0]);
        split_tf32(sgn * x0[8 * LD + 8 * k8], ah[1], al[1]);
        split_tf32(sgn * x0[8 * k8 + 4], ah[2], al[2]);
        split_tf32(sgn * x0[8 * LD + 8 * k8 + 4], ah[3], al[3]);
#pragma unroll
        for (int j = 0; j < 8; ++j) {
            const uint4 b = *reinterpret_cast<const uint4*>(b0 + 8 * j * kLdy + 16 * k8);
            mma_tf32(acc[j], al, b.x, b.y);
            mma_tf32(acc[j], ah, b.z, b.w);
            mma_tf32(acc[j], ah, b.x, b.y);
        }
    }
}

template <int NB>
__global__ void __launch_bounds__(32 * kPanelWarps, 1)
    k_panel32(float* __restrict__ a, int64_t ld, int64_t stride, int64_t k, int64_t row0, int64_t rows, int64_t rows_end,
              int64_t solve_row0, int64_t n_pad, float* __restrict__ panel, int keep, double* __restrict__ qacc,
              int64_t ldq) {
    extern __shared__ __align__(16) float fsm[];
    constexpr int kBlocks = NB == 128 ? 3 : 1;  // L11^{-1}, L21, L22^{-1}
    constexpr int LD = kLdr<NB>;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int g = lane >> 2, t = lane & 3;
    float* B = fsm;
    float* X = B + kBlocks * kBlk + warp * 16 * LD;
    float* A = a + (size_t)blockIdx.y * stride;
    {
        const float* D = A + (size_t)k * ld + k;
        for (int idx = threadIdx.x; idx < kBlocks * 64 * 32; idx += 32 * kPanelWarps) {
            const int blk = idx >> 11, r = (idx >> 5) & 63, k8 = (idx >> 2) & 7, tt = idx & 3;
            const float* src = D + (size_t)(r + (blk > 0 ? kNb : 0)) * ld + 8 * k8 + tt + (blk > 1 ? kNb : 0);
            uint4 v;
            split_tf32(src[0], v.x, v.z);
            split_tf32(src[4], v.y, v.w);
            *reinterpret_cast<uint4*>(B + blk * kBlk + r * kLdy + 16 * k8 + 4 * tt) = v;
        }
    }
    __syncthreads();
    const int64_t rp = rows_end - row0;
    float4* hi = reinterpret_cast<float4*>(panel + (size_t)blockIdx.y * 2 * (NB / 32) * rp * 32);
    float4* lo = hi + (size_t)(NB / 32) * rp * 8;
    auto store = [&](int col, const float (&acc)[8][4]) {  // fragments to this warp's rows
#pragma unroll
        for (int j = 0; j < 8; ++j)
#pragma unroll
            for (int h = 0; h < 2; ++h)
                *reinterpret_cast<float2*>(X + (g + 8 * h) * LD + col + 8 * j + 2 * t) =
                    make_float2(acc[j][2 * h], acc[j][2 * h + 1]);
    };
    for (int64_t r0 = row0 + (int64_t)(kPanelWarps * blockIdx.x + warp) * 16; r0 < rows_end;
         r0 += (int64_t)kPanelWarps * gridDim.x * 16) {
        const bool inside = r0 < rows;
        const bool solve = inside && r0 >= solve_row0;
        if (inside) {
            const float* src = A + (size_t)r0 * ld + k;
            for (int idx = lane; idx < 16 * (NB / 4); idx += 32)
                panel::cp_async16(X + idx / (NB / 4) * LD + 4 * (idx % (NB / 4)),
                                  src + (size_t)(idx / (NB / 4)) * ld + 4 * (idx % (NB / 4)));
        }
        asm volatile("cp.async.commit_group;\n" ::);
        asm volatile("cp.async.wait_group 0;\n" ::);
        __syncwarp();
        if (solve) {
            double s[2] = {0.0, 0.0};  // squared norms of rows g and g + 8, this lane's columns
            auto add_norms = [&](const float (&acc)[8][4]) {
#pragma unroll
                for (int j = 0; j < 8; ++j)
#pragma unroll
                    for (int e = 0; e < 4; ++e) {
                        const double y = (double)acc[j][e];
                        s[e >> 1] = fma(y, y, s[e >> 1]);
                    }
            };
            const bool norms = qacc && r0 >= n_pad;
            {
                float acc[8][4] = {};
                rows_mma<LD>(X, B, acc, 1.0f);
                __syncwarp();
                store(0, acc);
                if (norms) add_norms(acc);
                __syncwarp();
            }
            if (NB == 128) {
                {
                    float upd[8][4] = {};
                    rows_mma<LD>(X, B + kBlk, upd, -1.0f);
#pragma unroll
                    for (int j = 0; j < 8; ++j)
#pragma unroll
                        for (int h = 0; h < 2; ++h) {
                            float2* p = reinterpret_cast<float2*>(X + (g + 8 * h) * LD + kNb + 8 * j + 2 * t);
                            float2 v = *p;
                            v.x += upd[j][2 * h];
                            v.y += upd[j][2 * h + 1];
                            *p = v;
                        }
                    __syncwarp();
                }
                float acc[8][4] = {};
                rows_mma<LD>(X + kNb, B + 2 * kBlk, acc, 1.0f);
                __syncwarp();
                store(kNb, acc);
                if (norms) add_norms(acc);
                __syncwarp();
            }
            if (norms) {
#pragma unroll
                for (int h = 0; h < 2; ++h) {
                    s[h] += __shfl_xor_sync(0xffffffffu, s[h], 1);
                    s[h] += __shfl_xor_sync(0xffffffffu, s[h], 2);
                    if (t == 0) qacc[(size_t)blockIdx.y * ldq + (r0 - n_pad + g + 8 * h)] += s[h];
                }
            }
        }
        for (int idx = lane; idx < 16 * (NB / 4); idx += 32) {
            const int r = idx / (NB / 4), c4 = idx % (NB / 4);
            float4 x = make_float4(0.f, 0.f, 0.f, 0.f);
            if (inside) x = *reinterpret_cast<const float4*>(X + r * LD + 4 * c4);
            if (solve && keep) *reinterpret_cast<float4*>(A + (size_t)(r0 + r) * ld + k + 4 * c4) = x;
            if (panel) {
                unsigned h[4], l[4];
                split_tf32(x.x, h[0], l[0]);
                split_tf32(x.y, h[1], l[1]);
                split_tf32(x.z, h[2], l[2]);
                split_tf32(x.w, h[3], l[3]);
                const int64_t rr = r0 - row0 + r;
                const size_t dst = ((size_t)(c4 >> 3) * rp + rr) * 8 + ((c4 & 7) ^ (int)(rr & 7));  // K slice of 32, chunk
                hi[dst] = make_float4(__uint_as_float(h[0]), __uint_as_float(h[1]), __uint_as_float(h[2]), __uint_as_float(h[3]));
                lo[dst] = make_float4(__uint_as_float(l[0]), __uint_as_float(l[1]), __uint_as_float(l[2]), __uint_as_float(l[3]));
            }
        }
        __syncwarp();
    }
}

// Trailing update on FP32 tiles (3xTF32), same tile enumeration and K chunking as the
// FP64 k_update: output column tiles [tc0, tc0+T), lower square tiles then all RHS tiles
// (rhs_only: the RHS tiles alone, for the solve-only pass against a finished factor).
__global__ void __launch_bounds__(256, 3) k_update32(float* __restrict__ a, int64_t ld, int64_t stride, int64_t kb0,
                                                     int nk, int64_t tc0, int64_t T, int64_t nsq, int rhs_only) {
    extern __shared__ float fsm[];
    auto stage = [&](int st, int which) { return fsm + (2 * st + which) * 64 * kLdkf; };
    const int f = blockIdx.y;
    const int64_t Lr = nsq - tc0;
    const int64_t n_square = rhs_only ? 0 : T * Lr - T * (T - 1) / 2;
    const int64_t x = blockIdx.x;
    int64_t c, tr;
    if (x < n_square) {
        const double b = 2.0 * (double)Lr + 1.0;
        c = (int64_t)((b - sqrt(fmax(b * b - 8.0 * (double)x, 0.0))) * 0.5);
        auto cum = [Lr](int64_t cc) { return cc * Lr - cc * (cc - 1) / 2; };
        while (c > 0 && cum(c) > x) --c;
        while (c + 1 < T && cum(c + 1) <= x) ++c;
        tr = tc0 + c + (x - cum(c));
    } else {
        const int64_t y = x - n_square;
        c = y % T;
        tr = nsq + y / T;
    }
    const int64_t ri = tr * kNb, cj = (tc0 + c) * kNb;
    float* A = a + (size_t)f * stride;
    const int nsub = nk * (kNb / kKcf);
    load_f32_async<kKcf, kLdkf>(stage(0, 0), A + ri * ld + kb0, ld);
    load_f32_async<kKcf, kLdkf>(stage(0, 1), A + cj * ld + kb0, ld);
    asm volatile("cp.async.commit_group;\n" ::);
    float acc[4][4] = {};
    for (int sc = 0; sc < nsub; ++sc) {
        if (sc + 1 < nsub) {
            const int64_t kc = kb0 + (int64_t)(sc + 1) * kKcf;
            load_f32_async<kKcf, kLdkf>(stage((sc + 1) & 1, 0), A + ri * ld + kc, ld);
            load_f32_async<kKcf, kLdkf>(stage((sc + 1) & 1, 1), A + cj * ld + kc, ld);
            asm volatile("cp.async.commit_group;\n" ::);
            asm volatile("cp.async.wait_group 1;\n" ::);
        } else {
            asm volatile("cp.async.wait_group 0;\n" ::);
        }
        __syncthreads();
        tile_mma_3xtf32<kLdkf, kKcf>(stage(sc & 1, 0), stage(sc & 1, 1), acc, -1.0f);
        __syncthreads();
    }
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const int g = lane >> 2, t = lane & 3;
    const int rr = 16 * (w >> 1), cc = 32 * (w & 1);
#pragma unroll
    for (int j = 0; j < 4; ++j) {
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            float2* pc = reinterpret_cast<float2*>(A + (size_t)(ri + rr + g + 8 * h) * ld + cj + cc + 8 * j + 2 * t);
            float2 v = *pc;
            v.x += acc[j][2 * h];
            v.y += acc[j][2 * h + 1];
            *pc = v;
        }
    }
}

double update_flops32(const TallGeometry& g, int64_t kb0, int nk, int64_t c0, int64_t c1) {
    const int64_t kt = std::max<int64_t>(0, std::min<int64_t>(kb0 + (int64_t)nk * kNb, g.n) - kb0);
    const int64_t a0 = std::min(c0, g.n), a1 = std::min(c1, g.n);
    const double cols = (double)(a1 - a0);
    const double lower = cols * (double)g.n - 0.5 * (double)(a0 + a1 - 1) * cols;
    return 2.0 * (double)kt * (lower + (double)g.m * cols);
}

} // namespace

int launch_build_tall32(const TallGeometry& g, const double* v, const double* xt, const double* dvec, int64_t nf,
                        float* a, cudaStream_t s) {
    dim3 grid((unsigned)((g.n_pad + 255) / 256), (unsigned)std::min<int64_t>(g.rows, 65535));
    k_build_tall32<<<grid, 256, 0, s>>>(g.n, g.m, g.n_pad, g.ld, g.stride, g.rows, v, xt, dvec, (int)nf, a);
    GWB_LAUNCH("k_build_tall32");
    return 1;
}

namespace {

template <int NB>
void launch_diag32(const TallGeometry& g, int64_t nf, float* a, int64_t k, unsigned long long* err_pivot, cudaStream_t s) {
    GWB_CUDA(cudaFuncSetAttribute(k_diag32<NB>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kDiag32Smem));
    k_diag32<NB><<<(unsigned)nf, 256, kDiag32Smem, s>>>(a, g.ld, g.stride, k, err_pivot);
    GWB_LAUNCH("k_diag32");
}

// the rows below a diagonal block: all of them for the update's operands, else while factoring; the
// solve-only pass works on the right-hand sides alone
template <int NB>
int launch_rows32(const TallGeometry& g, int64_t nf, float* a, int64_t k, double* qacc, cudaStream_t s, float* panel,
                  bool solve_only, bool keep) {
    const int64_t row0 = solve_only && !panel ? g.n_pad : k + NB;
    const int64_t rows_end = panel ? row0 + tc_panel_rows(g, row0) : g.rows;
    const int64_t tiles = (rows_end - row0) / 16;
    if (tiles <= 0) return 0;
    GWB_CUDA(cudaFuncSetAttribute(k_panel32<NB>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kPanel32Smem<NB>));
    const int64_t gx = panel_grid((tiles + kPanelWarps - 1) / kPanelWarps, nf, 1);
    k_panel32<NB><<<dim3((unsigned)gx, (unsigned)nf), 32 * kPanelWarps, kPanel32Smem<NB>, s>>>(
        a, g.ld, g.stride, k, row0, g.rows, rows_end, solve_only ? g.n_pad : row0, g.n_pad, panel, keep ? 1 : 0, qacc,
        g.m_pad);
    GWB_LAUNCH("k_panel32");
    return 1;
}

}  // namespace

int launch_factor_chunk32(const TallGeometry& g, int64_t nf, float* a, double* qacc, unsigned long long* err_pivot,
                          cudaStream_t s, UpdateProfiler* prof, float* panel, unsigned long long* sched, int max_ctas,
                          bool keep_rows, bool solve_only, SideStream* side) {
    const size_t smem_update = 4 * 64 * kLdkf * sizeof(float);
    GWB_CUDA(cudaFuncSetAttribute(k_update32, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem_update));
    const int64_t nsq = g.n_pad / kNb, nrt = g.rows / kNb;
    constexpr int64_t kOuter = 2;
    int launches = 0;
    if (panel && nsq > kOuter) launches += launch_clear_sched(g, sched, s);
    // As in the plain form the next diagonal block is factored beside the trailing update; its own update
    // comes first, from the same kernel (its rounding is the form's): 2000 pairs x 64 frequencies 5029 -> 4912
    // us.  (Not in batches, whose lanes already overlap, nor in the refinement's solve.)
    if (prof || max_ctas > 0 || solve_only || !panel || nf >= tc::sm_count()) side = nullptr;
    auto diag = [&](int64_t ob) {
        if (solve_only) return;
        nsq - ob >= kOuter ? launch_diag32<128>(g, nf, a, ob * kNb, err_pivot, s)
                           : launch_diag32<64>(g, nf, a, ob * kNb, err_pivot, s);
        ++launches;
    };
    diag(0);
    for (int64_t ob = 0; ob < nsq; ob += kOuter) {
        const int64_t q = std::min(kOuter, nsq - ob), tc0 = ob + q;
        float* pan = tc0 < nsq ? panel : nullptr;  // operands of the trailing update, when there is one
        const bool keep = keep_rows || !panel;     // the mma.sync update reads the rows themselves
        launches += q == kOuter ? launch_rows32<128>(g, nf, a, ob * kNb, qacc, s, pan, solve_only, keep)
                                : launch_rows32<64>(g, nf, a, ob * kNb, qacc, s, pan, solve_only, keep);
        if (tc0 >= nsq) break;
        if (prof) prof->begin();
        if (side) {
            unsigned long long* counter = sched + ob / kOuter;
            launches += launch_update32_tc(g, nf, a, tc0 * kNb, pan, counter + sched_slots(g), err_pivot, s, 0, 0,
                                           TileRows::kFirst);
            SideScope beside(side, s);
            diag(tc0);
            launches += launch_update32_tc(g, nf, a, tc0 * kNb, pan, counter, err_pivot, beside.stream(), 0, 0,
                                           TileRows::kRest);
            beside.join();
        } else if (pan) {  // trailing update on tcgen05
            launches += launch_update32_tc(g, nf, a, tc0 * kNb, pan, sched + ob / kOuter, err_pivot, s, max_ctas,
                                           solve_only ? g.n_pad : 0);
        } else {
            const int64_t T = nsq - tc0;
            const int64_t tiles = (solve_only ? 0 : T * (T + 1) / 2) + T * (nrt - nsq);
            if (tiles > 0) {
                k_update32<<<dim3((unsigned)tiles, (unsigned)nf), 256, smem_update, s>>>(
                    a, g.ld, g.stride, ob * kNb, (int)q, tc0, T, nsq, solve_only ? 1 : 0);
                GWB_LAUNCH("k_update32");
                ++launches;
            }
        }
        if (prof) prof->end((double)nf * update_flops32(g, ob * kNb, (int)q, tc0 * kNb, nsq * kNb));
        if (!side) diag(tc0);
    }
    return launches;
}

} // namespace gwb200
