// panel_common.cuh -- the diagonal-block step of the blocked Cholesky: one CTA factors a 64- or
// 128-wide diagonal block in shared memory and forms its inverse factor on the way.
//
// What bounds it: a chain of NB dependent pivots.  Factoring the tall block [A ; I] instead of A
// makes the identity rows come out as I L^{-T}, the transposed inverse, with no chain of their own
// (a separate forward substitution is as long as the factorisation).  The columns are taken in
// panels of 16.  One warp holds a panel's 16 rows of A (lanes 0-15) and 16 identity rows (lanes
// 16-31) in registers and takes four columns at a time: every lane factors the 4 x 4 pivot block by
// itself, so a pivot costs a reciprocal square root and two multiply-adds (~65 cycles) and only one
// exchange through shared memory (~37 cycles) follows per four columns.  (Sixteen single columns
// with shuffled operands: ~375 cycles each.)  The remaining rows follow as FP64 tensor-core
// (m8n8k4) products over all warps, the next panel's diagonal block first, so that the other tiles
// are updated while warp 0 factors it.
#pragma once

#include "internal.cuh"

namespace gwb200 {
namespace panel {

constexpr int kWtLd = 20;  // row stride of the 16 x 16 inverse of a panel's diagonal block

template <int NB>
struct DiagShape {
    // Row stride (doubles) of the block: column j of L at [i][j] (j <= i), the identity row r's
    // column c at [r][c + 1] (c >= r), so the two triangles share one array.  = 4 mod 16: the 8
    // rows x 4 columns of one m8n8k4 fragment fall on distinct banks.
    static constexpr int kLd = NB + 4;
    static constexpr int kBlockDoubles = NB * kLd;
    // two 16 x 16 inverses of diagonal panels, warp 0's two row buffers [16][4] and pivot block [4][4]
    static constexpr int kWorkDoubles = 2 * 16 * kWtLd + 2 * 64 + 16;
    static constexpr size_t kSmem = sizeof(double) * (size_t)(kBlockDoubles + kWorkDoubles);
    static constexpr int kThreads = 4 * NB;  // enough warps to update the trailing tiles beside warp 0
};

// sqrt(D) with D = -Pi0(i w) = 4 delta / (w^2 + delta^2), rounded the same wherever it is formed.
__device__ __forceinline__ double scale_value(double delta, double w) {
    return sqrt(__dmul_rn(4.0, delta) / __fma_rn(w, w, __dmul_rn(delta, delta)));
}

// One m8n8k4 product.  Fragments (PTX ISA, mma.m8n8k4 .f64): a = A[lane/4][lane%4], b = B[lane%4][lane/4],
// c = C[lane/4][2*(lane%4)] and the next.
__device__ __forceinline__ void dmma(double (&c)[2], double a, double b) {
    asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0,%1}, {%2}, {%3}, {%0,%1};\n"
                 : "+d"(c[0]), "+d"(c[1])
                 : "d"(a), "d"(b));
}

// 16 bytes of global to shared memory, asynchronously
template <class T>
__device__ __forceinline__ void cp_async16(T* dst, const T* src) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"((unsigned)__cvta_generic_to_shared(dst)), "l"(src));
}

// d > 0 (infinity included, NaN not), on the integer pipe
__device__ __forceinline__ bool is_positive(double d) {
    const long long b = __double_as_longlong(d);
    return b > 0 && b <= 0x7ff0000000000000LL;
}

// 1 / sqrt(d) from the hardware's ~2^-20 approximation y by one step of Householder's third-order
// iteration: e = 1 - d y^2, y (1 + e / 2 + 3 e^2 / 8), error ~e^3; d positive, finite and normal.
__device__ __forceinline__ double rsqrt_iter(double d) {
    double y;
    asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(d));
    const double e = fma(-d, y * y, 1.0);
    return fma(fma(0.375, e, 0.5), y * e, y);
}

// The 4 x 4 pivot block l (lower triangle) factored in place by every lane, with 1 / L_jj in rs.
// kPlain: pairs of columns with both square roots at once -- the second pivot of [a b; b c] is
// det / a, det = a c - b^2, and 1 / sqrt(det / a) = rsqrt(det) a rsqrt(a) -- which shortens the
// chain by a third; values outside [2^-500, 2^500] (anything that is not a plain positive number)
// are reported in `odd` and the caller starts over without kPlain: there a pivot that is not > 0 is
// recorded in `bad` and counts as 1, and tiny or infinite ones are clamped to the normal range.
template <bool kPlain>
__device__ __forceinline__ void factor_pivots4(double (&l)[4][4], double (&rs)[4], int q, unsigned& bad) {
    if (kPlain) {
        auto plain = [](double d) { return (unsigned)(__double2hiint(d) - 0x20b00000) <= 0x3e800000u; };
#pragma unroll
        for (int j = 0; j < 4; j += 2) {
            const double a = l[j][j], b = l[j + 1][j], c = l[j + 1][j + 1];
            const double det = fma(a, c, -(b * b));
            rs[j] = rsqrt_iter(a);
            const double rdet = rsqrt_iter(det);
            rs[j + 1] = rdet * (a * rs[j]);
            bad |= (unsigned)!(plain(a) && plain(c) && plain(det));
            l[j + 1][j] = b * rs[j];
            if (j == 0) {
#pragma unroll
                for (int i = 2; i < 4; ++i) {
                    l[i][0] *= rs[0];
                    l[i][1] = fma(-l[i][0], l[1][0], l[i][1]) * rs[1];
                }
#pragma unroll
                for (int i = 2; i < 4; ++i)
#pragma unroll
                    for (int k = 2; k <= i; ++k)
                        l[i][k] = fma(-l[i][1], l[k][1], fma(-l[i][0], l[k][0], l[i][k]));
            }
        }
    } else {
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const double d = l[j][j];
            const bool fails = !is_positive(d);
            bad |= (unsigned)fails << (q + j);
            const int hi = min(max(__double2hiint(d), 0x00100000), 0x7fefffff);
            rs[j] = fails ? 1.0 : rsqrt_iter(__hiloint2double(hi, __double2loint(d)));
#pragma unroll
            for (int i = j + 1; i < 4; ++i) l[i][j] *= rs[j];
#pragma unroll
            for (int c = j + 1; c < 4; ++c)
#pragma unroll
                for (int i = c; i < 4; ++i) l[i][c] = fma(-l[i][j], l[c][j], l[i][c]);
        }
    }
}

// One warp: the 16 x 16 diagonal block at column c0 of S (lower triangle) in registers (lanes
// 0-15), with 16 identity rows (lanes 16-31), four columns at a time.  Returns `bad` of
// factor_pivots4 (kPlain: non-zero if the block has to be done without it).
template <int LD, bool kPlain>
__device__ __forceinline__ unsigned factor_rows16(const double* __restrict__ S, double (&x)[16],
                                                  double* __restrict__ rows2, double* __restrict__ piv, int c0) {
    const int lane = threadIdx.x & 31, r = lane & 15;
    const bool ident = lane >= 16;
#pragma unroll
    for (int c = 0; c < 16; ++c) x[c] = ident ? (c == r ? 1.0 : 0.0) : (c <= r ? S[(c0 + r) * LD + c0 + c] : 0.0);
    unsigned bad = 0;
#pragma unroll
    for (int q = 0; q < 16; q += 4) {
        // the pivot block's rows to every lane
        if (!ident && (r >> 2) == (q >> 2)) {
            double2* p = reinterpret_cast<double2*>(piv + 4 * (r & 3));
            p[0] = make_double2(x[q], x[q + 1]);
            p[1] = make_double2(x[q + 2], x[q + 3]);
        }
        __syncwarp();
        if (q > 0) {  // the previous four columns' update of the columns behind this block
            const double* rows = rows2 + ((q >> 2) & 1 ? 0 : 64);
#pragma unroll
            for (int c = q + 4; c < 16; ++c) {
                const double2 l0 = *reinterpret_cast<const double2*>(rows + 4 * c);
                const double2 l1 = *reinterpret_cast<const double2*>(rows + 4 * c + 2);
                x[c] = fma(-x[q - 3], l0.y, fma(-x[q - 4], l0.x, x[c]));
                x[c] = fma(-x[q - 1], l1.y, fma(-x[q - 2], l1.x, x[c]));
            }
        }
        double l[4][4], rs[4];
#pragma unroll
        for (int i = 0; i < 4; ++i)
#pragma unroll
            for (int c = 0; c <= i; ++c) l[i][c] = piv[4 * i + c];
        const unsigned before = bad;
        factor_pivots4<kPlain>(l, rs, q, bad);
#pragma unroll
        for (int j = 0; j < 4; ++j) {  // this lane's row against the block
#pragma unroll
            for (int c = 0; c < j; ++c) x[q + j] = fma(-x[q + c], l[j][c], x[q + j]);
            x[q + j] *= rs[j];
            // a failed pivot counts as 1
            if (!kPlain && ((bad & ~before) >> (q + j) & 1) && lane == q + j) x[q + j] = 1.0;
        }
        if (q < 12) {  // these columns of the block's rows, and their update of the next four columns
            double* rows = rows2 + ((q >> 2) & 1 ? 64 : 0);
            if (!ident) {
                double2* p = reinterpret_cast<double2*>(rows + 4 * r);
                p[0] = make_double2(x[q], x[q + 1]);
                p[1] = make_double2(x[q + 2], x[q + 3]);
            }
            __syncwarp();
#pragma unroll
            for (int c = q + 4; c < q + 8; ++c) {
                const double2 l0 = *reinterpret_cast<const double2*>(rows + 4 * c);
                const double2 l1 = *reinterpret_cast<const double2*>(rows + 4 * c + 2);
                x[c] = fma(-x[q + 1], l0.y, fma(-x[q], l0.x, x[c]));
                x[c] = fma(-x[q + 3], l1.y, fma(-x[q + 2], l1.x, x[c]));
            }
        }
    }
    return bad;
}

// Warp 0: factors the panel's diagonal block; the transposed inverse to Wt[c][r].  Returns the failed
// pivots as a bit mask.
template <int LD>
__device__ __forceinline__ unsigned factor_panel16(const double* __restrict__ S, double* __restrict__ Wt,
                                                   double* __restrict__ rows2, double* __restrict__ piv, int c0) {
    const int lane = threadIdx.x & 31, r = lane & 15;
    double x[16];
    unsigned bad = factor_rows16<LD, true>(S, x, rows2, piv, c0);
    if (bad) {  // the same for every lane
        __syncwarp();
        bad = factor_rows16<LD, false>(S, x, rows2, piv, c0);
    }
    if (lane >= 16) {
#pragma unroll
        for (int c = 0; c < 16; ++c) Wt[c * kWtLd + r] = x[c];
    }
    return bad;
}

// Factors the block in S (lower triangle given, everything above the diagonal zero) and leaves the
// transposed inverse: L^{-1}[c][r] = S[r][c + 1], c >= r (the lower triangle does not end as L).  A
// pivot that is not > 0 records the 1-based global row k0 + j + 1 in *err (the minimum) and counts as 1.
// work: DiagShape::kWorkDoubles, 16-byte aligned.  All DiagShape::kThreads threads call it after a
// barrier; ends with a barrier.
template <int NB>
__device__ __forceinline__ void factor_diag(double* __restrict__ S, double* __restrict__ work, int64_t k0,
                                            unsigned long long* err) {
    constexpr int LD = DiagShape<NB>::kLd, kWarps = DiagShape<NB>::kThreads / 32;
    double* rows2 = work;
    double* piv = work + 2 * 64;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int g = lane >> 2, t = lane & 3;
    for (int c0 = 0; c0 < NB; c0 += 16) {
        // a panel's update reads its own inverse while warp 0 writes the next panel's
        double* Wt = piv + 16 + (c0 & 16) * kWtLd;
        if (warp == 0) {
            const unsigned bad = factor_panel16<LD>(S, Wt, rows2, piv, c0);
            if (bad && lane == 0) atomicMin(err, (unsigned long long)(k0 + c0 + __ffs(bad)));
        }
        __syncthreads();
        // the other rows of the panel (A rows below, identity rows above): X <- X L_p^{-T}
        {
            constexpr int kRowTiles = (NB - 16) / 8;
            static_assert(kRowTiles <= kWarps, "one row tile per warp");
            if (warp < kRowTiles) {
                const bool below = 8 * warp >= c0;
                const int row = below ? 8 * warp + 16 : 8 * warp;
                double* X = S + (row + g) * LD + c0 + (below ? 0 : 1);
                double acc[2][2] = {};
                double af[4];
#pragma unroll
                for (int kk = 0; kk < 4; ++kk) af[kk] = X[4 * kk + t];
#pragma unroll
                for (int kk = 0; kk < 4; ++kk) {
                    dmma(acc[0], af[kk], Wt[g * kWtLd + 4 * kk + t]);
                    dmma(acc[1], af[kk], Wt[(8 + g) * kWtLd + 4 * kk + t]);
                }
                __syncwarp();
#pragma unroll
                for (int h = 0; h < 2; ++h) {
                    X[8 * h + 2 * t] = acc[h][0];
                    X[8 * h + 2 * t + 1] = acc[h][1];
                }
            } else if (warp == kWarps - 1 && lane < 16) {  // the panel's own identity rows into S
#pragma unroll
                for (int c = 0; c < 16; ++c)
                    if (c >= lane) S[(c0 + lane) * LD + c0 + c + 1] = Wt[c * kWtLd + lane];
            }
        }
        __syncthreads();
        // trailing columns c >= c0 + 16: X -= X_p (row c of L_p)^T over the rows below (their lower
        // triangle) and the identity rows up to this panel, as 16 x 16 tile groups
        const int c1 = c0 + 16;
        const int ng = (NB - c1) / 16;            // column groups left
        const int n_low = ng * (ng + 1) / 2;      // groups of the lower triangle
        const int n_all = n_low + (c1 / 16) * ng;  // and of the identity rows
        // group at (row, col); `shift` 1 for identity rows; X its A operand at [row][k], strides rs, ks
        auto group = [&](int row, int col, int shift, const double* X, int rs, int ks) {
            double acc[2][2][2];
            double af[2][4], bf[2][4];
#pragma unroll
            for (int h = 0; h < 2; ++h)
#pragma unroll
                for (int kk = 0; kk < 4; ++kk) {
                    af[h][kk] = -X[(8 * h + g) * rs + (4 * kk + t) * ks];
                    bf[h][kk] = S[(col + 8 * h + g) * LD + c0 + 4 * kk + t];
                }
            double* C = S + (row + g) * LD + col + 2 * t + shift;
#pragma unroll
            for (int h = 0; h < 2; ++h)
#pragma unroll
                for (int v = 0; v < 2; ++v) {
                    if (row == col && v > h) continue;  // above the diagonal: identity columns live there
                    acc[h][v][0] = C[8 * h * LD + 8 * v];
                    acc[h][v][1] = C[8 * h * LD + 8 * v + 1];
                }
#pragma unroll
            for (int kk = 0; kk < 4; ++kk)
#pragma unroll
                for (int h = 0; h < 2; ++h)
#pragma unroll
                    for (int v = 0; v < 2; ++v) dmma(acc[h][v], af[h][kk], bf[v][kk]);
#pragma unroll
            for (int h = 0; h < 2; ++h)
#pragma unroll
                for (int v = 0; v < 2; ++v) {
                    if (row == col && v > h) continue;
                    C[8 * h * LD + 8 * v] = acc[h][v][0];
                    C[8 * h * LD + 8 * v + 1] = acc[h][v][1];
                }
        };
        if (ng > 0) {
            // warp 0 updates the next panel's diagonal block and goes on to factor it; the others hold
            // back until it has (they have time to spare, and shared memory is what they contend for: a block
            // of 128 in 42,500 cycles without the barrier, 39,700 with it)
            if (warp == 0) {
                group(c1, c1, 0, S + c1 * LD + c0, LD, 1);
                __syncwarp();
                asm volatile("bar.arrive 1, %0;" ::"n"(32 * (1 + kWarps - kWarps / 4)) : "memory");
            } else if (warp & 3) {  // the warps that share warp 0's FP64 pipe stay out of its way
                asm volatile("bar.sync 1, %0;" ::"n"(32 * (1 + kWarps - kWarps / 4)) : "memory");
                for (int x = warp - (warp >> 2); x < n_all; x += kWarps - kWarps / 4) {  // group 0 is warp 0's
                    if (x < n_low) {
                        int gi = 0, base = 0;
                        while (base + gi + 1 <= x) base += ++gi;
                        const int row = c1 + 16 * gi;
                        group(row, c1 + 16 * (x - base), 0, S + row * LD + c0, LD, 1);
                    } else {
                        const int y = x - n_low, row = 16 * (y / ng), col = c1 + 16 * (y % ng);
                        if (row < c0)
                            group(row, col, 1, S + row * LD + c0 + 1, LD, 1);
                        else  // this panel's own identity rows: zeros below their diagonal, from Wt
                            group(row, col, 1, Wt, 1, kWtLd);
                    }
                }
            }
        }
    }
    __syncthreads();
}

}  // namespace panel
}  // namespace gwb200
