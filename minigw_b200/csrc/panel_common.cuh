// panel_common.cuh -- the diagonal-block step of the blocked Cholesky: one CTA factors a 64- or
// 128-wide diagonal block in shared memory and forms its inverse factor on the way.
//
// What bounds it: a chain of NB dependent pivots.  Factoring the tall block [A ; I] instead of A
// makes the identity rows come out as I L^{-T}, the transposed inverse, with no chain of their own
// (the separate forward substitution was as long as the factorisation).  The columns are taken in
// panels of 16.  One warp holds a panel's 16 rows of A (lanes 0-15) and 16 identity rows (lanes
// 16-31) in registers: a pivot costs one reciprocal square root and two dependent multiply-adds,
// because the operands of the next pivot are broadcast before the current column is scaled.  The
// remaining rows follow as FP64 tensor-core (m8n8k4) products over all warps, the next panel's
// diagonal block first, so that the other tiles are updated while warp 0 factors it.
#pragma once

#include "internal.cuh"

namespace gwb200 {
namespace panel {

constexpr int kPanelThreads = 256;
constexpr int kWtLd = 20;  // row stride of the 16 x 16 inverse of a panel's diagonal block

template <int NB>
struct DiagShape {
    // Row stride (doubles) of the block: column j of L at [i][j] (j <= i), the identity row r's
    // column c at [r][c + 1] (c >= r), so the two triangles share one array.  = 4 mod 16: the 8
    // rows x 4 columns of one m8n8k4 fragment fall on distinct banks.
    static constexpr int kLd = NB + 4;
    static constexpr int kBlockDoubles = NB * kLd;
    static constexpr size_t kSmem = sizeof(double) * (size_t)(kBlockDoubles + 2 * 16 * kWtLd);
};

__device__ __forceinline__ void dmma(double (&c)[2], double a, double b) {
    asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0,%1}, {%2}, {%3}, {%0,%1};\n"
                 : "+d"(c[0]), "+d"(c[1])
                 : "d"(a), "d"(b));
}

// 1 / sqrt(d) from the hardware's ~2^-20 approximation y by one step of Householder's third-order
// iteration: e = 1 - d y^2, y (1 + e / 2 + 3 e^2 / 8), error ~e^3.  d is clamped to the finite
// normal range first (subnormal and infinite pivots stay finite).
__device__ __forceinline__ double rsqrt_pivot(double d) {
    const int hi = min(max(__double2hiint(d), 0x00100000), 0x7fefffff);
    const double x = __hiloint2double(hi, __double2loint(d));
    double y;
    asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(x));
    const double e = fma(-x, y * y, 1.0);
    return fma(fma(0.375, e, 0.5), y * e, y);
}

// Factors the block in S (lower triangle given, everything above the diagonal zero) and leaves the
// transposed inverse: L^{-1}[c][r] = S[r][c + 1], c >= r.  With kKeepL the lower triangle of S is
// L.  A pivot that is not > 0 records the 1-based global row k0 + j + 1 in *err (the minimum) and
// counts as 1.  All kPanelThreads threads call it after a barrier; ends with a barrier.
template <int NB, bool kKeepL>
__device__ __forceinline__ void factor_diag(double* __restrict__ S, double* __restrict__ Wt2, int64_t k0,
                                            unsigned long long* err) {
    constexpr int LD = DiagShape<NB>::kLd;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int g = lane >> 2, t = lane & 3;
    for (int c0 = 0; c0 < NB; c0 += 16) {
        double* Wt = Wt2 + (c0 & 16) * kWtLd;
        if (warp == 0) {
            const int r = lane & 15;
            const bool ident = lane >= 16;
            double x[16];
#pragma unroll
            for (int c = 0; c < 16; ++c)
                x[c] = ident ? (c == r ? 1.0 : 0.0) : (c <= r ? S[(c0 + r) * LD + c0 + c] : 0.0);
            unsigned bad = 0;
            double d = __shfl_sync(0xffffffffu, x[0], 0);
#pragma unroll
            for (int j = 0; j < 16; ++j) {
                const bool fails = !(d > 0.0);
                bad |= (unsigned)fails << j;
                double rs = rsqrt_pivot(d);
                rs = fails ? 1.0 : rs;
                if (j < 15) {
                    // row j+1's entries of this column and the next, before this column is scaled:
                    // the next pivot is their update, the same arithmetic as lane j+1's own
                    const double a = __shfl_sync(0xffffffffu, x[j + 1], j + 1);
                    const double b = __shfl_sync(0xffffffffu, x[j], j + 1) * rs;
                    d = fma(-b, b, a);
                }
                x[j] = (fails && lane == j) ? 1.0 : x[j] * rs;
#pragma unroll
                for (int c = j + 1; c < 16; ++c)
                    x[c] = fma(-x[j], __shfl_sync(0xffffffffu, x[j], c), x[c]);
            }
            if (bad && lane == 0) atomicMin(err, (unsigned long long)(k0 + c0 + __ffs(bad)));
            if (ident) {
#pragma unroll
                for (int c = 0; c < 16; ++c) {
                    Wt[c * kWtLd + r] = x[c];
                    if (c >= r) S[(c0 + r) * LD + c0 + c + 1] = x[c];
                }
            } else if (kKeepL) {
#pragma unroll
                for (int c = 0; c < 16; ++c)
                    if (c <= r) S[(c0 + r) * LD + c0 + c] = x[c];
            }
        }
        __syncthreads();
        // the other rows of the panel (A rows below, identity rows above): X <- X L_p^{-T}
        for (int ti = warp; ti < (NB - 16) / 8; ti += 8) {
            const bool below = 8 * ti >= c0;
            const int row = below ? 8 * ti + 16 : 8 * ti;
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
        }
        __syncthreads();
        // trailing columns c >= c0 + 16: X -= X_p (row c of L_p)^T over the rows below (their lower
        // triangle) and the identity rows up to this panel
        const int c1 = c0 + 16;
        const int nt = (NB - c1) / 8;             // column tiles left
        const int n_low = nt * (nt + 1) / 2;      // tiles of the lower triangle
        const int n_all = n_low + (c1 / 8) * nt;  // and of the identity rows
        // A operand of a tile: X at [row][k], `rs` and `ks` the strides of row and column
        auto tile = [&](int row, int col, int shift, const double* X, int rs, int ks) {
            double* C = S + (row + g) * LD + col + 2 * t + shift;
            double acc[2] = {C[0], C[1]};
#pragma unroll
            for (int kk = 0; kk < 4; ++kk) dmma(acc, -X[g * rs + (4 * kk + t) * ks], S[(col + g) * LD + c0 + 4 * kk + t]);
            C[0] = acc[0];
            C[1] = acc[1];
        };
        auto tile_low = [&](int row, int col) { tile(row, col, 0, S + row * LD + c0, LD, 1); };
        if (nt > 0) {
            if (warp == 0) {  // the next panel's diagonal block, then on to factoring it
                tile_low(c1, c1);
                tile_low(c1 + 8, c1);
                tile_low(c1 + 8, c1 + 8);
                __syncwarp();
            } else {
                for (int x = 2 + warp; x < n_all; x += 7) {
                    if (x < n_low) {  // tiles 0-2 are warp 0's
                        int ti = (int)((sqrtf(8.0f * (float)x + 1.0f) - 1.0f) * 0.5f);
                        if (ti * (ti + 1) / 2 > x) --ti;
                        if ((ti + 1) * (ti + 2) / 2 <= x) ++ti;
                        tile_low(c1 + 8 * ti, c1 + 8 * (x - ti * (ti + 1) / 2));
                    } else {
                        const int y = x - n_low, row = 8 * (y / nt), col = c1 + 8 * (y % nt);
                        if (row < c0)
                            tile(row, col, 1, S + row * LD + c0 + 1, LD, 1);
                        else  // this panel's own identity rows: zeros below their diagonal, from Wt
                            tile(row, col, 1, Wt + (row - c0), 1, kWtLd);
                    }
                }
            }
        }
    }
    __syncthreads();
}

}  // namespace panel
}  // namespace gwb200
