// kernels_c64.cu -- screening for eta != 0 (complex FP64).
//
// With broadening eta the reference's Pi0 = 2[1/(w - d + i eta) - 1/(w + d - i eta)]
// (src/gw/sigma.cpp:41-54, w = i omega) is complex and eps_left = I - diag(Pi0) V is no longer
// SPD.  With S = diag(Pi0)^1/2 (any branch: only S*S = diag(Pi0) matters)
//     W_c = (I - diag(Pi0) V)^{-1} diag(Pi0) = S M^{-1} S,   M = I - S V S  (complex symmetric)
//     x^T W_c x = (S x)^T M^{-1} (S x) = sum_j (L^{-1} S x)_j^2,   M = L L^T  (no conjugation)
// so the same tall-matrix right-looking Cholesky runs in complex arithmetic without pivoting
// (M is a small perturbation of the SPD eta = 0 matrix).  A pivot of modulus < 1e-300 or a
// non-finite one is reported like the real path's non-positive pivot.  Every complex tile product
// is four FP64 DMMA tile products on separate real and imaginary planes.  At eta = 0 this path
// gives the real path's numbers (S = i D^1/2); the real path is used there.
#include "panel_common.cuh"
#include "tc_common.cuh"

#include <cmath>

namespace gwb200 {
namespace {

// principal square root of x + i y
__device__ __forceinline__ void csqrt_dev(double x, double y, double& sr, double& si) {
    const double r = hypot(x, y);
    if (r == 0.0) {
        sr = si = 0.0;
        return;
    }
    const double t = sqrt(0.5 * (fabs(x) + r));
    if (x >= 0.0) {
        sr = t;
        si = y / (2.0 * t);
    } else {
        sr = fabs(y) / (2.0 * t);
        si = copysign(t, y);
    }
}

// S_f[c] = sqrt(Pi0(i w_f)[c]) for eta != 0, as two planes (re, im) of n_pad each; zero padding.
__global__ void k_scale_vectors_c(const double* __restrict__ delta, int n, int n_pad, const double* __restrict__ omega,
                                  double eta, double* __restrict__ svec) {
    const int f = blockIdx.y;
    const double w = omega[f];
    double* sr_out = svec + (size_t)f * 2 * n_pad;
    double* si_out = sr_out + n_pad;
    for (int c = blockIdx.x * blockDim.x + threadIdx.x; c < n_pad; c += gridDim.x * blockDim.x) {
        double sr = 0.0, si = 0.0;
        if (c < n) {
            const double d = delta[c];
            // 1/(i w - d + i eta) = 1/(-d + i(w + eta)); 1/(i w + d - i eta) = 1/(d + i(w - eta))
            const double a1r = -d, a1i = w + eta, n1 = a1r * a1r + a1i * a1i;
            const double a2r = d, a2i = w - eta, n2 = a2r * a2r + a2i * a2i;
            const double pr = 2.0 * (a1r / n1 - a2r / n2);
            const double pi = 2.0 * (-a1i / n1 + a2i / n2);
            csqrt_dev(pr, pi, sr, si);
        }
        sr_out[c] = sr;
        si_out[c] = si;
    }
}

// Tall complex matrices: rows r < n_pad hold the lower triangle of M = I - S V S, rows >= n_pad
// hold (S x_j)^T.  Planes: a_re, a_im with the real geometry g.
__global__ void k_build_tall_c(int64_t n, int64_t m, int64_t n_pad, int64_t ld, int64_t stride, int64_t rows,
                               const double* __restrict__ v, const double* __restrict__ xt,
                               const double* __restrict__ svec, int nf, double* __restrict__ a_re,
                               double* __restrict__ a_im) {
    const int64_t c = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (c >= n_pad) return;
    for (int64_t r = blockIdx.y; r < rows; r += gridDim.y) {
        if (r < n_pad) {
            if (c > r) continue;
            const double vrc = (r < n && c < n) ? v[r * n + c] : 0.0;
            const double diag = (r == c) ? 1.0 : 0.0;
            for (int f = 0; f < nf; ++f) {
                const double* sr = svec + (size_t)f * 2 * n_pad;
                const double* si = sr + n_pad;
                // s_r * s_c
                const double pr = sr[r] * sr[c] - si[r] * si[c], pi = sr[r] * si[c] + si[r] * sr[c];
                a_re[(size_t)f * stride + r * ld + c] = diag - pr * vrc;
                a_im[(size_t)f * stride + r * ld + c] = -pi * vrc;
            }
        } else {
            const int64_t j = r - n_pad;
            const double x = (j < m && c < n) ? xt[j * n + c] : 0.0;
            for (int f = 0; f < nf; ++f) {
                const double* sr = svec + (size_t)f * 2 * n_pad;
                a_re[(size_t)f * stride + r * ld + c] = sr[c] * x;
                a_im[(size_t)f * stride + r * ld + c] = sr[n_pad + c] * x;
            }
        }
    }
}

// ---------------------------------------------------------------------------------------------
// Diagonal block, as in panel_common.cuh with complex entries: [A ; I] in 16-wide panels, the
// panel's 16 rows and 16 identity rows in one warp's registers, four columns per exchange; both
// planes of the 64-wide block share L (below) and the identity rows (column c at [r][c + 1]).
// Within a panel the columns stay unscaled (L D L^T): the chain takes 1 / d per pivot, and the
// square roots of the 16 pivots are taken at its end, one per lane.  (A complex pivot step with
// barriers and divisions per column and the inverse by substitution: 165 us per 64 columns.)

constexpr int kLdc = kNb + 4;
constexpr int kPlane = kNb * kLdc;
constexpr int kCWork = 2 * 2 * 16 * panel::kWtLd + 2 * 2 * 64 + 2 * 16 + 2 * 16;  // doubles

struct cd {
    double r, i;
};
__device__ __forceinline__ cd operator*(cd a, cd b) { return {fma(a.r, b.r, -(a.i * b.i)), fma(a.r, b.i, a.i * b.r)}; }
__device__ __forceinline__ void sub_prod(cd& c, cd a, cd b) {  // c -= a b
    c.r = fma(a.i, b.i, fma(-a.r, b.r, c.r));
    c.i = fma(-a.i, b.r, fma(-a.r, b.i, c.i));
}
__device__ __forceinline__ cd ld2(const double* p) {
    const double2 v = *reinterpret_cast<const double2*>(p);
    return {v.x, v.y};
}
__device__ __forceinline__ void st2(double* p, cd v) { *reinterpret_cast<double2*>(p) = make_double2(v.r, v.i); }

// 1 / d.  kPlain: conj(d) / |d|^2 with |d|^2's reciprocal from a third-order iteration; a pivot whose
// larger part is outside 2^-400 .. 2^400 clears the result's validity through `bad` and the caller
// starts over without kPlain: there a pivot of modulus <= 1e-300 or a non-finite one is recorded in
// `bad` and counts as 1, and the division is scaled.
template <bool kPlain>
__device__ __forceinline__ cd pivot_inverse(cd& d, int j, unsigned& bad) {
    if (kPlain) {
        const unsigned h = max((unsigned)__double2hiint(d.r) & 0x7fffffffu, (unsigned)__double2hiint(d.i) & 0x7fffffffu);
        bad |= (unsigned)!(h - ((1023u - 400u) << 20) < (800u << 20));
        const double m = fma(d.r, d.r, d.i * d.i);
        double y;
        asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(m));
        const double e = fma(-m, y, 1.0);
        y = fma(y, fma(e, e, e), y);
        return {d.r * y, -d.i * y};
    }
    const double mod = hypot(d.r, d.i);
    if (!(mod > 1e-300) || !isfinite(mod)) {
        bad |= 1u << j;
        d = {1.0, 0.0};
        return d;
    }
    return {d.r / mod / mod, -(d.i / mod / mod)};
}

template <bool kPlain>
__device__ __forceinline__ unsigned factor_rows16c(const double* __restrict__ Sr, const double* __restrict__ Si,
                                                   cd (&x)[16], double* __restrict__ rows2, double* __restrict__ piv,
                                                   double* __restrict__ scale, int c0) {
    const int lane = threadIdx.x & 31, r = lane & 15;
    const bool ident = lane >= 16;
#pragma unroll
    for (int c = 0; c < 16; ++c) {
        x[c] = {ident && c == r ? 1.0 : 0.0, 0.0};
        if (!ident && c <= r) x[c] = {Sr[(c0 + r) * kLdc + c0 + c], Si[(c0 + r) * kLdc + c0 + c]};
    }
    unsigned bad = 0;
    cd xt[4] = {};      // this lane's row of the last four columns times 1 / d
    cd mine = {1.0, 0.0};  // pivot r
#pragma unroll
    for (int q = 0; q < 16; q += 4) {
        if (!ident && (r >> 2) == (q >> 2))
#pragma unroll
            for (int c = 0; c < 4; ++c) st2(piv + 8 * (r & 3) + 2 * c, x[q + c]);
        __syncwarp();
        if (q > 0) {  // the previous four columns' update of the columns behind this block
            const double* rows = rows2 + ((q >> 2) & 1 ? 0 : 128);
#pragma unroll
            for (int c = q + 4; c < 16; ++c)
#pragma unroll
                for (int j = 0; j < 4; ++j) sub_prod(x[c], xt[j], ld2(rows + 8 * c + 2 * j));
        }
        cd l[4][4], inv[4];
#pragma unroll
        for (int i = 0; i < 4; ++i)
#pragma unroll
            for (int c = 0; c <= i; ++c) l[i][c] = ld2(piv + 8 * i + 2 * c);
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            inv[j] = pivot_inverse<kPlain>(l[j][j], q + j, bad);
            if (r == q + j) mine = l[j][j];
#pragma unroll
            for (int i = j + 1; i < 4; ++i) {
                const cd t = l[i][j] * inv[j];
#pragma unroll
                for (int c = j + 1; c <= i; ++c) sub_prod(l[i][c], t, l[c][j]);
            }
        }
#pragma unroll
        for (int j = 0; j < 4; ++j) {  // this lane's row against the block
#pragma unroll
            for (int c = 0; c < j; ++c) sub_prod(x[q + j], xt[c], l[j][c]);
            if (!ident && r == q + j) x[q + j] = l[j][j];
            xt[j] = x[q + j] * inv[j];
        }
        if (q < 12) {  // these columns of the block's rows, and their update of the next four columns
            double* rows = rows2 + ((q >> 2) & 1 ? 128 : 0);
            if (!ident)
#pragma unroll
                for (int j = 0; j < 4; ++j) st2(rows + 8 * r + 2 * j, x[q + j]);
            __syncwarp();
#pragma unroll
            for (int c = q + 4; c < q + 8; ++c)
#pragma unroll
                for (int j = 0; j < 4; ++j) sub_prod(x[c], xt[j], ld2(rows + 8 * c + 2 * j));
        }
    }
    // columns scaled by 1 / sqrt(d) (either root: only L L^T matters)
    cd s;
    csqrt_dev(mine.r, mine.i, s.r, s.i);
    unsigned none = 0;
    s = pivot_inverse<false>(s, 0, none);
    if (!ident) st2(scale + 2 * r, s);
    __syncwarp();
#pragma unroll
    for (int c = 0; c < 16; ++c) x[c] = x[c] * ld2(scale + 2 * c);
    return bad;
}

// The block in Sr / Si (lower triangle, zeros above) -> transposed inverse, L^{-1}[c][r] at
// [r][c + 1]; as panel::factor_diag.  256 threads, after a barrier; ends with a barrier.
__device__ void factor_diag_c(double* __restrict__ Sr, double* __restrict__ Si, double* __restrict__ work, int64_t k0,
                              unsigned long long* err) {
    constexpr int kWarps = 8;
    constexpr int WL = panel::kWtLd, kW = 16 * WL;
    double* rows2 = work;
    double* piv = rows2 + 2 * 128;
    double* scale = piv + 32;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int g = lane >> 2, t = lane & 3;
    for (int c0 = 0; c0 < kNb; c0 += 16) {
        double* Wr = scale + 32 + (c0 & 16 ? 2 * kW : 0);  // [c][r] of the panel's inverse, two buffers
        double* Wi = Wr + kW;
        if (warp == 0) {
            cd x[16];
            unsigned bad = factor_rows16c<true>(Sr, Si, x, rows2, piv, scale, c0);
            if (bad) {
                __syncwarp();
                bad = factor_rows16c<false>(Sr, Si, x, rows2, piv, scale, c0);
            }
            if (bad && lane == 0) atomicMin(err, (unsigned long long)(k0 + c0 + __ffs(bad)));
            if (lane >= 16)
#pragma unroll
                for (int c = 0; c < 16; ++c) {
                    Wr[c * WL + lane - 16] = x[c].r;
                    Wi[c * WL + lane - 16] = x[c].i;
                }
        }
        __syncthreads();
        // the panel's other rows (A below, identity above): X <- X L_p^{-T}
        constexpr int kRowTiles = (kNb - 16) / 8;
        if (warp < kRowTiles) {
            const bool below = 8 * warp >= c0;
            const int off = ((below ? 8 * warp + 16 : 8 * warp) + g) * kLdc + c0 + (below ? 0 : 1);
            double ar[2][2] = {}, ai[2][2] = {};
            double xr[4], xi[4];
#pragma unroll
            for (int kk = 0; kk < 4; ++kk) {
                xr[kk] = Sr[off + 4 * kk + t];
                xi[kk] = Si[off + 4 * kk + t];
            }
#pragma unroll
            for (int kk = 0; kk < 4; ++kk)
#pragma unroll
                for (int h = 0; h < 2; ++h) {
                    const double br = Wr[(8 * h + g) * WL + 4 * kk + t], bi = Wi[(8 * h + g) * WL + 4 * kk + t];
                    panel::dmma(ar[h], xr[kk], br);
                    panel::dmma(ai[h], xr[kk], bi);
                    panel::dmma(ar[h], -xi[kk], bi);
                    panel::dmma(ai[h], xi[kk], br);
                }
            __syncwarp();
#pragma unroll
            for (int h = 0; h < 2; ++h)
#pragma unroll
                for (int e = 0; e < 2; ++e) {
                    Sr[off + 8 * h + 2 * t + e] = ar[h][e];
                    Si[off + 8 * h + 2 * t + e] = ai[h][e];
                }
        } else if (warp == kWarps - 1 && lane < 16) {  // the panel's own identity rows
#pragma unroll
            for (int c = 0; c < 16; ++c)
                if (c >= lane) {
                    Sr[(c0 + lane) * kLdc + c0 + c + 1] = Wr[c * WL + lane];
                    Si[(c0 + lane) * kLdc + c0 + c + 1] = Wi[c * WL + lane];
                }
        }
        __syncthreads();
        // trailing columns, 16 x 16 tile groups: X -= X_p (row c of L_p)^T
        const int c1 = c0 + 16;
        const int ng = (kNb - c1) / 16, n_low = ng * (ng + 1) / 2, n_all = n_low + (c1 / 16) * ng;
        auto group = [&](int row, int col, int shift, const double* Xr, const double* Xi, int rs, int ks) {
            double br[2][4], bi[2][4];
#pragma unroll
            for (int v = 0; v < 2; ++v)
#pragma unroll
                for (int kk = 0; kk < 4; ++kk) {
                    br[v][kk] = Sr[(col + 8 * v + g) * kLdc + c0 + 4 * kk + t];
                    bi[v][kk] = Si[(col + 8 * v + g) * kLdc + c0 + 4 * kk + t];
                }
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                double ar[2][2], ai[2][2];
                const int off = (row + 8 * h + g) * kLdc + col + 2 * t + shift;
#pragma unroll
                for (int v = 0; v < 2; ++v)
#pragma unroll
                    for (int e = 0; e < 2; ++e) {
                        ar[v][e] = Sr[off + 8 * v + e];
                        ai[v][e] = Si[off + 8 * v + e];
                    }
#pragma unroll
                for (int kk = 0; kk < 4; ++kk) {
                    const int at = (8 * h + g) * rs + (4 * kk + t) * ks;
                    const double xr = Xr[at], xi = Xi[at];
#pragma unroll
                    for (int v = 0; v < 2; ++v) {
                        panel::dmma(ar[v], -xr, br[v][kk]);
                        panel::dmma(ai[v], -xr, bi[v][kk]);
                        panel::dmma(ar[v], xi, bi[v][kk]);
                        panel::dmma(ai[v], -xi, br[v][kk]);
                    }
                }
#pragma unroll
                for (int v = 0; v < 2; ++v) {
                    if (row == col && v > h) continue;  // above the diagonal: identity columns live there
#pragma unroll
                    for (int e = 0; e < 2; ++e) {
                        Sr[off + 8 * v + e] = ar[v][e];
                        Si[off + 8 * v + e] = ai[v][e];
                    }
                }
            }
        };
        auto group_low = [&](int row, int col) {
            group(row, col, 0, Sr + row * kLdc + c0, Si + row * kLdc + c0, kLdc, 1);
        };
        if (ng > 0) {
            if (warp == 0) {  // the next panel's diagonal block, then on to factoring it
                group_low(c1, c1);
                __syncwarp();
            } else if (warp & 3) {  // the warps that share warp 0's FP64 pipe stay out of its way
                for (int x = warp - (warp >> 2); x < n_all; x += kWarps - kWarps / 4) {
                    if (x < n_low) {
                        int gi = 0, base = 0;
                        while (base + gi + 1 <= x) base += ++gi;
                        group_low(c1 + 16 * gi, c1 + 16 * (x - base));
                    } else {
                        const int y = x - n_low, row = 16 * (y / ng), col = c1 + 16 * (y % ng);
                        const int at = row * kLdc + c0 + 1;
                        if (row < c0)
                            group(row, col, 1, Sr + at, Si + at, kLdc, 1);
                        else  // this panel's own identity rows, from the zero-filled copy
                            group(row, col, 1, Wr, Wi, 1, WL);
                    }
                }
            }
        }
    }
    __syncthreads();
}

// 32 or 64 rows of `w` doubles of both planes into shared memory (row stride ldm), one plane `plane` apart
__device__ __forceinline__ void load_rows_c(double* dst, int plane, int ldm, const double* re, const double* im, int64_t ld,
                                            int rows, int w) {
    for (int idx = threadIdx.x; idx < rows * (w / 2); idx += blockDim.x) {
        const int r = idx / (w / 2), c = 2 * (idx % (w / 2));
        panel::cp_async16(dst + r * ldm + c, re + (size_t)r * ld + c);
        panel::cp_async16(dst + plane + r * ldm + c, im + (size_t)r * ld + c);
    }
}

// One CTA per frequency: the diagonal block, first updated by the `depth` (0, 64 or 128) columns before it
// (the trailing update leaves it out, so that it is factored beside that update), replaced by its inverse
// factor.
__global__ void __launch_bounds__(256) k_diag_c(double* __restrict__ a_re, double* __restrict__ a_im, int64_t ld,
                                                int64_t stride, int64_t k, int depth, unsigned long long* err_pivot) {
    extern __shared__ __align__(16) double smem[];
    double* Sr = smem;
    double* Si = Sr + kPlane;
    const size_t base = (size_t)blockIdx.x * stride + k * ld + k;
    if (depth > 0) {
        // 64 columns of the panel's rows at a time through S, the block's lower 16 x 16 tiles in registers
        const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, g = lane >> 2, t = lane & 3;
        constexpr int kLower = 10;  // lower 16 x 16 tiles of the block
        double ar[2][2][2][2] = {}, ai[2][2][2][2] = {};
        int row[2], col[2];
        load_rows_c(Sr, kPlane, kLdc, a_re + base - depth, a_im + base - depth, ld, kNb, kNb);
        asm volatile("cp.async.commit_group;\n" ::);
#pragma unroll
        for (int u = 0; u < 2; ++u) {
            const int x = w + 8 * u;
            int gi = 0, first = 0;
            while (first + gi + 1 <= x) first += ++gi;
            row[u] = 16 * gi;
            col[u] = 16 * (x - first);
            if (x < kLower)
#pragma unroll
            for (int h = 0; h < 2; ++h)
#pragma unroll
                for (int v = 0; v < 2; ++v) {
                    const size_t at = base + (size_t)(row[u] + 8 * h + g) * ld + col[u] + 8 * v + 2 * t;
                    const double2 re = *reinterpret_cast<const double2*>(a_re + at);
                    const double2 im = *reinterpret_cast<const double2*>(a_im + at);
                    ar[u][h][v][0] = re.x;
                    ar[u][h][v][1] = re.y;
                    ai[u][h][v][0] = im.x;
                    ai[u][h][v][1] = im.y;
                }
        }
        for (int from = depth; from > 0; from -= kNb) {
            if (from < depth) {
                load_rows_c(Sr, kPlane, kLdc, a_re + base - from, a_im + base - from, ld, kNb, kNb);
                asm volatile("cp.async.commit_group;\n" ::);
            }
            asm volatile("cp.async.wait_group 0;\n" ::);
            __syncthreads();
#pragma unroll
            for (int u = 0; u < 2; ++u) {
                if (w + 8 * u >= kLower) continue;
                const double* X = Sr + (row[u] + g) * kLdc + t;
                const double* Y = Sr + (col[u] + g) * kLdc + t;
#pragma unroll 2
                for (int kk = 0; kk < kNb; kk += 4) {
                    double xr[2], xi[2];
#pragma unroll
                    for (int h = 0; h < 2; ++h) {
                        xr[h] = -X[8 * h * kLdc + kk];
                        xi[h] = X[kPlane + 8 * h * kLdc + kk];
                    }
#pragma unroll
                    for (int v = 0; v < 2; ++v) {
                        const double br = Y[8 * v * kLdc + kk], bi = Y[kPlane + 8 * v * kLdc + kk];
#pragma unroll
                        for (int h = 0; h < 2; ++h) {
                            panel::dmma(ar[u][h][v], xr[h], br);
                            panel::dmma(ai[u][h][v], xr[h], bi);
                            panel::dmma(ar[u][h][v], xi[h], bi);
                            panel::dmma(ai[u][h][v], -xi[h], br);
                        }
                    }
                }
            }
            __syncthreads();
        }
        // the block into S, zeros above its diagonal
#pragma unroll
        for (int u = 0; u < 2; ++u) {
            if (w + 8 * u < kLower)
#pragma unroll
            for (int h = 0; h < 2; ++h)
#pragma unroll
                for (int v = 0; v < 2; ++v) {
                    const int i = row[u] + 8 * h + g, j = col[u] + 8 * v + 2 * t;
#pragma unroll
                    for (int q = 0; q < 2; ++q) {
                        Sr[i * kLdc + j + q] = j + q <= i ? ar[u][h][v][q] : 0.0;
                        Si[i * kLdc + j + q] = j + q <= i ? ai[u][h][v][q] : 0.0;
                    }
                }
        }
        for (int idx = threadIdx.x; idx < kPlane; idx += 256) {
            const int i = idx / kLdc, j = idx % kLdc;
            if ((j & ~15) > i) Sr[idx] = Si[idx] = 0.0;
        }
    } else {
        for (int idx = threadIdx.x; idx < kPlane; idx += 256) {
            const int i = idx / kLdc, j = idx % kLdc;
            Sr[idx] = j <= i ? a_re[base + (size_t)i * ld + j] : 0.0;
            Si[idx] = j <= i ? a_im[base + (size_t)i * ld + j] : 0.0;
        }
    }
    __syncthreads();
    factor_diag_c(Sr, Si, Si + kPlane, k, err_pivot);
    for (int idx = threadIdx.x; idx < kNb * kNb; idx += 256) {  // the inverse in place of the block
        const int i = idx / kNb, j = idx % kNb;
        a_re[base + (size_t)i * ld + j] = j <= i ? Sr[j * kLdc + i + 1] : 0.0;
        a_im[base + (size_t)i * ld + j] = j <= i ? Si[j * kLdc + i + 1] : 0.0;
    }
}

// Rows below the block, 32-row tiles: P <- P L^{-T} with the triangular inverse (column tile c takes
// k < 8 (c + 1)); right-hand-side rows add sum_j p_j^2 to q.  A CTA keeps the inverse and walks its
// tiles; two CTAs per SM cover each other's loads.  Warp: 16 rows, column tiles {g, 7-g}.
constexpr int kTileC = 32 * kLdc;
constexpr size_t kPanelSmemC = sizeof(double) * (2 * kPlane + 2 * kTileC + 2 * 4 * 32);

__global__ void __launch_bounds__(256, 2) k_panel_c(double* __restrict__ a_re, double* __restrict__ a_im, int64_t ld,
                                                    int64_t stride, int64_t k, int64_t n_pad, int ntile,
                                                    double* __restrict__ qacc, int64_t ldq) {
    extern __shared__ __align__(16) double smem[];
    double* Y = smem;
    double* X = Y + 2 * kPlane;
    double* red = X + 2 * kTileC;
    const size_t f0 = (size_t)blockIdx.y * stride;
    const int64_t row0 = k + kNb;
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const int g = lane >> 2, t = lane & 3;
    const int r0 = 16 * (w & 1), cg = w >> 1;
    load_rows_c(Y, kPlane, kLdc, a_re + f0 + k * ld + k, a_im + f0 + k * ld + k, ld, kNb, kNb);
    for (int tile = blockIdx.x; tile < ntile; tile += gridDim.x) {
        const int64_t row = row0 + (int64_t)tile * 32;
        const size_t at = f0 + row * ld + k;
        load_rows_c(X, kTileC, kLdc, a_re + at, a_im + at, ld, 32, kNb);
        asm volatile("cp.async.commit_group;\n" ::);
        asm volatile("cp.async.wait_group 0;\n" ::);
        __syncthreads();
        double ar[2][2][2] = {}, ai[2][2][2] = {};
        auto steps = [&](int from, int to, int first) {
            for (int ks = from; ks < to; ++ks) {
                const double* xp = X + (r0 + g) * kLdc + 4 * ks + t;
                const double xr0 = xp[0], xr1 = xp[8 * kLdc], xi0 = xp[kTileC], xi1 = xp[kTileC + 8 * kLdc];
#pragma unroll
                for (int i = 0; i < 2; ++i) {
                    if (i < first) continue;
                    const double* yp = Y + (8 * (i ? 7 - cg : cg) + g) * kLdc + 4 * ks + t;
                    const double br = yp[0], bi = yp[kPlane];
                    panel::dmma(ar[0][i], xr0, br);
                    panel::dmma(ar[1][i], xr1, br);
                    panel::dmma(ai[0][i], xr0, bi);
                    panel::dmma(ai[1][i], xr1, bi);
                    panel::dmma(ar[0][i], -xi0, bi);
                    panel::dmma(ar[1][i], -xi1, bi);
                    panel::dmma(ai[0][i], xi0, br);
                    panel::dmma(ai[1][i], xi1, br);
                }
            }
        };
        steps(0, 2 * (cg + 1), 0);
        steps(2 * (cg + 1), 2 * (8 - cg), 1);
#pragma unroll
        for (int h = 0; h < 2; ++h)
#pragma unroll
            for (int i = 0; i < 2; ++i) {
                const size_t p = at + (size_t)(r0 + 8 * h + g) * ld + 8 * (i ? 7 - cg : cg) + 2 * t;
                *reinterpret_cast<double2*>(a_re + p) = make_double2(ar[h][i][0], ar[h][i][1]);
                *reinterpret_cast<double2*>(a_im + p) = make_double2(ai[h][i][0], ai[h][i][1]);
            }
        const bool rhs = row >= n_pad;
        if (rhs) {
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                double sr = 0.0, si = 0.0;
#pragma unroll
                for (int i = 0; i < 2; ++i)
#pragma unroll
                    for (int e = 0; e < 2; ++e) {
                        const double yr = ar[h][i][e], yi = ai[h][i][e];
                        sr += yr * yr - yi * yi;
                        si += 2.0 * yr * yi;
                    }
                for (int o = 1; o < 4; o <<= 1) {
                    sr += __shfl_xor_sync(0xffffffffu, sr, o);
                    si += __shfl_xor_sync(0xffffffffu, si, o);
                }
                if (t == 0) {
                    red[cg * 32 + r0 + 8 * h + g] = sr;
                    red[128 + cg * 32 + r0 + 8 * h + g] = si;
                }
            }
        }
        __syncthreads();
        if (rhs && threadIdx.x < 64) {
            const int r = threadIdx.x & 31, pl = threadIdx.x >> 5;
            const double* p = red + 128 * pl + r;
            qacc[((size_t)blockIdx.y * 2 + pl) * ldq + (row - n_pad) + r] += (p[0] + p[32]) + (p[64] + p[96]);
        }
    }
}

// C -= P_i P_j^T (complex) over K = 64 nk columns from kb0, output column tiles [tc0, tc0 + T): square
// tiles on or below the diagonal, then all right-hand-side rows; the real form's k_update with two
// planes.  64 x 64 tiles, K in 16-wide slices through a two-stage cp.async pipeline, two CTAs per SM
// (one 64-deep load per tile with one CTA per SM left the loads exposed: 18 TFLOP/s).
constexpr int kKcc = 16, kLdkc = kKcc + 4, kSliceC = 64 * kLdkc;
constexpr size_t kUpdateSmemC = sizeof(double) * 2 * 4 * kSliceC;

__global__ void __launch_bounds__(256, 2) k_update_c(double* __restrict__ a_re, double* __restrict__ a_im, int64_t ld,
                                                     int64_t stride, int64_t kb0, int nk, int64_t tc0, int64_t T,
                                                     int64_t nsq) {
    extern __shared__ __align__(16) double smem[];
    const int64_t x = blockIdx.x + 1, L = nsq - tc0;  // tile 0, the next diagonal block, is k_diag_c's
    const int64_t n_square = T * L - T * (T - 1) / 2;
    int64_t c, tr;
    if (x < n_square) {
        const double b = 2.0 * (double)L + 1.0;
        c = (int64_t)((b - sqrt(fmax(b * b - 8.0 * (double)x, 0.0))) * 0.5);
        auto cum = [L](int64_t cc) { return cc * L - cc * (cc - 1) / 2; };
        while (c > 0 && cum(c) > x) --c;
        while (c + 1 < T && cum(c + 1) <= x) ++c;
        tr = tc0 + c + (x - cum(c));
    } else {
        const int64_t y = x - n_square;
        c = y % T;
        tr = nsq + y / T;
    }
    const size_t f0 = (size_t)blockIdx.y * stride;
    const int64_t ri = tr * kNb, cj = (tc0 + c) * kNb;
    const int nsub = nk * (kNb / kKcc);
    auto stage = [&](int st) { return smem + (st & 1) * 4 * kSliceC; };
    auto load = [&](int sc) {
        const int64_t kc = kb0 + (int64_t)sc * kKcc;
        load_rows_c(stage(sc), kSliceC, kLdkc, a_re + f0 + ri * ld + kc, a_im + f0 + ri * ld + kc, ld, 64, kKcc);
        load_rows_c(stage(sc) + 2 * kSliceC, kSliceC, kLdkc, a_re + f0 + cj * ld + kc, a_im + f0 + cj * ld + kc, ld, 64,
                    kKcc);
        asm volatile("cp.async.commit_group;\n" ::);
    };
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const int g = lane >> 2, t = lane & 3;
    const int r0 = 16 * (w >> 1), c0 = 32 * (w & 1);
    double ar[2][4][2] = {}, ai[2][4][2] = {};
    load(0);
    for (int sc = 0; sc < nsub; ++sc) {
        if (sc + 1 < nsub) {
            load(sc + 1);
            asm volatile("cp.async.wait_group 1;\n" ::);
        } else {
            asm volatile("cp.async.wait_group 0;\n" ::);
        }
        __syncthreads();
        const double* A = stage(sc) + (r0 + g) * kLdkc + t;
        const double* B = stage(sc) + 2 * kSliceC + (c0 + g) * kLdkc + t;
#pragma unroll
        for (int kk = 0; kk < kKcc; kk += 4) {
            double xr[2], xi[2];
#pragma unroll
            for (int i = 0; i < 2; ++i) {
                xr[i] = -A[8 * i * kLdkc + kk];
                xi[i] = A[kSliceC + 8 * i * kLdkc + kk];
            }
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                const double br = B[8 * j * kLdkc + kk], bi = B[kSliceC + 8 * j * kLdkc + kk];
#pragma unroll
                for (int i = 0; i < 2; ++i) {
                    panel::dmma(ar[i][j], xr[i], br);
                    panel::dmma(ai[i][j], xr[i], bi);
                    panel::dmma(ar[i][j], xi[i], bi);
                    panel::dmma(ai[i][j], -xi[i], br);
                }
            }
        }
        __syncthreads();
    }
#pragma unroll
    for (int i = 0; i < 2; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const size_t off = f0 + (size_t)(ri + r0 + 8 * i + g) * ld + cj + c0 + 8 * j + 2 * t;
            double2 vr = *reinterpret_cast<double2*>(a_re + off), vi = *reinterpret_cast<double2*>(a_im + off);
            vr.x += ar[i][j][0];
            vr.y += ar[i][j][1];
            vi.x += ai[i][j][0];
            vi.y += ai[i][j][1];
            *reinterpret_cast<double2*>(a_re + off) = vr;
            *reinterpret_cast<double2*>(a_im + off) = vi;
        }
}

// q_out[f] (complex, interleaved) = qacc (planes re, im).
__global__ void k_forms_out_c(const double* __restrict__ qacc, int m, int64_t ldq, double* __restrict__ q,
                              int64_t ldq_out) {
    const int f = blockIdx.y;
    for (int j = blockIdx.x * blockDim.x + threadIdx.x; j < m; j += gridDim.x * blockDim.x) {
        q[(size_t)f * 2 * ldq_out + 2 * j] = qacc[(size_t)f * 2 * ldq + j];
        q[(size_t)f * 2 * ldq_out + 2 * j + 1] = qacc[(size_t)f * 2 * ldq + ldq + j];
    }
}

// Sigma contraction with complex forms (interleaved [f][2*ldq]):
// Sigma_c(p_s, i w_n) = -(1/pi) sum_{f', k} w_{f'} g(k, n, f') q[f', s, k].
__global__ void __launch_bounds__(256) k_sigma_contract_c(const double* __restrict__ qall, int nf_int, int nmo,
                                                          int64_t ldq,
                                                          const double* __restrict__ mo, double fermi,
                                                          const double* __restrict__ omega_int,
                                                          const double* __restrict__ weight_int,
                                                          const double* __restrict__ omega_out, int nf_out,
                                                          double* __restrict__ sigma) {
    const int fn = blockIdx.x, s = blockIdx.y;
    const double wn = omega_out[fn];
    double sr = 0.0, si = 0.0;
    const int total = nf_int * nmo;
    for (int idx = threadIdx.x; idx < total; idx += blockDim.x) {
        const int fp = idx / nmo, k = idx % nmo;
        const size_t qi = (size_t)fp * 2 * ldq + 2 * ((size_t)s * nmo + k);
        const double qr = qall[qi], qim = qall[qi + 1];
        const double ar = fermi - mo[k], ai = wn;
        const double wp = omega_int[fp];
        const double dr = ar * ar - ai * ai + wp * wp, di = 2.0 * ar * ai;
        const double inv = 1.0 / (dr * dr + di * di);
        const double gr = (ar * dr + ai * di) * inv, gi = (ai * dr - ar * di) * inv;
        const double wgt = -weight_int[fp];
        sr += wgt * (gr * qr - gi * qim);
        si += wgt * (gr * qim + gi * qr);
    }
    __shared__ double red[2][256];
    red[0][threadIdx.x] = sr;
    red[1][threadIdx.x] = si;
    __syncthreads();
    for (int off = blockDim.x / 2; off > 0; off >>= 1) {
        if (threadIdx.x < off) {
            red[0][threadIdx.x] += red[0][threadIdx.x + off];
            red[1][threadIdx.x] += red[1][threadIdx.x + off];
        }
        __syncthreads();
    }
    if (threadIdx.x == 0) {
        const double inv_pi = 1.0 / 3.141592653589793238462643383279502884;
        sigma[2 * ((size_t)s * nf_out + fn)] = red[0][0] * inv_pi;
        sigma[2 * ((size_t)s * nf_out + fn) + 1] = red[1][0] * inv_pi;
    }
}

} // namespace

int launch_factor_chunk_c(const TallGeometry& g, int64_t nf, const double* delta, const double* omega, double eta,
                          const double* v, const double* xt, double* a_re, double* a_im, double* svec, double* qacc,
                          unsigned long long* err_pivot, cudaStream_t s, SideStream* side) {
    const size_t smem_diag = sizeof(double) * (2 * kPlane + kCWork);
    GWB_CUDA(cudaFuncSetAttribute(k_diag_c, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem_diag));
    GWB_CUDA(cudaFuncSetAttribute(k_panel_c, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kPanelSmemC));
    GWB_CUDA(cudaFuncSetAttribute(k_update_c, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kUpdateSmemC));
    k_scale_vectors_c<<<dim3((unsigned)((g.n_pad + 255) / 256), (unsigned)nf), 256, 0, s>>>(delta, (int)g.n, (int)g.n_pad,
                                                                                          omega, eta, svec);
    GWB_LAUNCH("k_scale_vectors_c");
    k_build_tall_c<<<dim3((unsigned)((g.n_pad + 255) / 256), (unsigned)std::min<int64_t>(g.rows, 65535)), 256, 0, s>>>(
        g.n, g.m, g.n_pad, g.ld, g.stride, g.rows, v, xt, svec, (int)nf, a_re, a_im);
    GWB_LAUNCH("k_build_tall_c");
    GWB_CUDA(cudaMemsetAsync(qacc, 0, sizeof(double) * 2 * (size_t)nf * g.m_pad, s));
    int launches = 2;
    const int64_t nsq = g.n_pad / kNb, nrt = g.rows / kNb;
    // the next diagonal block beside the trailing update, as in the plain form
    if (nf >= tc::sm_count()) side = nullptr;
    auto diag = [&](int64_t b, int64_t depth) {
        k_diag_c<<<(unsigned)nf, 256, smem_diag, s>>>(a_re, a_im, g.ld, g.stride, b * kNb, (int)depth, err_pivot);
        GWB_LAUNCH("k_diag_c");
    };
    diag(0, 0);
    for (int64_t b = 0; b < nsq; ++b) {  // outer blocks of two 64-wide blocks
        const int64_t tiles = (g.rows - (b + 1) * kNb) / 32;
        k_panel_c<<<dim3((unsigned)panel_grid(tiles, nf, 2), (unsigned)nf), 256, kPanelSmemC, s>>>(
            a_re, a_im, g.ld, g.stride, b * kNb, g.n_pad, (int)tiles, qacc, g.m_pad);
        GWB_LAUNCH("k_panel_c");
        launches += 2;
        if (b + 1 == nsq) break;
        // behind the first block of two the second's columns (K = 64), behind the second all (K = 128)
        const int nk = 1 + (int)(b & 1);
        const int64_t tc0 = b + 1, T = nk == 1 ? 1 : nsq - tc0, L = nsq - tc0;
        SideScope beside(side, s);
        diag(b + 1, nk * kNb);
        k_update_c<<<dim3((unsigned)(T * L - T * (T - 1) / 2 + T * (nrt - nsq) - 1), (unsigned)nf), 256, kUpdateSmemC,
                     beside.stream()>>>(a_re, a_im, g.ld, g.stride, (tc0 - nk) * kNb, nk, tc0, T, nsq);
        GWB_LAUNCH("k_update_c");
        beside.join();
        ++launches;
    }
    return launches;
}

int launch_forms_out_c(const double* qacc, int64_t nf, int64_t m, int64_t ldq, double* q_out, int64_t ldq_out,
                       cudaStream_t s) {
    k_forms_out_c<<<dim3((unsigned)std::min<int64_t>((m + 255) / 256, 64), (unsigned)nf), 256, 0, s>>>(
        qacc, (int)m, ldq, q_out, ldq_out);
    GWB_LAUNCH("k_forms_out_c");
    return 1;
}

int launch_sigma_contract_c(const double* qall, int64_t nf_int, int64_t nstates, int64_t nmo, int64_t ldq,
                            const double* mo, double fermi, const double* omega_int, const double* weight_int,
                            const double* omega_out, int64_t nf_out, double* sigma, cudaStream_t s) {
    k_sigma_contract_c<<<dim3((unsigned)nf_out, (unsigned)nstates), 256, 0, s>>>(
        qall, (int)nf_int, (int)nmo, ldq, mo, fermi, omega_int, weight_int, omega_out, (int)nf_out, sigma);
    GWB_LAUNCH("k_sigma_contract_c");
    return 1;
}

} // namespace gwb200
