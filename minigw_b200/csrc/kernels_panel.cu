// kernels_panel.cu -- the panel step of the plain form's blocked Cholesky (FP64): per outer block
// of 128 columns (64 where only 64 are left) one kernel for the diagonal block and one for the
// rows below it.
//
//   k_diag64    one CTA per frequency: Cholesky of the diagonal block and its inverse
//               (panel_common.cuh); the inverse replaces the block in the tall matrix (the factor
//               itself is not read again: the screened forms need the solved rows alone).  A chain of
//               pivots on one SM, so the next block's runs beside the trailing update on the other
//               SMs: it takes its own update by the panel first, which the trailing update leaves out
//               (31 us without, 41 with 128 columns, 52 with 256, at any number of frequencies up to the
//               SMs).
//   k_panel64   rows below: P = A L^{-T} with the whole block's inverse, so the second 64 columns
//               need no separate update by the first.  The inverse is triangular, so column tile c
//               (8 wide) takes k < 8 (c + 1) only: 0.53 of the square product, less work than two
//               64-wide solves and the update between them (0.75).  Bound by the FP64 tensor pipe.
//               A CTA keeps the inverse in shared memory and walks row tiles of 32, the next tile
//               loaded while one is multiplied; each warp owns 16 rows and column tiles
//               {g, 7-g, 8+g, 15-g}, the same work for every g.
//
//   k_small64   systems of at most 128 particle-hole pairs: everything between the frequencies and
//               the forms in one kernel, see there.
#include "panel_common.cuh"

#include <algorithm>

namespace gwb200 {
namespace {

using namespace panel;

constexpr int kPanelThreads = 256;
constexpr int kRowTile = 32;

// With kUpdate the block first takes the update by the `depth` (128 or 256) columns before it, which the trailing
// update then leaves out: the block depends on the previous panel alone and is factored while the
// rest of the trailing update runs.
template <int NB, bool kUpdate>
__global__ void __launch_bounds__(DiagShape<NB>::kThreads) k_diag64(double* __restrict__ a, int64_t ld, int64_t stride, int64_t k,
                                                          int depth, unsigned long long* err_pivot) {
    extern __shared__ __align__(16) double psm[];
    constexpr int LD = DiagShape<NB>::kLd, kThreads = DiagShape<NB>::kThreads;
    double* S = psm;
    double* A = a + (size_t)blockIdx.x * stride + k * ld + k;
    if (kUpdate) {
        // the panel's rows through the space of S and beyond, the block's lower 16 x 16 tiles in
        // registers, tile x of the warps x mod kWarps
        constexpr int kK = 2 * kNb, kLdP = kK + 4, kWarps = kThreads / 32;
        constexpr int kTiles = (NB / 16) * (NB / 16 + 1) / 2, kPer = (kTiles + kWarps - 1) / kWarps;
        const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, g = lane >> 2, t = lane & 3;
        auto load_rows = [&](int from) {
            for (int idx = threadIdx.x; idx < NB * (kK / 2); idx += kThreads) {
                const int r = idx / (kK / 2), c = 2 * (idx % (kK / 2));
                cp_async16(psm + r * kLdP + c, A + (int64_t)r * ld + c - from);
            }
            asm volatile("cp.async.commit_group;\n" ::);
        };
        load_rows(depth);
        double acc[kPer][2][2][2];
        int row[kPer], col[kPer];
#pragma unroll
        for (int u = 0; u < kPer; ++u) {
            const int x = w + u * kWarps;
            int gi = 0, base = 0;
            while (base + gi + 1 <= x) base += ++gi;
            row[u] = 16 * gi;
            col[u] = 16 * (x - base);
            if (x < kTiles) {
#pragma unroll
                for (int h = 0; h < 2; ++h)
#pragma unroll
                    for (int v = 0; v < 2; ++v) {
                        const double2 e = *reinterpret_cast<const double2*>(A + (size_t)(row[u] + 8 * h + g) * ld +
                                                                             col[u] + 8 * v + 2 * t);
                        acc[u][h][v][0] = e.x;
                        acc[u][h][v][1] = e.y;
                    }
            }
        }
        for (int from = depth; from > 0; from -= kK) {
            if (from < depth) load_rows(from);
            asm volatile("cp.async.wait_group 0;\n" ::);
            __syncthreads();
#pragma unroll
            for (int u = 0; u < kPer; ++u) {
                if (w + u * kWarps >= kTiles) break;
                const double* X = psm + (row[u] + g) * kLdP + t;
                const double* Y = psm + (col[u] + g) * kLdP + t;
#pragma unroll 4
                for (int kk = 0; kk < kK; kk += 4) {
                    const double a0 = -X[kk], a1 = -X[8 * kLdP + kk], b0 = Y[kk], b1 = Y[8 * kLdP + kk];
                    dmma(acc[u][0][0], a0, b0);
                    dmma(acc[u][0][1], a0, b1);
                    dmma(acc[u][1][0], a1, b0);
                    dmma(acc[u][1][1], a1, b1);
                }
            }
            __syncthreads();
        }
        // the block into S, zeros above its diagonal
#pragma unroll
        for (int u = 0; u < kPer; ++u) {
            if (w + u * kWarps >= kTiles) break;
#pragma unroll
            for (int h = 0; h < 2; ++h)
#pragma unroll
                for (int v = 0; v < 2; ++v) {
                    const int i = row[u] + 8 * h + g, j = col[u] + 8 * v + 2 * t;
                    *reinterpret_cast<double2*>(S + i * LD + j) =
                        make_double2(j <= i ? acc[u][h][v][0] : 0.0, j + 1 <= i ? acc[u][h][v][1] : 0.0);
                }
        }
        for (int idx = threadIdx.x; idx < NB * (LD / 2); idx += kThreads) {
            const int i = idx / (LD / 2), j = 2 * (idx % (LD / 2));
            if ((j & ~15) > i) *reinterpret_cast<double2*>(S + i * LD + j) = make_double2(0.0, 0.0);
        }
    } else {
        for (int idx = threadIdx.x; idx < NB * (LD / 2); idx += kThreads) {
            const int i = idx / (LD / 2), j = 2 * (idx % (LD / 2));
            double2 v = make_double2(0.0, 0.0);
            if (j <= i) v = *reinterpret_cast<const double2*>(A + (size_t)i * ld + j);
            if (j + 1 > i) v.y = 0.0;
            *reinterpret_cast<double2*>(S + i * LD + j) = v;
        }
    }
    __syncthreads();
    factor_diag<NB>(S, S + DiagShape<NB>::kBlockDoubles, k, err_pivot);
    // the inverse in place of the block; above the diagonal zeros (not the upper right 64 x 64, which
    // nothing reads).  A warp takes 4 rows x 8 columns: the transposed reads are 2-way bank conflicts.
    const int rr = (threadIdx.x >> 3) & 3, cc = threadIdx.x & 7;
    for (int x = threadIdx.x >> 5; x < (NB / 4) * (NB / 8); x += kThreads / 32) {
        const int i = 4 * (x / (NB / 8)) + rr, j = 8 * (x % (NB / 8)) + cc;
        if (j < (i < kNb ? kNb : NB)) A[(size_t)i * ld + j] = j <= i ? S[j * LD + i + 1] : 0.0;
    }
}

// shared memory of k_diag64: the block and the workspace, or the panel's rows
template <int NB, bool kUpdate>
constexpr size_t diag_smem() {
    const size_t rows = sizeof(double) * (size_t)NB * (2 * kNb + 4);
    return kUpdate && rows > DiagShape<NB>::kSmem ? rows : DiagShape<NB>::kSmem;
}

template <int NB>
struct PanelShape {
    static constexpr int kLd = NB + 4;  // = 4 mod 16 (fragment loads on distinct banks)
    static constexpr int kTiles = NB / 32;  // column tiles of 8 per warp
    static constexpr size_t kSmem = sizeof(double) * ((size_t)NB * kLd + 2 * kRowTile * kLd + 8 * kRowTile);
};

template <int NB>
__global__ void __launch_bounds__(kPanelThreads, 1)
    k_panel64(double* __restrict__ a, int64_t ld, int64_t stride, int64_t k, int64_t n_pad, int ntile,
              double* __restrict__ qacc, int64_t ldq) {
    extern __shared__ __align__(16) double psm[];
    using Sh = PanelShape<NB>;
    constexpr int LD = Sh::kLd, NT = Sh::kTiles;
    double* Y = psm;
    double* Xs = Y + NB * LD;
    double* red = Xs + 2 * kRowTile * LD;
    double* A = a + (size_t)blockIdx.y * stride;
    const int64_t row0 = k + NB;
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const int g = lane >> 2, t = lane & 3;
    const int r0 = 16 * (w & 1), cg = w >> 1;
    auto load_rows = [&](int tile, int buf) {
        const double* src = A + (size_t)(row0 + (int64_t)tile * kRowTile) * ld + k;
        double* dst = Xs + buf * kRowTile * LD;
        for (int idx = threadIdx.x; idx < kRowTile * (NB / 2); idx += kPanelThreads) {
            const int r = idx / (NB / 2), c = 2 * (idx % (NB / 2));
            cp_async16(dst + r * LD + c, src + (size_t)r * ld + c);
        }
        asm volatile("cp.async.commit_group;\n" ::);
    };
    for (int idx = threadIdx.x; idx < NB * (NB / 2); idx += kPanelThreads) {
        const int r = idx / (NB / 2), c = 2 * (idx % (NB / 2));
        if (c < (r < kNb ? kNb : NB)) cp_async16(Y + r * LD + c, A + (size_t)(k + r) * ld + k + c);
    }
    load_rows(blockIdx.x, 0);
    // squared norms of a right-hand-side tile, from the warps' sums in red[its buffer], after a barrier
    auto add_norms = [&](int tile, int b) {
        const int64_t r = row0 + (int64_t)tile * kRowTile - n_pad + threadIdx.x;
        const double* v = red + b * 4 * kRowTile + threadIdx.x;
        if (r >= (int64_t)threadIdx.x && threadIdx.x < kRowTile)  // n_pad is a multiple of the tile
            qacc[(size_t)blockIdx.y * ldq + r] += (v[0] + v[kRowTile]) + (v[2 * kRowTile] + v[3 * kRowTile]);
    };
    // one barrier per tile: a warp stores its rows while others still multiply (4480 rows x 128 frequencies
    // 468 us with a second barrier, 458 without; multiplying alone takes 357)
    int buf = 0, tile = blockIdx.x;
    for (; tile < ntile; tile += gridDim.x, buf ^= 1) {
        asm volatile("cp.async.wait_group 0;\n" ::);
        __syncthreads();
        if (tile != (int)blockIdx.x) add_norms(tile - gridDim.x, buf ^ 1);
        if (tile + (int)gridDim.x < ntile) load_rows(tile + gridDim.x, buf ^ 1);
        const double* X = Xs + buf * kRowTile * LD + (r0 + g) * LD + t;
        // column tiles of this warp, ascending: cg, 7 - cg(, 8 + cg, 15 - cg)
        auto col = [&](int i) { return (i >> 1) * 8 + ((i & 1) ? 7 - cg : cg); };
        double acc[2][NT][2] = {};
        int ks = 0;
#pragma unroll
        for (int first = 0; first < NT; ++first) {  // tiles `first`.. still have columns k <= c
            const int kend = 2 * (col(first) + 1);
            for (; ks < kend; ++ks) {
                const double a0 = X[4 * ks], a1 = X[8 * LD + 4 * ks];
#pragma unroll
                for (int i = first; i < NT; ++i) {
                    const double b = Y[(8 * col(i) + g) * LD + 4 * ks + t];
                    dmma(acc[0][i], a0, b);
                    dmma(acc[1][i], a1, b);
                }
            }
        }
        const int64_t row = row0 + (int64_t)tile * kRowTile + r0 + g;
#pragma unroll
        for (int h = 0; h < 2; ++h)
#pragma unroll
            for (int i = 0; i < NT; ++i)
                *reinterpret_cast<double2*>(A + (size_t)(row + 8 * h) * ld + k + 8 * col(i) + 2 * t) =
                    make_double2(acc[h][i][0], acc[h][i][1]);
        if (row0 + (int64_t)tile * kRowTile >= n_pad) {  // squared row norms, summed in a fixed order
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                double s = 0.0;
#pragma unroll
                for (int i = 0; i < NT; ++i) s = fma(acc[h][i][1], acc[h][i][1], fma(acc[h][i][0], acc[h][i][0], s));
                s += __shfl_xor_sync(0xffffffffu, s, 1);
                s += __shfl_xor_sync(0xffffffffu, s, 2);
                if (t == 0) red[(buf * 4 + cg) * kRowTile + r0 + 8 * h + g] = s;
            }
        }
    }
    __syncthreads();
    add_norms(tile - gridDim.x, buf ^ 1);
}

// Whole frequencies of a small system (n <= NB <= 128), a CTA or more each: the scale vector, eps, its factor
// and inverse in shared memory, then the right-hand sides in 32-row tiles, of which only the forms
// leave the SM.  The arithmetic and its order are those of k_scale_vectors, k_build_tall, k_diag64,
// k_panel64 and k_negate_copy, whose five launches and tall matrices it replaces: at this size they
// spent their time in launches and the matrices' way through memory (24 orbitals, 200 frequencies:
// 113 us of kernels; this one 39).  NB is the next of 64, 96 and 128, so that up to n = 96 two CTAs
// share an SM.  The row tiles are dealt out over the grid's y; each of a frequency's CTAs factors its
// block again, on SMs that would be idle (116 pairs, 3600 rows: one CTA per frequency took 472 to 479 us
// at 1 to 64 frequencies, where the panel kernels take 57 to 312 and these 39 to 260).
template <int NB>
struct SmallShape {
    static constexpr int kXLd = NB + 4;
    static constexpr size_t kSmem = DiagShape<NB>::kSmem + sizeof(double) * ((size_t)kRowTile * kXLd + NB + 4 * kRowTile);
};

template <int NB>
__global__ void __launch_bounds__(DiagShape<NB>::kThreads) k_small64(int n, int m, const double* __restrict__ delta,
                                                                     const double* __restrict__ omega,
                                                                     const double* __restrict__ v,
                                                                     const double* __restrict__ xt, double* __restrict__ q,
                                                                     int64_t ldq, unsigned long long* err_pivot) {
    extern __shared__ __align__(16) double psm[];
    using Sh = DiagShape<NB>;
    constexpr int LD = Sh::kLd, XL = SmallShape<NB>::kXLd, NT = NB / 32;
    double* S = psm;
    double* work = S + Sh::kBlockDoubles;
    double* X = work + Sh::kWorkDoubles;
    double* d = X + kRowTile * XL;
    double* red = d + NB;
    const int f = blockIdx.x;
    const double w = omega[f];
    for (int c = threadIdx.x; c < NB; c += Sh::kThreads) d[c] = c < n ? scale_value(delta[c], w) : 0.0;
    __syncthreads();
    for (int idx = threadIdx.x; idx < NB * LD; idx += Sh::kThreads) {
        const int i = idx / LD, j = idx % LD;
        double x = 0.0;
        if (j <= i) x = fma(d[i] * (i < n ? v[(size_t)i * n + j] : 0.0), d[j], i == j ? 1.0 : 0.0);
        S[idx] = x;
    }
    __syncthreads();
    factor_diag<NB>(S, work, 0, err_pivot);
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int g = lane >> 2, t = lane & 3;
    const int r0 = 16 * (warp & 1), cg = warp >> 1;
    auto col = [&](int i) { return (i >> 1) * 8 + ((i & 1) ? 7 - cg : cg); };  // as in k_panel64
    for (int row = kRowTile * blockIdx.y; row < m; row += kRowTile * gridDim.y) {
        for (int idx = threadIdx.x; idx < kRowTile * NB; idx += Sh::kThreads) {
            const int r = idx / NB, c = idx % NB;
            X[r * XL + c] = (row + r < m && c < n) ? d[c] * xt[(size_t)(row + r) * n + c] : 0.0;
        }
        __syncthreads();
        if (warp < 8) {
            const double* Xp = X + (r0 + g) * XL + t;
            double acc[2][NT][2] = {};
            int ks = 0;
#pragma unroll
            for (int first = 0; first < NT; ++first) {
                const int kend = 2 * (col(first) + 1);
                for (; ks < kend; ++ks) {
                    const double a0 = Xp[4 * ks], a1 = Xp[8 * XL + 4 * ks];
                    const int k = 4 * ks + t;
#pragma unroll
                    for (int i = first; i < NT; ++i) {
                        const int c = 8 * col(i) + g;
                        const double b = k <= c ? S[k * LD + c + 1] : 0.0;
                        dmma(acc[0][i], a0, b);
                        dmma(acc[1][i], a1, b);
                    }
                }
            }
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                double s = 0.0;
#pragma unroll
                for (int i = 0; i < NT; ++i) s = fma(acc[h][i][1], acc[h][i][1], fma(acc[h][i][0], acc[h][i][0], s));
                s += __shfl_xor_sync(0xffffffffu, s, 1);
                s += __shfl_xor_sync(0xffffffffu, s, 2);
                if (t == 0) red[cg * kRowTile + r0 + 8 * h + g] = s;
            }
        }
        __syncthreads();
        if (threadIdx.x < kRowTile && row + (int)threadIdx.x < m) {
            const int r = threadIdx.x;
            q[(size_t)f * ldq + row + r] =
                -((red[r] + red[kRowTile + r]) + (red[2 * kRowTile + r] + red[3 * kRowTile + r]));
        }
    }
}

template <int NB>
int launch_small(const TallGeometry& g, int64_t nf, const double* delta, const double* omega, const double* v,
                 const double* xt, double* q, int64_t ldq, unsigned long long* err_pivot, cudaStream_t s) {
    const size_t smem = SmallShape<NB>::kSmem;
    GWB_CUDA(cudaFuncSetAttribute(k_small64<NB>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    // the factorisation costs as much as 8 row tiles at every NB; at NB = 64 two CTAs on an SM are as
    // fast as one (35 pairs, 288 rows, 148 frequencies: 33 us as 148 CTAs, 31 as 296), from 96 on they
    // take turns (80 pairs, 336 rows: 53 and 70)
    const int64_t gy = panel_grid((g.m + kRowTile - 1) / kRowTile, nf, NB == 64 ? 2 : 1, 8.0);
    k_small64<NB><<<dim3((unsigned)nf, (unsigned)gy), DiagShape<NB>::kThreads, smem, s>>>(
        (int)g.n, (int)g.m, delta, omega, v, xt, q, ldq, err_pivot);
    GWB_LAUNCH("k_small64");
    return 1;
}

template <int NB, bool kUpdate>
void launch_diag(const TallGeometry& g, int64_t nf, double* a, int64_t k, int64_t depth, unsigned long long* err_pivot,
                 cudaStream_t s) {
    constexpr size_t smem = diag_smem<NB, kUpdate>();
    GWB_CUDA(cudaFuncSetAttribute(k_diag64<NB, kUpdate>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    k_diag64<NB, kUpdate><<<(unsigned)nf, DiagShape<NB>::kThreads, smem, s>>>(a, g.ld, g.stride, k, (int)depth,
                                                                                 err_pivot);
    GWB_LAUNCH("k_diag64");
}

template <int NB>
int launch_rows(const TallGeometry& g, int64_t nf, double* a, int64_t k, double* qacc, cudaStream_t s) {
    const int64_t tiles = (g.rows - (k + NB)) / kRowTile;
    if (tiles <= 0) return 0;
    GWB_CUDA(cudaFuncSetAttribute(k_panel64<NB>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)PanelShape<NB>::kSmem));
    k_panel64<NB><<<dim3((unsigned)panel_grid(tiles, nf, 1), (unsigned)nf), kPanelThreads, PanelShape<NB>::kSmem, s>>>(
        a, g.ld, g.stride, k, g.n_pad, (int)tiles, qacc, g.m_pad);
    GWB_LAUNCH("k_panel64");
    return 1;
}

}  // namespace

// The fewest tile times over the waves.
int64_t panel_grid(int64_t tiles, int64_t nf, int64_t per_sm, double head) {
    const int64_t slots = 148 * per_sm;
    int64_t best = 1;
    double best_cost = 0.0;
    for (int64_t gx = 1; gx <= std::min<int64_t>(tiles, 64); ++gx) {
        const double waves = (double)((nf * gx + slots - 1) / slots);
        const double cost = waves * ((double)((tiles + gx - 1) / gx) + head);
        if (gx == 1 || cost < best_cost) {
            best = gx;
            best_cost = cost;
        }
    }
    return best;
}

bool small_system(const TallGeometry& g) { return g.n <= 128; }

int launch_small64(const TallGeometry& g, int64_t nf, const double* delta, const double* omega, const double* v,
                   const double* xt, double* q, int64_t ldq, unsigned long long* err_pivot, cudaStream_t s) {
    if (g.n <= 64) return launch_small<64>(g, nf, delta, omega, v, xt, q, ldq, err_pivot, s);
    if (g.n <= 96) return launch_small<96>(g, nf, delta, omega, v, xt, q, ldq, err_pivot, s);
    return launch_small<128>(g, nf, delta, omega, v, xt, q, ldq, err_pivot, s);
}

int launch_diag64(const TallGeometry& g, int64_t nf, double* a, int64_t k, int64_t width, int64_t depth,
                  unsigned long long* err_pivot, cudaStream_t s) {
    auto run = width == 2 * kNb ? (depth > 0 ? launch_diag<128, true> : launch_diag<128, false>)
                                : (depth > 0 ? launch_diag<64, true> : launch_diag<64, false>);
    run(g, nf, a, k, depth, err_pivot, s);
    return 1;
}

int launch_panel64(const TallGeometry& g, int64_t nf, double* a, int64_t k, int64_t width, double* qacc,
                   cudaStream_t s) {
    return width == 2 * kNb ? launch_rows<128>(g, nf, a, k, qacc, s) : launch_rows<64>(g, nf, a, k, qacc, s);
}

}  // namespace gwb200
