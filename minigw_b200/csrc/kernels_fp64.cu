// kernels_fp64.cu -- plain-form (FP64) screening kernels for sm_100a.
//
// Per frequency f the reference builds eps_left = I - diag(Pi0) V and forms
// W_c = eps_left^{-1} diag(Pi0) with a complex LU (src/workspace/screening_workspace.cpp:21-66,
// src/workspace/device_screening_workspace.cu:337-374), then evaluates x^T W_c x per panel
// (src/workspace/screening_workspace.cpp:69-102).  At eta = 0, Pi0 = -D with
// D = 4 delta / (w^2 + delta^2) > 0, and
//     x^T W_c x = -|| L^{-1} D^1/2 x ||^2,   L L^T = eps = I + D^1/2 V D^1/2  (SPD, eigenvalues >= 1).
// The kernels below factor the tall matrix [eps ; (D^1/2 X)^T] with one right-looking
// blocked Cholesky: its lower rows become (L^{-1} D^1/2 X)^T, whose row norms are the
// quadratic forms.  All arithmetic is FP64; the O(n^3) and O(n^2 m) work runs on FP64
// tensor cores (mma.sync m8n8k4 f64, DMMA).
#include "panel_common.cuh"
#include "tc_common.cuh"

#include <array>
#include <cstdio>
#include <cstring>
#include <map>
#include <mutex>

#include <cmath>
#include <cstdlib>

namespace gwb200 {
namespace {

// ---------------------------------------------------------------------------
// Gathers (bit-exact copies).

// The device keeps only the (pq|o.) block of the ERI: pqo[(p*nmo + q)*nocc + i][s] = eri[p,q,i,s]
// for i < nocc (every element the path reads except the exchange diagonal), uploaded by one 2D
// copy whose rows are nocc*nmo contiguous doubles.

// V[jb, ia] = eri[j, b, i, a]  (src/gw/sigma.cpp:56-71), row-major n x n.
// blockIdx.y strides over rows jb; threads over ia: for fixed (jb, i) the source run
// pqo[(j,b,i)][nocc:nmo] is contiguous, so loads coalesce in runs of nvir.
__global__ void k_gather_vph(const double* __restrict__ pqo, int nmo, int nocc, int n, double* __restrict__ v) {
    const int nvir = nmo - nocc;
    for (int jb = blockIdx.y; jb < n; jb += gridDim.y) {
        const int j = jb / nvir, b = nocc + jb % nvir;
        const size_t base = ((size_t)j * nmo + b) * (size_t)nocc * nmo;
        for (int ia = blockIdx.x * blockDim.x + threadIdx.x; ia < n; ia += gridDim.x * blockDim.x) {
            const int i = ia / nvir, a = nocc + ia % nvir;
            v[(size_t)jb * n + ia] = pqo[base + (size_t)i * nmo + a];
        }
    }
}

// Xt[s*nmo + k, ia] = eri[p_s, k, i, a]  (src/workspace/pq_ph_panel.cpp:25-47, transposed so
// that every right-hand side is a contiguous row), row-major m x n.
__global__ void k_gather_panel(const double* __restrict__ pqo, int nmo, int nocc, int n,
                               const int64_t* __restrict__ states, int m, double* __restrict__ xt) {
    const int nvir = nmo - nocc;
    for (int row = blockIdx.y; row < m; row += gridDim.y) {
        const int s = row / nmo, k = row % nmo;
        const size_t p = (size_t)states[s];
        const size_t base = (p * nmo + k) * (size_t)nocc * nmo;
        for (int ia = blockIdx.x * blockDim.x + threadIdx.x; ia < n; ia += gridDim.x * blockDim.x) {
            const int i = ia / nvir, a = nocc + ia % nvir;
            xt[(size_t)row * n + ia] = pqo[base + (size_t)i * nmo + a];
        }
    }
}

// Sigma_x[p,p] = -sum_{i<nocc} eri[p,i,p,i] in the reference's order (src/gw/sigma.cpp:29-36);
// xdiag[p*nocc + i] = eri[p,i,p,i] (gathered on the host).
__global__ void k_sigma_x_diag(const double* __restrict__ xdiag, int nmo, int nocc, double* __restrict__ out) {
    const int p = blockIdx.x * blockDim.x + threadIdx.x;
    if (p >= nmo) return;
    double value = 0.0;
    for (int i = 0; i < nocc; ++i) value = __dsub_rn(value, xdiag[(size_t)p * nocc + i]);
    out[p] = value;
}

// delta[ph] = e_a - e_i with ph = i*nvir + a_vir (include/gw/particle_hole.hpp:22-35).
__global__ void k_delta(const double* __restrict__ mo, int nmo, int nocc, double* __restrict__ delta) {
    const int nvir = nmo - nocc, n = nocc * nvir;
    const int ph = blockIdx.x * blockDim.x + threadIdx.x;
    if (ph >= n) return;
    const int i = ph / nvir, a = nocc + ph % nvir;
    delta[ph] = __dsub_rn(mo[a], mo[i]);
}

// dvec[f, c] = sqrt(D_f[c]) with D = -Pi0(i w_f) = 4 delta / (w^2 + delta^2); zero padding.
__global__ void k_scale_vectors(const double* __restrict__ delta, int n, int n_pad, const double* __restrict__ omega,
                                int nf, double* __restrict__ dvec) {
    const int f = blockIdx.y;
    const double w = omega[f];
    for (int c = blockIdx.x * blockDim.x + threadIdx.x; c < n_pad; c += gridDim.x * blockDim.x) {
        double val = 0.0;
        if (c < n) val = panel::scale_value(delta[c], w);
        dvec[(size_t)f * n_pad + c] = val;
    }
}

// Build the tall matrices of nf frequencies.  Thread (r, c): rows r < n_pad hold the lower
// triangle of eps (c <= r), rows r >= n_pad hold d_c * Xt[r - n_pad, c].  V and Xt are read
// once per chunk; the loop over frequencies reuses the value from registers.
__global__ void k_build_tall(int64_t n, int64_t m, int64_t n_pad, int64_t ld, int64_t stride,
                             const double* __restrict__ v, const double* __restrict__ xt,
                             const double* __restrict__ dvec, int nf, double* __restrict__ a) {
    const int64_t c = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (c >= n_pad) return;
    const int64_t rows = n_pad + ((m + kNb - 1) / kNb) * kNb;
    for (int64_t r = blockIdx.y; r < rows; r += gridDim.y) {
    if (r < n_pad) {
        if (c > r) continue;
        const bool inside = (r < n) && (c < n);
        const double vrc = inside ? v[r * n + c] : 0.0;
        const double diag = (r == c) ? 1.0 : 0.0;
        for (int f = 0; f < nf; ++f) {
            const double* d = dvec + (size_t)f * n_pad;
            a[(size_t)f * stride + r * ld + c] = fma(d[r] * vrc, d[c], diag);
        }
    } else {
        const int64_t j = r - n_pad;
        const double x = (j < m && c < n) ? xt[j * n + c] : 0.0;
        for (int f = 0; f < nf; ++f) {
            a[(size_t)f * stride + r * ld + c] = dvec[(size_t)f * n_pad + c] * x;
        }
    }
    }
}

// ---------------------------------------------------------------------------
// Trailing update C -= sum_chunks P_i P_j^T of the output column tiles [tc0, tc0+T) (64-wide,
// absolute tile indices): every tile on or below the diagonal in the square block but the first
// `skip` row tiles, then every tile of the right-hand-side rows.  The contraction runs over nk
// 64-wide column chunks of the factored panels starting at column kb0 in K slices, so K = 64*nk
// costs one read and one write of C: nk = 2 (16 flop per byte of C traffic).
//
// Update kernel family: 64x64 output tile per CTA, warp tile (8*WM) x (8*WN) of m8n8k4 DMMA
// fragments, K streamed in KC-wide slices through a STAGES-deep cp.async pipeline.
template <int KC>
__device__ __forceinline__ void load_slice_async(double* __restrict__ s, const double* __restrict__ gsrc, int64_t ld,
                                                 int nthreads) {
    constexpr int LD = KC + 4;  // (KC+4)*8 bytes per row: the 8 rows of one fragment load hit distinct banks
    for (int idx = threadIdx.x; idx < 64 * (KC / 2); idx += nthreads) {
        const int r = idx / (KC / 2), c2 = idx % (KC / 2);
        panel::cp_async16(s + r * LD + 2 * c2, gsrc + (size_t)r * ld + 2 * c2);
    }
}

template <int WM, int WN, int LD, int KD>
__device__ __forceinline__ void warp_mma(const double* __restrict__ As, const double* __restrict__ Bs,
                                         double (&acc)[WM][WN][2], int r0, int c0) {
    const int lane = threadIdx.x & 31;
    const int g = lane >> 2, t = lane & 3;
#pragma unroll 2
    for (int kk = 0; kk < KD; kk += 4) {
        double af[WM], bf[WN];
#pragma unroll
        for (int i = 0; i < WM; ++i) af[i] = -As[(r0 + 8 * i + g) * LD + kk + t];
#pragma unroll
        for (int j = 0; j < WN; ++j) bf[j] = Bs[(c0 + 8 * j + g) * LD + kk + t];
#pragma unroll
        for (int i = 0; i < WM; ++i)
#pragma unroll
            for (int j = 0; j < WN; ++j) panel::dmma(acc[i][j], af[i], bf[j]);
    }
}

template <int WM, int WN, int KC, int STAGES>
struct UpdateCfg {
    static constexpr int kWarpsM = 64 / (8 * WM), kWarpsN = 64 / (8 * WN);
    static constexpr int kThreads = 32 * kWarpsM * kWarpsN;
    static constexpr int kLd = KC + 4;
    static constexpr size_t kSmem = (size_t)STAGES * 2 * 64 * kLd * sizeof(double);
    static constexpr int kMinBlocks = (227 * 1024) / (int)kSmem < 4 ? (227 * 1024) / (int)kSmem : 4;
};

template <int WM, int WN, int KC, int STAGES>
__global__ void __launch_bounds__(UpdateCfg<WM, WN, KC, STAGES>::kThreads, UpdateCfg<WM, WN, KC, STAGES>::kMinBlocks)
    k_update(double* __restrict__ a, int64_t ld, int64_t stride, int64_t kb0, int nk, int64_t tc0, int64_t T,
             int64_t nsq, int64_t skip) {
    using Cfg = UpdateCfg<WM, WN, KC, STAGES>;
    constexpr int LD = Cfg::kLd;
    extern __shared__ double smem[];
    auto stage = [&](int st, int which) { return smem + (2 * st + which) * 64 * LD; };
    const int f = blockIdx.y;
    const int64_t x = blockIdx.x;
    const int64_t L = nsq - tc0;                     // square row tiles of the first column tile
    const int64_t n_square = T * L - T * (T - 1) / 2;
    int64_t c, tr;
    if (x < n_square) {
        // column offset c: largest c with cum(c) = c*L - c(c-1)/2 <= x
        const double b = 2.0 * (double)L + 1.0;
        c = (int64_t)((b - sqrt(fmax(b * b - 8.0 * (double)x, 0.0))) * 0.5);
        auto cum = [L](int64_t cc) { return cc * L - cc * (cc - 1) / 2; };
        while (c > 0 && cum(c) > x) --c;
        while (c + 1 < T && cum(c + 1) <= x) ++c;
        tr = tc0 + c + (x - cum(c));
        if (tr < tc0 + skip) return;
    } else {
        const int64_t y = x - n_square;
        c = y % T;
        tr = nsq + y / T;
    }
    const int64_t ri = tr * kNb, cj = (tc0 + c) * kNb;
    double* A = a + (size_t)f * stride;
    const int nsub = nk * (kNb / KC);
    // prologue: STAGES-1 slices in flight
#pragma unroll
    for (int p = 0; p < STAGES - 1; ++p) {
        if (p < nsub) {
            const int64_t kc = kb0 + (int64_t)p * KC;
            load_slice_async<KC>(stage(p, 0), A + ri * ld + kc, ld, Cfg::kThreads);
            load_slice_async<KC>(stage(p, 1), A + cj * ld + kc, ld, Cfg::kThreads);
        }
        asm volatile("cp.async.commit_group;\n" ::);
    }
    const int w = threadIdx.x >> 5;
    const int r0 = 8 * WM * (w / Cfg::kWarpsN), c0 = 8 * WN * (w % Cfg::kWarpsN);
    double acc[WM][WN][2] = {};
    for (int sc = 0; sc < nsub; ++sc) {
        const int pf = sc + STAGES - 1;  // slice to prefetch into the stage freed last iteration
        if (pf < nsub) {
            const int64_t kc = kb0 + (int64_t)pf * KC;
            load_slice_async<KC>(stage(pf % STAGES, 0), A + ri * ld + kc, ld, Cfg::kThreads);
            load_slice_async<KC>(stage(pf % STAGES, 1), A + cj * ld + kc, ld, Cfg::kThreads);
        }
        asm volatile("cp.async.commit_group;\n" ::);
        asm volatile("cp.async.wait_group %0;\n" ::"n"(STAGES - 1));
        __syncthreads();
        warp_mma<WM, WN, LD, KC>(stage(sc % STAGES, 0), stage(sc % STAGES, 1), acc, r0, c0);
        __syncthreads();
    }
    const int lane = threadIdx.x & 31;
    const int g = lane >> 2, t = lane & 3;
#pragma unroll
    for (int i = 0; i < WM; ++i)
#pragma unroll
        for (int j = 0; j < WN; ++j) {
            double2* pc = reinterpret_cast<double2*>(A + (size_t)(ri + r0 + 8 * i + g) * ld + cj + c0 + 8 * j + 2 * t);
            double2 v = *pc;
            v.x += acc[i][j][0];
            v.y += acc[i][j][1];
            *pc = v;
        }
}

// Variant table of the update kernel (selected by GWB200_UPDATE_VARIANT, default kDefaultUpdateVariant).
struct UpdateVariant {
    void (*fn)(double*, int64_t, int64_t, int64_t, int, int64_t, int64_t, int64_t, int64_t);
    int threads;
    size_t smem;
    const char* name;
};
template <int WM, int WN, int KC, int ST>
UpdateVariant make_variant(const char* name) {
    using Cfg = UpdateCfg<WM, WN, KC, ST>;
    return {k_update<WM, WN, KC, ST>, Cfg::kThreads, Cfg::kSmem, name};
}
const UpdateVariant kVariants[] = {
    make_variant<2, 4, 32, 2>("w16x32_k32_s2"),
    make_variant<4, 4, 32, 2>("w32x32_k32_s2"),
    make_variant<4, 4, 16, 3>("w32x32_k16_s3"),
    make_variant<2, 4, 32, 3>("w16x32_k32_s3"),
    make_variant<4, 8, 32, 2>("w32x64_k32_s2"),
    make_variant<4, 4, 32, 3>("w32x32_k32_s3"),
};
constexpr int kNumVariants = (int)(sizeof(kVariants) / sizeof(kVariants[0]));

}  // namespace

int fp64_update_mode() {  // GWB200_FP64_UPDATE: 1 = dmma (FP64 pipe only), 2 = ozaki (int8 emulation), 0 = tuned
    const char* env = std::getenv("GWB200_FP64_UPDATE");
    if (env && std::strcmp(env, "dmma") == 0) return 1;
    if (env && std::strcmp(env, "ozaki") == 0) return 2;
    return 0;
}

namespace {

int env_update_variant() {  // GWB200_UPDATE_VARIANT forces a variant; -1 if unset or out of range
    if (const char* env = std::getenv("GWB200_UPDATE_VARIANT")) {
        const int e = std::atoi(env);
        if (e >= 0 && e < kNumVariants) return e;
    }
    return -1;
}

void launch_variant(int v, const TallGeometry& g, int64_t nf, double* a, int64_t kb0, int nk, int64_t tc0, int64_t T,
                    cudaStream_t s, int64_t skip = 0) {
    const UpdateVariant& uv = kVariants[v];
    const int64_t nsq = g.n_pad / kNb, nrt = g.rows / kNb;
    const int64_t L = nsq - tc0;
    const int64_t tiles = T * L - T * (T - 1) / 2 + T * (nrt - nsq);
    if (tiles <= 0) return;
    uv.fn<<<dim3((unsigned)tiles, (unsigned)nf), uv.threads, uv.smem, s>>>(a, g.ld, g.stride, kb0, nk, tc0, T, nsq, skip);
    GWB_LAUNCH("k_update");
}

std::mutex g_tune_mu;
std::map<std::array<int64_t, 6>, int> g_tuned;  // (device, n_pad, rows, nf, int8 candidate, all) -> variant

// q_out[f, j] = -qacc[f, j]  (x^T W_c x = -||L^{-1} D^1/2 x||^2).
__global__ void k_negate_copy(const double* __restrict__ qacc, int nf, int m, int64_t ldq_in, double* __restrict__ q,
                              int64_t ldq_out) {
    const int f = blockIdx.y;
    for (int j = blockIdx.x * blockDim.x + threadIdx.x; j < m; j += gridDim.x * blockDim.x)
        q[(size_t)f * ldq_out + j] = -qacc[(size_t)f * ldq_in + j];
}

} // namespace

int launch_gather_vph(const double* pqo, int64_t nmo, int64_t nocc, double* v, cudaStream_t s) {
    const int n = (int)(nocc * (nmo - nocc));
    dim3 grid((unsigned)std::min<int64_t>((n + 255) / 256, 64), (unsigned)std::min(n, 65535));
    k_gather_vph<<<grid, 256, 0, s>>>(pqo, (int)nmo, (int)nocc, n, v);
    GWB_LAUNCH("k_gather_vph");
    return 1;
}

int launch_gather_panel(const double* pqo, int64_t nmo, int64_t nocc, const int64_t* states, int64_t nstates,
                        double* xt, cudaStream_t s) {
    const int n = (int)(nocc * (nmo - nocc));
    const int m = (int)(nstates * nmo);
    dim3 grid((unsigned)std::min<int64_t>((n + 255) / 256, 64), (unsigned)std::min(m, 65535));
    k_gather_panel<<<grid, 256, 0, s>>>(pqo, (int)nmo, (int)nocc, n, states, m, xt);
    GWB_LAUNCH("k_gather_panel");
    return 1;
}

int launch_sigma_x_diag(const double* xdiag, int64_t nmo, int64_t nocc, double* out, cudaStream_t s) {
    k_sigma_x_diag<<<(unsigned)((nmo + 127) / 128), 128, 0, s>>>(xdiag, (int)nmo, (int)nocc, out);
    GWB_LAUNCH("k_sigma_x_diag");
    return 1;
}

int launch_delta(const double* mo, int64_t nmo, int64_t nocc, double* delta, cudaStream_t s) {
    const int64_t n = nocc * (nmo - nocc);
    k_delta<<<(unsigned)((n + 255) / 256), 256, 0, s>>>(mo, (int)nmo, (int)nocc, delta);
    GWB_LAUNCH("k_delta");
    return 1;
}

int launch_scale_vectors(const double* delta, int64_t n, int64_t n_pad, const double* omega, int64_t nf,
                         double* dvec, cudaStream_t s) {
    dim3 grid((unsigned)((n_pad + 255) / 256), (unsigned)nf);
    k_scale_vectors<<<grid, 256, 0, s>>>(delta, (int)n, (int)n_pad, omega, (int)nf, dvec);
    GWB_LAUNCH("k_scale_vectors");
    return 1;
}

int launch_build_tall(const TallGeometry& g, const double* v, const double* xt, const double* dvec, int64_t nf,
                      double* a, cudaStream_t s) {
    dim3 grid((unsigned)((g.n_pad + 255) / 256), (unsigned)std::min<int64_t>(g.rows, 65535));
    k_build_tall<<<grid, 256, 0, s>>>(g.n, g.m, g.n_pad, g.ld, g.stride, v, xt, dvec, (int)nf, a);
    GWB_LAUNCH("k_build_tall");
    return 1;
}

// Algorithmic flops of one update: 2 * K_true * (true lower elements of the output columns
// [c0, c1) intersected with [0, n) + m per output column).
static double update_flops(const TallGeometry& g, int64_t kb0, int nk, int64_t c0, int64_t c1) {
    const int64_t kt = std::max<int64_t>(0, std::min<int64_t>(kb0 + (int64_t)nk * kNb, g.n) - kb0);
    const int64_t a0 = std::min(c0, g.n), a1 = std::min(c1, g.n);
    const double cols = (double)(a1 - a0);
    const double lower = cols * (double)g.n - 0.5 * (double)(a0 + a1 - 1) * cols;  // sum_{c} (n - c)
    return 2.0 * (double)kt * (lower + (double)g.m * cols);
}

// ... and of its diagonal block of columns [c0, c1)
static double diag_flops(const TallGeometry& g, int64_t kb0, int nk, int64_t c0, int64_t c1) {
    const int64_t kt = std::max<int64_t>(0, std::min<int64_t>(kb0 + (int64_t)nk * kNb, g.n) - kb0);
    const double cols = (double)(std::min(c1, g.n) - std::min(c0, g.n));
    return (double)kt * cols * (cols + 1.0);
}

int tune_update_variant(const TallGeometry& g, int64_t nf, double* a, cudaStream_t s, void* oz,
                        unsigned long long* sched, unsigned long long* err_pivot, bool timed) {
    const int forced = env_update_variant();
    if (forced >= 0) return forced;
    const int64_t nsq = g.n_pad / kNb;
    if (nsq <= 2) return kDefaultUpdateVariant;  // no outer trailing update to tune on
    if (oz && fp64_update_mode() == 2) return kUpdateOzaki;
    if (fp64_update_mode() == 1) oz = nullptr;  // the FP64 pipe only
    // Untimed (memory-capped handles: the serving loop's slots, whose requests run side by side):
    // the non-persistent DMMA kernel, which leaves SMs to the other slots' kernels (the persistent
    // int8 kernel holds one CTA on every SM it gets); GWB200_FP64_UPDATE=ozaki still forces it.
    if (!timed) return kDefaultUpdateVariant;
    const char* all_env = std::getenv("GWB200_TUNE_ALL");
    const bool all = all_env && all_env[0] == '1';  // every DMMA variant, not only the default
    int dev = 0;
    GWB_CUDA(cudaGetDevice(&dev));
    const std::array<int64_t, 6> key = {dev, g.n_pad, g.rows, nf, oz ? 1 : 0, all ? 1 : 0};
    std::lock_guard<std::mutex> lk(g_tune_mu);
    auto it = g_tuned.find(key);
    if (it != g_tuned.end()) return it->second;
    // Time the candidates on the first steps of this geometry's factorisation, in the workspace before the
    // tall matrix is built there: the values are irrelevant to the timing and are overwritten afterwards.  The
    // steps are those of launch_factor_chunk, without the diagonal blocks: the first block's trailing update
    // and, where the int8 update takes blocks in pairs, the second's too, so that its K = 256 kernel, which
    // does most of its work, is in the comparison (timed at K = 128 over all columns it was taken for 317
    // pairs x 64 frequencies, 261 us a call, where DMMA takes 236).
    cudaEvent_t e0, e1;
    GWB_CUDA(cudaEventCreate(&e0));
    GWB_CUDA(cudaEventCreate(&e1));
    float times[kNumVariants + 1] = {};
    auto time_it = [&](auto&& launch) {
        launch();  // warm-up
        GWB_CUDA(cudaEventRecord(e0, s));
        launch();
        GWB_CUDA(cudaEventRecord(e1, s));
        GWB_CUDA(cudaEventSynchronize(e1));
        float ms = 0.f;
        GWB_CUDA(cudaEventElapsedTime(&ms, e0, e1));
        return ms;
    };
    float best_ms = 0.f, def_ms = 0.f;
    int best = -1;
    const bool pair = nsq > 4;
    const int64_t first = std::min<int64_t>(2, nsq - 2), second = std::min<int64_t>(2, nsq - 4);  // tiles of the next blocks
    for (int v = 0; v < kNumVariants; ++v) {
        if (!all && v != kDefaultUpdateVariant) continue;
        GWB_CUDA(cudaFuncSetAttribute(kVariants[v].fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kVariants[v].smem));
        const float ms = time_it([&] {
            launch_variant(v, g, nf, a, 0, 2, 2, nsq - 2, s, first);
            if (pair) launch_variant(v, g, nf, a, 2 * kNb, 2, 4, nsq - 4, s, second);
        });
        times[v] = ms;
        if (v == kDefaultUpdateVariant) def_ms = ms;
        if (best < 0 || ms < best_ms) {
            best_ms = ms;
            best = v;
        }
    }
    if (oz) {  // the int8 emulation of the outer update (kernels_oz.cu), slicing included
        const float ms = time_it([&] {
            launch_clear_sched(g, sched, s);
            launch_update64_oz(g, nf, a, 0, 2 * kNb, pair ? 4 * kNb : g.n_pad, oz, sched, err_pivot, s, 0, first * kNb);
            if (pair) launch_update64_oz(g, nf, a, 0, 4 * kNb, g.n_pad, oz, sched + 1, err_pivot, s, 0, second * kNb);
        });
        times[kUpdateOzaki] = ms;
        if (ms < best_ms) {
            best_ms = ms;
            best = kUpdateOzaki;
        }
        // a wait that expired during the timing would have recorded pivot 0: start clean
        GWB_CUDA(cudaMemsetAsync(err_pivot, 0xFF, sizeof(unsigned long long), s));
    }
    cudaEventDestroy(e0);
    cudaEventDestroy(e1);
    if (def_ms <= 1.03f * best_ms) best = kDefaultUpdateVariant;  // keep the default unless clearly beaten
    g_tuned[key] = best;
    if (const char* verbose = std::getenv("GWB200_VERBOSE"); verbose && verbose[0] == '1') {
        std::fprintf(stderr, "gwb200: update kernel for n_pad=%lld rows=%lld nf=%lld:", (long long)g.n_pad,
                     (long long)g.rows, (long long)nf);
        for (int v = 0; v < kNumVariants; ++v)
            if (all || v == kDefaultUpdateVariant) std::fprintf(stderr, " %s %.3f ms", kVariants[v].name, times[v]);
        if (oz) std::fprintf(stderr, " int8_emulation %.3f ms", times[kUpdateOzaki]);
        std::fprintf(stderr, " -> %s\n", update_variant_name(best));
    }
    return best;
}

const char* update_variant_name(int v) {
    if (v == kUpdateOzaki) return "int8_emulation";
    return (v >= 0 && v < kNumVariants) ? kVariants[v].name : "?";
}

int launch_factor_chunk(const TallGeometry& g, int64_t nf, double* a, double* qacc, unsigned long long* err_pivot,
                        cudaStream_t s, UpdateProfiler* prof, int variant, void* oz, unsigned long long* sched,
                        int max_ctas, SideStream* side) {
    const bool use_oz = oz && variant == kUpdateOzaki;
    if (variant < 0 || variant >= kNumVariants)  // untuned caller: GWB200_UPDATE_VARIANT, else the default
        variant = env_update_variant() >= 0 ? env_update_variant() : kDefaultUpdateVariant;
    const int64_t nsq = g.n_pad / kNb;   // square tile rows/cols
    constexpr int64_t kOuter = 2;        // 64-wide tiles per outer block
    if (!use_oz && nsq > kOuter)
        GWB_CUDA(cudaFuncSetAttribute(kVariants[variant].fn, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                      (int)kVariants[variant].smem));
    int launches = 0;
    if (use_oz && nsq > kOuter) launches += launch_clear_sched(g, sched, s);
    launches += launch_diag64(g, nf, a, 0, std::min(kOuter, nsq) * kNb, 0, err_pivot, s);
    // The next diagonal block (one CTA per frequency, ~40 us) runs beside the trailing update: it is
    // launched first and takes nf SMs, the update's CTAs the others and those that become free: 1098 ->
    // 981 us for the forms of 737 pairs x 64 frequencies, 2845 -> 2634 for 1125 x 48.  With as many
    // frequencies as SMs there is nothing beside it.
    if (prof || max_ctas > 0 || nf >= tc::sm_count()) side = nullptr;
    for (int64_t ob = 0; ob < nsq; ob += kOuter) {
        const int64_t q = std::min(kOuter, nsq - ob), tc0 = ob + q;
        launches += launch_panel64(g, nf, a, ob * kNb, q * kNb, qacc, s);
        if (tc0 >= nsq) break;
        const int64_t next = std::min(kOuter, nsq - tc0);
        // int8: outer blocks in pairs while columns remain behind the pair.  The first updates the
        // second's columns alone, then both update the rest at K = 256.  (Pairs begin at multiples of
        // 256 columns whatever n_pad, so a molecule's columns take the same steps in a batch's geometry.)
        const bool wide = use_oz && nsq - ob / 4 * 4 > 4, second = wide && ob % 4 == 2;
        const int64_t kb = (second ? ob - kOuter : ob) * kNb, c_end = wide && !second ? tc0 + next : nsq;
        SideScope beside(side, s);
        launches += launch_diag64(g, nf, a, tc0 * kNb, next * kNb, tc0 * kNb - kb, err_pivot, s);
        // the rest of the trailing update (columns remain only behind a full outer block)
        if (prof) prof->begin();
        if (use_oz) {
            launches += launch_update64_oz(g, nf, a, kb, tc0 * kNb, c_end * kNb, oz, sched + ob / kOuter, err_pivot,
                                           beside.stream(), max_ctas, next * kNb);
        } else {
            launch_variant(variant, g, nf, a, kb, (int)q, tc0, nsq - tc0, beside.stream(), next);
            ++launches;
        }
        beside.join();
        const int nk = (int)(tc0 - kb / kNb);
        if (prof)
            prof->end((double)nf * (update_flops(g, kb, nk, tc0 * kNb, c_end * kNb) -
                                    diag_flops(g, kb, nk, tc0 * kNb, (tc0 + next) * kNb)));
    }
    return launches;
}

int launch_negate_copy(const double* qacc, int64_t nf, int64_t m, int64_t ldq_in, double* q_out, int64_t ldq_out,
                       cudaStream_t s) {
    dim3 grid((unsigned)std::min<int64_t>((m + 255) / 256, 64), (unsigned)nf);
    k_negate_copy<<<grid, 256, 0, s>>>(qacc, (int)nf, (int)m, ldq_in, q_out, ldq_out);
    GWB_LAUNCH("k_negate_copy");
    return 1;
}

} // namespace gwb200
