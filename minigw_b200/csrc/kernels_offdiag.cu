// kernels_offdiag.cu -- the correlation self-energy between the requested states, Sigma_c(p_s, p_t; i w):
// an extension beside the reference, which computes the diagonal only (docs/formulation.md:186).
//
// The plain form factors the tall matrix [eps ; (D^1/2 X)^T] per frequency; its lower block ends as
// the solved rows w_{s,k} = L^{-1} D^1/2 x_{p_s k} (tall row n_pad + s nmo + k), whose squared norms
// are the diagonal forms.  The same rows give every cross form at the cost of dot products:
//     q[f, k, s, t] = x_{p_s k}^T W_c(i w_f) x_{p_t k} = -w_{s,k} . w_{t,k}
// and the G0-weighted contraction of the diagonal (kernels_small.cu, src/gw/sigma_c_driver.cpp:
// 119-169) applies unchanged, the Green's function depending on k only:
//     Sigma_c(p_s, p_t; i w_n) = -(1/pi) sum_{f,k} w_f g_{n f k} q[f, k, s, t],
//     g_{n f k} = a / (a^2 + w_f^2),  a = i w_n + E_F - e_k.
//   k_cross_forms          one CTA per (k, frequency): the Gram matrix of the nstates rows on the FP64
//                          tensor cores straight from global memory, an eighth of the row length per
//                          warp, the warps' parts added in a fixed order;
//   k_sigma_contract_pairs one CTA per (output frequency, pair s <= t): the contraction, a fixed
//                          reduction tree; both triangles written.
#include "panel_common.cuh"

#include <type_traits>

namespace gwb200 {
namespace {

constexpr int kXWarps = 8;

// (s, t) with s <= t of upper-triangle index p (row-major: row s holds t = s .. ns-1).
__device__ __forceinline__ void pair_of(int p, int ns, int& s, int& t) {
    s = 0;
    while (p >= ns - s) {
        p -= ns - s;
        ++s;
    }
    t = s + p;
}

// The ns rows (tall rows n_pad + s nmo + k) in tiles of 8: in an m8n8k4 product of a tile with another
// the A fragment of the one and the B fragment of the other are both "row lane / 4, column lane % 4",
// so one register per tile and four columns serves every pair.  Bound by reading the rows once (8
// states, 1125 pairs, 90 orbitals, 48 frequencies: 311 MB in 64 us; one dot product per thread from
// staged rows left 220 of 256 threads idle and took 258).  NT: tiles of 8 states.
template <int NT>
__global__ void __launch_bounds__(32 * kXWarps) k_cross_forms(const double* __restrict__ a, int64_t ld, int64_t stride,
                                                              int64_t n_pad, int nmo, int ns, double* __restrict__ qx) {
    constexpr int kPairs = NT * (NT + 1) / 2;
    __shared__ double part[kXWarps][64];
    const int k = blockIdx.x, f = blockIdx.y;
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, g = lane >> 2, t = lane & 3;
    const double* rows[NT];
#pragma unroll
    for (int i = 0; i < NT; ++i) {  // a tile's missing states read the last one (their products are not stored)
        const int s = min(8 * i + g, ns - 1);
        rows[i] = a + (size_t)f * stride + (size_t)(n_pad + (int64_t)s * nmo + k) * ld + t;
    }
    double acc[kPairs][2] = {};
    // the rows are zero beyond n (identity padding), so whole 64-column blocks are read
#pragma unroll 4
    for (int64_t c = 4 * w; c < n_pad; c += 4 * kXWarps) {
        double x[NT];
#pragma unroll
        for (int i = 0; i < NT; ++i) x[i] = rows[i][c];
        int p = 0;
#pragma unroll
        for (int i = 0; i < NT; ++i)
#pragma unroll
            for (int j = i; j < NT; ++j, ++p)
                panel::dmma(acc[p], x[i], x[j]);
    }
    double* out = qx + ((size_t)f * nmo + k) * ns * ns;
    int p = 0;
#pragma unroll
    for (int i = 0; i < NT; ++i)
#pragma unroll
        for (int j = i; j < NT; ++j, ++p) {
            part[w][8 * g + 2 * t] = acc[p][0];
            part[w][8 * g + 2 * t + 1] = acc[p][1];
            __syncthreads();
            if (threadIdx.x < 64) {
                const int s = 8 * i + (threadIdx.x >> 3), u = 8 * j + (threadIdx.x & 7);
                double sum = 0.0;
#pragma unroll
                for (int v = 0; v < kXWarps; ++v) sum += part[v][threadIdx.x];
                if (s <= u && u < ns) {  // both triangles from one value
                    out[s * ns + u] = -sum;
                    out[u * ns + s] = -sum;
                }
            }
            __syncthreads();
        }
}

__global__ void __launch_bounds__(256) k_sigma_contract_pairs(const double* __restrict__ qx, int nf_int, int nmo,
                                                              int ns, const double* __restrict__ mo, double fermi,
                                                              const double* __restrict__ omega_int,
                                                              const double* __restrict__ weight_int,
                                                              const double* __restrict__ omega_out, int nf_out,
                                                              double* __restrict__ sigma) {
    const int fn = blockIdx.x;
    int s, t;
    pair_of(blockIdx.y, ns, s, t);
    const double wn = omega_out[fn];
    double sr = 0.0, si = 0.0;
    const int total = nf_int * nmo;
    for (int idx = threadIdx.x; idx < total; idx += blockDim.x) {
        const int fp = idx / nmo, k = idx - fp * nmo;
        const double q = qx[((size_t)fp * nmo + k) * ns * ns + (size_t)s * ns + t];
        const double ar = fermi - mo[k], ai = wn;
        const double wp = omega_int[fp];
        const double dr = ar * ar - ai * ai + wp * wp, di = 2.0 * ar * ai;
        const double inv = 1.0 / (dr * dr + di * di);
        const double gr = (ar * dr + ai * di) * inv, gi = (ai * dr - ar * di) * inv;
        const double scale = -weight_int[fp] * q;
        sr = fma(gr, scale, sr);
        si = fma(gi, scale, si);
    }
    __shared__ double red[2][256];
    red[0][threadIdx.x] = sr;
    red[1][threadIdx.x] = si;
    __syncthreads();
    for (int off = blockDim.x / 2; off > 0; off >>= 1) {
        if ((int)threadIdx.x < off) {
            red[0][threadIdx.x] += red[0][threadIdx.x + off];
            red[1][threadIdx.x] += red[1][threadIdx.x + off];
        }
        __syncthreads();
    }
    if (threadIdx.x == 0) {
        const double inv_pi = 1.0 / 3.141592653589793238462643383279502884;
        for (int e = 0; e < (s == t ? 1 : 2); ++e) {
            const size_t pos = (size_t)(e == 0 ? s * ns + t : t * ns + s) * nf_out + fn;
            sigma[2 * pos] = red[0][0] * inv_pi;
            sigma[2 * pos + 1] = red[1][0] * inv_pi;
        }
    }
}

} // namespace

int launch_cross_forms(const TallGeometry& g, int64_t nf, const double* a, int64_t nmo, int64_t nstates, double* qx,
                       cudaStream_t s) {
    const int ns = (int)nstates;
    if (ns < 1 || ns > 64) fail(GWB200_BAD_SHAPE, "too many states for the cross forms");
    const dim3 grid((unsigned)nmo, (unsigned)nf);
    auto run = [&](auto nt) {
        k_cross_forms<decltype(nt)::value><<<grid, 32 * kXWarps, 0, s>>>(a, g.ld, g.stride, g.n_pad, (int)nmo, ns, qx);
    };
    switch ((ns + 7) / 8) {
        case 1: run(std::integral_constant<int, 1>{}); break;
        case 2: run(std::integral_constant<int, 2>{}); break;
        case 3: run(std::integral_constant<int, 3>{}); break;
        case 4: run(std::integral_constant<int, 4>{}); break;
        case 5: run(std::integral_constant<int, 5>{}); break;
        case 6: run(std::integral_constant<int, 6>{}); break;
        case 7: run(std::integral_constant<int, 7>{}); break;
        default: run(std::integral_constant<int, 8>{}); break;
    }
    GWB_LAUNCH("k_cross_forms");
    return 1;
}

int launch_sigma_contract_pairs(const double* qx, int64_t nf_int, int64_t nmo, int64_t nstates, const double* mo,
                                double fermi, const double* omega_int, const double* weight_int,
                                const double* omega_out, int64_t nf_out, double* sigma, cudaStream_t s) {
    const int64_t npair = nstates * (nstates + 1) / 2;
    k_sigma_contract_pairs<<<dim3((unsigned)nf_out, (unsigned)npair), 256, 0, s>>>(
        qx, (int)nf_int, (int)nmo, (int)nstates, mo, fermi, omega_int, weight_int, omega_out, (int)nf_out, sigma);
    GWB_LAUNCH("k_sigma_contract_pairs");
    return 1;
}

} // namespace gwb200
