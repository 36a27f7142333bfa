// kernels_small.cu -- FP64 device kernels after the screening: the G0-weighted frequency
// contraction into Sigma_c(iw), the Pade continued fraction, the quasiparticle fixed point
// and the E_c.out sweep, plus the FP64 DMMA peak probe.
//
// The Pade / QP kernels reproduce the reference's std::complex<double> arithmetic operation
// by operation (src/gw/pade.cpp:10-101, src/gw/qp_solver.cpp:10-47): products are
// (ac - bd, ad + bc) with no fused multiply-add (explicit __dmul_rn / __dadd_rn), and
// quotients use Smith's algorithm (R. L. Smith, "Algorithm 116: Complex division",
// CACM 5(8), 1962), the method GCC's runtime applies for std::complex<double> division in
// the normal exponent range.  Given identical Sigma_c input the device quasiparticle
// energies therefore match a host build of the reference bit for bit.
#include "internal.cuh"

#include <cmath>

namespace gwb200 {
namespace {

struct cplx {
    double re, im;
};

__device__ __forceinline__ cplx c_add(cplx a, cplx b) { return {__dadd_rn(a.re, b.re), __dadd_rn(a.im, b.im)}; }
__device__ __forceinline__ cplx c_sub(cplx a, cplx b) { return {__dsub_rn(a.re, b.re), __dsub_rn(a.im, b.im)}; }
__device__ __forceinline__ cplx c_mul(cplx a, cplx b) {
    const double ac = __dmul_rn(a.re, b.re), bd = __dmul_rn(a.im, b.im);
    const double ad = __dmul_rn(a.re, b.im), bc = __dmul_rn(a.im, b.re);
    return {__dsub_rn(ac, bd), __dadd_rn(ad, bc)};
}
// Smith's algorithm, evaluated without contraction.
__device__ __forceinline__ cplx c_div(cplx x, cplx y) {
    const double a = x.re, b = x.im, c = y.re, d = y.im;
    if (fabs(c) < fabs(d)) {
        const double ratio = __ddiv_rn(c, d);
        const double denom = __dadd_rn(__dmul_rn(c, ratio), d);
        return {__ddiv_rn(__dadd_rn(__dmul_rn(a, ratio), b), denom),
                __ddiv_rn(__dsub_rn(__dmul_rn(b, ratio), a), denom)};
    }
    const double ratio = __ddiv_rn(d, c);
    const double denom = __dadd_rn(__dmul_rn(d, ratio), c);
    return {__ddiv_rn(__dadd_rn(__dmul_rn(b, ratio), a), denom),
            __ddiv_rn(__dsub_rn(b, __dmul_rn(a, ratio)), denom)};
}
// c_abs(a) < 1e-20 (hypot), decided without the square root wherever the larger part alone decides it:
// max(|re|, |im|) <= hypot <= sqrt(2) max up to rounding.
__device__ __noinline__ bool hypot_below(cplx a) { return hypot(a.re, a.im) < 1e-20; }
__device__ __forceinline__ bool c_small(cplx a) {
    if (fabs(a.re) > 1.001e-20 || fabs(a.im) > 1.001e-20) return false;
    return hypot_below(a);
}

// x / y by c_div's steps with shorter chains and no branch.  A quotient a / b comes from the
// correctly rounded reciprocal y of b, a quotient q within one ulp and its exact residual r = a - b q
// as fma(r, y, q), which is the correctly rounded quotient, the bits of __ddiv_rn (P. Markstein, IBM
// J. Res. Dev. 34(1), 1990; y likewise from a reciprocal within one ulp, unless b's significand is
// all ones).  Both parts share denom's reciprocal, whose first approximation comes from the
// unrounded ratio, so that it does not wait for the rounded one.  `ok` is cleared, and the result
// void, unless the divisor's larger part is within 2^-60 .. 2^400 (so it is not c_small), the ratio of
// its parts and both numerators are at least 2^-300 and finite (no residual underflows; zeros,
// infinities and NaN are out), its parts differ in their leading words (their order is decided on
// those) and neither divisor ends in 32 ones.
__device__ __noinline__ cplx c_div_general(cplx x, cplx y) { return c_div(x, y); }
__device__ __forceinline__ double rcp_iter(double b) {  // 1 / b within one ulp: a third-order iteration
    double y;
    asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(b));
    const double e = fma(-b, y, 1.0);
    return fma(y, fma(e, e, e), y);
}
__device__ __forceinline__ double rcp_step(double b, double y) { return fma(y, fma(-b, y, 1.0), y); }
// y0 within a few ulp of 1 / b, y its correct rounding
__device__ __forceinline__ double quotient(double a, double b, double y0, double y) {
    double q = a * y0;
    q = fma(fma(-b, q, a), y0, q);
    return fma(fma(-b, q, a), y, q);
}
__device__ __forceinline__ unsigned hi_abs(double v) { return (unsigned)__double2hiint(v) & 0x7fffffffu; }
__device__ __forceinline__ bool exponent_in(double v, unsigned lo, unsigned hi) {  // 2^(lo - 1023) <= |v| < 2^(hi - 1023)
    return hi_abs(v) - (lo << 20) < ((hi - lo) << 20);
}
__device__ __forceinline__ cplx c_div_chain(cplx x, cplx y, bool& ok) {
    const double a = x.re, b = x.im;
    const unsigned hre = hi_abs(y.re), him = hi_abs(y.im);
    const bool swap = hre < him;
    const double s = swap ? y.re : y.im, big = swap ? y.im : y.re;
    const double y0 = rcp_iter(big);
    const double d0 = rcp_iter(fma(s, s * y0, big));  // of denom, to a few ulp
    const double ratio = quotient(s, big, y0, rcp_step(big, y0));
    const double denom = __dadd_rn(__dmul_rn(s, ratio), big);
    const double p = swap ? a : b, q = swap ? b : a;
    const double nr = __dadd_rn(__dmul_rn(p, ratio), q);
    const double t = __dmul_rn(q, ratio);
    const double ni = swap ? __dsub_rn(t, a) : __dsub_rn(b, t);
    const double d1 = rcp_step(denom, rcp_step(denom, d0));
    const double re = quotient(nr, denom, d0, d1), im = quotient(ni, denom, d0, d1);
    ok = ok && hre != him && exponent_in(big, 1023 - 60, 1023 + 400) && exponent_in(ratio, 1023 - 300, 1024) &&
         exponent_in(nr, 1023 - 300, 1023 + 400) && exponent_in(ni, 1023 - 300, 1023 + 400) &&
         __double2loint(big) != -1 && __double2loint(denom) != -1;
    return {re, im};
}

constexpr int kMaxPade = 128;

// Thiele continued-fraction coefficients (src/gw/pade.cpp:10-63) by one warp: only the previous
// column of the reference's table g is live, kept as `coeffs` updated in place (lane i holds rows i,
// i + 32, ...), so after column ip coeffs[ip] = g(ip, ip).  The rows of a column are independent.
// row: sigma(i omega) as interleaved complex numbers; xs_im: the sample points i * xs_im.
__device__ int pade_coeffs(const double* __restrict__ row, const double* __restrict__ omega, int n, int npar,
                           cplx* coeffs, double* xs_im) {
    const int lane = threadIdx.x & 31;
    const int na = npar < n ? npar : n;
    const int step = na > 1 ? n / (na - 1) : 1;
    for (int i = lane; i < na; i += 32) {
        const int f = (na > 1 && i == na - 1) ? n - 1 : i * step;
        xs_im[i] = omega[f];
        coeffs[i] = {row[2 * f], row[2 * f + 1]};
    }
    __syncwarp();
    for (int ip = 1; ip < na; ++ip) {
        const cplx pivot = coeffs[ip - 1];
        const cplx x0{0.0, xs_im[ip - 1]};
        for (int id = ip + lane; id < na; id += 32) {
            const cplx c = coeffs[id];
            const cplx num = c_sub(pivot, c);
            const cplx den = c_mul(c_sub(cplx{0.0, xs_im[id]}, x0), c);
            bool ok = true;
            cplx v = c_div_chain(num, den, ok);
            if (!ok) v = c_div_general(num, c_small(den) ? cplx{1e-20, 0.0} : den);
            coeffs[id] = v;
        }
        __syncwarp();
    }
    return na;
}

// Backward evaluation at real z (src/gw/pade.cpp:65-101); num(k) = coeffs[k + 1] (z - xs[k]).  The
// chain runs through without a branch and is done again step by step if one of its steps was not
// covered.
template <class Num>
__device__ __noinline__ cplx pade_eval_general(cplx first, int npar, Num num) {
    cplx val{1.0, 0.0};
    for (int k = npar - 2; k >= 0; --k) {
        if (c_small(val)) val = cplx{1e-20, 0.0};
        val = c_add(cplx{1.0, 0.0}, c_div(num(k), val));
    }
    return c_div(first, c_small(val) ? cplx{1e-20, 0.0} : val);
}
template <class Num>
__device__ __forceinline__ cplx pade_eval(cplx first, int npar, Num num) {
    if (npar == 1) return first;
    // the innermost step divides by exactly 1: c_div(x, 1) is x + 0 componentwise
    const cplx inner = num(npar - 2);
    cplx val = c_add(cplx{1.0, 0.0}, cplx{__dadd_rn(__dmul_rn(inner.im, 0.0), inner.re),
                                          __dsub_rn(inner.im, __dmul_rn(inner.re, 0.0))});
    bool ok = true;
#pragma unroll 2
    for (int k = npar - 3; k >= 0; --k) val = c_add(cplx{1.0, 0.0}, c_div_chain(num(k), val, ok));
    val = c_div_chain(first, val, ok);
    return ok ? val : pade_eval_general(first, npar, num);
}
__device__ __forceinline__ cplx pade_num(const cplx* coeffs, const double* xs_im, double z, int k) {
    return c_mul(coeffs[k + 1], c_sub(cplx{z, 0.0}, cplx{0.0, xs_im[k]}));
}

// One warp per requested state (row of sigma, entry of qp): Pade fit of Sigma_c(p, iw) and the fixed-point QP update
// (src/gw/qp_solver.cpp:18-43), <= 200 iterations, tolerance 1e-6.  Bound by the chain of the
// evaluations (a state that does not settle takes all 200); the numerators of an evaluation do not
// depend on each other and are formed by the lanes before it.  60 states, 16 parameters, 100
// frequencies: 441 us (1347 us with one thread per state, __ddiv_rn and hypot at every step).
__global__ void __launch_bounds__(32) k_qp(const double* __restrict__ sigma, const double* __restrict__ omega,
                                           int nfreq, const int64_t* __restrict__ states, int npade,
                                           const double* __restrict__ mo, double fermi, const double* __restrict__ sigx,
                                           const double* __restrict__ vxc_diag, double* __restrict__ qp) {
    __shared__ cplx coeffs[kMaxPade], num[kMaxPade];
    __shared__ double xs_im[kMaxPade];
    const int lane = threadIdx.x;
    const int p = (int)states[blockIdx.x];
    const int na = pade_coeffs(sigma + 2 * (size_t)blockIdx.x * nfreq, omega, nfreq, npade, coeffs, xs_im);
    const double e = mo[p], sx = sigx[p], vx = vxc_diag[p];
    const cplx first = coeffs[0];
    double cur = e;
    for (int it = 0; it < 200; ++it) {
        const double target = __dsub_rn(cur, fermi);
        for (int k = lane; k < na - 1; k += 32) num[k] = pade_num(coeffs, xs_im, target, k);
        __syncwarp();
        const cplx sc = pade_eval(first, na, [&](int k) { return num[k]; });
        __syncwarp();
        const double nq = __dsub_rn(__dadd_rn(__dadd_rn(e, sc.re), sx), vx);
        const bool done = fabs(__dsub_rn(nq, cur)) < 1e-6;
        cur = nq;
        if (done) break;
    }
    if (lane == 0) qp[blockIdx.x] = cur;
}

// E_c.out sweep (src/io.cpp:94-108): coefficients once per block, one point per thread.
__global__ void __launch_bounds__(128) k_pade_sweep(const double* __restrict__ sigma_row,
                                                    const double* __restrict__ omega, int nfreq, int npade, int npts,
                                                    double fermi, double x_start, double interval,
                                                    double* __restrict__ out) {
    __shared__ cplx coeffs[kMaxPade];
    __shared__ double xs_im[kMaxPade];
    const int na = npade < nfreq ? npade : nfreq;
    if (threadIdx.x < 32) pade_coeffs(sigma_row, omega, nfreq, npade, coeffs, xs_im);
    __syncthreads();
    const cplx first = coeffs[0];
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < npts; i += gridDim.x * blockDim.x) {
        const double e = __dsub_rn(__dadd_rn(x_start, __dmul_rn((double)i, interval)), fermi);
        const cplx v = pade_eval(first, na, [&](int k) { return pade_num(coeffs, xs_im, e, k); });
        out[3 * (size_t)i + 0] = __dmul_rn(__dadd_rn(e, fermi), 27.211386245988);
        out[3 * (size_t)i + 1] = v.re;
        out[3 * (size_t)i + 2] = v.im;
    }
}

// Sigma_c(p_s, i w_n) = -(1/pi) sum_{f', k} w_{f'} g(k, n, f') q[f', s, k], with
// g = a / (a^2 + w_{f'}^2), a = i w_n + E_F - e_k, and q = x^T W_c x <= 0 the screened forms
// (the reference's accumulation, src/gw/sigma_c_driver.cpp:154-168, with W_c hoisted out of
// the loop over w_n).  The integration frequencies f' (omega_int, weight_int, rows of qall) may be
// a shard of the output grid (omega_out): the shards' results then add up to the full sum.
// sigma: [state][output frequency].  One block per (n, s); fixed-shape tree reduction (deterministic).
__global__ void __launch_bounds__(256) k_sigma_contract(const double* __restrict__ qall, int nf_int, int nmo,
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
        const double q = qall[(size_t)fp * ldq + (size_t)s * nmo + k];
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

// Short FP64 DMMA throughput probe (8 warps/block, 4 independent accumulators per warp).
__global__ void k_dmma_probe(double* out, int iters) {
    double a = threadIdx.x * 1e-3, b = 1.0 - threadIdx.x * 1e-4;
    double c[4][2] = {};
    for (int i = 0; i < iters; ++i) {
#pragma unroll
        for (int j = 0; j < 4; ++j)
            asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0,%1}, {%2}, {%3}, {%0,%1};\n"
                         : "+d"(c[j][0]), "+d"(c[j][1])
                         : "d"(a), "d"(b));
    }
    double s = 0;
    for (int j = 0; j < 4; ++j) s += c[j][0] + c[j][1];
    out[blockIdx.x * blockDim.x + threadIdx.x] = s;
}

} // namespace

int launch_sigma_contract(const double* qall, int64_t nf_int, int64_t nstates, int64_t nmo, int64_t ldq,
                          const double* mo, double fermi, const double* omega_int, const double* weight_int,
                          const double* omega_out, int64_t nf_out, double* sigma, cudaStream_t s) {
    dim3 grid((unsigned)nf_out, (unsigned)nstates);
    k_sigma_contract<<<grid, 256, 0, s>>>(qall, (int)nf_int, (int)nmo, ldq, mo, fermi, omega_int, weight_int,
                                          omega_out, (int)nf_out, sigma);
    GWB_LAUNCH("k_sigma_contract");
    return 1;
}

void check_npade(int64_t npade) {
    if (npade > kMaxPade) fail(GWB200_BAD_SHAPE, "npade exceeds the device Pade limit of 128");
}

int launch_qp(const double* sigma, const double* omega, int64_t nfreq, const int64_t* states, int64_t nstates,
              int64_t npade, const double* mo, double fermi, const double* sigx, const double* vxc_diag, double* qp,
              cudaStream_t s) {
    check_npade(npade);
    k_qp<<<(unsigned)nstates, 32, 0, s>>>(sigma, omega, (int)nfreq, states, (int)npade, mo, fermi, sigx, vxc_diag, qp);
    GWB_LAUNCH("k_qp");
    return 1;
}

int launch_pade_sweep(const double* sigma_row, const double* omega, int64_t nfreq, int64_t npade, int64_t npts,
                      double fermi, double x_start, double interval, double* out, cudaStream_t s) {
    check_npade(npade);
    k_pade_sweep<<<(unsigned)std::min<int64_t>((npts + 127) / 128, 8 * 148), 128, 0, s>>>(
        sigma_row, omega, (int)nfreq, (int)npade, (int)npts, fermi, x_start, interval, out);
    GWB_LAUNCH("k_pade_sweep");
    return 1;
}

double measure_fp64_peak_tflops(cudaStream_t s) {
    int dev = 0, sms = 0;
    GWB_CUDA(cudaGetDevice(&dev));
    GWB_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
    const int blocks = sms * 8, threads = 256, iters = 4096;
    double* d = nullptr;
    GWB_CUDA(cudaMalloc(&d, sizeof(double) * blocks * threads));
    cudaEvent_t e0, e1;
    GWB_CUDA(cudaEventCreate(&e0));
    GWB_CUDA(cudaEventCreate(&e1));
    k_dmma_probe<<<blocks, threads, 0, s>>>(d, 64);
    float best = 1e30f;
    for (int rep = 0; rep < 3; ++rep) {
        GWB_CUDA(cudaEventRecord(e0, s));
        k_dmma_probe<<<blocks, threads, 0, s>>>(d, iters);
        GWB_CUDA(cudaEventRecord(e1, s));
        GWB_CUDA(cudaEventSynchronize(e1));
        float ms = 0.f;
        GWB_CUDA(cudaEventElapsedTime(&ms, e0, e1));
        best = std::min(best, ms);
    }
    GWB_LAUNCH("k_dmma_probe");
    GWB_CUDA(cudaFree(d));
    GWB_CUDA(cudaEventDestroy(e0));
    GWB_CUDA(cudaEventDestroy(e1));
    const double flops = 2.0 * (blocks * threads / 32) * (double)iters * 4 * (8 * 8 * 4);
    return flops / (best * 1e-3) / 1e12;
}

} // namespace gwb200
