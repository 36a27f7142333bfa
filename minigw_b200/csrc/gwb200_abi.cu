// gwb200_abi.cu -- the C ABI (include/gwb200.h): handle, resident device state, frequency
// chunking by HBM budget, and the orchestration of the screening kernels.
#include "internal.cuh"

#include <algorithm>
#include <cmath>
#include <cstdlib>
#include <cstring>
#include <functional>
#include <initializer_list>
#include <limits>
#include <map>
#include <mutex>
#include <new>
#include <numeric>
#include <string>
#include <vector>

using namespace gwb200;

namespace {

thread_local std::string g_last_error;

// Device buffer.  Default: grow-only (cudaMalloc).  A handle with a memory limit sizes buffers
// exactly per request with the stream-ordered allocator on its own stream, so a sequence of
// different requests never holds more than one request's footprint and no cudaFree synchronises
// the device under concurrently running handles.
struct DevBuf {
    void* p = nullptr;
    size_t bytes = 0;
    cudaStream_t async_stream = nullptr;  // non-null: allocated stream-ordered on this stream
    void ensure(size_t want) {
        if (want <= bytes) return;
        release();
        GWB_CUDA(cudaMalloc(&p, want));
        bytes = want;
    }
    void ensure_exact(size_t want, cudaStream_t s, cudaMemPool_t pool) {
        if (p && want == bytes) return;
        release();
        if (pool) GWB_CUDA(cudaMallocFromPoolAsync(&p, want, pool, s));
        else GWB_CUDA(cudaMallocAsync(&p, want, s));
        bytes = want;
        async_stream = s;
    }
    void release() {
        if (p) {
            if (async_stream) cudaFreeAsync(p, async_stream);
            else cudaFree(p);
        }
        p = nullptr;
        bytes = 0;
        async_stream = nullptr;
    }
    template <class T>
    T* as() const {
        return static_cast<T*>(p);
    }
};

// Grow-only pinned host buffer: small per-call uploads/downloads go through it, so they are true
// asynchronous DMA (a pageable copy is staged by the driver and, for uploads, waits for the stream).
struct PinnedBuf {
    void* p = nullptr;
    size_t bytes = 0;
    void ensure(size_t want) {
        if (want <= bytes) return;
        release();
        GWB_CUDA(cudaMallocHost(&p, want));
        bytes = want;
    }
    void release() {
        if (p) cudaFreeHost(p);
        p = nullptr;
        bytes = 0;
    }
    template <class T>
    T* as() const {
        return static_cast<T*>(p);
    }
};

// One stream of a batched solve (gwb200_run_g0w0_batch) with its own workspaces; lane 0 runs on
// the lead handle's stream.
struct BatchLane {
    cudaStream_t stream = nullptr;  // lanes >= 1 (created on first use)
    cudaEvent_t done = nullptr;
    DevBuf a, qacc, panel, sched, refine;  // refine: the refined mixed form's correction terms
    size_t bytes() const { return a.bytes + qacc.bytes + panel.bytes + refine.bytes; }
};
constexpr int kMaxBatchLanes = 4;

template <class F>
int guarded(F&& body) {
    try {
        body();
        g_last_error.clear();
        return GWB200_OK;
    } catch (const Failure& e) {
        g_last_error = e.what();
        return e.code;
    } catch (const std::bad_alloc&) {
        g_last_error = "host allocation failed";
        return GWB200_OOM;
    } catch (const std::exception& e) {
        g_last_error = e.what();
        return GWB200_CUDA_ERROR;
    }
}

} // namespace

int gwb200_fail_status(int code, const char* message) {
    g_last_error = message ? message : "";
    return code;
}

struct gwb200_handle {
    int device = 0;
    cudaStream_t stream = nullptr;      // stream all work is issued on
    cudaStream_t own_stream = nullptr;  // the handle's own stream
    SideStream side;                    // work beside `stream`, joined to it before a call's results are read
    cudaEvent_t ev[6] = {};
    // resident system
    bool loaded = false;
    int64_t nmo = 0, nocc = 0, n = 0;
    double fermi = 0.0;
    bool bad_gap = false;
    bool complex_forms = false;  // the last compute_forms ran the eta != 0 (complex) path
    DevBuf pqo, xdiag, mo, vxc_diag, delta, v, sigx;  // pqo: the (pq|o.) block of the ERI
    // per-call workspaces (grow-only, reused across calls)
    DevBuf xt, dvec, a, qacc, qall, omega_out;
    // A call's small inputs and results, one copy each way: `in` holds the pivot word (set by the
    // upload), the grid, the state list (and a batch's group tables), `out` Sigma_c of the requested
    // states [nstates][nfreq] and their QP energies; `call` points into them (a batch member's into
    // its lead handle's).
    DevBuf in, out;
    struct {
        double *omega = nullptr, *weight = nullptr, *sigma = nullptr, *qp = nullptr;
        int64_t* states = nullptr;
    } call;
    unsigned long long* err() const { return in.as<unsigned long long>(); }
    DevBuf panel32;   // operand workspace of the tcgen05 trailing updates (mixed: FP32 hi/lo split;
                      // plain with GWB200_FP64_UPDATE=ozaki: int8 digit slices + exponents)
    DevBuf tc_sched;  // work counter of the tcgen05 update kernel
    // GWB200_MIXED_REFINED: pivoted Cholesky factor of the resident V_ph (computed on first use after
    // a load; pchol_rank < 0: not yet) and the per-chunk refinement workspace
    DevBuf pchol, pchol_sl, refine;  // pchol_sl: the factor's int8 digit slices
    DevBuf sweep;                    // gwb200_pade_sweep: grid, row, points
    DevBuf qx, sigmx;                // gwb200_sigma_c_matrix: cross forms, Sigma_c between the states
    int64_t pchol_rank = -1;
    double* pchol_ct = nullptr;
    BatchLane lanes[kMaxBatchLanes];  // streams + workspaces of the batches this handle leads
    cudaEvent_t batch_fork = nullptr;
    cudaGraphExec_t batch_exec = nullptr;   // the last batch sequence captured as a CUDA graph
    std::vector<int64_t> batch_graph_key;   // what it was captured for (sizes, plan, every pointer)
    std::vector<int64_t> batch_graph_seen;  // the last call's: captured when it comes twice in a row
    std::vector<int64_t> batch_graph_failed;  // a signature whose capture failed (issued eagerly)
    int64_t batch_graph_launches = 0;
    PinnedBuf stage_in, stage_out;
    // cached frequency-chunk size for a repeated geometry (avoids cudaMemGetInfo per call)
    int64_t chunk_key[5] = {-1, -1, -1, -1, -1};
    int64_t mem_limit = 0;          // 0: no cap
    cudaMemPool_t pool = nullptr;   // pool for exact-size buffers (set by a server), else the default
    int64_t chunk_fc = 0;
    int64_t last_update_kernel = -1;  // gwb200_update_kernel
    // gwb200_load_system_states: the state list whose panel rows are resident in xt (empty: the
    // (pq|o.) block is resident in pqo and the panel is gathered per call)
    std::vector<int64_t> bound_states;
    int persistent_ctas = 0;          // > 0: cap of the persistent kernels' grids (GPU shared by slots)
    // GWB200_PROFILE=1: the memory-bound kernels (kKprof* kinds) timed with CUDA events on the
    // handle's stream, resolved and summed when gwb200_kernel_profile reads them
    struct KprofPending {
        int kind;
        double bytes;
        cudaEvent_t start, stop;
    };
    std::vector<KprofPending> kprof_pending;
    double kprof_ms[4] = {}, kprof_bytes[4] = {};
    int64_t kprof_launches[4] = {};
};

void gwb200_attach_pool(gwb200_handle* h, cudaMemPool_t pool) { h->pool = pool; }

namespace {
// Kinds of gwb200_kernel_profile
constexpr int kKprofGatherVph = 0, kKprofGatherPanel = 1, kKprofBuildTall = 2, kKprofContract = 3;

bool kernel_profiling() {
    const char* e = std::getenv("GWB200_PROFILE");
    return e && e[0] == '1';
}

// Runs `launch` (kernels on h->stream); with GWB200_PROFILE=1 brackets it with two events whose
// elapsed time is credited to `kind` with `bytes` of algorithmic traffic when the profile is read
// (no synchronisation here).
template <class F>
int64_t kprof(gwb200_handle* h, int kind, double bytes, F&& launch) {
    if (!kernel_profiling()) return launch();
    cudaStreamCaptureStatus cap = cudaStreamCaptureStatusNone;
    GWB_CUDA(cudaStreamIsCapturing(h->stream, &cap));
    if (cap != cudaStreamCaptureStatusNone) return launch();  // a graph being captured: not timed
    gwb200_handle::KprofPending p{kind, bytes, nullptr, nullptr};
    GWB_CUDA(cudaEventCreate(&p.start));
    GWB_CUDA(cudaEventCreate(&p.stop));
    GWB_CUDA(cudaEventRecord(p.start, h->stream));
    const int64_t n = launch();
    GWB_CUDA(cudaEventRecord(p.stop, h->stream));
    h->kprof_pending.push_back(p);
    return n;
}

void kprof_release(gwb200_handle* h) {
    for (auto& p : h->kprof_pending) {
        cudaEventDestroy(p.start);
        cudaEventDestroy(p.stop);
    }
    h->kprof_pending.clear();
}
} // namespace
void gwb200_share_sms(gwb200_handle* h, int ways) {
    int dev = 0, sms = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess)
        sms = 148;
    h->persistent_ctas = ways > 1 ? std::max(1, sms / ways) : 0;
}

namespace {

// The mixed form's outer trailing updates: GWB200_MIXED_UPDATE=tc / =mma force the tcgen05 or the
// mma.sync kernel (same 3xTF32 arithmetic); by default tcgen05, except on memory-capped handles
// (the serving loop's slots), where the persistent tcgen05 kernel would hold every SM while the
// other slots' requests wait: measured, the non-persistent kernels serve 90.6 requests/s against 60
// (persistent kernels with grids shared between slots) and 41.6 (unshared).
bool mixed_update_on_tcgen05(const gwb200_handle* h) {
    const char* env = std::getenv("GWB200_MIXED_UPDATE");
    if (env && std::strcmp(env, "mma") == 0) return false;
    if (env && std::strcmp(env, "tc") == 0) return true;
    return h->mem_limit <= 0;
}


// Allocate `b` for `want` bytes: grow-only, or exact and stream-ordered when the handle is limited.
void size_buffer(gwb200_handle* h, DevBuf& b, size_t want) {
    if (h->mem_limit > 0) b.ensure_exact(want, h->stream, h->pool);
    else b.ensure(want);
}

void check_handle(gwb200_handle* h) {
    if (!h) fail(GWB200_BAD_ARGUMENT, "null gwb200_handle");
    GWB_CUDA(cudaSetDevice(h->device));
}

void check_system(gwb200_handle* h) {
    check_handle(h);
    if (!h->loaded) fail(GWB200_NO_SYSTEM, "no system loaded: call gwb200_load_system first");
}

void check_states(const gwb200_handle* h, const int64_t* states, int64_t nstates) {
    if (nstates <= 0 || !states) fail(GWB200_BAD_SHAPE, "at least one state is required");
    std::vector<int64_t> seen(states, states + nstates);
    for (int64_t s : seen)
        if (s < 0 || s >= h->nmo) fail(GWB200_BAD_SHAPE, "Selected state is out of range");
    std::sort(seen.begin(), seen.end());
    if (std::adjacent_find(seen.begin(), seen.end()) != seen.end()) fail(GWB200_BAD_SHAPE, "duplicate state in the state list");
}

// The pivoted Cholesky factor of the resident V_ph (and its int8 digit slices), computed on `s` on
// first use after a load (this synchronises `s`).
RefineFactor refine_factor(gwb200_handle* h, cudaStream_t s) {
    if (h->pchol_rank < 0) {
        size_buffer(h, h->pchol, pchol_bytes(h->n));
        const int64_t r = launch_pchol(h->v.as<double>(), h->n, h->pchol.p, &h->pchol_ct, s);
        const int64_t n_pad = round_up(h->n, kNb);
        if (gram_oz_fits(n_pad)) {
            size_buffer(h, h->pchol_sl, gram_oz_system_bytes(n_pad, r));
            launch_slice_ct(h->pchol_ct, r, n_pad, h->pchol_sl.p, s);
        }
        h->pchol_rank = r;
    }
    return RefineFactor{h->pchol_ct, std::max<int64_t>(kNb, round_up(h->pchol_rank, kNb)), h->pchol_sl.p,
                        h->pchol_rank};
}

float elapsed(cudaEvent_t a, cudaEvent_t b) {
    float ms = 0.f;
    GWB_CUDA(cudaEventElapsedTime(&ms, a, b));
    return ms;
}

// Screened quadratic forms for all requested frequencies into h->qall ([nfreq][m] doubles,
// x^T W_c x <= 0).  Records ev[0] (start), ev[1] (after gather), ev[2] (after screening).
// after_factor (plain form only): called on the stream after each frequency chunk [f0, f0 + nf) is
// factored, while h->a holds its tall matrices (the solved right-hand-side rows in their lower block).
using ChunkHook = std::function<void(const TallGeometry& g, int64_t f0, int64_t nf)>;

void compute_forms(gwb200_handle* h, const double* omega, int64_t nfreq, const int64_t* states, int64_t nstates,
                   double eta, int precision, gwb200_stats* st, const double* weight = nullptr,
                   const ChunkHook* after_factor = nullptr) {
    if (!omega) fail(GWB200_BAD_ARGUMENT, "null omega");
    if (nfreq <= 0) fail(GWB200_BAD_SHAPE, "--freq-points must be positive");
    check_states(h, states, nstates);
    if (!std::isfinite(eta)) fail(GWB200_BAD_ARGUMENT, "non-finite eta");
    if (precision != GWB200_FP64 && precision != GWB200_MIXED && precision != GWB200_MIXED_REFINED)
        fail(GWB200_BAD_ARGUMENT, "unknown precision");
    const bool mixed = precision != GWB200_FP64;
    const bool refine = precision == GWB200_MIXED_REFINED;
    if (mixed && eta != 0.0) fail(GWB200_BAD_ARGUMENT, "the mixed-precision form requires eta == 0");
    const bool cplx = eta != 0.0;  // eta != 0: complex symmetric factorisation
    if (!cplx && h->bad_gap)
        fail(GWB200_NONPOSITIVE_GAP, "some e_a - e_i <= 0: chi0(iw) is not negative definite, eps(iw) is not SPD");
    h->complex_forms = cplx;
    const int planes = cplx ? 2 : 1;
    for (int64_t f = 0; f < nfreq; ++f)
        if (!(std::isfinite(omega[f]))) fail(GWB200_BAD_ARGUMENT, "non-finite frequency");

    cudaStream_t s = h->stream;
    const int64_t m = nstates * h->nmo;
    const TallGeometry g = make_geometry(h->n, m);
    int64_t launches = 0;

    const bool bound = !h->bound_states.empty();
    if (bound && !std::equal(states, states + nstates, h->bound_states.begin(), h->bound_states.end()))
        fail(GWB200_BAD_ARGUMENT, "the state list must be the one given to gwb200_load_system_states");
    if (!bound) size_buffer(h, h->xt, sizeof(double) * (size_t)m * h->n);
    size_buffer(h, h->qall, sizeof(double) * planes * (size_t)nfreq * g.m_pad);
    {  // pivot word, grid, weights (optional) and states: one pinned upload
        const size_t nb_om = sizeof(double) * nfreq, nb_st = sizeof(int64_t) * nstates;
        const size_t nb_in = sizeof(unsigned long long) + 2 * nb_om + nb_st;
        h->in.ensure(nb_in);
        h->stage_in.ensure(nb_in);
        char* st_p = h->stage_in.as<char>();
        std::memset(st_p, 0xFF, sizeof(unsigned long long));
        st_p += sizeof(unsigned long long);
        std::memcpy(st_p, omega, nb_om);
        if (weight) std::memcpy(st_p + nb_om, weight, nb_om);
        else std::memset(st_p + nb_om, 0, nb_om);
        std::memcpy(st_p + 2 * nb_om, states, nb_st);
        GWB_CUDA(cudaMemcpyAsync(h->in.p, h->stage_in.p, nb_in, cudaMemcpyHostToDevice, s));
        h->call.omega = h->in.as<double>() + 1;
        h->call.weight = h->call.omega + nfreq;
        h->call.states = reinterpret_cast<int64_t*>(h->call.weight + nfreq);
    }

    // small systems need no tall matrices (unless the solved rows are wanted): one launch, one chunk
    const bool small = !mixed && !cplx && !after_factor && small_system(g);

    // Frequency chunk size from the HBM budget: tall matrices, scale vectors, accumulators, operands.
    const bool mixed_tc = mixed && mixed_update_on_tcgen05(h);
    // plain form: the int8 emulation of the outer updates is a candidate of the update autotuner
    // (its slice workspace is part of the budget) unless GWB200_FP64_UPDATE=dmma; memory-capped
    // handles use it only when it is forced (GWB200_FP64_UPDATE=ozaki)
    const bool fp64_oz = !mixed && !cplx && !small && fp64_update_mode() != 1 && (h->mem_limit <= 0 || fp64_update_mode() == 2);
    // refined mixed form: V_ph = C C^T once per loaded system (its rank sizes the correction's work)
    int64_t r_pad = 0;
    RefineFactor fac{};
    if (refine) {
        fac = refine_factor(h, s);
        r_pad = fac.r_pad;
    }
    const size_t per_freq = mixed ? sizeof(float) * (size_t)g.stride + sizeof(double) * (g.n_pad + g.m_pad) +
                                        (mixed_tc ? tc_panel_bytes_per_freq(g) : 0) +
                                        (refine ? refine_bytes_per_freq(g, r_pad) : 0)
                                  : sizeof(double) * planes * ((size_t)g.stride + g.n_pad + g.m_pad) +
                                        (fp64_oz ? oz_slice_bytes_per_freq(g) : 0);
    // GWB200_MAX_FREQ_CHUNK caps the chunk (tests use it to exercise the multi-chunk path).
    int64_t cap = 0;
    if (const char* env = std::getenv("GWB200_MAX_FREQ_CHUNK")) cap = std::max<long long>(0, std::atoll(env));
    const int64_t key[5] = {(int64_t)per_freq, nfreq, cap, (int64_t)g.stride, h->mem_limit};
    int64_t fc;
    if (small) {
        fc = cap > 0 ? std::min<int64_t>(nfreq, cap) : nfreq;
    } else if (std::equal(key, key + 5, h->chunk_key)) {
        fc = h->chunk_fc;  // same geometry as the last call: its buffers are already sized
    } else {
        size_t free_b = 0, total_b = 0;
        GWB_CUDA(cudaMemGetInfo(&free_b, &total_b));
        const size_t have =
            h->a.bytes + h->dvec.bytes + h->qacc.bytes + h->panel32.bytes + h->refine.bytes;
        size_t avail = free_b + have;  // what the chunk buffers may occupy
        size_t budget = (size_t)((double)avail * 0.85);
        if (h->mem_limit > 0) {  // the handle's cap minus what the system and panels already hold
            const size_t resident = h->pqo.bytes + h->xdiag.bytes + h->v.bytes + h->xt.bytes + h->qall.bytes +
                                    h->in.bytes + h->out.bytes + h->pchol.bytes + h->pchol_sl.bytes +
                                    h->qx.bytes + h->sigmx.bytes + ((size_t)1 << 20);
            const size_t lim = (size_t)h->mem_limit;
            const size_t room = lim > resident ? lim - resident : 0;
            budget = std::min(budget, room);
            avail = std::min(avail, room);
        }
        fc = (int64_t)std::min<size_t>((size_t)nfreq, std::max<size_t>(1, budget / per_freq));
        if (cap > 0) fc = std::min<int64_t>(fc, cap);
        if ((size_t)fc * per_freq > avail) fail(GWB200_OOM, "not enough device memory for one frequency of eps(iw)");
        std::copy(key, key + 5, h->chunk_key);
        h->chunk_fc = fc;
    }
    if (!small) {
        size_buffer(h, h->a, (mixed ? sizeof(float) : sizeof(double) * planes) * (size_t)fc * g.stride);
        size_buffer(h, h->dvec, sizeof(double) * planes * (size_t)fc * g.n_pad);
        size_buffer(h, h->qacc, sizeof(double) * planes * (size_t)fc * g.m_pad);
    }
    if (mixed_tc) {
        size_buffer(h, h->panel32, tc_panel_bytes_per_freq(g) * (size_t)fc);
        h->tc_sched.ensure(sched_bytes(g));
    }
    if (fp64_oz) {
        size_buffer(h, h->panel32, oz_slice_bytes_per_freq(g) * (size_t)fc);
        h->tc_sched.ensure(sched_bytes(g));
    }
    if (refine) size_buffer(h, h->refine, refine_bytes_per_freq(g, r_pad) * (size_t)fc);

    GWB_CUDA(cudaEventRecord(h->ev[0], s));
    if (!bound)
        launches += kprof(h, kKprofGatherPanel, 16.0 * (double)m * (double)h->n, [&] {
            return (int64_t)launch_gather_panel(h->pqo.as<double>(), h->nmo, h->nocc, h->call.states, nstates,
                                                h->xt.as<double>(), s);
        });
    GWB_CUDA(cudaEventRecord(h->ev[1], s));
    // algorithmic bytes of one build launch: V_ph and the panel rows read once, the lower triangle of
    // eps and the right-hand-side rows of every frequency written (el bytes per element)
    auto build_bytes = [&](int64_t nf, double el) {
        const double np = (double)g.n_pad, mp = (double)g.m_pad;
        return 8.0 * ((double)g.n * (double)g.n + (double)g.n * (double)m) + el * (double)nf * (np * (np + 1.0) / 2.0 + mp * np);
    };
    const char* prof_env = std::getenv("GWB200_PROFILE");
    UpdateProfiler prof(prof_env && prof_env[0] == '1', s);
    int64_t chunks = 0;
    // a capped handle's share of the GPU is taken by its own kernels
    SideStream* side = h->persistent_ctas == 0 ? &h->side : nullptr;
    int upd_variant = -1;  // FP64 update kernel, tuned on the first chunk (full size) of this geometry
    for (int64_t f0 = 0; f0 < nfreq; f0 += fc) {
        const int64_t nf = std::min(fc, nfreq - f0);
        if (small) {
            launches += launch_small64(g, nf, h->delta.as<double>(), h->call.omega + f0, h->v.as<double>(),
                                       h->xt.as<double>(), h->qall.as<double>() + f0 * g.m_pad, g.m_pad,
                                       h->err(), s);
            ++chunks;
            continue;
        }
        if (cplx) {
            double* a_re = h->a.as<double>();
            launches += launch_factor_chunk_c(g, nf, h->delta.as<double>(), h->call.omega + f0, eta,
                                              h->v.as<double>(), h->xt.as<double>(), a_re, a_re + (size_t)nf * g.stride,
                                              h->dvec.as<double>(), h->qacc.as<double>(),
                                              h->err(), s, side);
            launches += launch_forms_out_c(h->qacc.as<double>(), nf, m, g.m_pad,
                                           h->qall.as<double>() + f0 * 2 * g.m_pad, g.m_pad, s);
            ++chunks;
            continue;
        }
        launches += launch_scale_vectors(h->delta.as<double>(), g.n, g.n_pad, h->call.omega + f0, nf,
                                         h->dvec.as<double>(), s);
        GWB_CUDA(cudaMemsetAsync(h->qacc.p, 0, sizeof(double) * (size_t)nf * g.m_pad, s));
        if (mixed) {
            launches += kprof(h, kKprofBuildTall, build_bytes(nf, 4.0), [&] {
                return (int64_t)launch_build_tall32(g, h->v.as<double>(), h->xt.as<double>(), h->dvec.as<double>(), nf,
                                                    h->a.as<float>(), s);
            });
            launches += launch_factor_chunk32(g, nf, h->a.as<float>(), h->qacc.as<double>(),
                                              h->err(), s, prof.enabled ? &prof : nullptr,
                                              mixed_tc ? h->panel32.as<float>() : nullptr,
                                              h->tc_sched.as<unsigned long long>(), h->persistent_ctas,
                                              /*keep_rows=*/refine, /*solve_only=*/false, side);
            if (refine)  // qacc <- 2 x^T y - z^T z - y^T V y (FP64 energy functional at the FP32 solve)
                launches += launch_refine_chunk(g, nf, h->a.as<float>(), h->xt.as<double>(),
                                                h->dvec.as<double>(), fac, h->refine.p,
                                                h->qacc.as<double>(), h->err(), s,
                                                mixed_tc ? h->panel32.as<float>() : nullptr,
                                                h->tc_sched.as<unsigned long long>(), h->persistent_ctas);
        } else {
            if (upd_variant < 0)
                upd_variant = tune_update_variant(g, nf, h->a.as<double>(), s, fp64_oz ? h->panel32.p : nullptr,
                                                  h->tc_sched.as<unsigned long long>(), h->err(),
                                                  /*timed=*/h->mem_limit <= 0);
            launches += kprof(h, kKprofBuildTall, build_bytes(nf, 8.0), [&] {
                return (int64_t)launch_build_tall(g, h->v.as<double>(), h->xt.as<double>(), h->dvec.as<double>(), nf,
                                                  h->a.as<double>(), s);
            });
            launches += launch_factor_chunk(g, nf, h->a.as<double>(), h->qacc.as<double>(),
                                            h->err(), s, prof.enabled ? &prof : nullptr,
                                            upd_variant, fp64_oz ? h->panel32.p : nullptr,
                                            h->tc_sched.as<unsigned long long>(), h->persistent_ctas,
                                            side);
            if (after_factor) {
                (*after_factor)(g, f0, nf);
                ++launches;
            }
        }
        launches += launch_negate_copy(h->qacc.as<double>(), nf, m, g.m_pad, h->qall.as<double>() + f0 * g.m_pad,
                                       g.m_pad, s);
        ++chunks;
    }
    GWB_CUDA(cudaEventRecord(h->ev[2], s));
    h->last_update_kernel = -1;
    if (g.n_pad / kNb > 2 && !cplx) h->last_update_kernel = mixed ? (mixed_tc ? 7 : 8) : upd_variant;
    if (st) {
        const double nd = (double)g.n, md = (double)m;
        st->flops_screening = (double)nfreq * (nd * nd * nd / 3.0 + nd * nd * md + 3.0 * nd * md);
        st->frequency_chunks = chunks;
        st->kernel_launches = launches;
        st->nph = g.n;
        st->ncols = m;
    }
    if (prof.enabled && st) prof.collect(st);
}

// Reads the pivot word and `nb` bytes of results at `src` back (one synchronisation; the results at
// result_stage(h) afterwards) and reports a failed factorisation.
char* result_stage(gwb200_handle* h) { return h->stage_out.as<char>() + sizeof(unsigned long long); }

struct Readback {
    const void* src;
    size_t bytes;
};

void finish_forms(gwb200_handle* h, gwb200_stats* st, std::initializer_list<Readback> results = {}) {
    size_t nb = sizeof(unsigned long long);
    for (const Readback& r : results) nb += r.bytes;
    h->stage_out.ensure(nb);
    GWB_CUDA(cudaMemcpyAsync(h->stage_out.p, h->in.p, sizeof(unsigned long long), cudaMemcpyDeviceToHost, h->stream));
    char* o = result_stage(h);
    for (const Readback& r : results) {
        GWB_CUDA(cudaMemcpyAsync(o, r.src, r.bytes, cudaMemcpyDeviceToHost, h->stream));
        o += r.bytes;
    }
    GWB_CUDA(cudaStreamSynchronize(h->stream));
    const unsigned long long piv = *h->stage_out.as<unsigned long long>();
    if (piv == 0)  // a bounded device wait expired (pivots are 1-based)
        fail(GWB200_DEVICE_TIMEOUT, "a device-side wait of the tcgen05 update expired; results discarded");
    if (piv != std::numeric_limits<unsigned long long>::max()) {
        if (st) st->info = (int64_t)piv;
        fail(GWB200_NOT_SPD, "eps(iw) is not positive definite: Cholesky pivot " + std::to_string(piv) + " <= 0");
    }
    if (st) {
        st->device_ms_gather = elapsed(h->ev[0], h->ev[1]);
        st->device_ms_screening = elapsed(h->ev[1], h->ev[2]);
    }
}

// Sigma_c of the requested states ([nstates][nf] complex at `rows`) into the caller's nmo x nf array,
// zero elsewhere.
void scatter_sigma(const gwb200_handle* h, const char* rows, const int64_t* states, int64_t nstates, int64_t nf,
                   double* sigma_out) {
    const size_t nb_row = sizeof(double) * 2 * (size_t)nf;
    std::memset(sigma_out, 0, nb_row * (size_t)h->nmo);
    for (int64_t i = 0; i < nstates; ++i) std::memcpy(sigma_out + 2 * (size_t)(states[i] * nf), rows + (size_t)i * nb_row, nb_row);
}
void scatter_qp(const gwb200_handle* h, const char* rows, const int64_t* states, int64_t nstates, double* qp_out) {
    std::fill(qp_out, qp_out + h->nmo, std::numeric_limits<double>::quiet_NaN());
    for (int64_t i = 0; i < nstates; ++i) std::memcpy(qp_out + states[i], rows + sizeof(double) * (size_t)i, sizeof(double));
}
// Sizes `out` for nstates x nf results and points `call` at them.
void size_results(gwb200_handle* h, int64_t nstates, int64_t nf) {
    h->out.ensure(sizeof(double) * (size_t)nstates * (2 * (size_t)nf + 1));
    h->call.sigma = h->out.as<double>();
    h->call.qp = h->call.sigma + 2 * (size_t)nstates * nf;
}

// G0-weighted frequency contraction of h->qall (the nf_int frequencies compute_forms solved, with
// the weights it uploaded) into h->call.sigma ([nstates][nf_out] complex).
// omega_out_dev = NULL: the output grid is the integration grid.  Records ev[3].
void contract_on_device(gwb200_handle* h, int64_t nf_int, int64_t nstates, gwb200_stats* st,
                        const double* omega_out_dev = nullptr, int64_t nf_out = -1) {
    cudaStream_t s = h->stream;
    const int64_t m = nstates * h->nmo;
    const int64_t ldq = make_geometry(h->n, m).m_pad;
    if (!omega_out_dev) {
        omega_out_dev = h->call.omega;
        nf_out = nf_int;
    }
    const size_t sig_bytes = sizeof(double) * 2 * (size_t)h->nmo * nf_out;  // as the caller gets it
    if (h->complex_forms)
        st->kernel_launches += launch_sigma_contract_c(h->qall.as<double>(), nf_int, nstates, h->nmo, ldq,
                                                       h->mo.as<double>(), h->fermi, h->call.omega, h->call.weight, omega_out_dev,
                                                       nf_out, h->call.sigma, s);
    else  // algorithmic bytes: the forms read once, Sigma_c written once
        st->kernel_launches += kprof(h, kKprofContract, 8.0 * (double)nf_int * (double)m + (double)sig_bytes, [&] {
            return (int64_t)launch_sigma_contract(h->qall.as<double>(), nf_int, nstates, h->nmo, ldq,
                                                  h->mo.as<double>(), h->fermi, h->call.omega, h->call.weight, omega_out_dev, nf_out,
                                                  h->call.sigma, s);
        });
    GWB_CUDA(cudaEventRecord(h->ev[3], s));
}

// Pade + QP fixed point of the requested states on h->call's Sigma_c rows into h->call.qp.
void qp_on_device(gwb200_handle* h, int64_t nfreq, int64_t npade, int64_t nstates) {
    cudaStream_t s = h->stream;
    launch_qp(h->call.sigma, h->call.omega, nfreq, h->call.states, nstates, npade, h->mo.as<double>(), h->fermi,
              h->sigx.as<double>(), h->vxc_diag.as<double>(), h->call.qp, s);
}

// ---- many molecules in shared launches (gwb200_run_g0w0_batch; kernels in kernels_batch.cu) ----

// Batch work runs on the lead handle's stream; the members' own streams come back on exit.
struct StreamSwap {
    std::vector<gwb200_handle*> hs;
    std::vector<cudaStream_t> saved;
    ~StreamSwap() {
        for (size_t i = 0; i < hs.size(); ++i) hs[i]->stream = saved[i];
    }
};

// One launch sequence of a bucket: `nmat` matrices of geometry g, described by groups
// [group0, group0 + ngroups) of the device table.
struct BatchChunk {
    TallGeometry g;
    int64_t nmat, group0, ngroups;
};

// Chunks of one bucket plan (bucket sizes over `order`, the molecules sorted by size), at most
// `budget` bytes (and, if cap > 0, cap matrices) at once; appends the groups (device pointers of
// each member).
std::vector<BatchChunk> batch_chunks(const std::vector<gwb200_handle*>& hs, const std::vector<int64_t>& ms,
                                     const std::vector<int64_t>& fs, const std::vector<int>& order,
                                     const std::vector<int64_t>& sizes, bool mixed, bool oz, bool refine, size_t budget,
                                     int64_t cap, std::vector<BatchGroup>& groups) {
    std::vector<BatchChunk> chunks;
    size_t pos = 0;
    for (int64_t bsz : sizes) {
        int64_t nmax = 0, mmax = 0;
        for (int64_t t = 0; t < bsz; ++t) {
            const int i = order[pos + (size_t)t];
            nmax = std::max(nmax, hs[(size_t)i]->n);
            mmax = std::max(mmax, ms[(size_t)i]);
        }
        const TallGeometry g = make_geometry(nmax, mmax);
        int64_t fit = std::max<int64_t>(1, (int64_t)(budget / batch_bytes_per_matrix(g, mixed, oz, refine)));
        if (cap > 0) fit = std::min(fit, cap);
        BatchChunk cur{g, 0, (int64_t)groups.size(), 0};
        for (int64_t t = 0; t < bsz; ++t) {
            const int i = order[pos + (size_t)t];
            gwb200_handle* h = hs[(size_t)i];
            const TallGeometry gi = make_geometry(h->n, ms[(size_t)i]);
            const int64_t nfreq = fs[(size_t)i];
            for (int64_t f0 = 0; f0 < nfreq;) {
                if (cur.nmat == fit) {
                    chunks.push_back(cur);
                    cur = BatchChunk{g, 0, (int64_t)groups.size(), 0};
                }
                const int64_t nf = std::min(nfreq - f0, fit - cur.nmat);
                BatchGroup gr{};
                gr.v = h->v.as<double>();
                gr.xt = h->xt.as<double>();
                gr.dvec = h->dvec.as<double>() + f0 * gi.n_pad;
                gr.q_out = h->qall.as<double>() + f0 * gi.m_pad;
                gr.n = h->n;
                gr.m = ms[(size_t)i];
                gr.n_pad = gi.n_pad;
                gr.ldq_out = gi.m_pad;
                gr.mat0 = cur.nmat;
                gr.nf = nf;
                if (refine)
                    gr.fac = RefineFactor{h->pchol_ct, std::max<int64_t>(kNb, round_up(h->pchol_rank, kNb)),
                                          h->pchol_sl.p, h->pchol_rank};
                groups.push_back(gr);
                ++cur.ngroups;
                cur.nmat += nf;
                f0 += nf;
            }
        }
        if (cur.nmat > 0) chunks.push_back(cur);
        pos += (size_t)bsz;
    }
    return chunks;
}

// Workspace bytes of a set of chunks: the largest tall matrices, accumulators, operands, counters.
struct BatchNeed {
    size_t a = 0, qacc = 0, panel = 0, sched = 0, refine = 0;
    size_t total() const { return a + qacc + panel + refine; }
};
void batch_need(const std::vector<BatchChunk>& chunks, bool mixed, bool oz, bool refine, BatchNeed& need) {
    const size_t el = mixed ? sizeof(float) : sizeof(double);
    for (const BatchChunk& c : chunks) {
        const size_t nm = (size_t)c.nmat;
        need.a = std::max(need.a, el * nm * (size_t)c.g.stride);
        need.sched = std::max(need.sched, sched_bytes(c.g));
        need.qacc = std::max(need.qacc, sizeof(double) * nm * (size_t)c.g.m_pad);
        const size_t op = mixed ? tc_panel_bytes_per_freq(c.g) : (oz ? oz_slice_bytes_per_freq(c.g) : 0);
        need.panel = std::max(need.panel, op * nm);
        // the correction terms of one molecule at a time, bounded by the chunk's geometry
        if (refine) need.refine = std::max(need.refine, refine_bytes_per_freq(c.g, c.g.n_pad) * nm);
    }
}

// The chunks `idx` of a plan on one lane (build, factor, forms per chunk), on stream `s`.
int64_t batch_screen(gwb200_handle* w, BatchLane& lane, cudaStream_t s, int max_ctas,
                     const std::vector<BatchChunk>& chunks, const std::vector<size_t>& idx, const BatchGroup* dgroups,
                     const std::vector<BatchGroup>& hgroups, const std::vector<int>& variants, bool mixed,
                     bool mixed_tc, bool oz, bool refine) {
    int64_t launches = 0;
    unsigned long long* err = w->err();
    unsigned long long* sched = lane.sched.as<unsigned long long>();
    for (size_t k : idx) {
        const BatchChunk& c = chunks[k];
        const BatchGroup* gp = dgroups + c.group0;
        GWB_CUDA(cudaMemsetAsync(lane.qacc.p, 0, sizeof(double) * (size_t)c.nmat * c.g.m_pad, s));
        launches += launch_build_tall_batch(c.g, gp, c.ngroups, mixed, lane.a.p, s);
        if (mixed) {
            launches += launch_factor_chunk32(c.g, c.nmat, lane.a.as<float>(), lane.qacc.as<double>(), err, s,
                                              nullptr, mixed_tc ? lane.panel.as<float>() : nullptr, sched, max_ctas,
                                              /*keep_rows=*/refine);
            if (refine) {  // each molecule's factor reversed in its own n_pad, one backward solve of the
                           // chunk, then each molecule's correction in its own geometry
                for (int64_t q = 0; q < c.ngroups; ++q) {
                    const BatchGroup& gr = hgroups[(size_t)(c.group0 + q)];
                    launches += launch_refine_flip(c.g, gr.nf, lane.a.as<float>() + (size_t)gr.mat0 * c.g.stride,
                                                   gr.n_pad, s);
                }
                launches += launch_refine_solve(c.g, c.nmat, lane.a.as<float>(), err, s,
                                                mixed_tc ? lane.panel.as<float>() : nullptr, sched, max_ctas,
                                                /*flip=*/false);
                for (int64_t q = 0; q < c.ngroups; ++q) {
                    const BatchGroup& gr = hgroups[(size_t)(c.group0 + q)];
                    launches += launch_refine_terms(c.g, gr.nf, lane.a.as<float>() + (size_t)gr.mat0 * c.g.stride,
                                                    make_geometry(gr.n, gr.m), gr.xt, gr.dvec, gr.fac,
                                                    lane.refine.p, lane.qacc.as<double>() + (size_t)gr.mat0 * c.g.m_pad,
                                                    c.g.m_pad, err, s);
                }
            }
        } else
            launches += launch_factor_chunk(c.g, c.nmat, lane.a.as<double>(), lane.qacc.as<double>(), err, s, nullptr, variants[k],
                                            oz ? lane.panel.p : nullptr, sched, max_ctas);
        launches += launch_forms_scatter(gp, c.ngroups, lane.qacc.as<double>(), c.g.m_pad, s);
    }
    return launches;
}

// Chunks to lanes: longest modelled time first, each to the least loaded lane.
std::vector<std::vector<size_t>> batch_assign(const std::vector<BatchChunk>& chunks, int lanes, double step_us,
                                              double tflops) {
    std::vector<std::pair<double, size_t>> cost;
    for (size_t k = 0; k < chunks.size(); ++k) {
        const double N = (double)chunks[k].g.n_pad, M = (double)chunks[k].g.m_pad;
        cost.push_back({(N / kNb) * step_us * 1e-6 + (double)chunks[k].nmat * (N * N * N / 3.0 + N * N * M) / (tflops * 1e12),
                        k});
    }
    std::stable_sort(cost.begin(), cost.end(), [](const auto& x, const auto& y) { return x.first > y.first; });
    std::vector<std::vector<size_t>> out((size_t)lanes);
    std::vector<double> load((size_t)lanes, 0.0);
    for (const auto& [c, k] : cost) {
        const size_t l = (size_t)(std::min_element(load.begin(), load.end()) - load.begin());
        out[l].push_back(k);
        load[l] += c;
    }
    for (auto& v : out) std::sort(v.begin(), v.end());
    return out;
}

// Latency of one 64-wide block step, as far as the other lanes leave it bare, and the sustained rate of
// the padded work, the cost model's defaults (GWB200_BATCH_STEP_US / GWB200_BATCH_TFLOPS override).
// Measured on 16 molecules of 20 to 120 orbitals x 64 frequencies on 4 lanes, refined mixed form: 22.6
// ms at 8-15 us, 23.9 at 30, 25.4 at 60, 30.7 at 240 (one bucket per molecule 22.2); plain form, 16 to
// 96 orbitals: 9.7 ms at 8-15 us, 11.1 at 30, 12.2 at 80.  64 molecules of 20 to 160 orbitals, at 12 / 30 /
// 60 / 80 us: mixed 163 / 166 / 168 / 171 ms, plain 296 / 300 / 305 / 304, refined 260 / 265 / 265 / 271.
double batch_step_us() {
    if (const char* e = std::getenv("GWB200_BATCH_STEP_US")) return std::max(0.0, std::atof(e));
    return 12.0;
}
double batch_tflops(bool mixed) {
    if (const char* e = std::getenv("GWB200_BATCH_TFLOPS")) return std::max(1e-3, std::atof(e));
    return mixed ? 90.0 : 40.0;
}

std::mutex g_batch_mu;
std::map<std::vector<int64_t>, std::vector<int64_t>> g_batch_plans;  // batch signature -> bucket sizes

} // namespace

extern "C" {

const char* gwb200_last_error(void) { return g_last_error.c_str(); }

const char* gwb200_version(void) { return "gwb200 1.0 sm_100a fp64-dmma"; }

int gwb200_create(int device, gwb200_handle** out) {
    return guarded([&] {
        if (!out) fail(GWB200_BAD_ARGUMENT, "null output handle pointer");
        *out = nullptr;
        int count = 0;
        const cudaError_t e = cudaGetDeviceCount(&count);
        if (e != cudaSuccess || count == 0)
            fail(GWB200_CUDA_ERROR, std::string("no CUDA device available: ") + cudaGetErrorString(e));
        if (device < 0 || device >= count) fail(GWB200_BAD_ARGUMENT, "device index out of range");
        int major = 0;
        GWB_CUDA(cudaDeviceGetAttribute(&major, cudaDevAttrComputeCapabilityMajor, device));
        if (major != 10) fail(GWB200_CUDA_ERROR, "libgwb200 is built for sm_100a (B200); device has compute capability " +
                                                    std::to_string(major) + ".x");
        GWB_CUDA(cudaSetDevice(device));
        auto* h = new gwb200_handle();
        h->device = device;
        try {
            GWB_CUDA(cudaStreamCreateWithFlags(&h->own_stream, cudaStreamNonBlocking));
            h->stream = h->own_stream;
            for (auto& e2 : h->ev) GWB_CUDA(cudaEventCreate(&e2));
        } catch (...) {
            gwb200_destroy(h);
            throw;
        }
        *out = h;
    });
}

int gwb200_destroy(gwb200_handle* h) {
    if (!h) return GWB200_OK;
    cudaSetDevice(h->device);
    if (h->stream) cudaStreamSynchronize(h->stream);
    h->stage_in.release();
    h->stage_out.release();
    for (DevBuf* b : {&h->pchol, &h->pchol_sl, &h->refine, &h->pqo, &h->xdiag, &h->mo, &h->vxc_diag, &h->delta, &h->v, &h->sigx, &h->xt, &h->dvec, &h->a,
                      &h->qacc, &h->qall, &h->in, &h->out, &h->sweep, &h->omega_out, &h->panel32, &h->tc_sched, &h->qx,
                      &h->sigmx})
        b->release();
    for (BatchLane& l : h->lanes) {
        if (l.stream) cudaStreamSynchronize(l.stream);
        for (DevBuf* b : {&l.a, &l.qacc, &l.panel, &l.sched, &l.refine}) b->release();
        if (l.done) cudaEventDestroy(l.done);
        if (l.stream) cudaStreamDestroy(l.stream);
    }
    kprof_release(h);
    if (h->batch_fork) cudaEventDestroy(h->batch_fork);
    if (h->batch_exec) cudaGraphExecDestroy(h->batch_exec);
    for (auto& e : h->ev)
        if (e) cudaEventDestroy(e);
    h->side.destroy();
    if (h->own_stream) cudaStreamDestroy(h->own_stream);
    delete h;
    return GWB200_OK;
}

int gwb200_set_memory_limit(gwb200_handle* h, int64_t bytes) {
    return guarded([&] {
        check_handle(h);
        if (bytes < 0) fail(GWB200_BAD_ARGUMENT, "negative memory limit");
        h->mem_limit = bytes;
    });
}

int gwb200_set_stream(gwb200_handle* h, void* stream) {
    return guarded([&] {
        check_handle(h);
        GWB_CUDA(cudaStreamSynchronize(h->stream));
        h->stream = stream ? static_cast<cudaStream_t>(stream) : h->own_stream;
    });
}

namespace {
// Shared body of gwb200_load_system (states == NULL: the (pq|o.) block stays resident and panels
// are gathered per call) and gwb200_load_system_states (V_ph and the panel rows of `states` copied
// from the host straight into their device layouts; nothing else of the ERI is uploaded).
// Caller-sliced inputs of gwb200_load_system_slices (host memory, contiguous, row-major).
struct HostSlices {
    const double* vph;       // n x n
    const double* panel;     // nstates*nmo x n
    const double* xdiag;     // nmo x nocc: (p i|p i)
    const double* vxc_diag;  // nmo
};

void load_system_impl(gwb200_handle* h, int64_t nmo, int64_t nocc, const double* mo_energy, const double* eri,
                      const double* vxc, double fermi_energy, const int64_t* states, int64_t nstates,
                      const HostSlices* sl = nullptr) {
    check_handle(h);
    if (sl) {
        if (!mo_energy || !sl->vph || !sl->panel || !sl->xdiag || !sl->vxc_diag)
            fail(GWB200_BAD_ARGUMENT, "null input array");
        if (!states) fail(GWB200_BAD_ARGUMENT, "null state list");
    } else if (!mo_energy || !eri || !vxc) {
        fail(GWB200_BAD_ARGUMENT, "null input array");
    }
    if (nmo <= 0) fail(GWB200_BAD_SHAPE, "OrbitalSpace: empty MO energy vector");
    if (nocc <= 0 || nocc >= nmo) fail(GWB200_BAD_SHAPE, "OrbitalSpace: invalid number of occupied orbitals");
    if (nmo > 1024) fail(GWB200_BAD_SHAPE, "nmo > 1024 is not supported");
    const bool bound = states != nullptr;
    if (bound) {
        if (nstates <= 0) fail(GWB200_BAD_SHAPE, "at least one state is required");
        std::vector<int64_t> seen(states, states + nstates);
        for (int64_t st : seen)
            if (st < 0 || st >= nmo) fail(GWB200_BAD_SHAPE, "Selected state is out of range");
        std::sort(seen.begin(), seen.end());
        if (std::adjacent_find(seen.begin(), seen.end()) != seen.end())
            fail(GWB200_BAD_SHAPE, "duplicate state in the state list");
    }
    cudaStream_t s = h->stream;
    h->loaded = false;
    h->bound_states.clear();
    h->pchol_rank = -1;  // the factor of the previous system's V_ph is stale
    h->pchol_ct = nullptr;
    const size_t nmo2 = (size_t)nmo * nmo;
    const int64_t nvir = nmo - nocc, n = nocc * nvir;
    if (h->mem_limit > 0)  // drop the previous request's workspaces before sizing this system
        for (DevBuf* b : {&h->xt, &h->dvec, &h->a, &h->qacc, &h->qall, &h->panel32, &h->pchol, &h->pchol_sl,
                          &h->refine, &h->qx, &h->sigmx})
            b->release();
    if (bound) {
        h->pqo.release();
        size_buffer(h, h->xt, sizeof(double) * (size_t)nstates * nmo * n);
    } else {
        size_buffer(h, h->pqo, sizeof(double) * nmo2 * nocc * nmo);
    }
    size_buffer(h, h->xdiag, sizeof(double) * nmo * nocc);
    h->mo.ensure(sizeof(double) * nmo);
    h->vxc_diag.ensure(sizeof(double) * nmo);
    h->sigx.ensure(sizeof(double) * nmo);
    h->delta.ensure(sizeof(double) * n);
    size_buffer(h, h->v, sizeof(double) * (size_t)n * n);
    // the small arrays through the pinned buffer: orbital energies, the vxc diagonal and the exchange
    // diagonal eri[p,i,p,i], whose nocc elements per p lie nmo^2 + 1 apart (as copies of single
    // elements, one call per p, they took longer than the rest of the upload)
    h->stage_in.ensure(sizeof(double) * (size_t)(2 * nmo + nmo * nocc));
    double* hmo = h->stage_in.as<double>();
    double* hvxc = hmo + nmo;
    double* hxd = hvxc + nmo;
    std::memcpy(hmo, mo_energy, sizeof(double) * nmo);
    for (int64_t p = 0; p < nmo; ++p) hvxc[p] = sl ? sl->vxc_diag[p] : vxc[p * nmo + p];
    if (sl) {
        std::memcpy(hxd, sl->xdiag, sizeof(double) * nmo * nocc);
    } else {
        for (int64_t p = 0; p < nmo; ++p)
            for (int64_t i = 0; i < nocc; ++i) hxd[p * nocc + i] = eri[((size_t)(p * nmo + i) * nmo + p) * nmo + i];
    }
    GWB_CUDA(cudaMemcpyAsync(h->mo.p, hmo, sizeof(double) * nmo, cudaMemcpyHostToDevice, s));
    GWB_CUDA(cudaMemcpyAsync(h->vxc_diag.p, hvxc, sizeof(double) * nmo, cudaMemcpyHostToDevice, s));
    GWB_CUDA(cudaMemcpyAsync(h->xdiag.p, hxd, sizeof(double) * nmo * nocc, cudaMemcpyHostToDevice, s));
    // some e_a - e_i not > 0 (NaN included): the smallest virtual against the largest occupied energy
    bool bad = false;
    double top = -std::numeric_limits<double>::infinity(), bottom = std::numeric_limits<double>::infinity();
    for (int64_t p = 0; p < nmo; ++p) {
        if (std::isnan(mo_energy[p])) bad = true;
        if (p < nocc) top = std::max(top, mo_energy[p]);
        else bottom = std::min(bottom, mo_energy[p]);
    }
    bad = bad || !(bottom - top > 0.0);
    if (sl) {  // already in the device layouts: contiguous copies
        GWB_CUDA(cudaMemcpyAsync(h->v.p, sl->vph, sizeof(double) * (size_t)n * n, cudaMemcpyHostToDevice, s));
        GWB_CUDA(cudaMemcpyAsync(h->xt.p, sl->panel, sizeof(double) * (size_t)nstates * nmo * n, cudaMemcpyHostToDevice,
                                 s));
    } else if (bound) {
        // One 3D copy per source block eri[p, ., ., .] (an nmo x nmo x nmo array of rows of nmo
        // doubles): x = the virtual index s (nvir doubles from nocc), y = the occupied index
        // r < nocc, z = q.  The destination rows are the n = nocc * nvir columns (i, a) of
        //   V[j nvir + b, i nvir + a] = eri[j, nocc + b, i, nocc + a]   (p = j < nocc, z = b)
        //   Xt[t nmo + k, i nvir + a]  = eri[states[t], k, i, nocc + a]   (p = states[t], z = k),
        // the layouts k_gather_vph / k_gather_panel produce from the (pq|o.) block.
        auto copy_block = [&](int64_t p, int64_t q0, int64_t depth, double* dst) {
            cudaMemcpy3DParms c{};
            c.srcPtr = make_cudaPitchedPtr(const_cast<double*>(eri + (size_t)p * nmo2 * nmo), sizeof(double) * nmo,
                                           sizeof(double) * nmo, (size_t)nmo);
            c.srcPos = make_cudaPos(sizeof(double) * nocc, 0, (size_t)q0);
            c.dstPtr = make_cudaPitchedPtr(dst, sizeof(double) * nvir, sizeof(double) * nvir, (size_t)nocc);
            c.dstPos = make_cudaPos(0, 0, 0);
            c.extent = make_cudaExtent(sizeof(double) * nvir, (size_t)nocc, (size_t)depth);
            c.kind = cudaMemcpyHostToDevice;
            GWB_CUDA(cudaMemcpy3DAsync(&c, s));
        };
        for (int64_t j = 0; j < nocc; ++j) copy_block(j, nocc, nvir, h->v.as<double>() + (size_t)j * nvir * n);
        for (int64_t t = 0; t < nstates; ++t) copy_block(states[t], 0, nmo, h->xt.as<double>() + (size_t)t * nmo * n);
    } else {
        // Only the (pq|o.) block is uploaded: every V_ph / panel element has an occupied third
        // index.  One 2D copy: nmo^2 rows of nocc*nmo contiguous doubles, source pitch nmo^2.
        GWB_CUDA(cudaMemcpy2DAsync(h->pqo.p, sizeof(double) * nocc * nmo, eri, sizeof(double) * nmo2,
                                   sizeof(double) * nocc * nmo, nmo2, cudaMemcpyHostToDevice, s));
    }
    launch_delta(h->mo.as<double>(), nmo, nocc, h->delta.as<double>(), s);
    if (!bound)
        kprof(h, kKprofGatherVph, 16.0 * (double)n * (double)n,
              [&] { return (int64_t)launch_gather_vph(h->pqo.as<double>(), nmo, nocc, h->v.as<double>(), s); });
    launch_sigma_x_diag(h->xdiag.as<double>(), nmo, nocc, h->sigx.as<double>(), s);
    GWB_CUDA(cudaStreamSynchronize(s));
    h->nmo = nmo;
    h->nocc = nocc;
    h->n = n;
    h->fermi = fermi_energy;
    h->bad_gap = bad;
    if (bound) h->bound_states.assign(states, states + nstates);
    h->loaded = true;
}
} // namespace

int gwb200_load_system(gwb200_handle* h, int64_t nmo, int64_t nocc, const double* mo_energy, const double* eri,
                       const double* vxc, double fermi_energy) {
    return guarded([&] { load_system_impl(h, nmo, nocc, mo_energy, eri, vxc, fermi_energy, nullptr, 0); });
}

int gwb200_load_system_states(gwb200_handle* h, int64_t nmo, int64_t nocc, const double* mo_energy, const double* eri,
                              const double* vxc, double fermi_energy, const int64_t* states, int64_t nstates) {
    return guarded([&] {
        if (!states) fail(GWB200_BAD_ARGUMENT, "null state list");
        load_system_impl(h, nmo, nocc, mo_energy, eri, vxc, fermi_energy, states, nstates);
    });
}

int gwb200_read_resident(gwb200_handle* h, const int64_t* states, int64_t nstates, double* vph_out,
                         double* panel_out) {
    return guarded([&] {
        check_system(h);
        cudaStream_t s = h->stream;
        const int64_t n = h->n;
        if (vph_out) GWB_CUDA(cudaMemcpyAsync(vph_out, h->v.p, sizeof(double) * (size_t)n * n, cudaMemcpyDeviceToHost, s));
        if (panel_out) {
            check_states(h, states, nstates);
            const size_t nb = sizeof(double) * (size_t)nstates * h->nmo * n;
            if (!h->bound_states.empty()) {
                if (!std::equal(states, states + nstates, h->bound_states.begin(), h->bound_states.end()))
                    fail(GWB200_BAD_ARGUMENT, "the state list must be the one given to gwb200_load_system_states");
            } else {  // the panel rows a screening call would gather from the resident (pq|o.) block
                h->in.ensure(sizeof(int64_t) * nstates);
                size_buffer(h, h->xt, nb);
                GWB_CUDA(cudaMemcpyAsync(h->in.p, states, sizeof(int64_t) * nstates, cudaMemcpyHostToDevice, s));
                launch_gather_panel(h->pqo.as<double>(), h->nmo, h->nocc, h->in.as<int64_t>(), nstates,
                                    h->xt.as<double>(), s);
            }
            GWB_CUDA(cudaMemcpyAsync(panel_out, h->xt.p, nb, cudaMemcpyDeviceToHost, s));
        }
        GWB_CUDA(cudaStreamSynchronize(s));
    });
}

int gwb200_load_system_slices(gwb200_handle* h, int64_t nmo, int64_t nocc, const double* mo_energy,
                              const double* vph, const double* panel, const double* xdiag, const double* vxc_diag,
                              double fermi_energy, const int64_t* states, int64_t nstates) {
    return guarded([&] {
        const HostSlices sl{vph, panel, xdiag, vxc_diag};
        load_system_impl(h, nmo, nocc, mo_energy, nullptr, nullptr, fermi_energy, states, nstates, &sl);
    });
}

int gwb200_screened_forms(gwb200_handle* h, const double* omega, int64_t nfreq, const int64_t* states,
                          int64_t nstates, double eta, int precision, double* q_out, gwb200_stats* stats) {
    return guarded([&] {
        check_system(h);
        if (!q_out) fail(GWB200_BAD_ARGUMENT, "null output array");
        if (eta != 0.0)
            fail(GWB200_ETA_NONZERO, "real screened forms exist only at eta == 0; use gwb200_screened_forms_complex");
        gwb200_stats local{};
        gwb200_stats* st = stats ? stats : &local;
        *st = gwb200_stats{};
        compute_forms(h, omega, nfreq, states, nstates, eta, precision, st);
        finish_forms(h, st);
        const int64_t m = nstates * h->nmo;
        const int64_t ldq = make_geometry(h->n, m).m_pad;
        GWB_CUDA(cudaMemcpy2DAsync(q_out, sizeof(double) * m, h->qall.p, sizeof(double) * ldq, sizeof(double) * m,
                                   (size_t)nfreq, cudaMemcpyDeviceToHost, h->stream));
        GWB_CUDA(cudaStreamSynchronize(h->stream));
    });
}

int gwb200_screened_forms_complex(gwb200_handle* h, const double* omega, int64_t nfreq, const int64_t* states,
                                  int64_t nstates, double eta, double* q_out, gwb200_stats* stats) {
    return guarded([&] {
        check_system(h);
        if (!q_out) fail(GWB200_BAD_ARGUMENT, "null output array");
        gwb200_stats local{};
        gwb200_stats* st = stats ? stats : &local;
        *st = gwb200_stats{};
        compute_forms(h, omega, nfreq, states, nstates, eta, GWB200_FP64, st);
        finish_forms(h, st);
        const int64_t m = nstates * h->nmo;
        const int64_t ldq = make_geometry(h->n, m).m_pad;
        if (h->complex_forms) {
            GWB_CUDA(cudaMemcpy2DAsync(q_out, 2 * sizeof(double) * m, h->qall.p, 2 * sizeof(double) * ldq,
                                       2 * sizeof(double) * m, (size_t)nfreq, cudaMemcpyDeviceToHost, h->stream));
            GWB_CUDA(cudaStreamSynchronize(h->stream));
        } else {  // eta == 0: real forms, imaginary parts zero
            std::vector<double> re((size_t)nfreq * m);
            GWB_CUDA(cudaMemcpy2DAsync(re.data(), sizeof(double) * m, h->qall.p, sizeof(double) * ldq,
                                       sizeof(double) * m, (size_t)nfreq, cudaMemcpyDeviceToHost, h->stream));
            GWB_CUDA(cudaStreamSynchronize(h->stream));
            for (size_t i = 0; i < re.size(); ++i) {
                q_out[2 * i] = re[i];
                q_out[2 * i + 1] = 0.0;
            }
        }
    });
}

int gwb200_sigma_c(gwb200_handle* h, const double* omega, const double* weight, int64_t nfreq, const int64_t* states,
                   int64_t nstates, double eta, int precision, double* sigma_out, gwb200_stats* stats) {
    return guarded([&] {
        check_system(h);
        if (!weight || !sigma_out) fail(GWB200_BAD_ARGUMENT, "null weight or output array");
        gwb200_stats local{};
        gwb200_stats* st = stats ? stats : &local;
        *st = gwb200_stats{};
        compute_forms(h, omega, nfreq, states, nstates, eta, precision, st, weight);
        size_results(h, nstates, nfreq);
        contract_on_device(h, nfreq, nstates, st);
        finish_forms(h, st, {{h->call.sigma, sizeof(double) * 2 * (size_t)nstates * nfreq}});
        st->device_ms_contract = elapsed(h->ev[2], h->ev[3]);
        st->device_ms_total = elapsed(h->ev[0], h->ev[3]);
        scatter_sigma(h, result_stage(h), states, nstates, nfreq, sigma_out);
    });
}

int gwb200_sigma_c_matrix(gwb200_handle* h, const double* omega, const double* weight, int64_t nfreq,
                          const int64_t* states, int64_t nstates, double* sigma_out, gwb200_stats* stats) {
    return guarded([&] {
        check_system(h);
        if (!omega || !weight || !sigma_out || !states) fail(GWB200_BAD_ARGUMENT, "null input or output array");
        if (nstates < 1 || nstates > 64) fail(GWB200_BAD_SHAPE, "the state-pair self-energy takes 1 to 64 states");
        if (nfreq <= 0) fail(GWB200_BAD_SHAPE, "--freq-points must be positive");
        gwb200_stats local{};
        gwb200_stats* st = stats ? stats : &local;
        *st = gwb200_stats{};
        cudaStream_t s = h->stream;
        const int64_t ns = nstates;
        const size_t per_freq = (size_t)h->nmo * ns * ns;  // cross forms [k][s][t] of one frequency
        size_buffer(h, h->qx, sizeof(double) * per_freq * (size_t)nfreq);
        const ChunkHook hook = [&](const TallGeometry& g, int64_t f0, int64_t nf) {
            launch_cross_forms(g, nf, h->a.as<double>(), h->nmo, ns, h->qx.as<double>() + (size_t)f0 * per_freq, s);
        };
        compute_forms(h, omega, nfreq, states, nstates, 0.0, GWB200_FP64, st, weight, &hook);
        const size_t sig_bytes = sizeof(double) * 2 * (size_t)ns * ns * nfreq;
        size_buffer(h, h->sigmx, sig_bytes);
        st->kernel_launches += launch_sigma_contract_pairs(
            h->qx.as<double>(), nfreq, h->nmo, ns, h->mo.as<double>(), h->fermi, h->call.omega, h->call.weight,
            h->call.omega, nfreq, h->sigmx.as<double>(), s);
        GWB_CUDA(cudaEventRecord(h->ev[3], s));
        finish_forms(h, st, {{h->sigmx.p, sig_bytes}});
        st->device_ms_contract = elapsed(h->ev[2], h->ev[3]);
        st->device_ms_total = elapsed(h->ev[0], h->ev[3]);
        std::memcpy(sigma_out, result_stage(h), sig_bytes);
    });
}

int gwb200_sigma_c_shard(gwb200_handle* h, const double* omega, const double* weight, int64_t nfreq, int64_t f_begin,
                         int64_t f_end, const int64_t* states, int64_t nstates, double eta, int precision,
                         double* sigma_partial_out, gwb200_stats* stats) {
    return guarded([&] {
        check_system(h);
        if (!omega || !weight || !sigma_partial_out) fail(GWB200_BAD_ARGUMENT, "null input or output array");
        if (nfreq <= 0 || f_begin < 0 || f_end > nfreq || f_begin > f_end)
            fail(GWB200_BAD_SHAPE, "frequency shard must satisfy 0 <= f_begin <= f_end <= nfreq");
        gwb200_stats local{};
        gwb200_stats* st = stats ? stats : &local;
        *st = gwb200_stats{};
        if (f_begin == f_end) {  // empty shard: contributes nothing
            std::fill(sigma_partial_out, sigma_partial_out + 2 * (size_t)h->nmo * nfreq, 0.0);
            return;
        }
        cudaStream_t s = h->stream;
        h->omega_out.ensure(sizeof(double) * nfreq);
        GWB_CUDA(cudaMemcpyAsync(h->omega_out.p, omega, sizeof(double) * nfreq, cudaMemcpyHostToDevice, s));
        compute_forms(h, omega + f_begin, f_end - f_begin, states, nstates, eta, precision, st, weight + f_begin);
        size_results(h, nstates, nfreq);
        contract_on_device(h, f_end - f_begin, nstates, st, h->omega_out.as<double>(), nfreq);
        finish_forms(h, st, {{h->call.sigma, sizeof(double) * 2 * (size_t)nstates * nfreq}});
        st->device_ms_contract = elapsed(h->ev[2], h->ev[3]);
        st->device_ms_total = elapsed(h->ev[0], h->ev[3]);
        scatter_sigma(h, result_stage(h), states, nstates, nfreq, sigma_partial_out);
    });
}

int gwb200_run_g0w0(gwb200_handle* h, int64_t nfreq, int64_t npade, const int64_t* states, int64_t nstates,
                    double eta, int precision, double* omega_out, double* weight_out, double* sigma_out,
                    double* sigma_x_out, double* qp_out, gwb200_stats* stats) {
    return guarded([&] {
        check_system(h);
        if (nfreq <= 0) fail(GWB200_BAD_SHAPE, "--freq-points must be positive");
        if (npade <= 0) fail(GWB200_BAD_SHAPE, "--pade-params must be positive");
        gwb200_stats local{};
        gwb200_stats* st = stats ? stats : &local;
        *st = gwb200_stats{};
        std::vector<double> omega((size_t)nfreq), weight((size_t)nfreq);
        transformed_legendre_grid(nfreq, omega.data(), weight.data());
        compute_forms(h, omega.data(), nfreq, states, nstates, eta, precision, st, weight.data());
        size_results(h, nstates, nfreq);
        contract_on_device(h, nfreq, nstates, st);
        qp_on_device(h, nfreq, npade, nstates);
        st->kernel_launches += 1;
        const size_t nb_sig = sizeof(double) * 2 * (size_t)nstates * nfreq, nb_qp = sizeof(double) * nstates,
                     nb_v = sizeof(double) * h->nmo;
        finish_forms(h, st, {{h->call.sigma, nb_sig + nb_qp}, {h->sigx.p, nb_v}});
        st->device_ms_contract = elapsed(h->ev[2], h->ev[3]);
        st->device_ms_total = elapsed(h->ev[0], h->ev[3]);
        const char* o = result_stage(h);
        if (sigma_out) scatter_sigma(h, o, states, nstates, nfreq, sigma_out);
        if (qp_out) scatter_qp(h, o + nb_sig, states, nstates, qp_out);
        if (sigma_x_out) std::memcpy(sigma_x_out, o + nb_sig + nb_qp, nb_v);
        if (omega_out) std::copy(omega.begin(), omega.end(), omega_out);
        if (weight_out) std::copy(weight.begin(), weight.end(), weight_out);
    });
}

int gwb200_sigma_x_diag(gwb200_handle* h, double* out) {
    return guarded([&] {
        check_system(h);
        if (!out) fail(GWB200_BAD_ARGUMENT, "null output array");
        GWB_CUDA(cudaMemcpyAsync(out, h->sigx.p, sizeof(double) * h->nmo, cudaMemcpyDeviceToHost, h->stream));
        GWB_CUDA(cudaStreamSynchronize(h->stream));
    });
}

int gwb200_qp(gwb200_handle* h, const double* omega, int64_t nfreq, const double* sigma, int64_t npade,
              const int64_t* states, int64_t nstates, double* qp_out) {
    return guarded([&] {
        check_system(h);
        if (!omega || !sigma || !qp_out) fail(GWB200_BAD_ARGUMENT, "null input or output array");
        if (nfreq <= 0) fail(GWB200_BAD_SHAPE, "nfreq must be positive");
        if (npade <= 0) fail(GWB200_BAD_SHAPE, "Pade: npar must be positive");
        check_states(h, states, nstates);
        check_npade(npade);
        cudaStream_t s = h->stream;
        // grid, the states' rows and the state list: one pinned upload; one read back
        const size_t nb_om = sizeof(double) * nfreq, nb_st = sizeof(int64_t) * nstates;
        const size_t nb_sig = 2 * nb_om * (size_t)nstates, nb_qp = sizeof(double) * nstates;
        h->in.ensure(nb_om + nb_sig + nb_st);
        h->stage_in.ensure(nb_om + nb_sig + nb_st);
        char* p = h->stage_in.as<char>();
        std::memcpy(p, omega, nb_om);
        for (int64_t i = 0; i < nstates; ++i)
            std::memcpy(p + nb_om + 2 * nb_om * (size_t)i, sigma + 2 * (size_t)(states[i] * nfreq), 2 * nb_om);
        std::memcpy(p + nb_om + nb_sig, states, nb_st);
        GWB_CUDA(cudaMemcpyAsync(h->in.p, p, nb_om + nb_sig + nb_st, cudaMemcpyHostToDevice, s));
        h->call.omega = h->in.as<double>();
        h->call.sigma = h->call.omega + nfreq;
        h->call.states = reinterpret_cast<int64_t*>(h->call.sigma + 2 * (size_t)nstates * nfreq);
        h->out.ensure(nb_qp);
        h->call.qp = h->out.as<double>();
        qp_on_device(h, nfreq, npade, nstates);
        h->stage_out.ensure(nb_qp);
        GWB_CUDA(cudaMemcpyAsync(h->stage_out.p, h->call.qp, nb_qp, cudaMemcpyDeviceToHost, s));
        GWB_CUDA(cudaStreamSynchronize(s));
        scatter_qp(h, h->stage_out.as<char>(), states, nstates, qp_out);
    });
}

int gwb200_pade_sweep(gwb200_handle* h, const double* omega, int64_t nfreq, const double* sigma_row, int64_t npade,
                      int64_t npts, double fermi, double x_start, double interval, double* out) {
    return guarded([&] {
        check_handle(h);
        if (!omega || !sigma_row || !out) fail(GWB200_BAD_ARGUMENT, "null input or output array");
        if (nfreq <= 0 || npts <= 0) fail(GWB200_BAD_SHAPE, "nfreq and npts must be positive");
        if (npade <= 0) fail(GWB200_BAD_SHAPE, "Pade: npar must be positive");
        check_npade(npade);  // no copy of the caller's arrays is in flight when a call is refused
        cudaStream_t s = h->stream;
        // kept by the handle: allocating and freeing them per call synchronised the device each time.  A
        // capped handle gives them back, its cap is for the solves.
        h->sweep.ensure(sizeof(double) * ((size_t)nfreq * 3 + 3 * (size_t)npts));
        double* dom = h->sweep.as<double>();
        double* drow = dom + nfreq;
        double* dout = drow + 2 * nfreq;
        try {
            GWB_CUDA(cudaMemcpyAsync(dom, omega, sizeof(double) * nfreq, cudaMemcpyHostToDevice, s));
            GWB_CUDA(cudaMemcpyAsync(drow, sigma_row, sizeof(double) * 2 * nfreq, cudaMemcpyHostToDevice, s));
            launch_pade_sweep(drow, dom, nfreq, npade, npts, fermi, x_start, interval, dout, s);
            GWB_CUDA(cudaMemcpyAsync(out, dout, sizeof(double) * 3 * (size_t)npts, cudaMemcpyDeviceToHost, s));
        } catch (...) {
            cudaStreamSynchronize(s);
            throw;
        }
        GWB_CUDA(cudaStreamSynchronize(s));
        if (h->mem_limit > 0) h->sweep.release();
    });
}

int gwb200_grid(int64_t nfreq, double* omega, double* weight) {
    return guarded([&] {
        if (!omega || !weight) fail(GWB200_BAD_ARGUMENT, "null output array");
        transformed_legendre_grid(nfreq, omega, weight);
    });
}

int gwb200_read_input_h5(const char* path, int64_t* nmo, int64_t* nocc, double* fermi_energy, double* mo_energy,
                         double* eri, double* vxc) {
    return guarded([&] {
        if (!path || !nmo || !nocc || !fermi_energy) fail(GWB200_BAD_ARGUMENT, "null argument");
        read_gw_input_h5(path, nmo, nocc, fermi_energy, mo_energy, eri, vxc);
    });
}

int gwb200_read_input_h5_slices(const char* path, const int64_t* states, int64_t nstates, int64_t* nmo,
                                int64_t* nocc, double* fermi_energy, double* mo_energy, double* vph, double* panel,
                                double* xdiag, double* vxc_diag) {
    return guarded([&] {
        if (!path || !nmo || !nocc || !fermi_energy) fail(GWB200_BAD_ARGUMENT, "null argument");
        read_gw_input_h5_slices(path, states, nstates, nmo, nocc, fermi_energy, mo_energy, vph, panel, xdiag,
                                vxc_diag);
    });
}

int gwb200_screened_forms_noalloc(int64_t n, int64_t m, const double* d_v, const double* d_xt,
                                  const double* d_delta, const double* d_omega, int64_t nfreq, double* d_q_out,
                                  void* stream) {
    return guarded([&] {
        screened_forms_noalloc(n, m, d_v, d_xt, d_delta, d_omega, nfreq, d_q_out, static_cast<cudaStream_t>(stream));
    });
}

int gwb200_fp64_peak_tflops(gwb200_handle* h, double* tflops) {
    return guarded([&] {
        check_handle(h);
        if (!tflops) fail(GWB200_BAD_ARGUMENT, "null output");
        *tflops = measure_fp64_peak_tflops(h->stream);
    });
}

namespace {
// Molecule order of a batch: ascending (n, m), ties by position.
std::vector<int> batch_order(const std::vector<int64_t>& ns, const std::vector<int64_t>& ms) {
    std::vector<int> order(ns.size());
    std::iota(order.begin(), order.end(), 0);
    std::sort(order.begin(), order.end(), [&](int x, int y) {
        if (ns[(size_t)x] != ns[(size_t)y]) return ns[(size_t)x] < ns[(size_t)y];
        if (ms[(size_t)x] != ms[(size_t)y]) return ms[(size_t)x] < ms[(size_t)y];
        return x < y;
    });
    return order;
}

// Lanes of a batch: GWB200_BATCH_STREAMS concurrent streams (default 4, at most one per
// molecule), each with its own workspaces; GWB200_BATCH_SHARE_SMS=1 caps each lane's persistent
// update kernels at SMs / lanes CTAs (default: every lane's grid covers the GPU; those kernels take
// their work units from a counter and never wait on one another, so they need not be co-resident).
// Measured on the 64-molecule config-4 batch (mixed): 1 lane 261-274 ms, 2 lanes 233-244, 4 lanes
// 221-224.  Returns the lane count; *ctas the persistent-grid cap (0: none).
int batch_lanes(const gwb200_handle* w, int64_t nsys, int* ctas) {
    int lanes = kMaxBatchLanes;
    if (const char* e = std::getenv("GWB200_BATCH_STREAMS")) lanes = std::atoi(e);
    lanes = std::max(1, std::min<int>({kMaxBatchLanes, lanes, (int)nsys}));
    const char* share_env = std::getenv("GWB200_BATCH_SHARE_SMS");
    *ctas = w->persistent_ctas;
    if (lanes > 1 && share_env && std::strcmp(share_env, "1") == 0) {
        int sms = 148;
        GWB_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, w->device));
        *ctas = std::max(1, (w->persistent_ctas > 0 ? w->persistent_ctas : sms) / lanes);
    }
    return lanes;
}

// Device bytes the batch's lane workspaces may take: free memory plus what the lanes hold, and,
// for a capped lead handle, its cap minus what it holds besides the lanes.
size_t batch_avail(const gwb200_handle* w) {
    size_t free_b = 0, total_b = 0;
    GWB_CUDA(cudaMemGetInfo(&free_b, &total_b));
    size_t held = 0;
    for (const BatchLane& l : w->lanes) held += l.bytes();
    size_t avail = free_b + held;
    if (w->mem_limit > 0) {
        size_t resident = (size_t)1 << 20;
        for (const DevBuf* b : {&w->pqo, &w->xdiag, &w->v, &w->xt, &w->dvec, &w->qall, &w->in, &w->out, &w->a,
                                &w->qacc, &w->panel32})
            resident += b->bytes;
        const size_t lim = (size_t)w->mem_limit;
        avail = std::min(avail, lim > resident ? lim - resident : (size_t)0);
    }
    return avail;
}

// Bucket plans to run: GWB200_BATCH_PLAN=tuned (default: the plan cached for this signature, else
// the cost model's plans for three latency weights plus one bucket per molecule, to be timed),
// =model (the cost model alone), =each (one bucket per molecule), =single (one bucket).
std::vector<std::vector<int64_t>> batch_candidates(const std::vector<int64_t>& key, const std::vector<int64_t>& n_sorted,
                                                   const std::vector<int64_t>& m_sorted,
                                                   const std::vector<int64_t>& f_sorted, bool mixed,
                                                   size_t lane_budget) {
    const int64_t nsys = (int64_t)n_sorted.size();
    const char* mode_env = std::getenv("GWB200_BATCH_PLAN");
    const std::string mode = mode_env ? mode_env : "tuned";
    if (mode == "each") return {std::vector<int64_t>((size_t)nsys, 1)};
    if (mode == "single") return {{nsys}};
    if (mode == "tuned") {
        std::lock_guard<std::mutex> lk(g_batch_mu);
        auto it = g_batch_plans.find(key);
        if (it != g_batch_plans.end()) return {it->second};
    }
    std::vector<std::vector<int64_t>> cands;
    const double tau = batch_step_us(), rate = batch_tflops(mixed);
    for (double mult : (mode == "tuned" ? std::vector<double>{1.0, 0.25, 4.0} : std::vector<double>{1.0})) {
        std::vector<int64_t> p = plan_buckets(n_sorted, m_sorted, f_sorted, mixed, lane_budget, tau * mult, rate);
        if (std::find(cands.begin(), cands.end(), p) == cands.end()) cands.push_back(p);
    }
    if (mode == "tuned") {
        std::vector<int64_t> each((size_t)nsys, 1);
        if (std::find(cands.begin(), cands.end(), each) == cands.end()) cands.push_back(each);
    }
    return cands;
}

// What a captured batch graph depends on: the plan signature and plan, the launch sequences the plan
// was cut into (each chunk's geometry, matrix count and group range, and the chunks each lane runs:
// the chunk size follows the free device memory and GWB200_MAX_FREQ_CHUNK, so the same plan can be
// cut differently from call to call), the scalars its kernels take by value (E_F, sizes, Pade order,
// lanes, update variants) and every device pointer and stream it uses.  A replay is valid exactly
// while this is unchanged.
std::vector<int64_t> batch_graph_key(const gwb200_handle* w, const std::vector<gwb200_handle*>& hs,
                                     const std::vector<int64_t>& key, const std::vector<int64_t>& plan,
                                     const std::vector<BatchChunk>& chunks,
                                     const std::vector<std::vector<size_t>>& assign,
                                     const std::vector<int64_t>& fs, const std::vector<int64_t>& ps, int lanes,
                                     int lane_ctas, const std::vector<int>& variants, const int64_t* const* states,
                                     const int64_t* nstates) {
    std::vector<int64_t> gkey = key;
    auto put = [&](const void* ptr) { gkey.push_back((int64_t)reinterpret_cast<intptr_t>(ptr)); };
    gkey.insert(gkey.end(), plan.begin(), plan.end());
    gkey.push_back((int64_t)chunks.size());
    for (const BatchChunk& c : chunks)
        gkey.insert(gkey.end(), {c.g.n, c.g.m, c.g.n_pad, c.g.m_pad, c.nmat, c.group0, c.ngroups});
    for (const auto& lane : assign) {
        gkey.push_back(-1 - (int64_t)lane.size());
        gkey.insert(gkey.end(), lane.begin(), lane.end());
    }
    gkey.insert(gkey.end(), fs.begin(), fs.end());
    gkey.insert(gkey.end(), ps.begin(), ps.end());
    gkey.push_back(lanes);
    gkey.push_back(lane_ctas);
    gkey.insert(gkey.end(), variants.begin(), variants.end());
    for (size_t i = 0; i < hs.size(); ++i) {
        const gwb200_handle* h = hs[i];
        put(h);
        int64_t fermi_bits = 0;
        std::memcpy(&fermi_bits, &h->fermi, sizeof(fermi_bits));
        gkey.insert(gkey.end(), {fermi_bits, h->n, h->nmo, h->nocc});
        gkey.push_back(nstates[i]);
        gkey.insert(gkey.end(), states[i], states[i] + nstates[i]);
        gkey.push_back(h->bound_states.empty() ? 0 : 1);
        for (const DevBuf* b : {&h->pqo, &h->v, &h->xt, &h->dvec, &h->qall, &h->delta, &h->mo, &h->sigx, &h->vxc_diag})
            put(b->p);
        for (const void* p : {(const void*)h->call.omega, (const void*)h->call.weight, (const void*)h->call.states,
                              (const void*)h->call.sigma, (const void*)h->call.qp})
            put(p);
        put(h->pchol_ct);
        put(h->pchol_sl.p);
        gkey.push_back(h->pchol_rank);
    }
    put(w->in.p);
    put(w->stage_in.p);
    put(w->batch_fork);
    for (int l = 0; l < lanes; ++l) {
        const BatchLane& ln = w->lanes[l];
        for (const DevBuf* b : {&ln.a, &ln.qacc, &ln.panel, &ln.sched, &ln.refine}) put(b->p);
        put(ln.stream);
        put(ln.done);
    }
    return gkey;
}
} // namespace

int gwb200_plan_buckets(int64_t nsys, const int64_t* nph, const int64_t* ncols, int64_t nfreq, int precision,
                        int64_t budget_bytes, double step_us, double tflops, int64_t* bucket_of, int64_t* nbuckets) {
    return guarded([&] {
        if (nsys <= 0 || !nph || !ncols || !bucket_of || !nbuckets) fail(GWB200_BAD_ARGUMENT, "empty or null batch");
        if (nfreq <= 0 || budget_bytes <= 0) fail(GWB200_BAD_SHAPE, "nfreq and the budget must be positive");
        if (precision != GWB200_FP64 && precision != GWB200_MIXED && precision != GWB200_MIXED_REFINED)
            fail(GWB200_BAD_ARGUMENT, "unknown precision");
        const bool mixed = precision != GWB200_FP64;
        std::vector<int64_t> ns(nph, nph + nsys), ms(ncols, ncols + nsys);
        for (int64_t i = 0; i < nsys; ++i)
            if (ns[(size_t)i] <= 0 || ms[(size_t)i] <= 0) fail(GWB200_BAD_SHAPE, "nph and ncols must be positive");
        const std::vector<int> order = batch_order(ns, ms);
        std::vector<int64_t> n_sorted, m_sorted;
        for (int i : order) {
            n_sorted.push_back(ns[(size_t)i]);
            m_sorted.push_back(ms[(size_t)i]);
        }
        const std::vector<int64_t> sizes =
            plan_buckets(n_sorted, m_sorted, std::vector<int64_t>(n_sorted.size(), nfreq), mixed, (size_t)budget_bytes,
                         step_us > 0 ? step_us : batch_step_us(),
                         tflops > 0 ? tflops : batch_tflops(mixed));
        size_t pos = 0;
        for (size_t b = 0; b < sizes.size(); ++b)
            for (int64_t t = 0; t < sizes[b]; ++t) bucket_of[order[pos++]] = (int64_t)b;
        *nbuckets = (int64_t)sizes.size();
    });
}

int gwb200_run_g0w0_batch(gwb200_handle* const* systems, int64_t nsys, const int64_t* nfreq, const int64_t* npade,
                          const int64_t* const* states, const int64_t* nstates, int precision, double* const* sigma_out,
                          double* const* qp_out, int64_t* nbuckets_out, gwb200_stats* stats) {
    return guarded([&] {
        if (!systems || nsys <= 0) fail(GWB200_BAD_ARGUMENT, "empty batch");
        if (nsys > 65535) fail(GWB200_BAD_SHAPE, "at most 65535 systems per batch");  // one grid row per member run
        if (!states || !nstates) fail(GWB200_BAD_ARGUMENT, "null state lists");
        if (!nfreq || !npade) fail(GWB200_BAD_ARGUMENT, "null frequency or Pade counts");
        const std::vector<int64_t> fs(nfreq, nfreq + nsys), ps(npade, npade + nsys);
        for (int64_t i = 0; i < nsys; ++i) {
            if (fs[(size_t)i] <= 0) fail(GWB200_BAD_SHAPE, "--freq-points must be positive");
            if (ps[(size_t)i] <= 0) fail(GWB200_BAD_SHAPE, "--pade-params must be positive");
        }
        if (precision != GWB200_FP64 && precision != GWB200_MIXED && precision != GWB200_MIXED_REFINED)
            fail(GWB200_BAD_ARGUMENT, "unknown precision");
        std::vector<gwb200_handle*> hs(systems, systems + nsys);
        for (gwb200_handle* h : hs)
            if (!h) fail(GWB200_BAD_ARGUMENT, "null handle in the batch");
        gwb200_handle* w = hs[0];
        check_system(w);
        {
            std::vector<gwb200_handle*> uniq(hs);
            std::sort(uniq.begin(), uniq.end());
            if (std::adjacent_find(uniq.begin(), uniq.end()) != uniq.end())
                fail(GWB200_BAD_ARGUMENT, "a handle appears twice in the batch");
        }
        std::vector<int64_t> ns((size_t)nsys), ms((size_t)nsys);
        for (int64_t i = 0; i < nsys; ++i) {
            gwb200_handle* h = hs[(size_t)i];
            if (!h->loaded) fail(GWB200_NO_SYSTEM, "no system loaded: call gwb200_load_system first");
            if (h->device != w->device) fail(GWB200_BAD_ARGUMENT, "the systems of a batch must share one device");
            check_states(h, states[i], nstates[i]);
            if (!h->bound_states.empty() &&
                !std::equal(states[i], states[i] + nstates[i], h->bound_states.begin(), h->bound_states.end()))
                fail(GWB200_BAD_ARGUMENT, "the state list must be the one given to gwb200_load_system_states");
            if (h->bad_gap)
                fail(GWB200_NONPOSITIVE_GAP, "some e_a - e_i <= 0: chi0(iw) is not negative definite, eps(iw) is not SPD");
            ns[(size_t)i] = h->n;
            ms[(size_t)i] = nstates[i] * h->nmo;
        }
        const bool mixed = precision != GWB200_FP64;
        const bool refine = precision == GWB200_MIXED_REFINED;
        const bool mixed_tc = mixed && mixed_update_on_tcgen05(w);
        const bool oz = !mixed && fp64_update_mode() != 1 && (w->mem_limit <= 0 || fp64_update_mode() == 2);
        if (refine)  // each molecule's pivoted Cholesky factor of V, on its own stream, before any capture
            for (gwb200_handle* h : hs) refine_factor(h, h->stream);
        gwb200_stats local{};
        gwb200_stats* st = stats ? stats : &local;
        *st = gwb200_stats{};
        for (gwb200_handle* h : hs)
            if (h->stream != w->stream) GWB_CUDA(cudaStreamSynchronize(h->stream));
        StreamSwap swap;
        swap.hs = hs;
        for (gwb200_handle* h : hs) swap.saved.push_back(h->stream);
        for (gwb200_handle* h : hs) h->stream = w->stream;
        cudaStream_t s = w->stream;

        // members' own buffers first (they are not part of the batched-matrix budget)
        size_t nb_states = 0;
        for (int64_t i = 0; i < nsys; ++i) {
            gwb200_handle* h = hs[(size_t)i];
            const TallGeometry gi = make_geometry(h->n, ms[(size_t)i]);
            const int64_t nfreq = fs[(size_t)i];
            if (h->bound_states.empty()) size_buffer(h, h->xt, sizeof(double) * (size_t)ms[(size_t)i] * h->n);
            size_buffer(h, h->dvec, sizeof(double) * (size_t)nfreq * gi.n_pad);
            size_buffer(h, h->qall, sizeof(double) * (size_t)nfreq * gi.m_pad);
            h->complex_forms = false;
            nb_states += sizeof(int64_t) * nstates[i];
        }
        int lane_ctas = 0;
        const int lanes = batch_lanes(w, nsys, &lane_ctas);

        // plans over the molecules sorted by size (batch_candidates)
        const std::vector<int> order = batch_order(ns, ms);
        std::vector<int64_t> n_sorted, m_sorted, f_sorted;
        for (int i : order) {
            n_sorted.push_back(ns[(size_t)i]);
            m_sorted.push_back(ms[(size_t)i]);
            f_sorted.push_back(fs[(size_t)i]);
        }
        const size_t avail = batch_avail(w);
        std::vector<int64_t> key = {(int64_t)w->device, (int64_t)precision, (int64_t)oz, (int64_t)mixed_tc,
                                    (int64_t)lanes, (int64_t)lane_ctas};
        key.insert(key.end(), n_sorted.begin(), n_sorted.end());
        key.insert(key.end(), m_sorted.begin(), m_sorted.end());
        key.insert(key.end(), f_sorted.begin(), f_sorted.end());
        const std::vector<std::vector<int64_t>> cands =
            batch_candidates(key, n_sorted, m_sorted, f_sorted, mixed, (size_t)(0.85 * (double)avail / lanes));
        // chunks of every candidate inside one budget (all candidates share the workspaces)
        const TallGeometry gmax = make_geometry(n_sorted.back(), *std::max_element(m_sorted.begin(), m_sorted.end()));
        if (batch_bytes_per_matrix(gmax, mixed, oz, refine) > avail)
            fail(GWB200_OOM, "not enough device memory for one frequency of the largest eps(iw) in the batch");
        size_t budget = (size_t)(0.85 * (double)avail / lanes);  // per lane
        // GWB200_MAX_FREQ_CHUNK caps the matrices per launch sequence (tests use it to split buckets)
        int64_t cap = 0;
        if (const char* env = std::getenv("GWB200_MAX_FREQ_CHUNK")) cap = std::max<long long>(0, std::atoll(env));
        std::vector<std::vector<BatchChunk>> chunks;
        std::vector<BatchGroup> groups;
        BatchNeed need;
        for (int attempt = 0;; ++attempt) {
            chunks.clear();
            groups.clear();
            need = BatchNeed{};
            for (const auto& p : cands) {
                chunks.push_back(batch_chunks(hs, ms, fs, order, p, mixed, oz, refine, budget, cap, groups));
                batch_need(chunks.back(), mixed, oz, refine, need);
            }
            if (need.total() * (size_t)lanes <= (size_t)(0.9 * (double)avail) || attempt >= 12) break;
            budget = (size_t)(0.7 * (double)budget);
        }
        for (int l = 0; l < lanes; ++l) {
            BatchLane& ln = w->lanes[l];
            // batch_avail counted everything the lane holds as free: when a buffer must grow, or the
            // lane holds one this call does not use (the correction terms of an earlier refined
            // batch, the operand panel of another form), free them all before allocating, so the
            // new sizes fit the budget they were planned in
            const bool grow = need.a > ln.a.bytes || need.qacc > ln.qacc.bytes ||
                              need.panel > ln.panel.bytes || need.refine > ln.refine.bytes;
            const bool unused = (!need.panel && ln.panel.bytes) || (!need.refine && ln.refine.bytes);
            if (grow || unused)
                for (DevBuf* b : {&ln.a, &ln.qacc, &ln.panel, &ln.refine}) b->release();
            size_buffer(w, ln.a, need.a);
            size_buffer(w, ln.qacc, need.qacc);
            if (need.panel) size_buffer(w, ln.panel, need.panel);
            if (need.refine) size_buffer(w, ln.refine, need.refine);
            ln.sched.ensure(need.sched);
            if (l > 0 && !ln.stream) {
                GWB_CUDA(cudaStreamCreateWithFlags(&ln.stream, cudaStreamNonBlocking));
                GWB_CUDA(cudaEventCreateWithFlags(&ln.done, cudaEventDisableTiming));
            }
        }
        if (!w->batch_fork) GWB_CUDA(cudaEventCreateWithFlags(&w->batch_fork, cudaEventDisableTiming));
        // the call's inputs in one upload: the pivot word, one grid (omega, weights) per distinct frequency
        // count, the state lists, the group tables
        std::map<int64_t, size_t> grid_off;
        size_t groups_off = sizeof(unsigned long long);
        for (int64_t f : fs)
            if (grid_off.emplace(f, groups_off).second) groups_off += 2 * sizeof(double) * (size_t)f;
        const size_t states_off = groups_off;
        groups_off += nb_states;
        const size_t nb_in = groups_off + sizeof(BatchGroup) * groups.size();
        w->in.ensure(nb_in);
        std::vector<std::vector<std::vector<size_t>>> assign;
        for (const auto& ch : chunks) assign.push_back(batch_assign(ch, lanes, batch_step_us(), batch_tflops(mixed)));
        // FP64: the update kernel of each chunk geometry (timed before anything is built: the
        // autotuner overwrites the workspace)
        std::vector<std::vector<int>> variants(cands.size());
        for (size_t c = 0; c < cands.size(); ++c)
            for (const BatchChunk& ch : chunks[c])
                variants[c].push_back(mixed ? -1
                                            : tune_update_variant(ch.g, ch.nmat, w->lanes[0].a.as<double>(), s,
                                                                  oz ? w->lanes[0].panel.p : nullptr,
                                                                  w->lanes[0].sched.as<unsigned long long>(),
                                                                  w->err(), w->mem_limit <= 0));

        // the lead handle's pinned staging buffer, filled on the host before anything is issued
        w->stage_in.ensure(nb_in);
        char* sp = w->stage_in.as<char>();
        std::memset(sp, 0xFF, sizeof(unsigned long long));
        for (const auto& [f, off] : grid_off)
            transformed_legendre_grid(f, reinterpret_cast<double*>(sp + off),
                                      reinterpret_cast<double*>(sp + off) + f);
        std::memcpy(sp + groups_off, groups.data(), sizeof(BatchGroup) * groups.size());
        // results of all members, each [nstates][nfreq] complex and nstates QP energies, read back at once
        size_t nb_out = 0;
        std::vector<size_t> out_off;
        for (int64_t i = 0; i < nsys; ++i) {
            out_off.push_back(nb_out);
            nb_out += sizeof(double) * (size_t)nstates[i] * (2 * (size_t)fs[(size_t)i] + 1);
        }
        w->out.ensure(nb_out);
        {
            size_t off = states_off;
            for (int64_t i = 0; i < nsys; ++i) {
                gwb200_handle* h = hs[(size_t)i];
                const int64_t nfreq = fs[(size_t)i];
                std::memcpy(sp + off, states[i], sizeof(int64_t) * nstates[i]);
                h->call.omega = reinterpret_cast<double*>(w->in.as<char>() + grid_off.at(nfreq));
                h->call.weight = h->call.omega + nfreq;
                h->call.states = reinterpret_cast<int64_t*>(w->in.as<char>() + off);
                h->call.sigma = reinterpret_cast<double*>(w->out.as<char>() + out_off[(size_t)i]);
                h->call.qp = h->call.sigma + 2 * (size_t)nstates[i] * nfreq;
                off += sizeof(int64_t) * nstates[i];
            }
        }
        // the lanes fork off the lead stream and join back onto it around each phase
        auto lane_stream = [&](int l) { return l == 0 ? s : w->lanes[l].stream; };
        auto fork = [&]() {
            GWB_CUDA(cudaEventRecord(w->batch_fork, s));
            for (int l = 1; l < lanes; ++l) GWB_CUDA(cudaStreamWaitEvent(w->lanes[l].stream, w->batch_fork, 0));
        };
        auto join = [&]() {
            for (int l = 1; l < lanes; ++l) {
                GWB_CUDA(cudaEventRecord(w->lanes[l].done, w->lanes[l].stream));
                GWB_CUDA(cudaStreamWaitEvent(s, w->lanes[l].done, 0));
            }
        };
        const BatchGroup* dgroups = reinterpret_cast<const BatchGroup*>(w->in.as<char>() + groups_off);
        // the device sequence in three phases: uploads and member preparation; the screening of a
        // plan (each lane runs its chunks); members' contractions and QP updates
        auto prefix = [&]() {
            int64_t n_launch = 0;
            GWB_CUDA(cudaMemcpyAsync(w->in.p, sp, nb_in, cudaMemcpyHostToDevice, s));
            fork();
            for (int64_t i = 0; i < nsys; ++i) {
                gwb200_handle* h = hs[(size_t)i];
                cudaStream_t ls = lane_stream((int)(i % lanes));
                const int64_t nfreq = fs[(size_t)i];
                if (h->bound_states.empty())
                    n_launch += launch_gather_panel(h->pqo.as<double>(), h->nmo, h->nocc, h->call.states, nstates[i],
                                                    h->xt.as<double>(), ls);
                n_launch += launch_scale_vectors(h->delta.as<double>(), h->n, make_geometry(h->n, ms[(size_t)i]).n_pad,
                                                 h->call.omega, nfreq, h->dvec.as<double>(), ls);
            }
            join();
            return n_launch;
        };
        auto run_plan = [&](size_t c) {
            int64_t n_launch = 0;
            fork();
            for (int l = 0; l < lanes; ++l)
                n_launch += batch_screen(w, w->lanes[l], lane_stream(l), lane_ctas, chunks[c], assign[c][(size_t)l],
                                         dgroups, groups, variants[c], mixed, mixed_tc, oz, refine);
            join();
            return n_launch;
        };
        auto suffix = [&]() {
            gwb200_stats scratch{};
            fork();
            for (int64_t i = 0; i < nsys; ++i) {
                hs[(size_t)i]->stream = lane_stream((int)(i % lanes));
                contract_on_device(hs[(size_t)i], fs[(size_t)i], nstates[i], &scratch);
                qp_on_device(hs[(size_t)i], fs[(size_t)i], ps[(size_t)i], nstates[i]);
            }
            join();
            return scratch.kernel_launches + nsys;
        };

        // CUDA graph of the whole sequence for a repeated batch (one plan, nothing to time):
        // captured on the second such call in a row, replayed while every pointer it holds and every
        // scalar it passes by value is unchanged.  (A batch that never comes back, as most of a
        // server's, is issued directly: capturing, instantiating and destroying its graph cost more
        // than its launches, and other threads' calls waited for the destruction, 2.7 ms each.)
        // GWB200_BATCH_GRAPH=0 issues the launches one by one.
        const char* graph_env = std::getenv("GWB200_BATCH_GRAPH");
        const bool want_graph = cands.size() == 1 && !(graph_env && std::strcmp(graph_env, "0") == 0);
        const std::vector<int64_t> gkey = want_graph ? batch_graph_key(w, hs, key, cands[0], chunks[0], assign[0], fs,
                                                                        ps, lanes, lane_ctas, variants[0], states,
                                                                        nstates)
                                                     : std::vector<int64_t>{};
        int64_t launches = 0;
        size_t pick = 0;
        bool graphed = false;
        if (want_graph && gkey != w->batch_graph_failed) {
            if (gkey == w->batch_graph_seen && !(w->batch_exec && gkey == w->batch_graph_key)) {
                if (w->batch_exec) cudaGraphExecDestroy(w->batch_exec);
                w->batch_exec = nullptr;
                w->batch_graph_key.clear();
                cudaGraph_t graph = nullptr;
                bool capturing = false;
                try {
                    GWB_CUDA(cudaStreamBeginCapture(s, cudaStreamCaptureModeRelaxed));
                    capturing = true;
                    int64_t n = prefix();
                    n += run_plan(0);
                    n += suffix();
                    capturing = false;
                    GWB_CUDA(cudaStreamEndCapture(s, &graph));
                    GWB_CUDA(cudaGraphInstantiate(&w->batch_exec, graph, 0));
                    cudaGraphDestroy(graph);
                    w->batch_graph_key = gkey;
                    w->batch_graph_launches = n;
                } catch (...) {
                    // not capturable here: remember, and issue this signature's launches one by one
                    if (capturing) {
                        cudaGraph_t g2 = nullptr;
                        cudaStreamEndCapture(s, &g2);
                        if (g2) cudaGraphDestroy(g2);
                    }
                    if (graph) cudaGraphDestroy(graph);
                    if (w->batch_exec) cudaGraphExecDestroy(w->batch_exec);
                    w->batch_exec = nullptr;
                    cudaGetLastError();
                    w->batch_graph_failed = gkey;
                }
            }
            if (w->batch_exec && gkey == w->batch_graph_key) {
                GWB_CUDA(cudaEventRecord(w->ev[0], s));
                GWB_CUDA(cudaGraphLaunch(w->batch_exec, s));
                GWB_CUDA(cudaEventRecord(w->ev[3], s));
                launches = w->batch_graph_launches;
                graphed = true;
            }
        }
        if (want_graph) w->batch_graph_seen = gkey;
        if (!graphed) {
            GWB_CUDA(cudaEventRecord(w->ev[0], s));
            launches += prefix();
            GWB_CUDA(cudaEventRecord(w->ev[1], s));
            if (cands.size() > 1) {  // time each candidate plan once, keep the fastest for this signature
                float best = std::numeric_limits<float>::infinity();
                for (size_t c = 0; c < cands.size(); ++c) {
                    GWB_CUDA(cudaEventRecord(w->ev[4], s));
                    run_plan(c);
                    GWB_CUDA(cudaEventRecord(w->ev[5], s));
                    GWB_CUDA(cudaEventSynchronize(w->ev[5]));
                    const float t = elapsed(w->ev[4], w->ev[5]);
                    if (t < best) {
                        best = t;
                        pick = c;
                    }
                }
                std::lock_guard<std::mutex> lk(g_batch_mu);
                g_batch_plans[key] = cands[pick];
            }
            GWB_CUDA(cudaEventRecord(w->ev[4], s));
            launches += run_plan(pick);
            GWB_CUDA(cudaEventRecord(w->ev[2], s));
            launches += suffix();
            GWB_CUDA(cudaEventRecord(w->ev[3], s));
        }
        st->kernel_launches = launches;
        // results and the pivot word back in one synchronisation
        w->stage_out.ensure(sizeof(unsigned long long) + nb_out);
        char* op = w->stage_out.as<char>();
        GWB_CUDA(cudaMemcpyAsync(op, w->in.p, sizeof(unsigned long long), cudaMemcpyDeviceToHost, s));
        GWB_CUDA(cudaMemcpyAsync(op + sizeof(unsigned long long), w->out.p, nb_out, cudaMemcpyDeviceToHost, s));
        GWB_CUDA(cudaStreamSynchronize(s));
        unsigned long long piv = 0;
        std::memcpy(&piv, op, sizeof(piv));
        if (piv == 0) fail(GWB200_DEVICE_TIMEOUT, "a device-side wait of the tcgen05 update expired; results discarded");
        if (piv != std::numeric_limits<unsigned long long>::max()) {
            st->info = (int64_t)piv;
            fail(GWB200_NOT_SPD, "eps(iw) of a batch member is not positive definite: Cholesky pivot " +
                                     std::to_string(piv) + " <= 0");
        }
        for (int64_t i = 0; i < nsys; ++i) {
            const gwb200_handle* h = hs[(size_t)i];
            const char* rows = op + sizeof(unsigned long long) + out_off[(size_t)i];
            if (sigma_out && sigma_out[i]) scatter_sigma(h, rows, states[i], nstates[i], fs[(size_t)i], sigma_out[i]);
            if (qp_out && qp_out[i])
                scatter_qp(h, rows + sizeof(double) * 2 * (size_t)nstates[i] * fs[(size_t)i], states[i], nstates[i], qp_out[i]);
        }
        double flops = 0.0;
        int64_t nmax = 0, mmax = 0;
        for (int64_t i = 0; i < nsys; ++i) {
            const double nd = (double)ns[(size_t)i], md = (double)ms[(size_t)i];
            flops += (double)fs[(size_t)i] * (nd * nd * nd / 3.0 + nd * nd * md + 3.0 * nd * md);
            nmax = std::max(nmax, ns[(size_t)i]);
            mmax = std::max(mmax, ms[(size_t)i]);
        }
        st->flops_screening = flops;
        st->frequency_chunks = (int64_t)chunks[pick].size();
        st->nph = nmax;
        st->ncols = mmax;
        st->device_ms_total = elapsed(w->ev[0], w->ev[3]);
        if (graphed) {  // one graph launch: no phase split, the whole sequence counts as screening
            st->device_ms_screening = st->device_ms_total;
        } else {
            st->device_ms_gather = elapsed(w->ev[0], w->ev[1]);
            st->device_ms_screening = elapsed(w->ev[4], w->ev[2]);
            st->device_ms_contract = elapsed(w->ev[2], w->ev[3]);
        }
        if (nbuckets_out) *nbuckets_out = (int64_t)cands[pick].size();
    });
}

int gwb200_kernel_profile(gwb200_handle* h, double* ms_out, double* bytes_out, int64_t* launches_out) {
    return guarded([&] {
        check_handle(h);
        if (!ms_out || !bytes_out || !launches_out) fail(GWB200_BAD_ARGUMENT, "null output array");
        GWB_CUDA(cudaStreamSynchronize(h->stream));
        for (auto& p : h->kprof_pending) {
            float t = 0.f;
            GWB_CUDA(cudaEventElapsedTime(&t, p.start, p.stop));
            h->kprof_ms[p.kind] += t;
            h->kprof_bytes[p.kind] += p.bytes;
            h->kprof_launches[p.kind] += 1;
        }
        kprof_release(h);
        for (int k = 0; k < 4; ++k) {
            ms_out[k] = h->kprof_ms[k];
            bytes_out[k] = h->kprof_bytes[k];
            launches_out[k] = h->kprof_launches[k];
            h->kprof_ms[k] = h->kprof_bytes[k] = 0.0;
            h->kprof_launches[k] = 0;
        }
    });
}

int gwb200_update_kernel(gwb200_handle* h, int64_t* kernel) {
    return guarded([&] {
        if (!h) fail(GWB200_BAD_ARGUMENT, "null gwb200_handle");
        if (!kernel) fail(GWB200_BAD_ARGUMENT, "null output");
        *kernel = h->last_update_kernel;
    });
}

} // extern "C"
