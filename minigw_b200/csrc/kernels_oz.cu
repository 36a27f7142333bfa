// kernels_oz.cu -- FP64 trailing update emulated on the int8 tensor cores (tcgen05 kind::i8).
//
// The plain form's dominant work is C -= P_r . P_c over the trailing lower part after each outer
// block of K = 128 columns, or two of them at once, K = 256 (FP64; kernels_fp64.cu runs it on the FP64
// DMMA pipe, 37 TFLOP/s peak).  Here each panel row P_r (K values) is written as
//     P_r[k] = c_r * sum_{s=1..6} D_s[r][k] 2^{-8 s} + (remainder of at most 2^-49 c_r),
// with c_r = 2^e j / 64 (j = 33 .. 65) the smallest such scale above 2.008 max_k |P_r[k]| and D_s the
// balanced 8-bit digits (-128 .. 127) of P_r[k] / c_r rounded to 48 bits.  The product of two rows is
//     P_r . P_c ~= c_r c_c sum_{l=2..7} 2^{-8 l} S_l,   S_l = sum_{s+t=l} D_s[r] . D_t[c],
// dropping the terms with s + t > 7 (2^-64 D D', of random sign).  Each S_l is an exact int32 sum of
// int8 products (|S_l| <= 6 * 2^14 * 256 < 2^25), accumulated by 21 int8 tensor-core products per
// 32-deep K step; the levels are combined exactly in integers into two parts, converted, joined with
// one FP64 rounding and scaled by c_r c_c (an exact product).  This is the Ozaki splitting scheme
// restated for row scales of few bits.  Error of the screened forms against 80-bit arithmetic, 500 to
// 1000 pairs: 0.5e-14 to 0.7e-14 (rms, relative) where 7-bit digits with levels up to 8 (26 products,
// power-of-two scales, K = 128) leave 3.4e-14 to 4.3e-14, and 10 to 19 times less than those on
// strongly coupled systems, whose digits reach further below the row maximum.  (Of the forms; the largest
// error of Sigma_c, 2e-14 to 9e-14 of it against 64 bits, comes from other steps and is the same with either.)
//
// K = 256 shares what a tile costs beside its MMAs -- reading 6 levels, integer and FP64 arithmetic,
// 64 KB added to C -- between twice as many of them: 200 orbitals x 64 frequencies 246 ms with K = 128
// and 7-bit digits, 213 with K = 256, 190 with 8-bit digits (two scale steps per octave more: 193).
//
// Two launches per update:
//   k_slice_panel64  one warp per panel row: c_r, and the 6 digit slices of the row's values, each
//                    slice of 128 values a 128-byte row in the 128-byte-swizzled K-major layout
//                    ([128 columns][slice][row][128 bytes]) the tensor core reads;
//   k_update64_oz    persistent, warp-specialised, one CTA per SM (10 warps, 214 KB of shared
//                    memory, 512 TMEM columns):
//                      warp 0     producer: units from a global counter handed on through a
//                                 4-slot mbarrier ring; loads the unit's A slices 5-6 (128 rows,
//                                 32 KB, resident for the unit) and streams the B slices (64
//                                 rows, 8 KB each) through a ring of seven pairs; K = 256: three
//                                 pairs, and four stages through which the second half's A
//                                 slices pass once per tile;
//                      warp 1     TMEM allocation; lane 0 issues tcgen05.mma kind::i8 (M = 128,
//                                 N = 64, K = 32 per instruction; A slices 1-4, which take part
//                                 in 18 of the 21 products, from TMEM (columns 384-511), the
//                                 others and B from shared memory) into 6 int32 accumulators,
//                                 one per level l (columns 64 (l - 2));
//                      warps 2-9  epilogue: at each unit start, write A slices 1-4 into TMEM;
//                                 per tile, warp w reads lane quadrant w % 4, 32 columns (16
//                                 columns per tcgen05.wait::ld), combines the levels, scales by
//                                 c_r c_c, stages -value per row (256 bytes) and adds it to C
//                                 with one bulk reduction (cp.reduce.async.bulk .add.f64) per row.
// The accumulators are drained in two level groups so that the tensor core does not wait for the
// whole drain: with K = 128 the MMAs of group X (levels 4-7, 18 of the 21 products) run first and are
// committed, then those of group Y (levels 2-3, 3 products).  The epilogue reads group X (keeping its
// exact sum per element) and releases it while group Y runs; the next tile's group X then runs while
// the epilogue reads group Y and finishes the tile.  (At N = 64 a tcgen05.mma kind::i8 costs ~48 cycles
// whatever its operands; 6 levels x 64 columns leave no room for a second accumulator buffer.)
// K = 256, per tile: half 0 with B pairs 3, 2, 1 and A as above; half 1 with A slices 1-4 against B
// pairs 3-2, which frees those two for the next tile, then all A slices against pair 1.
// A work unit is (frequency, 128-row tile i, up to kOzSeg column tiles of 64); column tile c of
// row tile i has work iff c < 2 (i + 1); rows are written from the column tile's first column
// (the diagonal 64 x 64 blocks in full, as the other update kernels do).  Every mbarrier wait is
// bounded as in kernels_tc.cu (expiry -> pivot 0 -> GWB200_DEVICE_TIMEOUT).
#include "internal.cuh"
#include "tc_common.cuh"

#include <cstdlib>

namespace gwb200 {
namespace {

using namespace tc;

constexpr int kOzM = 128;                    // accumulator rows = TMEM lanes
constexpr int kOzN = 64;                     // accumulator columns per level
constexpr int kOzSlices = 6;                 // digit slices per value
constexpr int kOzLevels = 6;                 // levels s + t = 2..7, one accumulator each
constexpr int kOzMaxSum = kOzLevels - 1;     // 0-based slice indices: products with sa + t <= 5
constexpr int kOzSeg = 32;                   // column tiles per work unit
constexpr int kOzStages = 7;                 // 16 KB stages: pairs of B slices, and with KH = 2 A slices (3-6)
constexpr int kOzTmemSlices = 4;             // A slices 1-4 (18 of the 21 products) read from TMEM
constexpr int kSchedSlots = 4;
constexpr int kSliceA = kOzM * 128;          // one slice of 128 rows: 16 KB
constexpr int kSliceB = kOzN * 128;          // of 64 rows: 8 KB
constexpr int kStageB = 2 * kSliceB;
constexpr int kEpiWarps = 8;                 // 4 lane quadrants x 2 column halves of 32
constexpr int kOzThreads = 32 * (2 + kEpiWarps);
constexpr int kTmemCols = 512;               // 6 levels x 64 columns, then A slices 1-4 (32 each)
constexpr int kTmemA = kOzLevels * kOzN;     // first column of the A slices held in TMEM
static_assert(kTmemA + 32 * kOzTmemSlices <= kTmemCols, "TMEM columns");
constexpr int kStgRow = 256 + 16;            // staging row stride: 32 doubles + 16 bytes (banks)
constexpr int kStgBytes = 32 * kStgRow;      // per epilogue warp
constexpr int kHeader = 1024;
constexpr int kOzSmem = kHeader + 1024 + (kOzSlices - kOzTmemSlices) * kSliceA + kOzStages * kStageB + kEpiWarps * kStgBytes;

constexpr int kOffFull = 0;
constexpr int kOffEmpty = kOffFull + 8 * kOzStages;
constexpr int kOffTFull = kOffEmpty + 8 * kOzStages;    // level group g (0 = X, 1 = Y) ready (tcgen05.commit)
constexpr int kOffTEmpty = kOffTFull + 16;              // group g drained (kEpiWarps arrivals)
constexpr int kOffAFull = kOffTEmpty + 16;              // A slices 5-6 of the unit in smem (tx bytes)
constexpr int kOffAEmpty = kOffAFull + 8;               // MMAs of the unit complete
constexpr int kOffATmem = kOffAEmpty + 8;               // A slices 1-4 in TMEM (kEpiWarps arrivals)
constexpr int kOffDrain = kOffATmem + 8;
constexpr int kOffUFull = kOffDrain + 8;
constexpr int kOffUEmpty = kOffUFull + 8 * kSchedSlots;
constexpr int kOffUnit = kOffUEmpty + 8 * kSchedSlots;
constexpr int kOffTmem = kOffUnit + 8 * kSchedSlots;
constexpr int kOffAbort = kOffTmem + 4;
static_assert(kOffAbort + 4 <= kHeader, "header overflow");
static_assert(kOzSmem <= 227 * 1024, "shared memory");

// Instruction descriptor, kind::i8: D S32 (bits 4-5 = 2), A and B signed 8-bit (bits 7-9,
// 10-12 = 1), both K-major, N >> 3 at bits 17-22, M >> 4 at bits 24-28.
constexpr uint32_t kIdescI8 = (2u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(kOzN >> 3) << 17) |
                              ((uint32_t)(kOzM >> 4) << 24);

__device__ __forceinline__ void mma_i8(uint32_t tmem_d, uint64_t da, uint64_t db, uint32_t accumulate) {
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::i8 [%0], %1, %2, %3, p;\n\t}" ::"r"(tmem_d),
        "l"(da), "l"(db), "r"(kIdescI8), "r"(accumulate)
        : "memory");
}

// A from TMEM (lane = row, 4 consecutive K bytes per 32-bit column), B from shared memory.
__device__ __forceinline__ void mma_i8_ts(uint32_t tmem_d, uint32_t tmem_a, uint64_t db, uint32_t accumulate) {
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::i8 [%0], [%1], %2, %3, p;\n\t}" ::"r"(tmem_d),
        "r"(tmem_a), "l"(db), "r"(kIdescI8), "r"(accumulate)
        : "memory");
}
__device__ __forceinline__ void tmem_st32u(uint32_t taddr, const uint32_t (&v)[32]) {
    asm volatile(
        "tcgen05.st.sync.aligned.32x32b.x32.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16,"
        "%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31,%32};" ::"r"(taddr),
        "r"(v[0]), "r"(v[1]), "r"(v[2]), "r"(v[3]), "r"(v[4]), "r"(v[5]), "r"(v[6]), "r"(v[7]), "r"(v[8]), "r"(v[9]),
        "r"(v[10]), "r"(v[11]), "r"(v[12]), "r"(v[13]), "r"(v[14]), "r"(v[15]), "r"(v[16]), "r"(v[17]), "r"(v[18]),
        "r"(v[19]), "r"(v[20]), "r"(v[21]), "r"(v[22]), "r"(v[23]), "r"(v[24]), "r"(v[25]), "r"(v[26]), "r"(v[27]),
        "r"(v[28]), "r"(v[29]), "r"(v[30]), "r"(v[31])
        : "memory");
}

__device__ __forceinline__ double pow2(int k) {  // 2^k for -1022 <= k <= 1023, exact
    return __longlong_as_double((long long)(k + 1023) << 52);
}

// Per frequency: 6 slices of rp rows x 128 bytes for each 128 columns (KH of them), then rp row scales.
__host__ __device__ constexpr size_t oz_freq_bytes(int64_t rp, int kh) {
    return ((size_t)kh * kOzSlices * rp * 128 + (size_t)rp * 8 + 1023) / 1024 * 1024;
}

template <int KH>
__global__ void __launch_bounds__(256) k_slice_panel64(const double* __restrict__ a, int64_t ld, int64_t stride,
                                                       int64_t kb0, int64_t c_begin, int64_t rows, int64_t rp,
                                                       uint8_t* __restrict__ buf) {
    const int f = blockIdx.y;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int64_t rr = (int64_t)blockIdx.x * 8 + warp;  // panel row
    if (rr >= rp) return;
    const int64_t r = c_begin + rr;
    uint8_t* slices = buf + (size_t)f * oz_freq_bytes(rp, KH);
    double* scales = reinterpret_cast<double*>(slices + (size_t)KH * kOzSlices * rp * 128);
    double x[KH][4] = {};
    if (r < rows) {
        const double* row = a + (size_t)f * stride + (size_t)r * ld + kb0 + 4 * lane;
#pragma unroll
        for (int h = 0; h < KH; ++h)
#pragma unroll
            for (int j = 0; j < 4; j += 2) {
                const double2 v = *reinterpret_cast<const double2*>(row + 128 * h + j);
                x[h][j] = v.x;
                x[h][j + 1] = v.y;
            }
    }
    double m = 0.0;
#pragma unroll
    for (int h = 0; h < KH; ++h)
#pragma unroll
        for (int j = 0; j < 4; ++j) m = fmax(m, fabs(x[h][j]));
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) m = fmax(m, __shfl_xor_sync(0xffffffffu, m, o));
    // the row scale 2^e k / 64, k = 33 .. 65, with |x| <= 0.498 of it, so that six digits of -128 .. 127
    // reach it (a power of two alone leaves half a bit of each row unused on average)
    // (a row below the normal range, whose scale and its inverse a double does not hold, counts as zero)
    double scale = 1.0, inv = 1.0;
    if (m >= 0x1p-1022) {
        int e;
        const double k = ceil(frexp(m, &e) * (64.0 / 0.996));
        scale = pow2(e) * (k * 0x1p-5);
        inv = pow2(-e) * (32.0 / k);
    }
    const uint32_t chunk = (uint32_t)(lane >> 2), in_chunk = (uint32_t)(lane & 3) * 4;
    const size_t pos = (size_t)((chunk ^ (uint32_t)(rr & 7)) * 16 + in_chunk);
#pragma unroll
    for (int h = 0; h < KH; ++h) {
        // the bytes of round(2^48 v) + 80 80 80 80 80 80 (v = x / scale) are its digits, plus 128
        uint32_t lo[4], hi[4];
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const long long u = __double2ll_rn(x[h][j] * inv * 0x1p48) + 0x808080808080LL;
            lo[j] = (uint32_t)u;
            hi[j] = (uint32_t)(u >> 32);
        }
        // byte b of the four values side by side
        const uint32_t l01 = __byte_perm(lo[0], lo[1], 0x5140), l23 = __byte_perm(lo[2], lo[3], 0x5140);
        const uint32_t m01 = __byte_perm(lo[0], lo[1], 0x7362), m23 = __byte_perm(lo[2], lo[3], 0x7362);
        const uint32_t h01 = __byte_perm(hi[0], hi[1], 0x5140), h23 = __byte_perm(hi[2], hi[3], 0x5140);
        const uint32_t word[kOzSlices] = {__byte_perm(h01, h23, 0x7632), __byte_perm(h01, h23, 0x5410),
                                          __byte_perm(m01, m23, 0x7632), __byte_perm(m01, m23, 0x5410),
                                          __byte_perm(l01, l23, 0x7632), __byte_perm(l01, l23, 0x5410)};
#pragma unroll
        for (int s = 0; s < kOzSlices; ++s)
            *reinterpret_cast<uint32_t*>(slices + ((size_t)(h * kOzSlices + s) * rp + rr) * 128 + pos) =
                word[s] ^ 0x80808080u;
    }
    if (lane == 0) scales[rr] = scale;
}

struct UnitSpace {
    int64_t T, NI, NS, per_f, total;
    int64_t row_min;  // panel rows above it are left alone (the next diagonal block's); row tiles from row_min / 128
};

// unit -> (frequency, row tile i, column tiles [c0, c1)); the longest row tiles first
__device__ __forceinline__ bool decode_unit(const UnitSpace& us, int64_t u, int& f, int64_t& i, int64_t& c0,
                                            int64_t& c1) {
    f = (int)(u / us.per_f);
    const int64_t rem = u - (int64_t)f * us.per_f;
    const int64_t q = rem / us.NS;
    i = us.NI - 1 - q;
    c0 = (rem - q * us.NS) * kOzSeg;
    c1 = min(c0 + kOzSeg, min(us.T, 2 * i + 2));
    return c0 < c1;
}

template <int KH>
__global__ void __launch_bounds__(kOzThreads, 1)
    k_update64_oz(double* __restrict__ a, int64_t ld, int64_t stride, int64_t c_begin, int64_t rows,
                  const uint8_t* __restrict__ buf, int64_t rp, UnitSpace us, unsigned long long* __restrict__ sched,
                  unsigned long long* err, int withhold_first_stage) {
    extern __shared__ __align__(1024) uint8_t osm[];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const uint32_t base = smem_u32(osm);
    const uint32_t abuf = (base + kHeader + 1023u) & ~1023u;  // A slices 5-6, 1024-aligned
    const uint32_t ring = abuf + (kOzSlices - kOzTmemSlices) * kSliceA;  // B stages, and with KH = 2 A slices
    const uint32_t stg0 = ring + kOzStages * kStageB;          // epilogue staging rows
    volatile uint32_t* abort_flag = reinterpret_cast<volatile uint32_t*>(osm + kOffAbort);
    volatile int64_t* uslot = reinterpret_cast<volatile int64_t*>(osm + kOffUnit);
    auto full = [&](int s) { return base + kOffFull + 8 * s; };
    auto empty = [&](int s) { return base + kOffEmpty + 8 * s; };
    auto ufull = [&](int j) { return base + kOffUFull + 8 * j; };
    auto uempty = [&](int j) { return base + kOffUEmpty + 8 * j; };
    auto tfull = [&](int g) { return base + kOffTFull + 8 * g; };
    auto tempty = [&](int g) { return base + kOffTEmpty + 8 * g; };
    const uint32_t afull = base + kOffAFull, aempty = base + kOffAEmpty, drain = base + kOffDrain;
    const uint32_t atmem = base + kOffATmem;

    if (threadIdx.x == 0) {
        for (int s = 0; s < kOzStages; ++s) {
            mbar_init(full(s), 1);
            mbar_init(empty(s), 1);
        }
        for (int j = 0; j < kSchedSlots; ++j) {
            mbar_init(ufull(j), 1);
            mbar_init(uempty(j), 1 + kEpiWarps);
        }
        for (int g = 0; g < 2; ++g) {
            mbar_init(tfull(g), 1);
            mbar_init(tempty(g), kEpiWarps);
        }
        mbar_init(afull, 1);
        mbar_init(atmem, kEpiWarps);
        mbar_init(aempty, 1);
        mbar_init(drain, 1);
        *abort_flag = 0u;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    }
    if (warp == 1) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(base + kOffTmem),
                     "r"(kTmemCols)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = *reinterpret_cast<volatile uint32_t*>(osm + kOffTmem);
    const size_t fbytes = oz_freq_bytes(rp, KH);

    if (warp == 0 && lane == 0) {
        // ---- producer (one thread: handing a stage over costs ~400 cycles, ~1,300 with the warp in step) ----
        int s = 0, js = 0;
        uint32_t ph = 0, aph = 0, jph = 0;
        uint32_t filled = 0, fill_par = 0;
        bool a_filled = false, ok = true;
        const size_t slice_bytes = (size_t)rp * 128;
        while (ok) {
            int f = 0;
            int64_t i = 0, c0 = 0, c1 = 0, u = 0;
            do {
                u = (int64_t)atomicAdd(sched, 1ull);
            } while (u < us.total && !decode_unit(us, u, f, i, c0, c1));
            if (u > us.total) u = us.total;
            if (!mbar_wait(uempty(js), jph ^ 1u, abort_flag, err)) break;
            uslot[js] = u;
            mbar_arrive(ufull(js));
            if (++js == kSchedSlots) {
                js = 0;
                jph ^= 1u;
            }
            if (u >= us.total) break;
            const uint8_t* slices = buf + (size_t)f * fbytes;
            if (!mbar_wait(aempty, aph ^ 1u, abort_flag, err)) break;
            mbar_expect_tx(afull, (uint32_t)((kOzSlices - kOzTmemSlices) * kSliceA));
            for (int j = kOzTmemSlices; j < kOzSlices; ++j)  // one 16 KB copy per smem slice
                bulk_g2s(abuf + (j - kOzTmemSlices) * kSliceA, slices + (size_t)j * slice_bytes + i * kSliceA, kSliceA, afull);
            a_filled = true;
            aph ^= 1u;
            // a stage's two 8 KB parts, once its reader is done with what it held
            auto load = [&](int st, uint32_t par, const uint8_t* s0, const uint8_t* s1) {
                if (!ok || !mbar_wait_fast(empty(st), par ^ 1u, abort_flag, err)) {
                    ok = false;
                } else if (withhold_first_stage && blockIdx.x == 0 && filled == 0) {
                    withhold_first_stage = 0;  // test of the bounded waits (see kernels_tc.cu)
                } else {
                    mbar_expect_tx(full(st), (uint32_t)kStageB);
                    bulk_g2s(ring + st * kStageB, s0, kSliceB, full(st));
                    bulk_g2s(ring + st * kStageB + kSliceB, s1, kSliceB, full(st));
                    filled |= 1u << st;
                    fill_par = (fill_par & ~(1u << st)) | (par << st);
                }
            };
            for (int64_t c = c0; ok && c < c1; ++c) {
                if constexpr (KH == 1) {
                    const uint8_t* src = slices + c * kSliceB;
                    for (int t = 0; ok && t < kOzSlices; t += 2, src += 2 * slice_bytes) {
                        load(s, ph, src, src + slice_bytes);
                        if (++s == kOzStages) {
                            s = 0;
                            ph ^= 1u;
                        }
                    }
                } else {
                    // stage q holds B pair 3 - q of a half, stages 3-6 the second half's A slices 1-4,
                    // stages 3-4 then its slices 5-6
                    auto load_b = [&](int64_t col, int h, int q) {
                        const uint8_t* src = slices + (size_t)(h * kOzSlices + 2 * (2 - q)) * slice_bytes + col * kSliceB;
                        load(q, (uint32_t)h, src, src + slice_bytes);
                    };
                    auto load_a = [&](int sa) {
                        const uint8_t* src = slices + (size_t)(kOzSlices + sa) * slice_bytes + i * kSliceA;
                        load(3 + (sa & 3), sa == 2 || sa == 3 ? ph : (uint32_t)(sa >> 2), src, src + kSliceB);
                    };
                    if (c == c0) {
                        load_b(c, 0, 0);
                        load_b(c, 0, 1);
                    }
                    load_b(c, 0, 2);
                    for (int sa = 0; sa < 4; ++sa) load_a(sa);
                    for (int q = 0; q < 3; ++q) load_b(c, 1, q);
                    if (c + 1 < c1) {
                        load_b(c + 1, 0, 0);
                        load_b(c + 1, 0, 1);
                    }
                    load_a(4);
                    load_a(5);
                    ph ^= 1u;  // one turn of stages 5-6 per tile (two of the others)
                }
            }
        }
        for (int q = 0; q < kOzStages; ++q)
            if (filled & (1u << q)) mbar_drain(full(q), (fill_par >> q) & 1u);
        if (a_filled) mbar_drain(afull, aph ^ 1u);
    } else if (warp == 1 && lane == 0) {
        // ---- MMA issuer ----
        const uint64_t desc_a0 = smem_desc_sw128(abuf), desc_b0 = smem_desc_sw128(ring);
        int s = 0, js = 0;
        uint32_t ph = 0, acc_ph = 0, aph = 0, jph = 0;
        bool issued = false, ok = true;
        for (;;) {
            const int64_t u = take_unit(ufull(js), uempty(js), uslot + js, jph, abort_flag, err);
            if (++js == kSchedSlots) {
                js = 0;
                jph ^= 1u;
            }
            if (u < 0 || u >= us.total) break;
            int f;
            int64_t i, c0, c1;
            decode_unit(us, u, f, i, c0, c1);
            if (!mbar_wait(afull, aph, abort_flag, err)) break;
            if (!mbar_wait(atmem, aph, abort_flag, err)) break;
            tc_fence_after();
            aph ^= 1u;
            // A slice sa+1 against B slice t+1 (of stage st) into level sa + t + 2, with t ascending: a
            // level's first product has t = 0 and starts the accumulator at kk = 0
            auto pair = [&](int sa, int t, int st) {
                // descriptors differ from the stage / A bases only in the address field (bytes >>
                // 4, below 2^14 for shared memory): constant offsets, no carries
                const uint64_t db0 = desc_b0 + (uint64_t)((uint32_t)(st * kStageB + (t & 1) * kSliceB) >> 4);
                const uint32_t d = tmem + (uint32_t)((sa + t) * kOzN);
                const bool starts = t == 0;
#pragma unroll
                for (int kk = 0; kk < 4; ++kk) {
                    const uint32_t acc = (!starts || kk > 0) ? 1u : 0u;
                    if (sa < kOzTmemSlices)  // A slice from TMEM: 32 bytes of K = 8 columns
                        mma_i8_ts(d, tmem + (uint32_t)(kTmemA + 32 * sa + 8 * kk), db0 + (uint64_t)(2 * kk), acc);
                    else
                        mma_i8(d, desc_a0 + (uint64_t)(((sa - kOzTmemSlices) * kSliceA + 32 * kk) >> 4),
                               db0 + (uint64_t)(2 * kk), acc);
                }
            };
            if constexpr (KH == 2) {
                // product (sa, t) of half h into level sa + t + 2; A of half 0 from TMEM or its resident
                // slices, of half 1 from stage 3 + (sa & 3); B pair t / 2 from stage 2 - t / 2
                auto product = [&](int h, int sa, int t) {
                    const uint64_t db = desc_b0 + (uint64_t)((uint32_t)((2 - t / 2) * kStageB + (t & 1) * kSliceB) >> 4);
                    const uint32_t d = tmem + (uint32_t)((sa + t) * kOzN);
                    // the first product of a level, in the order of half 0
                    const bool starts = h == 0 && sa < 2 && t % 2 == 0;
#pragma unroll
                    for (int kk = 0; kk < 4; ++kk) {
                        const uint32_t acc = (!starts || kk > 0) ? 1u : 0u;
                        if (h == 0 && sa < kOzTmemSlices)
                            mma_i8_ts(d, tmem + (uint32_t)(kTmemA + 32 * sa + 8 * kk), db + (uint64_t)(2 * kk), acc);
                        else if (h == 0)
                            mma_i8(d, desc_a0 + (uint64_t)(((sa - kOzTmemSlices) * kSliceA + 32 * kk) >> 4),
                                   db + (uint64_t)(2 * kk), acc);
                        else
                            mma_i8(d, desc_b0 + (uint64_t)(((3 + (sa & 3)) * kStageB + 32 * kk) >> 4),
                                   db + (uint64_t)(2 * kk), acc);
                    }
                };
                auto wait_b = [&](int h, int q) { return mbar_wait_fast(full(q), (uint32_t)h, abort_flag, err); };
                auto wait_a = [&](int sa) {
                    return mbar_wait_fast(full(3 + (sa & 3)), sa == 2 || sa == 3 ? ph : (uint32_t)(sa >> 2), abort_flag, err);
                };
                for (int64_t c = c0; ok && c < c1; ++c) {
                    // ---- half 0: B pairs 3, 2, 1 ----
                    ok = mbar_wait_fast(tempty(0), acc_ph ^ 1u, abort_flag, err);
#pragma unroll
                    for (int q = 0; q < 3; ++q) {
                        if (!ok || !wait_b(0, q)) {
                            ok = false;
                            break;
                        }
                        tc_fence_after();
                        issued = true;
#pragma unroll
                        for (int t = 2 * (2 - q); t < 2 * (2 - q) + 2; ++t)
#pragma unroll
                            for (int sa = 0; sa < kOzSlices; ++sa)
                                if (sa + t >= 2 && sa + t <= kOzMaxSum) product(0, sa, t);
                        if (q < 2) mma_commit(empty(q));
                    }
                    if (!ok || !mbar_wait_fast(tempty(1), acc_ph ^ 1u, abort_flag, err)) {
                        ok = false;
                        break;
                    }
                    tc_fence_after();
                    product(0, 0, 0);
                    product(0, 1, 0);
                    product(0, 0, 1);
                    mma_commit(empty(2));
                    // ---- half 1: A slices 1-4 against B pairs 3-2 while pair 1 arrives, then pair 1 ----
                    if (!wait_b(1, 0) || !wait_b(1, 1)) {
                        ok = false;
                        break;
                    }
#pragma unroll
                    for (int sa = 0; sa < 4; ++sa) {
                        if (!ok || !wait_a(sa)) {
                            ok = false;
                            break;
                        }
                        tc_fence_after();
#pragma unroll
                        for (int t = kOzMaxSum - sa; t >= 2; --t) product(1, sa, t);
                        if (sa == 1) mma_commit(empty(0));  // B slices 5-6 are done
                    }
                    mma_commit(empty(1));
                    if (!ok || !wait_b(1, 2)) {
                        ok = false;
                        break;
                    }
                    tc_fence_after();
#pragma unroll
                    for (int sa = 0; sa < kOzSlices; ++sa) {
                        if (sa >= 4 && (!ok || !wait_a(sa))) {
                            ok = false;
                            break;
                        }
                        tc_fence_after();
#pragma unroll
                        for (int t = sa < 5 ? 1 : 0; t >= 0; --t) product(1, sa, t);
                        mma_commit(empty(3 + (sa & 3)));
                    }
                    if (!ok) break;
                    mma_commit(empty(2));
                    mma_commit(tfull(0));
                    mma_commit(tfull(1));
                    acc_ph ^= 1u;
                    ph ^= 1u;
                }
            } else {
                for (int64_t c = c0; ok && c < c1; ++c) {
                    // group X (levels 4-7, sa + t >= 2) once the epilogue has read the previous tile's
                    if (!mbar_wait_fast(tempty(0), acc_ph ^ 1u, abort_flag, err)) {
                        ok = false;
                        break;
                    }
                    tc_fence_after();
                    const int s0 = s;  // B slices 1-2, held for group Y
#pragma unroll
                    for (int t2 = 0; t2 < kOzSlices; t2 += 2) {
                        if (!mbar_wait_fast(full(s), ph, abort_flag, err)) {
                            ok = false;
                            break;
                        }
                        tc_fence_after();
                        issued = true;
#pragma unroll
                        for (int t = t2; t < t2 + 2; ++t)
#pragma unroll
                            for (int sa = 0; sa < kOzSlices; ++sa)
                                if (sa + t >= 2 && sa + t <= kOzMaxSum) pair(sa, t, s);
                        if (t2 > 0) mma_commit(empty(s));
                        if (++s == kOzStages) {
                            s = 0;
                            ph ^= 1u;
                        }
                    }
                    if (!ok) break;
                    mma_commit(tfull(0));
                    // group Y (levels 2-3) once the epilogue has read the previous tile's
                    if (!mbar_wait_fast(tempty(1), acc_ph ^ 1u, abort_flag, err)) {
                        ok = false;
                        break;
                    }
                    tc_fence_after();
                    pair(0, 0, s0);
                    pair(1, 0, s0);
                    pair(0, 1, s0);
                    mma_commit(empty(s0));
                    mma_commit(tfull(1));
                    acc_ph ^= 1u;
                }
            }
            if (!ok) break;
            mma_commit(aempty);
        }
        if (issued) {
            mma_commit(drain);
            mbar_drain(drain, 0);
        }
    } else if (warp >= 2) {
        // ---- epilogue ----
        const int q = warp & 3, half = (warp - 2) >> 2;
        const uint32_t stg = stg0 + (uint32_t)(warp - 2) * kStgBytes + (uint32_t)lane * kStgRow;
        int js = 0;
        uint32_t acc_ph = 0, jph = 0, aph = 0;
        bool ok = true, reduced = false;
        while (ok) {
            int64_t u = 0;
            if (lane == 0) u = take_unit(ufull(js), uempty(js), uslot + js, jph, abort_flag, err);
            u = __shfl_sync(0xffffffffu, u, 0);
            if (++js == kSchedSlots) {
                js = 0;
                jph ^= 1u;
            }
            if (u < 0 || u >= us.total) break;
            int f;
            int64_t i, c0, c1;
            decode_unit(us, u, f, i, c0, c1);
            const uint8_t* slices = buf + (size_t)f * fbytes;
            const double* scales = reinterpret_cast<const double*>(slices + (size_t)KH * kOzSlices * rp * 128);
            const int64_t rr = i * kOzM + q * 32 + lane;  // panel row of this lane
            {   // A slices 1-4 of the unit into TMEM (warp half h writes slices h + 1 and h + 3 of its
                // lane quadrant) once the previous unit's MMAs are done with them
                uint32_t got = 1;
                if (lane == 0) got = mbar_wait(aempty, aph ^ 1u, abort_flag, err) ? 1u : 0u;
                got = __shfl_sync(0xffffffffu, got, 0);
                if (!got) break;
                aph ^= 1u;
                tc_fence_after();
#pragma unroll
                for (int sl = half; sl < kOzTmemSlices; sl += 2) {
                    const uint4* row = reinterpret_cast<const uint4*>(slices + ((size_t)sl * rp + rr) * 128);
                    uint32_t w[32];
#pragma unroll
                    for (int c = 0; c < 8; ++c) {  // undo the 128-byte swizzle of the slice row
                        const uint4 x = row[c ^ (int)(rr & 7)];
                        w[4 * c] = x.x;
                        w[4 * c + 1] = x.y;
                        w[4 * c + 2] = x.z;
                        w[4 * c + 3] = x.w;
                    }
                    tmem_st32u(tmem + ((uint32_t)(q * 32) << 16) + (uint32_t)(kTmemA + 32 * sl), w);
                }
                asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
                tc_fence_before();
                __syncwarp();
                if (lane == 0) mbar_arrive(atmem);
            }
            const int64_t r = c_begin + rr;
            const double row_scale = scales[rr] * -0x1p-56;
            for (int64_t c = c0; c < c1; ++c) {
                const int64_t cj = c_begin + c * kOzN + half * 32;  // this warp's first column
                const bool valid = r < rows && rr >= max(us.row_min, c * kOzN);
                const double2* sc = reinterpret_cast<const double2*>(scales + c * kOzN + half * 32);  // the columns' scales
                // Levels combined exactly: adjacent pairs S2 2^8 + S3 (|S2| <= 128^2 256, below 2^31), S4 2^8
                // + S5 and S6 2^8 + S7 (below 2^33), the latter two as one integer m of at most 49 bits (an
                // exact double between the groups); value = p23 2^-24 + m 2^-56 with one rounding, scaled
                // by c_r c_c.
                const uint32_t lanes = tmem + ((uint32_t)(q * 32) << 16) + (uint32_t)(half * 32);
                auto wait_group = [&](int g) {
                    uint32_t got = 1;
                    if (lane == 0) got = mbar_wait(tfull(g), acc_ph, abort_flag, err) ? 1u : 0u;
                    got = __shfl_sync(0xffffffffu, got, 0);
                    if (got) tc_fence_after();
                    return got != 0u;
                };
                auto release_group = [&](int g) {  // the group's levels are in registers
                    tc_fence_before();
                    __syncwarp();
                    if (lane == 0) mbar_arrive(tempty(g));
                };
                if (!wait_group(0)) {
                    ok = false;
                    break;
                }
                double m_d[32];
#pragma unroll
                for (int h16 = 0; h16 < 2; ++h16) {  // group X: levels 4-7, 16 columns per wait
                    uint32_t v[kOzLevels - 2][16];
#pragma unroll
                    for (int L = 2; L < kOzLevels; ++L) tmem_ld16_nowait(lanes + (uint32_t)(L * kOzN + 16 * h16), v[L - 2]);
                    tmem_wait_ld();
                    if (h16 == 1) release_group(0);
#pragma unroll
                    for (int j = 0; j < 16; ++j) {
                        const long long p45 = (long long)(int32_t)v[0][j] * 256 + (int32_t)v[1][j];
                        const long long p67 = (long long)(int32_t)v[2][j] * 256 + (int32_t)v[3][j];
                        m_d[16 * h16 + j] = (double)(p45 * (1LL << 16) + p67);  // exact
                    }
                }
                if (!wait_group(1)) {
                    ok = false;
                    break;
                }
                acc_ph ^= 1u;
#pragma unroll
                for (int h16 = 0; h16 < 2; ++h16) {  // group Y: levels 2-3, then the half's 16 columns to C
                    uint32_t v[2][16];
                    tmem_ld16_nowait(lanes + (uint32_t)(16 * h16), v[0]);
                    tmem_ld16_nowait(lanes + (uint32_t)(kOzN + 16 * h16), v[1]);
                    tmem_wait_ld();
                    if (h16 == 1) release_group(1);
                    // the staged row's last reduction has read it
                    if (h16 == 0 && reduced) asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory");
#pragma unroll
                    for (int j4 = 0; j4 < 4; ++j4) {
                        const double2 s0 = __ldg(sc + 8 * h16 + 2 * j4), s1 = __ldg(sc + 8 * h16 + 2 * j4 + 1);  // the same for every lane
                        const double sj[4] = {s0.x, s0.y, s1.x, s1.y};
                        double val[4];
#pragma unroll
                        for (int k = 0; k < 4; ++k) {
                            const int j = 4 * j4 + k;
                            const int32_t p23 = (int32_t)v[0][j] * 256 + (int32_t)v[1][j];
                            // (p23 2^32 + m) rounded once is 2^56 times the value rounded once: the
                            // 2^-56 is in row_scale
                            val[k] = fma((double)p23, 0x1p32, m_d[16 * h16 + j]) *
                                     (row_scale * sj[k]);  // an exact product
                        }
                        if (valid) {
                            const uint32_t dst = stg + (uint32_t)(128 * h16 + 32 * j4);
                            asm volatile("st.shared.v2.f64 [%0], {%1, %2};" ::"r"(dst), "d"(val[0]), "d"(val[1]) : "memory");
                            asm volatile("st.shared.v2.f64 [%0], {%1, %2};" ::"r"(dst + 16u), "d"(val[2]), "d"(val[3])
                                         : "memory");
                        }
                    }
                }
                // one bulk reduction per row: issuing one takes ~55 cycles per lane, whatever its size
                asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
                if (valid) {
                    double* dst = a + (size_t)f * stride + (size_t)r * ld + cj;
                    asm volatile("cp.reduce.async.bulk.global.shared::cta.bulk_group.add.f64 [%0], [%1], 256;" ::"l"(dst),
                                 "r"(stg)
                                 : "memory");
                    asm volatile("cp.async.bulk.commit_group;" ::: "memory");
                    reduced = true;
                }
            }
        }
        if (reduced) asm volatile("cp.async.bulk.wait_group 0;" ::: "memory");  // this lane's reductions done
    }
    tc_fence_before();
    __syncthreads();
    if (warp == 1) {
        __syncwarp();
        tc_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(kTmemCols) : "memory");
    }
}

} // namespace

size_t oz_slice_bytes_per_freq(const TallGeometry& g) { return oz_freq_bytes((g.rows + kOzM - 1) / kOzM * kOzM, 2); }

namespace {
template <int KH>
int launch_update(const TallGeometry& g, int64_t nf, double* a, int64_t kb0, int64_t c_begin, int64_t c_end,
                  void* slices, unsigned long long* sched, unsigned long long* err, cudaStream_t s, int max_ctas,
                  int64_t row_min) {
    const int64_t T = (c_end - c_begin) / kOzN;
    if (T <= 0 || nf <= 0) return 0;
    const int64_t H = g.rows - c_begin;
    const int64_t NI = (H + kOzM - 1) / kOzM, rp = NI * kOzM;
    uint8_t* buf = static_cast<uint8_t*>(slices);
    k_slice_panel64<KH><<<dim3((unsigned)(rp / 8), (unsigned)nf), 256, 0, s>>>(a, g.ld, g.stride, kb0, c_begin, g.rows,
                                                                              rp, buf);
    GWB_LAUNCH("k_slice_panel64");
    GWB_CUDA(cudaFuncSetAttribute(k_update64_oz<KH>, cudaFuncAttributeMaxDynamicSharedMemorySize, kOzSmem));
    UnitSpace us;
    us.T = T;
    us.NI = NI;
    us.NS = (T + kOzSeg - 1) / kOzSeg;
    us.per_f = (NI - row_min / kOzM) * us.NS;
    us.total = nf * us.per_f;
    us.row_min = row_min;
    const char* expire = std::getenv("GWB200_TEST_EXPIRE_WAIT");
    const int withhold = (expire && expire[0] == '1') ? 1 : 0;
    const unsigned grid = (unsigned)std::min<int64_t>(us.total, max_ctas > 0 ? std::min(max_ctas, sm_count()) : sm_count());
    k_update64_oz<KH><<<grid, kOzThreads, kOzSmem, s>>>(a, g.ld, g.stride, c_begin, g.rows, buf, rp, us, sched, err,
                                                         withhold);
    GWB_LAUNCH("k_update64_oz");
    return 2;
}
}  // namespace

int launch_update64_oz(const TallGeometry& g, int64_t nf, double* a, int64_t kb0, int64_t c_begin, int64_t c_end,
                       void* slices, unsigned long long* sched, unsigned long long* err, cudaStream_t s, int max_ctas,
                       int64_t row_min) {
    return c_begin - kb0 == 256 ? launch_update<2>(g, nf, a, kb0, c_begin, c_end, slices, sched, err, s, max_ctas, row_min)
                                : launch_update<1>(g, nf, a, kb0, c_begin, c_end, slices, sched, err, s, max_ctas, row_min);
}

} // namespace gwb200
