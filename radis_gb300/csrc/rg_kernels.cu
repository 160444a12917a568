// Device kernels of the LDM/DIT synthesis for sm_103a.
//
// Pipeline of one spectrum (radis/gpu/gpu.py:255-282 is the reference order):
//   k_scatter       fused per-line scaling + 2x2x2 scatter into a shared-memory
//                   LDM tile, flushed once to HBM with plain stores
//                   (replaces cmdFillLDM.comp:75-145 and the buffer clear)
//   k_col_fft_fwd, k_row_fft_voigt, k_col_ifft   the FFT stage (rg_fft.cu)
// Two real node rows a, b are transformed as one complex row z = a + i b.
// With W = V_a - i V_b, sum_j Z_j W_j = G and abscoeff = Re(IFFT(G)) / (N dv):
// the Hermitian pairing of bins k and N-k is absorbed by taking the real part.
#include <cuda_runtime.h>

#include <algorithm>
#include <atomic>
#include <cstdio>

#include "rg_device.cuh"

namespace rg {

// ---------------------------------------------------------------------------
// small helpers
// ---------------------------------------------------------------------------
__device__ __forceinline__ float lg2(float x) {
    float y;
    asm("lg2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}
// Knuth's TwoSum: s + e == a + b exactly.
__device__ __forceinline__ void two_sum(float a, float b, float& s, float& e) {
    s = a + b;
    float bb = s - a;
    e = (a - (s - bb)) + (b - bb);
}
// ---------------------------------------------------------------------------
// line preparation at upload: (hi, lo) split of v0 and log2 of the intensity
// ---------------------------------------------------------------------------
__global__ void k_prepare_lines(const double* __restrict__ v0, const double* __restrict__ s, int64_t n,
                                double c2_tref, float* __restrict__ vh, float* __restrict__ vl,
                                float* __restrict__ ls2, int* unsorted) {
    int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (i >= n) return;
    double v = v0[i];
    float hi = (float)v;
    float lo = (float)(v - (double)hi);
    vh[i] = hi;
    vl[i] = lo;
    double si = s[i];
    // log2 S_ref - log2(1 - exp(-c2 v0 / Tref)) : the stimulated-emission
    // denominator of base.py:2676 is constant per line
    double l = si > 0.0 ? log2(si) - log2(-expm1(-c2_tref * v)) : -INFINITY;
    ls2[i] = (float)l;
    if (i + 1 < n && v0[i + 1] < v) atomicExch(unsorted, 1);
}

// A position as v0 is stored (hi rounded to nearest, lo the rest) and the
// comparison "v0 < target" in FP32: hi decides unless equal, then lo against
// the rest of the target rounded up (exact for a float lo).  FP64 adds and
// compares would bound the searches (2 lanes per clock and SM on this part).
struct SplitTarget {
    float hi, lo;
};
__device__ __forceinline__ SplitTarget split_target(double t) {
    SplitTarget s;
    s.hi = __double2float_rn(t);
    s.lo = __double2float_ru(t - (double)s.hi);
    return s;
}
struct SplitList {   // a list's positions
    const float* __restrict__ hi;
    const float* __restrict__ lo;
};
__device__ __forceinline__ bool below(float hi, float lo, SplitTarget t) { return hi < t.hi || (hi == t.hi && lo < t.lo); }
__device__ __forceinline__ bool below(SplitList v, int64_t i, SplitTarget t) { return below(v.hi[i], v.lo[i], t); }

// First line index with v0 >= target, by one warp: 32 pivots per step, so a list
// of 10M lines takes 5 dependent loads instead of 24.
__device__ __forceinline__ int64_t warp_lower_bound(SplitList v0, int64_t n, SplitTarget target, int lane) {
    int64_t lo = 0, hi = n;   // the answer lies in [lo, hi]
    while (lo < hi) {
        // pivots lo <= p_0 <= ... <= p_31 < hi; v0 ascends, so the lanes below the target come first
        const int64_t p = lo + ((hi - lo) * lane >> 5);
        const int nb = __popc(__ballot_sync(0xffffffffu, below(v0, p, target)));
        const int64_t a = lo + ((hi - lo) * (nb - 1) >> 5), b = lo + ((hi - lo) * nb >> 5);
        if (nb == 0) return lo;
        if (nb < 32) hi = b;
        lo = a + 1;
    }
    return lo;
}

// First line index with v0 >= vmin + c dv, for c = c_min + idx.  Bound by the
// latency of dependent loads: a block finds the lines between its first and
// last column with two warps (above), and its threads search between them, in
// shared memory when they are few enough.  (One binary search of the whole
// list per column, compared in FP64: 76 us on 5M lines x 400 001 columns, 20 us on
// 600k lines x 116k columns, alone on a cold GPU; now 25 and 9.)
constexpr int kColStage = 2048;
__global__ void __launch_bounds__(256) k_col_index(SplitList v0, int64_t n, double vmin, double dv, int c_min, int count,
                                                   int64_t* __restrict__ col_start) {
    __shared__ int64_t ends[2];
    __shared__ float2 part[kColStage];
    const int idx = blockIdx.x * 256 + threadIdx.x;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    auto target_of = [&](int i) { return split_target(vmin + (double)(c_min + i) * dv); };
    if (warp < 2) {
        const int i = min((int)blockIdx.x * 256 + (warp ? 255 : 0), count - 1);
        const int64_t b = warp_lower_bound(v0, n, target_of(i), lane);
        if (lane == 0) ends[warp] = b;
    }
    __syncthreads();
    const int64_t first = ends[0];
    const int m = (int)min(ends[1] - first, (int64_t)0x7fffffff);
    const bool staged = m <= kColStage;
    if (staged) {
        for (int i = threadIdx.x; i < m; i += 256) part[i] = make_float2(v0.hi[first + i], v0.lo[first + i]);
        __syncthreads();
    }
    if (idx >= count) return;
    const SplitTarget target = target_of(idx);
    int64_t lo = first, hi = ends[1];
    if (staged) {
        int l = 0, h = m;
        while (l < h) {
            const int mid = (l + h) >> 1;
            if (below(part[mid].x, part[mid].y, target))
                l = mid + 1;
            else
                h = mid;
        }
        lo = first + l;
    } else {
        while (lo < hi) {   // eight parts per step: seven independent loads
            const int64_t span = hi - lo;
            int nb = 0;
#pragma unroll
            for (int i = 1; i < 8; ++i) nb += below(v0, lo + (span * i >> 3), target);
            const int64_t a = lo + (span * nb >> 3), b = lo + (span * (nb + 1) >> 3);
            if (nb < 7) hi = b;   // v0[b] is not below the target
            if (nb > 0)
                lo = a + 1;          // v0[a] is
            else if (span < 8) {     // the first part may be empty: look at lo itself
                if (below(v0, lo, target))
                    ++lo;
                else
                    hi = lo;
            }
        }
    }
    col_start[idx] = lo;
}

// most lines with v0 in columns [c - 1 - E, c + 1 + E) over the grid columns
__global__ void k_col_cmax(const int64_t* __restrict__ col_start, int col_off, int col_count, int n_v, int E,
                           int* __restrict__ cmax) {
    int m = 0;
    for (int c = blockIdx.x * blockDim.x + threadIdx.x; c < n_v; c += gridDim.x * blockDim.x) {
        const int lo = max(0, min(c - 1 - E + col_off, col_count - 1));
        const int hi = max(0, min(c + 1 + E + col_off, col_count - 1));
        m = max(m, (int)min(col_start[hi] - col_start[lo], (int64_t)0x3fffffff));
    }
    for (int o = 16; o; o >>= 1) m = max(m, __shfl_xor_sync(0xffffffffu, m, o));
    if ((threadIdx.x & 31) == 0 && m) atomicMax(cmax, m);
}

// ---------------------------------------------------------------------------
// K1: fused line scaling + LDM scatter into a shared-memory tile
// ---------------------------------------------------------------------------
// A tile holds only the node rows that its lines can reach.  The Gaussian
// width is proportional to v0, so the lines of a few hundred columns lie
// between two neighbouring Gaussian nodes, or around one: two or three of the
// grid's Gaussian rows times all Lorentzian ones, from row l_base on.  (Tiles
// of every node: 128 rows instead of 32-48 on the 8 x 16 grid, 288 instead of
// 48-72 on 12 x 24; with them went 3-4 times the flush work and, on the larger
// grid, 1.7 GB of zeros written and read back per spectrum.)  Row pitch 4 (mod
// 32) words: the flush's fragment loads (4 nodes two apart x 8 columns) touch
// 32 banks, and the nodes of one column eight.

// --- TMA (cp.async.bulk) + mbarrier helpers ---------------------------------
__device__ __forceinline__ uint32_t smem_u32(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }

__device__ __forceinline__ void mbar_init(uint64_t* bar, uint32_t count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count) : "memory");
}
__device__ __forceinline__ void mbar_expect_tx(uint64_t* bar, uint32_t bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)), "r"(bytes)
                 : "memory");
}
__device__ __forceinline__ void tma_load_1d(void* dst, const void* src, uint32_t bytes, uint64_t* bar) {
    asm volatile(
        "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
            smem_u32(dst)),
        "l"(src), "r"(bytes), "r"(smem_u32(bar))
        : "memory");
}
// The thread may stay suspended inside try_wait until the phase completes or
// the hint (ns) runs out, so waiting warps do not spin on the issue slots.
__device__ __forceinline__ bool mbar_try_wait(uint64_t* bar, uint32_t parity) {
    constexpr uint32_t kSuspendHintNs = 1000000;
    uint32_t ok;
    asm volatile(
        "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2, %3;\n selp.u32 %0, 1, 0, p;\n}\n"
        : "=r"(ok)
        : "r"(smem_u32(bar)), "r"(parity), "n"(kSuspendHintNs)
        : "memory");
    return ok != 0;
}
__device__ __forceinline__ void mbar_arrive(uint64_t* bar) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(bar)) : "memory");
}
// Bounded wait (`limit` SM clock cycles); false when it gives up.
__device__ __forceinline__ bool mbar_wait(uint64_t* bar, uint32_t parity, long long limit = kScatWaitCycles) {
    if (mbar_try_wait(bar, parity)) return true;
    const long long t0 = clock64();
    for (;;) {   // the clock every 16 tries: the waiting warps share the issue slots
#pragma unroll 1
        for (int i = 0; i < 16; ++i)
            if (mbar_try_wait(bar, parity)) return true;
        if (clock64() - t0 > limit) return false;
    }
}

// One thread: copy lines [start, start + count) of every column into a stage
// buffer (16-line granularity: the arrays are padded to a multiple of 16).
__device__ __forceinline__ void issue_chunk(const ScatterArgs& a, unsigned char* base, uint64_t* bar, int start,
                                            int count) {
    const uint32_t cp = (uint32_t)((count + kLinePad - 1) / kLinePad * kLinePad);
    const int ch = a.chunk;
    // the buffer was last read through the generic proxy
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    mbar_expect_tx(bar, cp * (28 + (a.dl ? 4 : 0) + (a.iso ? 1 : 0)));
    tma_load_1d(base, a.vh + start, cp * 4, bar);
    tma_load_1d(base + 4 * ch, a.vl + start, cp * 4, bar);
    tma_load_1d(base + 8 * ch, a.ls2 + start, cp * 4, bar);
    tma_load_1d(base + 12 * ch, a.el + start, cp * 4, bar);
    tma_load_1d(base + 16 * ch, a.ga + start, cp * 4, bar);
    tma_load_1d(base + 20 * ch, a.gs + start, cp * 4, bar);
    tma_load_1d(base + 24 * ch, a.na + start, cp * 4, bar);
    if (a.dl) tma_load_1d(base + 28 * ch, a.dl + start, cp * 4, bar);
    if (a.iso) tma_load_1d(base + (a.dl ? 32 : 28) * ch, a.iso + start, cp, bar);
}

// TF32 operands (round to nearest, ties away) and mma.sync m16n8k8 with FP32
// accumulators: a[0..3] = A (row g, col t), (g + 8, t), (g, t + 4),
// (g + 8, t + 4); b0, b1 = B (row t, col g), (t + 4, g); d = (g, 2t), (g, 2t
// + 1), (g + 8, 2t), (g + 8, 2t + 1), with g = lane / 4, t = lane % 4.
// TF32 rounding to nearest, ties away from zero (the rna mode) on the bit
// pattern: half a TF32 unit (bit 12) added to the magnitude bits, the 13 low
// mantissa bits cleared; a carry out of the mantissa bumps the exponent, as
// rounding up must.  Two integer instructions; finite inputs only (the
// operands here are sums of finite line contributions).
__device__ __forceinline__ uint32_t tf32_rna(float x) { return (__float_as_uint(x) + 0x1000u) & 0xFFFFE000u; }
__device__ __forceinline__ void mma_tf32(float (&d)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
    asm volatile("mma.sync.aligned.m16n8k8.row.col.f32.tf32.tf32.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, "
                 "{%0,%1,%2,%3};"
                 : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
                 : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}

// --- per-line quantities at the conditions of a ScatterArgs -----------------
// (shared by the scatter, the tangent scatter and the adjoint gather)

// Fractional grid position of the (pressure-shifted) line centre, in
// double-float: ((hi - vmin_hi) + (lo - vmin_lo + shift)) / dv = fk + tv,
// fk integral, tv in [0, 1).
__device__ __forceinline__ void line_position(const ScatterArgs& a, float2 v, float dl, float& fk, float& tv) {
    float s, e1;
    two_sum(v.x, -a.vmin_hi, s, e1);
    e1 += (v.y - a.vmin_lo) + dl * a.p_atm;
    const float p = s * a.inv_dv_hi;
    const float pe = fmaf(s, a.inv_dv_hi, -p) + fmaf(s, a.inv_dv_lo, e1 * a.inv_dv_hi);
    fk = floorf(p);
    tv = (p - fk) + pe;
    const float fl = floorf(tv);
    fk += fl;
    tv -= fl;
}

// Gaussian / Lorentzian node cell and fractions (FWHM, log space); log v0 is
// taken relative to v_ref so the FP32 log and offset do not cancel.
__device__ __forceinline__ void line_nodes(const ScatterArgs& a, float v0, float ga, float gs, float na, int is,
                                           int& l0, int& m0, float& tG, float& tL) {
    const float pl = fmaf(lg2(v0 * a.inv_vref), a.lgG_scale, a.cG[is]);
    const float gam = fmaf(a.x_self, gs - ga, ga);
    const float pm = fmaf(lg2(gam), a.lgL_scale, fmaf(na, a.tL, a.cL));
    l0 = min(max((int)floorf(pl), 0), a.NG - 2);
    m0 = min(max((int)floorf(pm), 0), a.NL - 2);
    tG = pl - (float)l0;
    tL = pm - (float)m0;
}

// Scaled intensity S(T) N x Qr exp(-log_scale): exponent log2(S') + a_T El +
// b_iso in double-float, times the stimulated-emission factor.
__device__ __forceinline__ float line_intensity(const ScatterArgs& a, float v0, float el, float ls2, int is) {
    const float ph = el * a.aT_hi;
    const float pe2 = fmaf(el, a.aT_hi, -ph) + el * a.aT_lo;
    float s1, f1, s2, f2;
    two_sum(ph, a.bI_hi[is], s1, f1);
    two_sum(s1, ls2, s2, f2);
    const float arg = s2 + (f1 + f2 + pe2 + a.bI_lo[is]);
    return ex2(arg) * (1.f - ex2(-a.stim_c * v0));
}

// Fixed-point accumulators of the tile: 32-bit words, or 64-bit sums for dense
// columns (see fx_wide) held as two planes of 32-bit words `hi_off` words
// apart.  Shared memory has native 32-bit integer adds only (a 64-bit
// atomicAdd runs as a compare-and-swap loop: 6.6 rounds per add on a band core
// of 2400 lines per column), so a 64-bit add is a native add of the low word
// and one of the high word plus the carry that the old low word tells, left
// out when it is zero.  Integer sums: exact and order-independent.
template <bool W> struct Fx;
template <> struct Fx<false> {
    static constexpr int kWidth = 31;
    // the 8 cells of a line: columns c and c + 1 of rows 0, 1, dg, dg + 1 (in pitches)
    __device__ static void add8(unsigned* t, int pitch, int dg, int, const float (&a)[4], const float (&b)[4]) {
        unsigned* row[4] = {t, t + pitch, t + dg, t + dg + pitch};
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            atomicAdd(row[i], __float2uint_rn(a[i]));
            atomicAdd(row[i] + 1, __float2uint_rn(b[i]));
        }
    }
    __device__ static float value(const unsigned* t, int) { return __uint2float_rn(*t); }
};
template <> struct Fx<true> {
    static constexpr int kWidth = 63;
    // all low words first: the old values come back while the next adds go out
    __device__ static void add8(unsigned* t, int pitch, int dg, int hi_off, const float (&a)[4], const float (&b)[4]) {
        unsigned* row[4] = {t, t + pitch, t + dg, t + dg + pitch};
        unsigned hi[8], lo[8], old[8];
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            const unsigned long long u = __float2ull_rn(i & 1 ? b[i >> 1] : a[i >> 1]);
            lo[i] = (unsigned)u;
            hi[i] = (unsigned)(u >> 32);
            old[i] = atomicAdd(row[i >> 1] + (i & 1), lo[i]);
        }
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            hi[i] += old[i] + lo[i] < lo[i] ? 1u : 0u;
            if (hi[i]) atomicAdd(row[i >> 1] + (i & 1) + hi_off, hi[i]);
        }
    }
    __device__ static float value(const unsigned* t, int hi_off) {
        return __ull2float_rn(((unsigned long long)t[hi_off] << 32) | *t);
    }
};

// --- the same on two lines per thread ----------------------------------------
// Packed FP32 (fadd2 / ffma2): a pair of lines costs the issue slots of one.
__device__ __forceinline__ float2 neg2(float2 a) { return make_float2(-a.x, -a.y); }
__device__ __forceinline__ float2 dup2(float x) { return make_float2(x, x); }
__device__ __forceinline__ float2 sub2(float2 a, float2 b) { return __fadd2_rn(a, neg2(b)); }
__device__ __forceinline__ void two_sum2(float2 a, float2 b, float2& s, float2& e) {
    s = __fadd2_rn(a, b);
    const float2 bb = sub2(s, a);
    e = __fadd2_rn(sub2(a, sub2(s, bb)), sub2(b, bb));
}
// floor for |x| < 2^22: 1.5 2^23 + x rounded down has ulp 1.  From 2^22 to
// 2^24 the result is the even number below (a position's fraction is floored
// once more); values beyond stay out of every window.
__device__ __forceinline__ float2 floor2(float2 x) {
    const float m = 12582912.f;
    return __fadd2_rn(__fadd2_rd(x, dup2(m)), dup2(-m));
}
__device__ __forceinline__ float2 clamp2(float2 x, float lo, float hi) {
    return make_float2(fminf(fmaxf(x.x, lo), hi), fminf(fmaxf(x.y, lo), hi));
}

// What a tile's lines need of it.
struct TileView {
    float k_start, k_lo, k_hi;   // first column; positions whose line touches the tile's columns
    float l_lo, l_hi;            // Gaussian cells (l0) of its lines
    int l_base, l_rows;          // first Gaussian row, rows in use
};
__device__ __forceinline__ TileView tile_view(const ScatterArgs& a, int tile) {
    TileView t;
    const int k0 = tile * a.TK, tk = min(a.TK, a.n_v - k0);
    t.k_start = (float)k0;
    t.k_lo = (float)max(k0 - 1, 0);
    t.k_hi = (float)min(k0 + tk - 1, a.n_v - 2);   // dropped beyond (cmdFillLDM.comp:102)
    // Gaussian coordinates of the first and last line position, with room for rounding
    const float va = fmaxf(fmaf((float)(k0 - 1 - a.margin_cols), a.v_step, a.v_lo), a.v_bot);
    const float vb = fmaxf(fmaf((float)(k0 + tk + a.margin_cols), a.v_step, a.v_lo), a.v_bot);
    const float pa = fmaf(lg2(va * a.inv_vref), a.lgG_scale, a.cG_lo) - 0.05f;
    const float pb = fmaf(lg2(vb * a.inv_vref), a.lgG_scale, a.cG_hi) + 0.05f;
    const float lb = fminf(fmaxf(floorf(pa), 0.f), (float)(a.NG - a.win));
    const float le = fminf(fmaxf(floorf(pb), lb), lb + (float)(a.win - 2));
    t.l_lo = lb;
    t.l_hi = le;
    t.l_base = (int)lb;
    t.l_rows = (int)(le - lb) + 2;
    return t;
}

// Lines 2p and 2p + 1 of a staged chunk (`two`: the second exists) into the
// tile accumulator (`tile`: this lane's copy).  A line one column left of the
// tile or on its last column also adds to a word beyond that column: padding
// that nothing reads.  Returns the lines that count as the tile's.
template <bool W>
__device__ __forceinline__ unsigned scatter_pair(const ScatterArgs& a, const TileView& tv, const unsigned char* st, int p,
                                                 bool two, unsigned* tile, float fxs) {
    const LinePairs& k = a.k2;
    const int ch4 = 4 * a.chunk;
    const unsigned char* q = st + 8 * p;
    auto col = [&](int i) { return *reinterpret_cast<const float2*>(q + i * ch4); };
    const float2 vh = col(0);
    // position (line_position)
    float2 s, e;
    two_sum2(vh, k.neg_vmin_hi, s, e);
    float2 t = sub2(col(1), k.vmin_lo);
    if (a.dl) t = __ffma2_rn(col(7), k.p_atm, t);
    e = __fadd2_rn(e, t);
    const float2 pos = __fmul2_rn(s, k.inv_dv_hi);
    const float2 pe = __fadd2_rn(__ffma2_rn(s, k.inv_dv_hi, neg2(pos)), __ffma2_rn(s, k.inv_dv_lo, __fmul2_rn(e, k.inv_dv_hi)));
    float2 fk = floor2(pos);
    float2 f = __fadd2_rn(sub2(pos, fk), pe);
    const float2 fl = floor2(f);
    fk = __fadd2_rn(fk, fl);
    f = sub2(f, fl);
    const bool ok0 = fk.x >= tv.k_lo && fk.x <= tv.k_hi;
    const bool ok1 = two && fk.y >= tv.k_lo && fk.y <= tv.k_hi;
    if (!(ok0 || ok1)) return 0;
    // nodes (line_nodes)
    float2 cG = k.cG, bh = k.bI_hi, bl = k.bI_lo;
    if (a.iso) {
        const unsigned char* is = st + (a.dl ? 8 : 7) * ch4 + 2 * p;
        const int i0 = is[0], i1 = two ? is[1] : i0;
        cG = make_float2(a.cG[i0], a.cG[i1]);
        bh = make_float2(a.bI_hi[i0], a.bI_hi[i1]);
        bl = make_float2(a.bI_lo[i0], a.bI_lo[i1]);
    }
    const float2 xv = __fmul2_rn(vh, k.inv_vref);
    const float2 pl = __ffma2_rn(make_float2(lg2(xv.x), lg2(xv.y)), k.lgG_scale, cG);
    const float2 ga = col(4);
    const float2 gam = __ffma2_rn(k.x_self, sub2(col(5), ga), ga);
    const float2 pm = __ffma2_rn(make_float2(lg2(gam.x), lg2(gam.y)), k.lgL_scale, __ffma2_rn(col(6), k.tL, k.cL));
    const float2 l0 = clamp2(floor2(pl), tv.l_lo, tv.l_hi);
    const float2 m0 = clamp2(floor2(pm), 0.f, (float)(a.NL - 2));
    const float2 tG = sub2(pl, l0), tL = sub2(pm, m0);
    const float2 row = __ffma2_rn(sub2(l0, dup2(tv.l_lo)), k.n_l, m0);
    const float2 at = __ffma2_rn(row, dup2((float)a.pitch), sub2(fk, dup2(tv.k_start)));
    // intensity (line_intensity), in accumulator units
    const float2 el = col(3);
    const float2 ph = __fmul2_rn(el, k.aT_hi);
    const float2 pe2 = __ffma2_rn(el, k.aT_lo, __ffma2_rn(el, k.aT_hi, neg2(ph)));
    float2 s1, f1, s2, f2;
    two_sum2(ph, bh, s1, f1);
    two_sum2(s1, col(2), s2, f2);
    const float2 arg = __fadd2_rn(s2, __fadd2_rn(__fadd2_rn(__fadd2_rn(f1, f2), pe2), bl));
    const float2 xs = __fmul2_rn(vh, k.stim);
    const float2 em = sub2(dup2(1.f), make_float2(ex2(-xs.x), ex2(-xs.y)));
    const float2 I = __fmul2_rn(__fmul2_rn(make_float2(ex2(arg.x), ex2(arg.y)), em), dup2(fxs));
    // weights
    const float2 I1 = __fmul2_rn(f, I), I0 = sub2(I, I1);
    const float2 w11 = __fmul2_rn(tG, tL);
    const float2 w10 = sub2(tG, w11);                  // tG (1 - tL)
    const float2 w01 = sub2(tL, w11);                  // (1 - tG) tL
    const float2 w00 = sub2(sub2(dup2(1.f), tG), w01);   // (1 - tG)(1 - tL)
    const float2 a00 = __fmul2_rn(I0, w00), a01 = __fmul2_rn(I0, w01), a10 = __fmul2_rn(I0, w10), a11 = __fmul2_rn(I0, w11);
    const float2 b00 = __fmul2_rn(I1, w00), b01 = __fmul2_rn(I1, w01), b10 = __fmul2_rn(I1, w10), b11 = __fmul2_rn(I1, w11);
    const int pitch = a.pitch, dG = a.NL * pitch, hi_off = a.rows * pitch;
    if (ok0) {
        const float x0[4] = {a00.x, a01.x, a10.x, a11.x}, x1[4] = {b00.x, b01.x, b10.x, b11.x};
        Fx<W>::add8(tile + __float2int_rn(at.x), pitch, dG, hi_off, x0, x1);
    }
    if (ok1) {
        const float x0[4] = {a00.y, a01.y, a10.y, a11.y}, x1[4] = {b00.y, b01.y, b10.y, b11.y};
        Fx<W>::add8(tile + __float2int_rn(at.y), pitch, dG, hi_off, x0, x1);
    }
    return a.in_window ? (ok0 && fk.x >= tv.k_start) + (ok1 && fk.y >= tv.k_start) : 0u;
}

// Columns [c, c + NC) of a finished tile, by one warp.
// Sum of the tile's copies into the first (integer sums: exact), the others zeroed.
template <bool W, int NC>
__device__ __forceinline__ void fold_copies(const ScatterArgs& a, unsigned* tile, int c, int rows, int lane) {
    const int hi_off = a.rows * a.pitch;
    for (int i = lane; i < rows * NC; i += 32) {
        unsigned* w = tile + (i / NC) * a.pitch + c + i % NC;
        unsigned long long s = 0;
        for (int q = 0; q < a.copies; ++q, w += a.copy_words) {
            s += W ? ((unsigned long long)w[hi_off] << 32) | w[0] : w[0];
            w[0] = 0;
            if (W) w[hi_off] = 0;
        }
        w -= a.copies * a.copy_words;
        w[0] = (unsigned)s;
        if (W) w[hi_off] = (unsigned)(s >> 32);
    }
    __syncwarp();
}
template <bool W, int NC>
__device__ __forceinline__ void zero_columns(const ScatterArgs& a, unsigned* tile, int c, int rows, int lane) {
    __syncwarp();
    for (int i = lane; i < rows * (NC / 4); i += 32) {
        unsigned* w = tile + (i / (NC / 4)) * a.pitch + c + 4 * (i % (NC / 4));
        *reinterpret_cast<uint4*>(w) = make_uint4(0u, 0u, 0u, 0u);
        if (W) *reinterpret_cast<uint4*>(w + a.rows * a.pitch) = make_uint4(0u, 0u, 0u, 0u);
        else if (a.copies == 2) {   // (the second copy is not 16-byte aligned)
            w += a.copy_words;
            w[0] = w[1] = w[2] = w[3] = 0u;
        }
    }
}

// Coefficients of eight nodes from `node` on, rows 8 nr .. 8 nr + 7, as one
// lane's B fragment (the window's padding rows hold zeros: any coefficient does).
__device__ __forceinline__ float4 proj_frag(const ScatterArgs& a, int nr, int node, int lane) {
    const float2* p = a.proj + ((nr * a.proj_np + min(node + 2 * (lane & 3), a.proj_np - 2)) << 3) + (lane >> 2);
    const float2 u = __ldg(p), v = __ldg(p + 8);
    return make_float4(u.x, u.y, v.x, v.y);
}

// Skeleton rows of 16 columns on the tensor cores: Y^T[columns x rows] =
// T^T[columns x nodes] C^T[nodes x rows] with mma.sync m16n8k8 TF32, each
// product split into three (hi hi + lo hi + hi lo; x = hi + lo, hi = tf32(x),
// lo = tf32(x - hi)): columns as M, the NR row blocks of 8 as N, the tile's
// nodes as K, eight per step (past the rows in use the tile holds zeros); k =
// t, t + 4 are nodes 2 t, 2 t + 1 of a step, 8 banks apart.  Two sums per
// output keep the chains of dependent MMAs short.  frag: the coefficients of
// the tile's nodes as B fragments, [step][row block][lane] (node 2 t hi, lo,
// node 2 t + 1 hi, lo), in shared memory (through L1 the reads missed: a
// third of the 5M-line scatter's time), where it has the room (kFrags).
template <bool W, int NR, bool kFrags>
__device__ __forceinline__ void project_columns(const ScatterArgs& a, int steps, int first, const unsigned* tile,
                                                const float4* frag, int c, int nr0, int k_start, int tk, float inv_fx,
                                                int lane) {
    const int g = lane >> 2, t = lane & 3;
    const int hi_off = a.rows * a.pitch;
    const bool two = !W && a.copies == 2;   // two copies are added up here, more by fold_copies
    const unsigned* col = tile + 2 * t * a.pitch + c + g;
    const float4* cf = frag + nr0 * 32 + lane;
    float d[NR][4], e[NR][4];
#pragma unroll
    for (int nr = 0; nr < NR; ++nr)
#pragma unroll
        for (int i = 0; i < 4; ++i) d[nr][i] = e[nr][i] = 0.f;
#pragma unroll 2
    for (int s = 0; s < steps; ++s, col += 8 * a.pitch, cf += 32 * a.proj_nr) {
        const unsigned* p[4] = {col, col + 8, col + a.pitch, col + a.pitch + 8};
        {   // Leave out nodes and columns that hold nothing: 0 x coefficient.  A
            // line fills 4 of a window's nodes, so in a 5M-line list of 12 lines
            // per column and in sparser ones many steps are empty (spectrum 114 ->
            // 108 us; 0.03 lines per column 41.2 -> 38.8, 100M lines 1214 -> 1164 us).
            // Loading the next step's words before this one's MMAs as well: 117 us.
            unsigned any = p[0][0] | p[1][0] | p[2][0] | p[3][0];
            if (W) any |= p[0][hi_off] | p[1][hi_off] | p[2][hi_off] | p[3][hi_off];
            if (two) any |= p[0][a.copy_words] | p[1][a.copy_words] | p[2][a.copy_words] | p[3][a.copy_words];
            if (!__any_sync(0xffffffffu, any)) continue;
        }
        float4 b[NR];
#pragma unroll
        for (int nr = 0; nr < NR; ++nr) b[nr] = kFrags ? cf[nr * 32] : proj_frag(a, nr0 + nr, first + 8 * s, lane);
        uint32_t ah[4], al[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            float v;
            if constexpr (W) v = Fx<W>::value(p[i], hi_off);
            else v = __uint2float_rn(two ? p[i][0] + p[i][a.copy_words] : p[i][0]);
            ah[i] = tf32_rna(v);
            al[i] = tf32_rna(v - __uint_as_float(ah[i]));
        }
#pragma unroll
        for (int nr = 0; nr < NR; ++nr) mma_tf32(e[nr], al, __float_as_uint(b[nr].x), __float_as_uint(b[nr].z));
#pragma unroll
        for (int nr = 0; nr < NR; ++nr) mma_tf32(d[nr], ah, __float_as_uint(b[nr].x), __float_as_uint(b[nr].z));
#pragma unroll
        for (int nr = 0; nr < NR; ++nr) mma_tf32(e[nr], ah, __float_as_uint(b[nr].y), __float_as_uint(b[nr].w));
    }
    // d[nr][i]: column c + g + 8 (i / 2), row 8 (nr0 + nr) + 2 t + i % 2
#pragma unroll
    for (int nr = 0; nr < NR; ++nr)
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const int r = 8 * (nr0 + nr) + 2 * t + (i & 1);
            const int cc = c + g + 8 * (i >> 1);
            if (r < a.proj_rows && cc < tk)
                __stcs(a.ldm + (int64_t)r * a.row_stride + k_start + cc, (d[nr][i] + e[nr][i]) * inv_fx);
        }
}
// Persistent, warp-specialised scatter: CTA b owns tiles b, b + G, b + 2G, ...
//  * warp 0 (one thread): streams the tiles' line records chunk by chunk into a
//    ring of buffers with TMA bulk copies, each buffer guarded by a "full"
//    mbarrier (TMA completion) and an "empty" one (one arrival per line warp);
//  * line warps: two lines per lane and chunk, scattered into the tile (fixed
//    point, native integer shared atomics, deterministic).  The lanes of a
//    warp take pairs `stride` (odd) apart, so that they lie in different
//    columns and their adds in different banks;
//  * flush warps: project (or copy) a finished tile's columns to HBM and zero
//    them, 16 (32) columns a warp at a time, while the line warps fill the other
//    of two tile slots ("tfull": one arrival per line warp, "tfree": one per
//    flush warp; "fmeet": the flush warps around a change of the coefficients
//    they share).
// Every wait is bounded; a wait that gives up sets the error flag and its warp
// stops, the others' waits run out in turn, and the producer stays until the
// copies it issued have landed (bounded).  W: 64-bit sums.
// A tile holds the `win` Gaussian rows that its lines can reach, not all of the
// grid's: 12 x 24 nodes need 72 of 288 rows, so that two tiles of hundreds of
// columns fit and the flush reads a quarter.  One kernel projects every grid:
// the node rows never reach memory.  Against one tile of all rows filled and
// flushed in turn: 5M lines x 400k points 94 -> 55 us (28 bytes a line are 21
// us of HBM; the shared atomics' wavefronts, the flush's MMA chains and its
// last tile are the rest), 100M x 1.5M points 1130 + 407 (a projection pass) ->
// 760 us (HBM: 414 us).  Two CTAs per SM of half the size: 58.6 and 957 us where
// one took 57 and 800.
template <bool W>
__device__ __forceinline__ void scatter_body(const ScatterArgs& a) {
    extern __shared__ __align__(128) unsigned char smem[];
    const int ch = a.chunk, S = a.stages, sb = a.stage_bytes;
    uint64_t* full = reinterpret_cast<uint64_t*>(smem + S * sb);
    uint64_t* empty = full + kScatMaxStages;
    uint64_t* tfull = empty + kScatMaxStages;
    uint64_t* tfree = tfull + 2;
    uint64_t* fmeet = tfree + 2;
    int2* rng = reinterpret_cast<int2*>(smem + S * sb + 192);
    unsigned* tiles = reinterpret_cast<unsigned*>(smem + scatter_fixed_smem(sb, S, a.rng_cap));
    const int slot_words = (a.copies * a.copy_words + 3) & ~3;
    const int G = gridDim.x;
    const int nq = (a.n_tiles - (int)blockIdx.x + G - 1) / G;   // tiles of this CTA (<= a.rng_cap)
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int lw = a.line_warps, fw = (int)(blockDim.x >> 5) - 1 - lw;

    {
        uint4* z = reinterpret_cast<uint4*>(tiles - 4);   // with the words before the first tile
        for (int i = threadIdx.x; i <= a.slots * slot_words / 4; i += blockDim.x) z[i] = make_uint4(0u, 0u, 0u, 0u);
    }
    if (threadIdx.x == 0) {
        for (int b = 0; b < S; ++b) {
            mbar_init(&full[b], 1);
            mbar_init(&empty[b], lw);
        }
        for (int b = 0; b < 2; ++b) {
            mbar_init(&tfull[b], lw);
            mbar_init(&tfree[b], fw);
        }
        mbar_init(fmeet, fw);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    chain_begin();
    if (nq > a.rng_cap) {   // the host sizes the table for every CTA: never taken
        if (threadIdx.x == 0) atomicExch(a.err, 1u);
        return;
    }
    auto col_idx = [&](int c) { return max(0, min(c + a.col_off, a.col_count - 1)); };
    for (int q = threadIdx.x; q < nq; q += blockDim.x) {
        const int k_start = ((int)blockIdx.x + q * G) * a.TK;
        const int tk = min(a.TK, a.n_v - k_start);
        const int lo = (int)a.col_start[col_idx(k_start - 1 - a.margin_cols)];
        const int hi = (int)a.col_start[col_idx(k_start + tk + a.margin_cols)];
        rng[q] = make_int2(lo / kLinePad * kLinePad, hi);   // 16-line aligned start
    }
    __syncthreads();

    if (warp == 0) {   // producer
        if (lane != 0) return;
        uint32_t c = 0;       // chunks issued
        int buf = 0;          // ring slot of chunk c (c mod S, kept incrementally)
        uint32_t round = 0;   // c / S: slot reuse number
        bool bad = false;
        for (int q = 0; q < nq && !bad && !a.withhold; ++q)
            for (int cs = rng[q].x; cs < rng[q].y; cs += ch) {
                if (round > 0 && !mbar_wait(&empty[buf], (round - 1) & 1, a.wait_limit)) {
                    bad = true;
                    break;
                }
                issue_chunk(a, smem + buf * sb, &full[buf], cs, min(ch, rng[q].y - cs));
                ++c;
                if (++buf == S) {
                    buf = 0;
                    ++round;
                }
            }
        if (bad) atomicExch(a.err, 1u);
        // the last copies must land before the CTA may end (normally already
        // consumed); this drain keeps the full bound whatever a.wait_limit is
        for (uint32_t k = c > (uint32_t)S ? c - S : 0; k < c; ++k)
            mbar_wait(&full[k % (uint32_t)S], (k / (uint32_t)S) & 1);
        return;
    }

    const float fxs = fx_scale_of(*a.cmax, Fx<W>::kWidth);
    if (warp <= lw) {   // line warps
        const int w = warp - 1;
        int buf = 0;            // ring slot of the next chunk (chunks consumed mod S)
        uint32_t par = 0;       // phase parity of its "full" barrier
        unsigned counted = 0;
        for (int q = 0; q < nq; ++q) {
            const int slot = a.slots == 2 ? q & 1 : 0, use = a.slots == 2 ? q >> 1 : q;
            const TileView tv = tile_view(a, (int)blockIdx.x + q * G);
            unsigned* tile = tiles + slot * slot_words + (lane & (a.copies - 1)) * a.copy_words;
            bool ok = use == 0 || __all_sync(0xffffffffu, mbar_wait(&tfree[slot], (use - 1) & 1, a.wait_limit));
            const int b = rng[q].y;
            for (int cs = rng[q].x; cs < b && ok; cs += ch) {
                // every lane acquires the TMA data through the mbarrier itself
                ok = __all_sync(0xffffffffu, mbar_wait(&full[buf], par, a.wait_limit));
                if (!ok) break;
                const int count = min(ch, b - cs);
                const int stride = ((count + 63) >> 6) | 1;   // odd, <= lw
                const int p = lane * stride + w;
                if (w < stride && 2 * p < count)
                    counted += scatter_pair<W>(a, tv, smem + buf * sb, p, 2 * p + 1 < count, tile, fxs);
                __syncwarp();
                if (lane == 0) mbar_arrive(&empty[buf]);   // this warp is done with the buffer
                if (++buf == S) {
                    buf = 0;
                    par ^= 1u;
                }
            }
            if (!ok) {   // the same on every lane
                if (lane == 0) atomicExch(a.err, 1u);
                return;
            }
            __syncwarp();
            if (lane == 0) mbar_arrive(&tfull[slot]);   // this warp is done with the tile
        }
        if (a.in_window) {   // one atomic per warp: per-thread atomics on one word serialise in L2
            const unsigned tot = __reduce_add_sync(0xffffffffu, counted);
            if (lane == 0 && tot) atomicAdd(a.in_window, (unsigned long long)tot);
        }
        return;
    }

    // flush warps
    const float inv_fx = 1.f / fxs;
    const int w = warp - 1 - lw;
    float4* frag = reinterpret_cast<float4*>(tiles + a.slots * slot_words);   // of the Gaussian rows from frag_base on
    int frag_base = -1;
    uint32_t meet_par = 0;
    auto meet = [&] {   // the flush warps, bounded as every wait
        __syncwarp();
        if (lane == 0) mbar_arrive(fmeet);
        const bool ok = __all_sync(0xffffffffu, mbar_wait(fmeet, meet_par, a.wait_limit));
        meet_par ^= 1u;
        if (!ok && lane == 0) atomicExch(a.err, 1u);
        return ok;
    };
    for (int q = 0; q < nq; ++q) {
        const int slot = a.slots == 2 ? q & 1 : 0, use = a.slots == 2 ? q >> 1 : q;
        const int ti = (int)blockIdx.x + q * G;
        const TileView tv = tile_view(a, ti);
        const int k_start = ti * a.TK, tk = min(a.TK, a.n_v - k_start);
        unsigned* tile = tiles + slot * slot_words;
        const int first = tv.l_base * a.NL;
        if (a.proj && a.proj_frags && tv.l_base != frag_base) {   // rarely: neighbouring tiles share it
            frag_base = tv.l_base;
            if (q && !meet()) return;   // every read of the old ones done
            for (int i = 32 * w + lane; i < (a.rows >> 3) * a.proj_nr * 32; i += 32 * fw) {
                const int s = i / (32 * a.proj_nr), nr = (i >> 5) - s * a.proj_nr;
                frag[i] = proj_frag(a, nr, first + 8 * s, i & 31);
            }
            if (!meet()) return;
        }
        if (!__all_sync(0xffffffffu, mbar_wait(&tfull[slot], use & 1, a.wait_limit))) {
            if (lane == 0) atomicExch(a.err, 1u);
            return;
        }
        const int rows = tv.l_rows * a.NL;
        if (a.proj) {
            const int steps = (rows + 7) >> 3;
            for (int c = 16 * w; c < tk; c += 16 * fw) {
                if (a.copies > (W ? 1 : 2)) fold_copies<W, 16>(a, tile, c, rows, lane);
                for (int nr0 = 0; nr0 < a.proj_nr; nr0 += 3) {   // up to three row blocks in registers
                    const int nr = a.proj_nr - nr0;
                    if (!a.proj_frags)
                        for (int i = 0; i < min(nr, 3); ++i)
                            project_columns<W, 1, false>(a, steps, first, tile, frag, c, nr0 + i, k_start, tk, inv_fx, lane);
                    else if (nr >= 3) project_columns<W, 3, true>(a, steps, first, tile, frag, c, nr0, k_start, tk, inv_fx, lane);
                    else if (nr == 2) project_columns<W, 2, true>(a, steps, first, tile, frag, c, nr0, k_start, tk, inv_fx, lane);
                    else project_columns<W, 1, true>(a, steps, first, tile, frag, c, nr0, k_start, tk, inv_fx, lane);
                }
                zero_columns<W, 16>(a, tile, c, rows, lane);
            }
        } else {
            // node rows as floats, word / fx_scale (a power of two: exact
            // scaling of the rounded word); zero rows outside the tile's
            const int hi_off = a.rows * a.pitch;
            for (int c = 32 * w; c < tk; c += 32 * fw) {
                if (a.copies > 1) fold_copies<W, 32>(a, tile, c, rows, lane);
                float* dst = a.ldm + k_start + c + lane;
                const unsigned* src = tile + c + lane;
                if (c + lane < tk)
                    for (int n = 0; n < a.n_nodes; ++n) {
                        const int r = n - first;
                        const float v = (unsigned)r < (unsigned)rows ? Fx<W>::value(src + r * a.pitch, hi_off) * inv_fx : 0.f;
                        // streaming store: the LDM is read once by the next stage, long after
                        __stcs(dst + n * a.row_stride, v);
                    }
                zero_columns<W, 32>(a, tile, c, rows, lane);
            }
        }
        __syncwarp();
        if (lane == 0) mbar_arrive(&tfree[slot]);
    }
}

template <bool W>
__global__ void __launch_bounds__(kScatThreads, 1) k_scatter(const __grid_constant__ ScatterArgs a) {
    scatter_body<W>(a);
}

// The accumulator chosen on the device from the column bound *cmax (served and
// allocation-free spectra, whose bound is never read back): a32 / a64 are the
// shapes of the two variants; the launch covers the larger grid and shared
// memory (tiles are dealt out by gridDim.x, so the extra CTAs of the smaller
// variant only take fewer tiles each).
__global__ void __launch_bounds__(kScatThreads, 1) k_scatter_auto(const __grid_constant__ ScatterArgs a32,
                                                                  const __grid_constant__ ScatterArgs a64) {
    chain_begin();
    if (fx_wide(*a32.cmax))
        scatter_body<true>(a64);
    else
        scatter_body<false>(a32);
}

// ---------------------------------------------------------------------------
// Derivatives with respect to (T, p, x), node axes held fixed.
//
// With the axes fixed the Voigt weights of the nodes are constants, so the
// spectrum is a fixed linear map C of the LDM and only the LDM depends on
// (T, p, x): dA/dtheta = C dLDM/dtheta.  Per line, the LDM holds
// I w(tv, tG, tL) in 8 cells (trilinear weights of the three fractional
// coordinates), so dLDM/dtheta is a scatter of
//   I (dlnI/dtheta w + dw/dtv dtv/dtheta + dw/dtG dtG/dtheta + dw/dtL dtL/dtheta).
// Forward mode (tangent): scatter that into a float LDM and run it through C
// (the ordinary FFT / Voigt / inverse FFT kernels).
// Reverse mode (adjoint): C restricted to one node is a symmetric circular
// convolution (V is real and even), so C^T g for node n is the same
// convolution of the upstream gradient g: Re(IFFT(FFT(g) V_n)) / (N dv).  The
// adjoint LDM for all nodes comes from one forward FFT of g and one inverse
// FFT per node pair (k_row_ifft_adj, k_col_ifft_adj; V_a + i V_b puts node a
// in the real and node b in the imaginary part), and the per-line chain rule
// gathers it back at each line's 8 cells (k_gather_grad).
// ---------------------------------------------------------------------------

// Gaussian stage of the merged layout (see GaussArgs).  One CTA: one merged
// row (wL node), kGaussTile consecutive outputs, kGaussPer per thread.  A merged row is
// sum over wide nodes l of (d_l conv LDM_{l,m}) with the symmetric residual
// kernel d_l[j] = c_l 2^(-a2_l j^2), |j| <= K_l, i.e. out[p] = sum_jj d[jj]
// x[p - ext - K + jj]; each thread keeps its outputs' input window in registers
// and advances it 8 taps at a time (two half-windows used alternately, so the
// window never moves between registers).  The shared base Gaussian of the
// wide nodes is applied after the FFT, by the row kernel.
template <int P>
__device__ __forceinline__ void gauss_step(float (&acc)[P], const float (&lo)[P], const float (&hi)[8],
                                           const float (&g)[8]) {
    // window = lo[0..P) followed by hi[0..8): acc[i] += sum_u g[u] window[i + u]
#pragma unroll
    for (int u = 0; u < 8; ++u)
#pragma unroll
        for (int i = 0; i < P; ++i) acc[i] = fmaf(g[u], i + u < P ? lo[i + u] : hi[i + u - P], acc[i]);
}

__device__ __forceinline__ void load8(float (&d)[8], const float* s) {
    const float4 a = *reinterpret_cast<const float4*>(s);
    const float4 b = *reinterpret_cast<const float4*>(s + 4);
    d[0] = a.x; d[1] = a.y; d[2] = a.z; d[3] = a.w;
    d[4] = b.x; d[5] = b.y; d[6] = b.z; d[7] = b.w;
}

// acc[i] += sum_jj taps[jj] xs[t0 + i + jj], jj < KP (a multiple of 4; xs
// readable up to t0 + KP + 7): three 8-value register blocks rotate through
// the window (no moves): taps jj..jj+7 use A ++ B, jj+8.. use B ++ C, jj+16..
// use C ++ A'; a tail of up to two 8-tap steps and one 4-tap step ends the
// row of taps.
// Four taps on the same window form (the tail of a row of taps whose count
// is 4 mod 8): acc[i] += sum_{u < 4} g[u] window[i + u], window = lo ++ hi.
__device__ __forceinline__ void gauss_step4(float (&acc)[8], const float (&lo)[8], const float4 hi, const float4 g4) {
    const float hv[3] = {hi.x, hi.y, hi.z};
    const float g[4] = {g4.x, g4.y, g4.z, g4.w};
#pragma unroll
    for (int u = 0; u < 4; ++u)
#pragma unroll
        for (int i = 0; i < 8; ++i) acc[i] = fmaf(g[u], i + u < 8 ? lo[i + u] : hv[i + u - 8], acc[i]);
}

__device__ __forceinline__ void conv_window(float (&acc)[8], const float* xs, const float* taps, int t0, int KP) {
    float A[8], B[8], C[8], g[8];
    load8(A, &xs[t0]);
    int jj = 0;
    for (; jj + 24 <= KP; jj += 24) {
        load8(B, &xs[t0 + jj + 8]);
        load8(g, &taps[jj]);
        gauss_step<8>(acc, A, B, g);
        load8(C, &xs[t0 + jj + 16]);
        load8(g, &taps[jj + 8]);
        gauss_step<8>(acc, B, C, g);
        load8(A, &xs[t0 + jj + 24]);
        load8(g, &taps[jj + 16]);
        gauss_step<8>(acc, C, A, g);
    }
    // tail of 0-20 taps: up to two 8-tap steps, then one 4-tap step
    const int r = KP - jj;
    if (r >= 8) {
        load8(B, &xs[t0 + jj + 8]);
        load8(g, &taps[jj]);
        gauss_step<8>(acc, A, B, g);
        if (r >= 16) {
            load8(C, &xs[t0 + jj + 16]);
            load8(g, &taps[jj + 8]);
            gauss_step<8>(acc, B, C, g);
            if (r & 4)
                gauss_step4(acc, C, *reinterpret_cast<const float4*>(&xs[t0 + jj + 24]),
                            *reinterpret_cast<const float4*>(&taps[jj + 16]));
        } else if (r & 4) {
            gauss_step4(acc, B, *reinterpret_cast<const float4*>(&xs[t0 + jj + 16]),
                        *reinterpret_cast<const float4*>(&taps[jj + 8]));
        }
    } else if (r & 4) {
        gauss_step4(acc, A, *reinterpret_cast<const float4*>(&xs[t0 + jj + 8]),
                    *reinterpret_cast<const float4*>(&taps[jj]));
    }
}

// Nodes are streamed through a ring of kGaussStages shared-memory slots, each
// holding one node's taps and window, filled with cp.async (zero-filled
// outside the row) kGaussStages - 1 nodes ahead of the convolution: one
// barrier per node and no staging through registers.
constexpr int kGaussStages = 4;

__device__ __forceinline__ void cp_async16(float* dst, const float* src, int bytes) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(smem_u32(dst)), "l"(src), "r"(bytes)
                 : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_async_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }

__global__ void __launch_bounds__(256) k_gauss_merge(const GaussArgs a) {
    extern __shared__ __align__(16) float gsm[];
    chain_begin();
    constexpr int TW = kGaussTile;
    constexpr int P = kGaussPer;                     // outputs per thread (8)
    constexpr int S = kGaussStages;
    const int r = blockIdx.y;
    const int p0 = blockIdx.x * TW;                  // first output (buffer position)
    const int Lr = a.n_v + 2 * a.ext;
    float* orow = a.out + (int64_t)r * a.out_stride;
    const int m = r;   // merged row of wL node m
    float acc[P];
#pragma unroll
    for (int i = 0; i < P; ++i) acc[i] = 0.f;
    const int t0 = threadIdx.x * P;
    // Node w's window starts at LDM index base = p0 - ext - K_w; it is staged
    // from the 16-byte aligned index base & ~3, and the offset s = base & 3 is
    // absorbed by s leading zero taps.
    auto shift_of = [&](int w) { return (p0 - a.ext - a.K[w]) & 3; };
    auto taps_of = [&](int w) { return (2 * a.K[w] + 1 + shift_of(w) + 3) & ~3; };   // multiple of 4
    auto slot_taps = [&](int w) { return gsm + (w % S) * a.slot_len; };
    auto issue = [&](int w) {   // taps (plain stores) and window (cp.async) of node w into its slot
        float* taps = slot_taps(w);
        float* xs = taps + a.slot_taps;
        const int K = a.K[w];
        const int sh = shift_of(w);
        const int KP = taps_of(w);
        for (int jj = threadIdx.x; jj < KP; jj += blockDim.x) {
            const float j = (float)(jj - sh - K);
            taps[jj] = jj >= sh && jj <= sh + 2 * K ? a.c[w] * ex2(-a.a2[w] * j * j) : 0.f;
        }
        const int k0 = (p0 - a.ext - K) & ~3;        // LDM index of xs[0]
        const int n4 = (TW + KP + 8 + 3) / 4;        // 4 n4 <= slot_len - slot_taps
        const float* src = a.ldm + (int64_t)(a.wide_l[w] * a.NL + m) * a.row_stride;
        for (int q = threadIdx.x; q < n4; q += blockDim.x) {
            const int k = k0 + 4 * q;                // rows start 128-byte aligned; k is a multiple of 4
            const int bytes = (k >= 0 && k < a.n_v) ? 4 * min(4, a.n_v - k) : 0;   // zeros outside [0, n_v)
            cp_async16(xs + 4 * q, bytes ? src + k : src, bytes);
        }
    };
#pragma unroll
    for (int w = 0; w < S - 1; ++w) {
        if (w < a.n_wide) issue(w);
        cp_async_commit();
    }
    for (int w = 0; w < a.n_wide; ++w) {
        cp_async_wait<S - 2>();   // this thread's copies of node w have landed
        __syncthreads();          // everyone's have, and everyone is done with node w - 1
        if (w + S - 1 < a.n_wide) issue(w + S - 1);   // into node w - 1's slot
        cp_async_commit();
        const float* taps = slot_taps(w);
        conv_window(acc, taps + a.slot_taps, taps, t0, taps_of(w));
    }
    const int p = p0 + t0;
#pragma unroll
    for (int i = 0; i < P; i += 4) {
        if (p + i + 4 <= Lr) {
            *reinterpret_cast<float4*>(&orow[p + i]) = make_float4(acc[i], acc[i + 1], acc[i + 2], acc[i + 3]);
        } else {
#pragma unroll
            for (int u = 0; u < 4; ++u)
                if (p + i + u < Lr) orow[p + i + u] = acc[i + u];
        }
    }
}

// Instrument slit (radis/tools/slit.py:737 and remove_boundary, :1063-1072):
// out[i] = scale sum_j slit[j] in[i + (m-1)/2 - j], the 'same' part of the
// full convolution, zero outside [0, n); written as a correlation with the
// reversed slit r[u] = slit[m-1-u]: out[i] = scale sum_u r[u] in[i - m/2 + u].
// One CTA: two groups of threads over the same outputs, 8 per thread, each
// with half of the taps (their parts are summed at the end); taps in passes of
// kSlitPass with a staged input window, through the same register-window
// convolution as the Gaussian stage.  'valid' mode: the first (la-1)/2 and last
// la/2 outputs are NaN, la = min(n, m).  Bound by the FP32 pipe and its
// operand reads (84% of the instructions are FMAs of three registers, which
// measured 3.2 of 4 per cycle), so every SM gets the same number of outputs
// (slit_threads) and the second group keeps enough warps in flight.  400 001
// points x 1001 taps, time per call: 196 CTAs of 2048 outputs 28.7 us, equal
// CTAs 26.7, with two groups 22.6 (three 22.5, four 28.2: registers allow one
// CTA less).  A padded window without bank conflicts: 24.6.
constexpr int kSlitGroups = 2;
__global__ void __launch_bounds__(128 * kSlitGroups) k_slit_conv(const SlitArgs a) {
    extern __shared__ __align__(16) float ssm[];
    constexpr int P = kGaussPer;
    constexpr int G = kSlitGroups;
    const int T = (int)blockDim.x / G;       // threads of a group
    const int TW = T * P;
    const int grp = threadIdx.x / T, gt = threadIdx.x - grp * T;
    float* taps = ssm;                       // kSlitPass (padded to 4)
    float* xs = ssm + kSlitPass + 16;        // TW + KP + 8 <= TW + kSlitPass + 16
    const int64_t p0 = (int64_t)blockIdx.x * TW;
    const int t0 = gt * P;
    const int64_t half = a.m / 2;
    float acc[P];
#pragma unroll
    for (int i = 0; i < P; ++i) acc[i] = 0.f;
    for (int u0 = 0; u0 < a.m; u0 += kSlitPass) {
        const int kb = min(kSlitPass, a.m - u0);
        const int KP = (kb + 3) & ~3;
        const int64_t base = p0 - half + u0;   // input index of xs[0]
        __syncthreads();   // previous pass consumed
        for (int jj = threadIdx.x; jj < KP; jj += blockDim.x) taps[jj] = jj < kb ? a.slit[a.m - 1 - (u0 + jj)] : 0.f;
        for (int t = threadIdx.x; t < TW + KP + 8; t += blockDim.x) {
            const int64_t k = base + t;
            xs[t] = k >= 0 && k < a.n ? __ldg(&a.in[k]) : 0.f;
        }
        __syncthreads();
        // this group's share of the pass's taps
        const int share = ((KP + G - 1) / G + 7) & ~7;
        const int k0 = min(grp * share, KP), k1 = min(k0 + share, KP);
        conv_window(acc, xs, taps + k0, t0 + k0, k1 - k0);
    }
    if (G > 1) {   // sum the groups' parts into the first one's
        __syncthreads();
        float* part = xs;   // [G - 1][P][T]
        if (grp) {
#pragma unroll
            for (int i = 0; i < P; ++i) part[((grp - 1) * P + i) * T + gt] = acc[i];
        }
        __syncthreads();
        if (grp) return;
        for (int q = 0; q < G - 1; ++q)
#pragma unroll
            for (int i = 0; i < P; ++i) acc[i] += part[(q * P + i) * T + gt];
    }
    const int64_t la = a.n < (int64_t)a.m ? a.n : (int64_t)a.m;
    const int64_t ea = a.valid ? (la - 1) / 2 : 0, eb = a.valid ? la / 2 : 0;
#pragma unroll
    for (int i = 0; i < P; ++i) {
        const int64_t idx = p0 + t0 + i;
        if (idx < a.n) a.out[idx] = idx < ea || idx >= a.n - eb ? __int_as_float(0x7fc00000) : acc[i] * a.scale;
    }
}

// Per-line derivative coefficients: dlnI/dtheta and the rates of the three
// fractional coordinates, for theta = T, p_bar, x (radis/lbl/base.py:2664-2677
// for I, broadening.py:170-172 and 368-381 for the widths, base.py:2351-2370
// for the shift; number density p x / (k T)).
struct LineRates {
    float lnI[3], tv[3], tG[3], tL[3];
};

__device__ __forceinline__ LineRates line_rates(const GradArgs& g, float v0, float el, float ga, float gs, float na,
                                                float dl, int is) {
    LineRates r;
    const float x = g.c2_T * v0;
    // d/dT of ln(exp(-c2 El/T) (1 - exp(-c2 v0/T))), partition ratio and density
    r.lnI[0] = g.c2_T2 * el - g.c2_T2 * v0 / expm1f(x) + g.cT0[is];
    r.lnI[1] = g.iP;
    r.lnI[2] = g.iX;
    r.tv[0] = 0.f;
    r.tv[1] = dl * g.kP;
    r.tv[2] = 0.f;
    r.tG[0] = g.gT;
    r.tG[1] = 0.f;
    r.tG[2] = 0.f;
    const float gam = fmaf(g.s.x_self, gs - ga, ga);
    r.tL[0] = -na * g.lT;
    r.tL[1] = g.lP;
    r.tL[2] = (gs - ga) / gam * g.lX;
    return r;
}

// Reverse mode: out[theta] += sum over lines of I (dlnI S0 + dtv Sk + dtG SG +
// dtL SL), with S0 the adjoint LDM interpolated at the line and Sk, SG, SL its
// differences along the three cell axes.  One FP64 atomic per block and theta.
__global__ void __launch_bounds__(256) k_gather_grad(const GradArgs g) {
    extern __shared__ float gcs[];   // skeleton layout: the coefficients [proj_n][proj_rp]
    const ScatterArgs& a = g.s;
    if (g.proj_coef) {
        for (int i = threadIdx.x; i < g.proj_n * g.proj_rp; i += blockDim.x) gcs[i] = __ldg(&g.proj_coef[i]);
        __syncthreads();
    }
    float acc[3] = {0.f, 0.f, 0.f};
    const int64_t stride = (int64_t)gridDim.x * blockDim.x;
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < g.n_lines; i += stride) {
        const float2 v = make_float2(a.vh[i], a.vl[i]);
        const float dl = a.dl ? a.dl[i] : 0.f;
        float fk, tv;
        line_position(a, v, dl, fk, tv);
        if (!(fk >= 0.f) || fk + 1.f >= (float)a.n_v) continue;
        const int k0 = (int)fk;
        const int is = a.iso ? (int)a.iso[i] : 0;
        const float ga = a.ga[i], gs = a.gs[i], na = a.na[i], el = a.el[i];
        int l0, m0;
        float tG, tL;
        line_nodes(a, v.x, ga, gs, na, is, l0, m0, tG, tL);
        const float I = line_intensity(a, v.x, el, a.ls2[i], is);
        if (!(I > 0.f)) continue;
        // the adjoint at the line's 4 nodes, columns k0 and k0 + 1
        float u0[4], u1[4];   // node order (l0, m0), (l0, m0 + 1), (l0 + 1, m0), (l0 + 1, m0 + 1)
        const int n00 = l0 * a.NL + m0;
        if (g.proj_coef) {   // from the skeleton rows
            const int nd[4] = {n00, n00 + 1, n00 + a.NL, n00 + a.NL + 1};
#pragma unroll
            for (int j = 0; j < 4; ++j) u0[j] = u1[j] = 0.f;
            const float* z = g.adj + k0;
            for (int r = 0; r < g.proj_rows; ++r, z += g.row_stride) {
                const float z0 = z[0], z1 = z[1];
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    const float c = gcs[nd[j] * g.proj_rp + r];
                    u0[j] = fmaf(c, z0, u0[j]);
                    u1[j] = fmaf(c, z1, u1[j]);
                }
            }
        } else {
            const float* r00 = g.adj + (int64_t)n00 * g.row_stride + k0;
            const float* rr[4] = {r00, r00 + g.row_stride, r00 + (int64_t)a.NL * g.row_stride,
                                  r00 + (int64_t)(a.NL + 1) * g.row_stride};
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                u0[j] = rr[j][0];
                u1[j] = rr[j][1];
            }
        }
        const float d00 = u1[0] - u0[0], d01 = u1[1] - u0[1];
        const float d10 = u1[2] - u0[2], d11 = u1[3] - u0[3];
        const float e00 = fmaf(tv, d00, u0[0]), e01 = fmaf(tv, d01, u0[1]);
        const float e10 = fmaf(tv, d10, u0[2]), e11 = fmaf(tv, d11, u0[3]);
        const float uG = 1.f - tG, uL = 1.f - tL;
        const float S0 = uG * (uL * e00 + tL * e01) + tG * (uL * e10 + tL * e11);
        const float Sk = uG * (uL * d00 + tL * d01) + tG * (uL * d10 + tL * d11);
        const float SG = uL * (e10 - e00) + tL * (e11 - e01);
        const float SL = uG * (e01 - e00) + tG * (e11 - e10);
        const LineRates r = line_rates(g, v.x, el, ga, gs, na, dl, is);
#pragma unroll
        for (int q = 0; q < 3; ++q) acc[q] += I * (r.lnI[q] * S0 + r.tv[q] * Sk + r.tG[q] * SG + r.tL[q] * SL);
    }
    __shared__ double part[3][8];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
    for (int q = 0; q < 3; ++q) {
        double s = acc[q];
        for (int o = 16; o; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
        if (lane == 0) part[q][warp] = s;
    }
    __syncthreads();
    if (threadIdx.x < 3) {
        double s = 0.0;
        for (int w = 0; w < (int)(blockDim.x >> 5); ++w) s += part[threadIdx.x][w];
        atomicAdd(&g.out[threadIdx.x], s);
    }
}

// Forward mode: scatter the tangent of each line's 8 LDM values in direction
// g.theta into the float rows g.tan (FP32 global atomics): node rows, or the
// skeleton rows.
__global__ void __launch_bounds__(256) k_scatter_tangent(const GradArgs g) {
    const ScatterArgs& a = g.s;
    const int th = g.theta;
    const int64_t stride = (int64_t)gridDim.x * blockDim.x;
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < g.n_lines; i += stride) {
        const float2 v = make_float2(a.vh[i], a.vl[i]);
        const float dl = a.dl ? a.dl[i] : 0.f;
        float fk, tv;
        line_position(a, v, dl, fk, tv);
        if (!(fk >= 0.f) || fk + 1.f >= (float)a.n_v) continue;
        const int k0 = (int)fk;
        const int is = a.iso ? (int)a.iso[i] : 0;
        const float ga = a.ga[i], gs = a.gs[i], na = a.na[i], el = a.el[i];
        int l0, m0;
        float tG, tL;
        line_nodes(a, v.x, ga, gs, na, is, l0, m0, tG, tL);
        const float I = line_intensity(a, v.x, el, a.ls2[i], is);
        if (!(I > 0.f)) continue;
        const LineRates r = line_rates(g, v.x, el, ga, gs, na, dl, is);
        const float K[2] = {1.f - tv, tv}, dK[2] = {-r.tv[th], r.tv[th]};
        const float Gw[2] = {1.f - tG, tG}, dG[2] = {-r.tG[th], r.tG[th]};
        const float Lw[2] = {1.f - tL, tL}, dL[2] = {-r.tL[th], r.tL[th]};
        const float ln = r.lnI[th];
        float u[4][2];   // node order (l0, m0), (l0, m0 + 1), (l0 + 1, m0), (l0 + 1, m0 + 1)
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const float gl = Gw[j >> 1] * Lw[j & 1];
            const float dgl = dG[j >> 1] * Lw[j & 1] + Gw[j >> 1] * dL[j & 1];
#pragma unroll
            for (int ck = 0; ck < 2; ++ck) u[j][ck] = I * fmaf(ln, K[ck] * gl, dK[ck] * gl + K[ck] * dgl);
        }
        const int n00 = l0 * a.NL + m0;
        if (g.proj_coef) {
            const float* c00 = g.proj_coef + n00 * g.proj_rp;
            const float* c10 = c00 + a.NL * g.proj_rp;
            float* row = g.tan + k0;
#pragma unroll 4
            for (int r = 0; r < g.proj_rows; ++r, row += g.row_stride) {
                const float c[4] = {__ldg(c00 + r), __ldg(c00 + g.proj_rp + r), __ldg(c10 + r), __ldg(c10 + g.proj_rp + r)};
#pragma unroll
                for (int ck = 0; ck < 2; ++ck)
                    atomicAdd(&row[ck], fmaf(c[3], u[3][ck], fmaf(c[2], u[2][ck], fmaf(c[1], u[1][ck], c[0] * u[0][ck]))));
            }
            continue;
        }
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            float* row = g.tan + (int64_t)(n00 + (j >> 1) * a.NL + (j & 1)) * g.row_stride + k0;
#pragma unroll
            for (int ck = 0; ck < 2; ++ck) atomicAdd(&row[ck], u[j][ck]);
        }
    }
}

// ---------------------------------------------------------------------------
// launchers
// ---------------------------------------------------------------------------
static thread_local const char* g_launch_err = nullptr;
const char* last_launch_error() { return g_launch_err; }

int check_launch() {
    cudaError_t e = cudaGetLastError();
    g_launch_err = e == cudaSuccess ? nullptr : cudaGetErrorString(e);
    return e == cudaSuccess ? RG_OK : RG_ERR_CUDA;
}

int launch_prepare_lines(const double* v0_d, const double* s_d, int64_t n, double c2_tref, float* vh_out,
                         float* vl_out, float* ls2_out, int* unsorted_flag, cudaStream_t st) {
    if (n <= 0) return RG_OK;
    int64_t blocks = (n + 255) / 256;
    k_prepare_lines<<<(unsigned)blocks, 256, 0, st>>>(v0_d, s_d, n, c2_tref, vh_out, vl_out, ls2_out,
                                                          unsorted_flag);
    return check_launch();
}

int launch_col_index(const float* vh, const float* vl, int64_t n, double vmin, double dv, int c_min, int count,
                     int64_t* col_start, cudaStream_t st) {
    k_col_index<<<(count + 255) / 256, 256, 0, st>>>(SplitList{vh, vl}, n, vmin, dv, c_min, count, col_start);
    return check_launch();
}

int launch_col_cmax(const int64_t* col_start, int col_off, int col_count, int n_v, int E, int* cmax,
                    cudaStream_t st) {
    if (cudaMemsetAsync(cmax, 0, sizeof(int), st) != cudaSuccess) return RG_ERR_CUDA;
    const int blocks = std::min((n_v + 255) / 256, 1024);
    k_col_cmax<<<std::max(blocks, 1), 256, 0, st>>>(col_start, col_off, col_count, n_v, E, cmax);
    return check_launch();
}

int launch_scatter(const ScatterArgs& a, int grid, int threads, size_t smem, bool wide, cudaStream_t st) {
    if (wide) {
        ALLOW_SMEM(k_scatter<true>, smem);
        return launch_chained(k_scatter<true>, grid, threads, smem, st, a);
    }
    ALLOW_SMEM(k_scatter<false>, smem);
    return launch_chained(k_scatter<false>, grid, threads, smem, st, a);
}

int launch_scatter_auto(const ScatterArgs& a32, const ScatterArgs& a64, int grid, int threads, size_t smem,
                        cudaStream_t st) {
    ALLOW_SMEM(k_scatter_auto, smem);
    return launch_chained(k_scatter_auto, grid, threads, smem, st, a32, a64);
}

// Dynamic shared memory a scatter variant may have (one CTA per SM).
template <bool W>
static int scatter_optin(size_t* avail) {
    static std::atomic<size_t> cached{0};   // one GPU model per process
    size_t a = cached.load();
    if (!a) {
        int dev = 0, optin = 0;
        if (cudaGetDevice(&dev) != cudaSuccess) return RG_ERR_CUDA;
        if (cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev) != cudaSuccess)
            return RG_ERR_CUDA;
        cudaFuncAttributes fa;
        if (cudaFuncGetAttributes(&fa, k_scatter<W>) != cudaSuccess) return RG_ERR_CUDA;
        a = (size_t)optin - fa.sharedSizeBytes;
        cached.store(a);
    }
    *avail = a;
    return RG_OK;
}
int scatter_smem_optin(size_t* avail, bool wide) {
    // every variant (and k_scatter_auto) has the same static shared memory
    // (none); the opt-in limit of one serves for all
    return wide ? scatter_optin<true>(avail) : scatter_optin<false>(avail);
}

// Row pitch of the projection coefficients: the rows rounded up to a multiple of 4.
int proj_rows_pad(int rows) { return (rows + 3) & ~3; }

// Tensor-core form of the projection pass: Y^T[columns x rows] = X^T[columns
// x nodes] C^T[nodes x rows] with mma.sync m16n8k8 TF32 (columns as M, rows
// as N in steps of 8, nodes as K), each product split into three TF32
// products (hi hi + lo hi + hi lo; x = hi + lo with hi = tf32(x), lo =
// tf32(x - hi)): ~22 significant bits per operand, FP32-level sums.  CTA = 8
// warps over a 256-column tile; warp w owns columns 32 w .. 32 w + 31 as two
// 16-column m-tiles, for every 8-row n-tile (NR of them), accumulators in
// registers; the three products of a k-step are issued part by part over all
// 2 NR accumulators (independent MMAs between dependent ones).  Node rows
// stream through kTcStages shared-memory stages of 16 rows (cp.async,
// zero-filled past n_v and past the last node), row pitch 264 floats: the A
// fragment loads (node t / t + 4, column g / g + 8 of each m-tile) are
// conflict-free.  The B fragments (coefficients, hi and lo parts, prepared on
// the host in fragment order) sit in shared memory, 8 bytes per lane per part.
constexpr int kTcTC = 256;                // columns per CTA tile (8 warps x 32)
constexpr int kTcKC = 16;                 // node rows per stage (two k-steps)
constexpr int kTcPitch = kTcTC + 8;       // staged row pitch (floats)
constexpr int kTcStages = 3;

size_t proj_tc_smem(int row_blocks, int ksteps) {
    return sizeof(float) * ((size_t)row_blocks * ksteps * 128 + (size_t)kTcStages * kTcKC * kTcPitch);
}


template <int NR>
__global__ void __launch_bounds__(256, 2) k_node_project_tc(const ProjArgs a) {
    constexpr int S = kTcStages;
    extern __shared__ __align__(16) float tsm[];
    const int KSP = a.ksteps;                             // node steps of 8 (even, covers n_nodes)
    const int n_chunks = KSP / 2;                         // 16-node chunks per tile
    float* fr = tsm;                                      // fragments [NR][KSP][2][32][2]
    float* xs = tsm + NR * KSP * 128;                     // stages [S][kTcKC][kTcPitch]
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int g = lane >> 2, t = lane & 3;
    const int n_tiles = (int)((a.n_v + kTcTC - 1) / kTcTC);
    const int my_tiles = (n_tiles - (int)blockIdx.x + (int)gridDim.x - 1) / (int)gridDim.x;
    const int total = my_tiles * n_chunks;
    auto tile_k0 = [&](int tt) { return (int64_t)((int)blockIdx.x + tt * (int)gridDim.x) * kTcTC; };
    // this thread's 16-byte pieces of a stage: rows r_0 + 4 i, columns 4 c4_t
    const int r_0 = threadIdx.x / (kTcTC / 4), c4_t = threadIdx.x % (kTcTC / 4);
    auto issue = [&](int gq) {
        const int64_t k = tile_k0(gq / n_chunks) + 4 * c4_t;
        const int nd0 = (gq % n_chunks) * kTcKC + r_0;
        float* dst = xs + (gq % S) * kTcKC * kTcPitch + r_0 * kTcPitch + 4 * c4_t;
        const float* src = a.ldm + (int64_t)nd0 * a.row_stride + k;
        const bool col_ok = k < a.n_v;   // a piece past n_v stays in the row's padding
#pragma unroll
        for (int i = 0; i < kTcKC * kTcTC / 4 / 256; ++i) {
            const bool ok = col_ok && nd0 + 4 * i < a.n_nodes;
            cp_async16(dst + 4 * i * kTcPitch, ok ? src + (int64_t)4 * i * a.row_stride : a.ldm, ok ? 16 : 0);
        }
    };
#pragma unroll
    for (int q = 0; q < S - 1; ++q) {
        if (q < total) issue(q);
        cp_async_commit();
    }
    {
        const float4* src = reinterpret_cast<const float4*>(a.frag);
        float4* dst = reinterpret_cast<float4*>(fr);
        for (int i = threadIdx.x; i < NR * KSP * 32; i += blockDim.x) dst[i] = __ldg(&src[i]);
    }
    for (int tt = 0; tt < my_tiles; ++tt) {
        float d[2][NR][4];
#pragma unroll
        for (int m = 0; m < 2; ++m)
#pragma unroll
            for (int nr = 0; nr < NR; ++nr)
#pragma unroll
                for (int i = 0; i < 4; ++i) d[m][nr][i] = 0.f;
        for (int ch = 0; ch < n_chunks; ++ch) {
            const int gq = tt * n_chunks + ch;
            cp_async_wait<S - 2>();
            __syncthreads();
            if (gq + S - 1 < total) issue(gq + S - 1);
            cp_async_commit();
            const float* xb = xs + (gq % S) * kTcKC * kTcPitch + warp * 32 + g;
#pragma unroll
            for (int s2 = 0; s2 < 2; ++s2) {
                const int ks = 2 * ch + s2;
                // A fragments (two m-tiles): (col g / g + 8, node t / t + 4), hi and lo
                uint32_t ah[2][4], al[2][4];
#pragma unroll
                for (int m = 0; m < 2; ++m) {
                    const float* xm = xb + (8 * s2 + t) * kTcPitch + 16 * m;
                    const float v[4] = {xm[0], xm[8], xm[4 * kTcPitch], xm[4 * kTcPitch + 8]};
#pragma unroll
                    for (int i = 0; i < 4; ++i) {
                        ah[m][i] = tf32_rna(v[i]);
                        al[m][i] = tf32_rna(v[i] - __uint_as_float(ah[m][i]));
                    }
                }
                uint32_t bh[NR][2], bl[NR][2];
#pragma unroll
                for (int nr = 0; nr < NR; ++nr) {
                    const float* f = fr + ((nr * KSP + ks) * 2) * 64 + lane * 2;
                    const float2 h = *reinterpret_cast<const float2*>(f);
                    const float2 l = *reinterpret_cast<const float2*>(f + 64);
                    bh[nr][0] = __float_as_uint(h.x);
                    bh[nr][1] = __float_as_uint(h.y);
                    bl[nr][0] = __float_as_uint(l.x);
                    bl[nr][1] = __float_as_uint(l.y);
                }
#pragma unroll
                for (int m = 0; m < 2; ++m)
#pragma unroll
                    for (int nr = 0; nr < NR; ++nr) mma_tf32(d[m][nr], ah[m], bh[nr][0], bh[nr][1]);
#pragma unroll
                for (int m = 0; m < 2; ++m)
#pragma unroll
                    for (int nr = 0; nr < NR; ++nr) mma_tf32(d[m][nr], al[m], bh[nr][0], bh[nr][1]);
#pragma unroll
                for (int m = 0; m < 2; ++m)
#pragma unroll
                    for (int nr = 0; nr < NR; ++nr) mma_tf32(d[m][nr], ah[m], bl[nr][0], bl[nr][1]);
            }
        }
        // the tile is complete: d[m][nr] = (column g / g + 8 of m-tile m, row 8 nr + 2 t / + 1)
        const int64_t kc = tile_k0(tt) + warp * 32 + g;
#pragma unroll
        for (int m = 0; m < 2; ++m)
#pragma unroll
            for (int nr = 0; nr < NR; ++nr)
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    const int r = 8 * nr + 2 * t + (i & 1);
                    const int64_t k = kc + 16 * m + 8 * (i >> 1);
                    if (r < a.rows && k < a.n_v) a.ldm[(int64_t)r * a.row_stride + k] = d[m][nr][i];
                }
    }
}

template <int NR>
int launch_proj_tc(const ProjArgs& a, cudaStream_t st) {
    const size_t smem = proj_tc_smem(NR, a.ksteps);
    ALLOW_SMEM((k_node_project_tc<NR>), smem);
    const int64_t tiles = (a.n_v + kTcTC - 1) / kTcTC;
    // two CTAs per SM where their shared memory fits (fragments of up to ~4 row
    // blocks of a 288-node grid), else one
    const int per_sm = smem <= 110 * 1024 ? 2 : 1;
    const int grid = (int)std::min<int64_t>(tiles, (int64_t)per_sm * std::max(a.sms, 1));
    k_node_project_tc<NR><<<grid, 256, smem, st>>>(a);
    return check_launch();
}

int launch_node_project(const ProjArgs& a, cudaStream_t st) {
    if (a.rows <= 0 || a.rows > kProjMaxRows || a.rows_pad != proj_rows_pad(a.rows) || a.n_nodes <= 0 ||
        a.n_v <= 0 || a.row_stride % 4 != 0 || !a.frag)
        return RG_ERR_ARG;
    if (a.mtiles != (a.rows + 7) / 8 || a.ksteps < (a.n_nodes + 7) / 8 || a.ksteps % 2) return RG_ERR_ARG;
    if (proj_tc_smem(a.mtiles, a.ksteps) > kProjTcSmemMax) return RG_ERR_RANGE;
    switch (a.mtiles) {
    case 1: return launch_proj_tc<1>(a, st);
    case 2: return launch_proj_tc<2>(a, st);
    case 3: return launch_proj_tc<3>(a, st);
    case 4: return launch_proj_tc<4>(a, st);
    case 5: return launch_proj_tc<5>(a, st);
    case 6: return launch_proj_tc<6>(a, st);
    case 7: return launch_proj_tc<7>(a, st);
    case 8: return launch_proj_tc<8>(a, st);
    default: return RG_ERR_ARG;
    }
}

int launch_gauss_merge(const GaussArgs& a0, int out_rows, cudaStream_t st) {
    GaussArgs a = a0;
    const int Lr = a.n_v + 2 * a.ext;
    if (a.n_wide < 0 || a.n_wide > kMaxAxis || a.row_stride % 4) return RG_ERR_RANGE;
    int kp_max = 4;   // taps of the widest node: 2 K + 1 + shift (<= 3), rounded up to 4
    for (int w = 0; w < a.n_wide; ++w) {
        if (a.K[w] < 0 || a.K[w] > kGaussMaxK) return RG_ERR_RANGE;
        kp_max = std::max(kp_max, (2 * a.K[w] + 1 + 3 + 3) & ~3);
    }
    a.slot_taps = kp_max;
    a.slot_len = kp_max + ((kGaussTile + kp_max + 8 + 3) / 4) * 4;   // taps + staged window, 16-byte multiple
    const size_t smem = sizeof(float) * (size_t)kGaussStages * a.slot_len;
    ALLOW_SMEM(k_gauss_merge, smem);
    dim3 grid((Lr + kGaussTile - 1) / kGaussTile, out_rows);
    return launch_chained(k_gauss_merge, grid, 256, smem, st, a);
}

// Threads per group of the slit convolution: the outputs dealt out in the
// fewest whole CTAs per SM of at most 128 threads a group, all equally large,
// so that no SM works while the others have finished.
static int slit_threads(int64_t n, int sms) {
    const int64_t per_sm = (n + (int64_t)sms * kGaussPer - 1) / ((int64_t)sms * kGaussPer);   // threads
    const int64_t ctas = (per_sm + 127) / 128;
    return (int)std::max<int64_t>(8, (per_sm + ctas - 1) / ctas);
}

int launch_slit_conv(const SlitArgs& a, int sms, cudaStream_t st) {
    if (a.n <= 0) return RG_OK;
    if (a.m <= 0) return RG_ERR_RANGE;
    const int threads = slit_threads(a.n, sms);
    const int tile = threads * kGaussPer;
    const size_t window = std::max(tile + kSlitPass + 16, (kSlitGroups - 1) * tile);
    const size_t smem = sizeof(float) * (kSlitPass + 16 + window);
    const int64_t blocks = (a.n + tile - 1) / tile;
    if (blocks > 0x7fffffff) return RG_ERR_RANGE;
    k_slit_conv<<<(unsigned)blocks, threads * kSlitGroups, smem, st>>>(a);
    return check_launch();
}

int launch_gather_grad(const GradArgs& a, int grid, cudaStream_t st) {
    if (a.n_lines <= 0) return RG_OK;
    const size_t smem = a.proj_coef ? sizeof(float) * (size_t)a.proj_n * a.proj_rp : 0;
    ALLOW_SMEM(k_gather_grad, smem);
    k_gather_grad<<<(int)std::min<int64_t>(grid, (a.n_lines + 255) / 256), 256, smem, st>>>(a);
    return check_launch();
}

int launch_scatter_tangent(const GradArgs& a, int grid, cudaStream_t st) {
    if (a.n_lines <= 0) return RG_OK;
    k_scatter_tangent<<<(int)std::min<int64_t>(grid, (a.n_lines + 255) / 256), 256, 0, st>>>(a);
    return check_launch();
}

}  // namespace rg
