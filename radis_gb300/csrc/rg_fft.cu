// The four-step FFT of the synthesis and of its adjoint, for sm_103a.
//
//   k_col_fft_fwd(_f)  length-n1 DFTs down the columns of two packed node rows
//                      z = a + i b, and the four-step twiddle
//   k_row_fft_voigt    length-n2 DFT of each row and pair, times the analytic
//                      Voigt FT of the two nodes, summed over the pairs, and the
//                      inverse row DFT of the sum (replaces the R2C FFT and
//                      cmdApplyLineshapes.comp:51-90)
//   k_col_ifft         inverse twiddle, inverse column DFTs, real part, scaled,
//                      first n_v samples (replaces the C2R IFFT)
//   k_row_ifft_adj, k_col_ifft_adj   the adjoint's inverse half, per pair
//
// Everything works on two complex values side by side (P2: neighbouring
// columns t = 2c, 2c + 1 of the n1 x n2 array), with the packed FP32
// instructions of sm_103a.  A packed add or multiply takes the pipe as long as two
// scalar ones (measured: 1.95 warp instructions per clock and SM against
// 3.77) but one issue slot instead of two, and issue slots are what bounds
// these kernels: their FP32 pipes were 24% busy at 48-59% issue.  The column
// DFTs treat the two columns alike.  The row DFT of length n2 then is two
// packed DFTs of length h = n2 / 2 over the even and the odd t, joined by one
// radix-2 step on the two lanes of a P2; the inverse row DFT starts with that
// step and ends with the even and odd t in the two lanes again, which is what
// the inverse column kernel reads.  No value ever changes lanes through a shuffle.
// The scalar form it replaces (one butterfly of two pairs per thread, pairs in
// turn): rows of 819 200 points x 6 pairs 24.8 M warp instructions and 49.8 us,
// now 15.0 M and 36.9; 10 240 points 28.4 -> 8.6 us; 1024 points with 13 folded
// copies 20.5 -> 6.7 us.
//
// Arrays between the kernels: y[pair][k1][c] and g[k1][c], c < h, 16 bytes per
// element (re 2c, re 2c + 1, im 2c, im 2c + 1).  The frequency form of g (the
// adjoint's transform of its input) holds bins k2 = c and c + h in the two lanes.
#include <algorithm>
#include <type_traits>

#include "rg_device.cuh"

namespace rg {

// ---------------------------------------------------------------------------
// pairs of complex values
// ---------------------------------------------------------------------------
struct P2 {
    float2 re, im;
};
__device__ __forceinline__ float2 dup2(float x) { return make_float2(x, x); }
__device__ __forceinline__ float2 neg2(float2 a) { return make_float2(-a.x, -a.y); }   // folds into an operand
__device__ __forceinline__ P2 dup(float2 w) { return {dup2(w.x), dup2(w.y)}; }
__device__ __forceinline__ P2 zero_p2() { return {dup2(0.f), dup2(0.f)}; }
__device__ __forceinline__ P2 cadd(P2 a, P2 b) { return {__fadd2_rn(a.re, b.re), __fadd2_rn(a.im, b.im)}; }
__device__ __forceinline__ P2 csub(P2 a, P2 b) { return {__fadd2_rn(a.re, neg2(b.re)), __fadd2_rn(a.im, neg2(b.im))}; }
__device__ __forceinline__ P2 cmul(P2 a, P2 w) {
    return {__ffma2_rn(a.re, w.re, neg2(__fmul2_rn(a.im, w.im))), __ffma2_rn(a.im, w.re, __fmul2_rn(a.re, w.im))};
}
__device__ __forceinline__ P2 mul_mi(P2 a) { return {a.im, neg2(a.re)}; }   // times -i
__device__ __forceinline__ P2 axpy(float c, P2 t, P2 a) {                   // a + c t
    return {__ffma2_rn(dup2(c), t.re, a.re), __ffma2_rn(dup2(c), t.im, a.im)};
}
__device__ __forceinline__ P2 scale(float c, P2 t) { return {__fmul2_rn(dup2(c), t.re), __fmul2_rn(dup2(c), t.im)}; }
__device__ __forceinline__ P2 from4(float4 v) { return {make_float2(v.x, v.y), make_float2(v.z, v.w)}; }
__device__ __forceinline__ float4 to4(P2 v) { return make_float4(v.re.x, v.re.y, v.im.x, v.im.y); }
__device__ __forceinline__ float2 cmulf(float2 a, float2 b) {
    return make_float2(a.x * b.x - a.y * b.y, a.x * b.y + a.y * b.x);
}

// ---------------------------------------------------------------------------
// forward DFTs in registers (exp(-2 pi i n k / R)), natural order
// ---------------------------------------------------------------------------
__device__ __forceinline__ void dft2(P2* v) {
    const P2 a = v[0], b = v[1];
    v[0] = cadd(a, b);
    v[1] = csub(a, b);
}
__device__ __forceinline__ void dft4(P2* v) {
    const P2 s02 = cadd(v[0], v[2]), d02 = csub(v[0], v[2]);
    const P2 s13 = cadd(v[1], v[3]), d13 = mul_mi(csub(v[1], v[3]));
    v[0] = cadd(s02, s13);
    v[2] = csub(s02, s13);
    v[1] = cadd(d02, d13);
    v[3] = csub(d02, d13);
}
__device__ __forceinline__ void dft3(P2* v) {
    const float c1 = -0.5f, s1 = 0.86602540378443864676f;   // cos, sin(2 pi / 3)
    const P2 t = cadd(v[1], v[2]), d = mul_mi(csub(v[1], v[2]));
    const P2 m = axpy(c1, t, v[0]);
    v[0] = cadd(v[0], t);
    v[1] = axpy(s1, d, m);
    v[2] = axpy(-s1, d, m);
}
__device__ __forceinline__ void dft5(P2* v) {
    const float c1 = 0.30901699437494742410f, s1 = 0.95105651629515357212f;    // 2 pi / 5
    const float c2 = -0.80901699437494742410f, s2 = 0.58778525229247312917f;   // 4 pi / 5
    const P2 t1 = cadd(v[1], v[4]), d1 = csub(v[1], v[4]);
    const P2 t2 = cadd(v[2], v[3]), d2 = csub(v[2], v[3]);
    const P2 m1 = axpy(c2, t2, axpy(c1, t1, v[0]));
    const P2 m2 = axpy(c1, t2, axpy(c2, t1, v[0]));
    const P2 q1 = mul_mi(axpy(s2, d2, scale(s1, d1)));
    const P2 q2 = mul_mi(axpy(-s1, d2, scale(s2, d1)));
    v[0] = cadd(v[0], cadd(t1, t2));
    v[1] = cadd(m1, q1);
    v[4] = csub(m1, q1);
    v[2] = cadd(m2, q2);
    v[3] = csub(m2, q2);
}
// the last step of an 8-point DFT: v[k], v[k + 4] from the even (e) and odd (o) halves' 4-point DFTs
__device__ __forceinline__ void dft8_join(P2* v, const P2* e, const P2* o) {
    const float r = 0.70710678118654752440f;
    const P2 a1 = cadd(o[1], mul_mi(o[1]));   // w8 o1 = r (1 - i) o1
    const P2 a3 = csub(mul_mi(o[3]), o[3]);   // w8^3 o3 = r (-1 - i) o3
    const P2 o2 = mul_mi(o[2]);
    v[0] = cadd(e[0], o[0]);
    v[4] = csub(e[0], o[0]);
    v[1] = axpy(r, a1, e[1]);
    v[5] = axpy(-r, a1, e[1]);
    v[2] = cadd(e[2], o2);
    v[6] = csub(e[2], o2);
    v[3] = axpy(r, a3, e[3]);
    v[7] = axpy(-r, a3, e[3]);
}
__device__ __forceinline__ void dft8(P2* v) {
    P2 e[4] = {v[0], v[2], v[4], v[6]}, o[4] = {v[1], v[3], v[5], v[7]};
    dft4(e);
    dft4(o);
    dft8_join(v, e, o);
}
// the same where v[4..7] are zero (the padded half of the rows)
__device__ __forceinline__ void dft8_half(P2* v) {
    const P2 ei = mul_mi(v[2]), oi = mul_mi(v[3]);
    const P2 e[4] = {cadd(v[0], v[2]), cadd(v[0], ei), csub(v[0], v[2]), csub(v[0], ei)};
    const P2 o[4] = {cadd(v[1], v[3]), cadd(v[1], oi), csub(v[1], v[3]), csub(v[1], oi)};
    dft8_join(v, e, o);
}

// exp(-2 pi i M / N) at compile time: octant-free quadrant reduction of the
// exact fraction M / N, then Taylor series on [0, pi/2) (double, ~1e-16)
constexpr double kPiC = 3.14159265358979323846;
__host__ __device__ constexpr double csin_q(double y) {
    double t = y, s = y;
    for (int k = 1; k < 14; ++k) {
        t *= -y * y / ((2.0 * k) * (2.0 * k + 1.0));
        s += t;
    }
    return s;
}
__host__ __device__ constexpr double ccos_q(double y) {
    double t = 1.0, s = 1.0;
    for (int k = 1; k < 14; ++k) {
        t *= -y * y / ((2.0 * k - 1.0) * (2.0 * k));
        s += t;
    }
    return s;
}
__host__ __device__ constexpr double ctw(int m, int n, bool sine) {
    const int mm = ((m % n) + n) % n;
    const int q = 4 * mm / n;                                  // quadrant
    const double y = 2.0 * kPiC * (double)(4 * mm - q * n) / (4.0 * n);   // in [0, pi/2)
    const double c = ccos_q(y), sn = csin_q(y);
    if (!sine) return q == 0 ? c : q == 1 ? -sn : q == 2 ? -c : sn;
    return q == 0 ? sn : q == 1 ? c : q == 2 ? -sn : -c;
}
template <int M, int N>
struct TwConst {   // exp(-2 pi i M / N)
    static constexpr float re = (float)ctw(M, N, false);
    static constexpr float im = (float)-ctw(M, N, true);
};
// exp(-2 pi i t / 1024), duplicated into both lanes: the twiddles of the column
// DFTs, one 16-byte read each
constexpr int kColMax = 1024;
struct ColTable {
    float4 w[kColMax];
};
constexpr ColTable make_col_table() {
    ColTable t{};
    for (int i = 0; i < kColMax; ++i) {
        const float c = (float)ctw(i, kColMax, false), s = (float)-ctw(i, kColMax, true);
        t.w[i].x = c;
        t.w[i].y = c;
        t.w[i].z = s;
        t.w[i].w = s;
    }
    return t;
}
__device__ const ColTable kColTable = make_col_table();

template <int R>
__device__ __forceinline__ void dftR(P2* v);

// Stage 1 of a length-A B DFT, in place: for column n2 (N2), the A-point DFT
// of v[B n1 + n2] over n1, each output k1 times exp(-2 pi i n2 k1 / (A B))
// (compile-time constants), written back to v[B k1 + n2].
template <int A, int B, int N2, int K1>
__device__ __forceinline__ void twiddle_col(P2* v, const P2* t) {
    if constexpr (K1 < A) {
        constexpr int e = N2 * K1 % (A * B);
        if constexpr (e == 0)
            v[B * K1 + N2] = t[K1];
        else if constexpr (4 * e == A * B)
            v[B * K1 + N2] = mul_mi(t[K1]);
        else
            v[B * K1 + N2] = cmul(t[K1], dup(make_float2(TwConst<e, A * B>::re, TwConst<e, A * B>::im)));
        twiddle_col<A, B, N2, K1 + 1>(v, t);
    }
}
template <int A, int B, int N2>
__device__ __forceinline__ void dft_stage1(P2* v) {
    if constexpr (N2 < B) {
        P2 t[A];
#pragma unroll
        for (int n1 = 0; n1 < A; ++n1) t[n1] = v[B * n1 + N2];
        dftR<A>(t);
        twiddle_col<A, B, N2, 0>(v, t);
        dft_stage1<A, B, N2 + 1>(v);
    }
}
// DFT of length A B in registers, natural order in and out (Cooley-Tukey,
// n = B n1 + n2, k = k1 + A k2): stage 1 above, then the B-point DFTs of
// v[B k1 + n2] over n2 back into the same slots, which leaves X[k1 + A k2] in
// v[B k1 + k2]; a compile-time register permutation restores natural order.
template <int A, int B>
__device__ __forceinline__ void dftAB(P2* v) {
    constexpr int N = A * B;
    dft_stage1<A, B, 0>(v);
#pragma unroll
    for (int k1 = 0; k1 < A; ++k1) dftR<B>(v + B * k1);
    P2 t[N];
#pragma unroll
    for (int r = 0; r < N; ++r) t[r] = v[B * (r % A) + r / A];
#pragma unroll
    for (int r = 0; r < N; ++r) v[r] = t[r];
}
template <int R>
__device__ __forceinline__ void dftR(P2* v) {
    if constexpr (R == 2) dft2(v);
    else if constexpr (R == 3) dft3(v);
    else if constexpr (R == 4) dft4(v);
    else if constexpr (R == 5) dft5(v);
    else if constexpr (R == 6) dftAB<2, 3>(v);
    else if constexpr (R == 8) dft8(v);
    else if constexpr (R == 9) dftAB<3, 3>(v);
    else if constexpr (R == 10) dftAB<2, 5>(v);
    else if constexpr (R == 12) dftAB<4, 3>(v);
}
// dispatch of a run-time radix to f(integral_constant<R>)
template <class F>
__device__ __forceinline__ void with_radix(int R, F&& f) {
    switch (R) {
        case 2: f(std::integral_constant<int, 2>()); break;
        case 3: f(std::integral_constant<int, 3>()); break;
        case 4: f(std::integral_constant<int, 4>()); break;
        case 5: f(std::integral_constant<int, 5>()); break;
        case 6: f(std::integral_constant<int, 6>()); break;
        case 9: f(std::integral_constant<int, 9>()); break;
        case 10: f(std::integral_constant<int, 10>()); break;
        case 12: f(std::integral_constant<int, 12>()); break;
        default: f(std::integral_constant<int, 8>()); break;
    }
}

// v[r] *= w^r, w = tw[s] (tw[t] = exp(-2 pi i t / n)): a table read for the
// powers 1, 2, 4 and every 4th beyond, the others by products of two.
template <int R>
__device__ __forceinline__ void twiddle(P2* v, const float2* __restrict__ tw, int s) {
    const P2 w1 = dup(__ldg(&tw[s]));
    v[1] = cmul(v[1], w1);
    if constexpr (R > 2) {
        const P2 w2 = dup(__ldg(&tw[2 * s]));
        v[2] = cmul(v[2], w2);
        const P2 w3 = R > 3 ? cmul(w1, w2) : w2;
        if constexpr (R > 3) v[3] = cmul(v[3], w3);
#pragma unroll
        for (int b = 4; b < R; b += 4) {
            const P2 wb = dup(__ldg(&tw[b * s]));
            v[b] = cmul(v[b], wb);
            if (b + 1 < R) v[b + 1] = cmul(v[b + 1], cmul(wb, w1));
            if (b + 2 < R) v[b + 2] = cmul(v[b + 2], cmul(wb, w2));
            if (b + 3 < R) v[b + 3] = cmul(v[b + 3], cmul(wb, w3));
        }
    }
}

// exp(-2 pi i t / N) from a two-level table (t = hi * 1024 + lo)
__device__ __forceinline__ float2 twiddle_n(const float2* __restrict__ hi, const float2* __restrict__ lo, int t) {
    return cmulf(__ldg(&hi[t >> 10]), __ldg(&lo[t & 1023]));
}
// the same for t and t + d: a P2
__device__ __forceinline__ P2 twiddle_n2(const float2* __restrict__ hi, const float2* __restrict__ lo, int t, int d) {
    const float2 a = twiddle_n(hi, lo, t), b = twiddle_n(hi, lo, t + d);
    return {make_float2(a.x, b.x), make_float2(a.y, b.y)};
}

// ---------------------------------------------------------------------------
// column DFTs, length n1 = 8^d, 2 8^d or 4 8^d
// ---------------------------------------------------------------------------
// A CTA takes B elements (2 B columns) of one pair, n1/8 threads per element
// with eight values each; radix-8 passes (and a last one of radix 2 or 4 over
// the same eight values) exchange through one shared buffer [n1][B].  The
// four-step twiddles of the CTA's columns are made once per CTA, in shared
// memory, while the samples are on their way.  64 registers and 256 threads:
// 1024 threads an SM.
template <int N1>
struct ColShape {
    static constexpr int TPC = N1 / 8;
    static constexpr int B = N1 >= 512 ? 4 : N1 >= 64 ? 2048 / N1 : 32;
    static constexpr int THREADS = TPC * B;
    static constexpr int CTAS = THREADS >= 256 ? 1024 / THREADS : 8;
    static constexpr int A8 = TPC >= 8 ? TPC / 8 : 1;
    static constexpr int TWS = 8 + A8 + 3;   // twiddle entries per element
    static constexpr size_t SMEM = ((N1 > 8 ? (size_t)N1 * B : 0) + (size_t)TWS * B) * sizeof(float4);
};
__device__ __forceinline__ P2 col_tw(int t) { return from4(__ldg(&kColTable.w[t])); }

// On entry v[q] = x[j + q N1/8] of element b (HALF: zero for q >= 4); on
// return v[r] = X[j + r N1/8].
template <int N1, bool HALF>
__device__ __forceinline__ void col_fft8(P2 (&v)[8], float4* sm, int j, int b) {
    constexpr int TPC = ColShape<N1>::TPC;
    constexpr int B = ColShape<N1>::B;
    if constexpr (HALF) dft8_half(v);
    else dft8(v);
    // write out[(j - k) 8 + k + Ns r] of the pass before, read in[j + q N1/8]
    auto exchange = [&](int ns) {
        const int k = j & (ns - 1);
        if (ns > 1) __syncthreads();
#pragma unroll
        for (int r = 0; r < 8; ++r) sm[((j - k) * 8 + k + ns * r) * B + b] = to4(v[r]);
        __syncthreads();
#pragma unroll
        for (int r = 0; r < 8; ++r) v[r] = from4(sm[(j + r * TPC) * B + b]);
    };
    auto pass8 = [&](int s) {   // times w^r, w = exp(-2 pi i s / 1024), and an 8-point DFT
        const P2 w1 = col_tw(s), w2 = col_tw(2 * s), w4 = col_tw(4 * s);
        const P2 w3 = cmul(w1, w2);
        v[1] = cmul(v[1], w1);
        v[2] = cmul(v[2], w2);
        v[3] = cmul(v[3], w3);
        v[4] = cmul(v[4], w4);
        v[5] = cmul(v[5], cmul(w1, w4));
        v[6] = cmul(v[6], cmul(w2, w4));
        v[7] = cmul(v[7], cmul(w3, w4));
        dft8(v);
    };
    if constexpr (N1 >= 64) {
        exchange(1);
        pass8((j & 7) * (kColMax / 64));
    }
    if constexpr (N1 >= 512) {
        exchange(8);
        pass8((j & 63) * (kColMax / 512));
    }
    constexpr int D = N1 >= 512 ? 512 : N1 >= 64 ? 64 : 8;   // done so far
    if constexpr (N1 == 2 * D) {
        exchange(D / 8);
#pragma unroll
        for (int i = 0; i < 4; ++i) {   // butterflies j + i N1/8
            const P2 t = cmul(v[i + 4], col_tw((j + i * TPC) * (kColMax / N1)));
            v[i + 4] = csub(v[i], t);
            v[i] = cadd(v[i], t);
        }
    } else if constexpr (N1 == 4 * D) {
        exchange(D / 8);
#pragma unroll
        for (int i = 0; i < 2; ++i) {
            const int m = (j + i * TPC) * (kColMax / N1);
            P2 t[4] = {v[i], cmul(v[i + 2], col_tw(m)), cmul(v[i + 4], col_tw(2 * m)), cmul(v[i + 6], col_tw(3 * m))};
            dft4(t);
#pragma unroll
            for (int r = 0; r < 4; ++r) v[i + 2 * r] = t[r];
        }
    }
}

// Four-step twiddles w_N^{n2i k1} of the CTA's elements (n2i = 2c, 2c + 1) in
// shared memory: k1 = b < 8, k1 = 8 a < n1/8, and the powers 1, 2, 4 of n1/8,
// each from the tables of N.
template <int N1>
__device__ __forceinline__ void make_four_step(float4* tws, const ColFftArgs& a, int c0) {
    using S = ColShape<N1>;
    for (int i = threadIdx.x; i < S::TWS * S::B; i += S::THREADS) {
        const int e = i / S::B, c = c0 + i % S::B;
        const int k1 = e < 8 ? e : e < 8 + S::A8 ? 8 * (e - 8) : S::TPC << (e - 8 - S::A8);
        if (c < (a.n2 >> 1)) tws[i] = to4(twiddle_n2(a.tw_hi, a.tw_lo, 2 * c * k1, k1));
    }
    __syncthreads();
}
// v[r] *= w_N^{n2i (j + r n1/8)}: products of at most five table values
template <int N1>
__device__ __forceinline__ void four_step(P2 (&v)[8], const float4* tws, int j, int b) {
    using S = ColShape<N1>;
    auto at = [&](int e) { return from4(tws[e * S::B + b]); };
    const P2 s1 = at(8 + S::A8), s2 = at(9 + S::A8), s4 = at(10 + S::A8);
    const P2 w0 = S::TPC >= 16 ? cmul(at(j & 7), at(8 + (j >> 3))) : at(j & 7);
    const P2 w1 = cmul(w0, s1), w2 = cmul(w0, s2), w3 = cmul(w1, s2);
    v[0] = cmul(v[0], w0);
    v[1] = cmul(v[1], w1);
    v[2] = cmul(v[2], w2);
    v[3] = cmul(v[3], w3);
    v[4] = cmul(v[4], cmul(w0, s4));
    v[5] = cmul(v[5], cmul(w1, s4));
    v[6] = cmul(v[6], cmul(w2, s4));
    v[7] = cmul(v[7], cmul(w3, s4));
}

template <int N1>
__device__ __forceinline__ void store_y(const P2 (&v)[8], const ColFftArgs& a, int pair, int j, int c) {
    constexpr int TPC = ColShape<N1>::TPC;
    const int h = a.n2 >> 1;
    float4* y = a.y + ((int64_t)(a.pair_base + pair) * N1 + j) * h + c;
#pragma unroll
    for (int r = 0; r < 8; ++r) y[(int64_t)r * TPC * h] = to4(v[r]);
}

// Node rows 2 pair and 2 pair + 1 of the LDM (or through the row map of the
// merged layout's narrow nodes).  Samples from n1/2 rows on are the
// transform's zero padding (N >= 2 n_v).
template <int N1>
__global__ void __launch_bounds__(ColShape<N1>::THREADS, ColShape<N1>::CTAS) k_col_fft_fwd(const ColFftArgs a) {
    constexpr int TPC = ColShape<N1>::TPC;
    constexpr int B = ColShape<N1>::B;
    extern __shared__ float4 sm[];
    float4* tws = sm + (N1 > 8 ? N1 * B : 0);
    chain_begin();
    const int b = threadIdx.x % B;
    const int j = threadIdx.x / B;
    const int c = blockIdx.x * B + b;
    const bool in = c < (a.n2 >> 1);   // the last CTA may be partly empty
    const int pair = blockIdx.y;
    auto node_of = [&](int v) {   // -1: zero row (padding of an odd n_L block)
        if (!a.map_n) return v;
        const int m = v % a.map_NLv;
        return m < a.map_NL ? a.map_l[v / a.map_NLv] * a.map_NL + m : -1;
    };
    const int na = node_of(2 * pair), nb = node_of(2 * pair + 1);
    const float* ra = a.ldm + (int64_t)max(na, 0) * a.row_stride + 2 * c;
    const float* rb = a.ldm + (int64_t)max(nb, 0) * a.row_stride + 2 * c;
    P2 v[8];
    // all loads first, masks after them.  Rows start on 128 bytes and end with
    // padding: the 8-byte read of an odd n_v's last sample stays inside.
#pragma unroll
    for (int q = 0; q < 4; ++q) {
        const int64_t o = (int64_t)(j + q * TPC) * a.n2;
        const bool ok = in && o + 2 * c < a.n_v;
        v[q].re = ok && na >= 0 ? *reinterpret_cast<const float2*>(ra + o) : dup2(0.f);
        v[q].im = ok && nb >= 0 ? *reinterpret_cast<const float2*>(rb + o) : dup2(0.f);
    }
#pragma unroll
    for (int q = 0; q < 4; ++q)   // the sample after an odd n_v's last one is padding
        if ((int64_t)(j + q * TPC) * a.n2 + 2 * c + 1 >= a.n_v) v[q].re.y = v[q].im.y = 0.f;
    make_four_step<N1>(tws, a, blockIdx.x * B);
    col_fft8<N1, true>(v, sm, j, b);
    four_step<N1>(v, tws, j, b);
    if (in) store_y<N1>(v, a, pair, j, c);
}

// Float rows 2 pair and 2 pair + 1 of a.src (the merged rows, with their
// wrap-around extension), or (a.single) the row a.src with a zero partner,
// of any alignment.
template <int N1>
__global__ void __launch_bounds__(ColShape<N1>::THREADS, ColShape<N1>::CTAS) k_col_fft_fwd_f(const ColFftArgs a) {
    constexpr int TPC = ColShape<N1>::TPC;
    constexpr int B = ColShape<N1>::B;
    extern __shared__ float4 sm[];
    float4* tws = sm + (N1 > 8 ? N1 * B : 0);
    chain_begin();
    const int b = threadIdx.x % B;
    const int j = threadIdx.x / B;
    const int c = blockIdx.x * B + b;
    const bool in = c < (a.n2 >> 1);   // the last CTA may be partly empty
    const int pair = blockIdx.y;
    const float* ra = a.src + (a.single ? 0 : (int64_t)(2 * pair) * a.row_stride);
    const float* rb = a.single ? nullptr : ra + a.row_stride;
    P2 v[8];
#pragma unroll
    for (int q = 0; q < 8; ++q) {
        float x[2] = {0.f, 0.f}, z[2] = {0.f, 0.f};
#pragma unroll
        for (int i = 0; i < 2; ++i) {
            const int64_t nidx = (int64_t)(j + q * TPC) * a.n2 + 2 * c + i;
            // buffer offset of FFT index nidx, or -1 where the row is zero
            int64_t off = -1;
            if (a.ext == 0) {
                if (nidx < a.n_v) off = nidx;
            } else if (nidx < a.n_v + a.ext) {
                off = nidx + a.ext;
            } else if (nidx >= a.n - a.ext) {
                off = nidx - (a.n - a.ext);
            }
            if (in && off >= 0) {
                x[i] = ra[off];
                if (rb) z[i] = rb[off];
            }
        }
        v[q] = {make_float2(x[0], x[1]), make_float2(z[0], z[1])};
    }
    make_four_step<N1>(tws, a, blockIdx.x * B);
    col_fft8<N1, false>(v, sm, j, b);
    four_step<N1>(v, tws, j, b);
    if (in) store_y<N1>(v, a, pair, j, c);
}

// Post-processing epilogue (radis/lbl/factory.py:1284-1297 and
// radis/spectrum/equations.py:21-44): absorbance A L, emissivity
// -expm1(-A L), transmittance 1 - emissivity, radiance emissivity x Planck
// (radis/phys/blackbody.py:35-74, mW / cm2 / sr / nm at lambda = 1e7/nu nm).
__device__ __forceinline__ void quantities_at(const ColFftArgs& a, int64_t k, float A) {
    const float tau = A * a.q_scale * a.q_path;      // absorbance in physical units
    const float eps = -expm1f(-tau);
    const float nu = (float)(a.q_vmin + a.q_dv * (double)k);
    const float lam = 0.01f / nu;                    // m
    // 2 h c^2 / lambda^5 / expm1(h c / (lambda k T)) W m-3 sr-1 -> mW cm-2 sr-1 nm-1 (x 1e-10)
    const float l2 = lam * lam;
    const float planck = 1.19104297e-16f / (l2 * l2 * lam) / expm1f(a.q_c2_T * nu) * 1e-10f;
    const int64_t n = a.n_v;
    a.q_out[k] = A * a.q_path;
    a.q_out[n + k] = eps;
    a.q_out[2 * n + k] = 1.f - eps;
    a.q_out[3 * n + k] = eps * planck;
}

// The inverse row DFTs arrive as conj(z) (a forward DFT of conj(G)), so the
// inverse column DFT conj(DFT(conj(.))) and the inverse twiddle conj(w) are a
// forward twiddle and a forward DFT of what is read.  Only the samples of the
// first n1/2 rows are kept.
template <int N1>
__device__ __forceinline__ void inverse_columns(P2 (&v)[8], const ColFftArgs& a, const float4* src, float4* sm,
                                                float4* tws, int j, int b, int c, bool in) {
    constexpr int TPC = ColShape<N1>::TPC;
    const int h = a.n2 >> 1;
    const float4* s = src + (int64_t)j * h + c;
#pragma unroll
    for (int q = 0; q < 8; ++q) v[q] = in ? from4(s[(int64_t)q * TPC * h]) : zero_p2();
    make_four_step<N1>(tws, a, c - b);
    four_step<N1>(v, tws, j, b);
    col_fft8<N1, false>(v, sm, j, b);
}

template <int N1>
__global__ void __launch_bounds__(ColShape<N1>::THREADS, ColShape<N1>::CTAS) k_col_ifft(const ColFftArgs a) {
    constexpr int TPC = ColShape<N1>::TPC;
    constexpr int B = ColShape<N1>::B;
    extern __shared__ float4 sm[];
    float4* tws = sm + (N1 > 8 ? N1 * B : 0);
    chain_begin();
    const int b = threadIdx.x % B;
    const int j = threadIdx.x / B;
    const int c = blockIdx.x * B + b;
    const bool in = c < (a.n2 >> 1);   // the last CTA may be partly empty
    P2 v[8];
    inverse_columns<N1>(v, a, a.h, sm, tws, j, b, c, in);
#pragma unroll
    for (int r = 0; r < 4; ++r) {
        const int64_t k = in ? (int64_t)(j + r * TPC) * a.n2 + 2 * c : a.n_v;
        const float2 A = make_float2(v[r].re.x * a.out_scale, v[r].re.y * a.out_scale);   // Re(conj(z)) = Re(z)
        if (k + 1 < a.n_v && a.out_vec) {
            *reinterpret_cast<float2*>(a.out + k) = A;
        } else {
            if (k < a.n_v) a.out[k] = A.x;
            if (k + 1 < a.n_v) a.out[k + 1] = A.y;
        }
        if (a.q_out) {
            if (k < a.n_v) quantities_at(a, k, A.x);
            if (k + 1 < a.n_v) quantities_at(a, k + 1, A.y);
        }
    }
    // last kernel of the spectrum: hand the error flag to the host (mapped
    // memory, read after the stream synchronises) and clear it
    if (a.err_pub && blockIdx.x == 0 && threadIdx.x == 0) {
        *a.err_pub = *a.err;
        *a.err = 0u;
    }
}

// Adjoint column stage: real part of pair `blockIdx.y` -> float row 2 pair,
// imaginary part -> row 2 pair + 1 of a.out (first n_v samples, x out_scale).
template <int N1>
__global__ void __launch_bounds__(ColShape<N1>::THREADS, ColShape<N1>::CTAS) k_col_ifft_adj(const ColFftArgs a) {
    constexpr int TPC = ColShape<N1>::TPC;
    constexpr int B = ColShape<N1>::B;
    extern __shared__ float4 sm[];
    float4* tws = sm + (N1 > 8 ? N1 * B : 0);
    chain_begin();
    const int b = threadIdx.x % B;
    const int j = threadIdx.x / B;
    const int c = blockIdx.x * B + b;
    const bool in = c < (a.n2 >> 1);   // the last CTA may be partly empty
    const int pair = blockIdx.y;
    P2 v[8];
    inverse_columns<N1>(v, a, a.h + (int64_t)pair * N1 * (a.n2 >> 1), sm, tws, j, b, c, in);
    float* oa = a.out + (int64_t)(2 * pair) * a.row_stride + 2 * c;
#pragma unroll
    for (int r = 0; r < 4; ++r) {
        const int64_t o = (int64_t)(j + r * TPC) * a.n2;
        if (in && o + 2 * c < a.n_v) {   // an odd n_v's last pair ends in the row's padding
            *reinterpret_cast<float2*>(oa + o) = make_float2(v[r].re.x * a.out_scale, v[r].re.y * a.out_scale);
            *reinterpret_cast<float2*>(oa + a.row_stride + o) =
                make_float2(-v[r].im.x * a.out_scale, -v[r].im.y * a.out_scale);   // Im(conj(z))
        }
    }
}

// ---------------------------------------------------------------------------
// Voigt transforms
// ---------------------------------------------------------------------------
// Arguments of the row kernels: geometry and one 16-byte record per
// transformed row, so that a bin's two nodes take two uniform loads.  CAP: 64
// rows (1 KB of parameters; the skeleton and most merged layouts), or every
// node of the largest grid.
template <int CAP>
struct RowArgs {
    FftLen f;
    int n1, n_pairs, units, bins, any_fold;
    int half_n;           // N / 2
    float inv_ndv, half_fs;
    const float4* y;
    float4* g;
    float4* out;          // adjoint: inverse rows [pair][n1][h]
    // unfolded rows: (-alpha, -beta, log2 norm, 0): nrm 2^-(al f^2 + bm f) =
    // 2^(lnrm - bm f - al f^2), two FMAs and one ex2; with folded copies in
    // the grid: (alpha, beta, norm, copies)
    float4 node[CAP];
};
// One node's transform at the two frequencies f (f2 = f^2).  FOLD: with its
// folded copies (broadening.py:1914-1926) at q/(2 dv) + (f or 1/(2 dv) - f);
// the node, and so their number, is the same for the whole CTA.
template <bool FOLD>
__device__ __forceinline__ float2 voigt_of(float4 n, float half_fs, float2 f, float2 f2) {
    if constexpr (!FOLD) {
        const float2 e = __ffma2_rn(dup2(n.x), f2, __ffma2_rn(dup2(n.y), f, dup2(n.z)));
        return make_float2(ex2(e.x), ex2(e.y));
    }
    auto at = [&](float2 g) {
        const float2 e = __ffma2_rn(__fmul2_rn(dup2(n.x), g), g, __fmul2_rn(dup2(n.y), g));
        return make_float2(ex2(-e.x), ex2(-e.y));
    };
    float2 v = at(f);
    const int nf = (int)n.w;
    for (int q = 1; q <= nf; ++q) {
        const float b = q * half_fs;
        v = __fadd2_rn(v, at(q & 1 ? make_float2(b + (half_fs - f.x), b + (half_fs - f.y)) : make_float2(b + f.x, b + f.y)));
    }
    return __fmul2_rn(v, dup2(n.z));
}
// frequencies of bins k2 = t and t + h of row k1 (the second is aliased from
// the negative side: N - k = N/2 - (k1 + n1 t))
template <class A>
__device__ __forceinline__ float2 bin_freqs(const A& a, int k1, int t) {
    const int kk = k1 + a.n1 * t;
    return make_float2((float)kk * a.inv_ndv, (float)(a.half_n - kk) * a.inv_ndv);
}

// ---------------------------------------------------------------------------
// row DFTs
// ---------------------------------------------------------------------------
// Stockham passes over `units` transforms of length h = f.L side by side, one
// butterfly per thread and step: butterfly j of a transform reads in[j + r
// M], M = h / R, twiddles by w_{Ns R}^{r (j mod Ns)} and writes out[(j / Ns)
// Ns R + (j mod Ns) + r Ns].  The first pass writes runs of R elements; with
// even R the buffer skips one element after each run (rpad), so that the
// strided 16-byte writes spread over the banks; the second pass reads them so,
// later passes use plain indices.  The pass twiddles come from the table of
// n2 = 2 h entries, read through L1.
__device__ __forceinline__ int rpad(int i, unsigned mag) { return i + (int)__umulhi((unsigned)i, mag); }

template <int R, bool FIRST, class LD>
__device__ __forceinline__ void row_pass(const FftLen& f, int p, int units, float4* out, int ub, LD ld) {
    const int M = f.L / R;
    const int items = units * M;
    const int Ns = FIRST ? 1 : f.ns[p];
    const unsigned mag = f.mag[p], mm = f.mag_m[p], pm = f.pad_mag;
    const int ts = FIRST ? 0 : 2 * f.L / (Ns * R);
    for (int i = threadIdx.x; i < items; i += blockDim.x) {
        const int u = (int)__umulhi((unsigned)i, mm);
        const int j = i - u * M;
        const int q = FIRST ? j : (int)__umulhi((unsigned)j, mag);
        const int k = FIRST ? 0 : j - q * Ns;
        P2 v[R];
        ld(v, u, j, M);
        if (!FIRST) twiddle<R>(v, f.tw, k * ts);
        dftR<R>(v);
        float4* o = out + u * ub;
        if constexpr (FIRST) {
            o += rpad(j * R, pm);
#pragma unroll
            for (int r = 0; r < R; ++r) o[r] = to4(v[r]);
        } else {
            o += q * Ns * R + k;
#pragma unroll
            for (int r = 0; r < R; ++r) o[r * Ns] = to4(v[r]);
        }
    }
}

// first pass: `src(u)` = element 0 of transform u
template <class SRC>
__device__ __forceinline__ void row_first(const FftLen& f, int units, float4* out, int ub, SRC src) {
    with_radix(f.radix[0], [&](auto rc) {
        constexpr int R = decltype(rc)::value;
        row_pass<R, true>(f, 0, units, out, ub, [&](P2* v, int u, int j, int M) {
            const float4* s = src(u) + j;
#pragma unroll
            for (int r = 0; r < R; ++r) v[r] = from4(s[r * M]);
        });
    });
    __syncthreads();
}

template <bool PIN>
__device__ __forceinline__ void row_mid(const FftLen& f, int p, int units, const float4* in, int ub, float4* out,
                                        int out_ub) {
    with_radix(f.radix[p], [&](auto rc) {
        constexpr int R = decltype(rc)::value;
        row_pass<R, false>(f, p, units, out, out_ub, [&](P2* v, int u, int j, int M) {
            const float4* s = in + u * ub;
#pragma unroll
            for (int r = 0; r < R; ++r) v[r] = from4(s[PIN ? rpad(j + r * M, f.pad_mag) : j + r * M]);
        });
    });
}

// passes 1 .. npass - 1 over what row_first left in buf0, through buf1 and
// back; GLOBAL: the last pass writes `dst` (unit stride dst_ub), else the
// result's buffer is returned, after a barrier.
template <bool GLOBAL>
__device__ __forceinline__ float4* row_rest(const FftLen& f, int units, float4* buf0, float4* buf1, int ub,
                                            float4* dst, int dst_ub) {
    float4* in = buf0;
    float4* out = buf1;
    const int n = GLOBAL ? f.npass - 1 : f.npass;
    for (int p = 1; p < n; ++p) {
        if (p == 1) row_mid<true>(f, p, units, in, ub, out, ub);
        else row_mid<false>(f, p, units, in, ub, out, ub);
        __syncthreads();
        float4* t = in;
        in = out;
        out = t;
    }
    if constexpr (GLOBAL) {
        if (n == 1) row_mid<true>(f, n, units, in, ub, dst, dst_ub);
        else row_mid<false>(f, n, units, in, ub, dst, dst_ub);
    }
    return in;
}

// the radix-2 join of a length-n2 DFT from the even (x) and odd (y) lanes at
// bin t: lanes X[t], X[t + h]
__device__ __forceinline__ P2 join2(P2 e, float2 w) {
    const float2 o = cmulf(make_float2(e.re.y, e.im.y), w);
    return {make_float2(e.re.x + o.x, e.re.x - o.x), make_float2(e.im.x + o.y, e.im.x - o.y)};
}
// the radix-2 split that starts the inverse DFT, on conj(G): lanes
// (D_t + D_{t+h}, (D_t - D_{t+h}) w^t), D = conj(G)
__device__ __forceinline__ P2 split2(P2 g, float2 w) {
    const float2 s = make_float2(g.re.x + g.re.y, -(g.im.x + g.im.y));
    const float2 d = cmulf(make_float2(g.re.x - g.re.y, g.im.y - g.im.x), w);
    return {make_float2(s.x, d.x), make_float2(s.y, d.y)};
}

// One thread per bin pair (t, t + h) of a row: joins the lanes of `nu` pairs'
// spectra x, applies their Voigt weights and adds them up; the sum goes to
// `sum` (more pairs to come), to g, or, split for the inverse, to `split`.
template <bool FOLD, class A>
__device__ __forceinline__ void weigh(const A& a, const float4* x, int ub, int j0, int nu, bool last, float4* sum,
                                      float4* split, int k1) {
    const int h = a.f.L;
    for (int t = threadIdx.x; t < h; t += blockDim.x) {
        P2 c = j0 ? from4(sum[t]) : zero_p2();
        const float2 w = __ldg(&a.f.tw[t]);
        const float2 fr = bin_freqs(a, k1, t), f2 = __fmul2_rn(fr, fr);
        for (int u = 0; u < nu; ++u) {
            const P2 z = join2(from4(x[u * ub + t]), w);
            const float2 va = voigt_of<FOLD>(a.node[2 * (j0 + u)], a.half_fs, fr, f2);
            const float2 vb = voigt_of<FOLD>(a.node[2 * (j0 + u) + 1], a.half_fs, fr, f2);
            // G += Z (V_a - i V_b)
            c.re = __ffma2_rn(z.re, va, __ffma2_rn(z.im, vb, c.re));
            c.im = __ffma2_rn(z.im, va, __ffma2_rn(neg2(z.re), vb, c.im));
        }
        if (!last) sum[t] = to4(c);
        else if (a.bins) a.g[(int64_t)k1 * h + t] = to4(c);
        else split[t] = to4(split2(c, w));
    }
}

// One CTA: row k1 of every pair, a.units pairs at a time: their DFTs pass by
// pass side by side in two shared buffers, then the weights and the sum; the
// inverse row DFT of the sum (bins == 0) goes straight to g, or (bins) the sum
// itself.
template <int CAP>
__global__ void __launch_bounds__(kRowMaxThreads, 1) k_row_fft_voigt(const RowArgs<CAP> a) {
    extern __shared__ float4 sm4[];
    chain_begin();
    const FftLen& f = a.f;
    const int h = f.L;
    const int ub = f.row_len;
    float4* buf0 = sm4;
    float4* buf1 = buf0 + a.units * ub;
    float4* sum = buf1 + a.units * ub;   // [h], only with more than one batch
    const int k1 = blockIdx.x;
    float4* free_buf = buf0;   // what the weights below do not read
    float4* x = buf1;
    for (int j0 = 0; j0 < a.n_pairs; j0 += a.units) {
        const int nu = min(a.units, a.n_pairs - j0);
        float4* first = free_buf;
        float4* second = x;
        row_first(f, nu, first, ub, [&](int u) { return a.y + ((int64_t)(j0 + u) * a.n1 + k1) * h; });
        x = row_rest<false>(f, nu, first, second, ub, nullptr, 0);
        free_buf = x == first ? second : first;
        const bool last = j0 + a.units >= a.n_pairs;
        if (a.any_fold) weigh<true>(a, x, ub, j0, nu, last, sum, free_buf, k1);
        else weigh<false>(a, x, ub, j0, nu, last, sum, free_buf, k1);
    }
    if (a.bins) return;
    __syncthreads();
    // the inverse's first pass reads the split bins and overwrites the spectra
    row_first(f, 1, x, ub, [&](int) { return free_buf; });
    row_rest<true>(f, 1, x, free_buf, ub, a.g + (int64_t)k1 * h, 0);
}

// Adjoint row stage, one CTA per row k1 and a.units pairs: H = Ghat (V_2j + i
// V_2j+1) on the row's bins, inverse row DFT; output [j][k1][c].
template <bool FOLD, class A>
__device__ __forceinline__ void weigh_adj(const A& a, float4* out, int ub, int j0, int nu, int k1) {
    const int h = a.f.L;
    for (int t = threadIdx.x; t < h; t += blockDim.x) {
        const P2 z = from4(a.g[(int64_t)k1 * h + t]);
        const float2 w = __ldg(&a.f.tw[t]);
        const float2 fr = bin_freqs(a, k1, t), f2 = __fmul2_rn(fr, fr);
        for (int u = 0; u < nu; ++u) {
            const float2 va = voigt_of<FOLD>(a.node[2 * (j0 + u)], a.half_fs, fr, f2);
            const float2 vb = voigt_of<FOLD>(a.node[2 * (j0 + u) + 1], a.half_fs, fr, f2);
            P2 c;
            c.re = __ffma2_rn(z.re, va, neg2(__fmul2_rn(z.im, vb)));
            c.im = __ffma2_rn(z.im, va, __fmul2_rn(z.re, vb));
            out[u * ub + t] = to4(split2(c, w));
        }
    }
}
template <int CAP>
__global__ void __launch_bounds__(kRowMaxThreads, 1) k_row_ifft_adj(const RowArgs<CAP> a) {
    extern __shared__ float4 sm4[];
    chain_begin();
    const FftLen& f = a.f;
    const int h = f.L;
    const int ub = f.row_len;
    float4* buf0 = sm4;
    float4* buf1 = buf0 + a.units * ub;
    const int k1 = blockIdx.x;
    const int j0 = blockIdx.y * a.units;
    const int nu = min(a.units, a.n_pairs - j0);
    if (a.any_fold) weigh_adj<true>(a, buf0, ub, j0, nu, k1);
    else weigh_adj<false>(a, buf0, ub, j0, nu, k1);
    __syncthreads();
    row_first(f, nu, buf1, ub, [&](int u) { return buf0 + u * ub; });
    row_rest<true>(f, nu, buf1, buf0, ub, a.out + ((int64_t)j0 * a.n1 + k1) * h, a.n1 * h);
}

// ---------------------------------------------------------------------------
// launchers
// ---------------------------------------------------------------------------
template <int N1, class K>
static int launch_col(K kernel, const ColFftArgs& a, int pairs, cudaStream_t st) {
    dim3 grid((a.n2 / 2 + ColShape<N1>::B - 1) / ColShape<N1>::B, pairs);
    return launch_chained(kernel, grid, ColShape<N1>::THREADS, ColShape<N1>::SMEM, st, a);
}
#define RG_COL(name, fn, pairs)                                             \
    template <int N1>                                                       \
    static int name##_n1(const ColFftArgs& a, cudaStream_t st) {            \
        ALLOW_SMEM(fn<N1>, ColShape<N1>::SMEM);                             \
        return launch_col<N1>(fn<N1>, a, pairs, st);                        \
    }                                                                       \
    int name(const ColFftArgs& a, cudaStream_t st) {                        \
        switch (a.n1) {                                                     \
            case 8: return name##_n1<8>(a, st);                                \
            case 16: return name##_n1<16>(a, st);                              \
            case 32: return name##_n1<32>(a, st);                              \
            case 64: return name##_n1<64>(a, st);                              \
            case 128: return name##_n1<128>(a, st);                            \
            case 256: return name##_n1<256>(a, st);                            \
            case 512: return name##_n1<512>(a, st);                            \
            case 1024: return name##_n1<1024>(a, st);                          \
            default: return RG_ERR_RANGE;                                   \
        }                                                                   \
    }
RG_COL(launch_col_fft_fwd, k_col_fft_fwd, a.n_pairs)
RG_COL(launch_col_fft_fwd_f, k_col_fft_fwd_f, (a.single ? 1 : a.n_pairs))
RG_COL(launch_col_ifft, k_col_ifft, 1)
RG_COL(launch_col_ifft_adj, k_col_ifft_adj, a.n_pairs)

static size_t row_smem(const FftLen& f, int units, bool batches) {
    return sizeof(float4) * ((size_t)2 * units * f.row_len + (batches ? f.L : 0));
}

// Pairs side by side and threads of the row kernels.  All rows resident at
// once when that takes at most four CTAs an SM (n1 = 512 rows on 152 SMs: four
// of 56 KB; 256: two of 112 KB), then as many pairs as fit: fewer barriers per
// row.  Threads: a butterfly of ~8 points each, about two per thread where the
// grid fills the machine, within 80 registers x threads of the resident CTAs.
// (GB300 sweeps over units x threads: 400-point transforms of 6 pairs, 512
// rows: 3 x 160 threads 18.7 us, 2 x 160 20.7, 6 x 256 22.5; 480 points, 256
// rows: 6 x 288 15.0, 3 x 320 16.5; 800 points, 512 rows: 1 x 160 37.1, 3 x 320
// 41.3; 1536 points of 11 pairs, 1024 rows: 1 x 384 283, 3 x 768 290.)  The
// adjoint's rows are independent: one pair per CTA.
RowShape row_shape(const FftLen& f, int n1, int n_pairs, int sms, bool adjoint) {
    RowShape s{};
    const size_t room = (size_t)224 * 1024;
    const int want = adjoint ? 4 : std::max(1, std::min(4, (n1 + sms - 1) / std::max(sms, 1)));
    s.units = 1;
    if (!adjoint)
        while (s.units < n_pairs && row_smem(f, s.units + 1, s.units + 1 < n_pairs) <= room / want) ++s.units;
    const size_t smem = row_smem(f, s.units, !adjoint && s.units < n_pairs);
    const int ctas = (int)std::max<size_t>(1, std::min<size_t>(want, room / smem));
    const int points = s.units * f.L;
    const int t = points <= 1100 || ctas < want ? points / 4 : points * 2 / 15;
    const int cap = std::min(kRowMaxThreads, 800 / ctas / 32 * 32);
    s.threads = std::max(64, std::min(cap, (t + 16) / 32 * 32));
    return s;
}

template <int CAP>
static int launch_row(const VoigtArgs& v, float4* adj_out, cudaStream_t st) {
    RowArgs<CAP> a;
    a.f = v.f2;
    a.n1 = v.n1;
    a.n_pairs = v.n_pairs;
    a.units = v.units;
    a.bins = v.bins;
    a.any_fold = v.any_fold;
    a.half_n = (int)(v.n / 2);
    a.inv_ndv = v.inv_ndv;
    a.half_fs = v.half_fs;
    a.y = v.y;
    a.g = v.g;
    a.out = adj_out;
    for (int r = 0; r < 2 * v.n_pairs; ++r) {
        const float al = v.alpha[v.rowwise ? r : r / v.NL], bm = v.beta[v.rowwise ? r : r % v.NL];
        a.node[r] = v.any_fold ? float4{al, bm, v.norm[r], (float)v.nfold[r]} : float4{-al, -bm, v.lnorm[r], 0.f};
    }
    const bool adj = adj_out != nullptr;
    const size_t smem = row_smem(v.f2, v.units, !adj && v.units < v.n_pairs);
    if (adj) {
        ALLOW_SMEM(k_row_ifft_adj<CAP>, smem);
        return launch_chained(k_row_ifft_adj<CAP>, dim3(v.n1, (v.n_pairs + v.units - 1) / v.units), v.threads, smem, st, a);
    }
    ALLOW_SMEM(k_row_fft_voigt<CAP>, smem);
    return launch_chained(k_row_fft_voigt<CAP>, v.n1, v.threads, smem, st, a);
}
static int launch_row_any(const VoigtArgs& v, float4* adj_out, cudaStream_t st) {
    if (v.f2.L != v.n2 / 2 || v.f2.npass < 2 || v.units < 1 || v.threads < 32 || v.threads > kRowMaxThreads || v.threads % 32 ||
        2 * v.n_pairs > kMaxNodes || v.n > ((int64_t)1 << 31))
        return RG_ERR_RANGE;
    return 2 * v.n_pairs <= 64 ? launch_row<64>(v, adj_out, st) : launch_row<kMaxNodes>(v, adj_out, st);
}
int launch_row_fft_voigt(const VoigtArgs& a, cudaStream_t st) { return launch_row_any(a, nullptr, st); }
int launch_row_ifft_adj(const AdjRowArgs& a, cudaStream_t st) { return launch_row_any(a.v, a.y, st); }

}  // namespace rg
