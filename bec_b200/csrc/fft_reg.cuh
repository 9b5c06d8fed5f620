// fft_reg.cuh -- register-resident DFTs of compile-time size.
//
// A thread holds a whole line (N <= 32 elements) in registers; the DFT is a
// fully unrolled radix-2 Cooley-Tukey recursion whose twiddles are
// compile-time constants, so trivial twiddles (1, -i, +i) cost nothing and
// the rest become FMA immediates of six-FMA butterflies (bfly_w). Elements are float2 (one complex value) or
// cpair (the two components a, b of one cell, transformed together by packed FP32x2 instructions).
//
// Twiddle values come from cos_2pi / sin_2pi below: exact octant reduction on the
// integer angle 2 pi k / n, then Taylor series on [0, pi/2) in double
// precision (error ~1e-16), evaluated by the compiler.
#pragma once

#include <utility>

#include "common.cuh"
#include "twiddle_fp32.h"

namespace fftreg {

constexpr double kPi = 3.14159265358979323846264338327950288;

__host__ __device__ constexpr double taylor_sin(double x)
{
    double t = x, s = x;
    for (int i = 1; i < 24; ++i) {
        t *= -x * x / ((2.0 * i) * (2.0 * i + 1.0));
        s += t;
    }
    return s;
}

__host__ __device__ constexpr double taylor_cos(double x)
{
    double t = 1.0, s = 1.0;
    for (int i = 1; i < 24; ++i) {
        t *= -x * x / ((2.0 * i - 1.0) * (2.0 * i));
        s += t;
    }
    return s;
}

// cos(2 pi k / n) and sin(2 pi k / n) for integer k, n > 0
__host__ __device__ constexpr double cos_2pi(long k, long n)
{
    k %= n;
    if (k < 0) k += n;
    const long q = (4 * k) / n, r = 4 * k - q * n;
    const double a = (kPi / 2.0) * (double)r / (double)n;
    const double sa = taylor_sin(a), ca = taylor_cos(a);
    return q == 0 ? ca : q == 1 ? -sa : q == 2 ? -ca : sa;
}

__host__ __device__ constexpr double sin_2pi(long k, long n)
{
    k %= n;
    if (k < 0) k += n;
    const long q = (4 * k) / n, r = 4 * k - q * n;
    const double a = (kPi / 2.0) * (double)r / (double)n;
    const double sa = taylor_sin(a), ca = taylor_cos(a);
    return q == 0 ? sa : q == 1 ? ca : q == 2 ? -sa : -ca;
}

// ---- packed pairs ------------------------------------------------------------
// Two FP32 values in one 64-bit register, operated on by one packed instruction (fma.rn.f32x2 and the like,
// sm_100): each half rounds exactly as the scalar instruction does. A packed FMA takes the FMA pipe twice as long
// as a scalar one (62.9 against 121.2 thread-instructions per clock and SM, measured), so the transforms alone gain
// nothing (0.147 clocks per point and SM for a 16-point DFT in scalar FMAs, 0.155 packed, at 20 warps per SM); the
// passes are bound by issue, and there the freed slots count: on 365 trajectories of 32x32x256 the plane pass went
// from 352.7 to 303.5 thread-instructions per cell and from 1.288 to 1.257 ms, the nz = 256 pencil pass from 0.632
// to 0.614 ms, on 333 of 16x16x128 from 0.140 to 0.131 and from 0.0686 to 0.0666 ms; the same bits.
typedef unsigned long long f32x2;

__device__ __forceinline__ f32x2 pack2(float a, float b)
{
    f32x2 r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b));
    return r;
}
__device__ __forceinline__ f32x2 both(float a) { return pack2(a, a); }
__device__ __forceinline__ float2 unpack2(f32x2 v)
{
    float2 r;
    asm("mov.b64 {%0, %1}, %2;" : "=f"(r.x), "=f"(r.y) : "l"(v));
    return r;
}
__device__ __forceinline__ f32x2 fma2(f32x2 a, f32x2 b, f32x2 c)
{
    f32x2 d;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
    return d;
}
__device__ __forceinline__ f32x2 mul2(f32x2 a, f32x2 b)
{
    f32x2 d;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
    return d;
}
__device__ __forceinline__ f32x2 add2(f32x2 a, f32x2 b)
{
    f32x2 d;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
    return d;
}
__device__ __forceinline__ f32x2 sub2(f32x2 a, f32x2 b)
{
    f32x2 d;
    asm("sub.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
    return d;
}

// The two components of one cell: re = (a.re, b.re), im = (a.im, b.im), the order in which a cell is stored.
struct __align__(16) cpair {
    f32x2 re, im;
};
__device__ __forceinline__ cpair make_cpair(float2 a, float2 b) { return cpair{pack2(a.x, b.x), pack2(a.y, b.y)}; }
// (a.re, a.im) and (b.re, b.im)
__device__ __forceinline__ float2 comp_a(const cpair &v) { return make_float2(unpack2(v.re).x, unpack2(v.im).x); }
__device__ __forceinline__ float2 comp_b(const cpair &v) { return make_float2(unpack2(v.re).y, unpack2(v.im).y); }

// ---- element operations ----------------------------------------------------
__device__ __forceinline__ float2 add(float2 a, float2 b) { return make_float2(a.x + b.x, a.y + b.y); }
__device__ __forceinline__ float2 sub(float2 a, float2 b) { return make_float2(a.x - b.x, a.y - b.y); }
__device__ __forceinline__ cpair add(cpair a, cpair b) { return cpair{add2(a.re, b.re), add2(a.im, b.im)}; }
__device__ __forceinline__ cpair sub(cpair a, cpair b) { return cpair{sub2(a.re, b.re), sub2(a.im, b.im)}; }

// Complex products with the fused multiply-adds written out, so that a float2 and a cpair caller round
// every component the same way (left to the compiler, the contraction of a*b - c*d can differ between them).
// v * (c + i s)
__device__ __forceinline__ float2 cmulc(float2 v, float c, float s)
{
    return make_float2(fmaf(v.x, c, -(v.y * s)), fmaf(v.x, s, v.y * c));
}
// the same on both components, the factor as packed pairs (c, c), (s, s), (-s, -s)
__device__ __forceinline__ cpair cmul2(cpair v, f32x2 c, f32x2 s, f32x2 ns)
{
    return cpair{fma2(v.re, c, mul2(v.im, ns)), fma2(v.re, s, mul2(v.im, c))};
}
__device__ __forceinline__ cpair cmulc(cpair v, float c, float s) { return cmul2(v, both(c), both(s), both(-s)); }
// v * (-i), v * (+i)
__device__ __forceinline__ float2 mul_negi(float2 v) { return make_float2(v.y, -v.x); }
__device__ __forceinline__ float2 mul_posi(float2 v) { return make_float2(-v.y, v.x); }

// (a - b) * (+i), without a negation of its own for packed pairs
__device__ __forceinline__ float2 sub_posi(float2 a, float2 b) { return mul_posi(sub(a, b)); }
__device__ __forceinline__ cpair sub_posi(cpair a, cpair b) { return cpair{sub2(b.im, a.im), sub2(a.re, b.re)}; }

// v * w with w a runtime complex (float2). On a cell by scalar instructions: packed ones would need the factor
// duplicated, (c, c), (s, s) and (-s, -s), by three moves or a table three times as large (measured on the nz = 256
// pencil pass: 0.613 ms with scalar, 0.639 ms with packed products).
__device__ __forceinline__ float2 cmulw(float2 v, float2 w) { return cmulc(v, w.x, w.y); }
__device__ __forceinline__ cpair cmulw(cpair v, float2 w)
{
    return make_cpair(cmulc(comp_a(v), w.x, w.y), cmulc(comp_b(v), w.x, w.y));
}
// m0 a + m1 b, every rounding fixed
__device__ __forceinline__ float2 cmix(float2 m0, float2 a, float2 m1, float2 b)
{
    return make_float2(fmaf(m0.x, a.x, fmaf(-m0.y, a.y, fmaf(m1.x, b.x, -(m1.y * b.y)))),
                       fmaf(m0.x, a.y, fmaf(m0.y, a.x, fmaf(m1.x, b.y, m1.y * b.x))));
}

// ---- butterfly with a constant twiddle -------------------------------------------
// x0 = e + w o, x1 = e - w o for the compile-time twiddle w = c + i s, in six FMAs per complex value
// (Linzer and Feig, "Implementation of efficient FFT algorithms on fused multiply-add architectures",
// IEEE Trans. Signal Processing 41, 1993): the larger of |c|, |s| is factored out, so with r = s / c
// (or c / s) of magnitude <= 1, w o = c (o.re - r o.im, o.im + r o.re) (or s (r o.re - o.im, o.re + r o.im)),
// and both outputs are one FMA each from e.
__device__ __forceinline__ void bfly_c(float2 &x0, float2 &x1, float2 e, float2 o, float f, float r)
{
    const float ur = fmaf(-r, o.y, o.x), ui = fmaf(r, o.x, o.y);
    x0 = make_float2(fmaf(f, ur, e.x), fmaf(f, ui, e.y));
    x1 = make_float2(fmaf(-f, ur, e.x), fmaf(-f, ui, e.y));
}
__device__ __forceinline__ void bfly_s(float2 &x0, float2 &x1, float2 e, float2 o, float f, float r)
{
    const float ur = fmaf(r, o.x, -o.y), ui = fmaf(r, o.y, o.x);
    x0 = make_float2(fmaf(f, ur, e.x), fmaf(f, ui, e.y));
    x1 = make_float2(fmaf(-f, ur, e.x), fmaf(-f, ui, e.y));
}

__device__ __forceinline__ void bfly_c(cpair &x0, cpair &x1, cpair e, cpair o, float f, float r)
{
    const f32x2 F = both(f), NF = both(-f);
    const f32x2 ur = fma2(both(-r), o.im, o.re), ui = fma2(both(r), o.re, o.im);
    x0 = cpair{fma2(F, ur, e.re), fma2(F, ui, e.im)};
    x1 = cpair{fma2(NF, ur, e.re), fma2(NF, ui, e.im)};
}
__device__ __forceinline__ void bfly_s(cpair &x0, cpair &x1, cpair e, cpair o, float f, float r)
{
    const f32x2 F = both(f), NF = both(-f);
    const f32x2 nur = fma2(both(-r), o.re, o.im), ui = fma2(both(r), o.im, o.re);   // nur = -ur
    x0 = cpair{fma2(NF, nur, e.re), fma2(F, ui, e.im)};
    x1 = cpair{fma2(F, nur, e.re), fma2(NF, ui, e.im)};
}
// x0 = e + i o, x1 = e - i o (INV) or e - i o, e + i o
template <bool INV>
__device__ __forceinline__ void bfly_i(float2 &x0, float2 &x1, float2 e, float2 o)
{
    const float2 t = INV ? mul_posi(o) : mul_negi(o);
    x0 = add(e, t);
    x1 = sub(e, t);
}
template <bool INV>
__device__ __forceinline__ void bfly_i(cpair &x0, cpair &x1, cpair e, cpair o)
{
    const cpair p{sub2(e.re, o.im), add2(e.im, o.re)}, m{add2(e.re, o.im), sub2(e.im, o.re)};
    x0 = INV ? p : m;
    x1 = INV ? m : p;
}

// the butterfly of twiddle w = e^{-+2 pi i K / N} (sign - forward, + when INV)
// UNIT: the factors of modulus closest to 1 (twiddle_fp32.h; the real-time passes, where a modulus error
// drains the norm at every step), else the nearest FP32 factors (the imaginary-time passes, which
// renormalise at every step and gain nothing from the modulus)
template <int K, int N, bool INV, bool UNIT = true, typename T>
__device__ __forceinline__ void bfly_w(T &x0, T &x1, T e, T o)
{
    constexpr double c = cos_2pi(K, N), s = INV ? sin_2pi(K, N) : -sin_2pi(K, N);
    if constexpr ((c < 0 ? -c : c) >= (s < 0 ? -s : s)) {
        constexpr Twid t = UNIT ? unit_fr(c, s / c) : Twid{(float)c, (float)(s / c)};
        bfly_c(x0, x1, e, o, t.a, t.b);
    } else {
        constexpr Twid t = UNIT ? unit_fr(s, c / s) : Twid{(float)s, (float)(c / s)};
        bfly_s(x0, x1, e, o, t.a, t.b);
    }
}

// ---- DFT ---------------------------------------------------------------------
// x[k] <- sum_n x[n] exp(-+2 pi i n k / N) (sign - forward, + when INV), unnormalised; UNIT as bfly_w.
template <int N, bool INV, bool UNIT = true, typename T>
__device__ __forceinline__ void dft(T *x);

template <int N, bool INV, bool UNIT, int K, typename T>
__device__ __forceinline__ void combine_one(T *x, const T *e, const T *o)
{
    if constexpr (K == 0) {
        x[K] = add(e[K], o[K]);
        x[K + N / 2] = sub(e[K], o[K]);
    } else if constexpr (4 * K == N) {
        bfly_i<INV>(x[K], x[K + N / 2], e[K], o[K]);
    } else {
        bfly_w<K, N, INV, UNIT>(x[K], x[K + N / 2], e[K], o[K]);
    }
}

template <int N, bool INV, bool UNIT, typename T, int... K>
__device__ __forceinline__ void combine_all(T *x, const T *e, const T *o, std::integer_sequence<int, K...>)
{
    (combine_one<N, INV, UNIT, K>(x, e, o), ...);
}

template <int N, bool INV, bool UNIT, typename T>
__device__ __forceinline__ void dft(T *x)
{
    if constexpr (N == 1) {
        return;
    } else if constexpr (N == 2) {
        const T a = x[0], b = x[1];
        x[0] = add(a, b);
        x[1] = sub(a, b);
    } else {
        T e[N / 2], o[N / 2];
#pragma unroll
        for (int k = 0; k < N / 2; ++k) {
            e[k] = x[2 * k];
            o[k] = x[2 * k + 1];
        }
        dft<N / 2, INV, UNIT>(e);
        dft<N / 2, INV, UNIT>(o);
        combine_all<N, INV, UNIT>(x, e, o, std::make_integer_sequence<int, N / 2>{});
    }
}

} // namespace fftreg
