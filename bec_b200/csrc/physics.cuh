// physics.cuh -- the per-cell real-space step of the FP32 path, shared by the
// plane-pass kernels.
//
// propagateXSpaceTwoComponent (programs/bec_wigner_3d.cuda/wigner_kernel.cu:184-229):
// itmax midpoint iterations of the exponential integrator
//   pa = -(l111 na^2 + l12 nb)/2 + i (V + g11 na + g12 nb)
//   pb = -(l22 nb + l12 na)/2  + i (V + g22 nb + g12 na - detuning)
//   d  = exp(p dt/2),  psi = psi0 d  (x itmax),  out = psi d
// (the reference's sign: evolution by e^{+i H dt}, wigner_kernel.cu:206-215),
// followed by the Wigner loss-noise increment at the start of the substep:
//   a += 3 sqrt(l111/6) conj(a0)^2 dW1 + sqrt(l12/2) conj(b0) dW2
//   b +=   sqrt(l12/2)  conj(a0)   dW2 + sqrt(l22)   conj(b0) dW3,
// dW complex normal with <|dW|^2> = dt / dV; the six normals of a cell and step
// come from one Philox4x32-10 draw keyed by the ensemble seed with counter
// (cell, step, trajectory, 1) (loss_normals6, common.cuh).
#pragma once

#include "common.cuh"
#include "engine.h"
#include "fft_reg.cuh"

// Per-thread constants of a trajectory's cell step, computed once per thread from its GroupParamsF:
// the nonlinear coefficients scaled by dt/2 and the squared loss-noise amplitudes.
struct CellConsts {
    float hdt;                      // dt / 2
    float hg11, hg12, hg22, hdet;   // g_ij dt/2, detuning dt/2
    float hl111, hl12, hl22;        // -l dt/4 (the drift -(l111 na^2 + l12 nb)/2 times dt/2)
    float n1, n2, n3;               // -2 ln 2 (noise_amp c_i)^2
    int itmax;
};

__device__ __forceinline__ CellConsts cell_consts(const GroupParamsF &P)
{
    CellConsts K;
    K.hdt = 0.5f * P.dt;
    K.hg11 = P.g11 * K.hdt;
    K.hg12 = P.g12 * K.hdt;
    K.hg22 = P.g22 * K.hdt;
    K.hdet = P.detuning * K.hdt;
    K.hl111 = -0.5f * K.hdt * P.l111;
    K.hl12 = -0.5f * K.hdt * P.l12;
    K.hl22 = -0.5f * K.hdt * P.l22;
    const float a1 = P.noise_amp * P.c1, a2 = P.noise_amp * P.c2, a3 = P.noise_amp * P.c3;
    K.n1 = -1.38629436112f * a1 * a1;
    K.n2 = -1.38629436112f * a2 * a2;
    K.n3 = -1.38629436112f * a3 * a3;
    K.itmax = P.itmax;
    return K;
}

// One Box-Muller pair of loss_normals6 scaled by an amplitude amp, with the SFU log2/sqrt/sin/cos:
// r = amp sqrt(-2 ln u1) = sqrt(n log2 u1) for n = -2 ln 2 amp^2, u1 = (f1 + 1/2) / 2^21 in (0, 1);
// (n1, n2) = r (cos, sin)(2 pi f2 / 2^21). log2 u1 < 0 for every u1 here: its largest value,
// log2(1 - 2^-22) = -3.4e-7, is twice the SFU log2's absolute error bound on [0.5, 2].
__device__ __forceinline__ float2 box_muller21_scaled(uint32_t f1, uint32_t f2, float n)
{
    const float y = n * __log2f(fmaf((float)f1, 0x1p-21f, 0x1p-22f));
    float r;
    asm("sqrt.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(y));
    float s, c;
    __sincosf((float)f2 * (6.28318530717958648f * 0x1p-21f), &s, &c);
    return make_float2(r * c, r * s);
}

// Phase and decay factors of the nonlinear substep. On the bench workloads |t| = |Im p| dt/2 stays below
// 0.38 and |Re p| dt/2 below 1e-6, so every cell takes the polynomial branch:
//   cos t, sin t: Taylor in u = t^2, Horner form, for |t| <= 0.5; sin to t^7 (truncation <= 0.5^9/9! = 5.4e-9),
//     cos to t^8 (<= 0.5^10/10! = 2.7e-10), both below half an FP32 ulp of the result;
//   exp x: Taylor to x^3 for |x| <= 1/64 (truncation <= (1/64)^4/4! = 2.5e-9).
// Arguments outside those ranges take sincosf / expf; one branch covers all four arguments of a cell.
// Both components of the cell at once, in packed pairs (fft_reg.cuh).
__device__ __forceinline__ void cis_taylor2(fftreg::f32x2 t, fftreg::f32x2 &c, fftreg::f32x2 &s)
{
    using namespace fftreg;
    const f32x2 u = mul2(t, t);
    s = fma2(mul2(t, u), fma2(u, fma2(u, both(-1.f / 5040.f), both(1.f / 120.f)), both(-1.f / 6.f)), t);
    c = fma2(u, fma2(u, fma2(u, fma2(u, both(1.f / 40320.f), both(-1.f / 720.f)), both(1.f / 24.f)), both(-0.5f)),
             both(1.f));
}

__device__ __forceinline__ fftreg::f32x2 exp_taylor2(fftreg::f32x2 x)
{
    using namespace fftreg;
    return fma2(x, fma2(x, fma2(x, both(1.f / 6.f), both(0.5f)), both(1.f)), both(1.f));
}

// The substep's factor pair (da, db) from the midpoint estimate x = (xa, xb): real parts, imaginary parts and
// negated imaginary parts. Every fused multiply-add is written out, so that every kernel that inlines the cell
// step rounds it the same way.
struct CellFactor {
    fftreg::f32x2 re, im, nim;
};
__device__ __forceinline__ CellFactor nonlinear_factors(const fftreg::cpair &x, float hV, float hVd, const CellConsts &K)
{
    using namespace fftreg;
    const f32x2 n = fma2(x.re, x.re, mul2(x.im, x.im));
    const float na = unpack2(n).x, nb = unpack2(n).y;
    const float ra = fmaf(K.hl111 * na, na, K.hl12 * nb);
    const float rb = fmaf(K.hl22, nb, K.hl12 * na);
    const float ta = fmaf(K.hg11, na, fmaf(K.hg12, nb, hV));
    const float tb = fmaf(K.hg22, nb, fmaf(K.hg12, na, hVd));
    f32x2 c, s, m;
    if (fmaxf(fabsf(ta), fabsf(tb)) <= 0.5f && fmaxf(fabsf(ra), fabsf(rb)) <= 0.015625f) {
        cis_taylor2(pack2(ta, tb), c, s);
        m = exp_taylor2(pack2(ra, rb));
    } else {
        float2 ea, eb;
        sincosf(ta, &ea.y, &ea.x);
        sincosf(tb, &eb.y, &eb.x);
        c = pack2(ea.x, eb.x);
        s = pack2(ea.y, eb.y);
        m = pack2(expf(ra), expf(rb));
    }
    return CellFactor{mul2(m, c), mul2(m, s), mul2(mul2(m, both(-1.f)), s)};
}

// One cell: v = (a, b) at the start of the substep, V the trap potential.
__device__ __forceinline__ fftreg::cpair nonlinear_cell(const fftreg::cpair &v, float V, const CellConsts &K)
{
    using namespace fftreg;
    const float hV = __fmul_rn(V, K.hdt), hVd = __fsub_rn(hV, K.hdet);   // never contracted
    CellFactor d;
    if (K.itmax == 1) {
        // one midpoint iteration (every workload here): the factors of the start values, applied twice
        d = nonlinear_factors(v, hV, hVd, K);
        return cmul2(cmul2(v, d.re, d.im, d.nim), d.re, d.im, d.nim);
    }
    cpair x = v;
    d = CellFactor{0, 0, 0};
    for (int it = 0; it < K.itmax; ++it) {
        d = nonlinear_factors(x, hV, hVd, K);
        x = cmul2(v, d.re, d.im, d.nim);
    }
    return cmul2(x, d.re, d.im, d.nim);
}

// The loss-noise increment of one cell from its Philox output, accumulated into out as FMA chains:
//   a += conj(a0)^2 w1 + conj(b0) w2,  b += conj(a0) w2 + conj(b0) w3.
__device__ __forceinline__ fftreg::cpair loss_noise_apply(const fftreg::cpair &o, const fftreg::cpair &v0,
                                                          const CellConsts &K, u32x4 w)
{
    uint32_t f[6];
    loss_fields(w, f);
    const float2 w1 = box_muller21_scaled(f[0], f[1], K.n1);
    const float2 w2 = box_muller21_scaled(f[2], f[3], K.n2);
    const float2 w3 = box_muller21_scaled(f[4], f[5], K.n3);
    const float2 a = fftreg::comp_a(v0), b = fftreg::comp_b(v0), oa = fftreg::comp_a(o), ob = fftreg::comp_b(o);
    const float ax = a.x, ay = a.y, bx = b.x, by = b.y;
    const float qx = fmaf(ax, ax, -ay * ay), qy = -2.f * ax * ay;       // conj(a0)^2
    return fftreg::make_cpair(
        make_float2(fmaf(qx, w1.x, fmaf(-qy, w1.y, fmaf(bx, w2.x, fmaf(by, w2.y, oa.x)))),
                    fmaf(qx, w1.y, fmaf(qy, w1.x, fmaf(bx, w2.y, fmaf(-by, w2.x, oa.y))))),
        make_float2(fmaf(ax, w2.x, fmaf(ay, w2.y, fmaf(bx, w3.x, fmaf(by, w3.y, ob.x)))),
                    fmaf(ax, w2.y, fmaf(-ay, w2.x, fmaf(bx, w3.y, fmaf(-by, w3.x, ob.y))))));
}

// Adds the loss-noise increments of two cells of the same trajectory and step, evaluated at v0 and v1, to
// out0 and out1: per cell the six normals of one Philox4x32-10 draw (loss_fields) as three complex Wiener
// increments already scaled by their amplitudes. The two draws' rounds interleave; keys: the round keys of
// the ensemble seed (philox_keys).
__device__ __forceinline__ void loss_noise_cell2(fftreg::cpair &out0, const fftreg::cpair &v0, fftreg::cpair &out1,
                                                 const fftreg::cpair &v1, const CellConsts &K,
                                                 const PhiloxKeys &keys, uint32_t traj, uint32_t step,
                                                 uint32_t cell0, uint32_t cell1)
{
    const u32x4x2 w = philox4x32_10_x2(cell0, step, traj, RNG_TAG_LOSS, cell1, step, traj, RNG_TAG_LOSS, keys);
    out0 = loss_noise_apply(out0, v0, K, w.a);
    out1 = loss_noise_apply(out1, v1, K, w.b);
}


// The loss-noise increments of four cells cell0 + d i, i < 4, of the same trajectory and step:
// one interleaved group of four Philox4x32-10 draws.
__device__ __forceinline__ void loss_noise_cell4(fftreg::cpair out[4], const fftreg::cpair v0[4], const CellConsts &K,
                                                 const PhiloxKeys &keys, uint32_t traj, uint32_t step, uint32_t cell0,
                                                 uint32_t d = 1u)
{
    const u32x4x4 w = philox4x32_10_x4(cell0, step, traj, RNG_TAG_LOSS, keys, d);
    out[0] = loss_noise_apply(out[0], v0[0], K, w.a);
    out[1] = loss_noise_apply(out[1], v0[1], K, w.b);
    out[2] = loss_noise_apply(out[2], v0[2], K, w.c);
    out[3] = loss_noise_apply(out[3], v0[3], K, w.d);
}
