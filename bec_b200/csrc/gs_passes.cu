// gs_passes.cu -- batched FP32 imaginary-time ground states.
//
// calculateSteadyState (programs/bec_wigner_3d.cuda/wigner.cu:84-175) for many
// ensembles at once: every step is K/2 -> FFT -> N(dt) -> IFFT -> K/2 ->
// renormalise to N (wigner_kernel.cu:128-134, :154-181), regrouped like the
// real-time path into a pencil pass (IFFT_z, kinetic factor, FFT_z) and a plane
// pass (FFT_xy, nonlinear factor, IFFT_xy) over single-component float2 states
// in the same stored representation (k-space along x and y, x-space along z).
//
// The norm after the second half-kick is measured in k-space by Parseval
// (N' = cells dV sum |psi_k|^2), accumulated per trajectory in FP64, and the
// factor sqrt(N / N') is applied by the next plane pass before the nonlinear
// step (scaling commutes with the linear kick and transforms). Norm buffers
// alternate between steps: the pencil pass of step n adds into buffer n % 2,
// the plane pass of step n + 1 reads it and clears the other one.
#include "engine.h"
#include "fft_reg.cuh"

namespace {

using fftreg::dft;

struct GsArgs {
    float frac1, frac2;       // kick fractions of dt_steady before / after the measurement
    float scale;              // 1/cells (makes the inverse z transform the normalised k-space state)
    float out_scale;          // nx*ny when the pass ends a step, else 1
};

// ---------------------------------------------------------------- pencil pass
// 2^LP pencils a trajectory. STEADY: the pass between two steps (two equal kicks, the norm); otherwise the fractions differ
// and norm and ekin may be null.
//
// On 256 states of 32x32x256 the pencil pass moves 1.01 GB in 229 us, 69 % of the measured HBM copy rate, and the plane pass as
// much in 260 us, 60 % (ncu, one launch each): what keeps them from the memory is the few warps that a line of 16 or 32
// complex values a thread leaves room for. So registers and instructions count: with the shared lines padded by one element instead
// of swizzled, and the grid's sizes known to the compiler, every shared and global access has an address and a constant
// offset. The nz = 256 pencil pass then fits four CTAs an SM at 64 registers without a spill (three at 80 with one before),
// the 32 x 32 plane pass five at 96 (four at 128). A step of 256 states of 32x32x256: 633 us before, 487 here; of 200 of
// 16x16x128: 67.2 and 50.5; of 16 of 32x32x256: 49.3 and 40.7. (Two warps a plane with 16 values a thread: 532 us.)
template <int NZ, int LP, bool STEADY>
__global__ void __launch_bounds__(NZ, 4 * 256 / NZ) k_gs_pencil(float2 *__restrict__ state, const GroupParamsF *__restrict__ gp,
                                                  const GsParamsF *__restrict__ gs, const int *__restrict__ tgroup,
                                                  const float2 *__restrict__ tw_g, GsArgs a,
                                                  double *__restrict__ norm, double *__restrict__ ekin,
                                                  const int *__restrict__ active)
{
    constexpr int R = 16, G = NZ / 16, LX = LP / 2, NX = 1 << LX, PLANE = 1 << LP, TILES = PLANE / 16;
    constexpr int LD = NZ + 1;                   // of a pencil in the buffer: its 16 first elements on different banks
    extern __shared__ float2 dyn2[];
    float2 *buf = dyn2;                          // 16 pencils
    float2 *tw = buf + 16 * LD;                  // W_NZ^e
    float *ez1 = reinterpret_cast<float *>(tw + NZ), *exy1 = ez1 + NZ;   // exp(-dt frac1 kz^2/2) per kz, per pencil x scale
    float *ez2 = exy1 + 16, *exy2 = ez2 + NZ;    // the same for frac2, x out_scale
    float *kz2 = exy2 + 16, *kxy2 = kz2 + NZ;    // kz^2/2 per kz, (kx^2 + ky^2)/2 per pencil
    __shared__ double red[2][NZ / 32];

    const int t = threadIdx.x;
    const int lt = blockIdx.x / TILES;                   // position in the launch's trajectory list
    const int traj = active ? active[lt] : lt;
    const int pen0 = (blockIdx.x - lt * TILES) * 16;
    const int gi = tgroup[traj];
    const float dts = gs[gi].dt_steady;
    {
        const GroupParamsF &P = gp[gi];
        tw[t] = tw_g[t];
        const float kz = getk<float>(t, P.dkz, NZ);
        const float kz2t = 0.5f * kz * kz;
        ez1[t] = expf(-dts * a.frac1 * kz2t);
        if (!STEADY) {
            kz2[t] = kz2t;
            ez2[t] = expf(-dts * a.frac2 * kz2t);
        }
        if (t < 16) {
            const int pen = pen0 + t;
            const float kx = getk<float>(pen & (NX - 1), P.dkx, NX);
            const float ky = getk<float>(pen >> LX, P.dky, NX);
            const float kxyt = 0.5f * (kx * kx + ky * ky);
            kxy2[t] = kxyt;
            exy1[t] = expf(-dts * a.frac1 * kxyt) * a.scale;
            exy2[t] = expf(-dts * a.frac2 * kxyt) * a.out_scale;
        }
    }

    const int p = t & 15, j = t >> 4;
    float2 *__restrict__ g = state + ((size_t)traj * (NZ * PLANE) + (size_t)(pen0 + p + j * PLANE));
    float2 x[R];
#pragma unroll
    for (int m = 0; m < R; ++m) x[m] = g[G * m * PLANE];
    __syncthreads();
    dft<R, true, false>(x);
#pragma unroll
    for (int k1 = 1; k1 < R; ++k1) {
        const float2 w = tw[j * k1];
        x[k1] = fftreg::cmulw(x[k1], make_float2(w.x, -w.y));
    }
    float2 *b1 = buf + p * LD + j * R;
#pragma unroll
    for (int k1 = 0; k1 < R; ++k1) b1[k1] = x[k1];
    __syncthreads();

    const int q = t % G, p2 = t / G;
    float2 *b2 = buf + p2 * LD + q;
    float2 y[R];
#pragma unroll
    for (int r = 0; r < R / G; ++r)
#pragma unroll
        for (int jj = 0; jj < G; ++jj) y[r * G + jj] = b2[jj * R + G * r];
#pragma unroll
    for (int r = 0; r < R / G; ++r) dft<G, true, false>(y + r * G);

    // propagateKSpaceImaginaryTime (wigner_kernel.cu:128-134): exp(-dt_steady frac k^2/2), real, as the
    // product of its (kx, ky) and kz factors
    double n_acc = 0.0, e_acc = 0.0;
    const float fxy1 = exy1[p2], fxy2 = exy2[p2];
#pragma unroll
    for (int r = 0; r < R / G; ++r)
#pragma unroll
        for (int k2 = 0; k2 < G; ++k2) {
            const int k = q + G * r + R * k2;
            float2 v = y[r * G + k2];
            const float z1 = ez1[k];
            const float e1 = fxy1 * z1;
            v = make_float2(v.x * e1, v.y * e1);
            if (STEADY || norm) {
                const double nk = (double)v.x * v.x + (double)v.y * v.y;
                n_acc += nk;
                if (!STEADY && ekin) e_acc += nk * (kxy2[p2] + kz2[k]);
            }
            const float e2 = fxy2 * (STEADY ? z1 : ez2[k]);
            y[r * G + k2] = make_float2(v.x * e2, v.y * e2);
        }
    if (STEADY || norm) {
        for (int off = 16; off > 0; off >>= 1) {
            n_acc += __shfl_down_sync(0xffffffffu, n_acc, off);
            if (!STEADY) e_acc += __shfl_down_sync(0xffffffffu, e_acc, off);
        }
        if ((t & 31) == 0) { red[0][t >> 5] = n_acc; red[1][t >> 5] = e_acc; }
    }

#pragma unroll
    for (int r = 0; r < R / G; ++r) dft<G, false, false>(y + r * G);
#pragma unroll
    for (int r = 0; r < R / G; ++r)
#pragma unroll
        for (int jj = 1; jj < G; ++jj) y[r * G + jj] = fftreg::cmulw(y[r * G + jj], tw[(q + G * r) * jj]);
    __syncthreads();
    if ((STEADY || norm) && t == 0) {
        double sn = 0.0, se = 0.0;
        for (int w = 0; w < NZ / 32; ++w) { sn += red[0][w]; se += red[1][w]; }
        atomicAdd(norm + traj, sn);
        if (!STEADY && ekin) atomicAdd(ekin + traj, se);
    }
#pragma unroll
    for (int r = 0; r < R / G; ++r)
#pragma unroll
        for (int jj = 0; jj < G; ++jj) b2[jj * R + G * r] = y[r * G + jj];
    __syncthreads();
#pragma unroll
    for (int k1 = 0; k1 < R; ++k1) x[k1] = b1[k1];
    dft<R, false, false>(x);
#pragma unroll
    for (int m = 0; m < R; ++m) g[G * m * PLANE] = x[m];
}

// ---------------------------------------------------------------- plane passes
// propagateXSpaceOneComponent (wigner_kernel.cu:154-181) of a renormalised cell; one midpoint iteration, every workload
// here, runs without its loop
__device__ __forceinline__ float2 nonlinear_gs(float2 a0, float V, float g11, float hdt, int itmax)
{
    float2 xa = a0;
    float da = 0.0f;
    if (itmax == 1) {
        da = expf(hdt * fmaf(-g11, fmaf(a0.x, a0.x, a0.y * a0.y), -V));
        xa = make_float2(a0.x * da, a0.y * da);
    } else {
        for (int it = 0; it < itmax; ++it) {
            da = expf(hdt * fmaf(-g11, fmaf(xa.x, xa.x, xa.y * xa.y), -V));
            xa = make_float2(a0.x * da, a0.y * da);
        }
    }
    return make_float2(xa.x * da, xa.y * da);
}

// MODE 0: step (FFT_xy -> renormalise -> nonlinear -> IFFT_xy)
// MODE 1: prep (x-space natural in -> IFFT_xy)
// MODE 2: measure / output (FFT_xy, renormalise, write x-space rows to out, x-space sums)
template <int N, int MODE>
__global__ void __launch_bounds__(128, N == 32 && MODE == 0 ? 5 : 4) k_gs_plane(float2 *__restrict__ state, int nz, int cells,
                                                  const GroupParamsF *__restrict__ gp,
                                                  const GsParamsF *__restrict__ gs, const int *__restrict__ tgroup,
                                                  const double *__restrict__ norm_in, double *__restrict__ norm_clear,
                                                  float2 *__restrict__ out, double *__restrict__ xsums, float in_scale,
                                                  const int *__restrict__ active)
{
    constexpr int W = 32 / N;
    constexpr int PLANE = N * N, LD = N + 1;
    extern __shared__ float2 tile2[];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int wp = lane / N, c = lane % N;
    const int plane_id = (blockIdx.x * 4 + warp) * W + wp;
    const int lt = plane_id / nz, z = plane_id - lt * nz;
    const int traj = active ? active[lt] : lt;
    float2 *__restrict__ g = state + (size_t)traj * cells + (size_t)z * PLANE;
    float2 *s = tile2 + (warp * W + wp) * (N * LD);
    const int gi = tgroup[traj];
    const GroupParamsF P = gp[gi];
    const GsParamsF Q = gs[gi];

    float scale = in_scale;
    if (norm_in) scale *= sqrtf((float)(Q.N / (norm_in[traj] * Q.parseval)));
    if (norm_clear && z == 0 && c == 0) norm_clear[traj] = 0.0;

    float2 v[N];
#pragma unroll
    for (int y = 0; y < N; ++y) v[y] = (MODE == 1) ? g[c * N + y] : g[y * N + c];   // prep starts from rows
    const int p_begin = (MODE == 1) ? 2 : 0;
    const int p_end = (MODE == 2) ? 2 : 4;
#pragma unroll 1
    for (int pass = p_begin; pass < p_end; ++pass) {
        if (pass >= 2) dft<N, true, false>(v);
        else dft<N, false, false>(v);
        if (pass == 0) {
#pragma unroll
            for (int y = 0; y < N; ++y) s[y * LD + c] = v[y];
            __syncwarp();
#pragma unroll
            for (int x = 0; x < N; ++x) v[x] = s[c * LD + x];
        } else if (pass == 1 && MODE == 0) {
#pragma unroll
            for (int x = 0; x < N; ++x) s[c * LD + x] = v[x];
            // coordinates and potential with the fused multiply-adds written out; four cells per iteration, their
            // exponentials independent
            const float Y = fmaf(P.dy, (float)c, -P.ymax);
            const float Z = fmaf(P.dz, (float)z, -P.zmax);
            const float base = fmaf(Y, Y, (Z * Z) * P.inv_lambda2);
            const float hdt = 0.5f * Q.dt_steady;
#pragma unroll 1
            for (int x = 0; x < N; x += 4) {
                float2 o[4];
#pragma unroll
                for (int k = 0; k < 4; ++k) {
                    const float X = fmaf(P.dx, (float)(x + k), -P.xmax);
                    const float V = 0.5f * fmaf(X, X, base);
                    const float2 w = s[c * LD + x + k];
                    o[k] = nonlinear_gs(make_float2(w.x * scale, w.y * scale), V, P.g11, hdt, P.itmax);
                }
#pragma unroll
                for (int k = 0; k < 4; ++k) s[c * LD + x + k] = o[k];
            }
#pragma unroll
            for (int x = 0; x < N; ++x) v[x] = s[c * LD + x];
        } else if (pass == 2) {
#pragma unroll
            for (int x = 0; x < N; ++x) s[c * LD + x] = v[x];
            __syncwarp();
#pragma unroll
            for (int y = 0; y < N; ++y) v[y] = s[y * LD + c];
        }
    }
    if (MODE == 2) {
        // lane c holds row y = c of the x-space state
        const float Y = -P.ymax + P.dy * (float)c;
        const float Z = -P.zmax + P.dz * (float)z;
        const float base = Y * Y + Z * Z * P.inv_lambda2;
        // sums: n V, n^2, n and |u - previous output|^2 (the state's change since the last output)
        double sv = 0.0, s2 = 0.0, s1 = 0.0, sd = 0.0;
        float2 *o = out + (size_t)traj * cells + (size_t)z * PLANE + c * N;
#pragma unroll
        for (int x = 0; x < N; ++x) {
            const float2 u = make_float2(v[x].x * scale, v[x].y * scale);
            const float2 w = o[x];
            o[x] = u;
            const float X = -P.xmax + P.dx * (float)x;
            const double n = (double)u.x * u.x + (double)u.y * u.y;
            const float ex = u.x - w.x, ey = u.y - w.y;
            sv += n * (double)(0.5f * (X * X + base));
            s2 += n * n;
            s1 += n;
            sd += (double)(ex * ex + ey * ey);
        }
        if (xsums) {
            for (int off = N / 2; off > 0; off >>= 1) {
                sv += __shfl_down_sync(0xffffffffu, sv, off, N);
                s2 += __shfl_down_sync(0xffffffffu, s2, off, N);
                s1 += __shfl_down_sync(0xffffffffu, s1, off, N);
                sd += __shfl_down_sync(0xffffffffu, sd, off, N);
            }
            if (c == 0) {
                atomicAdd(xsums + 4 * traj + 0, sv);
                atomicAdd(xsums + 4 * traj + 1, s2);
                atomicAdd(xsums + 4 * traj + 2, s1);
                atomicAdd(xsums + 4 * traj + 3, sd);
            }
        }
    } else {
#pragma unroll
        for (int y = 0; y < N; ++y) g[y * N + c] = v[y];
    }
}

// x-space Thomas-Fermi start (fillWithTFGroundState, wigner_kernel.cu:116-125) or a copy of a warm start
__global__ void k_gs_init(float2 *state, int nx, int lx, int ny, int ly, int cells, int n_traj,
                          const GroupParamsF *gp, const GsParamsF *gs, const int *tgroup, const float2 *warm)
{
    const size_t n = (size_t)cells * n_traj;
    for (size_t idx = blockIdx.x * (size_t)blockDim.x + threadIdx.x; idx < n; idx += (size_t)gridDim.x * blockDim.x) {
        const int t = (int)(idx / cells), i = (int)(idx - (size_t)t * cells);
        if (warm) { state[idx] = warm[idx]; continue; }
        const int gi = tgroup[t];
        const GroupParamsF P = gp[gi];
        const int x = i & (nx - 1), y = (i >> lx) & (ny - 1), z = i >> (lx + ly);
        const float X = -P.xmax + P.dx * (float)x;
        const float Y = (ny > 1) ? -P.ymax + P.dy * (float)y : 0.0f;
        const float Z = -P.zmax + P.dz * (float)z;
        const float e = gs[gi].mu - 0.5f * (X * X + Y * Y + Z * Z * P.inv_lambda2);
        state[idx] = make_float2(e > 0.0f ? sqrtf(e / P.g11) : 0.0f, 0.0f);
    }
}

template <int N, int MODE>
void launch_gs_plane(float2 *state, const ClassGeom &c, const GroupParamsF *gp, const GsParamsF *gs,
                     const int *tgroup, const double *norm_in, double *norm_clear, float2 *out, double *xsums,
                     float in_scale, const int *active, cudaStream_t s)
{
    constexpr int W = 32 / N;
    const size_t smem = sizeof(float2) * 4 * W * N * (N + 1);
    ensure_smem_limit((const void *)k_gs_plane<N, MODE>, (int)smem);
    k_gs_plane<N, MODE><<<c.n_traj * c.nz / (4 * W), 128, smem, s>>>(state, c.nz, c.cells, gp, gs, tgroup, norm_in,
                                                                      norm_clear, out, xsums, in_scale, active);
    g_launches++;
}

template <int NZ, int LP>
void launch_gs_pencil(float2 *state, const ClassGeom &c, const GroupParamsF *gp, const GsParamsF *gs,
                      const int *tgroup, const float2 *tw, const GsArgs &a, double *norm, double *ekin,
                      const int *active, cudaStream_t s)
{
    const bool steady = a.frac1 == a.frac2 && norm && !ekin;
    const size_t smem = sizeof(float2) * (16 * (NZ + 1) + NZ) + sizeof(float) * (3 * NZ + 3 * 16);
    auto kernel = steady ? k_gs_pencil<NZ, LP, true> : k_gs_pencil<NZ, LP, false>;
    ensure_smem_limit((const void *)kernel, (int)smem);
    kernel<<<c.n_traj << (LP - 4), NZ, smem, s>>>(state, gp, gs, tgroup, tw, a, norm, ekin, active);
    g_launches++;
}
template <int NZ>
void dispatch_pencil(float2 *state, const ClassGeom &c, const GroupParamsF *gp, const GsParamsF *gs, const int *tgroup,
                     const float2 *tw, const GsArgs &a, double *norm, double *ekin, const int *active, cudaStream_t s)
{
    switch (c.nx) {
    case 8: launch_gs_pencil<NZ, 6>(state, c, gp, gs, tgroup, tw, a, norm, ekin, active, s); break;
    case 16: launch_gs_pencil<NZ, 8>(state, c, gp, gs, tgroup, tw, a, norm, ekin, active, s); break;
    case 32: launch_gs_pencil<NZ, 10>(state, c, gp, gs, tgroup, tw, a, norm, ekin, active, s); break;
    default: break;
    }
}

template <int MODE>
void dispatch_plane(float2 *state, const ClassGeom &c, const GroupParamsF *gp, const GsParamsF *gs, const int *tgroup,
                    const double *norm_in, double *norm_clear, float2 *out, double *xsums, float in_scale,
                    const int *active, cudaStream_t s)
{
    switch (c.nx) {
    case 8: launch_gs_plane<8, MODE>(state, c, gp, gs, tgroup, norm_in, norm_clear, out, xsums, in_scale, active, s); break;
    case 16: launch_gs_plane<16, MODE>(state, c, gp, gs, tgroup, norm_in, norm_clear, out, xsums, in_scale, active, s); break;
    case 32: launch_gs_plane<32, MODE>(state, c, gp, gs, tgroup, norm_in, norm_clear, out, xsums, in_scale, active, s); break;
    default: break;
    }
}

} // namespace

bool gs_batched_supported(const ClassGeom &c)
{
    return fp32_fast_plane_supported(c) && fp32_fast_pencil_supported(c);
}

void gs_init(float2 *state, const ClassGeom &c, const GroupParamsF *gp, const GsParamsF *gs, const int *tgroup,
             const float2 *warm, cudaStream_t s)
{
    size_t n = (size_t)c.cells * c.n_traj;
    int blocks = (int)((n + 255) / 256);
    if (blocks > 148 * 32) blocks = 148 * 32;
    k_gs_init<<<blocks, 256, 0, s>>>(state, c.nx, c.lx, c.ny, c.ly, c.cells, c.n_traj, gp, gs, tgroup, warm);
    g_launches++;
}

void gs_prep(float2 *state, const ClassGeom &c, const GroupParamsF *gp, const GsParamsF *gs, const int *tgroup,
             cudaStream_t s)
{
    dispatch_plane<1>(state, c, gp, gs, tgroup, nullptr, nullptr, nullptr, nullptr, 1.0f, nullptr, s);
}

void gs_plane_step(float2 *state, const ClassGeom &c, const GroupParamsF *gp, const GsParamsF *gs, const int *tgroup,
                   const double *norm_in, double *norm_clear, cudaStream_t s, const int *active)
{
    dispatch_plane<0>(state, c, gp, gs, tgroup, norm_in, norm_clear, nullptr, nullptr, 1.0f, active, s);
}

void gs_output(float2 *state, const ClassGeom &c, const GroupParamsF *gp, const GsParamsF *gs, const int *tgroup,
               const double *norm_in, float2 *out, double *xsums, float in_scale, cudaStream_t s, const int *active)
{
    dispatch_plane<2>(state, c, gp, gs, tgroup, norm_in, nullptr, out, xsums, in_scale, active, s);
}

void gs_pencil(float2 *state, const ClassGeom &c, const GroupParamsF *gp, const GsParamsF *gs, const int *tgroup,
               const float2 *tw_full, float frac1, float frac2, float scale, float out_scale, double *norm,
               double *ekin, cudaStream_t s, const int *active)
{
    GsArgs a{frac1, frac2, scale, out_scale};
    switch (c.nz) {
    case 64: dispatch_pencil<64>(state, c, gp, gs, tgroup, tw_full, a, norm, ekin, active, s); break;
    case 128: dispatch_pencil<128>(state, c, gp, gs, tgroup, tw_full, a, norm, ekin, active, s); break;
    case 256: dispatch_pencil<256>(state, c, gp, gs, tgroup, tw_full, a, norm, ekin, active, s); break;
    default: break;
    }
}
