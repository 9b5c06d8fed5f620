// fp64_passes.cu -- FP64 imaginary-time steps of single-component states and real-time steps of both components, each in
// two fused passes, and the FP64 measures of ground states.
//
// Imaginary time:
// calculateSteadyState (programs/bec_wigner_3d.cuda/wigner.cu:84-175) takes a kick, three transform axes, the
// nonlinear factor, three axes, a scaling, a kick, three axes and a renormalisation per step, each a kernel of its
// own. Here a step is a pencil pass (IFFT_z -> 1/cells -> half kick -> norm -> half kick of the next step -> FFT_z)
// and a plane pass (FFT_xy -> renormalise -> nonlinear factor -> IFFT_xy) over a state kept as k-space along x and
// y, x-space along z, as in the FP32 passes. The norm after the second half kick is taken in k-space (Parseval):
// every pencil CTA writes its partial sum, and the next plane pass adds them in a fixed order, so a step is
// deterministic and holds no synchronisation with the host.
//
// What bounds it: latency. A 16x16x128 state is 512 KiB; at HBM rate the two passes would take 0.3 us. A pass is a
// launch, one trip to L2 and back, and two to three radix-8 stages per axis in shared memory. Tiles are therefore
// small (a plane, or two to eight pencils), so that one trajectory fills the chip. Measured on one 16x16x128 ground
// state of 500 steps: 83.4 ms with one kernel per operation (30 launches a step), 5.1 ms here (8.43 ms before the
// twiddles and kick factors lay in shared memory at the pass's start and a launch overlapped the end of the one before). The measures of a
// batch (mu, energy, norm, residual) took twenty launches and two synchronisations a state; here they take eight
// launches for half the batch (96 states of 32x32x256 with 60 steps: the whole call 42.6 -> 23.2 ms).
//
// Real time (wigner.cu:178-199): the passes of k64_evo_plane and k64_evo_pencil below, over every trajectory of an ensemble.
#include <algorithm>
#include <climits>

#include "engine.h"
#include "launch.cuh"
#include "reduce.cuh"

namespace {

// ---------------------------------------------------------------- radix-8 transforms in shared memory
__device__ __forceinline__ double2 mul_i(double2 v, bool inv) { return inv ? make_double2(-v.y, v.x) : make_double2(v.y, -v.x); }

template <bool INV>
__device__ __forceinline__ void dft2(double2 &a, double2 &b)
{
    const double2 t = a;
    a = cadd(t, b);
    b = csub(t, b);
}
template <bool INV>
__device__ __forceinline__ void dft4(double2 &a, double2 &b, double2 &c, double2 &d)
{
    dft2<INV>(a, c);
    dft2<INV>(b, d);
    d = mul_i(d, INV);
    dft2<INV>(a, b);
    dft2<INV>(c, d);
    const double2 t = b;      // natural order: a, c, b, d -> X0 X1 X2 X3
    b = c;
    c = t;
}
// v / sqrt(2), rounded once. The double nearest to 1 / sqrt(2) is 4.8e-17 larger, which every radix-8 stage would put into a
// quarter of its values: the population then grows by 1.3e-16 to 2.6e-16 a step (six transforms) on every grid, against a
// few 1e-17 so or with radix-2 stages.
__device__ __forceinline__ double over_root2(double v) { return fma(0x1.6a09e667f3bcdp-1, v, -0x1.bdd3413b26456p-55 * v); }
// x[k] <- sum_n x[n] e^{-+2 pi i n k / R}, R = 2, 4, 8
template <int R, bool INV>
__device__ __forceinline__ void dft_small(double2 *x)
{
    if constexpr (R == 2) {
        dft2<INV>(x[0], x[1]);
    } else if constexpr (R == 4) {
        dft4<INV>(x[0], x[1], x[2], x[3]);
    } else {
        dft4<INV>(x[0], x[2], x[4], x[6]);      // even samples -> E0..E3 in x[0], x[2], x[4], x[6]
        dft4<INV>(x[1], x[3], x[5], x[7]);
        const double2 o0 = x[1], o1 = x[3], o2 = x[5], o3 = x[7];
        const double2 i1 = mul_i(o1, INV), i3 = mul_i(o3, INV);
        const double2 t1 = make_double2(over_root2(o1.x + i1.x), over_root2(o1.y + i1.y));       // W o1
        const double2 t2 = mul_i(o2, INV);                                                       // W^2 o2
        const double2 t3 = make_double2(over_root2(i3.x - o3.x), over_root2(i3.y - o3.y));       // W^3 o3
        const double2 e0 = x[0], e1 = x[2], e2 = x[4], e3 = x[6];
        x[0] = cadd(e0, o0); x[4] = csub(e0, o0);
        x[1] = cadd(e1, t1); x[5] = csub(e1, t1);
        x[2] = cadd(e2, t2); x[6] = csub(e2, t2);
        x[3] = cadd(e3, t3); x[7] = csub(e3, t3);
    }
}

// Lines of n = 2^logn elements at base(line) + e * es: base = (line & (2^lin - 1)) * ls_in + (line >> lin) * ls_out.
struct Lines {
    int logn, log_lines, es, lin, ls_in, ls_out;
    __device__ __forceinline__ int base(int line) const { return (line & ((1 << lin) - 1)) * ls_in + (line >> lin) * ls_out; }
};

// One stage of span m = 2^lm and radix R over every line. Decimation in time (DIF = false): twiddles before the
// small transform; in frequency: after it.
template <int R, bool INV, bool DIF>
__device__ __forceinline__ void stage(double2 *buf, const Lines &L, const double2 *tw, int lm)
{
    constexpr int LR = R == 8 ? 3 : R == 4 ? 2 : 1;
    const int total = 1 << (L.log_lines + L.logn - LR);
    const int shift = L.logn - LR - lm;
    for (int w = threadIdx.x; w < total; w += blockDim.x) {
        const int line = w & ((1 << L.log_lines) - 1), jj = w >> L.log_lines;
        const int j = jj & ((1 << lm) - 1);
        double2 *p = buf + L.base(line) + (((jj >> lm) << (lm + LR)) + j) * L.es;
        const int step = L.es << lm;
        double2 x[R];
#pragma unroll
        for (int r = 0; r < R; ++r) x[r] = p[r * step];
        if constexpr (DIF) dft_small<R, INV>(x);
        if (lm > 0) {
#pragma unroll
            for (int r = 1; r < R; ++r) {
                double2 t = tw[(j * r) << shift];
                if (INV) t.y = -t.y;
                x[r] = cmul(x[r], t);
            }
        }
        if constexpr (!DIF) dft_small<R, INV>(x);
#pragma unroll
        for (int r = 0; r < R; ++r) p[r * step] = x[r];
    }
    __syncthreads();
}

// Position of element k of a line in the digit-reversed order that the transforms start from (in time) or end in
// (in frequency): radix 8 as often as logn allows, a last radix of 2 or 4.
__device__ __forceinline__ int digit_rev(int k, int logn)
{
    int p = 0, s = logn;
    while (s >= 3) {
        s -= 3;
        p |= (k & 7) << s;
        k >>= 3;
    }
    return p | k;
}

// digit-reversed -> natural, every line of the tile
template <bool INV>
__device__ __forceinline__ void fft_time(double2 *buf, const Lines &L, const double2 *tw)
{
    int lm = 0;
    if (L.logn % 3 == 1) { stage<2, INV, false>(buf, L, tw, 0); lm = 1; }
    else if (L.logn % 3 == 2) { stage<4, INV, false>(buf, L, tw, 0); lm = 2; }
    for (; lm < L.logn; lm += 3) stage<8, INV, false>(buf, L, tw, lm);
}
// natural -> digit-reversed
template <bool INV>
__device__ __forceinline__ void fft_freq(double2 *buf, const Lines &L, const double2 *tw)
{
    int lm = L.logn - 3;
    for (; lm >= 0; lm -= 3) stage<8, INV, true>(buf, L, tw, lm);
    if (lm == -2) stage<2, INV, true>(buf, L, tw, 0);
    else if (lm == -1) stage<4, INV, true>(buf, L, tw, 0);
}

__device__ __forceinline__ void copy16(double2 *dst_smem, const double2 *src)
{
    const unsigned d = (unsigned)__cvta_generic_to_shared(dst_smem);
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(d), "l"(src) : "memory");
}
__device__ __forceinline__ void copy_wait() { asm volatile("cp.async.wait_all;" ::: "memory"); }

// Sum of K values over the block in a fixed order, valid in every thread; red holds K * 32 + K doubles.
template <int K>
__device__ __forceinline__ void block_sum(double (&v)[K], double *red)
{
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
#pragma unroll
    for (int k = 0; k < K; ++k)
#pragma unroll
        for (int off = 16; off > 0; off >>= 1) v[k] += __shfl_xor_sync(0xffffffffu, v[k], off);
    if (lane == 0)
#pragma unroll
        for (int k = 0; k < K; ++k) red[k * 32 + warp] = v[k];
    __syncthreads();
#pragma unroll
    for (int k = 0; k < K; ++k) {
        double s = 0.0;
        for (int w = 0; w < nw; ++w) s += red[k * 32 + w];
        v[k] = s;
    }
    __syncthreads();
}

__device__ __forceinline__ double2 load_psi(const double2 *p, size_t i) { return p[i]; }
__device__ __forceinline__ double2 load_psi(const float2 *p, size_t i) { return make_double2(p[i].x, p[i].y); }

// ---------------------------------------------------------------- plane pass
// A CTA holds ppc planes (nx x ny, rows padded by one element against bank conflicts).
//   START    x-space in (src, or the Thomas-Fermi profile when src is null) -> IFFT_xy -> state
//   MEASURE  START with the sums n V, n^2, n of src per CTA
//   STEP     state -> FFT_xy -> renormalise -> nonlinear factor -> IFFT_xy -> state
//   OUT      state -> FFT_xy -> renormalise -> out (x-space); sums n V, n^2, n, |u - previous out|^2 and the
//            reference's energy integrand (wigner_kernel.cu:232-258) when the k-space state kout is given
//   RESIDUAL state (k^2/2 psi_k along z) -> FFT_xy = kinetic part; sum |(H - mu) psi|^2 of src
enum { START, MEASURE, STEP, OUT, RESIDUAL };

template <int MODE, typename S>
__global__ void __launch_bounds__(256) k64_plane(double2 *__restrict__ state, const Gs64Par *__restrict__ par, int lx, int ly,
                                                 int lz, int lppc, const double2 *__restrict__ tx,
                                                 const double2 *__restrict__ ty, const double *norm_part, int norm_tiles,
                                                 const S *src, double2 *out, const double2 *kout, const double *sums4,
                                                 double *part)
{
    // (what the kernel before this one writes is not declared __restrict__: such loads might move above the wait)
    extern __shared__ double2 sm64[];
    __shared__ double red[5 * 32];
    const int nx = 1 << lx, ny = 1 << ly, ld = nx + 1, lplane = lx + ly;
    const int lchunk = lppc + lplane, chunk = 1 << lchunk;
    const int chunks = 1 << (lz - lppc);                        // per trajectory
    const int traj = blockIdx.x >> (lz - lppc), c0 = blockIdx.x & (chunks - 1);
    const size_t cell0 = (size_t)c0 << lchunk;
    const size_t first = ((size_t)traj << (lplane + lz)) + cell0;
    auto natural = [&](int i) { return (i >> lx) * ld + (i & (nx - 1)); };
    auto reversed = [&](int i) {
        return ((i >> lplane) * ny + digit_rev((i >> lx) & (ny - 1), ly)) * ld + digit_rev(i & (nx - 1), lx);
    };
    const Lines rows{lx, lppc + ly, 1, 30, ld, 0}, cols{ly, lppc + lx, ld, lx, 1, ny * ld};
    // the twiddles beside the tile: read from L2 stage by stage they would add a trip to every barrier
    double2 *twx = sm64 + ((ny << lppc) * ld), *twy = twx + nx;
    for (int i = threadIdx.x; i < nx; i += blockDim.x) copy16(twx + i, tx + i);
    for (int i = threadIdx.x; i < ny; i += blockDim.x) copy16(twy + i, ty + i);

    wait_predecessor();
    allow_successor();
    if (MODE == STEP || MODE == OUT || MODE == RESIDUAL)
        for (int i = threadIdx.x; i < chunk; i += blockDim.x) copy16(sm64 + reversed(i), state + first + i);
    const Gs64Par &Q = par[traj];
    const GeomD &g = Q.g;
    double scale = 1.0;
    if (MODE == STEP || MODE == OUT) {
        double s[1] = {0.0};
        for (int t = threadIdx.x; t < norm_tiles; t += blockDim.x) s[0] += norm_part[((size_t)traj * norm_tiles + t) * 2];
        block_sum<1>(s, red);
        scale = sqrt(Q.N / (s[0] * ((double)g.cells * g.dV)));
    }
    auto potential = [&](int i) {
        const double X = -g.xmax + g.dx * (double)(i & (nx - 1));
        const double Y = ny > 1 ? -g.ymax + g.dy * (double)((i >> lx) & (ny - 1)) : 0.0;
        const double Z = -g.zmax + g.dz * (double)((c0 << lppc) + (i >> lplane));
        return (X * X + Y * Y + Z * Z / (g.lambda * g.lambda)) / 2.0;
    };
    if (MODE == STEP || MODE == OUT || MODE == RESIDUAL) {
        copy_wait();
        __syncthreads();
        fft_time<false>(sm64, rows, twx);
        if (ly > 0) fft_time<false>(sm64, cols, twy);
    }
    double v[5] = {0.0, 0.0, 0.0, 0.0, 0.0};
    for (int i = threadIdx.x; i < chunk; i += blockDim.x) {
        double2 &w = sm64[natural(i)];
        if (MODE == START || MODE == MEASURE) {
            double2 u;
            if (src) {
                u = load_psi(src, first + i);
            } else {
                const double e = Q.mu - potential(i);
                u = make_double2(e > 0 ? sqrt(e / g.g11) : 0.0, 0.0);
            }
            w = u;
            if (MODE == MEASURE) {
                const double n = u.x * u.x + u.y * u.y;
                v[0] += n * potential(i);
                v[1] += n * n;
                v[2] += n;
            }
        } else if (MODE == STEP) {
            // propagateXSpaceOneComponent (wigner_kernel.cu:154-181)
            const double V = potential(i);
            const double2 a0 = cscale(w, scale);
            double2 x = a0;
            double d = 0.0;
            for (int it = 0; it < g.itmax; ++it) {
                d = exp(g.dt_steady / 2.0 * (-V - g.g11 * (x.x * x.x + x.y * x.y)));
                x = cscale(a0, d);
            }
            w = cscale(x, d);
        } else if (MODE == OUT) {
            const double2 u = cscale(w, scale), p = out[first + i];
            out[first + i] = u;
            const double V = potential(i), n = u.x * u.x + u.y * u.y;
            v[0] += n * V;
            v[1] += n * n;
            v[2] += n;
            const double dx = u.x - p.x, dy = u.y - p.y;
            v[3] += dx * dx + dy * dy;
            if (kout) {
                const int x = i & (nx - 1), y = (i >> lx) & (ny - 1), z = (c0 << lppc) + (i >> lplane);
                const double kx = getk<double>(x, g.dkx, nx), ky = ny > 1 ? getk<double>(y, g.dky, ny) : 0.0;
                const double kz = getk<double>(z, g.dkz, 1 << lz);
                const double2 ak = cscale(kout[first + i], scale * ((kx * kx + ky * ky + kz * kz) / 2.0));
                v[4] += n * (V + g.g11 * n / 2.0) + (u.x * ak.x - u.y * ak.y);
            }
        } else {
            const double2 u = load_psi(src, first + i);
            const double *m = sums4 + 4 * (size_t)traj;            // n V, n^2, n, kinetic
            const double mu = (m[3] * g.cells + m[0] + g.g11 * m[1]) / m[2];
            const double f = potential(i) + g.g11 * (u.x * u.x + u.y * u.y) - mu;
            const double hx = w.x + u.x * f, hy = w.y + u.y * f;
            v[0] += hx * hx + hy * hy;
        }
    }
    if (MODE == START || MODE == MEASURE || MODE == STEP) {
        copy_wait();
        __syncthreads();
        if (ly > 0) fft_freq<true>(sm64, cols, twy);
        fft_freq<true>(sm64, rows, twx);
        for (int i = threadIdx.x; i < chunk; i += blockDim.x) state[first + i] = sm64[reversed(i)];
    }
    if (MODE == MEASURE || MODE == OUT || MODE == RESIDUAL) {
        constexpr int K = MODE == MEASURE ? 3 : MODE == OUT ? 5 : 1;
        double s[K];
#pragma unroll
        for (int k = 0; k < K; ++k) s[k] = v[k];
        block_sum<K>(s, red);
        if (threadIdx.x == 0)
#pragma unroll
            for (int k = 0; k < K; ++k) part[(size_t)blockIdx.x * K + k] = s[k];
    }
}

// ---------------------------------------------------------------- pencil pass
// A CTA holds 2^lp adjacent pencils of a trajectory, laid out [z][pencil]: IFFT_z -> scale -> [half kick] -> [sums
// |psi_k|^2 and |psi_k|^2 k^2/2 per CTA] -> [psi_k to kout] -> [half kick, or k^2/2] -> FFT_z.
enum { KICK1 = 1, SUMS = 2, KICK2 = 4, TIMES_K2 = 8 };

__global__ void __launch_bounds__(256) k64_pencil(double2 *__restrict__ state, const Gs64Par *__restrict__ par, int lx, int ly,
                                                  int lz, int lp, const double2 *__restrict__ tz,
                                                  const double *__restrict__ kick, double scale, int what,
                                                  double *__restrict__ part, double2 *__restrict__ kout)
{
    extern __shared__ double2 sm64[];
    __shared__ double red[2 * 32];
    __shared__ double exy[8], kxy[8];
    const int nx = 1 << lx, nz = 1 << lz, lplane = lx + ly, P = 1 << lp, chunk = nz << lp;
    double2 *tw = sm64 + chunk;
    double *ez = reinterpret_cast<double *>(tw + nz);          // half-kick factors per kz, then kz^2/2
    double *kz2 = ez + nz;
    const int traj = blockIdx.x >> (lplane - lp), pen0 = (blockIdx.x & ((1 << (lplane - lp)) - 1)) << lp;
    double2 *g0 = state + ((size_t)traj << (lplane + lz)) + pen0;
    const Gs64Par &Q = par[traj];
    const GeomD &g = Q.g;
    for (int i = threadIdx.x; i < nz + P; i += blockDim.x) {
        double k2;
        if (i < nz) {
            const double kz = getk<double>(i, g.dkz, nz);
            k2 = kz * kz / 2.0;
        } else {
            const int pen = pen0 + i - nz;
            const double kx = getk<double>(pen & (nx - 1), g.dkx, nx);
            const double ky = ly > 0 ? getk<double>(pen >> lx, g.dky, 1 << ly) : 0.0;
            k2 = (kx * kx + ky * ky) / 2.0;
        }
        // the half-kick factors come from k64_kick's table
        const double e = (what & (KICK1 | KICK2)) ? kick[i < nz ? i : i + pen0] : 1.0;
        if (i < nz) { ez[i] = e; kz2[i] = k2; }
        else { exy[i - nz] = e; kxy[i - nz] = k2; }
    }
    for (int i = threadIdx.x; i < nz; i += blockDim.x) copy16(tw + i, tz + i);
    wait_predecessor();
    allow_successor();
    for (int i = threadIdx.x; i < chunk; i += blockDim.x)
        copy16(sm64 + (digit_rev(i >> lp, lz) << lp) + (i & (P - 1)), g0 + ((size_t)(i >> lp) << lplane) + (i & (P - 1)));
    copy_wait();
    __syncthreads();
    const Lines L{lz, lp, P, 30, 1, 0};
    fft_time<true>(sm64, L, tw);
    double v[2] = {0.0, 0.0};
    for (int i = threadIdx.x; i < chunk; i += blockDim.x) {
        const int z = i >> lp, p = i & (P - 1);
        const double e = ez[z] * exy[p], k2 = kz2[z] + kxy[p];
        double2 u = cscale(sm64[i], scale);
        if (what & KICK1) u = cscale(u, e);
        if (what & SUMS) {
            const double n = u.x * u.x + u.y * u.y;
            v[0] += n;
            v[1] += n * k2;
        }
        if (kout) kout[((size_t)traj << (lplane + lz)) + ((size_t)z << lplane) + pen0 + p] = u;
        if (what & KICK2) u = cscale(u, e);
        if (what & TIMES_K2) u = cscale(u, k2);
        sm64[i] = u;
    }
    __syncthreads();
    fft_freq<false>(sm64, L, tw);
    for (int i = threadIdx.x; i < chunk; i += blockDim.x)
        g0[((size_t)(i >> lp) << lplane) + (i & (P - 1))] = sm64[(digit_rev(i >> lp, lz) << lp) + (i & (P - 1))];
    if (what & SUMS) {
        block_sum<2>(v, red);
        if (threadIdx.x == 0) {
            part[(size_t)blockIdx.x * 2] = v[0];
            part[(size_t)blockIdx.x * 2 + 1] = v[1];
        }
    }
}

// half-kick factors exp(-dt/2 k^2/2) of one trajectory (propagateKSpaceImaginaryTime, wigner_kernel.cu:128-134): nz of the
// kz, then nx ny of (kx, ky)
__global__ void k64_kick(const Gs64Par *__restrict__ par, int lx, int ly, int lz, double *__restrict__ kick)
{
    const GeomD &g = par->g;
    const int nx = 1 << lx, nz = 1 << lz, n = nz + (1 << (lx + ly));
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        double k2;
        if (i < nz) {
            const double kz = getk<double>(i, g.dkz, nz);
            k2 = kz * kz / 2.0;
        } else {
            const int pen = i - nz;
            const double kx = getk<double>(pen & (nx - 1), g.dkx, nx);
            const double ky = ly > 0 ? getk<double>(pen >> lx, g.dky, 1 << ly) : 0.0;
            k2 = (kx * kx + ky * ky) / 2.0;
        }
        kick[i] = exp(-g.dt_steady / 2.0 * k2);
    }
}

// out[traj * stride + off + k] = sum over n of part[(traj * n + i) * K + first + k], k < count; one block per trajectory
__global__ void k64_fold(const double *__restrict__ part, int n, int K, int first, int count, double *__restrict__ out,
                         int stride, int off)
{
    __shared__ double red[32];
    for (int k = 0; k < count; ++k) {
        double s[1] = {0.0};
        for (int i = threadIdx.x; i < n; i += blockDim.x) s[0] += part[((size_t)blockIdx.x * n + i) * K + first + k];
        block_sum<1>(s, red);
        if (threadIdx.x == 0) out[(size_t)blockIdx.x * stride + off + k] = s[0];
    }
}

// ---------------------------------------------------------------- real time
// Between calls an ensemble's state is k-space on every axis, as the reference keeps it. n steps take 2 n + 1 launches:
//   pencils   k-space -> half kick -> FFT_z                      \
//   planes    FFT_xy -> nonlinear step, loss noise -> IFFT_xy     | the last pencil pass ends
//   pencils   IFFT_z -> 1/cells, two half kicks -> FFT_z         /  after one half kick, in k-space
// The two half kicks between steps are applied one after the other, so that a run has the same bits however it is cut
// into calls. Where one kernel per operation and trajectory moved the state nine times a step, it moves twice. The plane
// pass is bound by FP64 arithmetic (most of it exp, sincos and the normals): 15 us of a step of four 16x16x128
// trajectories, whose pencil pass takes 7, near its latency. Measured, a step: 22.7 us for those four, 201 for 64, and 184
// for eight of 32x32x256; with one kernel per operation and trajectory 565, 9154 and 1311. Against an 80-bit reference the
// states are as far off as with one kernel per operation (nine runs of 20 to 100 steps on five grids: median 8.1e-15 of
// the state, 1.1e-14).

// A CTA holds ppc planes of both components, the second's after the first's.
//   E_STEP    state -> FFT_xy -> midpoint iteration (wigner_kernel.cu:184-229) and loss noise -> IFFT_xy -> state
//   E_OBSERVE state -> FFT_xy -> per-z sums |a|^2, |b|^2, Re and Im conj(a) b, times dV
//   E_TO_X    state -> FFT_xy -> state;   E_FROM_X  state -> IFFT_xy -> state
enum { E_STEP, E_OBSERVE, E_TO_X, E_FROM_X };

__device__ __forceinline__ double2 cexp64(double re, double im)
{
    double s, c;
    sincos(im, &s, &c);
    const double m = exp(re);
    return make_double2(m * c, m * s);
}

template <int MODE>
__global__ void __launch_bounds__(256) k64_evo_plane(double2 *A, double2 *B, const GeomD g, int lppc, const double2 *__restrict__ tx,
                                                     const double2 *__restrict__ ty, uint32_t traj0, uint32_t step, double *obs,
                                                     int row)
{
    extern __shared__ double2 sm64[];
    const int lx = g.lx, ly = g.ly, nx = 1 << lx, ny = 1 << ly, ld = nx + 1, lplane = lx + ly;
    const int lchunk = lppc + lplane, chunk = 1 << lchunk;
    const int lcta = g.lz - lppc;                               // CTAs per trajectory
    const int traj = blockIdx.x >> lcta, c0 = blockIdx.x & ((1 << lcta) - 1);
    const size_t cell0 = (size_t)c0 << lchunk;
    const size_t first = ((size_t)traj << (lplane + g.lz)) + cell0;
    double2 *const gA = A + first, *const gB = B + first;
    auto natural = [&](int i) { return (i >> lx) * ld + (i & (nx - 1)); };
    auto reversed = [&](int i) {
        return ((i >> lplane) * ny + digit_rev((i >> lx) & (ny - 1), ly)) * ld + digit_rev(i & (nx - 1), lx);
    };
    const Lines rows{lx, lppc + ly + 1, 1, 30, ld, 0}, cols{ly, lppc + lx + 1, ld, lx, 1, ny * ld};
    double2 *twx = sm64 + ((2 * ny << lppc) * ld), *twy = twx + nx;
    for (int i = threadIdx.x; i < nx; i += blockDim.x) copy16(twx + i, tx + i);
    for (int i = threadIdx.x; i < ny; i += blockDim.x) copy16(twy + i, ty + i);
    wait_predecessor();
    allow_successor();
    for (int i = threadIdx.x; i < 2 * chunk; i += blockDim.x)
        copy16(sm64 + (MODE == E_FROM_X ? natural(i) : reversed(i)), i < chunk ? gA + i : gB + (i - chunk));
    copy_wait();
    __syncthreads();
    if (MODE != E_FROM_X) {
        fft_time<false>(sm64, rows, twx);
        if (ly > 0) fft_time<false>(sm64, cols, twy);
    }
    if (MODE == E_STEP) {
        const double dt = g.dt_evo, h = dt / 2.0, iz = 1.0 / (g.lambda * g.lambda);
        const double ns = sqrt(dt / (2.0 * g.dV));
        const double c1 = sqrt(g.l111 / 6.0) * 3.0, c2 = sqrt(g.l12 / 2.0), c3 = sqrt(g.l22);
        for (int i = threadIdx.x; i < chunk; i += blockDim.x) {
            double2 &wa = sm64[natural(i)], &wb = sm64[natural(i + chunk)];
            const double X = -g.xmax + g.dx * (double)(i & (nx - 1));
            const double Y = ny > 1 ? -g.ymax + g.dy * (double)((i >> lx) & (ny - 1)) : 0.0;
            const double Z = -g.zmax + g.dz * (double)((c0 << lppc) + (i >> lplane));
            const double V = (X * X + Y * Y + Z * Z * iz) / 2.0;
            const double2 a0 = wa, b0 = wb;
            double2 x = a0, y = b0, da = make_double2(0, 0), db = make_double2(0, 0);
            for (int it = 0; it < g.itmax; ++it) {
                const double na = x.x * x.x + x.y * x.y, nb = y.x * y.x + y.y * y.y;
                const double pa_re = -(g.l111 * na * na + g.l12 * nb) / 2.0, pb_re = -(g.l22 * nb + g.l12 * na) / 2.0;
                const double pa_im = V + g.g11 * na + g.g12 * nb, pb_im = V + g.g22 * nb + g.g12 * na - g.detuning;
                da = cexp64(pa_re * h, pa_im * h);
                db = cexp64(pb_re * h, pb_im * h);
                x = cmul(a0, da);
                y = cmul(b0, db);
            }
            double2 ao = cmul(x, da), bo = cmul(y, db);
            if (g.noise) {
                double r[6];
                loss_normals6<double>(g.seed, traj0 + (uint32_t)traj, step, (uint32_t)(cell0 + i), r);
                const double2 w1 = make_double2(ns * r[0], ns * r[1]), w2 = make_double2(ns * r[2], ns * r[3]),
                              w3 = make_double2(ns * r[4], ns * r[5]);
                const double2 ca = cconj(a0), cb = cconj(b0);
                ao = cadd(ao, cadd(cmul(cscale(cmul(ca, ca), c1), w1), cmul(cscale(cb, c2), w2)));
                bo = cadd(bo, cadd(cmul(cscale(ca, c2), w2), cmul(cscale(cb, c3), w3)));
            }
            wa = ao;
            wb = bo;
        }
        __syncthreads();
    }
    if (MODE == E_STEP || MODE == E_FROM_X) {
        if (ly > 0) fft_freq<true>(sm64, cols, twy);
        fft_freq<true>(sm64, rows, twx);
    }
    if constexpr (MODE == E_OBSERVE) {
        const int plane = 1 << lplane;
        auto sums = [&](int pl, int i0, int di) {
            KVec<4> acc;
            for (int i = i0; i < plane; i += di) {
                const double2 u = sm64[natural((pl << lplane) + i)], v = sm64[natural(chunk + (pl << lplane) + i)];
                acc.v[0].add(u.x * u.x + u.y * u.y);
                acc.v[1].add(v.x * v.x + v.y * v.y);
                acc.v[2].add(u.x * v.x + u.y * v.y);
                acc.v[3].add(u.x * v.y - u.y * v.x);
            }
            return acc;
        };
        double *o = obs + ((size_t)traj * row + ((size_t)c0 << lppc)) * 4;
        if (lppc == 0) {
            const KVec<4> r = block_reduce<4>(sums(0, threadIdx.x, blockDim.x));
            if (threadIdx.x == 0)
                for (int k = 0; k < 4; ++k) o[k] = r.v[k].value() * g.dV;
        } else {                                                // planes of 128 cells at most: a warp each
            for (int pl = threadIdx.x >> 5; pl < 1 << lppc; pl += blockDim.x >> 5) {
                KVec<4> r = sums(pl, threadIdx.x & 31, 32);
                for (int k = 0; k < 4; ++k)
                    for (int off = 16; off > 0; off >>= 1)
                        ksum_merge(r.v[k], __shfl_down_sync(0xffffffffu, r.v[k].s, off),
                                   __shfl_down_sync(0xffffffffu, r.v[k].c, off));
                if ((threadIdx.x & 31) == 0)
                    for (int k = 0; k < 4; ++k) o[4 * pl + k] = r.v[k].value() * g.dV;
            }
        }
    } else {
        for (int i = threadIdx.x; i < 2 * chunk; i += blockDim.x)
            (i < chunk ? gA + i : gB + (i - chunk))[0] = sm64[MODE == E_TO_X ? natural(i) : reversed(i)];
    }
}

// v times a kick's phase, with the fused multiply-adds written out: the same bits in every pass
__device__ __forceinline__ double2 kicked(double2 v, double2 e)
{
    return make_double2(fma(v.x, e.x, -(v.y * e.y)), fma(v.x, e.y, v.y * e.x));
}

// A CTA holds 2^lp adjacent pencils of one component: [IFFT_z ->] scale -> `kicks` half kicks [-> FFT_z], from (sA, sB) to
// (dA, dB), which may be the same. kick: e^{i k^2/2 dt/2} of every cell (k64_evo_kick), copied beside the tile before the
// predecessor ends.
template <bool FROM_Z, bool TO_Z>
__global__ void __launch_bounds__(256) k64_evo_pencil(const double2 *sA, const double2 *sB, double2 *dA, double2 *dB, int lx, int ly,
                                                      int lz, int lp, int n, const double2 *__restrict__ tz,
                                                      const double2 *__restrict__ kick, double scale, int kicks)
{
    extern __shared__ double2 sm64[];
    const int nz = 1 << lz, lplane = lx + ly, P = 1 << lp, chunk = nz << lp, ltiles = lplane - lp;
    double2 *tw = sm64 + chunk, *ek = tw + nz;
    const bool second = (int)blockIdx.x >= n << ltiles;
    const int blk = second ? blockIdx.x - (n << ltiles) : blockIdx.x;
    const int traj = blk >> ltiles, pen0 = (blk & ((1 << ltiles) - 1)) << lp;
    const size_t off = ((size_t)traj << (lplane + lz)) + pen0;
    const double2 *src = (second ? sB : sA) + off;
    double2 *dst = (second ? dB : dA) + off;
    for (int i = threadIdx.x; i < nz; i += blockDim.x) copy16(tw + i, tz + i);
    if (kicks)
        for (int i = threadIdx.x; i < chunk; i += blockDim.x)
            copy16(ek + i, kick + ((size_t)(i >> lp) << lplane) + pen0 + (i & (P - 1)));
    wait_predecessor();
    allow_successor();
    for (int i = threadIdx.x; i < chunk; i += blockDim.x)
        copy16(sm64 + (FROM_Z ? (digit_rev(i >> lp, lz) << lp) + (i & (P - 1)) : i), src + ((size_t)(i >> lp) << lplane) + (i & (P - 1)));
    copy_wait();
    __syncthreads();
    const Lines L{lz, lp, P, 30, 1, 0};
    if (FROM_Z) fft_time<true>(sm64, L, tw);
    for (int i = threadIdx.x; i < chunk; i += blockDim.x) {
        double2 u = cscale(sm64[i], scale);
        if (kicks) {
            const double2 e = ek[i];
            u = kicked(u, e);
            if (kicks > 1) u = kicked(u, e);
        }
        if (TO_Z) sm64[i] = u;
        else dst[((size_t)(i >> lp) << lplane) + (i & (P - 1))] = u;
    }
    if (!TO_Z) return;
    __syncthreads();
    fft_freq<false>(sm64, L, tw);
    for (int i = threadIdx.x; i < chunk; i += blockDim.x)
        dst[((size_t)(i >> lp) << lplane) + (i & (P - 1))] = sm64[(digit_rev(i >> lp, lz) << lp) + (i & (P - 1))];
}

// e^{i k^2/2 dt/2} of every cell (propagateKSpaceRealTime, wigner_kernel.cu:137-151), one sine and cosine each. As the product
// of a (kx, ky) and a kz factor it had an error of the modulus that the many cells of a factor share, and with it the
// population drifted by up to 1.3e-14 in 100 steps of 8x8x64; now by up to 5e-15, as with one kernel per operation. The pass
// takes the same time, since a tile's phases are copied while the pass before it ends (a step of four 16x16x128 trajectories
// 22.75 us with factors, 22.7).
__global__ void k64_evo_kick(const GeomD g, double2 *__restrict__ kick)
{
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < g.cells; i += gridDim.x * blockDim.x) {
        const double kx = getk<double>(i & (g.nx - 1), g.dkx, g.nx), kz = getk<double>(i >> (g.lx + g.ly), g.dkz, g.nz);
        const double ky = g.ly > 0 ? getk<double>((i >> g.lx) & (g.ny - 1), g.dky, g.ny) : 0.0;
        double s, c;
        sincos((kx * kx + ky * ky + kz * kz) / 2.0 * g.dt_evo / 2.0, &s, &c);
        kick[i] = make_double2(c, s);
    }
}

size_t plane_smem(int lx, int ly, int lppc)
{
    return sizeof(double2) * ((((size_t)1 << (ly + lppc)) * ((1 << lx) + 1)) + ((size_t)1 << lx) + ((size_t)1 << ly));
}
size_t evo_plane_smem(int lx, int ly, int lppc) { return 2 * plane_smem(lx, ly, lppc); }    // (the twiddles' share is ample)
size_t evo_pencil_smem(int lz, int lp) { return sizeof(double2) * (((size_t)2 << (lz + lp)) + ((size_t)1 << lz)); }
size_t pencil_smem(int lz, int lp) { return sizeof(double2) * (((size_t)1 << (lz + lp)) + ((size_t)2 << lz)); }
constexpr size_t kMaxSmem = 200 * 1024;

int ilog(int n) { int r = 0; while ((1 << r) < n) ++r; return r; }
// A tile of 2048 elements or more takes 256 threads; so does one of 256 or more where the launch has no more than four CTAs an
// SM, which then wait for one another's latency less (a step of one ground state of 32x32x256 29.8 -> 20.4 us, of 16x16x128
// 10.3 -> 9.8; the pencil passes of four FP64 trajectories of 16x16x128, 256 CTAs: 27.4 -> 22.7 us a step; of 64, 4096 CTAs: 199
// -> 208). The real-time plane pass, bound by arithmetic, keeps 128 (four trajectories 27.4 -> 26.3 us, 64: 199 -> 248).
int threads_for(int log_elems, long long ctas) { return log_elems >= 11 || (log_elems >= 8 && ctas <= 4 * 148) ? 256 : 128; }

template <int MODE, typename S>
cudaError_t plane_launch(const Gs64Dims &d, const Gs64Tab &t, double2 *state, const Gs64Par *par, const double *norm_part,
                         const S *src, double2 *out, const double2 *kout, const double *sums4, double *part, cudaStream_t s)
{
    const size_t smem = plane_smem(d.lx, d.ly, d.lppc);
    cudaError_t e = ensure_smem_limit((const void *)k64_plane<MODE, S>, (int)kMaxSmem);
    if (e) return e;
    return launch_after(k64_plane<MODE, S>, d.n * d.plane_ctas(), threads_for(d.lppc + d.lx + d.ly, (long long)d.n * d.plane_ctas()), smem, s, state, par, d.lx,
                        d.ly, d.lz, d.lppc, t.x, t.y, norm_part, d.pencil_ctas(), src, out, kout, sums4, part);
}

cudaError_t pencil_launch(const Gs64Dims &d, const Gs64Tab &t, double2 *state, const Gs64Par *par, double scale, int what,
                          double *part, double2 *kout, cudaStream_t s)
{
    cudaError_t e = ensure_smem_limit((const void *)k64_pencil, (int)kMaxSmem);
    if (e) return e;
    return launch_after(k64_pencil, d.n * d.pencil_ctas(), threads_for(d.lz + d.lp, (long long)d.n * d.pencil_ctas()), pencil_smem(d.lz, d.lp), s, state, par, d.lx,
                        d.ly, d.lz, d.lp, t.z, t.kick, scale, what, part, kout);
}

void fold_launch(const Gs64Dims &d, const double *part, int n, int K, int first, int count, double *out, int off, cudaStream_t s)
{
    k64_fold<<<d.n, 128, 0, s>>>(part, n, K, first, count, out, kGs64Sums, off);
    g_launches++;
}

template <bool FROM_Z, bool TO_Z>
cudaError_t evo_pencil(const Evo64 &e, const double2 *sA, const double2 *sB, double2 *dA, double2 *dB, int n, double scale, int kicks,
                       cudaStream_t s)
{
    cudaError_t err = ensure_smem_limit((const void *)k64_evo_pencil<FROM_Z, TO_Z>, (int)kMaxSmem);
    if (err) return err;
    const GeomD &g = e.g;
    return launch_after(k64_evo_pencil<FROM_Z, TO_Z>, 2 * n << (g.lx + g.ly - e.lp), threads_for(g.lz + e.lp, (long long)2 * n << (g.lx + g.ly - e.lp)),
                        evo_pencil_smem(g.lz, e.lp), s, sA, sB, dA, dB, g.lx, g.ly, g.lz, e.lp, n, e.z, (const double2 *)e.kick, scale,
                        kicks);
}

template <int MODE>
cudaError_t evo_plane(const Evo64 &e, double2 *A, double2 *B, int n, uint32_t traj0, uint32_t step, double *obs, int row,
                      cudaStream_t s)
{
    cudaError_t err = ensure_smem_limit((const void *)k64_evo_plane<MODE>, (int)kMaxSmem);
    if (err) return err;
    const GeomD &g = e.g;
    return launch_after(k64_evo_plane<MODE>, n << (g.lz - e.lppc), threads_for(e.lppc + g.lx + g.ly, LLONG_MAX),
                        evo_plane_smem(g.lx, g.ly, e.lppc), s, A, B, g, e.lppc, e.x, e.y, traj0, step, obs, row);
}

} // namespace

// As gs64_dims; both components of a plane lie in shared memory.
bool evo64_dims(const GeomD &g, int n, Evo64 &e)
{
    e.g = g;
    e.lppc = std::max(0, std::min(8 - g.lx - g.ly, g.lz));
    e.lp = std::min(3, g.lx + g.ly);
    while (e.lp > 1 && (((long long)2 * n << (g.lx + g.ly - e.lp)) < 148 || sizeof(double2) << (g.lz + e.lp) > 32 * 1024)) --e.lp;
    e.ready = g.lx >= 1 && g.lz >= 1 && g.lx <= 10 && g.ly <= 10 && g.lz <= 10 && evo_plane_smem(g.lx, g.ly, e.lppc) <= kMaxSmem &&
              evo_pencil_smem(g.lz, e.lp) <= kMaxSmem && ((long long)2 * n << (g.lx + g.ly - e.lp)) < (1ll << 31) &&
              ((long long)n << (g.lz - e.lppc)) < (1ll << 31);
    return e.ready;
}

void evo64_kick_table(const Evo64 &e, cudaStream_t s)
{
    k64_evo_kick<<<std::min((e.g.cells + 127) / 128, 148 * 16), 128, 0, s>>>(e.g, e.kick);
    g_launches++;
}

cudaError_t evo64_steps(const Evo64 &e, double2 *a, double2 *b, int n, uint32_t step, int n_steps, cudaStream_t s)
{
    const double norm = 1.0 / e.g.cells;
    cudaError_t err = n_steps > 0 ? evo_pencil<false, true>(e, a, b, a, b, n, 1.0, 1, s) : cudaSuccess;
    for (int i = 0; i < n_steps && !err; ++i) {
        if ((err = evo_plane<E_STEP>(e, a, b, n, 0, step + (uint32_t)i, nullptr, 0, s))) break;
        err = i + 1 < n_steps ? evo_pencil<true, true>(e, a, b, a, b, n, norm, 2, s)
                              : evo_pencil<true, false>(e, a, b, a, b, n, norm, 1, s);
    }
    return err;
}

cudaError_t evo64_observe(const Evo64 &e, const double2 *a, const double2 *b, double2 *wa, double2 *wb, int n, double *obs, int row,
                          cudaStream_t s)
{
    const cudaError_t err = evo_pencil<false, true>(e, a, b, wa, wb, n, 1.0, 0, s);
    return err ? err : evo_plane<E_OBSERVE>(e, wa, wb, n, 0, 0, obs, row, s);
}

cudaError_t evo64_to_x(const Evo64 &e, const double2 *a, const double2 *b, double2 *wa, double2 *wb, int n, cudaStream_t s)
{
    const cudaError_t err = evo_pencil<false, true>(e, a, b, wa, wb, n, 1.0, 0, s);
    return err ? err : evo_plane<E_TO_X>(e, wa, wb, n, 0, 0, nullptr, 0, s);
}

cudaError_t evo64_from_x(const Evo64 &e, double2 *a, double2 *b, int n, cudaStream_t s)
{
    const cudaError_t err = evo_plane<E_FROM_X>(e, a, b, n, 0, 0, nullptr, 0, s);
    return err ? err : evo_pencil<true, false>(e, a, b, a, b, n, 1.0 / e.g.cells, 0, s);
}

// Tiles: a plane pass takes planes up to 256 cells together, a pencil pass 8 pencils (128-byte rows), fewer while one
// launch has fewer CTAs than the chip has SMs (down to 2: 32-byte sectors) or the tile would not fit.
bool gs64_dims(int nx, int ny, int nz, int n_traj, Gs64Dims &d)
{
    d.lx = ilog(nx); d.ly = ilog(ny); d.lz = ilog(nz);
    d.n = n_traj;
    d.lppc = std::max(0, std::min(8 - d.lx - d.ly, d.lz));
    d.lp = std::min(3, d.lx + d.ly);
    while (d.lp > 1 && ((long long)d.n * d.pencil_ctas() < 148 || pencil_smem(d.lz, d.lp) > 64 * 1024)) --d.lp;
    return d.lx >= 1 && d.lz >= 1 && d.lx <= 10 && d.ly <= 10 && d.lz <= 10 &&
           plane_smem(d.lx, d.ly, d.lppc) <= kMaxSmem && pencil_smem(d.lz, d.lp) <= kMaxSmem &&
           (long long)d.n * std::max(d.plane_ctas(), d.pencil_ctas()) < (1ll << 31);
}

cudaError_t gs64_start(const Gs64Dims &d, const Gs64Tab &t, double2 *state, const Gs64Par *par, const double2 *warm,
                       double *norm_part, cudaStream_t s)
{
    k64_kick<<<(d.cells() >> d.lz) / 128 + 1, 128, 0, s>>>(par, d.lx, d.ly, d.lz, t.kick);
    g_launches++;
    cudaError_t e = plane_launch<START, double2>(d, t, state, par, nullptr, warm, nullptr, nullptr, nullptr, nullptr, s);
    return e ? e : pencil_launch(d, t, state, par, 1.0 / d.cells(), SUMS | KICK2, norm_part, nullptr, s);
}

cudaError_t gs64_plane_step(const Gs64Dims &d, const Gs64Tab &t, double2 *state, const Gs64Par *par, const double *norm_part,
                            cudaStream_t s)
{
    return plane_launch<STEP, double2>(d, t, state, par, norm_part, nullptr, nullptr, nullptr, nullptr, nullptr, s);
}

cudaError_t gs64_pencil_step(const Gs64Dims &d, const Gs64Tab &t, double2 *state, const Gs64Par *par, double *norm_part,
                             cudaStream_t s)
{
    return pencil_launch(d, t, state, par, 1.0 / d.cells(), KICK1 | SUMS | KICK2, norm_part, nullptr, s);
}

cudaError_t gs64_boundary(const Gs64Dims &d, const Gs64Tab &t, double2 *state, const Gs64Par *par, double *norm_part,
                          double2 *out, double2 *kout, double *part, double *sums, cudaStream_t s)
{
    cudaError_t e = pencil_launch(d, t, state, par, 1.0 / d.cells(), KICK1 | SUMS, norm_part, kout, s);
    if (e) return e;
    e = plane_launch<OUT, double2>(d, t, state, par, norm_part, nullptr, out, kout, nullptr, part, s);
    if (e || !sums) return e;
    fold_launch(d, part, d.plane_ctas(), 5, 0, 5, sums, 0, s);
    fold_launch(d, norm_part, d.pencil_ctas(), 2, 0, 2, sums, 5, s);
    return cudaGetLastError();
}

cudaError_t gs64_resume(const Gs64Dims &d, const Gs64Tab &t, double2 *state, const Gs64Par *par, cudaStream_t s)
{
    return pencil_launch(d, t, state, par, 1.0 / (1 << d.lz), KICK2, nullptr, nullptr, s);
}

template <typename S>
static cudaError_t measures(const Gs64Dims &d, const Gs64Tab &t, const S *psi, double2 *work, const Gs64Par *par, double *part,
                            double *sums4, double *sums, cudaStream_t s)
{
    cudaError_t e = plane_launch<MEASURE, S>(d, t, work, par, nullptr, psi, nullptr, nullptr, nullptr, part, s);
    if (e) return e;
    k64_fold<<<d.n, 128, 0, s>>>(part, d.plane_ctas(), 3, 0, 3, sums4, 4, 0);
    if ((e = pencil_launch(d, t, work, par, 1.0 / d.cells(), SUMS | TIMES_K2, part, nullptr, s))) return e;
    k64_fold<<<d.n, 128, 0, s>>>(part, d.pencil_ctas(), 2, 1, 1, sums4, 4, 3);
    if ((e = plane_launch<RESIDUAL, S>(d, t, work, par, nullptr, psi, nullptr, nullptr, sums4, part, s))) return e;
    fold_launch(d, sums4, 1, 4, 0, 4, sums, 0, s);
    fold_launch(d, part, d.plane_ctas(), 1, 0, 1, sums, 4, s);
    g_launches += 2;
    return cudaGetLastError();
}

cudaError_t gs64_measures(const Gs64Dims &d, const Gs64Tab &t, const double2 *psi, double2 *work, const Gs64Par *par, double *part,
                          double *sums4, double *sums, cudaStream_t s)
{
    return measures(d, t, psi, work, par, part, sums4, sums, s);
}
cudaError_t gs64_measures(const Gs64Dims &d, const Gs64Tab &t, const float2 *psi, double2 *work, const Gs64Par *par, double *part,
                          double *sums4, double *sums, cudaStream_t s)
{
    return measures(d, t, psi, work, par, part, sums4, sums, s);
}
