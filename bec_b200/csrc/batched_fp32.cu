// batched_fp32.cu -- the general FP32 passes: any power-of-two grid, the initial states, and the reductions.
//
// One split step of the reference (propagate, programs/bec_wigner_3d.cuda/
// wigner.cu:178-199: K/2 -> FFT -> N(dt) -> IFFT -> 1/cells -> K/2) is
// regrouped into two fused passes over the state of every trajectory:
//
//   z pass (pencils along z):  IFFT_z -> 1/cells -> K (the previous step's
//                              second half-kick merged with this step's first)
//                              [-> pulse] -> FFT_z [-> observe]
//   plane pass (x-y planes):   FFT_xy -> nonlinear + losses + loss noise
//                              -> IFFT_xy
//
// The stored representation between passes is "k-space along x and y,
// x-space along z", in two scalings: a plane pass reads ifft_xy(psi_x)
// (normalised), so that FFT_xy returns psi_x exactly, and writes
// IFFT_xy(psi_x) (unnormalised, nx*ny times larger), which the next z pass
// turns into ifftn(psi_x) with its 1/cells. A z pass that ends a step (no
// plane pass follows) multiplies by nx*ny on the way out so the state is
// again in the form a z pass reads. Both components of a cell travel together as one 16-byte
// value (a.re, b.re, a.im, b.im).
//
// The shapes that most runs use take the register passes (fused_passes.cu); these kernels
// serve the others (2D slices, planes that are not square or not 8, 16 or 32 wide, other nz), and the transforms of
// every grid's initial and fetched states. They are bound by latency: a run on such a grid has a few thousand to a few
// hundred thousand cells, whose HBM time is well under a microsecond. So a CTA's tile is small (a plane or a few, 128 cells
// or more; two to sixteen pencils), which fills the chip with one trajectory, three radix-2 stages share a barrier, and the
// kinetic phases, the same at every step, come from a table per ensemble. A step of one 32x128 slice takes 6.6 us and one
// of a 4x4x512 trajectory 9.9 us; with 2048-cell tiles, a barrier per stage and the phases evaluated in FP64 in every pass
// they took 21.9 and 51.5 us, with the same bits. (256 trajectories of 64x32x16: 516 us a step, 887 then.)
#include <algorithm>

#include "common.cuh"
#include "engine.h"
#include "launch.cuh"
#include "reduce.cuh"

namespace {

// ---------------------------------------------------------------- cells
// A cell in the stored order (a.re, b.re, a.im, b.im), and the operations of the transforms on it.
struct __align__(16) Cell {
    float ar, br, ai, bi;
};
__device__ __forceinline__ Cell make_cell(float2 a, float2 b) { return Cell{a.x, b.x, a.y, b.y}; }
__device__ __forceinline__ float2 cell_a(const Cell &v) { return make_float2(v.ar, v.ai); }
__device__ __forceinline__ float2 cell_b(const Cell &v) { return make_float2(v.br, v.bi); }
__device__ __forceinline__ Cell cell_add(Cell p, Cell q) { return Cell{p.ar + q.ar, p.br + q.br, p.ai + q.ai, p.bi + q.bi}; }
__device__ __forceinline__ Cell cell_sub(Cell p, Cell q) { return Cell{p.ar - q.ar, p.br - q.br, p.ai - q.ai, p.bi - q.bi}; }
__device__ __forceinline__ Cell cell_scale(Cell v, float s) { return Cell{v.ar * s, v.br * s, v.ai * s, v.bi * s}; }
__device__ __forceinline__ Cell cell_mul(Cell v, float2 w) { return make_cell(cmul(cell_a(v), w), cmul(cell_b(v), w)); }

// ---------------------------------------------------------------- transforms in shared memory
// Radix-2 butterflies over lines of n = 2^logn cells at base(line) + e * es, base = (line & (2^lin - 1)) * ls_in + (line >>
// lin) * ls_out: decimation in time (bit-reversed -> natural) and in frequency (natural -> bit-reversed), one after the
// other in tw = W_n^k = e^{-2 pi i k / n} (conjugated when INV). A thread takes the 2^LR cells that LR consecutive stages
// combine through its registers, so a barrier separates three stages instead of one.
struct Lines {
    int logn, log_lines, es, lin, ls_in, ls_out;
    __device__ __forceinline__ int base(int line) const { return (line & ((1 << lin) - 1)) * ls_in + (line >> lin) * ls_out; }
};

// stages s .. s + LR - 1 in time
template <int LR, bool INV>
__device__ __forceinline__ void stages_time(Cell *buf, const Lines &L, const float2 *tw, int s)
{
    constexpr int R = 1 << LR;
    const int total = 1 << (L.log_lines + L.logn - LR);
    for (int w = threadIdx.x; w < total; w += blockDim.x) {
        const int line = w & ((1 << L.log_lines) - 1), jj = w >> L.log_lines;
        const int j = jj & ((1 << s) - 1);
        Cell *p = buf + L.base(line) + (((jj >> s) << (s + LR)) + j) * L.es;
        const int step = L.es << s;
        Cell x[R];
#pragma unroll
        for (int r = 0; r < R; ++r) x[r] = p[r * step];
#pragma unroll
        for (int q = 0; q < LR; ++q) {
            const int shift = L.logn - 1 - s - q;       // stage s + q: W_n^{pos << shift}, pos < 2^(s + q)
#pragma unroll
            for (int m = 0; m < 1 << q; ++m) {
                float2 t = tw[(j + (m << s)) << shift];
                if (INV) t.y = -t.y;
#pragma unroll
                for (int r = m; r < R; r += 2 << q) {
                    const Cell u = x[r], v = cell_mul(x[r + (1 << q)], t);
                    x[r] = cell_add(u, v);
                    x[r + (1 << q)] = cell_sub(u, v);
                }
            }
        }
#pragma unroll
        for (int r = 0; r < R; ++r) p[r * step] = x[r];
    }
    __syncthreads();
}

// stages s + LR - 1 .. s in frequency
template <int LR, bool INV>
__device__ __forceinline__ void stages_freq(Cell *buf, const Lines &L, const float2 *tw, int s)
{
    constexpr int R = 1 << LR;
    const int total = 1 << (L.log_lines + L.logn - LR);
    for (int w = threadIdx.x; w < total; w += blockDim.x) {
        const int line = w & ((1 << L.log_lines) - 1), jj = w >> L.log_lines;
        const int j = jj & ((1 << s) - 1);
        Cell *p = buf + L.base(line) + (((jj >> s) << (s + LR)) + j) * L.es;
        const int step = L.es << s;
        Cell x[R];
#pragma unroll
        for (int r = 0; r < R; ++r) x[r] = p[r * step];
#pragma unroll
        for (int q = LR - 1; q >= 0; --q) {
            const int shift = L.logn - 1 - s - q;
#pragma unroll
            for (int m = 0; m < 1 << q; ++m) {
                float2 t = tw[(j + (m << s)) << shift];
                if (INV) t.y = -t.y;
#pragma unroll
                for (int r = m; r < R; r += 2 << q) {
                    const Cell u = x[r], v = x[r + (1 << q)];
                    x[r] = cell_add(u, v);
                    x[r + (1 << q)] = cell_mul(cell_sub(u, v), t);
                }
            }
        }
#pragma unroll
        for (int r = 0; r < R; ++r) p[r * step] = x[r];
    }
    __syncthreads();
}

template <bool INV>
__device__ __forceinline__ void fft_time(Cell *buf, const Lines &L, const float2 *tw)
{
    const int first = L.logn % 3;
    if (first == 1) stages_time<1, INV>(buf, L, tw, 0);
    else if (first == 2) stages_time<2, INV>(buf, L, tw, 0);
    for (int s = first; s < L.logn; s += 3) stages_time<3, INV>(buf, L, tw, s);
}
template <bool INV>
__device__ __forceinline__ void fft_freq(Cell *buf, const Lines &L, const float2 *tw)
{
    const int first = L.logn % 3;
    for (int s = L.logn - 3; s >= first; s -= 3) stages_freq<3, INV>(buf, L, tw, s);
    if (first == 1) stages_freq<1, INV>(buf, L, tw, 0);
    else if (first == 2) stages_freq<2, INV>(buf, L, tw, 0);
}

__device__ __forceinline__ void copy16(Cell *dst_smem, const Cell *src)
{
    const unsigned d = (unsigned)__cvta_generic_to_shared(dst_smem);
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(d), "l"(src) : "memory");
}
__device__ __forceinline__ void copy8(float2 *dst_smem, const float2 *src)
{
    const unsigned d = (unsigned)__cvta_generic_to_shared(dst_smem);
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(d), "l"(src) : "memory");
}
__device__ __forceinline__ void copy_wait() { asm volatile("cp.async.wait_all;" ::: "memory"); }

// ---------------------------------------------------------------- initial states
// initializeEnsembles (wigner_kernel.cu:295-317): x-space a = gs + Va eta_a / sqrt(dV),
// b = Vb eta_b / sqrt(dV), eta = (n0 + i n1) / 2 from Philox or injected.
__device__ __forceinline__ Cell initial_cell(float2 g, const GroupParamsF &P, float2 ea, float2 eb)
{
    return Cell{g.x + P.init_a * ea.x, P.init_b * eb.x, g.y + P.init_a * ea.y, P.init_b * eb.y};
}
__device__ __forceinline__ Cell initial_cell_philox(float2 g, const GroupParamsF &P, uint32_t traj, uint32_t cell)
{
    float r[4];
    const uint64_t seed = ((uint64_t)P.seed_hi << 32) | P.seed_lo;
    normals4<float>(seed, traj, 0u, cell, RNG_TAG_INIT, r);
    return initial_cell(g, P, make_float2(0.5f * r[0], 0.5f * r[1]), make_float2(0.5f * r[2], 0.5f * r[3]));
}

// sources of the x-space cells of a preparation pass, by trajectory t of the launch and cell i
// the state itself, (a.re, a.im, b.re, b.im) as float4 (an uploaded trajectory)
struct FromState {
    const float4 *x;
    __device__ __forceinline__ Cell operator()(size_t at, int, int) const
    {
        const float4 v = x[at];
        return Cell{v.x, v.z, v.y, v.w};
    }
};
// one ensemble's ground state and its noise (injected, or Philox stream t)
struct FromGroup {
    GroupParamsF P;
    const double2 *gs;
    const float2 *noise;
    int cells;
    __device__ __forceinline__ Cell operator()(size_t, int t, int i) const
    {
        const float2 g = make_float2((float)gs[i].x, (float)gs[i].y);
        if (noise) return initial_cell(g, P, noise[((size_t)t * 2 + 0) * cells + i], noise[((size_t)t * 2 + 1) * cells + i]);
        return initial_cell_philox(g, P, (uint32_t)t, (uint32_t)i);
    }
};
// ground-state value i of a complex128 (double2), complex64 (float2) or real FP32 (float) array, as float2
__device__ __forceinline__ float2 gs_value(const double2 *p, int i) { return make_float2((float)p[i].x, (float)p[i].y); }
__device__ __forceinline__ float2 gs_value(const float2 *p, int i) { return p[i]; }
__device__ __forceinline__ float2 gs_value(const float *p, int i) { return make_float2(p[i], 0.f); }
// the same initial states for a run of trajectories that may belong to many ensembles: trajectory t takes its ensemble's
// parameters, its ground state gs_ptrs[tgroup[t]] and its Philox stream tlocal[t]
template <typename T>
struct FromGroups {
    const int *tgroup, *tlocal;
    const GroupParamsF *gp;
    const void *const *gs_ptrs;
    __device__ __forceinline__ Cell operator()(size_t, int t, int i) const
    {
        const int grp = tgroup[t];
        return initial_cell_philox(gs_value(static_cast<const T *>(gs_ptrs[grp]), i), gp[grp], (uint32_t)tlocal[t], (uint32_t)i);
    }
};

// ---------------------------------------------------------------- plane passes
// A CTA holds 2^lppc planes, rows padded by one cell against bank conflicts.
struct PlaneTile {
    int lx, ly, lz, lppc;
    const float2 *tx, *ty;      // W_nx^k, k < nx / 2, and W_ny^k (global; copied beside the tile)
    __host__ __device__ __forceinline__ int ld() const { return (1 << lx) + 1; }
    __device__ __forceinline__ int natural(int i) const { return (i >> lx) * ld() + (i & ((1 << lx) - 1)); }
    __device__ __forceinline__ int reversed(int i) const
    {
        const int y = (i >> lx) & ((1 << ly) - 1);
        return (((i >> (lx + ly)) << ly) + brev_bits(y, ly)) * ld() + brev_bits(i & ((1 << lx) - 1), lx);
    }
    __device__ __forceinline__ Lines rows() const { return Lines{lx, lppc + ly, 1, 30, ld(), 0}; }
    __device__ __forceinline__ Lines cols() const { return Lines{ly, lppc + lx, ld(), lx, 1, ld() << ly}; }
    __host__ __device__ __forceinline__ int cells() const { return ld() << (ly + lppc); }
    __device__ __forceinline__ float2 *tw(Cell *sm) const { return reinterpret_cast<float2 *>(sm + cells()); }
    // the twiddles beside the tile: read from L2 stage by stage they would add a trip to every barrier
    __device__ __forceinline__ void fetch_twiddles(Cell *sm) const
    {
        const int hx = 1 << lx >> 1, hy = 1 << ly >> 1;
        for (int i = threadIdx.x; i < hx + hy; i += blockDim.x) copy8(tw(sm) + i, i < hx ? tx + i : ty + i - hx);
    }
    __device__ __forceinline__ void forward(Cell *sm) const
    {
        fft_time<false>(sm, rows(), tw(sm));
        if (ly > 0) fft_time<false>(sm, cols(), tw(sm) + (1 << lx >> 1));
    }
    __device__ __forceinline__ void inverse(Cell *sm) const
    {
        if (ly > 0) fft_freq<true>(sm, cols(), tw(sm) + (1 << lx >> 1));
        fft_freq<true>(sm, rows(), tw(sm));
    }
};

// x-space cells of src -> IFFT_xy -> stored representation
template <typename Src>
__global__ void __launch_bounds__(256) k_prep(Cell *__restrict__ state, PlaneTile T, Src src)
{
    extern __shared__ Cell smw[];
    const int lchunk = T.lppc + T.lx + T.ly, lcells = T.lx + T.ly + T.lz;
    const size_t first = (size_t)blockIdx.x << lchunk;
    const int traj = (int)(first >> lcells), cell0 = (int)(first & ((1u << lcells) - 1));
    T.fetch_twiddles(smw);
    for (int i = threadIdx.x; i < 1 << lchunk; i += blockDim.x) smw[T.natural(i)] = src(first + i, traj, cell0 + i);
    copy_wait();
    __syncthreads();
    T.inverse(smw);
    for (int i = threadIdx.x; i < 1 << lchunk; i += blockDim.x) state[first + i] = smw[T.reversed(i)];
}

// where x-space cells go: (a.re, a.im, b.re, b.im), or the components times scale in FP64, as the caller of a state wants them
// (NULL: not that one)
struct ToCells {
    float4 *out;
    __device__ void operator()(size_t i, const Cell &v) const { out[i] = make_float4(v.ar, v.ai, v.br, v.bi); }
};
struct ToComponents {
    double2 *a, *b;
    double scale;
    __device__ void operator()(size_t i, const Cell &v) const
    {
        if (a) a[i] = make_double2(v.ar * scale, v.ai * scale);
        if (b) b[i] = make_double2(v.br * scale, v.bi * scale);
    }
};
// stored representation -> FFT_xy -> x-space cells
template <class Out>
__global__ void __launch_bounds__(256) k_unprep(const Cell *__restrict__ state, PlaneTile T, Out out)
{
    extern __shared__ Cell smw[];
    const int lchunk = T.lppc + T.lx + T.ly;
    const size_t first = (size_t)blockIdx.x << lchunk;
    T.fetch_twiddles(smw);
    for (int i = threadIdx.x; i < 1 << lchunk; i += blockDim.x) copy16(smw + T.reversed(i), state + first + i);
    copy_wait();
    __syncthreads();
    T.forward(smw);
    for (int i = threadIdx.x; i < 1 << lchunk; i += blockDim.x) {
        out(first + i, smw[T.natural(i)]);
    }
}

// the plane pass of a step
__global__ void __launch_bounds__(256) k_plane_any(Cell *__restrict__ state, PlaneTile T, const GroupParamsF *__restrict__ gp,
                                                   const int *__restrict__ tgroup, const int *__restrict__ tlocal,
                                                   const StepRef sr)
{
    extern __shared__ Cell smw[];
    const int lplane = T.lx + T.ly, lchunk = T.lppc + lplane, lcells = lplane + T.lz;
    const size_t first = (size_t)blockIdx.x << lchunk;
    const int traj = (int)(first >> lcells), cell0 = (int)(first & ((1u << lcells) - 1));
    T.fetch_twiddles(smw);
    const GroupParamsF P = gp[tgroup[traj]];
    const uint32_t tl = (uint32_t)tlocal[traj];
    wait_predecessor();
    allow_successor();
    for (int i = threadIdx.x; i < 1 << lchunk; i += blockDim.x) copy16(smw + T.reversed(i), state + first + i);
    const uint32_t step = *sr.step + sr.off;                 // Philox step index (device scalar, see fp32_put_step)
    const uint64_t seed = ((uint64_t)P.seed_hi << 32) | P.seed_lo;
    const float hdt = P.dt * 0.5f;
    copy_wait();
    __syncthreads();
    T.forward(smw);
    for (int i = threadIdx.x; i < 1 << lchunk; i += blockDim.x) {
        const int cell = cell0 + i;
        const int x = cell & ((1 << T.lx) - 1), y = (cell >> T.lx) & ((1 << T.ly) - 1), z = cell >> lplane;
        const float X = -P.xmax + P.dx * (float)x;
        const float Y = (T.ly > 0) ? -P.ymax + P.dy * (float)y : 0.0f;
        const float Z = -P.zmax + P.dz * (float)z;
        const float V = (X * X + Y * Y + Z * Z * P.inv_lambda2) * 0.5f;
        Cell *at = smw + T.natural(i);
        float2 a0 = cell_a(*at), b0 = cell_b(*at);
        float2 xa = a0, xb = b0, da = make_float2(0.f, 0.f), db = make_float2(0.f, 0.f);
        for (int it = 0; it < P.itmax; ++it) {
            const float na = xa.x * xa.x + xa.y * xa.y;
            const float nb = xb.x * xb.x + xb.y * xb.y;
            // propagateXSpaceTwoComponent (wigner_kernel.cu:203-223), reference sign
            // (fused multiply-adds written out where the compiler's choice could change with the code around them)
            const float pa_re = -fmaf(P.l111 * na, na, P.l12 * nb) * 0.5f;
            const float pa_im = V + P.g11 * na + P.g12 * nb;
            const float pb_re = -fmaf(P.l12, na, P.l22 * nb) * 0.5f;
            const float pb_im = V + P.g22 * nb + P.g12 * na - P.detuning;
            float sa, ca, sb, cb;
            sincosf(pa_im * hdt, &sa, &ca);
            sincosf(pb_im * hdt, &sb, &cb);
            const float ma = expf(pa_re * hdt), mb = expf(pb_re * hdt);
            da = make_float2(ma * ca, ma * sa);
            db = make_float2(mb * cb, mb * sb);
            xa = cmul(a0, da);
            xb = cmul(b0, db);
        }
        float2 ao = cmul(xa, da), bo = cmul(xb, db);
        if (P.noise) {
            float r[6];
            loss_normals6<float>(seed, tl, step, (uint32_t)cell, r);
            const float s = P.noise_amp;
            const float2 w1 = make_float2(s * r[0], s * r[1]);
            const float2 w2 = make_float2(s * r[2], s * r[3]);
            const float2 w3 = make_float2(s * r[4], s * r[5]);
            const float2 ca2 = cconj(a0), cb2 = cconj(b0);
            ao = cadd(ao, cadd(cmul(cscale(cmul(ca2, ca2), P.c1), w1), cmul(cscale(cb2, P.c2), w2)));
            bo = cadd(bo, cadd(cmul(cscale(ca2, P.c2), w2), cmul(cscale(cb2, P.c3), w3)));
        }
        *at = make_cell(ao, bo);
    }
    __syncthreads();
    T.inverse(smw);
    for (int i = threadIdx.x; i < 1 << lchunk; i += blockDim.x) state[first + i] = smw[T.reversed(i)];
    advance_step(sr);
}

// ---------------------------------------------------------------- z pass
// (a, b) <- M (a, b) with M row-major (m11, m12, m21, m22): a Rabi pulse
// (report.tex rotation matrix; applyHalfPiPulse / applyPiPulse,
// wigner_kernel.cu:320-341). It acts identically on every cell, so it
// commutes with the transforms and the kinetic phase.
__device__ __forceinline__ Cell apply_m(const float2 *m, Cell v)
{
    const float2 a = cell_a(v), b = cell_b(v);
    return make_cell(cadd(cmul(m[0], a), cmul(m[1], b)), cadd(cmul(m[2], a), cmul(m[3], b)));
}

// v times a kinetic phase, with the fused multiply-adds written out (as above)
__device__ __forceinline__ float2 kick(float2 v, float2 w)
{
    return make_float2(fmaf(v.x, w.x, -(v.y * w.y)), fmaf(v.y, w.x, v.x * w.y));
}
__device__ __forceinline__ Cell kick_cell(Cell v, float2 w) { return make_cell(kick(cell_a(v), w), kick(cell_b(v), w)); }

// e^{+i k^2/2 dt frac} of cell i of an ensemble (wigner_kernel.cu:143-144)
__device__ __forceinline__ float2 kick_phase(const GroupParamsF &P, int x, int y, int z, int nx, int ny, int nz, float frac)
{
    const int ix = kidx(x, nx), iy = ny > 1 ? kidx(y, ny) : 0, iz = kidx(z, nz);
    const double k2h = P.kin_x * (double)(ix * ix) + P.kin_y * (double)(iy * iy) + P.kin_z * (double)(iz * iz);
    return kin_phase(k2h * (double)frac);
}

// the phases of every cell of each of the class's n ensembles (ensemble e: parameters gp[groups[e]])
__global__ void k_kick_table(float2 *__restrict__ tab, const GroupParamsF *__restrict__ gp, const int *__restrict__ groups, int n,
                             int lx, int ly, int lz, float frac)
{
    const int lcells = lx + ly + lz;
    const size_t total = (size_t)n << lcells;
    for (size_t at = blockIdx.x * (size_t)blockDim.x + threadIdx.x; at < total; at += (size_t)gridDim.x * blockDim.x) {
        const int i = (int)(at & ((1u << lcells) - 1));
        tab[at] = kick_phase(gp[groups[at >> lcells]], i & ((1 << lx) - 1), (i >> lx) & ((1 << ly) - 1), i >> (lx + ly), 1 << lx,
                             1 << ly, 1 << lz, frac);
    }
}

struct ZArgs {
    int lx, ly, lz, lp;          // 2^lp pencils per CTA
    const float2 *tz;            // W_nz^k, k < nz / 2
    const float2 *kick;          // k_kick_table of the kick fraction, or NULL: evaluated here
    const int *tindex;           // ensemble of the table per trajectory
    float frac;                  // 0: no kick
    float scale, out_scale;      // 1/cells; nx ny when the pass ends a step, else 1
    int has_m;
    float2 m[4];
};

// OBS: the pass ends a step and writes, per z, the FP64 sums of |a|^2, |b|^2 and conj(a) b over the tile's pencils
template <bool OBS>
__global__ void __launch_bounds__(256) k_z_any(Cell *__restrict__ state, ZArgs A, const GroupParamsF *__restrict__ gp,
                                               const int *__restrict__ tgroup, double *__restrict__ obs)
{
    extern __shared__ Cell smw[];
    const int lplane = A.lx + A.ly, P2 = 1 << A.lp, nz = 1 << A.lz, chunk = nz << A.lp;
    float2 *tw = reinterpret_cast<float2 *>(smw + chunk);
    const int tile = blockIdx.x & ((1 << (lplane - A.lp)) - 1), traj = blockIdx.x >> (lplane - A.lp);
    const int pen0 = tile << A.lp;
    Cell *__restrict__ g = state + ((size_t)traj << (lplane + A.lz)) + pen0;
    for (int i = threadIdx.x; i < nz / 2; i += blockDim.x) copy8(tw + i, A.tz + i);
    const GroupParamsF P = gp[tgroup[traj]];
    const float2 *table = A.kick ? A.kick + ((size_t)A.tindex[traj] << (lplane + A.lz)) + pen0 : nullptr;
    wait_predecessor();
    allow_successor();
    for (int i = threadIdx.x; i < chunk; i += blockDim.x)
        copy16(smw + (brev_bits(i >> A.lp, A.lz) << A.lp) + (i & (P2 - 1)), g + ((size_t)(i >> A.lp) << lplane) + (i & (P2 - 1)));
    copy_wait();
    __syncthreads();
    const Lines L{A.lz, A.lp, P2, 30, 1, 0};
    fft_time<true>(smw, L, tw);       // IFFT_z: now full k-space (unnormalised)
    for (int i = threadIdx.x; i < chunk; i += blockDim.x) {
        const int z = i >> A.lp, p = i & (P2 - 1);
        Cell v = cell_scale(smw[i], OBS ? A.scale : A.scale * A.out_scale);
        if (A.frac != 0.0f)
            v = kick_cell(v, table ? table[((size_t)z << lplane) + p]
                                 : kick_phase(P, (pen0 + p) & ((1 << A.lx) - 1), (pen0 + p) >> A.lx, z, 1 << A.lx, 1 << A.ly, nz,
                                              A.frac));
        if (A.has_m) v = apply_m(A.m, v);
        smw[i] = v;
    }
    __syncthreads();
    if (OBS) {
        // per-z moments: transform the boundary state along z, sum over the tile's pencils
        fft_freq<false>(smw, L, tw);
        for (int z = threadIdx.x; z < nz; z += blockDim.x) {
            const Cell *row = smw + (brev_bits(z, A.lz) << A.lp);
            KSum s0, s1, s2, s3;
            for (int p = 0; p < P2; ++p) {
                const Cell v = row[p];
                s0.add((double)v.ar * v.ar + (double)v.ai * v.ai);
                s1.add((double)v.br * v.br + (double)v.bi * v.bi);
                s2.add((double)v.ar * v.br + (double)v.ai * v.bi);
                s3.add((double)v.ar * v.bi - (double)v.ai * v.br);
            }
            double *o = obs + ((size_t)blockIdx.x * nz + z) * 4;
            o[0] = s0.value(); o[1] = s1.value(); o[2] = s2.value(); o[3] = s3.value();
        }
        __syncthreads();
        fft_time<true>(smw, L, tw);   // back to k-space (times nz)
        const float inv_n = A.out_scale / (float)nz;
        for (int i = threadIdx.x; i < chunk; i += blockDim.x) smw[i] = cell_scale(smw[i], inv_n);
        __syncthreads();
    }
    fft_freq<false>(smw, L, tw);      // FFT_z back to the stored representation (bit-reversed slots)
    for (int i = threadIdx.x; i < chunk; i += blockDim.x)
        g[((size_t)(i >> A.lp) << lplane) + (i & (P2 - 1))] = smw[(brev_bits(i >> A.lp, A.lz) << A.lp) + (i & (P2 - 1))];
}

// obs_partial[traj][tile][z][4] -> traj_axial[traj][z][4] (scaled), traj_tot[traj][4]
__global__ void k_obs_reduce(const double *part, int tiles, int nz, const double *traj_scale, double *axial,
                             double *tot)
{
    const int traj = blockIdx.x;
    const double sc = traj_scale ? traj_scale[traj] : 1.0;
    KVec<4> acc;
    for (int z = threadIdx.x; z < nz; z += blockDim.x) {
        KSum s[4];
        for (int t = 0; t < tiles; ++t) {
            const double *p = part + (((size_t)traj * tiles + t) * nz + z) * 4;
            for (int k = 0; k < 4; ++k) s[k].add(p[k]);
        }
        for (int k = 0; k < 4; ++k) {
            const double v = s[k].value() * sc;
            if (axial) axial[((size_t)traj * nz + z) * 4 + k] = v;
            acc.v[k].add(v);
        }
    }
    KVec<4> r = block_reduce<4>(acc);
    if (threadIdx.x == 0)
        for (int k = 0; k < 4; ++k) tot[(size_t)traj * 4 + k] = r.v[k].value();
}

// FP64 sums of |a|^2, |b|^2 and Re, Im of conj(a) b over the stored state of a class, times `scale`: block
// `idx` sums range idx % blocks (of `blocks` equal ranges) of trajectory idx / blocks and writes
// part[idx * 4 + k], the [traj][tile][z = 0][4] layout of k_obs_reduce with `blocks` tiles.
__global__ void k_state_sums(const float4 *__restrict__ state, int cells, int blocks, double scale,
                             double *__restrict__ part)
{
    const int traj = blockIdx.x / blocks, b = blockIdx.x - traj * blocks;
    const int chunk = (cells + blocks - 1) / blocks;
    const int i0 = b * chunk, i1 = min(cells, i0 + chunk);
    const float4 *p = state + (size_t)traj * cells;
    // plain FP64 sums over a thread's few dozen cells (rounding ~1e-15 relative), compensated across threads
    double s0 = 0.0, s1 = 0.0, s2 = 0.0, s3 = 0.0;
    for (int i = i0 + threadIdx.x; i < i1; i += blockDim.x) {
        const float4 v = p[i];
        const double ax = v.x, bx = v.y, ay = v.z, by = v.w;
        s0 = fma(ax, ax, fma(ay, ay, s0));
        s1 = fma(bx, bx, fma(by, by, s1));
        s2 = fma(ax, bx, fma(ay, by, s2));
        s3 = fma(ax, by, fma(-ay, bx, s3));
    }
    KVec<4> acc;
    acc.v[0].add(s0);
    acc.v[1].add(s1);
    acc.v[2].add(s2);
    acc.v[3].add(s3);
    KVec<4> r = block_reduce<4>(acc);
    if (threadIdx.x == 0)
        for (int k = 0; k < 4; ++k) part[(size_t)blockIdx.x * 4 + k] = r.v[k].value() * scale;
}

// (a.re, b.re, a.im, b.im) <-> (a.re, a.im, b.re, b.im)
__global__ void k_swap_cells(float4 *state, size_t n)
{
    for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x)
        state[i] = make_float4(state[i].x, state[i].z, state[i].y, state[i].w);
}

__global__ void k_group_reduce(const double *traj_tot, const int *first, const int *count, double *out)
{
    const int gidx = blockIdx.x;
    KVec<4> acc;
    for (int t = threadIdx.x; t < count[gidx]; t += blockDim.x)
        for (int k = 0; k < 4; ++k) acc.v[k].add(traj_tot[((size_t)first[gidx] + t) * 4 + k]);
    KVec<4> r = block_reduce<4>(acc);
    if (threadIdx.x == 0)
        for (int k = 0; k < 4; ++k) out[(size_t)gidx * 4 + k] = r.v[k].value();
}


// ---------------------------------------------------------------- tiles
constexpr size_t kMaxTile = 64 * 1024;      // shared memory of a z tile
constexpr int kEnoughCtas = 2 * 148;

// Planes per CTA: as many as 1024 cells hold while the launch keeps two CTAs per SM, at least one, at least 128 cells (a
// cell per thread).
PlaneTile plane_tile(const ClassGeom &c, const float2 *tx, const float2 *ty)
{
    PlaneTile T{c.lx, c.ly, c.lz, 0, tx, ty};
    const int lplane = c.lx + c.ly;
    T.lppc = std::max(0, std::min(10 - lplane, c.lz));
    while (T.lppc > 0 && T.lppc + lplane > 7 && ((long long)c.n_traj << (c.lz - T.lppc)) < kEnoughCtas) --T.lppc;
    return T;
}
int plane_ctas(const ClassGeom &c, const PlaneTile &T) { return c.n_traj << (c.lz - T.lppc); }
int tile_threads(int log_cells) { return log_cells >= 10 ? 256 : 128; }
size_t plane_bytes(const PlaneTile &T) { return sizeof(Cell) * (size_t)T.cells() + sizeof(float2) * ((1 << T.lx >> 1) + (1 << T.ly >> 1)); }
constexpr int kMaxPlaneBytes = 16 * 3 * 1024 + 8 * 1024;    // planes of up to 2048 cells, rows of two padded to three

// Pencils per CTA: 16 (256-byte rows) for observing passes, whose sums take memory per tile; else 8 (128 bytes), fewer, down
// to two 32-byte sectors' worth, while the launch has fewer than two CTAs per SM; never more than fit.
int z_log_pencils(const ClassGeom &c, bool observe)
{
    int lp = std::min(observe ? 4 : 3, c.lx + c.ly);
    while (lp > 0 && (sizeof(Cell) << (lp + c.lz)) > kMaxTile) --lp;
    while (!observe && lp > 1 && ((long long)c.n_traj << (c.lx + c.ly - lp)) < kEnoughCtas) --lp;
    return lp;
}

template <typename Src>
void launch_prep(float4 *state, const ClassGeom &c, const float2 *tx, const float2 *ty, const Src &src, cudaStream_t s)
{
    if (c.n_traj <= 0) return;
    const PlaneTile T = plane_tile(c, tx, ty);
    ensure_smem_limit((const void *)k_prep<Src>, kMaxPlaneBytes);
    k_prep<Src><<<plane_ctas(c, T), tile_threads(T.lppc + c.lx + c.ly), plane_bytes(T), s>>>(reinterpret_cast<Cell *>(state), T, src);
    g_launches++;
}

} // namespace

void fp32_init_group(float4 *state, const ClassGeom &c, const GroupParamsF &gp, const double2 *gs, const float2 *noise,
                     const float2 *tx, const float2 *ty, cudaStream_t s)
{
    launch_prep(state, c, tx, ty, FromGroup{gp, gs, noise, c.cells}, s);
}

void fp32_init_batched(float4 *state, const ClassGeom &c, const int *tgroup, const int *tlocal, const GroupParamsF *gp,
                       const void *const *gs_ptrs, int host_type, const float2 *tx, const float2 *ty, cudaStream_t s)
{
    if (host_type == BEC_HOST_R32) launch_prep(state, c, tx, ty, FromGroups<float>{tgroup, tlocal, gp, gs_ptrs}, s);
    else if (host_type == BEC_HOST_C64) launch_prep(state, c, tx, ty, FromGroups<float2>{tgroup, tlocal, gp, gs_ptrs}, s);
    else launch_prep(state, c, tx, ty, FromGroups<double2>{tgroup, tlocal, gp, gs_ptrs}, s);
}

void fp32_prep(float4 *state, const ClassGeom &c, const float4 *x, const float2 *tx, const float2 *ty, cudaStream_t s)
{
    launch_prep(state, c, tx, ty, FromState{x}, s);
}

template <class Out>
static void unprep(const float4 *state, const ClassGeom &c, const Out &out, const float2 *tx, const float2 *ty, cudaStream_t s)
{
    if (c.n_traj <= 0) return;
    const PlaneTile T = plane_tile(c, tx, ty);
    ensure_smem_limit((const void *)k_unprep<Out>, kMaxPlaneBytes);
    k_unprep<Out><<<plane_ctas(c, T), tile_threads(T.lppc + c.lx + c.ly), plane_bytes(T), s>>>(reinterpret_cast<const Cell *>(state),
                                                                                              T, out);
    g_launches++;
}
void fp32_unprep(const float4 *state, const ClassGeom &c, float4 *x, const float2 *tx, const float2 *ty, cudaStream_t s)
{
    unprep(state, c, ToCells{x}, tx, ty, s);
}
void fp32_unprep_components(const float4 *state, const ClassGeom &c, double scale, double2 *a, double2 *b, const float2 *tx,
                            const float2 *ty, cudaStream_t s)
{
    unprep(state, c, ToComponents{a, b, scale}, tx, ty, s);
}

void fp32_ppass(float4 *state, const ClassGeom &c, const GroupParamsF *gp, const int *tgroup, const int *tlocal,
                const float2 *tx, const float2 *ty, const StepRef &sr, cudaStream_t s)
{
    if (c.n_traj <= 0) return;
    const PlaneTile T = plane_tile(c, tx, ty);
    ensure_smem_limit((const void *)k_plane_any, kMaxPlaneBytes);
    launch_after(k_plane_any, plane_ctas(c, T), tile_threads(T.lppc + c.lx + c.ly), plane_bytes(T), s,
                 reinterpret_cast<Cell *>(state), T, gp, tgroup, tlocal, sr);
}

namespace {
__global__ void k_put_step(uint32_t *d, int n, uint32_t v)
{
    for (int i = threadIdx.x; i < n; i += blockDim.x) d[i] = v;
}
} // namespace

void fp32_put_step(uint32_t *d_step, int n, uint32_t v, cudaStream_t s)
{
    k_put_step<<<1, 32, 0, s>>>(d_step, n, v);
    g_launches++;
}

int fp32_zpass_tiles(const ClassGeom &c) { return (c.nx * c.ny) >> z_log_pencils(c, true); }

void fp32_kick_table(float2 *tab, const ClassGeom &c, const GroupParamsF *gp, const int *groups, int n_groups, float frac,
                     cudaStream_t s)
{
    if (n_groups <= 0) return;
    const size_t blocks = ((size_t)n_groups * c.cells + 127) / 128;
    k_kick_table<<<(int)std::min<size_t>(blocks, 148 * 128), 128, 0, s>>>(tab, gp, groups, n_groups, c.lx, c.ly, c.lz, frac);
    g_launches++;
}

void fp32_zpass(float4 *state, const ClassGeom &c, const GroupParamsF *gp, const int *tgroup, const float2 *tz,
                const float2 *kick, const int *tindex, float frac, float scale, float out_scale, const float2 *m, double *obs,
                cudaStream_t s)
{
    if (c.n_traj <= 0) return;
    ZArgs A{};
    A.lx = c.lx; A.ly = c.ly; A.lz = c.lz;
    A.lp = z_log_pencils(c, obs != nullptr);
    A.tz = tz;
    A.kick = kick;
    A.tindex = tindex;
    A.frac = frac;
    A.scale = scale;
    A.out_scale = out_scale;
    A.has_m = m ? 1 : 0;
    for (int i = 0; m && i < 4; ++i) A.m[i] = m[i];
    const int ctas = c.n_traj << (c.lx + c.ly - A.lp), threads = tile_threads(c.lz + A.lp);
    const size_t bytes = (sizeof(Cell) << (c.lz + A.lp)) + sizeof(float2) * ((size_t)c.nz / 2);
    const int most = (int)(kMaxTile + sizeof(float2) * 256);
    Cell *st = reinterpret_cast<Cell *>(state);
    if (obs) {
        ensure_smem_limit((const void *)k_z_any<true>, most);
        launch_after(k_z_any<true>, ctas, threads, bytes, s, st, A, gp, tgroup, obs);
    } else {
        ensure_smem_limit((const void *)k_z_any<false>, most);
        launch_after(k_z_any<false>, ctas, threads, bytes, s, st, A, gp, tgroup, obs);
    }
}

void obs_reduce(const double *obs_partial, int n_traj, int tiles, int nz, const double *traj_scale,
                double *traj_axial, double *traj_tot, cudaStream_t s)
{
    if (n_traj <= 0) return;
    k_obs_reduce<<<n_traj, 256, 0, s>>>(obs_partial, tiles, nz, traj_scale, traj_axial, traj_tot);
    g_launches++;
}

void fp32_state_sums(const float4 *state, int cells, int n_traj, int blocks, double scale, double *part,
                     cudaStream_t s)
{
    if (n_traj <= 0) return;
    k_state_sums<<<n_traj * blocks, 256, 0, s>>>(state, cells, blocks, scale, part);
    g_launches++;
}

void fp32_swap_cells(float4 *state, size_t n, cudaStream_t s)
{
    if (n == 0) return;
    const size_t blocks = (n + 255) / 256;
    k_swap_cells<<<(int)(blocks > 148 * 32 ? 148 * 32 : blocks), 256, 0, s>>>(state, n);
    g_launches++;
}

void group_reduce(const double *traj_tot, const int *group_first, const int *group_count, int n_groups,
                  double *out, cudaStream_t s)
{
    if (n_groups <= 0) return;
    k_group_reduce<<<n_groups, 256, 0, s>>>(traj_tot, group_first, group_count, out);
    g_launches++;
}

namespace {
// the profile of an ensemble: the compensated sum over its trajectories, in order; several loads in flight (one at a time, each
// adds a trip to L2: 3000 trajectories of 8x8x64 745 us a profile, 407 so)
__global__ void k_group_axial(const double *__restrict__ traj_axial, int row, const int *__restrict__ groups,
                              const int *__restrict__ first, const int *__restrict__ count, int base,
                              const int *__restrict__ off, double *__restrict__ out)
{
    const int g = groups ? groups[blockIdx.x] : blockIdx.x, i = blockIdx.y * blockDim.x + threadIdx.x;
    if (i >= off[g + 1] - off[g]) return;
    const double *src = traj_axial + (size_t)(first[g] - base) * row * 4 + i;
    KSum acc;
    constexpr int U = 16;
    const int n = count[g];
    int t = 0;
    for (; t + U <= n; t += U) {
        double v[U];
#pragma unroll
        for (int u = 0; u < U; ++u) v[u] = src[(size_t)(t + u) * row * 4];
#pragma unroll
        for (int u = 0; u < U; ++u) acc.add(v[u]);
    }
    for (; t < n; ++t) acc.add(src[(size_t)t * row * 4]);
    out[off[g] + i] = acc.value();
}

// the same for thousands of trajectories, a warp per value (20,000 of 2x2x2: 362 us a profile, 1690 in order)
__global__ void __launch_bounds__(128) k_group_axial_long(const double *__restrict__ traj_axial, int row,
                                                          const int *__restrict__ groups, const int *__restrict__ first,
                                                          const int *__restrict__ count, int base, const int *__restrict__ off,
                                                          double *__restrict__ out)
{
    const int g = groups ? groups[blockIdx.x] : blockIdx.x, i = blockIdx.y * 4 + (threadIdx.x >> 5);
    if (i >= off[g + 1] - off[g]) return;
    const double *src = traj_axial + (size_t)(first[g] - base) * row * 4 + i;
    KSum acc;
    const int n = count[g];
#pragma unroll 8
    for (int t = threadIdx.x & 31; t < n; t += 32) acc.add(src[(size_t)t * row * 4]);
    for (int o = 16; o > 0; o >>= 1)
        ksum_merge(acc, __shfl_down_sync(0xffffffffu, acc.s, o), __shfl_down_sync(0xffffffffu, acc.c, o));
    if ((threadIdx.x & 31) == 0) out[off[g] + i] = acc.value();
}
constexpr int kLongEnsemble = 4096;
} // namespace

void group_axial(const double *traj_axial, int row, const int *groups, int n, const int *first, const int *count, int base,
                 int longest, const int *off, double *out, cudaStream_t s)
{
    if (n <= 0) return;
    if (longest > kLongEnsemble)
        k_group_axial_long<<<dim3(n, row), 128, 0, s>>>(traj_axial, row, groups, first, count, base, off, out);
    else
        k_group_axial<<<dim3(n, (4 * row + 127) / 128), 128, 0, s>>>(traj_axial, row, groups, first, count, base, off, out);
    g_launches++;
}
