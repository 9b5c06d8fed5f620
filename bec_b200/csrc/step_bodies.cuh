// step_bodies.cuh -- the register-resident plane and pencil passes of the FP32 path as device bodies.
//
// One split step of the reference (propagate, programs/bec_wigner_3d.cuda/wigner.cu:178-199) is
// regrouped into a pencil pass (IFFT_z -> kinetic phase [-> pulse] -> FFT_z) and a plane pass
// (FFT_xy -> nonlinear + losses + loss noise -> IFFT_xy) over the stored representation (k-space
// along x and y, x-space along z; see batched_fp32.cu). Every line of the 3D transform lives in one
// thread's registers (or, for 32-point lines, in one lane of each of two warps); shared memory only
// transposes.
//
// The bodies run on a "virtual block" (VBlock): a contiguous group of a CTA's threads with its own
// index and barrier. The standalone kernels (fused_passes.cu) give each body a whole CTA; the fused
// step kernel (step_kernel.cu) runs several virtual blocks of one item side by side in a 256-thread
// CTA, each synchronising on its own named barrier.
//
// plane pass (square planes N x N, N = 8, 16): one warp per 32/N planes. Lane c loads column c of its
//   plane from HBM (each load instruction of the warp reads consecutive 16-byte cells), transforms it
//   along y, writes it to a padded shared tile, reads back row c, transforms along x, applies
//   the nonlinear / loss / loss-noise step to its N cells, and returns the same way. Both components of
//   a cell are one 16-byte cpair (fft_reg.cuh).
// plane pass, 32 x 32 planes: two warps per plane, a 32-point line shared by lane L of each warp
//   (split32.cuh).
// pencil pass (nz = 64, 128, 256 = 16 G): 16 (or 8) adjacent pencils of a trajectory per virtual block of
//   nz (or nz / 2) threads. A four-step decomposition nz = 16 x G: each thread holds 16 elements (z = j + G m)
//   and does a 16-point DFT, twiddles, and after one shared-memory transpose a G-point DFT across j;
//   the kinetic phase e^{i k^2/2 dt} (wigner_kernel.cu:137-151) is applied in full k-space as the
//   product of a per-pencil (kx, ky) factor and a per-kz factor; the forward transform retraces the
//   same steps.
//
// Shared lines are padded by one 16-byte cell, so that both the row-wise and the column-wise access of a quarter warp touch
// eight different bank groups and every access has an address and a constant offset. (A tile that must stay dense, the
// state held in shared memory, is swizzled on the cell index instead, col ^ (row & 7), at an instruction or two an access:
// with every tile swizzled the 32 x 32 plane pass took 303.5 thread-instructions a cell, 283 padded, and a step of 256
// trajectories of 32x32x256 1.309 ms, 1.247; with eight pencils a CTA besides, and the line exchange in the plane's tile,
// 1.215 to 1.231.)
//
// The plane bodies read the state with ld.global.cg (L2 only): inside the fused step kernel another
// SM's pencil item wrote those lines during the same launch, and L1 is not coherent across SMs.
#pragma once

#include "engine.h"
#include "fft_reg.cuh"
#include "physics.cuh"
#include "split32.cuh"

namespace stepk {

using fftreg::cpair;
using fftreg::dft;
using fftreg::f32x2;

// a cell from L2 (ld.global.cg; a volatile load, which keeps its place among waits and barriers)
__device__ __forceinline__ cpair ld_cg(const cpair *p)
{
    const ulonglong2 u = __ldcg(reinterpret_cast<const ulonglong2 *>(p));
    return cpair{u.x, u.y};
}

// A group of nthr consecutive threads of a CTA acting as one block.
struct VBlock {
    int tid;     // thread index within the group
    int bid;     // block index the body works on
    int bar;     // barrier: 0 = the whole CTA (__syncthreads), else a named barrier of nthr threads
    int nthr;
    __device__ __forceinline__ void sync() const
    {
        if (bar == 0) __syncthreads();
        else asm volatile("bar.sync %0, %1;" ::"r"(bar), "r"(nthr) : "memory");
    }
};

// ---------------------------------------------------------------- plane pass, N = 8, 16
// 4 warps (128 threads); tile: plane_tile_cells<N> cells, 4 warps x (32 / N) planes of N rows
// SMEM: `state` is a trajectory held in shared memory and `tile` is the same memory (the transposes run in
// place): plain loads instead of L2-only ones, and the warp's loads all done before its first store.
template <int N>
constexpr int plane_tile_cells = 4 * (32 / N) * N * (N + 1);
template <int N, bool SMEM = false>
__device__ __forceinline__ void plane_body(const VBlock &vb, cpair *__restrict__ state, int nz, int cells,
                                           const GroupParamsF *__restrict__ gp, const int *__restrict__ tgroup,
                                           const int *__restrict__ tlocal, uint32_t step, cpair *tile)
{
    constexpr int W = 32 / N;          // planes per warp
    constexpr int PLANE = N * N;
    const int warp = vb.tid >> 5, lane = vb.tid & 31;
    const int wp = lane / N, c = lane % N;
    const int plane_id = (vb.bid * 4 + warp) * W + wp;
    const int traj = plane_id / nz, z = plane_id - traj * nz;
    cpair *__restrict__ g = state + (size_t)traj * cells + (size_t)z * PLANE;
    // row and column c of the plane in shared memory: padded rows, or swizzled ones where the state lies there
    constexpr int LD = SMEM ? N : N + 1;
    cpair *s = tile + (warp * W + wp) * (N * LD);
    cpair *row = s + c * LD;
    auto in_row = [&](int x) -> cpair & { return row[SMEM ? x ^ (c & 7) : x]; };
    auto in_col = [&](int y) -> cpair & { return s[y * LD + (SMEM ? c ^ (y & 7) : c)]; };

    const GroupParamsF P = gp[tgroup[traj]];

    cpair v[N];
#pragma unroll
    for (int y = 0; y < N; ++y) v[y] = SMEM ? g[y * N + c] : ld_cg(g + y * N + c);
    if (SMEM) __syncwarp();

    // Four transforms share one loop body (the kernel is otherwise bound by
    // instruction fetch): pass 0 forward along y, pass 1 forward along x,
    // passes 2 and 3 inverse along x and y (the inverse DFT body, no sign flips).
#pragma unroll 1
    for (int pass = 0; pass < 4; ++pass) {
        if (pass >= 2) dft<N, true>(v);
        else dft<N, false>(v);
        if (pass == 0) {
            // column c -> row c
#pragma unroll
            for (int y = 0; y < N; ++y) in_col(y) = v[y];
            __syncwarp();
#pragma unroll
            for (int x = 0; x < N; ++x) v[x] = in_row(x);
        } else if (pass == 1) {
            // lane c owns row y = c: the cells go through the physics one at a time
            // from its own shared row (a rolled loop keeps the kernel small)
#pragma unroll
            for (int x = 0; x < N; ++x) in_row(x) = v[x];
            // coordinates and trap potential with every fused multiply-add written out (same bits in every kernel)
            const float Y = fmaf(P.dy, (float)c, -P.ymax);
            const float Z = fmaf(P.dz, (float)z, -P.zmax);
            const float base = fmaf(Y, Y, (Z * Z) * P.inv_lambda2);
            const uint32_t tl = (uint32_t)tlocal[traj];
            const CellConsts K = cell_consts(P);
            const uint32_t cell0 = (uint32_t)(z * PLANE + c * N);
            const PhiloxKeys keys = philox_keys(P.seed_lo, P.seed_hi);
            // cells in fours: the four Philox draws interleave (loss_noise_cell4)
#pragma unroll 1
            for (int x = 0; x < N; x += 4) {
                cpair v0[4], o[4];
#pragma unroll
                for (int q = 0; q < 4; ++q) {
                    const float X = fmaf(P.dx, (float)(x + q), -P.xmax);
                    v0[q] = in_row(x + q);
                    o[q] = nonlinear_cell(v0[q], 0.5f * fmaf(X, X, base), K);
                }
                if (P.noise) loss_noise_cell4(o, v0, K, keys, tl, step, cell0 + x);
#pragma unroll
                for (int q = 0; q < 4; ++q) in_row(x + q) = o[q];
            }
#pragma unroll
            for (int x = 0; x < N; ++x) v[x] = in_row(x);
        } else if (pass == 2) {
            // row c -> column c
#pragma unroll
            for (int x = 0; x < N; ++x) in_row(x) = v[x];
            __syncwarp();
#pragma unroll
            for (int y = 0; y < N; ++y) v[y] = in_col(y);
        }
    }
    if (SMEM) __syncwarp();
#pragma unroll
    for (int y = 0; y < N; ++y) g[y * N + c] = v[y];
}

// ---------------------------------------------------------------- plane pass, 32 x 32, two warps a plane
// 64 threads; every 32-point line is shared by lane L of warp 0 and lane L of warp 1, 16 elements
// each, half the registers of a one-lane line, so more warps fit on an SM. tile: kPlane32Cells cells, the
// plane and, between its transposes, the line exchange slots (slots of their own would take a third of the shared memory
// from L1: 365 trajectories of 32x32x256 1.171 ms with them, 1.158 without, for five barriers more).
constexpr int kPlane32Cells = 32 * 33;
__device__ __forceinline__ void plane32_body(const VBlock &vb, cpair *__restrict__ state, int nz, int cells,
                                             const GroupParamsF *__restrict__ gp, const int *__restrict__ tgroup,
                                             const int *__restrict__ tlocal, uint32_t step, cpair *tile)
{
    using namespace split32;
    const int h = vb.tid >> 5, lane = vb.tid & 31;
    const int plane_id = vb.bid;
    const int traj = plane_id / nz, z = plane_id - traj * nz;
    cpair *__restrict__ g = state + (size_t)traj * cells + (size_t)z * 1024;
    const GroupParamsF P = gp[tgroup[traj]];
    auto bar = [&vb]() { vb.sync(); };
    cpair *row = tile + lane * 33, *col = tile + lane;

    cpair v[16];
    // forward along y (lane = column), then along x (lane = row); shared code body
#pragma unroll 1
    for (int pass = 0; pass < 2; ++pass) {
        if (pass == 0) {
#pragma unroll
            for (int j = 0; j < 16; ++j) v[j] = ld_cg(g + (2 * j + h) * 32 + lane);
        } else {
#pragma unroll
            for (int j = 0; j < 16; ++j) v[j] = row[2 * j + h];
            vb.sync();
        }
        fwd_line(v, tile, h, lane, bar);
        vb.sync();
        if (pass == 0) {
#pragma unroll
            for (int s = 0; s < 16; ++s) col[kblk(s, h) * 33] = v[s];
            vb.sync();
        }
    }
    // x-space: lane owns row y = lane, cells x = kblk(s, h); the physics runs as a rolled loop
    // over those cells in the tile
    {
#pragma unroll
        for (int s = 0; s < 16; ++s) row[kblk(s, h)] = v[s];
        const float Y = fmaf(P.dy, (float)lane, -P.ymax);
        const float Z = fmaf(P.dz, (float)z, -P.zmax);
        const float base = fmaf(Y, Y, (Z * Z) * P.inv_lambda2);
        const uint32_t tl = (uint32_t)tlocal[traj];
        const CellConsts K = cell_consts(P);
        const uint32_t cell0 = (uint32_t)(z * 1024 + lane * 32);
        const PhiloxKeys keys = philox_keys(P.seed_lo, P.seed_hi);
        // cells in pairs (x, x + 1; kblk keeps pairs of even s adjacent): the two Philox draws interleave.
        // (Fours measured slower here: the larger loop body misses in the instruction cache.)
#pragma unroll 1
        for (int s = 0; s < 16; s += 2) {
            const int x = kblk(s, h);
            const float X0 = fmaf(P.dx, (float)x, -P.xmax), X1 = fmaf(P.dx, (float)(x + 1), -P.xmax);
            cpair *s0 = row + x, *s1 = row + x + 1;
            const cpair v0 = *s0, v1 = *s1;
            cpair o0 = nonlinear_cell(v0, 0.5f * fmaf(X0, X0, base), K);
            cpair o1 = nonlinear_cell(v1, 0.5f * fmaf(X1, X1, base), K);
            if (P.noise)
                loss_noise_cell2(o0, v0, o1, v1, K, keys, tl, step, cell0 + x, cell0 + x + 1);
            *s0 = o0;
            *s1 = o1;
        }
#pragma unroll
        for (int s = 0; s < 16; ++s) v[s] = row[kblk(s, h)];
    }
    vb.sync();    // every row is read
    // inverse along x (lane = row), then along y (lane = column); shared code body
#pragma unroll 1
    for (int pass = 0; pass < 2; ++pass) {
        if (pass == 1) {
#pragma unroll
            for (int s = 0; s < 16; ++s) v[s] = col[kblk(s, h) * 33];
            vb.sync();
        }
        inv_line(v, tile, h, lane, bar);
        if (pass == 0) {
            vb.sync();
#pragma unroll
            for (int m = 0; m < 16; ++m) row[2 * m + h] = v[m];
            vb.sync();
        }
    }
#pragma unroll
    for (int m = 0; m < 16; ++m) g[(2 * m + h) * 32 + lane] = v[m];
}

// ---------------------------------------------------------------- pencil pass
// 8-byte global -> shared copy that completes asynchronously (cp.async), and the wait for this thread's copies
__device__ __forceinline__ void copy_async8(float2 *dst_smem, const float2 *src)
{
    const unsigned d = (unsigned)__cvta_generic_to_shared(dst_smem);
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(d), "l"(src) : "memory");
}
__device__ __forceinline__ void copy_async_wait() { asm volatile("cp.async.wait_all;" ::: "memory"); }

struct PencilArgs {
    float frac;          // kick in units of dt (0.5 + 0.5 for a full step)
    float scale;         // 1/cells times the output scale
    int has_m;
    float2 m[4];         // pulse matrix, row-major
};

// The four-step z transform of a tile of PEN adjacent pencils (nz = 16 G; PEN * G threads), in three
// stages separated by barriers of the tile's threads. buf holds CELLS cells.
//   inv1:  thread (p, j) = (t % PEN, t / PEN) holds z = j + G m, m < 16: inverse 16-point DFT over
//          m -> k1, twiddle W^{-j k1}, to buf
//   mid:   thread (q, p2) = (t % G, t / G) gathers k1 = q + G r (r < 16 / G) for all j: inverse G-point
//          DFT over j -> k2 (k = k1 + 16 k2), kinetic phase (and pulse), forward G-point DFT, twiddle;
//          mid_store writes it back after the caller's barrier
//   fwd3:  thread (p, j) gathers its k1 < 16 and finishes with the forward 16-point DFT over k1 -> m
// The buffer is a cell pointer or an accessor (a functor mapping the buffer index to a cell slot, e.g.
// into a tile of a state held in shared memory).
__device__ __forceinline__ cpair &zat(cpair *b, int i) { return b[i]; }
template <class F>
__device__ __forceinline__ cpair &zat(const F &f, int i) { return f(i); }

// PAD: a pencil takes NZ + 1 cells of buf, so that every access has a base and a constant offset; otherwise NZ, its rows of
// 16 swizzled.
template <int NZ, int PEN, bool PAD = true>
struct ZTile {
    static constexpr int R = 16, G = NZ / 16, CELLS = PEN * (PAD ? NZ + 1 : NZ);
    static_assert(NZ % 16 == 0 && G <= 16, "nz = 16 G with G <= 16");

    __device__ static __forceinline__ int bix(int p, int jj, int k1)
    {
        return PAD ? p * (NZ + 1) + jj * R + k1 : (p * G + jj) * R + (k1 ^ (p & 7));
    }

    template <class Buf>
    __device__ static __forceinline__ void inv1(cpair (&x)[R], Buf buf, const float2 *tw, int p, int j)
    {
        dft<R, true>(x);                                            // over m -> k1 (inverse)
#pragma unroll
        for (int k1 = 1; k1 < R; ++k1) {
            const float2 w = tw[j * k1];
            x[k1] = fftreg::cmulw(x[k1], make_float2(w.x, -w.y));   // W^{-j k1}
        }
#pragma unroll
        for (int k1 = 0; k1 < R; ++k1) zat(buf, bix(p, j, k1)) = x[k1];
    }

    // pxy: the pencil's (kx, ky) factor times the scale; kzp: the kz factors
    template <class Buf>
    __device__ static __forceinline__ void mid(cpair (&y)[R], Buf buf, const float2 *tw, const float2 *kzp,
                                               float2 pxy, const PencilArgs &pa, int q, int p2)
    {
#pragma unroll
        for (int r = 0; r < R / G; ++r)
#pragma unroll
            for (int jj = 0; jj < G; ++jj) y[r * G + jj] = zat(buf, bix(p2, jj, q + G * r));
#pragma unroll
        for (int r = 0; r < R / G; ++r) dft<G, true>(y + r * G);   // over j -> k2: k = k1 + 16 k2

        // the two unit-modulus factors are applied to the data one after the other: their product, the same
        // every step for a mode, would round the same way every step and drift the norm of the most
        // populated modes coherently
#pragma unroll
        for (int r = 0; r < R / G; ++r)
#pragma unroll
            for (int k2 = 0; k2 < G; ++k2) {
                const int k = q + G * r + R * k2;
                cpair v = fftreg::cmulw(fftreg::cmulw(y[r * G + k2], pxy), kzp[k]);
                if (pa.has_m) {
                    const float2 a = fftreg::comp_a(v), b = fftreg::comp_b(v);
                    v = fftreg::make_cpair(fftreg::cmix(pa.m[0], a, pa.m[1], b), fftreg::cmix(pa.m[2], a, pa.m[3], b));
                }
                y[r * G + k2] = v;
            }

#pragma unroll
        for (int r = 0; r < R / G; ++r) dft<G, false>(y + r * G); // over k2 -> j (forward)
#pragma unroll
        for (int r = 0; r < R / G; ++r)
#pragma unroll
            for (int jj = 1; jj < G; ++jj) y[r * G + jj] = fftreg::cmulw(y[r * G + jj], tw[(q + G * r) * jj]);
    }

    template <class Buf>
    __device__ static __forceinline__ void mid_store(const cpair (&y)[R], Buf buf, int q, int p2)
    {
#pragma unroll
        for (int r = 0; r < R / G; ++r)
#pragma unroll
            for (int jj = 0; jj < G; ++jj) zat(buf, bix(p2, jj, q + G * r)) = y[r * G + jj];
    }

    template <class Buf>
    __device__ static __forceinline__ void fwd3(cpair (&x)[R], Buf buf, int p, int j)
    {
#pragma unroll
        for (int k1 = 0; k1 < R; ++k1) x[k1] = zat(buf, bix(p, j, k1));
        dft<R, false>(x);
    }
};

// shared memory of one pencil body: PEN pencils of NZ + 1 cells, then W_NZ^e, the kz phase and the
// per-pencil (kx, ky) phase (float2 each)
template <int NZ, int PEN = 16>
__host__ __device__ constexpr size_t pencil_smem_bytes() { return sizeof(cpair) * PEN * (NZ + 1) + sizeof(float2) * (2 * NZ + PEN); }

// OBS: the pass ends a step (no plane pass follows) and also writes, per z, the
// FP64 sums over the tile's 16 pencils of |a|^2, |b|^2 and conj(a) b of the
// z-transformed boundary state: obs[((traj * tiles + tile) * NZ + z) * 4 + k].
// PEN G threads; dyn: pencil_smem_bytes<NZ, PEN>() of shared memory. LP: log2 of nx ny, or 0 where only run time tells.
template <int NZ, bool OBS, int LP = 0, int PEN = 16>
__device__ __forceinline__ void pencil_body(const VBlock &vb, cpair *__restrict__ state, int nx, int lx, int ny,
                                            int cells, int tiles, const GroupParamsF *__restrict__ gp,
                                            const int *__restrict__ tgroup, const float2 *__restrict__ tw_g,
                                            const PencilArgs &pa, double *__restrict__ obs, float inv_out_scale,
                                            const float2 *__restrict__ kin, cpair *dyn)
{
    using Z = ZTile<NZ, PEN>;
    constexpr int R = 16, G = NZ / 16;
    static_assert(!OBS || PEN == 16, "the layout of obs");
    (void)gp; (void)tgroup; (void)lx;
    cpair *buf = dyn;                                           // PEN pencils x NZ
    float2 *tw = reinterpret_cast<float2 *>(dyn + Z::CELLS);    // W_NZ^e, e < NZ
    float2 *kzp = tw + NZ;                                       // kz phase
    float2 *kxyp = kzp + NZ;                                    // (kx, ky) phase x scale, per pencil

    const int t = vb.tid;
    const int traj = vb.bid / tiles;
    const int pen0 = (vb.bid - traj * tiles) * PEN;
    const int plane = LP ? 1 << LP : nx * ny;

    // kinetic phase e^{+i k^2/2 dt frac} (wigner_kernel.cu:137-151) as the product of the per-kz and the
    // per-pencil factors, from the class's table for this kick fraction (fp32_kin_tables); kin == NULL
    // means frac == 0, no kick.
    // The table entries go to shared memory by asynchronous copies, so the state loads below issue at once
    // and no register holds a table value in between.
    const float2 *kt = kin ? kin + (size_t)traj * (NZ + plane) : nullptr;
#pragma unroll
    for (int e = 0; e < NZ; e += PEN * G) {
        copy_async8(tw + e + t, tw_g + e + t);
        if (kt) copy_async8(kzp + e + t, kt + e + t);
        else kzp[e + t] = make_float2(1.f, 0.f);
    }
    if (t < PEN) {
        if (kt) copy_async8(kxyp + t, kt + NZ + pen0 + t);
        else kxyp[t] = make_float2(1.f, 0.f);
    }

    const int p = t % PEN, j = t / PEN;
    cpair *__restrict__ g = state + (size_t)traj * cells + pen0 + p + j * plane;
    cpair x[R];
#pragma unroll
    for (int m = 0; m < R; ++m) x[m] = g[G * m * plane];
    copy_async_wait();
    if (t < PEN) kxyp[t] = make_float2(pa.scale * kxyp[t].x, pa.scale * kxyp[t].y);
    vb.sync();                                                  // tables ready
    Z::inv1(x, buf, tw, p, j);
    vb.sync();

    const int q = t % G, p2 = t / G;
    cpair y[R];
    Z::mid(y, buf, tw, kzp, kxyp[p2], pa, q, p2);
    vb.sync();                                                  // stage-2 reads done
    Z::mid_store(y, buf, q, p2);
    vb.sync();

    Z::fwd3(x, buf, p, j);
    if constexpr (OBS) {
        // the output is out_scale * FFT_z(boundary state); undo the scale for the moments
        vb.sync();                                              // stage-3 reads of buf done
        float4 *sums = reinterpret_cast<float4 *>(buf);
#pragma unroll
        for (int m = 0; m < R; ++m) {
            const float2 a = fftreg::comp_a(x[m]), b = fftreg::comp_b(x[m]);
            const float ax = a.x * inv_out_scale, ay = a.y * inv_out_scale;
            const float bx = b.x * inv_out_scale, by = b.y * inv_out_scale;
            const int z = j + G * m;
            sums[p * NZ + (z ^ (p & 7))] = make_float4(ax * ax + ay * ay, bx * bx + by * by, ax * bx + ay * by,
                                                      ax * by - ay * bx);
        }
        vb.sync();
        const int tile = vb.bid - traj * tiles;
        for (int z = t; z < NZ; z += NZ) {
            KSum s0, s1, s2, s3;
#pragma unroll
            for (int q2 = 0; q2 < 16; ++q2) {
                const float4 u = sums[q2 * NZ + (z ^ (q2 & 7))];
                s0.add(u.x); s1.add(u.y); s2.add(u.z); s3.add(u.w);
            }
            double *o = obs + (((size_t)traj * tiles + tile) * NZ + z) * 4;
            o[0] = s0.value(); o[1] = s1.value(); o[2] = s2.value(); o[3] = s3.value();
        }
    }
#pragma unroll
    for (int m = 0; m < R; ++m) g[G * m * plane] = x[m];
}

} // namespace stepk
