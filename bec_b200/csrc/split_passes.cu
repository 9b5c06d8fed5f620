// split_passes.cu -- the register passes with every line shared by several threads, for classes too small to fill the chip.
//
// The passes of fused_passes.cu give a thread sixteen cells of a line, which is the best use of the issue slots once
// every SM holds sixteen warps. A class of a few trajectories has fewer warps than that in all, and a pass then takes as
// long as one thread's sixteen cells: transforms, Philox draws and physics one after the other. Here a line belongs to S
// threads of different warps (four, or two for 8-point lines) holding the elements q + S j each: S times the threads, a
// quarter of the work in each. A thread transforms its own elements, exchanges the results through shared memory and
// computes the last two levels (one) of butterflies for the outputs q + S j, which are again the elements that the next
// transform wants from it. The butterflies are those of fftreg::dft, decimation in time, in the same order, so every cell
// gets the same bits as in the other kernels.
//
// Measured, microseconds per step of a captured run, sixteen cells per thread -> four: 16x16x128 with one trajectory
// 11.8 -> 6.2, with 4 12.7 -> 8.8, with 16 17.0 -> 15.2 (split plane pass alone), with 64 40.6 -> 41.5; 8x8x64 with 8
// 8.5 -> 5.7, with 256 22.4 -> 23.2; the pencil pass of a 32x128 slice 3.8 -> 2.5. The autotuner times both for classes of
// up to kSplitCells cells (bec_api.cpp).
#include <algorithm>

#include "engine.h"
#include "launch.cuh"
#include "step_bodies.cuh"

namespace {

using fftreg::cpair;
using stepk::PencilArgs;
using stepk::ld_cg;

// x0 = e + W_N^K o, x1 = e - W_N^K o as fftreg::dft computes them
template <int K, int N, bool INV>
__device__ __forceinline__ void butterfly(cpair &x0, cpair &x1, cpair e, cpair o)
{
    if constexpr (K == 0) {
        x0 = fftreg::add(e, o);
        x1 = fftreg::sub(e, o);
    } else if constexpr (4 * K == N) {
        fftreg::bfly_i<INV>(x0, x1, e, o);
    } else {
        fftreg::bfly_w<K, N, INV>(x0, x1, e, o);
    }
}

// the outputs q + S j of an N-point transform from the S sub-transforms d[r][k] (r: n mod S) in ex[(r * N/S + k) * lanes + lane]
template <int N, bool INV, int S, int Q, int KK>
__device__ __forceinline__ void combine_one(cpair *v, const cpair *ex, int lanes)
{
    constexpr int E = N / S, K = Q + S * KK;
    if constexpr (S == 2) {
        butterfly<K, N, INV>(v[KK], v[KK + E / 2], ex[K * lanes], ex[(E + K) * lanes]);
    } else {
        cpair e0, e1, o0, o1;
        butterfly<K, N / 2, INV>(e0, e1, ex[K * lanes], ex[(2 * E + K) * lanes]);
        butterfly<K, N / 2, INV>(o0, o1, ex[(E + K) * lanes], ex[(3 * E + K) * lanes]);
        butterfly<K, N, INV>(v[KK], v[KK + E / 2], e0, o0);
        butterfly<K + E, N, INV>(v[KK + E / 4], v[KK + 3 * E / 4], e1, o1);
    }
}
template <int N, bool INV, int S, int Q, int... KK>
__device__ __forceinline__ void combine_all(cpair *v, const cpair *ex, int lanes, std::integer_sequence<int, KK...>)
{
    (combine_one<N, INV, S, Q, KK>(v, ex, lanes), ...);
}

// v[j] = x[q + S j] -> X[q + S j]; ex: exchange slots of N x lanes cells (this thread's lane already added)
template <int N, bool INV, int S, class Sync>
__device__ __forceinline__ void line(cpair *v, cpair *ex, int lanes, int q, Sync sync)
{
    constexpr int E = N / S;
    fftreg::dft<E, INV>(v);
    if constexpr (S > 1) {
#pragma unroll
        for (int k = 0; k < E; ++k) ex[(q * E + k) * lanes] = v[k];
        sync();
        using Seq = std::make_integer_sequence<int, E / S>;
        // q is the same for every thread of a warp
        if constexpr (S == 2) {
            if (q == 0) combine_all<N, INV, 2, 0>(v, ex, lanes, Seq{});
            else combine_all<N, INV, 2, 1>(v, ex, lanes, Seq{});
        } else {
            if (q == 0) combine_all<N, INV, 4, 0>(v, ex, lanes, Seq{});
            else if (q == 1) combine_all<N, INV, 4, 1>(v, ex, lanes, Seq{});
            else if (q == 2) combine_all<N, INV, 4, 2>(v, ex, lanes, Seq{});
            else combine_all<N, INV, 4, 3>(v, ex, lanes, Seq{});
        }
    }
}

// ---------------------------------------------------------------- plane pass, N = 8, 16
// 32 S threads per 32 / N planes: warp q, lane = column, then row, of its plane.
template <int N>
constexpr int kSplit = N / 4;        // threads per line: four elements each

template <int N>
__global__ void __launch_bounds__(32 * kSplit<N>) k_plane_split(cpair *__restrict__ state, int nz, int cells,
                                                                  const GroupParamsF *__restrict__ gp,
                                                                  const int *__restrict__ tgroup,
                                                                  const int *__restrict__ tlocal, const StepRef sr)
{
    constexpr int S = kSplit<N>, E = 4, W = 32 / N, PLANE = N * N;
    constexpr int LD = N + 1;
    __shared__ cpair tile[32 * LD], ex[2][32 * N];
    const int q = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int wp = lane / N, c = lane % N;
    const int plane_id = blockIdx.x * W + wp;
    const int traj = plane_id / nz, z = plane_id - traj * nz;
    cpair *__restrict__ g = state + (size_t)traj * cells + (size_t)z * PLANE;
    cpair *s = tile + wp * (N * LD);
    auto sync = []() { __syncthreads(); };
    const GroupParamsF P = gp[tgroup[traj]];
    wait_predecessor();
    allow_successor();
    const uint32_t step = *sr.step + sr.off;

    cpair v[E];
#pragma unroll
    for (int j = 0; j < E; ++j) v[j] = ld_cg(g + (q + S * j) * N + c);
    line<N, false, S>(v, ex[0] + lane, 32, q, sync);
#pragma unroll
    for (int j = 0; j < E; ++j) s[(q + S * j) * LD + c] = v[j];
    __syncthreads();
#pragma unroll
    for (int j = 0; j < E; ++j) v[j] = s[c * LD + q + S * j];
    line<N, false, S>(v, ex[1] + lane, 32, q, sync);
    {
        // this thread's cells x = q + S j of row y = c (plane_body's arithmetic)
        const float Y = fmaf(P.dy, (float)c, -P.ymax);
        const float Z = fmaf(P.dz, (float)z, -P.zmax);
        const float base = fmaf(Y, Y, (Z * Z) * P.inv_lambda2);
        const CellConsts K = cell_consts(P);
        cpair v0[E];
#pragma unroll
        for (int j = 0; j < E; ++j) {
            const float X = fmaf(P.dx, (float)(q + S * j), -P.xmax);
            v0[j] = v[j];
            v[j] = nonlinear_cell(v0[j], 0.5f * fmaf(X, X, base), K);
        }
        if (P.noise)
            loss_noise_cell4(v, v0, K, philox_keys(P.seed_lo, P.seed_hi), (uint32_t)tlocal[traj], step,
                             (uint32_t)(z * PLANE + c * N + q), S);
    }
    line<N, true, S>(v, ex[0] + lane, 32, q, sync);
#pragma unroll
    for (int j = 0; j < E; ++j) s[c * LD + q + S * j] = v[j];
    __syncthreads();
#pragma unroll
    for (int j = 0; j < E; ++j) v[j] = s[(q + S * j) * LD + c];
    line<N, true, S>(v, ex[1] + lane, 32, q, sync);
#pragma unroll
    for (int j = 0; j < E; ++j) g[(q + S * j) * N + c] = v[j];
    advance_step(sr);
}

// ---------------------------------------------------------------- pencil pass
// ZTile's stages (step_bodies.cuh) on PEN pencils by 4 PEN G threads (nz = 16 G), four elements each: thread group q of
// PEN G threads holds m = q + 4 i of the 16-point transforms over m, and of the G-point ones over j: j = q + 4 i (G = 16),
// one of the two transforms and a parity (G = 8), one transform (G = 4).
template <int NZ>
struct PencilSplit {
    static constexpr int G = NZ / 16, PEN = G == 4 ? 8 : 4, LANES = PEN * G, THREADS = 4 * LANES;
};

template <int NZ>
__global__ void __launch_bounds__(PencilSplit<NZ>::THREADS) k_pencil_split(cpair *__restrict__ state, int plane, int cells,
                                                                         int tiles, const float2 *__restrict__ tw_g,
                                                                         PencilArgs pa, const float2 *__restrict__ kin)
{
    using C = PencilSplit<NZ>;
    constexpr int G = C::G, PEN = C::PEN, LANES = C::LANES, R = 16;
    constexpr int SG = G == 16 ? 4 : G == 8 ? 2 : 1;      // threads per G-point line
    __shared__ cpair buf[PEN * (NZ + 1)], ex[PEN * NZ];
    __shared__ float2 tw[NZ], kzp[NZ];
    const int t = threadIdx.x, q = t / LANES, u = t % LANES;
    const int traj = blockIdx.x / tiles, pen0 = (blockIdx.x - traj * tiles) * PEN;
    auto sync = []() { __syncthreads(); };
    auto bix = [](int p, int j, int k1) { return p * (NZ + 1) + j * R + k1; };
    const float2 *kt = kin ? kin + (size_t)traj * (NZ + plane) : nullptr;
    for (int e = t; e < NZ; e += C::THREADS) {
        tw[e] = tw_g[e];
        kzp[e] = kt ? kt[e] : make_float2(1.f, 0.f);
    }
    const int p = u % PEN, j = u / PEN;                   // stages 1 and 3
    const int kq = u % G, p2 = u / G;                     // stage 2: k1 = kq + G r
    float2 pxy = kt ? kt[NZ + pen0 + p2] : make_float2(1.f, 0.f);
    pxy = make_float2(pa.scale * pxy.x, pa.scale * pxy.y);
    cpair *__restrict__ g = state + (size_t)traj * cells + pen0 + p;
    wait_predecessor();
    allow_successor();

    cpair x[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) x[i] = ld_cg(g + (size_t)(j + G * (q + 4 * i)) * plane);
    line<16, true, 4>(x, ex + u, LANES, q, sync);         // over m -> k1 = q + 4 i
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const int k1 = q + 4 * i;
        if (k1 > 0) {
            const float2 w = tw[j * k1];
            x[i] = fftreg::cmulw(x[i], make_float2(w.x, -w.y));       // W^{-j k1}
        }
        buf[bix(p, j, k1)] = x[i];
    }
    __syncthreads();
    // over j -> k2 (k = k1 + 16 k2): h: this thread's place in its line, r: which of the 16 / G lines of kq
    const int h = G == 16 ? q : G == 8 ? q & 1 : 0, r = G == 16 ? 0 : G == 8 ? q >> 1 : q;
    const int k1 = kq + G * r;
    cpair y[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) y[i] = buf[bix(p2, h + SG * i, k1)];
    // each G-point line exchanges in its own slots
    cpair *const ex2 = ex + (G == 8 ? r * G * LANES : 0) + u;
    line<G, true, SG>(y, ex2, LANES, h, sync);
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const int k = k1 + R * (h + SG * i);
        cpair v = fftreg::cmulw(fftreg::cmulw(y[i], pxy), kzp[k]);
        if (pa.has_m) {
            const float2 a = fftreg::comp_a(v), b = fftreg::comp_b(v);
            v = fftreg::make_cpair(fftreg::cmix(pa.m[0], a, pa.m[1], b), fftreg::cmix(pa.m[2], a, pa.m[3], b));
        }
        y[i] = v;
    }
    __syncthreads();                                      // the exchange slots are free again
    line<G, false, SG>(y, ex2, LANES, h, sync);           // over k2 -> j
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const int jj = h + SG * i;
        if (jj > 0) y[i] = fftreg::cmulw(y[i], tw[k1 * jj]);
        buf[bix(p2, jj, k1)] = y[i];
    }
    __syncthreads();
#pragma unroll
    for (int i = 0; i < 4; ++i) x[i] = buf[bix(p, j, q + 4 * i)];
    line<16, false, 4>(x, ex + u, LANES, q, sync);        // over k1 -> m = q + 4 i
#pragma unroll
    for (int i = 0; i < 4; ++i) g[(size_t)(j + G * (q + 4 * i)) * plane] = x[i];
}

template <int N>
void launch_plane(float4 *state, const ClassGeom &c, const GroupParamsF *gp, const int *tgroup, const int *tlocal,
                  const StepRef &sr, cudaStream_t s)
{
    launch_after(k_plane_split<N>, c.n_traj * c.nz / (32 / N), 32 * kSplit<N>, 0, s, reinterpret_cast<cpair *>(state), c.nz,
                 c.cells, gp, tgroup, tlocal, sr);
}

template <int NZ>
void launch_pencil(float4 *state, const ClassGeom &c, const float2 *tw, const PencilArgs &pa, const float2 *kin, cudaStream_t s)
{
    const int tiles = c.nx * c.ny / PencilSplit<NZ>::PEN;
    launch_after(k_pencil_split<NZ>, c.n_traj * tiles, PencilSplit<NZ>::THREADS, 0, s, reinterpret_cast<cpair *>(state),
                 c.nx * c.ny, c.cells, tiles, tw, pa, kin);
}

} // namespace

bool fp32_plane_split_supported(const ClassGeom &c)
{
    return c.nx == c.ny && (c.nx == 8 || c.nx == 16) && ((long long)c.n_traj * c.nz) % (32 / c.nx) == 0;
}

void fp32_plane_split(float4 *state, const ClassGeom &c, const GroupParamsF *gp, const int *tgroup, const int *tlocal,
                      const StepRef &sr, cudaStream_t s)
{
    if (c.n_traj <= 0) return;
    if (c.nx == 8) launch_plane<8>(state, c, gp, tgroup, tlocal, sr, s);
    else launch_plane<16>(state, c, gp, tgroup, tlocal, sr, s);
}

void fp32_pencil_split(float4 *state, const ClassGeom &c, const float2 *tw_full, float scale, const float2 *m,
                       const float2 *kin, cudaStream_t s)
{
    if (c.n_traj <= 0) return;
    PencilArgs pa{};
    pa.scale = scale;
    pa.has_m = m ? 1 : 0;
    for (int i = 0; m && i < 4; ++i) pa.m[i] = m[i];
    switch (c.nz) {
    case 64: launch_pencil<64>(state, c, tw_full, pa, kin, s); break;
    case 128: launch_pencil<128>(state, c, tw_full, pa, kin, s); break;
    case 256: launch_pencil<256>(state, c, tw_full, pa, kin, s); break;
    default: break;
    }
}
