// fused_passes.cu -- the register-resident plane and pencil passes of the FP32 path as standalone
// kernels, one launch per pass and grid class; the bodies are in step_bodies.cuh (each kernel gives its
// body the whole CTA). Same two-pass regrouping of the reference's split step as batched_fp32.cu
// (propagate, programs/bec_wigner_3d.cuda/wigner.cu:178-199) and the same stored representation.
// A steady step of the fast classes runs instead as one launch of the fused step kernel
// (step_kernel.cu); these kernels serve the steps that observe, and the launch-per-pass schedule.
#include <algorithm>

#include "engine.h"
#include "launch.cuh"
#include "step_bodies.cuh"

namespace {

using fftreg::cpair;
using stepk::PencilArgs;
using stepk::VBlock;

// ---------------------------------------------------------------- plane pass, N = 8, 16
template <int N, int MINB>
__global__ void __launch_bounds__(128, MINB) k_plane(cpair *__restrict__ state, int nz, int cells,
                                               const GroupParamsF *__restrict__ gp, const int *__restrict__ tgroup,
                                               const int *__restrict__ tlocal, const StepRef sr)
{
    extern __shared__ cpair tile[];   // plane_tile_cells<N>
    stepk::plane_body<N>(VBlock{(int)threadIdx.x, (int)blockIdx.x, 0, 128}, state, nz, cells, gp, tgroup, tlocal,
                         *sr.step + sr.off, tile);
    advance_step(sr);
}

// ---------------------------------------------------------------- plane pass, 32 x 32, two warps a plane
template <int MINB>
__global__ void __launch_bounds__(64, MINB) k_plane32s(cpair *__restrict__ state, int nz, int cells,
                                                      const GroupParamsF *__restrict__ gp,
                                                      const int *__restrict__ tgroup, const int *__restrict__ tlocal,
                                                      const StepRef sr)
{
    __shared__ cpair tile[stepk::kPlane32Cells];
    stepk::plane32_body(VBlock{(int)threadIdx.x, (int)blockIdx.x, 0, 64}, state, nz, cells, gp, tgroup, tlocal,
                        *sr.step + sr.off, tile);
    advance_step(sr);
}

// ---------------------------------------------------------------- pencil pass
// Pencils per CTA: 16 as the sums of an observing pass are laid out, else 128 threads' worth at nz = 256. Twenty warps an SM
// (96 registers, no spill) come to 87 % of the measured HBM rate at nz = 256: 365 trajectories of 32x32x256 take 0.546 ms,
// 0.596 with 16 pencils and 256 threads (of which only two CTAs fit), 0.614 with swizzled lines and a run-time plane size
// besides; sixteen warps 0.550, twenty-four (80 registers, spilling) 0.652.
template <int NZ, bool OBS>
constexpr int kPen = !OBS && NZ == 256 ? 8 : 16;

template <int NZ, bool OBS, int LP>
__global__ void __launch_bounds__(kPen<NZ, OBS> * NZ / 16, OBS ? 1 : 640 / (kPen<NZ, OBS> * NZ / 16)) k_pencil(cpair *__restrict__ state, int nx, int lx, int ny, int cells,
                                               int tiles, const GroupParamsF *__restrict__ gp,
                                               const int *__restrict__ tgroup, const float2 *__restrict__ tw_g,
                                               PencilArgs pa, double *__restrict__ obs, float inv_out_scale,
                                               const float2 *__restrict__ kin)
{
    extern __shared__ cpair dyn[];
    constexpr int PEN = kPen<NZ, OBS>;
    stepk::pencil_body<NZ, OBS, LP, PEN>(VBlock{(int)threadIdx.x, (int)blockIdx.x, 0, PEN * NZ / 16}, state, nx, lx, ny, cells, tiles,
                                gp, tgroup, tw_g, pa, obs, inv_out_scale, kin, dyn);
}

__global__ void k_kin_tables(float2 *__restrict__ tab, const GroupParamsF *__restrict__ gp,
                             const int *__restrict__ tgroup, int nx, int ny, int nz, int lx, int n_traj, float frac)
{
    const int per = nz + nx * ny;
    const size_t n = (size_t)n_traj * per;
    for (size_t idx = blockIdx.x * (size_t)blockDim.x + threadIdx.x; idx < n; idx += (size_t)gridDim.x * blockDim.x) {
        const int t = (int)(idx / per), i = (int)(idx - (size_t)t * per);
        const GroupParamsF &P = gp[tgroup[t]];
        double turns;
        if (i < nz) {
            const int iz = kidx(i, nz);
            turns = P.kin_z * (double)(iz * iz);
        } else {
            const int pen = i - nz;
            const int ix = kidx(pen & (nx - 1), nx), iy = ny > 1 ? kidx(pen >> lx, ny) : 0;
            turns = P.kin_x * (double)(ix * ix) + P.kin_y * (double)(iy * iy);
        }
        tab[idx] = kin_phase(turns * (double)frac);
    }
}

template <int NZ, bool OBS, int LP>
void launch_pencil_lp(cpair *state, const ClassGeom &c, const GroupParamsF *gp, const int *tgroup, const float2 *tw,
                   const PencilArgs &pa, double *obs, float inv_out_scale, const float2 *kin, cudaStream_t s)
{
    constexpr int PEN = kPen<NZ, OBS>;
    const int tiles = c.nx * c.ny / PEN;
    const size_t smem = stepk::pencil_smem_bytes<NZ, PEN>();
    ensure_smem_limit((const void *)k_pencil<NZ, OBS, LP>, (int)smem);
    k_pencil<NZ, OBS, LP><<<c.n_traj * tiles, PEN * NZ / 16, smem, s>>>(state, c.nx, c.lx, c.ny, c.cells, tiles, gp, tgroup, tw,
                                                         pa, obs, inv_out_scale, kin);
    g_launches++;
}

// square planes with their size known to the compiler
template <int NZ, bool OBS>
void launch_pencil(cpair *state, const ClassGeom &c, const GroupParamsF *gp, const int *tgroup, const float2 *tw,
                   const PencilArgs &pa, double *obs, float inv_out_scale, const float2 *kin, cudaStream_t s)
{
    switch (c.nx * c.ny) {
    case 64: launch_pencil_lp<NZ, OBS, 6>(state, c, gp, tgroup, tw, pa, obs, inv_out_scale, kin, s); break;
    case 256: launch_pencil_lp<NZ, OBS, 8>(state, c, gp, tgroup, tw, pa, obs, inv_out_scale, kin, s); break;
    case 1024: launch_pencil_lp<NZ, OBS, 10>(state, c, gp, tgroup, tw, pa, obs, inv_out_scale, kin, s); break;
    default: launch_pencil_lp<NZ, OBS, 0>(state, c, gp, tgroup, tw, pa, obs, inv_out_scale, kin, s); break;
    }
}

template <int N, int MINB>
void launch_plane(cpair *state, const ClassGeom &c, const GroupParamsF *gp, const int *tgroup, const int *tlocal,
                  const StepRef &sr, cudaStream_t s)
{
    constexpr int W = 32 / N;
    const int planes = c.n_traj * c.nz;
    const size_t smem = sizeof(cpair) * stepk::plane_tile_cells<N>;
    ensure_smem_limit((const void *)k_plane<N, MINB>, (int)smem);
    k_plane<N, MINB><<<planes / (4 * W), 128, smem, s>>>(state, c.nz, c.cells, gp, tgroup, tlocal, sr);
    g_launches++;
}

template <int MINB>
void launch_plane32s(cpair *state, const ClassGeom &c, const GroupParamsF *gp, const int *tgroup, const int *tlocal,
                     const StepRef &sr, cudaStream_t s)
{
    k_plane32s<MINB><<<c.n_traj * c.nz, 64, 0, s>>>(state, c.nz, c.cells, gp, tgroup, tlocal, sr);
    g_launches++;
}

} // namespace

bool fp32_fast_plane_supported(const ClassGeom &c)
{
    if (c.nx != c.ny || (c.nx != 8 && c.nx != 16 && c.nx != 32)) return false;
    const int W = 32 / c.nx;
    return ((long long)c.n_traj * c.nz) % (4 * W) == 0;
}

bool fp32_fast_pencil_supported(const ClassGeom &c)
{
    return (c.nz == 64 || c.nz == 128 || c.nz == 256) && (c.nx * c.ny) % 16 == 0 && c.nx * c.ny >= 16;
}

void fp32_plane_fast(float4 *cells, const ClassGeom &c, const GroupParamsF *gp, const int *tgroup, const int *tlocal,
                     const StepRef &sr, int occupancy, cudaStream_t s)
{
    if (c.n_traj <= 0) return;
    cpair *state = reinterpret_cast<cpair *>(cells);
    // occupancy 0: 16 warps per SM (8x8 / 16x16: 4 CTAs of 128 threads; 32x32: 8 CTAs of 64), no register spill;
    // occupancy 1: 20 warps per SM (5 and 10 CTAs), 96 registers with a small spill
    switch (c.nx) {
    case 8:
        if (occupancy) launch_plane<8, 5>(state, c, gp, tgroup, tlocal, sr, s);
        else launch_plane<8, 4>(state, c, gp, tgroup, tlocal, sr, s);
        break;
    case 16:
        if (occupancy) launch_plane<16, 5>(state, c, gp, tgroup, tlocal, sr, s);
        else launch_plane<16, 4>(state, c, gp, tgroup, tlocal, sr, s);
        break;
    case 32:
        if (occupancy) launch_plane32s<10>(state, c, gp, tgroup, tlocal, sr, s);
        else launch_plane32s<8>(state, c, gp, tgroup, tlocal, sr, s);
        break;
    default: break;
    }
}

void fp32_kin_tables(float2 *tab, const ClassGeom &c, const GroupParamsF *gp, const int *tgroup, float frac,
                     cudaStream_t s)
{
    if (c.n_traj <= 0) return;
    const size_t n = (size_t)c.n_traj * (c.nz + c.nx * c.ny);
    const int blocks = (int)std::min<size_t>((n + 255) / 256, 148 * 16);
    k_kin_tables<<<blocks, 256, 0, s>>>(tab, gp, tgroup, c.nx, c.ny, c.nz, c.lx, c.n_traj, frac);
    g_launches++;
}

void fp32_pencil_fast(float4 *cells, const ClassGeom &c, const GroupParamsF *gp, const int *tgroup,
                      const float2 *tw_full, float frac, float scale, const float2 *m, double *obs,
                      float out_scale, const float2 *kin, cudaStream_t s)
{
    if (c.n_traj <= 0) return;
    cpair *state = reinterpret_cast<cpair *>(cells);
    PencilArgs pa{};
    pa.frac = frac;
    pa.scale = scale;
    pa.has_m = m ? 1 : 0;
    if (m)
        for (int i = 0; i < 4; ++i) pa.m[i] = m[i];
    const float inv = 1.0f / out_scale;
    switch (c.nz) {
    case 64:
        if (obs) launch_pencil<64, true>(state, c, gp, tgroup, tw_full, pa, obs, inv, kin, s);
        else launch_pencil<64, false>(state, c, gp, tgroup, tw_full, pa, nullptr, inv, kin, s);
        break;
    case 128:
        if (obs) launch_pencil<128, true>(state, c, gp, tgroup, tw_full, pa, obs, inv, kin, s);
        else launch_pencil<128, false>(state, c, gp, tgroup, tw_full, pa, nullptr, inv, kin, s);
        break;
    case 256:
        if (obs) launch_pencil<256, true>(state, c, gp, tgroup, tw_full, pa, obs, inv, kin, s);
        else launch_pencil<256, false>(state, c, gp, tgroup, tw_full, pa, nullptr, inv, kin, s);
        break;
    default: break;
    }
}

int fp32_fast_pencil_tiles(const ClassGeom &c) { return c.nx * c.ny / 16; }
