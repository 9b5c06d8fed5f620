// nn.cu -- the warm-start network: a small MLP trained and evaluated on the GPU.
//
// No counterpart in the reference. The network maps an ensemble's parameters
// to the coefficients of a correction to the Thomas-Fermi profile; its output
// only seeds the imaginary-time ground-state loop (bec_ground_state_batch),
// which alone decides convergence.
//
// Layers are Y = act(X W^T + b) (W is [out x in], row-major, as a linear layer),
// tanh on hidden layers, identity on the last. GEMMs run on the 5th-generation
// tensor cores (tcgen05.mma, BF16 operands from shared memory, FP32 accumulator in
// tensor memory) with split operands: every FP32 operand x is held as two BF16
// values, hi = bf16(x) and lo = bf16(x - hi), and a product is accumulated as
// hi*hi + hi*lo + lo*hi (three MMAs), about 16 significant bits per operand instead
// of 8. Single BF16 products limited the trained network (its loss stalled at the
// BF16 rounding level and its warm starts needed 1.6x the steps of the same
// network trained in FP32). Master weights, Adam moments, activations' pre-images
// and gradients are FP32.
//
// What bounds it: latency. A training step of the 256-wide network at batch 256 is
// 0.23 GFLOP and 4 MB, under a microsecond of either; it is a chain of dependent
// GEMMs. So a step is one launch per link of that chain (four forward, four backward)
// and nothing else: every GEMM's epilogue applies the bias, the activation or its
// derivative, the loss or Adam, and writes its result as the split operands that the
// next GEMMs read, plain and transposed, already in the tiles' shared-memory layout; a
// layer's weight gradient, bias gradient and input gradient share a launch, and the
// next minibatch is gathered beside the first layer's. A launch sets itself up (barriers, tensor memory) while the one
// before it finishes (launch.cuh), and an epilogue fetches what it reads while the tile's operands load. Weights' operands alternate
// between two buffers, so that a launch can update a layer that another tile of it
// still reads. 55 us a step (batch 256, 400 steps with the set-up) against 314 us with one kernel per
// operation.
#include <algorithm>
#include <cstdlib>
#include <cmath>
#include <cstring>
#include <random>
#include <string>
#include <vector>

#include <cuda_bf16.h>

#include "engine.h"
#include "launch.cuh"
#include "mlp_tiles.h"

namespace {

typedef __nv_bfloat16 bf16;

// ---------------------------------------------------------------- operands
// A split matrix [R x K] (R, K multiples of 64) as its hi and its lo values, each in the K-major canonical order of
// the tensor core without swizzle: 64 columns after another, 8-row groups of 1024 bytes, in a group 16-byte chunks of 8
// columns (128 bytes apart) of 8 rows (16 bytes apart). The rows r0 .. r0 + T of a 64-column block are then T * 128
// contiguous bytes: one bulk copy brings an operand tile to shared memory.
struct Split {
    bf16 *hi, *lo;
};
__host__ __device__ __forceinline__ size_t blk(int R, int r, int k)
{
    return ((size_t)(k >> 6) * (R >> 3) + (r >> 3)) * 512 + ((k >> 3) & 7) * 64 + (r & 7) * 8 + (k & 7);
}

// the split of an FP32 value into hi = bf16(v) and lo = bf16(v - hi)
__device__ __forceinline__ void split_bf16(float v, bf16 &hi, bf16 &lo)
{
    hi = __float2bfloat16(v);
    lo = __float2bfloat16(v - __bfloat162float(hi));
}

// ---------------------------------------------------------------- GEMM on the 5th-generation tensor cores
// C[M x N] = A[M x K] * B[N x K]^T with A = A_hi + A_lo, B = B_hi + B_lo; M, N, K multiples of 64. One CTA of 256
// threads per 64 x tn tile of C (tn = 16, 32, 64 or 128: the narrowest that keeps a launch within one CTA per SM, so that
// a 256 x 256 product spreads over 64 SMs). The FP32 accumulator lives in tensor memory (row i of the tile in lane
// 32 (i / 16) + i % 16). K runs in 64-wide stages through a ring of four: one thread issues the bulk copies of a stage's
// four tiles onto an mbarrier, and, as each stage lands, per 16-wide K step the three tcgen05.mma (M 64, N tn, K 16, BF16
// in, FP32 accumulate) lo*hi, hi*lo, hi*hi; tcgen05.commit arrives on the stage's second mbarrier when they are done.
// Every wait is bounded. What a link reads besides the operand that the one before it has just written (the weights, the
// epilogue's inputs) it fetches before it waits for that one (GemmJob::early).
//
// A link of the 256-wide chain at batch 256 is the arrival of its operands, then the last MMAs, then the epilogue. With
// 128 x 16 tiles (144 KB of operands a CTA, 3.4 us to arrive; 0.6 us of MMAs; 1.9 us of tanh or 3.6 us of Adam in sixteen
// columns a thread) a training step took 65 us of launches; with 64 x 16 tiles, four columns a thread and early fetches 45.
//
// The epilogue reads the accumulator with tcgen05.ld: warps w and w + 4 own the 16 rows of lanes 32 w, eight columns each
// in turn, of which the idle upper lanes take half: EC columns a thread.
constexpr int kThreads = 256;
constexpr int GM = kTileRows, GK = 64, GSTAGES = 4;
constexpr int kTileA = GM * GK * 2;                           // 8 KiB each of hi and lo
__host__ __device__ constexpr int stage_bytes(int tn) { return 2 * (kTileA + tn * GK * 2); }
__host__ __device__ constexpr int gemm_smem(int tn) { return GSTAGES * stage_bytes(tn) + 128; }   // + mbarriers and TMEM slot

enum Epilogue {
    EPI_TANH,       // y = tanh(acc + bias): f32 and operands
    EPI_LINEAR,     // y = acc + bias
    EPI_LOSS,       // the output layer in training: y = acc + bias, dz = 2 (y - t) / (valid * real_cols), loss
    EPI_DX,         // dz = acc (1 - y^2): f32 and operands
    EPI_GRAD,       // the weight gradient: f32
    EPI_ADAM        // the weight gradient applied at once: master weight, moments, operands
};

struct AdamArgs {
    float lr, c1, c2;           // step size, 1 - beta1^t, 1 - beta2^t
};
struct GemmJob {
    const bf16 *Ahi, *Alo, *Bhi, *Blo;   // operands; Ahi == nullptr: no job
    int Ra, Rb;                 // rows of the operand matrices
    int M, N, K, tn, ctas;
    int epi;
    bool early;                 // B and the epilogue's inputs are older than the launch before this one
    const float *bias;          // [N]
    float *f32;                 // row-major [M x N] result (y, dz, gradient), may be NULL
    int f32_ld, f32_rows, f32_cols;      // ... stored for rows and columns below these
    Split out, outT;            // [M x N] and [N x M] operands, may be NULL
    const float *y;             // EPI_DX: activation [M x N]
    const float *tgt;           // EPI_LOSS: targets [M x N]
    int valid, real_cols;
    float *loss;
    float *w, *m, *v;           // EPI_ADAM: master weights and moments, [M x N]
    AdamArgs adam;
};
struct BiasJob {                // db[c] = sum_r dz[r][c], rows in order
    const float *dz;
    int rows, cols, ctas;
    float *g;                   // gradient out, or NULL: Adam on w, m, v
    float *w, *m, *v;
    AdamArgs adam;
};
struct GatherJob {              // a minibatch: rows idx[r] (or r) of x, zero rows past valid and columns past in_real
    const float *x, *t;
    const int *idx;
    int rows, valid, in_real, in, out_real, out, ctas;
    Split X, XT;                // [rows x in], [in x rows]; XT and tgt may be NULL
    float *tgt;                 // [rows x out]
};
struct Jobs {
    GemmJob gemm[2];
    BiasJob bias;
    GatherJob gather;
    int *err;
    const int *never;
    int stall;
    unsigned long long limit_ns;
};

__device__ __forceinline__ float adam_update(float &w, float &m, float &v, float gi, const AdamArgs &a)
{
    const float b1 = 0.9f, b2 = 0.999f, eps = 1e-8f;
    const float mi = b1 * m + (1.0f - b1) * gi;
    const float vi = b2 * v + (1.0f - b2) * gi * gi;
    m = mi;
    v = vi;
    // (a zero moment changes nothing, and zeros, the padding's, would take the slow paths of division and square root:
    // they made the epilogue of a layer of six inputs, padded to 64, 6.2 us long)
    if (mi == 0.0f) return w;
    w -= a.lr * (mi / a.c1) / (sqrtf(vi / a.c2) + eps);
    return w;
}

__device__ __forceinline__ uint32_t saddr(const void *p) { return (uint32_t)__cvta_generic_to_shared(p); }

// shared-memory matrix descriptor: start address >> 4 (bits 0-13), leading byte offset >> 4 (16-29) = the K-chunk
// stride 128 B, stride byte offset >> 4 (32-45) = the 8-row group stride 1024 B, descriptor version 1 (46-47),
// no swizzle (61-63 = 0)
__device__ __forceinline__ uint64_t kmajor_desc(uint32_t addr)
{
    return (uint64_t)((addr >> 4) & 0x3FFFu) | ((uint64_t)(128 >> 4) << 16) | ((uint64_t)(1024 >> 4) << 32) |
           (1ull << 46);
}

__device__ __forceinline__ unsigned long long now_ns()
{
    unsigned long long t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    return t;
}

__device__ __forceinline__ bool mbar_test(uint32_t bar, uint32_t parity)
{
    uint32_t done;
    asm volatile("{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
                 "selp.u32 %0, 1, 0, p;\n\t}"
                 : "=r"(done)
                 : "r"(bar), "r"(parity)
                 : "memory");
    return done != 0;
}

__device__ __forceinline__ bool mbar_wait_bounded(uint32_t bar, uint32_t parity, unsigned long long limit_ns)
{
    if (mbar_test(bar, parity)) return true;
    const unsigned long long t0 = now_ns();
    while (!mbar_test(bar, parity))
        if (now_ns() - t0 > limit_ns) return false;
    return true;
}

// a wait for a flag that nothing sets (fault injection): false after limit_ns
__device__ __noinline__ bool wait_flag(const int *flag, unsigned long long limit_ns)
{
    const unsigned long long t0 = now_ns();
    while (*(volatile const int *)flag == 0) {
        __nanosleep(1000);
        if (now_ns() - t0 > limit_ns) return false;
    }
    return true;
}

// one tcgen05.mma of the tile: D (+)= A B^T from the shared-memory descriptors; accumulate = 0 overwrites D
__device__ __forceinline__ void mma_f16(uint32_t tmem, uint64_t ad, uint64_t bd, uint32_t idesc, uint32_t accumulate)
{
    asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
                 "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}"
                 ::"r"(tmem), "l"(ad), "l"(bd), "r"(idesc), "r"(accumulate)
                 : "memory");
}

__device__ __forceinline__ void bulk_load(uint32_t dst, const void *src, uint32_t bytes, uint32_t bar)
{
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
                 ::"r"(dst), "l"(src), "r"(bytes), "r"(bar)
                 : "memory");
}

// EC consecutive columns of one row, as operands: half a chunk of the plain matrix, and of the transposed one
// a 2-byte value per column (8 rows of consecutive lanes make a chunk)
constexpr int EC = 4;
__device__ __forceinline__ void store_operands(const GemmJob &J, int row, int col, const float (&o)[EC])
{
    __align__(8) bf16 hi[EC], lo[EC];
#pragma unroll
    for (int q = 0; q < EC; ++q) split_bf16(o[q], hi[q], lo[q]);
    if (J.out.hi) {
        const size_t at = blk(J.M, row, col);
        *reinterpret_cast<uint2 *>(J.out.hi + at) = *reinterpret_cast<const uint2 *>(hi);
        *reinterpret_cast<uint2 *>(J.out.lo + at) = *reinterpret_cast<const uint2 *>(lo);
    }
    if (J.outT.hi) {
#pragma unroll
        for (int q = 0; q < EC; ++q) {
            const size_t at = blk(J.N, col + q, row);
            J.outT.hi[at] = hi[q];
            J.outT.lo[at] = lo[q];
        }
    }
}

__device__ __forceinline__ void load_cols(float (&o)[EC], const float *p)
{
#pragma unroll
    for (int q = 0; q < EC / 4; ++q) {
        const float4 v = reinterpret_cast<const float4 *>(p)[q];
        o[4 * q] = v.x; o[4 * q + 1] = v.y; o[4 * q + 2] = v.z; o[4 * q + 3] = v.w;
    }
}
__device__ __forceinline__ void store_cols(float *p, const float (&o)[EC])
{
#pragma unroll
    for (int q = 0; q < EC / 4; ++q) reinterpret_cast<float4 *>(p)[q] = make_float4(o[4 * q], o[4 * q + 1], o[4 * q + 2], o[4 * q + 3]);
}

// what the epilogue reads beside the accumulator: the thread's first EC columns are fetched while the tile's operands load
struct Aux {
    float a[EC], b[EC], c[EC];
};
__device__ __forceinline__ void load_aux(const GemmJob &J, Aux &x, int row, int col)
{
    const size_t at = (size_t)row * J.N + col;
    if (J.epi <= EPI_LOSS) load_cols(x.a, J.bias + col);
    if (J.epi == EPI_LOSS) load_cols(x.b, J.tgt + at);
    if (J.epi == EPI_DX) load_cols(x.a, J.y + at);
    if (J.epi == EPI_ADAM) {
        load_cols(x.a, J.w + at);
        load_cols(x.b, J.m + at);
        load_cols(x.c, J.v + at);
    }
}

// row's EC accumulator columns from col on; returns the row's share of the loss (EPI_LOSS)
__device__ __forceinline__ float epilogue(const GemmJob &J, int row, int col, float (&o)[EC], Aux &x)
{
    float l = 0.0f;
    const size_t at = (size_t)row * J.N + col;
    if (J.epi <= EPI_LOSS) {
#pragma unroll
        for (int q = 0; q < EC; ++q) o[q] += x.a[q];
    }
    if (J.epi == EPI_TANH) {
#pragma unroll
        for (int q = 0; q < EC; ++q) o[q] = tanhf(o[q]);
    } else if (J.epi == EPI_LOSS) {
        // the padding columns of y and t are zero, padding rows get no gradient
        const float s = 2.0f / ((float)J.valid * J.real_cols);
#pragma unroll
        for (int q = 0; q < EC; ++q) {
            const float d = row < J.valid ? o[q] - x.b[q] : 0.0f;
            l += d * d;
            o[q] = s * d;
        }
    } else if (J.epi == EPI_DX) {
#pragma unroll
        for (int q = 0; q < EC; ++q) o[q] *= 1.0f - x.a[q] * x.a[q];
    } else if (J.epi == EPI_ADAM) {
#pragma unroll
        for (int q = 0; q < EC; ++q) o[q] = adam_update(x.a[q], x.b[q], x.c[q], o[q], J.adam);
        store_cols(J.w + at, x.a);
        store_cols(J.m + at, x.b);
        store_cols(J.v + at, x.c);
    }
    if (J.f32 && row < J.f32_rows) {
        float *dst = J.f32 + (size_t)row * J.f32_ld + col;
        if (col + EC <= J.f32_cols && (J.f32_ld & 3) == 0) {
            store_cols(dst, o);
        } else {
            for (int q = 0; q < EC; ++q)
                if (col + q < J.f32_cols) dst[q] = o[q];
        }
    }
    store_operands(J, row, col, o);
    return l;
}

__device__ void gemm_tile(const GemmJob &J, const Jobs &all, int tile, unsigned char *sm)
{
    const int tn = J.tn, tiles_n = J.N / tn, sbytes = stage_bytes(tn);
    const int t = threadIdx.x, warp = t >> 5;
    const int m0 = tile / tiles_n * GM, n0 = tile % tiles_n * tn;
    const int nk = J.K / GK;
    // stage g at g * sbytes: A_hi (64 rows x 64 K), A_lo, B_hi (tn rows x 64 K), B_lo; then full and done barriers
    const uint32_t full = saddr(sm + GSTAGES * sbytes), done = full + 8 * GSTAGES;
    uint32_t *tslot = reinterpret_cast<uint32_t *>(sm + GSTAGES * sbytes + 16 * GSTAGES);

    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], 128;" ::"r"(saddr(tslot)) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    if (t == 0) {
        for (int g = 0; g < 2 * GSTAGES; ++g)
            asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(full + 8 * g) : "memory");
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem = *tslot;

    // this thread's row and first columns in the tile
    const int lr = (warp & 3) * 16 + (t & 15), c0 = (warp >> 2) * 2 * EC + ((t >> 4) & 1) * EC;
    const uint32_t ab = GM * GK * 2, bb = tn * GK * 2;
    auto load_b = [&](int kb) {
        const uint32_t dst = saddr(sm + (kb % GSTAGES) * sbytes) + 2 * kTileA, bar = full + 8 * (kb % GSTAGES);
        asm volatile("mbarrier.expect_tx.relaxed.cta.shared::cta.b64 [%0], %1;" ::"r"(bar), "r"(2 * bb) : "memory");
        const size_t b0 = blk(J.Rb, n0, kb * GK);
        bulk_load(dst, J.Bhi + b0, bb, bar);
        bulk_load(dst + bb, J.Blo + b0, bb, bar);
    };
    auto load_a = [&](int kb) {       // the stage's one arrival
        const uint32_t dst = saddr(sm + (kb % GSTAGES) * sbytes), bar = full + 8 * (kb % GSTAGES);
        asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(2 * ab) : "memory");
        const size_t a0 = blk(J.Ra, m0, kb * GK);
        bulk_load(dst, J.Ahi + a0, ab, bar);
        bulk_load(dst + kTileA, J.Alo + a0, ab, bar);
    };
    const int first = min(GSTAGES, nk);
    Aux x;
    if (J.early) {
        if (t == 0)
            for (int kb = 0; kb < first; ++kb) load_b(kb);
        load_aux(J, x, m0 + lr, n0 + c0);
    }
    wait_predecessor();
    allow_successor();
    if (!J.early) load_aux(J, x, m0 + lr, n0 + c0);
    bool ok = true;
    if (t == 0) {
        // instruction descriptor, kind::f16: D F32 (bits 4-5 = 1), A and B BF16 (bits 7-9, 10-12 = 1), both K-major,
        // N >> 3 at bits 17-22, M >> 4 at bits 24-28
        const uint32_t idesc = (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(tn >> 3) << 17) | ((uint32_t)(GM >> 4) << 24);
        for (int kb = 0; kb < first; ++kb) {
            if (!J.early) load_b(kb);
            load_a(kb);
        }
        auto landed = [&](int kb) { return mbar_wait_bounded(full + 8 * (kb % GSTAGES), (kb / GSTAGES) & 1, all.limit_ns); };
        auto multiplied = [&](int kb) { return mbar_wait_bounded(done + 8 * (kb % GSTAGES), (kb / GSTAGES) & 1, all.limit_ns); };
        int loaded = first, waited = 0, issued = 0;
        for (int kb = 0; kb < nk && ok; ++kb) {
            ok = landed(kb);
            // stall (fault injection): the first stage also waits for a flag that nothing sets
            if (ok) ++waited;
            if (ok && all.stall && kb == 0) ok = wait_flag(all.never, all.limit_ns);
            if (!ok) break;
            const uint32_t as = saddr(sm + (kb % GSTAGES) * sbytes), als = as + kTileA, bs = als + kTileA, bls = bs + tn * GK * 2;
#pragma unroll
            for (int kk = 0; kk < GK / 16; ++kk) {
                const uint64_t ad = kmajor_desc(as + 256 * kk), bd = kmajor_desc(bs + 256 * kk);
                const uint64_t ald = kmajor_desc(als + 256 * kk), bld = kmajor_desc(bls + 256 * kk);
                // the small products first; only the very first MMA of the tile starts D afresh
                mma_f16(tmem, ald, bd, idesc, (kb > 0 || kk > 0) ? 1u : 0u);
                mma_f16(tmem, ad, bld, idesc, 1u);
                mma_f16(tmem, ad, bd, idesc, 1u);
            }
            asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];"
                         ::"r"(done + 8 * (kb % GSTAGES)) : "memory");
            ++issued;
            // refill the stage before this one once its MMAs have read it
            if (kb >= 1 && loaded < nk) {
                ok = multiplied(kb - 1);
                if (ok) {
                    load_b(loaded);
                    load_a(loaded++);
                }
            }
        }
        if (ok) ok = multiplied(nk - 1);
        if (!ok) {
            // a wait that ran out: report it and give the copies and MMAs in flight once more the limit
            atomicExch(all.err, 1);
            for (int kb = waited; kb < loaded; ++kb) landed(kb);
            if (issued) multiplied(issued - 1);
        }
    }
    const bool failed = __syncthreads_or(!ok);
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    if (!failed) {
        float l = 0.0f;
        for (int cb = 0; cb < tn; cb += 4 * EC) {
            uint32_t r[2 * EC];
            asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
                         : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7])
                         : "r"(tmem + ((uint32_t)((warp & 3) * 32) << 16) + (uint32_t)(cb + (warp >> 2) * 2 * EC)));
            asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
            float o[EC];
#pragma unroll
            for (int q = 0; q < EC; ++q) {
                const uint32_t upper = __shfl_sync(0xffffffffu, r[EC + q], t & 15);
                o[q] = __uint_as_float(t & 16 ? upper : r[q]);
            }
            if (cb > 0) load_aux(J, x, m0 + lr, n0 + cb + c0);
            l += epilogue(J, m0 + lr, n0 + cb + c0, o, x);
        }
        if (J.epi == EPI_LOSS) {
            for (int off = 16; off > 0; off >>= 1) l += __shfl_down_sync(0xffffffffu, l, off);
            if ((t & 31) == 0) atomicAdd(J.loss, l / ((float)J.valid * J.real_cols));
        }
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    if (warp == 0) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, 128;" ::"r"(tmem) : "memory");
}

// 32 columns per CTA, 128 rows at a time through shared memory, so that the loads overlap while the sum keeps its order
constexpr int kBiasCols = 32, kBiasRows = 128;
__device__ __forceinline__ void bias_columns(const BiasJob &J, int cta, float *sm)
{
    const int t = threadIdx.x, c = cta * kBiasCols + (t & 31);
    float s = 0.0f;
    for (int r0 = 0; r0 < J.rows; r0 += kBiasRows) {
        const int n = min(kBiasRows, J.rows - r0);
        float v[kBiasRows / 8];
#pragma unroll
        for (int i = 0; i < kBiasRows / 8; ++i) {
            const int r = i * 8 + (t >> 5);
            v[i] = r < n ? J.dz[(size_t)(r0 + r) * J.cols + c] : 0.0f;
        }
        __syncthreads();
#pragma unroll
        for (int i = 0; i < kBiasRows / 8; ++i) sm[(i * 8 + (t >> 5)) * 32 + (t & 31)] = v[i];
        __syncthreads();
        if (t < 32)
#pragma unroll 16
            for (int r = 0; r < n; ++r) s += sm[r * 32 + t];
    }
    if (t >= 32) return;
    if (J.g) J.g[c] = s;
    else adam_update(J.w[c], J.m[c], J.v[c], s, J.adam);
}

// a row group (8 rows) of a minibatch per CTA; every thread finds its row once and has several loads in flight (a loop of
// one load an iteration made the last link of a training step 19 us long)
__device__ __forceinline__ void gather_rows(const GatherJob &J, int cta)
{
    constexpr int U = 4;
    const int t = threadIdx.x;
    auto source = [&](int r) { return r < J.valid ? (J.idx ? J.idx[r] : r) : -1; };
    const int r = cta * 8 + (t & 7), from = source(r);            // inputs: a thread's row, 32 columns a round
    const int rt = cta * 8 + (t >> 5), from_t = J.tgt ? source(rt) : -1;   // targets: a warp's row
    for (int c0 = t >> 3; c0 < J.in; c0 += 32 * U) {
        float x[U];
#pragma unroll
        for (int u = 0; u < U; ++u) {
            const int c = c0 + 32 * u;
            x[u] = from >= 0 && c < J.in_real ? J.x[(size_t)from * J.in_real + c] : 0.0f;
        }
#pragma unroll
        for (int u = 0; u < U; ++u) {
            const int c = c0 + 32 * u;
            if (c >= J.in) break;
            bf16 hi, lo;
            split_bf16(x[u], hi, lo);
            J.X.hi[blk(J.rows, r, c)] = hi;
            J.X.lo[blk(J.rows, r, c)] = lo;
            if (J.XT.hi) {
                J.XT.hi[blk(J.in, c, r)] = hi;
                J.XT.lo[blk(J.in, c, r)] = lo;
            }
        }
    }
    for (int c0 = t & 31; J.tgt && c0 < J.out; c0 += 32 * U) {
        float y[U];
#pragma unroll
        for (int u = 0; u < U; ++u) {
            const int c = c0 + 32 * u;
            y[u] = from_t >= 0 && c < J.out_real ? J.t[(size_t)from_t * J.out_real + c] : 0.0f;
        }
#pragma unroll
        for (int u = 0; u < U; ++u)
            if (c0 + 32 * u < J.out) J.tgt[(size_t)rt * J.out + c0 + 32 * u] = y[u];
    }
}

// one link of the chain: the tiles of up to two GEMMs, a bias gradient, the gathering of a minibatch
__global__ void __launch_bounds__(kThreads) k_mlp(const __grid_constant__ Jobs jobs)
{
    extern __shared__ __align__(1024) unsigned char sm[];
    int b = blockIdx.x;
    for (int j = 0; j < 2; ++j) {
        if (b < jobs.gemm[j].ctas) {
            gemm_tile(jobs.gemm[j], jobs, b, sm);
            return;
        }
        b -= jobs.gemm[j].ctas;
    }
    wait_predecessor();
    allow_successor();
    if (b < jobs.bias.ctas) {
        bias_columns(jobs.bias, b, reinterpret_cast<float *>(sm));
        return;
    }
    gather_rows(jobs.gather, b - jobs.bias.ctas);
}

// the operands of a weight matrix [out x in]: plain and transposed
__global__ void k_split_weights(const float *__restrict__ w, int out, int in, Split W, Split WT)
{
    const size_t n = (size_t)out * in;
    for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x) {
        const int r = (int)(i / in), c = (int)(i - (size_t)r * in);
        bf16 hi, lo;
        split_bf16(w[i], hi, lo);
        W.hi[blk(out, r, c)] = hi;
        W.lo[blk(out, r, c)] = lo;
        WT.hi[blk(in, c, r)] = hi;
        WT.lo[blk(in, c, r)] = lo;
    }
}

inline int grid_for(size_t n) { size_t b = (n + 255) / 256; return (int)(b > 4096 ? 4096 : (b < 1 ? 1 : b)); }

} // namespace

struct bec_mlp {
    std::vector<int> w;              // widths (padded): w[0] = padded inputs
    std::vector<int> w_real;         // caller's widths
    int L = 0;                       // weight layers
    std::vector<size_t> woff, boff;  // offsets into the parameter vector
    size_t n_params = 0;
    // device memory, one slab per use: parameters and their operands; Adam moments and the second set of operands; the
    // buffers of a batch for inference, for its gradients, and for training. The first and, for kFirstBatch rows, the third
    // and fourth exist from the start, in one allocation, the others from the first call that needs them: a network that only
    // predicts keeps 5 MB (256 wide) that it does not use, and creating one (with its parameters set) takes 1.8 ms for 6-256-256-256-64
    // and 0.57 for 5-70-130-3 (2.2 and 0.58 with an allocation per buffer), a first gradient call 0.30 and 0.13 ms (0.56, 0.30).
    char *slab[5] = {};              // the allocations, and
    size_t size[5] = {};             // ... their bytes
    char *base[5] = {};              // where each use's buffers lie
    int cap[5] = {};                 // 1, or the batch capacity of slabs 2 to 4
    size_t bytes = 0, limit = 0;     // device bytes in use; BEC_DEVICE_BYTES_LIMIT at creation (0: none)
    float *p = nullptr, *g = nullptr, *m = nullptr, *v = nullptr;   // FP32 params, grads, Adam moments
    std::vector<Split> W[2], WT[2];  // per layer the weights' operands, plain and transposed: the current set and the
    int cur = 0;                     // one that a training step writes
    std::vector<float *> y, dz;      // per layer: activation, its gradient before the activation (FP32) [cap x w]
    std::vector<Split> X, XT, D, DT; // their operands, plain and transposed
    Split X0[2], XT0[2];             // the operands of the inputs of this minibatch and of the next
    float *tgt[2] = {nullptr, nullptr};
    float *io = nullptr;             // raw inputs, and the raw result
    float *raw_t = nullptr;          // raw targets
    float *loss = nullptr;
    int *d_err = nullptr;            // [0] set by a GEMM whose wait ran out, [1] a flag nothing sets
    int sms = 148;
    long long adam_t = 0;
    cudaStream_t s = nullptr;
    std::string err;
    cudaError_t launched = cudaSuccess;      // the first launch since the last check that was refused
    // waits of the device side (read from the environment at every call): limit, fault injection
    int stall = 0;
    unsigned long long limit_ns = 2000000000ull;
};

namespace {

int round_up(int v, int q) { return (v + q - 1) / q * q; }

// hands out 256-byte aligned pieces of a slab; with base == NULL it only counts
struct Carve {
    char *base;
    size_t used = 0;
    template <typename T>
    T *take(size_t n)
    {
        T *p = base ? reinterpret_cast<T *>(base + used) : nullptr;
        used += (n * sizeof(T) + 255) / 256 * 256;
        return p;
    }
    Split split(size_t n)
    {
        Split s;
        s.hi = take<bf16>(n);
        s.lo = take<bf16>(n);
        return s;
    }
};

enum Slab { SLAB_PARAMS, SLAB_ADAM, SLAB_FORWARD, SLAB_BACKWARD, SLAB_TRAIN };
constexpr int kFirstBatch = 256;

size_t carve(bec_mlp *m, Slab which, char *base, int cap)
{
    Carve c{base};
    const int L = m->L;
    auto operands = [&](int k) {
        m->W[k].resize(L);
        m->WT[k].resize(L);
        for (int l = 0; l < L; ++l) {
            m->W[k][l] = c.split((size_t)m->w[l] * m->w[l + 1]);
            m->WT[k][l] = c.split((size_t)m->w[l] * m->w[l + 1]);
        }
    };
    switch (which) {
    case SLAB_PARAMS:
        m->p = c.take<float>(m->n_params);
        operands(0);
        m->loss = c.take<float>(1);
        m->d_err = c.take<int>(2);
        break;
    case SLAB_ADAM:
        m->m = c.take<float>(m->n_params);
        m->v = c.take<float>(m->n_params);
        operands(1);
        break;
    case SLAB_FORWARD:
        m->X.assign(L + 1, Split{nullptr, nullptr});
        m->X0[0] = c.split((size_t)cap * m->w[0]);
        for (int l = 1; l < L; ++l) m->X[l] = c.split((size_t)cap * m->w[l]);
        m->io = c.take<float>((size_t)cap * (m->w_real[0] + m->w_real[L]) + 64);
        break;
    case SLAB_BACKWARD:
        m->y.assign(L + 1, nullptr);
        m->dz.assign(L + 1, nullptr);
        for (auto *v : {&m->XT, &m->D, &m->DT}) v->assign(L + 1, Split{nullptr, nullptr});
        m->g = c.take<float>(m->n_params);
        m->XT0[0] = c.split((size_t)cap * m->w[0]);
        m->tgt[0] = c.take<float>((size_t)cap * m->w[L]);
        m->raw_t = c.take<float>((size_t)cap * m->w_real[L]);
        for (int l = 1; l <= L; ++l) {
            const size_t n = (size_t)cap * m->w[l];
            m->dz[l] = c.take<float>(n);
            m->D[l] = c.split(n);
            m->DT[l] = c.split(n);
            if (l < L) {
                m->y[l] = c.take<float>(n);
                m->XT[l] = c.split(n);
            }
        }
        break;
    case SLAB_TRAIN:
        m->X0[1] = c.split((size_t)cap * m->w[0]);
        m->XT0[1] = c.split((size_t)cap * m->w[0]);
        m->tgt[1] = c.take<float>((size_t)cap * m->w[L]);
        break;
    }
    return c.used;
}

// With a byte limit set, an allocation that would take the network past it fails without reaching the device.
bec_status slab_alloc(bec_mlp *m, char **p, size_t bytes)
{
    *p = nullptr;
    if (m->limit && m->bytes + bytes > m->limit) return BEC_ERR_OUT_OF_MEMORY;
    if (cudaMalloc((void **)p, bytes) != cudaSuccess) { cudaGetLastError(); *p = nullptr; return BEC_ERR_OUT_OF_MEMORY; }
    m->bytes += bytes;
    return BEC_OK;
}

void slab_free(bec_mlp *m, char *p, size_t bytes)
{
    if (!p) return;
    cudaStreamSynchronize(m->s);
    cudaFree(p);
    m->bytes -= bytes;
}

// makes a slab hold at least cap rows (batch slabs; 1 for the others). When the memory is not to be had the first batch's
// buffers, which lie in the parameters' slab, stay as they are; others are given back to make room, and cap says so.
bec_status reserve(bec_mlp *m, Slab which, int cap)
{
    if (cap <= m->cap[which]) return BEC_OK;
    slab_free(m, m->slab[which], m->size[which]);
    if (m->slab[which]) {
        m->slab[which] = m->base[which] = nullptr;
        m->cap[which] = 0;
    }
    const size_t bytes = carve(m, which, nullptr, cap);     // (leaves the slab's pointers null)
    const bec_status st = slab_alloc(m, &m->slab[which], bytes);
    if (st) {
        if (m->base[which]) carve(m, which, m->base[which], m->cap[which]);
        return st;
    }
    m->size[which] = bytes;
    m->base[which] = m->slab[which];
    carve(m, which, m->slab[which], cap);
    if (which == SLAB_ADAM && (cudaMemsetAsync(m->m, 0, sizeof(float) * m->n_params, m->s) != cudaSuccess ||
                               cudaMemsetAsync(m->v, 0, sizeof(float) * m->n_params, m->s) != cudaSuccess))
        return BEC_ERR_CUDA;
    m->cap[which] = cap;
    return BEC_OK;
}

// BEC_STEP_WAIT_LIMIT_MS bounds the device-side waits (2 s by default); BEC_GEMM_INJECT_STALL=1 makes the
// first stage of every tile also wait for a flag that nothing sets (the error path, without a fault)
void read_env(bec_mlp *m)
{
    m->limit_ns = 2000000000ull;
    if (const char *v = std::getenv("BEC_STEP_WAIT_LIMIT_MS")) m->limit_ns = 1000000ull * std::strtoull(v, nullptr, 10);
    const char *inj = std::getenv("BEC_GEMM_INJECT_STALL");
    m->stall = inj && std::atoi(inj) ? 1 : 0;
}

GemmJob make_job(const Split &A, int Ra, const Split &B, int Rb, int M, int N, int K, int epi)
{
    GemmJob j{};
    j.Ahi = A.hi; j.Alo = A.lo; j.Bhi = B.hi; j.Blo = B.lo;
    j.Ra = Ra; j.Rb = Rb;
    j.M = M; j.N = N; j.K = K;
    j.epi = epi;
    return j;
}

// launches the jobs: column tiles as narrow as one CTA per SM allows. A launch that is refused is reported by check_gemm.
void launch(bec_mlp *m, Jobs &J)
{
    J.err = m->d_err;
    J.never = m->d_err + 1;
    J.stall = m->stall;
    J.limit_ns = m->limit_ns;
    int tn = 16, total = 0;
    for (;; tn *= 2) {
        total = J.bias.ctas + J.gather.ctas;
        for (auto &g : J.gemm) {
            g.tn = tile_cols(g.N, tn);
            g.ctas = g.Ahi ? tile_ctas(g.M, g.N, tn) : 0;
            total += g.ctas;
        }
        if (total <= m->sms || tn == kWidestTile) break;
    }
    const bool gemm = J.gemm[0].Ahi != nullptr;
    cudaError_t e = gemm ? ensure_smem_limit((const void *)k_mlp, gemm_smem(kWidestTile)) : cudaSuccess;
    if (!e) e = launch_after(k_mlp, total, kThreads, gemm ? gemm_smem(tn) : 0, m->s, J);
    if (!m->launched) m->launched = e;
}

GatherJob gather_job(bec_mlp *m, int k, const float *x, const float *t, const int *idx, int rows, int valid, bool train)
{
    GatherJob g{};
    g.x = x; g.t = t; g.idx = idx;
    g.rows = rows; g.valid = valid;
    g.in_real = m->w_real[0]; g.in = m->w[0];
    g.out_real = m->w_real[m->L]; g.out = m->w[m->L];
    g.ctas = rows / 8;
    g.X = m->X0[k];
    if (train) {
        g.XT = m->XT0[k];
        g.tgt = m->tgt[k];
    }
    return g;
}

// the forward chain on the inputs in buffer k; train: up to the loss and the output layer's dz, else the outputs of the
// first `valid` rows to out
void forward_chain(bec_mlp *m, int k, int rows, int valid, bool train, float *out, float *loss)
{
    for (int l = 0; l < m->L; ++l) {
        const int in = m->w[l], ow = m->w[l + 1];
        const bool last = l == m->L - 1;
        Jobs J{};
        GemmJob &g = J.gemm[0];
        g = make_job(l ? m->X[l] : m->X0[k], rows, m->W[m->cur][l], ow, rows, ow, in, !last ? EPI_TANH : train ? EPI_LOSS : EPI_LINEAR);
        // (the launch before the first layer's gathered its inputs and may have updated its weights)
        g.early = l > 0;
        g.bias = m->p + m->boff[l];
        if (!last) {
            g.out = m->X[l + 1];
            if (train) {
                g.outT = m->XT[l + 1];
                g.f32 = m->y[l + 1];
            }
        } else if (train) {
            g.tgt = m->tgt[k];
            g.valid = valid;
            g.real_cols = m->w_real[m->L];
            g.loss = loss;
            g.f32 = m->dz[l + 1];
            g.out = m->D[l + 1];
            g.outT = m->DT[l + 1];
        } else {
            g.f32 = out;
        }
        g.f32_ld = last && !train ? m->w_real[m->L] : ow;
        g.f32_rows = last && !train ? valid : rows;
        g.f32_cols = last && !train ? m->w_real[m->L] : ow;
        launch(m, J);
    }
}

// the backward chain from the output layer's dz: gradients into m->g, or (adam) applied to the weights, whose operands go
// to the other set; next: gathered beside the first layer's gradient
void backward_chain(bec_mlp *m, int k, int rows, const AdamArgs *adam, const GatherJob *next)
{
    for (int l = m->L - 1; l >= 0; --l) {
        const int in = m->w[l], ow = m->w[l + 1];
        Jobs J{};
        // dW [out x in] = dZ^T [out x rows] * (X^T [in x rows])^T
        GemmJob &g = J.gemm[0];
        g = make_job(m->DT[l + 1], ow, l ? m->XT[l] : m->XT0[k], in, ow, in, rows, adam ? EPI_ADAM : EPI_GRAD);
        g.early = true;
        if (adam) {
            g.w = m->p + m->woff[l];
            g.m = m->m + m->woff[l];
            g.v = m->v + m->woff[l];
            g.adam = *adam;
            g.out = m->W[1 - m->cur][l];
            g.outT = m->WT[1 - m->cur][l];
        } else {
            g.f32 = m->g + m->woff[l];
            g.f32_ld = in;
            g.f32_rows = ow;
            g.f32_cols = in;
        }
        if (l > 0) {
            // dX [rows x in] = dZ [rows x out] * (W^T [in x out])^T, times the tanh derivative: the next layer's dZ
            GemmJob &d = J.gemm[1];
            d = make_job(m->D[l + 1], rows, m->WT[m->cur][l], in, rows, in, ow, EPI_DX);
            d.early = true;
            d.y = m->y[l];
            d.f32 = m->dz[l];
            d.f32_ld = in;
            d.f32_rows = rows;
            d.f32_cols = in;
            d.out = m->D[l];
            d.outT = m->DT[l];
        }
        BiasJob &b = J.bias;
        b.dz = m->dz[l + 1];
        b.rows = rows;
        b.cols = ow;
        b.ctas = ow / kBiasCols;
        if (adam) {
            b.w = m->p + m->boff[l];
            b.m = m->m + m->boff[l];
            b.v = m->v + m->boff[l];
            b.adam = *adam;
        } else {
            b.g = m->g + m->boff[l];
        }
        if (l == 0 && next) J.gather = *next;
        launch(m, J);
    }
    if (adam) m->cur = 1 - m->cur;
}

void split_weights(bec_mlp *m)
{
    for (int l = 0; l < m->L; ++l) {
        k_split_weights<<<grid_for((size_t)m->w[l] * m->w[l + 1]), 256, 0, m->s>>>(
            m->p + m->woff[l], m->w[l + 1], m->w[l], m->W[m->cur][l], m->WT[m->cur][l]);
        g_launches++;
    }
}

// BEC_ERR_CUDA when a launch since the last check was refused, or a GEMM gave up a wait (synchronises the stream)
bec_status check_gemm(bec_mlp *m)
{
    int e = 0;
    const cudaError_t launched = m->launched;
    m->launched = cudaSuccess;
    if (cudaMemcpyAsync(&e, m->d_err, sizeof(int), cudaMemcpyDeviceToHost, m->s) != cudaSuccess ||
        cudaStreamSynchronize(m->s) != cudaSuccess) {
        m->err = cudaGetErrorString(cudaGetLastError());
        return BEC_ERR_CUDA;
    }
    if (e) {
        cudaMemsetAsync(m->d_err, 0, sizeof(int), m->s);
        m->err = "MLP GEMM: a tensor-core wait gave up";
        return BEC_ERR_CUDA;
    }
    if (launched != cudaSuccess) {
        m->err = cudaGetErrorString(launched);
        cudaGetLastError();
        return BEC_ERR_CUDA;
    }
    return BEC_OK;
}

} // namespace

extern "C" {

bec_status bec_mlp_create(const int32_t *widths, int32_t n_layers, uint64_t seed, bec_mlp **out)
{
    if (!out) return BEC_ERR_INVALID_ARG;
    *out = nullptr;
    if (!widths || n_layers < 1 || n_layers > 16) return BEC_ERR_INVALID_ARG;
    for (int l = 0; l <= n_layers; ++l)
        if (widths[l] < 1 || widths[l] > 4096) return BEC_ERR_INVALID_ARG;
    int ndev = 0;
    if (cudaGetDeviceCount(&ndev) != cudaSuccess || ndev == 0) { cudaGetLastError(); return BEC_ERR_NO_DEVICE; }
    bec_mlp *m = new bec_mlp();
    if (const char *lim = std::getenv("BEC_DEVICE_BYTES_LIMIT")) m->limit = (size_t)std::strtoull(lim, nullptr, 10);
    m->L = n_layers;
    m->w_real.assign(widths, widths + n_layers + 1);
    m->w.resize(n_layers + 1);
    for (int l = 0; l <= n_layers; ++l) m->w[l] = round_up(widths[l], 64);   // GEMM tiles are 64 wide
    for (int l = 0; l < n_layers; ++l) {
        m->woff.push_back(m->n_params);
        m->n_params += (size_t)m->w[l] * m->w[l + 1];
        m->boff.push_back(m->n_params);
        m->n_params += (size_t)m->w[l + 1];
    }
    auto bail = [&](bec_status st) { bec_mlp_destroy(m); return st; };
    bec_status st;
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || cudaDeviceGetAttribute(&m->sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess ||
        cudaStreamCreateWithFlags(&m->s, cudaStreamNonBlocking) != cudaSuccess)
        return bail(BEC_ERR_CUDA);
    // the parameters, and the buffers of a first batch, in one allocation (a later, larger batch gets slabs of its own)
    const Slab at_once[3] = {SLAB_PARAMS, SLAB_FORWARD, SLAB_BACKWARD};
    size_t used = 0;
    for (Slab k : at_once) used += carve(m, k, nullptr, kFirstBatch);
    if ((st = slab_alloc(m, &m->slab[SLAB_PARAMS], used))) return bail(st);
    m->size[SLAB_PARAMS] = used;
    used = 0;
    for (Slab k : at_once) {
        m->base[k] = m->slab[SLAB_PARAMS] + used;
        used += carve(m, k, m->base[k], kFirstBatch);
        m->cap[k] = kFirstBatch;
    }
    if (cudaMemsetAsync(m->d_err, 0, 2 * sizeof(int), m->s) != cudaSuccess) return bail(BEC_ERR_CUDA);
    // Glorot-uniform weights on the real block, zero padding and biases
    std::vector<float> h(m->n_params, 0.0f);
    std::mt19937_64 rng(seed);
    for (int l = 0; l < n_layers; ++l) {
        const float a = std::sqrt(6.0f / (float)(widths[l] + widths[l + 1]));
        std::uniform_real_distribution<float> U(-a, a);
        for (int o = 0; o < widths[l + 1]; ++o)
            for (int i = 0; i < widths[l]; ++i) h[m->woff[l] + (size_t)o * m->w[l] + i] = U(rng);
    }
    cudaMemcpyAsync(m->p, h.data(), sizeof(float) * h.size(), cudaMemcpyHostToDevice, m->s);
    split_weights(m);
    if (cudaStreamSynchronize(m->s) != cudaSuccess) return bail(BEC_ERR_CUDA);
    *out = m;
    return BEC_OK;
}

void bec_mlp_destroy(bec_mlp *m)
{
    if (!m) return;
    if (m->s) cudaStreamSynchronize(m->s);
    for (char *p : m->slab) cudaFree(p);
    if (m->s) cudaStreamDestroy(m->s);
    delete m;
}

int64_t bec_mlp_param_count(const bec_mlp *m)
{
    if (!m) return 0;
    int64_t n = 0;
    for (int l = 0; l < m->L; ++l) n += (int64_t)m->w_real[l] * m->w_real[l + 1] + m->w_real[l + 1];
    return n;
}

// host layout: for each layer W [out x in] row-major then b [out] (caller's widths)
bec_status bec_mlp_get_params(bec_mlp *m, float *params)
{
    if (!m || !params) return BEC_ERR_INVALID_ARG;
    std::vector<float> h(m->n_params);
    cudaMemcpyAsync(h.data(), m->p, sizeof(float) * h.size(), cudaMemcpyDeviceToHost, m->s);
    if (cudaStreamSynchronize(m->s) != cudaSuccess) return BEC_ERR_CUDA;
    size_t k = 0;
    for (int l = 0; l < m->L; ++l) {
        for (int o = 0; o < m->w_real[l + 1]; ++o)
            for (int i = 0; i < m->w_real[l]; ++i) params[k++] = h[m->woff[l] + (size_t)o * m->w[l] + i];
        for (int o = 0; o < m->w_real[l + 1]; ++o) params[k++] = h[m->boff[l] + o];
    }
    return BEC_OK;
}

bec_status bec_mlp_set_params(bec_mlp *m, const float *params)
{
    if (!m || !params) return BEC_ERR_INVALID_ARG;
    std::vector<float> h(m->n_params, 0.0f);
    size_t k = 0;
    for (int l = 0; l < m->L; ++l) {
        for (int o = 0; o < m->w_real[l + 1]; ++o)
            for (int i = 0; i < m->w_real[l]; ++i) h[m->woff[l] + (size_t)o * m->w[l] + i] = params[k++];
        for (int o = 0; o < m->w_real[l + 1]; ++o) h[m->boff[l] + o] = params[k++];
    }
    if (cudaMemcpyAsync(m->p, h.data(), sizeof(float) * h.size(), cudaMemcpyHostToDevice, m->s) != cudaSuccess) return BEC_ERR_CUDA;
    split_weights(m);
    return cudaStreamSynchronize(m->s) == cudaSuccess ? BEC_OK : BEC_ERR_CUDA;
}

bec_status bec_mlp_forward(bec_mlp *m, const float *x, int32_t batch, float *y)
{
    if (!m || !x || !y || batch < 1) return BEC_ERR_INVALID_ARG;
    const int rows = round_up(batch, 64);
    bec_status st;
    if ((st = reserve(m, SLAB_FORWARD, rows))) return st;
    read_env(m);
    const size_t nx = (size_t)batch * m->w_real[0], ny = (size_t)batch * m->w_real[m->L];
    float *out = m->io + (nx + 63) / 64 * 64;     // aligned for 16-byte stores
    // x is pageable or pinned memory that the caller may reuse on return: this call waits for its result
    if (cudaMemcpyAsync(m->io, x, sizeof(float) * nx, cudaMemcpyHostToDevice, m->s) != cudaSuccess) return BEC_ERR_CUDA;
    Jobs J{};
    J.gather = gather_job(m, 0, m->io, nullptr, nullptr, rows, batch, false);
    launch(m, J);
    forward_chain(m, 0, rows, batch, false, out, nullptr);
    if (cudaMemcpyAsync(y, out, sizeof(float) * ny, cudaMemcpyDeviceToHost, m->s) != cudaSuccess) return BEC_ERR_CUDA;
    return check_gemm(m);
}

// Loss and gradients of mean((y - target)^2) over the batch (host params layout).
bec_status bec_mlp_gradients(bec_mlp *m, const float *x, const float *target, int32_t batch, float *loss,
                             float *grads)
{
    if (!m || !x || !target || batch < 1) return BEC_ERR_INVALID_ARG;
    const int rows = round_up(batch, 64);
    bec_status st;
    if ((st = reserve(m, SLAB_FORWARD, rows)) || (st = reserve(m, SLAB_BACKWARD, rows))) return st;
    read_env(m);
    const size_t nx = (size_t)batch * m->w_real[0], ny = (size_t)batch * m->w_real[m->L];
    if (cudaMemcpyAsync(m->io, x, sizeof(float) * nx, cudaMemcpyHostToDevice, m->s) != cudaSuccess ||
        cudaMemcpyAsync(m->raw_t, target, sizeof(float) * ny, cudaMemcpyHostToDevice, m->s) != cudaSuccess ||
        cudaMemsetAsync(m->loss, 0, sizeof(float), m->s) != cudaSuccess)
        return BEC_ERR_CUDA;
    Jobs J{};
    J.gather = gather_job(m, 0, m->io, m->raw_t, nullptr, rows, batch, true);
    launch(m, J);
    forward_chain(m, 0, rows, batch, true, nullptr, m->loss);
    backward_chain(m, 0, rows, nullptr, nullptr);
    float l = 0.f;
    cudaMemcpyAsync(&l, m->loss, sizeof(float), cudaMemcpyDeviceToHost, m->s);
    std::vector<float> h(m->n_params);
    cudaMemcpyAsync(h.data(), m->g, sizeof(float) * h.size(), cudaMemcpyDeviceToHost, m->s);
    if ((st = check_gemm(m))) return st;
    if (loss) *loss = l;
    if (grads) {
        size_t k = 0;
        for (int li = 0; li < m->L; ++li) {
            for (int o = 0; o < m->w_real[li + 1]; ++o, k += m->w_real[li])
                std::memcpy(grads + k, &h[m->woff[li] + (size_t)o * m->w[li]], sizeof(float) * m->w_real[li]);
            std::memcpy(grads + k, &h[m->boff[li]], sizeof(float) * m->w_real[li + 1]);
            k += m->w_real[li + 1];
        }
    }
    return BEC_OK;
}

// Adam on minibatches drawn (seeded) from n samples; loss_history[s] = loss of step s. The samples are uploaded once and
// the losses stay on the device until the end; the indices of kDrawSteps minibatches at a time are drawn and uploaded
// while the GPU works on earlier ones, so the step loop issues work without waiting on the GPU.
bec_status bec_mlp_train(bec_mlp *m, const float *x, const float *target, int32_t n, int32_t batch, int32_t steps,
                         float lr, int32_t schedule, uint64_t seed, float *loss_history)
{
    if (!m || !x || !target || n < 1 || batch < 1 || steps < 0) return BEC_ERR_INVALID_ARG;
    if (schedule != BEC_LR_CONSTANT && schedule != BEC_LR_COSINE) return BEC_ERR_INVALID_ARG;
    constexpr int kDrawSteps = 64;
    const int rows = round_up(batch, 64);
    bec_status st;
    read_env(m);
    if (steps == 0) return check_gemm(m);
    if ((st = reserve(m, SLAB_ADAM, 1)) || (st = reserve(m, SLAB_FORWARD, rows)) || (st = reserve(m, SLAB_BACKWARD, rows)) ||
        (st = reserve(m, SLAB_TRAIN, rows)))
        return st;
    const int in_r = m->w_real[0], out_r = m->w_real[m->L];
    const int valid = std::min(batch, n);
    float *dx = nullptr, *dt = nullptr, *dhist = nullptr;
    int *didx = nullptr;
    auto samples = [&](char *base) {
        Carve c{base};
        dx = c.take<float>((size_t)n * in_r);
        dt = c.take<float>((size_t)n * out_r);
        dhist = c.take<float>(steps);
        didx = c.take<int>((size_t)valid * steps);
        return c.used;
    };
    char *slab = nullptr;
    const size_t slab_bytes = samples(nullptr);
    if ((st = slab_alloc(m, &slab, slab_bytes))) return st;
    struct F { bec_mlp *m; char *p; size_t n; ~F() { slab_free(m, p, n); } } f{m, slab, slab_bytes};
    samples(slab);
    if (cudaMemcpyAsync(dx, x, sizeof(float) * (size_t)n * in_r, cudaMemcpyHostToDevice, m->s) != cudaSuccess ||
        cudaMemcpyAsync(dt, target, sizeof(float) * (size_t)n * out_r, cudaMemcpyHostToDevice, m->s) != cudaSuccess ||
        cudaMemsetAsync(dhist, 0, sizeof(float) * steps, m->s) != cudaSuccess)
        return BEC_ERR_CUDA;
    // minibatches: consecutive slices of seeded shuffles of the n samples
    std::mt19937_64 rng(seed);
    std::vector<int> order(n), drawn;
    for (int i = 0; i < n; ++i) order[i] = i;
    int pos = n, ready = 0;
    auto draw = [&]() -> bec_status {
        const int k = std::min(kDrawSteps, steps - ready);
        drawn.resize((size_t)valid * k);
        for (int &i : drawn) {
            if (pos >= n) { std::shuffle(order.begin(), order.end(), rng); pos = 0; }
            i = order[pos++];
        }
        // the copy from this pageable buffer is staged before the call returns
        const cudaError_t e = cudaMemcpyAsync(didx + (size_t)valid * ready, drawn.data(), sizeof(int) * drawn.size(),
                                              cudaMemcpyHostToDevice, m->s);
        ready += k;
        return e == cudaSuccess ? BEC_OK : BEC_ERR_CUDA;
    };
    auto minibatch = [&](int s) { return gather_job(m, s & 1, dx, dt, didx + (size_t)valid * s, rows, valid, true); };
    const double pi = 3.14159265358979323846;
    for (int s = 0; s < steps; ++s) {
        if (s == 0) {
            if ((st = draw())) return st;
            Jobs J{};
            J.gather = minibatch(0);
            launch(m, J);
        }
        if (s + 1 < steps && s + 1 == ready && (st = draw())) return st;
        forward_chain(m, s & 1, rows, valid, true, nullptr, dhist + s);
        ++m->adam_t;
        AdamArgs a;
        a.c1 = 1.0f - std::pow(0.9f, (float)m->adam_t);
        a.c2 = 1.0f - std::pow(0.999f, (float)m->adam_t);
        a.lr = schedule == BEC_LR_COSINE ? (float)(lr * 0.5 * (1.0 + std::cos(pi * s / steps))) : lr;
        GatherJob next{};
        if (s + 1 < steps) next = minibatch(s + 1);
        backward_chain(m, s & 1, rows, &a, s + 1 < steps ? &next : nullptr);
    }
    std::vector<float> hist(steps, 0.0f);
    cudaMemcpyAsync(hist.data(), dhist, sizeof(float) * steps, cudaMemcpyDeviceToHost, m->s);
    if ((st = check_gemm(m))) {
        // a tile that gave up has written neither its weights nor their operands in the set that is current now
        split_weights(m);
        cudaStreamSynchronize(m->s);
        return st;
    }
    if (loss_history)
        for (int s = 0; s < steps; ++s) loss_history[s] = hist[s];
    return cudaGetLastError() == cudaSuccess ? BEC_OK : BEC_ERR_CUDA;
}

} // extern "C"
