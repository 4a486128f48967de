// Learned T2 initial guess: a 4-layer MLP (8 -> 256 -> 256 -> 256 -> 1, SiLU)
// that predicts, per amplitude, t2(converged) - t2(reference guess).
//
// Inputs of the amplitude t2(i,a,j,b) with (ia) <= (jb):
//   the reference guess L(iajb)/D(iajb) (guessCC), e_i, e_j, e_a, e_b (MO Fock
//   diagonal), (ia|jb), (ib|ja) and 8/N (molecule size).
// Only canonical pairs are evaluated and the result is written to both t2
// entries of the pair, so the guess keeps the pair symmetry of t2 exactly.
//
// Inference (mlp_infer, one CTA per SM looping over 128-row tiles): layer 1
// runs on the CUDA cores and writes bf16 activations straight into shared
// memory in the 128-byte-swizzled K-major layout the tensor core reads;
// layers 2 and 3 are tcgen05.mma (kind::f16, BF16 x BF16 -> FP32, M = 128,
// N = 256, K = 256) with the bf16 weights brought in by TMA and the
// accumulator in 256 TMEM columns; their epilogues (tcgen05.ld, bias, SiLU,
// bf16) feed the next layer through shared memory; the output layer is a dot
// product in the last epilogue. In the engine the features are computed from
// the molecules' device state inside the kernel, one launch for all of them,
// and the result goes straight into t2. What bounds a tile is the activation
// arithmetic (98k SiLUs) and the FP64 features; the weights' TMA loads run
// behind them (W2 from the tile's start, W3 from the moment the layer-2
// products are done). Sixteen warps share the columns of a tile (eight left each
// scheduler two warps, and most of a tile was their latency), and four more
// compute the next tile's inputs meanwhile, one thread per row. Measured
// (16 warps and the inputs ahead, from eight and none): 128 molecules of 8 to
// 64 sites 23.5 -> 14.9 ms, the initialisation of 160 sites 109 -> 99 ms, both
// with an approximate division in the SiLU. With the correctly rounded one the
// guess takes 14.8 ms of those 128 molecules' initialisation (12.2 before) and
// 21.0 ms at 160 sites (18.6).
//
// Training (hx_mlp_grad / hx_mlp_train): the six 256-wide products of a step
// (layers 2 and 3 forward, their weight gradients and the gradients of their
// inputs) on the tensor cores (bgemm: bf16 operands brought in by TMA, FP32
// accumulation in TMEM), with the same bf16 roundings as inference (W2, W3
// and the activations entering layers 2 and 3) plus the loss gradients
// entering those products (straight-through in the backward pass); the
// 8-wide first layer, the output unit and the bias sums on the CUDA cores.
// Mean-squared error in units of y_scale, Adam with a cosine learning-rate
// decay. The gradients are those of the CPU reference in oracle/mlp.py.
#include <cuda.h>
#include <cuda_bf16.h>
#include <cudaTypedefs.h>

#include <algorithm>
#include <cmath>
#include <cstring>
#include <numeric>
#include <random>
#include <vector>

#include "hx_common.cuh"
#include "hx_mlp.h"

namespace mlp {

__device__ __forceinline__ float silu(float z) { return z / (1.f + __expf(-z)); }
__device__ __forceinline__ float dsilu(float z)
{
    const float s = 1.f / (1.f + __expf(-z));
    return s * (1.f + z * (1.f - s));
}
__device__ __forceinline__ float bf16r(float x) { return __bfloat162float(__float2bfloat16_rn(x)); }

// ------------------------------------------------------------------ features
// canonical pair index r -> (p, q), p <= q, rows of the upper triangle of an n x n matrix
__device__ __forceinline__ void tri_index(long long r, long long n, long long &p, long long &q)
{
    const double nn = (double)n + 0.5;
    long long pp = (long long)(nn - sqrt(fmax(nn * nn - 2.0 * (double)r, 0.0)));
    if (pp < 0) pp = 0;
    if (pp > n - 1) pp = n - 1;
    while (pp > 0 && pp * n - pp * (pp - 1) / 2 > r) --pp;
    while (pp + 1 < n && (pp + 1) * n - (pp + 1) * pp / 2 <= r) ++pp;
    p = pp;
    q = pp + (r - (pp * n - pp * (pp - 1) / 2));
}

// features of canonical pair (p, q); returns the flat pair index p*ov + q
__device__ long long pair_features(const CCMol &m, long long p, long long q, float *f, double &guess)
{
    const int o = m.o, v = m.v, n = m.N;
    const long long ov = (long long)o * v;
    const int i = (int)(p / v), a = (int)(p % v), j = (int)(q / v), b = (int)(q % v);
    const long long pq = p * ov + q;
    const long long p2 = (long long)i * v + b, q2 = (long long)j * v + a;
    guess = m.Lov[pq] / m.D2[pq];
    f[0] = (float)guess;
    f[1] = (float)m.Fmo[(long long)i * n + i];
    f[2] = (float)m.Fmo[(long long)j * n + j];
    f[3] = (float)m.Fmo[(long long)(o + a) * n + o + a];
    f[4] = (float)m.Fmo[(long long)(o + b) * n + o + b];
    f[5] = (float)m.gov[pq];
    f[6] = (float)m.gov[(p2 < q2 ? p2 : q2) * ov + (p2 < q2 ? q2 : p2)];
    f[7] = 8.f / (float)n;
    return pq;
}

// training rows: features and target t2 - guess of the given canonical pairs
__global__ void k_sample(const CCMol *mols, int mol, const long long *rows, int n, float *X, float *T)
{
    const CCMol &m = mols[mol];
    const long long ov = (long long)m.o * m.v;
    for (int k = blockIdx.x * blockDim.x + threadIdx.x; k < n; k += gridDim.x * blockDim.x) {
        long long p, q;
        tri_index(rows[k], ov, p, q);
        double g;
        const long long pq = pair_features(m, p, q, X + (long long)k * F, g);
        T[k] = (float)(m.t2[pq] - g);
    }
}

// ------------------------------------------------------------------ tcgen05 inference
__device__ __forceinline__ uint32_t smem_u32(const void *p) { return (uint32_t)__cvta_generic_to_shared(p); }
__device__ __forceinline__ unsigned long long gtimer()
{
    unsigned long long t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    return t;
}
// bounded wait (4 s): false and an error code if the phase never completes
__device__ __forceinline__ bool wait_bar(uint64_t *bar, uint32_t parity, int *err, int code)
{
    const unsigned long long t0 = gtimer();
    for (;;) {
        uint32_t ok;
        asm volatile(
            "{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\tselp.u32 %0, 1, 0, p;\n\t}\n"
            : "=r"(ok)
            : "r"(smem_u32(bar)), "r"(parity)
            : "memory");
        if (ok) return true;
        if (gtimer() - t0 > 4000000000ull) {
            if (err) atomicCAS(err, 0, code);
            return false;
        }
    }
}
// shared-memory descriptor: K-major, 128-byte swizzle, 8-row groups 1024 B apart
__device__ __forceinline__ uint64_t sw128_desc(uint32_t addr)
{
    return (uint64_t)((addr & 0x3FFFF) >> 4) | ((uint64_t)1 << 16) | ((uint64_t)(1024 >> 4) << 32) |
           ((uint64_t)1 << 46) | ((uint64_t)2 << 61);
}
// byte offset of the 16-byte chunk c (elements 8c..8c+7) of row `row` in a [rows x 64] bf16 K-block
__device__ __forceinline__ uint32_t sw128_chunk(int row, int c) { return (uint32_t)(row * 128 + (((c ^ row) & 7) << 4)); }

constexpr int TILE = 128;
constexpr int A_KB = TILE * 128;               // one K-block of activations: 128 rows x 64 bf16
constexpr int B_KB = H * 128;                  // one K-block of weights: 256 rows x 64 bf16
constexpr int A_BYTES = 4 * A_KB;              // 64 KB
constexpr int B_BYTES = 4 * B_KB;              // 128 KB
constexpr int MLP_PARTS = 4;                   // column parts of a tile: 4 warps each
constexpr int MLP_COMPUTE = MLP_PARTS * TILE;  // threads of the layers; 128 more work out the next tile's inputs
constexpr int MLP_THREADS = MLP_COMPUTE + TILE;
constexpr int MLP_SMEM = 1024 + A_BYTES + B_BYTES + (H * F + 4 * H + MLP_PARTS * TILE + 2 * TILE * F) * 4 + 2 * TILE * 24;

struct InferArgs {
    const float *X;          // [n x F] features (hx_mlp_predict) or NULL (engine)
    float *Y;                // [n] predictions (hx_mlp_predict)
    const CCMol *mols;       // engine: molecules, first tile of each and the total
    const int *tile_start;
    int nmol;
    long long n;             // rows (hx_mlp_predict)
    const float *P;
    int *err;
};

// one row's input and the pair it belongs to (m: the molecule, NULL for hx_mlp_predict)
__device__ __forceinline__ void load_row(const InferArgs &a, const CCMol *m, long long gr, long long n, float *x,
                                         long long &pq, long long &qp, double &guess)
{
    pq = qp = -1;
    guess = 0.0;
    if (gr >= n) {
#pragma unroll
        for (int f = 0; f < F; ++f) x[f] = 0.f;
        return;
    }
    if (!m) {
#pragma unroll
        for (int f = 0; f < F; ++f) x[f] = a.X[gr * F + f];
        return;
    }
    const long long ov = (long long)m->o * m->v;
    long long p, q;
    tri_index(gr, ov, p, q);
    pq = pair_features(*m, p, q, x, guess);
    qp = q * ov + p;
}

__global__ void __launch_bounds__(MLP_THREADS, 1) mlp_infer(InferArgs a, const __grid_constant__ CUtensorMap mapW2,
                                                            const __grid_constant__ CUtensorMap mapW3)
{
    extern __shared__ __align__(1024) uint8_t smem_raw[];
    uint8_t *smem = (uint8_t *)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
    uint8_t *sA = smem, *sB = smem + A_BYTES;
    float *sW1 = (float *)(sB + B_BYTES);       // [H x F]
    float *sb1 = sW1 + H * F;                   // [H] biases of layers 1, 2, 3
    float *sb2 = sb1 + H;
    float *sb3 = sb2 + H;
    float *sw4 = sb3 + H;                       // [H] output weights
    float *sred = sw4 + H;                      // [MLP_PARTS][TILE] dot products of the column parts
    float *sx = sred + MLP_PARTS * TILE;        // [2][F][TILE] normalised inputs, of this tile and the next
    double *sguess = (double *)(sx + 2 * TILE * F);               // [2][TILE] reference guesses
    long long *spq = (long long *)(sguess + 2 * TILE);            // [2][TILE] pairs' positions in t2 (-1: no row)
    long long *sqp = spq + 2 * TILE;
    __shared__ const CCMol *smol[2];
    __shared__ __align__(8) uint64_t bar_full, bar_done;
    __shared__ uint32_t tmem_slot;
    __shared__ int s_abort;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int row = (warp & 3) * 32 + lane;     // TMEM lane = tile row of this thread
    const int part = warp >> 2;                 // column part [PC*part, +PC) of this thread; MLP_PARTS: the inputs' warps
    constexpr int PC = H / MLP_PARTS;
    auto compute_sync = [&]() { asm volatile("bar.sync 1, %0;" ::"n"(MLP_COMPUTE) : "memory"); };
    for (int k = tid; k < H * F; k += MLP_THREADS) sW1[k] = a.P[O_W1 + k];
    for (int k = tid; k < H; k += MLP_THREADS) {
        sb1[k] = a.P[O_B1 + k];
        sb2[k] = a.P[O_B2 + k];
        sb3[k] = a.P[O_B3 + k];
        sw4[k] = a.P[O_W4 + k];
    }
    float xs[F], xc[F];
#pragma unroll
    for (int f = 0; f < F; ++f) { xs[f] = a.P[O_XS + f]; xc[f] = a.P[O_XC + f]; }
    const float b4 = a.P[O_B4], ys = a.P[O_YS];
    if (tid == 0) {
        s_abort = 0;
        asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(smem_u32(&bar_full)));
        asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(smem_u32(&bar_done)));
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&tmem_slot)),
                     "r"(H));
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem = tmem_slot;
    const uint32_t idesc = (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(H >> 3) << 17) | ((uint32_t)(TILE >> 4) << 24);
    const uint32_t lane_base = (uint32_t)((warp & 3) * 32) << 16;
    uint32_t ph_full = 0, ph_done = 0;
    const long long ntiles = a.mols ? a.tile_start[a.nmol] : (a.n + TILE - 1) / TILE;
    // weights of a hidden layer into sB (free: every MMA that read it has completed)
    auto load_weights = [&](const CUtensorMap *map) {
        asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(&bar_full)), "r"(B_BYTES)
                     : "memory");
        for (int kb = 0; kb < 4; ++kb)
            asm volatile(
                "cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4}], [%2];" ::"r"(
                    smem_u32(sB + kb * B_KB)),
                "l"(map), "r"(smem_u32(&bar_full)), "r"(kb * 64), "r"(0)
                : "memory");
    };
    // inputs of a tile into buffer b, one thread per row
    auto load_tile = [&](long long tile, int b) {
        const CCMol *m = nullptr;
        long long gr = tile * TILE + row, n = a.n;
        if (a.mols) {
            int lo = 0, hi = a.nmol - 1;                // the last molecule whose first tile is at or below this one
            while (lo < hi) {
                const int mid = (lo + hi + 1) >> 1;
                if (a.tile_start[mid] <= tile) lo = mid; else hi = mid - 1;
            }
            m = a.mols + lo;
            gr = (tile - a.tile_start[lo]) * TILE + row;
            const long long ov = (long long)m->o * m->v;
            n = ov * (ov + 1) / 2;
        }
        float x[F];
        long long pq = -1, qp = -1;
        double guess = 0.0;
        load_row(a, m, gr, n, x, pq, qp, guess);
#pragma unroll
        for (int f = 0; f < F; ++f) sx[(b * F + f) * TILE + row] = (x[f] - xs[f]) * xc[f];
        spq[b * TILE + row] = m ? pq : gr < n ? gr : -1;
        sqp[b * TILE + row] = qp;
        sguess[b * TILE + row] = guess;
        if (row == 0) smol[b] = m;
    };
    int buf = 0;
    if (part == MLP_PARTS && blockIdx.x < ntiles) load_tile(blockIdx.x, 0);
    for (long long tile = blockIdx.x; tile < ntiles; tile += gridDim.x, buf ^= 1) {
        __syncthreads();                                // this tile's inputs are there; the other buffer is free
        if (s_abort) break;
        if (part == MLP_PARTS) {
            if (tile + gridDim.x < ntiles) load_tile(tile + gridDim.x, buf ^ 1);
            continue;
        }
        if (tid == 0) load_weights(&mapW2);
        float x[F];
#pragma unroll
        for (int f = 0; f < F; ++f) x[f] = sx[(buf * F + f) * TILE + row];
        // layer 1: hidden units [PC*part, +PC) of this row, 8 per 16-byte store
        for (int c = part * (PC / 8); c < (part + 1) * (PC / 8); ++c) {
            __align__(16) __nv_bfloat16 h8[8];
#pragma unroll
            for (int e = 0; e < 8; ++e) {
                const int j = c * 8 + e;
                float z = sb1[j];
                const float4 wa = *reinterpret_cast<const float4 *>(sW1 + j * F), wb = *reinterpret_cast<const float4 *>(sW1 + j * F + 4);
                z = fmaf(wa.x, x[0], z); z = fmaf(wa.y, x[1], z); z = fmaf(wa.z, x[2], z); z = fmaf(wa.w, x[3], z);
                z = fmaf(wb.x, x[4], z); z = fmaf(wb.y, x[5], z); z = fmaf(wb.z, x[6], z); z = fmaf(wb.w, x[7], z);
                h8[e] = __float2bfloat16_rn(silu(z));
            }
            *reinterpret_cast<uint4 *>(sA + (c >> 3) * A_KB + sw128_chunk(row, c & 7)) = *reinterpret_cast<uint4 *>(h8);
        }
        float dot = 0.f;
        for (int layer = 0; layer < 2; ++layer) {
            const float *sb = layer == 0 ? sb2 : sb3;
            asm volatile("fence.proxy.async.shared::cta;" ::: "memory");   // generic smem writes -> tensor core
            compute_sync();
            if (tid == 0) {
                if (!wait_bar(&bar_full, ph_full, a.err, 11)) {
                    s_abort = 1;
                } else {
                    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                    for (int kb = 0; kb < 4; ++kb)
                        for (int kk = 0; kk < 4; ++kk) {
                            const uint64_t ad = sw128_desc(smem_u32(sA + kb * A_KB) + kk * 32);
                            const uint64_t bd = sw128_desc(smem_u32(sB + kb * B_KB) + kk * 32);
                            const uint32_t acc = (kb | kk) ? 1u : 0u;
                            asm volatile(
                                "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
                                "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}\n" ::"r"(tmem),
                                "l"(ad), "l"(bd), "r"(idesc), "r"(acc));
                        }
                }
                // arrives once the MMAs issued above (if any) have completed
                asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(
                                 smem_u32(&bar_done))
                             : "memory");
            }
            ph_full ^= 1;
            if (!wait_bar(&bar_done, ph_done, a.err, 12)) s_abort = 1;
            ph_done ^= 1;
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            compute_sync();
            if (s_abort) break;
            if (layer == 0 && tid == 0) load_weights(&mapW3);
            // epilogue: this row, columns [PC*part, +PC)
            for (int c0 = part * PC; c0 < (part + 1) * PC; c0 += 16) {
                uint32_t r[16];
                asm volatile(
                    "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
                    : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
                      "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
                    : "r"(tmem + lane_base + (uint32_t)c0));
                asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
                if (layer == 0) {
                    __align__(16) __nv_bfloat16 h8[16];
#pragma unroll
                    for (int e = 0; e < 16; ++e) h8[e] = __float2bfloat16_rn(silu(__uint_as_float(r[e]) + sb[c0 + e]));
                    const int c = c0 >> 3;
                    *reinterpret_cast<uint4 *>(sA + (c >> 3) * A_KB + sw128_chunk(row, c & 7)) = *reinterpret_cast<uint4 *>(h8);
                    *reinterpret_cast<uint4 *>(sA + ((c + 1) >> 3) * A_KB + sw128_chunk(row, (c + 1) & 7)) =
                        *reinterpret_cast<uint4 *>(h8 + 8);
                } else {
#pragma unroll
                    for (int e = 0; e < 16; ++e) dot = fmaf(silu(__uint_as_float(r[e]) + sb[c0 + e]), sw4[c0 + e], dot);
                }
            }
            asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
        }
        if (part) sred[part * TILE + row] = dot;
        compute_sync();
        const long long pq = spq[buf * TILE + row];
        if (part == 0 && pq >= 0 && !s_abort) {
            for (int k = 1; k < MLP_PARTS; ++k) dot += sred[k * TILE + row];
            const float y = (dot + b4) * ys;
            const CCMol *m = smol[buf];
            if (!m) {
                a.Y[pq] = y;
            } else {
                const double t = sguess[buf * TILE + row] + (double)y;
                m->t2[pq] = t;
                m->t2[sqp[buf * TILE + row]] = t;
            }
        }
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    if (warp == 0) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(H));
}

// ------------------------------------------------------------------ tcgen05 training GEMM
// C[M x 256] = A[M x K] B[256 x K]^T (+ bias[n]) from bf16 operands, both
// K-major (row m of A, row n of B, K contiguous), FP32 accumulation in 256
// TMEM columns. CTA (x, y) = 128-row tile x a split of kb_per 64-deep
// K-blocks; with more than one split the CTAs add into C with atomics (C
// cleared first). Thread 0 streams the K-blocks with TMA through two
// stages and issues the MMAs (M = 128, N = 256, K = 16); the four warps
// then drain TMEM (a lane per row). Every wait is bounded; a CTA that gives
// up records a code, waits (bounded) for the loads it issued and still
// frees its TMEM.
constexpr int BG_STAGE = A_KB + B_KB;                 // 16 KB of A + 32 KB of B per K-block
constexpr int BG_SMEM = 1024 + 2 * BG_STAGE;
constexpr int BG_THREADS = 128;

__global__ void __launch_bounds__(BG_THREADS, 1) bgemm(const __grid_constant__ CUtensorMap mapA,
                                                       const __grid_constant__ CUtensorMap mapB, float *C, int ldc,
                                                       const float *bias, int nkb, int kb_per, int *err)
{
    extern __shared__ __align__(1024) uint8_t bg_raw[];
    uint8_t *smem = (uint8_t *)(((uintptr_t)bg_raw + 1023) & ~(uintptr_t)1023);
    __shared__ __align__(8) uint64_t full[2], freed[2], done;
    __shared__ uint32_t tmem_slot;
    __shared__ int s_abort;
    const int tid = threadIdx.x, warp = tid >> 5;
    const int m0 = blockIdx.x * TILE;
    const int kb0 = blockIdx.y * kb_per, n = min(nkb, kb0 + kb_per) - kb0;
    if (tid == 0) {
        s_abort = 0;
        for (int q = 0; q < 2; ++q) {
            asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(smem_u32(&full[q])));
            asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(smem_u32(&freed[q])));
        }
        asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(smem_u32(&done)));
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&tmem_slot)),
                     "r"(H));
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem = tmem_slot;
    if (tid == 0) {
        const uint32_t idesc = (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(H >> 3) << 17) | ((uint32_t)(TILE >> 4) << 24);
        auto load = [&](int i) {
            uint8_t *sa = smem + (i & 1) * BG_STAGE, *sb = sa + A_KB;
            asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(&full[i & 1])),
                         "r"(BG_STAGE)
                         : "memory");
            asm volatile(
                "cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4}], [%2];" ::"r"(
                    smem_u32(sa)),
                "l"(&mapA), "r"(smem_u32(&full[i & 1])), "r"((kb0 + i) * 64), "r"(m0)
                : "memory");
            asm volatile(
                "cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4}], [%2];" ::"r"(
                    smem_u32(sb)),
                "l"(&mapB), "r"(smem_u32(&full[i & 1])), "r"((kb0 + i) * 64), "r"(0)
                : "memory");
        };
        int issued = 0, consumed = 0;
        for (; issued < n && issued < 2; ++issued) load(issued);
        bool ok = true;
        for (int i = 0; i < n && ok; ++i) {
            ok = wait_bar(&full[i & 1], (uint32_t)((i >> 1) & 1), err, 21);
            if (!ok) break;
            ++consumed;
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            const uint32_t sa = smem_u32(smem + (i & 1) * BG_STAGE), sb = sa + A_KB;
            for (int kk = 0; kk < 4; ++kk) {
                const uint64_t ad = sw128_desc(sa + kk * 32), bd = sw128_desc(sb + kk * 32);
                const uint32_t acc = (i | kk) ? 1u : 0u;
                asm volatile(
                    "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
                    "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}\n" ::"r"(tmem),
                    "l"(ad), "l"(bd), "r"(idesc), "r"(acc));
            }
            asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(
                             smem_u32(&freed[i & 1]))
                         : "memory");
            if (issued < n) {                  // stage i & 1 is free once these MMAs complete
                ok = wait_bar(&freed[i & 1], (uint32_t)((i >> 1) & 1), err, 22);
                if (ok) load(issued++);
            }
        }
        if (!ok) {
            s_abort = 1;
            for (int j = consumed; j < issued; ++j) wait_bar(&full[j & 1], (uint32_t)((j >> 1) & 1), nullptr, 0);
        }
        // arrives once every MMA issued above has completed
        asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(smem_u32(&done))
                     : "memory");
    }
    const bool fin = wait_bar(&done, 0u, err, 23);
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    __syncthreads();
    if (fin && !s_abort) {
        const uint32_t lane_base = (uint32_t)(warp * 32) << 16;
        float *crow = C + (long long)(m0 + tid) * ldc;
        const bool atomic = gridDim.y > 1;
        for (int c0 = 0; c0 < H; c0 += 16) {
            uint32_t r[16];
            asm volatile(
                "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
                : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
                  "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
                : "r"(tmem + lane_base + (uint32_t)c0));
            asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
            float v[16];
#pragma unroll
            for (int e = 0; e < 16; ++e) v[e] = __uint_as_float(r[e]) + (bias ? bias[c0 + e] : 0.f);
            if (atomic) {
#pragma unroll
                for (int e = 0; e < 16; ++e) atomicAdd(crow + c0 + e, v[e]);
            } else {
#pragma unroll
                for (int e = 0; e < 16; e += 4) *reinterpret_cast<float4 *>(crow + c0 + e) = make_float4(v[e], v[e + 1], v[e + 2], v[e + 3]);
            }
        }
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    if (warp == 0) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(H));
}

// bf16 copies, row-major (dst) and transposed (dstT), of the two hidden weight
// matrices W2 and W3 of the blob, through 32 x 32 shared tiles so that both
// are written coalesced; block = one tile.
__global__ void __launch_bounds__(256) k_weight_copies(const float *P, __nv_bfloat16 *W2, __nv_bfloat16 *W2T,
                                                       __nv_bfloat16 *W3, __nv_bfloat16 *W3T)
{
    __shared__ float t[32][33];
    const int tx = threadIdx.x & 31, ty = threadIdx.x >> 5, ct = H / 32;
    const bool second = blockIdx.x >= ct * ct;
    const int u = second ? blockIdx.x - ct * ct : blockIdx.x;
    const float *src = P + (second ? O_W3 : O_W2);
    __nv_bfloat16 *dst = second ? W3 : W2, *dstT = second ? W3T : W2T;
    const int r0 = (u / ct) * 32, c0 = (u % ct) * 32;
    for (int y = ty; y < 32; y += 8) {
        const float v = src[(r0 + y) * H + c0 + tx];
        t[y][tx] = v;
        dst[(r0 + y) * H + c0 + tx] = __float2bfloat16_rn(v);
    }
    __syncthreads();
    for (int y = ty; y < 32; y += 8) dstT[(c0 + y) * H + r0 + tx] = __float2bfloat16_rn(t[tx][y]);
}

__global__ void k_to_bf16(const float *src, __nv_bfloat16 *dst, int n)
{
    for (int k = blockIdx.x * blockDim.x + threadIdx.x; k < n; k += gridDim.x * blockDim.x) dst[k] = __float2bfloat16_rn(src[k]);
}

// ------------------------------------------------------------------ SIMT training kernels
// x = (X[idx] - shift) * scale and t = T[idx] for the rows of one batch (idx NULL = identity)
__global__ void k_gather_norm(const float *X, const float *T, const long long *idx, const float *P, float *x,
                              float *t, int n)
{
    for (int e = blockIdx.x * blockDim.x + threadIdx.x; e < n * F; e += gridDim.x * blockDim.x) {
        const int r = e / F, f = e % F;
        const long long src = idx ? idx[r] : r;
        x[e] = (X[src * F + f] - P[O_XS + f]) * P[O_XC + f];
        if (f == 0) t[r] = T[src];
    }
}
// The element-wise kernels between the products: a block takes TR rows of the
// batch x all H columns, in TR x 32 column tiles (thread = (column, every
// eighth row)), writes the bf16 operand of the next product in both orders
// and adds its column sums (bias and output-weight gradients) to G, so every
// activation is read once and no product is spent on a sum. The sums over
// the batch as one-column products on the 64 x 64 SIMT tile took 0.2 ms each,
// a step of 4096 rows 3.0 ms.
constexpr int TR = 32;
struct Tile {
    float t[TR][33];
    float red[8][32];
};

// bf16 copies of the staged tile (rows r0.., columns c0..): dst [rows x H], dstT [H x rows]
__device__ __forceinline__ void store_tile(const Tile &s, int r0, int c0, int rows, __nv_bfloat16 *dst, __nv_bfloat16 *dstT)
{
    const int tx = threadIdx.x & 31, ty = threadIdx.x >> 5;
    for (int y = ty; y < TR; y += 8) dst[(long long)(r0 + y) * H + c0 + tx] = __float2bfloat16_rn(s.t[y][tx]);
    for (int y = ty; y < 32; y += 8) dstT[(long long)(c0 + y) * rows + r0 + tx] = __float2bfloat16_rn(s.t[tx][y]);
}
// adds the block's sums of a column tile to out[c0 ..] (v: this thread's share of column tx)
__device__ __forceinline__ void add_columns(Tile &s, float v, float *out)
{
    const int tx = threadIdx.x & 31, ty = threadIdx.x >> 5;
    __syncthreads();
    s.red[ty][tx] = v;
    __syncthreads();
    if (ty == 0) {
        float a = 0.f;
#pragma unroll
        for (int k = 0; k < 8; ++k) a += s.red[k][tx];
        atomicAdd(out + tx, a);
    }
}

// layer 1: z1 = x W1^T + b1, h1 = bf16(silu(z1))
__global__ void __launch_bounds__(256) k_layer1(const float *x, const float *P, float *z1, __nv_bfloat16 *h, __nv_bfloat16 *hT, int rows)
{
    __shared__ Tile s;
    __shared__ float xs[TR][F];
    const int tx = threadIdx.x & 31, ty = threadIdx.x >> 5, r0 = blockIdx.x * TR;
    for (int e = threadIdx.x; e < TR * F; e += 256) xs[e / F][e % F] = x[(long long)r0 * F + e];
    for (int c0 = 0; c0 < H; c0 += 32) {
        const int c = c0 + tx;
        float w[F];
#pragma unroll
        for (int f = 0; f < F; ++f) w[f] = P[O_W1 + c * F + f];
        const float b = P[O_B1 + c];
        __syncthreads();
        for (int y = ty; y < TR; y += 8) {
            float a = 0.f;
#pragma unroll
            for (int f = 0; f < F; ++f) a = fmaf(xs[y][f], w[f], a);
            const float z = a + b;
            z1[(long long)(r0 + y) * H + c] = z;
            s.t[y][tx] = silu(z);
        }
        __syncthreads();
        store_tile(s, r0, c0, rows, h, hT);
    }
}
// h = bf16(silu(z))
__global__ void __launch_bounds__(256) k_act(const float *z, __nv_bfloat16 *h, __nv_bfloat16 *hT, int rows)
{
    __shared__ Tile s;
    const int tx = threadIdx.x & 31, ty = threadIdx.x >> 5, r0 = blockIdx.x * TR;
    for (int c0 = 0; c0 < H; c0 += 32) {
        __syncthreads();
        for (int y = ty; y < TR; y += 8) s.t[y][tx] = silu(z[(long long)(r0 + y) * H + c0 + tx]);
        __syncthreads();
        store_tile(s, r0, c0, rows, h, hT);
    }
}
// output unit, loss and the gradient of z3: h3 = silu(z3), residual in network
// units r = h3 w4 + b4 - T / y_scale, dy = 2 r / n (0 for the padded rows
// >= n), loss += mean r^2, dz3 = dy w4 silu'(z3); dw4, db4, db3 added to G
__global__ void __launch_bounds__(256) k_out(const float *z3, const float *T, const float *P, float *G, float *loss,
                                             __nv_bfloat16 *dz, __nv_bfloat16 *dzT, int n, int rows)
{
    __shared__ Tile s;
    __shared__ float dy[TR], rr[TR];
    const int tx = threadIdx.x & 31, ty = threadIdx.x >> 5, r0 = blockIdx.x * TR;
    const float *W4 = P + O_W4;
    for (int y = ty; y < TR; y += 8) {
        float a = 0.f;
#pragma unroll
        for (int c = 0; c < H; c += 32) a = fmaf(silu(z3[(long long)(r0 + y) * H + c + tx]), W4[c + tx], a);
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) a += __shfl_xor_sync(0xffffffffu, a, o);
        if (tx == 0) {
            const bool live = r0 + y < n;
            const float r = live ? a + P[O_B4] - T[r0 + y] / P[O_YS] : 0.f;
            dy[y] = 2.f * r / n;
            rr[y] = r * r;
        }
    }
    __syncthreads();
    if (ty == 0) {
        float d = dy[tx], q = rr[tx];
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) { d += __shfl_xor_sync(0xffffffffu, d, o); q += __shfl_xor_sync(0xffffffffu, q, o); }
        if (tx == 0) { atomicAdd(G + O_B4, d); atomicAdd(loss, q / n); }
    }
    for (int c0 = 0; c0 < H; c0 += 32) {
        float gw = 0.f, gb = 0.f;
        for (int y = ty; y < TR; y += 8) {
            const float z = z3[(long long)(r0 + y) * H + c0 + tx], g = dy[y] * W4[c0 + tx] * dsilu(z);
            gw = fmaf(dy[y], silu(z), gw);
            gb += g;
            s.t[y][tx] = g;
        }
        add_columns(s, gw, G + O_W4 + c0);
        add_columns(s, gb, G + O_B3 + c0);
        store_tile(s, r0, c0, rows, dz, dzT);
        __syncthreads();
    }
}
// dz = dh silu'(z), its column sums added to db
__global__ void __launch_bounds__(256) k_dact(const float *dh, const float *z, float *db, __nv_bfloat16 *dz, __nv_bfloat16 *dzT, int rows)
{
    __shared__ Tile s;
    const int tx = threadIdx.x & 31, ty = threadIdx.x >> 5, r0 = blockIdx.x * TR;
    for (int c0 = 0; c0 < H; c0 += 32) {
        float gb = 0.f;
        for (int y = ty; y < TR; y += 8) {
            const long long e = (long long)(r0 + y) * H + c0 + tx;
            const float g = dh[e] * dsilu(z[e]);
            gb += g;
            s.t[y][tx] = g;
        }
        add_columns(s, gb, db + c0);
        store_tile(s, r0, c0, rows, dz, dzT);
        __syncthreads();
    }
}
// layer 1's gradients: dz1 = dh silu'(z1), db1 and dW1 = dz1^T x added to G; thread = column
__global__ void __launch_bounds__(H) k_dlayer1(const float *dh, const float *z1, const float *x, float *G)
{
    __shared__ float xs[TR][F];
    const int c = threadIdx.x, r0 = blockIdx.x * TR;
    for (int e = threadIdx.x; e < TR * F; e += H) xs[e / F][e % F] = x[(long long)r0 * F + e];
    __syncthreads();
    float gb = 0.f, gw[F] = {};
#pragma unroll 4
    for (int y = 0; y < TR; ++y) {
        const long long e = (long long)(r0 + y) * H + c;
        const float g = dh[e] * dsilu(z1[e]);
        gb += g;
#pragma unroll
        for (int f = 0; f < F; ++f) gw[f] = fmaf(g, xs[y][f], gw[f]);
    }
    atomicAdd(G + O_B1 + c, gb);
#pragma unroll
    for (int f = 0; f < F; ++f) atomicAdd(G + O_W1 + c * F + f, gw[f]);
}
// Adam on the trainable prefix of the blob
__global__ void k_adam(float *P, const float *G, float *m1, float *m2, int n, float lr, float b1, float b2, float eps,
                       float c1, float c2)
{
    for (int e = blockIdx.x * blockDim.x + threadIdx.x; e < n; e += gridDim.x * blockDim.x) {
        const float g = G[e];
        m1[e] = b1 * m1[e] + (1.f - b1) * g;
        m2[e] = b2 * m2[e] + (1.f - b2) * g * g;
        P[e] -= lr * (m1[e] / c1) / (sqrtf(m2[e] / c2) + eps);
    }
}

// ------------------------------------------------------------------ host helpers
static inline unsigned nblocks(long long n, int t = 256)
{
    long long b = (n + t - 1) / t;
    return (unsigned)std::max(1LL, std::min(b, 65535LL));
}

static PFN_cuTensorMapEncodeTiled_v12000 encode_fn()
{
    static PFN_cuTensorMapEncodeTiled_v12000 fn = nullptr;
    if (!fn) {
        void *p = nullptr;
        cudaDriverEntryPointQueryResult q;
        if (cudaGetDriverEntryPointByVersion("cuTensorMapEncodeTiled", &p, 12000, cudaEnableDefault, &q) == cudaSuccess &&
            q == cudaDriverEntryPointSuccess)
            fn = (PFN_cuTensorMapEncodeTiled_v12000)p;
    }
    return fn;
}

// 2D map over a bf16 [rows x cols] matrix: 64 x box_rows boxes, 128-byte swizzle
static int map_bf16(CUtensorMap *map, const void *base, long long rows, int cols, int box_rows)
{
    auto fn = encode_fn();
    if (!fn) { hx_set_error("cuTensorMapEncodeTiled is unavailable"); return HX_ERR_CUDA; }
    cuuint64_t dims[2] = {(cuuint64_t)cols, (cuuint64_t)rows};
    cuuint64_t strides[1] = {(cuuint64_t)cols * 2};
    cuuint32_t box[2] = {64, (cuuint32_t)box_rows};
    cuuint32_t es[2] = {1, 1};
    CUresult r = fn(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<void *>(base), dims, strides, box, es,
                    CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                    CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (r != CUDA_SUCCESS) { hx_set_error("cuTensorMapEncodeTiled failed (%d)", (int)r); return HX_ERR_CUDA; }
    return HX_OK;
}

// device workspace for batches of up to M rows (padded to Mp, a multiple of
// the 128-row tile: the padded rows have zero inputs and zero loss gradient)
struct Work {
    int M = 0, Mp = 0;
    float *x = nullptr, *t = nullptr, *z1 = nullptr, *z2 = nullptr, *z3 = nullptr, *dh = nullptr, *G = nullptr,
          *loss = nullptr;
    // bf16 operands of the tensor-core GEMMs: activations and gradients (and
    // their transposes, [H x Mp]) and the two hidden weight matrices
    __nv_bfloat16 *h1b = nullptr, *h2b = nullptr, *h1T = nullptr, *h2T = nullptr, *dzb = nullptr, *dzT = nullptr,
                  *W2b = nullptr, *W3b = nullptr, *W2T = nullptr, *W3T = nullptr;
    CUtensorMap mH1b, mH2b, mW2b, mW3b, mDzT, mH1T, mH2T, mDzb, mW2T, mW3T;
    int *err = nullptr;
    int alloc(int m)
    {
        M = m;
        Mp = (m + TILE - 1) / TILE * TILE;
        const size_t act = (size_t)Mp * H * 4, actb = (size_t)Mp * H * 2, wb = (size_t)H * H * 2;
        float **big[] = {&z1, &z2, &z3, &dh};
        for (float **b : big)
            if (cudaMalloc(b, act) != cudaSuccess) return HX_ERR_NOMEM;
        __nv_bfloat16 **bb[] = {&h1b, &h2b, &h1T, &h2T, &dzb, &dzT};
        for (__nv_bfloat16 **b : bb)
            if (cudaMalloc(b, actb) != cudaSuccess) return HX_ERR_NOMEM;
        __nv_bfloat16 **wbs[] = {&W2b, &W3b, &W2T, &W3T};
        for (__nv_bfloat16 **b : wbs)
            if (cudaMalloc(b, wb) != cudaSuccess) return HX_ERR_NOMEM;
        if (cudaMalloc(&x, (size_t)Mp * F * 4) != cudaSuccess || cudaMalloc(&t, (size_t)Mp * 4) != cudaSuccess ||
            cudaMalloc(&G, (size_t)NPARAM * 4) != cudaSuccess || cudaMalloc(&loss, 4) != cudaSuccess ||
            cudaMalloc(&err, 4) != cudaSuccess)
            return HX_ERR_NOMEM;
        // padded rows: zero inputs and targets (and a zero loss gradient, k_out)
        if (cudaMemset(x, 0, (size_t)Mp * F * 4) != cudaSuccess || cudaMemset(t, 0, (size_t)Mp * 4) != cudaSuccess ||
            cudaMemset(err, 0, 4) != cudaSuccess)
            return HX_ERR_CUDA;
        int rc = HX_OK;
        if (rc == HX_OK) rc = map_bf16(&mH1b, h1b, Mp, H, TILE);
        if (rc == HX_OK) rc = map_bf16(&mH2b, h2b, Mp, H, TILE);
        if (rc == HX_OK) rc = map_bf16(&mDzb, dzb, Mp, H, TILE);
        if (rc == HX_OK) rc = map_bf16(&mDzT, dzT, H, Mp, TILE);
        if (rc == HX_OK) rc = map_bf16(&mH1T, h1T, H, Mp, H);
        if (rc == HX_OK) rc = map_bf16(&mH2T, h2T, H, Mp, H);
        if (rc == HX_OK) rc = map_bf16(&mW2b, W2b, H, H, H);
        if (rc == HX_OK) rc = map_bf16(&mW3b, W3b, H, H, H);
        if (rc == HX_OK) rc = map_bf16(&mW2T, W2T, H, H, H);
        if (rc == HX_OK) rc = map_bf16(&mW3T, W3T, H, H, H);
        if (rc != HX_OK) return rc;
        if (cudaFuncSetAttribute(bgemm, cudaFuncAttributeMaxDynamicSharedMemorySize, BG_SMEM) != cudaSuccess) {
            hx_set_error("cannot reserve shared memory for the training GEMM");
            return HX_ERR_CUDA;
        }
        return HX_OK;
    }
    int error_word() const
    {
        int v = 0;
        if (err) cudaMemcpy(&v, err, 4, cudaMemcpyDeviceToHost);
        return v;
    }
    ~Work()
    {
        float *all[] = {x, t, z1, z2, z3, dh, G, loss};
        for (float *b : all) cudaFree(b);
        __nv_bfloat16 *allb[] = {h1b, h2b, h1T, h2T, dzb, dzT, W2b, W3b, W2T, W3T};
        for (__nv_bfloat16 *b : allb) cudaFree(b);
        cudaFree(err);
    }
};

// tensor-core GEMM C[rows x H] = A B^T (+ bias) over nkb 64-deep K-blocks; splits > 1
// add into C (zero before) from that many K ranges
static void bf16_gemm(cudaStream_t s, const CUtensorMap &a, const CUtensorMap &b, int rows, int nkb, int splits,
                    float *C, const float *bias, int *err)
{
    const int kb_per = (nkb + splits - 1) / splits;
    const dim3 grid(rows / TILE, (nkb + kb_per - 1) / kb_per);
    bgemm<<<grid, BG_THREADS, BG_SMEM, s>>>(a, b, C, H, bias, nkb, kb_per, err);
}

// forward + backward of one batch already normalised in w.x / w.t (M rows);
// gradients into w.G (overwritten), mean squared error added to w.loss. The
// six 256-wide products (layers 2 and 3 forward, their weight gradients and
// the gradients of their inputs) run on the tensor cores in BF16 with FP32
// accumulation (bgemm); the 8-wide first layer, the 1-wide output and the
// bias sums are part of the element-wise kernels between them. The loss
// gradient dz entering a bf16 product is rounded to bf16 (oracle/mlp.py
// applies the same roundings).
static void fwd_bwd(cudaStream_t s, Work &w, const float *P, int M)
{
    const int Mp = w.Mp, nk = H / 64, nkm = Mp / 64;
    const unsigned g = (unsigned)(Mp / TR);
    cudaMemsetAsync(w.G, 0, (size_t)O_XS * 4, s);
    k_weight_copies<<<2 * (H / 32) * (H / 32), 256, 0, s>>>(P, w.W2b, w.W2T, w.W3b, w.W3T);
    k_layer1<<<g, 256, 0, s>>>(w.x, P, w.z1, w.h1b, w.h1T, Mp);
    bf16_gemm(s, w.mH1b, w.mW2b, Mp, nk, 1, w.z2, P + O_B2, w.err);
    k_act<<<g, 256, 0, s>>>(w.z2, w.h2b, w.h2T, Mp);
    bf16_gemm(s, w.mH2b, w.mW3b, Mp, nk, 1, w.z3, P + O_B3, w.err);
    k_out<<<g, 256, 0, s>>>(w.z3, w.t, P, w.G, w.loss, w.dzb, w.dzT, M, Mp);
    // layer 3
    bf16_gemm(s, w.mDzT, w.mH2T, H, nkm, std::max(1, nkm / 4), w.G + O_W3, nullptr, w.err);   // dW3 = bf16(dz3)^T h2
    bf16_gemm(s, w.mDzb, w.mW3T, Mp, nk, 1, w.dh, nullptr, w.err);          // dh2 = bf16(dz3) bf16(W3)
    k_dact<<<g, 256, 0, s>>>(w.dh, w.z2, w.G + O_B2, w.dzb, w.dzT, Mp);
    // layer 2
    bf16_gemm(s, w.mDzT, w.mH1T, H, nkm, std::max(1, nkm / 4), w.G + O_W2, nullptr, w.err);
    bf16_gemm(s, w.mDzb, w.mW2T, Mp, nk, 1, w.dh, nullptr, w.err);
    // layer 1
    k_dlayer1<<<g, H, 0, s>>>(w.dh, w.z1, w.x, w.G);
    hx_count_launches(12);
}


int Model::load(const float *host_blob)
{
    release();
    if (cudaMalloc(&P, (size_t)NPARAM * 4) != cudaSuccess || cudaMalloc(&W2, (size_t)H * H * 2) != cudaSuccess ||
        cudaMalloc(&W3, (size_t)H * H * 2) != cudaSuccess || cudaMalloc(&err, 4) != cudaSuccess) {
        hx_set_error("learned guess: device allocation failed");
        return HX_ERR_NOMEM;
    }
    if (cudaMemcpy(P, host_blob, (size_t)NPARAM * 4, cudaMemcpyHostToDevice) != cudaSuccess ||
        cudaMemset(err, 0, 4) != cudaSuccess) {
        hx_set_error("learned guess: upload failed");
        return HX_ERR_CUDA;
    }
    k_to_bf16<<<64, 256>>>(P + O_W2, W2, H * H);
    k_to_bf16<<<64, 256>>>(P + O_W3, W3, H * H);
    auto fn = encode_fn();
    if (!fn) { hx_set_error("cuTensorMapEncodeTiled is unavailable"); return HX_ERR_CUDA; }
    for (int k = 0; k < 2; ++k) {
        cuuint64_t dims[2] = {(cuuint64_t)H, (cuuint64_t)H};
        cuuint64_t strides[1] = {(cuuint64_t)H * 2};
        cuuint32_t box[2] = {64, (cuuint32_t)H};
        cuuint32_t es[2] = {1, 1};
        CUresult r = fn(k == 0 ? &mapW2 : &mapW3, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, k == 0 ? (void *)W2 : (void *)W3,
                        dims, strides, box, es, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B,
                        CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
        if (r != CUDA_SUCCESS) { hx_set_error("cuTensorMapEncodeTiled failed (%d)", (int)r); return HX_ERR_CUDA; }
    }
    if (cudaFuncSetAttribute(mlp_infer, cudaFuncAttributeMaxDynamicSharedMemorySize, MLP_SMEM) != cudaSuccess) {
        hx_set_error("cannot reserve shared memory for mlp_infer");
        return HX_ERR_CUDA;
    }
    hx_count_launches(2);
    return cudaDeviceSynchronize() == cudaSuccess ? HX_OK : HX_ERR_CUDA;
}

void Model::release()
{
    cudaFree(P);
    cudaFree(W2);
    cudaFree(W3);
    cudaFree(err);
    cudaFree(tile_start);
    P = nullptr;
    W2 = W3 = nullptr;
    err = nullptr;
    tile_start = nullptr;
    tiles_cap = 0;
}

int Model::error_word() const
{
    int v = 0;
    if (err) cudaMemcpy(&v, err, 4, cudaMemcpyDeviceToHost);
    return v;
}

static cudaError_t launch_infer(const InferArgs &a, const Model &m, long long tiles, cudaStream_t s)
{
    if (tiles <= 0) return cudaSuccess;
    int dev = 0, nsm = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev);
    const unsigned grid = (unsigned)std::min<long long>(tiles, nsm > 0 ? nsm : 1);
    mlp_infer<<<grid, MLP_THREADS, MLP_SMEM, s>>>(a, m.mapW2, m.mapW3);
    hx_count_launches(1);
    return cudaGetLastError();
}

cudaError_t Model::apply(const CCMol *d_mols, const long long *npairs, int nmol, cudaStream_t s)
{
    std::vector<int> start(nmol + 1, 0);
    for (int k = 0; k < nmol; ++k) start[k + 1] = start[k] + (int)((npairs[k] + TILE - 1) / TILE);
    if (nmol > tiles_cap) {
        cudaFree(tile_start);
        tile_start = nullptr;
        tiles_cap = 0;
        const cudaError_t e = cudaMalloc(&tile_start, sizeof(int) * (nmol + 1));
        if (e != cudaSuccess) return e;
        tiles_cap = nmol;
    }
    cudaError_t e = cudaMemcpyAsync(tile_start, start.data(), sizeof(int) * (nmol + 1), cudaMemcpyHostToDevice, s);
    InferArgs a{nullptr, nullptr, d_mols, tile_start, nmol, 0, P, err};
    if (e == cudaSuccess) e = launch_infer(a, *this, start[nmol], s);
    if (e == cudaSuccess) e = cudaStreamSynchronize(s);      // (the prefix sums are pageable host memory)
    return e;
}

}  // namespace mlp

// ------------------------------------------------------------------ C ABI
using namespace mlp;

extern "C" {

int hx_mlp_nparam(void) { return NPARAM; }

int hx_mlp_predict(const float *params, const float *X, int64_t n, float *Y)
{
    if (!params || n < 0 || (n > 0 && (!X || !Y))) { hx_set_error("hx_mlp_predict: bad arguments"); return HX_ERR_ARG; }
    if (n == 0) return HX_OK;
    Model m;
    int rc = m.load(params);
    float *dX = nullptr, *dY = nullptr;
    if (rc == HX_OK && (cudaMalloc(&dX, (size_t)n * F * 4) != cudaSuccess || cudaMalloc(&dY, (size_t)n * 4) != cudaSuccess)) {
        hx_set_error("hx_mlp_predict: allocation failed");
        rc = HX_ERR_NOMEM;
    }
    if (rc == HX_OK) {
        cudaError_t e = cudaMemcpy(dX, X, (size_t)n * F * 4, cudaMemcpyHostToDevice);
        InferArgs a{dX, dY, nullptr, nullptr, 0, n, m.P, m.err};
        if (e == cudaSuccess) e = launch_infer(a, m, (n + TILE - 1) / TILE, 0);
        if (e == cudaSuccess) e = cudaDeviceSynchronize();
        if (e != cudaSuccess) { hx_set_error("hx_mlp_predict: %s", cudaGetErrorString(e)); rc = HX_ERR_CUDA; }
        else if (int w = m.error_word()) { hx_set_error("hx_mlp_predict: a tensor-core wait timed out (%d)", w); rc = HX_ERR_KERNEL; }
        else if (cudaMemcpy(Y, dY, (size_t)n * 4, cudaMemcpyDeviceToHost) != cudaSuccess) rc = HX_ERR_CUDA;
    }
    cudaFree(dX);
    cudaFree(dY);
    m.release();
    return rc;
}

int hx_mlp_grad(const float *params, const float *X, const float *T, int32_t n, float *loss, float *grad)
{
    if (!params || !X || !T || n <= 0) { hx_set_error("hx_mlp_grad: bad arguments"); return HX_ERR_ARG; }
    Work w;
    float *dP = nullptr, *dX = nullptr, *dT = nullptr;
    int rc = w.alloc(n);
    if (rc == HX_OK && (cudaMalloc(&dP, (size_t)NPARAM * 4) != cudaSuccess || cudaMalloc(&dX, (size_t)n * F * 4) != cudaSuccess ||
                        cudaMalloc(&dT, (size_t)n * 4) != cudaSuccess))
        rc = HX_ERR_NOMEM;
    if (rc == HX_ERR_NOMEM) hx_set_error("hx_mlp_grad: allocation failed");
    if (rc == HX_OK) {
        cudaMemcpy(dP, params, (size_t)NPARAM * 4, cudaMemcpyHostToDevice);
        cudaMemcpy(dX, X, (size_t)n * F * 4, cudaMemcpyHostToDevice);
        cudaMemcpy(dT, T, (size_t)n * 4, cudaMemcpyHostToDevice);
        cudaMemset(w.loss, 0, 4);
        k_gather_norm<<<nblocks((long long)n * F), 256>>>(dX, dT, nullptr, dP, w.x, w.t, n);
        fwd_bwd(0, w, dP, n);
        cudaError_t e = cudaDeviceSynchronize();
        if (e != cudaSuccess) { hx_set_error("hx_mlp_grad: %s", cudaGetErrorString(e)); rc = HX_ERR_CUDA; }
        else if (int we = w.error_word()) { hx_set_error("hx_mlp_grad: a tensor-core wait timed out (%d)", we); rc = HX_ERR_KERNEL; }
        else {
            if (loss) cudaMemcpy(loss, w.loss, 4, cudaMemcpyDeviceToHost);
            if (grad) {
                cudaMemcpy(grad, w.G, (size_t)O_XS * 4, cudaMemcpyDeviceToHost);
                for (int k = O_XS; k < NPARAM; ++k) grad[k] = 0.f;     // normalisation constants are not trained
            }
        }
    }
    cudaFree(dP);
    cudaFree(dX);
    cudaFree(dT);
    return rc;
}

int hx_mlp_train(float *params, const float *X, const float *T, int64_t n, int32_t epochs, int32_t batch, float lr,
                 uint64_t seed, float *epoch_loss)
{
    if (!params || !X || !T || batch <= 0 || n < batch || epochs <= 0 || !(lr > 0.f)) {
        hx_set_error("hx_mlp_train: bad arguments");
        return HX_ERR_ARG;
    }
    Work w;
    float *dP = nullptr, *dX = nullptr, *dT = nullptr, *m1 = nullptr, *m2 = nullptr;
    long long *dperm = nullptr;
    const int ntrain = O_XS;          // W1 .. b4; the normalisation constants stay fixed
    int rc = w.alloc(batch);
    if (rc == HX_OK &&
        (cudaMalloc(&dP, (size_t)NPARAM * 4) != cudaSuccess || cudaMalloc(&dX, (size_t)n * F * 4) != cudaSuccess ||
         cudaMalloc(&dT, (size_t)n * 4) != cudaSuccess || cudaMalloc(&m1, (size_t)ntrain * 4) != cudaSuccess ||
         cudaMalloc(&m2, (size_t)ntrain * 4) != cudaSuccess || cudaMalloc(&dperm, (size_t)n * 8) != cudaSuccess))
        rc = HX_ERR_NOMEM;
    if (rc == HX_ERR_NOMEM) hx_set_error("hx_mlp_train: allocation failed");
    if (rc == HX_OK) {
        cudaMemcpy(dP, params, (size_t)NPARAM * 4, cudaMemcpyHostToDevice);
        cudaMemcpy(dX, X, (size_t)n * F * 4, cudaMemcpyHostToDevice);
        cudaMemcpy(dT, T, (size_t)n * 4, cudaMemcpyHostToDevice);
        cudaMemset(m1, 0, (size_t)ntrain * 4);
        cudaMemset(m2, 0, (size_t)ntrain * 4);
        std::mt19937_64 rng(seed);
        std::vector<long long> perm(n);
        std::iota(perm.begin(), perm.end(), 0LL);
        const long long nb = n / batch;
        const long long total = nb * epochs;
        long long step = 0;
        const float b1 = 0.9f, b2 = 0.999f;
        for (int ep = 0; ep < epochs && rc == HX_OK; ++ep) {
            std::shuffle(perm.begin(), perm.end(), rng);
            cudaMemcpy(dperm, perm.data(), (size_t)n * 8, cudaMemcpyHostToDevice);
            cudaMemset(w.loss, 0, 4);
            for (long long b = 0; b < nb; ++b) {
                k_gather_norm<<<nblocks((long long)batch * F), 256>>>(dX, dT, dperm + b * batch, dP, w.x, w.t, batch);
                fwd_bwd(0, w, dP, batch);
                ++step;
                const float lr_t = 0.5f * lr * (1.f + cosf(3.14159265f * (float)(step - 1) / (float)total));
                k_adam<<<nblocks(ntrain), 256>>>(dP, w.G, m1, m2, ntrain, lr_t, b1, b2, 1e-8f,
                                                 1.f - powf(b1, (float)step), 1.f - powf(b2, (float)step));
                hx_count_launches(2);
            }
            float l = 0.f;
            cudaError_t e = cudaMemcpy(&l, w.loss, 4, cudaMemcpyDeviceToHost);
            if (e != cudaSuccess) { hx_set_error("hx_mlp_train: %s", cudaGetErrorString(e)); rc = HX_ERR_CUDA; }
            else if (int we = w.error_word()) { hx_set_error("hx_mlp_train: a tensor-core wait timed out (%d)", we); rc = HX_ERR_KERNEL; }
            if (epoch_loss) epoch_loss[ep] = l / (float)(nb > 0 ? nb : 1);
        }
        if (rc == HX_OK && cudaMemcpy(params, dP, (size_t)ntrain * 4, cudaMemcpyDeviceToHost) != cudaSuccess) rc = HX_ERR_CUDA;
    }
    cudaFree(dP);
    cudaFree(dX);
    cudaFree(dT);
    cudaFree(m1);
    cudaFree(m2);
    cudaFree(dperm);
    return rc;
}

}  // extern "C"

// training rows of a solved molecule (engine side, declared in hx_engine.cu)
cudaError_t hx_mlp_sample(const CCMol *d_mols, int mol, const long long *d_rows, int n, float *dX, float *dT,
                          cudaStream_t s)
{
    k_sample<<<nblocks(n), 256, 0, s>>>(d_mols, mol, d_rows, n, dX, dT);
    hx_count_launches(1);
    return cudaGetLastError();
}
