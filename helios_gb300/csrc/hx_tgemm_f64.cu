// FP64 grouped tensor-GEMM on the CUDA cores (the plain-FP64 contraction backend).
//
// One launch runs a whole group of TgemmDesc problems (e.g. the same
// contraction for every molecule of a batch): CTAs are laid out over the
// concatenated tile lists and each finds its problem by counting the
// tile_starts at or below its tile. Tiles of molecules whose `active` flag is
// 0 exit at once.
//
// What bounds it: GB300 issues two FP64 multiply-adds per clock and SM, so a
// warp-wide FMA occupies the pipe for 16 clocks and everything else (loads,
// index arithmetic, shared memory) fits beside it even with one output per
// thread. The time of a launch is therefore the FMAs of the busiest SM, and
// the tile is as small as that allows: T x T outputs, T = 16 (256 threads) or,
// when a launch would not give every SM two such tiles, T = 8, whose k-blocks
// are then shared by four groups of 64 threads (a quarter of the chain of
// dependent FMAs, one sum through shared memory at the end).
// Warps whose outputs all lie outside M x N skip their FMAs. k runs in
// ascending order for every output (of its group), 32 at a time, the next
// k-block fetched into registers while the current one is multiplied. Operand
// elements are gathered through the descriptor's split strides, so any index
// permutation of a 4-index tensor is read in place; the loader walks the
// operand's contiguous dimension first.
// Measured against 64 x 64 tiles computed in full (16 us per 16 k on one SM,
// whatever M and N): the 12-site solve 45 -> 11.5 ms, 24 molecules of 8-24
// sites 141 -> 42 ms, one iteration of a 50-site ladder 6.2 -> 3.4 ms.
#include <algorithm>
#include "hx_common.cuh"
#include "hx_kernels.h"

namespace {
constexpr int BKG = 32;      // k per group and block

__device__ __forceinline__ long long split_off(int x, int xi, long long s0, long long s1)
{
    const int q = x / xi;
    return (long long)q * s0 + (long long)(x - q * xi) * s1;
}

template <int T, int G>
__global__ void __launch_bounds__(T * T * G) tgemm_f64_kernel(const TgemmDesc *__restrict__ descs, int ndesc,
                                                          const int *__restrict__ active)
{
    constexpr int BK = BKG * G, NT = T * T * G, R = T * BK / NT;   // R elements of each operand per thread and k-block
    __shared__ double As[BK][T + 1];
    __shared__ double Bs[BK][T + 1];
    const long long tile = blockIdx.x;
    int di = 0;
    if (ndesc > 1) {                                      // the last descriptor with tile_start <= tile
        int n = 0;
        for (int k0 = 0; k0 < ndesc; k0 += NT) {
            const int k = k0 + threadIdx.x;
            n += __syncthreads_count(k < ndesc && descs[k].tile_start <= tile);
        }
        di = n - 1;
    }
    const TgemmDesc &d = descs[di];
    if (active && !active[d.mol]) return;
    const int M = d.M, N = d.N, ksplit = d.ksplit, tiles_n = d.tiles_n;
    int local = (int)(tile - d.tile_start);               // a problem's tiles number below 2^31
    const int ks = local % ksplit;
    local /= ksplit;
    const int per_batch = d.tiles_m * tiles_n;
    const int bt = local / per_batch;
    local -= bt * per_batch;
    const int m0 = local / tiles_n * T, n0 = local % tiles_n * T;
    // K slice of this CTA (multiples of 16)
    const int kslice = ((d.K + ksplit - 1) / ksplit + 15) / 16 * 16;
    const int kbeg = ks * kslice, kend = min(d.K, kbeg + kslice);
    const double *__restrict__ A = d.A + (long long)bt * d.a[4];
    const double *__restrict__ B = d.B + (long long)bt * d.b[4];
    // K is contiguous for an operand when its inner k stride is 1 and it is the fast axis.
    const bool a_kfast = (d.a[3] == 1) || (d.a[1] != 1);
    const bool b_kfast = (d.b[3] == 1) || (d.b[1] != 1);
    const int Ki = d.Ki;
    const long long a2 = d.a[2], a3 = d.a[3], b2 = d.b[2], b3 = d.b[3];
    // this thread's rows of the operand tiles and their offsets (fixed over k)
    int am[R], ak[R], bn[R], bk[R];
    long long aoff[R], boff[R];
#pragma unroll
    for (int r = 0; r < R; ++r) {
        const int e = threadIdx.x + NT * r;
        if (a_kfast) { ak[r] = e % BK; am[r] = e / BK; } else { am[r] = e % T; ak[r] = e / T; }
        if (b_kfast) { bk[r] = e % BK; bn[r] = e / BK; } else { bn[r] = e % T; bk[r] = e / T; }
        aoff[r] = m0 + am[r] < M ? split_off(m0 + am[r], d.Mi, d.a[0], d.a[1]) : -1;
        boff[r] = n0 + bn[r] < N ? split_off(n0 + bn[r], d.Ni, d.b[0], d.b[1]) : -1;
    }
    double av[R], bv[R];
    auto fetch = [&](int k0) {
#pragma unroll
        for (int r = 0; r < R; ++r) {
            const int ka = k0 + ak[r], kb = k0 + bk[r];
            av[r] = (aoff[r] >= 0 && ka < kend) ? A[aoff[r] + split_off(ka, Ki, a2, a3)] : 0.0;
            bv[r] = (boff[r] >= 0 && kb < kend) ? B[boff[r] + split_off(kb, Ki, b2, b3)] : 0.0;
        }
    };
    // a warp computes T rows of 32 / T consecutive columns, for its group's k
    const int grp = threadIdx.x / (T * T), tid = threadIdx.x % (T * T);
    const int mm = tid % T, nn = tid / T;
    const bool live = n0 + (tid / 32) * (32 / T) < N;                  // uniform over the warp
    double acc = 0.0;
    fetch(kbeg);
    for (int k0 = kbeg; k0 < kend; k0 += BK) {
#pragma unroll
        for (int r = 0; r < R; ++r) { As[ak[r]][am[r]] = av[r]; Bs[bk[r]][bn[r]] = bv[r]; }
        __syncthreads();
        if (k0 + BK < kend) fetch(k0 + BK);
        if (live) {
            const int kb = grp * BKG, kn = min(BKG, kend - k0 - kb);
            if (kn == BKG) {
#pragma unroll
                for (int kk = 0; kk < BKG; ++kk) acc = fma(As[kb + kk][mm], Bs[kb + kk][nn], acc);
            } else {
#pragma unroll 4
                for (int kk = 0; kk < kn; ++kk) acc = fma(As[kb + kk][mm], Bs[kb + kk][nn], acc);
            }
        }
        __syncthreads();
    }
    if (G > 1) {                                              // the groups' sums in order
        double *red = &As[0][0];
        if (grp > 0) red[(grp - 1) * T * T + tid] = acc;
        __syncthreads();
        if (grp > 0) return;
#pragma unroll
        for (int g = 1; g < G; ++g) acc += red[(g - 1) * T * T + tid];
    }
    const int m = m0 + mm, n = n0 + nn;
    if (m >= M || n >= N) return;
    double *p = d.C + (long long)bt * d.c[4] + split_off(m, d.Mi, d.c[0], d.c[1]) + split_off(n, d.Ni, d.c[2], d.c[3]);
    double r = d.alpha * acc;
    if (ksplit > 1) { atomicAdd(p, r); return; }
    if (d.beta != 0.0) r += d.beta * *p;
    *p = r;
}

// Tiles of T x T outputs over the group, and the K slices of each problem:
// accumulating problems (beta = 1) whose output has few tiles but whose K is
// long are cut so that the launch reaches about two CTAs per SM.
long long layout(TgemmDesc *descs, int n, int T)
{
    long long start = 0;
    for (int i = 0; i < n; ++i) {
        TgemmDesc &d = descs[i];
        d.tiles_m = (d.M + T - 1) / T;
        d.tiles_n = (d.N + T - 1) / T;
        d.ksplit = 1;
        const long long out_tiles = (long long)d.batch * d.tiles_m * d.tiles_n;
        if (d.beta == 1.0 && d.K >= 512 && out_tiles < 304) {
            long long want = (304 + out_tiles - 1) / out_tiles;
            long long maxk = d.K / 128;
            d.ksplit = (int)std::max(1LL, std::min(want, maxk));
        }
        d.tile_start = start;
        if (d.M > 0 && d.N > 0 && d.batch > 0) start += out_tiles * d.ksplit;
    }
    return start;
}
}  // namespace

// Fill tiles/tile_start of the group on the host; returns the total tile count
// and the tile size: 8 when 16 x 16 tiles would leave SMs with fewer than two.
F64Tiles hx_tgemm_f64_prepare(TgemmDesc *descs, int n)
{
    F64Tiles t;
    t.size = 16;
    t.count = layout(descs, n, 16);
    if (t.count > 0 && t.count < 304) {
        t.size = 8;
        t.count = layout(descs, n, 8);
    }
    return t;
}

cudaError_t hx_tgemm_f64_launch(const TgemmDesc *d_descs, int n, F64Tiles tiles, const int *d_active, cudaStream_t s)
{
    if (tiles.count <= 0) return cudaSuccess;
    if (tiles.size == 8) tgemm_f64_kernel<8, 4><<<(unsigned)tiles.count, 256, 0, s>>>(d_descs, n, d_active);
    else tgemm_f64_kernel<16, 1><<<(unsigned)tiles.count, 256, 0, s>>>(d_descs, n, d_active);
    hx_count_launches(1);
    return cudaGetLastError();
}
