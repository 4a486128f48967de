// (T) triples correction of a converged closed-shell CCSD: the energy kernels.
//
// The spin-adapted form of the perturbative triples on spatial orbitals:
//   X_ijk^abc = sum_d (bd|ai) t_kj^cd - sum_l (ck|jl) t_il^ab
//   W_ijk^abc = X summed over the six simultaneous permutations of the pairs
//               (ia), (jb), (kc): twelve GEMMs per block of triples on the
//               tensor cores (hx_ccsd_triples in hx_engine.cu)
//   Z_ijk^abc = (jb|kc) t_i^a + (ia|kc) t_j^b + (ia|jb) t_k^c
//   Y_ijk^abc = 4 W_abc + W_bca + W_cab - 2 W_acb - 2 W_bac - 2 W_cba  (ijk fixed)
//   E[4] = sum W Y / (3 D),  E[5] = sum Z Y / (3 D),  D = e_i+e_j+e_k-e_a-e_b-e_c
// (k_t_energy), over the triples i <= j <= k, each weighted by its number of
// distinct permutations. E[4] + E[5] equals the spin-orbital (T) of the
// connected and disconnected triples amplitudes. One block per occupied
// triple, its threads over the virtual triples a >= b >= c: the FP64 pipe is
// the bound, and the six permutations of (a, b, c) share D and the sums
// P = W_abc + W_bca + W_cab, Q = W_acb + W_bac + W_cba (Y = 3W + P - 2Q on the
// first three, 3W + Q - 2P on the others): 9 FP64 operations per element
// instead of about 50 with two divisions each.
#include <algorithm>

#include "hx_common.cuh"
#include "hx_kernels.h"

namespace {
constexpr int TNT = 256;

__device__ __forceinline__ double t_warp_sum(double v)
{
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}

// Bvv0[mu][(b d)] = C_mu,o+b C_mu,o+d ; Boo0[mu][(j l)] = C_mu,j C_mu,l
__global__ void k_t_pairs(const double *__restrict__ C, int N, int o, double *__restrict__ Bvv0,
                          double *__restrict__ Boo0)
{
    const int v = N - o;
    const long long nvv = (long long)N * v * v, noo = (long long)N * o * o;
    for (long long e = (long long)blockIdx.x * blockDim.x + threadIdx.x; e < nvv + noo;
         e += (long long)gridDim.x * blockDim.x) {
        if (e < nvv) {
            const int mu = (int)(e / ((long long)v * v)), r = (int)(e % ((long long)v * v));
            Bvv0[e] = C[(long long)mu * N + o + r / v] * C[(long long)mu * N + o + r % v];
        } else {
            const long long f = e - nvv;
            const int mu = (int)(f / ((long long)o * o)), r = (int)(f % ((long long)o * o));
            Boo0[f] = C[(long long)mu * N + r / o] * C[(long long)mu * N + r % o];
        }
    }
}

// Per-block partials of 3 E[4] and 3 E[5] for one triple (i, j, k), i <= j <= k:
// the block's W_ijk^abc (v^3, [a][b][c]) sits in the slab at triple `blockIdx.x`;
// the triple counts w = 6, 3 or 1 times (its distinct permutations: the
// energy of a triple is unchanged by a simultaneous permutation of (ia),
// (jb), (kc)). abc: the nabc virtual triples a >= b >= c, packed 8 bits each.
__global__ void __launch_bounds__(TNT) k_t_energy(const double *__restrict__ W, const int3 *__restrict__ triples,
                                                  const unsigned *__restrict__ abc, int nabc,
                                                  const double *__restrict__ t1, const double *__restrict__ gov,
                                                  const double *__restrict__ Fmo, int N, int o, int v,
                                                  double *__restrict__ part)
{
    __shared__ double ev[256];
    const int i = triples[blockIdx.x].x, j = triples[blockIdx.x].y, k = triples[blockIdx.x].z;
    const int v2 = v * v;
    const long long ov = (long long)o * v;
    const double *Wb = W + (long long)blockIdx.x * v2 * v;
    // (jb|kc), (ia|kc), (ia|jb) as v x v blocks of gov, and the rows of t1
    const double *gjk = gov + (long long)j * v * ov + (long long)k * v, *gik = gov + (long long)i * v * ov + (long long)k * v,
                 *gij = gov + (long long)i * v * ov + (long long)j * v;
    const double *ti = t1 + (long long)i * v, *tj = t1 + (long long)j * v, *tk = t1 + (long long)k * v;
    for (int a = threadIdx.x; a < v; a += TNT) ev[a] = Fmo[(long long)(o + a) * N + o + a];
    __syncthreads();
    const double eijk = Fmo[(long long)i * N + i] + Fmo[(long long)j * N + j] + Fmo[(long long)k * N + k];
    const double wt = (i == j && j == k) ? 1.0 : ((i == j || j == k) ? 3.0 : 6.0);
    double e4 = 0.0, e5 = 0.0;
    for (int e = threadIdx.x; e < nabc; e += TNT) {
        const unsigned x = abc[e];
        const int a = x >> 16, b = (x >> 8) & 255, c = x & 255;
        // the six permutations (p, q, r) of (a, b, c): even ones first
        const int p[6] = {a, b, c, a, b, c}, q[6] = {b, c, a, c, a, b}, r[6] = {c, a, b, b, c, a};
        double w[6], s4 = 0.0, s5 = 0.0;
#pragma unroll
        for (int m = 0; m < 6; ++m) w[m] = Wb[(p[m] * v + q[m]) * v + r[m]];
        const double P = (w[0] + w[1]) + w[2], Q = (w[3] + w[4]) + w[5];
        const double ye = fma(-2.0, Q, P), yo = fma(-2.0, P, Q);
#pragma unroll
        for (int m = 0; m < 6; ++m) {
            const double y = fma(3.0, w[m], m < 3 ? ye : yo);
            double z = gjk[q[m] * ov + r[m]] * ti[p[m]];
            z = fma(gik[p[m] * ov + r[m]], tj[q[m]], z);
            z = fma(gij[p[m] * ov + q[m]], tk[r[m]], z);
            s4 = fma(w[m], y, s4);
            s5 = fma(z, y, s5);
        }
        // equal indices: the six permutations repeat the distinct ones two or six times
        const double rep = a == c ? 6.0 : (a == b || b == c) ? 2.0 : 1.0;
        const double d = 1.0 / (rep * (eijk - ((ev[a] + ev[b]) + ev[c])));
        e4 = fma(s4, d, e4);
        e5 = fma(s5, d, e5);
    }
    __shared__ double sh[2][TNT / 32];
    e4 = t_warp_sum(e4);
    e5 = t_warp_sum(e5);
    if ((threadIdx.x & 31) == 0) { sh[0][threadIdx.x >> 5] = e4; sh[1][threadIdx.x >> 5] = e5; }
    __syncthreads();
    if (threadIdx.x == 0) {
        double s4 = 0.0, s5 = 0.0;
        for (int w = 0; w < TNT / 32; ++w) { s4 += sh[0][w]; s5 += sh[1][w]; }
        part[2 * (long long)blockIdx.x] = wt * s4;
        part[2 * (long long)blockIdx.x + 1] = wt * s5;
    }
}

// ordered sum of the block partials (deterministic)
__global__ void k_t_final(const double *__restrict__ part, long long nblk, double *__restrict__ out)
{
    __shared__ double sh[2][32];
    double s4 = 0.0, s5 = 0.0;
#pragma unroll 8
    for (long long b = threadIdx.x; b < nblk; b += 32) { s4 += part[2 * b]; s5 += part[2 * b + 1]; }
    sh[0][threadIdx.x] = s4;
    sh[1][threadIdx.x] = s5;
    __syncthreads();
    if (threadIdx.x == 0) {
        double a = 0.0, b = 0.0;
        for (int t = 0; t < 32; ++t) { a += sh[0][t]; b += sh[1][t]; }
        out[0] = a / 3.0;
        out[1] = b / 3.0;
    }
}
}  // namespace

cudaError_t hx_triples_pairs(const double *C, int N, int o, double *Bvv0, double *Boo0, cudaStream_t s)
{
    const long long work = (long long)N * ((long long)(N - o) * (N - o) + (long long)o * o);
    const unsigned g = (unsigned)std::min<long long>((work + TNT - 1) / TNT, 4096);
    k_t_pairs<<<g, TNT, 0, s>>>(C, N, o, Bvv0, Boo0);
    hx_count_launches(1);
    return cudaGetLastError();
}

cudaError_t hx_triples_energy(const double *W, const int3 *triples, int ntriples, const unsigned *abc, int nabc,
                              const double *t1, const double *gov, const double *Fmo, int N, int o, double *part,
                              double *out, cudaStream_t s)
{
    k_t_energy<<<(unsigned)ntriples, TNT, 0, s>>>(W, triples, abc, nabc, t1, gov, Fmo, N, o, N - o, part);
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return e;
    k_t_final<<<1, 32, 0, s>>>(part, ntriples, out);
    hx_count_launches(2);
    return cudaGetLastError();
}
