// Elementwise, reduction and DIIS kernels of the CCSD iteration (FP64, HBM bound).
//
// All kernels are grouped over the molecules of a batch with a balanced
// schedule (HxSched, hx_plan.h): every molecule owns a run of blocks in
// proportion to its work, a block finds its molecule by binary search over
// the prefix sums, and blocks of molecules whose `active` flag is 0 return at
// once. Reductions are two-pass (fixed per-block partials, then an ordered
// sum per molecule), so repeated runs are bitwise identical.
//
// The amplitude tail of an iteration (stepCC, pushCCVectors, diisDotProduct,
// newCCVectors and energyCC; mod_cc.f90:987-1017, 1390-1423, 1514-1555,
// 2133-2193, 1916-1952) works on "pair units": v x v blocks [a][b] of the
// pair matrix for occupied pairs (i, j), staged in shared memory so that the
// (a, b) transposes the equations need are read and written coalesced.
//   k_step_push   residual assembly (r2, the C, D and E terms and their pair
//                 transposes), the Jacobi step, the push into the DIIS ring and
//                 the dots of the new error vector with every stored one, per unit;
//   k_diis_solve  per molecule: maxima, Gram row, bordered solve by one warp;
//   k_amplitudes_energy  t = sum c_k t_k written to both halves of t2 and the
//                 energy of the result (the last block sums the partials).
// Only the canonical blocks i <= j are stepped and stored, as the reference
// stores only the pairs (ia) <= (jb).
#include <mutex>

#include "hx_common.cuh"
#include "hx_plan.h"
#include "hx_kernels.h"
#include "hx_quotient.h"

namespace {
constexpr int NT = 256;

__device__ double warp_sum(double v)
{
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}
__device__ double warp_max(double v)
{
    for (int o = 16; o > 0; o >>= 1) v = fmax(v, __shfl_xor_sync(0xffffffffu, v, o));
    return v;
}
// block-wide reduction (sum or max) of blockDim.x == NT threads; the result is
// valid in thread 0 and the shared scratch may be reused after the call
__device__ double block_red(double v, bool mx)
{
    __shared__ double sh[NT / 32];
    v = mx ? warp_max(v) : warp_sum(v);
    int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    __syncthreads();
    if (lane == 0) sh[w] = v;
    __syncthreads();
    v = (threadIdx.x < NT / 32) ? sh[threadIdx.x] : 0.0;
    if (w == 0) v = mx ? warp_max(v) : warp_sum(v);
    return v;
}

// molecule of block b: the last m with start[m] <= b
__device__ __forceinline__ int sched_mol(const int *__restrict__ start, int nmol, int b)
{
    int lo = 0, hi = nmol - 1;
    while (lo < hi) {
        const int mid = (lo + hi + 1) >> 1;
        if (start[mid] <= b) lo = mid; else hi = mid - 1;
    }
    return lo;
}

// Element-wise kernels: block b of molecule mol covers HX_EW_CHUNK elements.
#define EW_PROLOGUE                                                                      \
    const int mol_ = sched_mol(start, nmol, blockIdx.x);                                 \
    if (active && !active[mol_]) return;                                                 \
    const CCMol &m = mols[mol_];                                                         \
    const long long base_ = (long long)(blockIdx.x - start[mol_]) * HX_EW_CHUNK;
#define EW_LOOP(e, n)                                                                    \
    for (long long e = base_ + threadIdx.x, end_ = min(base_ + HX_EW_CHUNK, (long long)(n)); e < end_; e += NT)
#define EW_ARGS const CCMol *__restrict__ mols, const int *__restrict__ active, const int *__restrict__ start, int nmol

// ---------------------------------------------------------------- dressing
// H2 = h - G o Pm + 2 diag(G diag Pm), Pm = Yo Xo^T (dressed half density)
__global__ void __launch_bounds__(NT) k_dress_fock(EW_ARGS)
{
    __shared__ double diag[HX_EW_CHUNK / 2 + 2];
    EW_PROLOGUE
    const int n = m.N;
    // the diagonal elements of this block's stretch: rows r0 .. r1 - 1, a warp per sum
    const long long end = min(base_ + HX_EW_CHUNK, (long long)n * n);
    const int r0 = (int)((base_ + n) / (n + 1)), r1 = (int)((end + n) / (n + 1));
    for (int i = r0 + (int)(threadIdx.x >> 5); i < r1; i += NT / 32) {
        double s = 0.0;
        for (int l = threadIdx.x & 31; l < n; l += 32) s += m.G[i * n + l] * m.Pm[l * n + l];
        s = warp_sum(s);
        if ((threadIdx.x & 31) == 0) diag[i - r0] = s;
    }
    __syncthreads();
    EW_LOOP(e, (long long)n * n) {
        const int i = (int)(e / n), j = (int)(e % n);
        double f = m.h[e] - m.G[e] * m.Pm[e];
        if (i == j) f += 2.0 * diag[i - r0];
        m.H2[e] = f;
    }
}

// ZDO pair products of the dressed factors.
__global__ void k_zdo_products(EW_ARGS)
{
    EW_PROLOGUE
    const int n = m.N, o = m.o, v = m.v;
    const long long nia = (long long)n * o * v, noo = (long long)n * o * o, nvv = (long long)n * v * v;
    EW_LOOP(e, nia + noo + nvv) {
        if (e < nia) {
            int mu = (int)(e / (o * v)), r = (int)(e % (o * v)), i = r / v, a = r % v;
            m.Bia[e] = m.X[mu * n + o + a] * m.Y[mu * n + i];
        } else if (e < nia + noo) {
            long long f = e - nia;
            int mu = (int)(f / (o * o)), r = (int)(f % (o * o)), k = r / o, i = r % o;
            m.Boo[f] = m.X[mu * n + k] * m.Y[mu * n + i];
        } else {
            long long f = e - nia - noo;
            int mu = (int)(f / (v * v)), r = (int)(f % (v * v)), a = r / v, c = r % v;
            m.Bvv[f] = m.X[mu * n + o + a] * m.Y[mu * n + o + c];
        }
    }
}

// Ts[i][mu][j][nu] *= G[mu][nu]  (a molecule's o N o N < 2^32 elements: 32-bit index arithmetic)
__global__ void k_gamma_scale(EW_ARGS)
{
    EW_PROLOGUE
    const unsigned n = (unsigned)m.N, no = n * (unsigned)m.o;
    double *__restrict__ Ts = m.Ts;
    const double *__restrict__ G = m.G;
    EW_LOOP(e, (long long)no * no) {
        const unsigned x = (unsigned)e;
        const unsigned nu = x % n, mu = (x / no) % n;
        Ts[e] *= G[mu * n + nu];
    }
}

// ---------------------------------------------------------------- pair units
// Units of one molecule: unit 0 is the singles; unit u >= 1 holds the v x v
// blocks [(u-1) g, min(u g, nb)) of the occupied pairs (i, j), in row-major
// order of the upper triangle i <= j (SK_UP) or of the whole o x o grid
// (SK_FULL), g = hx_unit_blocks(v). A unit's blocks sit in shared memory as
// [block][a][b] with rows padded to v + 1 (transposed reads spread over banks).
struct Unit {
    int mol, u, k0, nb;   // molecule, unit, first block, blocks in this unit
};

// (i, j) of block k of the upper triangle (row i starts at i o - i (i - 1) / 2)
__device__ __forceinline__ void up_block(int k, int o, int &i, int &j)
{
    const double s = 2.0 * o + 1.0;
    int r = (int)((s - sqrt(s * s - 8.0 * k)) * 0.5);
    r = r < 0 ? 0 : (r > o - 1 ? o - 1 : r);
    while (r > 0 && r * o - r * (r - 1) / 2 > k) --r;
    while (r + 1 < o && (r + 1) * o - (r + 1) * r / 2 <= k) ++r;
    i = r;
    j = r + (k - (r * o - r * (r - 1) / 2));
}

// This block's unit, and the (i, j) of its pair blocks in bi/bj (shared).
__device__ __forceinline__ Unit unit_of(const CCMol *mols, const int *start, int nmol, bool upper, int *bi, int *bj)
{
    Unit w;
    w.mol = sched_mol(start, nmol, blockIdx.x);
    w.u = blockIdx.x - start[w.mol];
    const CCMol &m = mols[w.mol];
    const int g = hx_unit_blocks(m.v);
    const int nbt = upper ? m.o * (m.o + 1) / 2 : m.o * m.o;
    w.k0 = w.u > 0 ? (w.u - 1) * g : 0;
    w.nb = w.u > 0 ? min(g, nbt - w.k0) : 0;
    for (int lb = threadIdx.x; lb < w.nb; lb += blockDim.x) {
        int i, j;
        if (upper) up_block(w.k0 + lb, m.o, i, j);
        else { i = (w.k0 + lb) / m.o; j = (w.k0 + lb) % m.o; }
        bi[lb] = i;
        bj[lb] = j;
    }
    __syncthreads();
    return w;
}

__device__ __forceinline__ long long pair_off(int i, int a, int j, int b, int o, int v)
{
    return (((long long)i * v + a) * o + j) * v + b;
}

// Tile loops of a unit: warp w walks the rows (block lb, row a) of the unit's
// tile, its lanes the columns b, so global reads and writes run along b (one
// division per row, none per element); shared-memory index of (lb, a, b) is
// (lb v + a)(v + 1) + b.
// A warp walks several rows at once with as many lanes per row (32, 16, 8 or 4;
// lg_: the log2) as leave the fewest idle, so that its FP64 slots are not spent
// on idle lanes (v = 80: 16 lanes x 5 instead of 32 x 3; v = 18: 8 x 3).
__device__ __forceinline__ int row_lanes(int v)
{
    int lg = 5, width = (v + 31) & ~31;
    for (int l = 4; l >= 2; --l) {
        const int w = (v + (1 << l) - 1) >> l << l;
        if (w < width && (l > 2 || v <= 4)) { width = w; lg = l; }
    }
    return lg;
}
#define ROW_LANES(v) const int lg_ = row_lanes(v);
#define ROW_LOOP(nrows) for (int row_ = threadIdx.x >> lg_; row_ < (nrows); row_ += NT >> lg_)
#define COL_LOOP(b, v) for (int b = threadIdx.x & ((1 << lg_) - 1); b < (v); b += 1 << lg_)

// K sums over the block at once (two barriers); valid in thread 0
template <int K>
__device__ __forceinline__ void block_sum_n(double (&x)[K])
{
    __shared__ double sh[K][NT / 32];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
#pragma unroll
    for (int k = 0; k < K; ++k) x[k] = warp_sum(x[k]);
    __syncthreads();
    if (lane == 0)
#pragma unroll
        for (int k = 0; k < K; ++k) sh[k][w] = x[k];
    __syncthreads();
#pragma unroll
    for (int k = 0; k < K; ++k) {
        x[k] = (threadIdx.x < NT / 32) ? sh[k][threadIdx.x] : 0.0;
        if (w == 0) x[k] = warp_sum(x[k]);
    }
}

// Eight sums over the block; thread q < 8 returns sum q. Each exchange of the
// warp stage halves the values a lane carries (9 FP64 adds per lane instead
// of 40: on GB300's FP64 pipe the full butterflies of 20 DIIS dots cost more
// than the dots of a 1024-element unit).
__device__ __forceinline__ double block_sum8(double (&x)[8])
{
    __shared__ double sh[8][NT / 32];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
#pragma unroll
    for (int n = 4, o = 16; n >= 1; n >>= 1, o >>= 1) {
        const bool up = (lane & o) != 0;
#pragma unroll
        for (int q = 0; q < n; ++q) {
            const double send = up ? x[q] : x[q + n], keep = up ? x[q + n] : x[q];
            x[q] = keep + __shfl_xor_sync(0xffffffffu, send, o);
        }
    }
    x[0] += __shfl_xor_sync(0xffffffffu, x[0], 2);
    x[0] += __shfl_xor_sync(0xffffffffu, x[0], 1);
    __syncthreads();
    if ((lane & 3) == 0) sh[lane >> 2][w] = x[0];      // bits 4, 3, 2 of the lane: values 4, 2, 1
    __syncthreads();
    double r = 0.0;
    if (threadIdx.x < 8)
#pragma unroll
        for (int k = 0; k < NT / 32; ++k) r += sh[threadIdx.x][k];
    return r;
}

// max of two magnitudes by their bit patterns (NaN ignored, as fmax does;
// integer compares instead of the FP64 pipe)
__device__ __forceinline__ double max_abs(double mx, double x)
{
    const unsigned long long b = (unsigned long long)__double_as_longlong(x) & 0x7FFFFFFFFFFFFFFFull;
    const unsigned long long m = (unsigned long long)__double_as_longlong(mx);
    return b > m && b <= 0x7FF0000000000000ull ? __longlong_as_double((long long)b) : mx;
}

// u[i][a][j][b] = 2 t[i][a][j][b] - t[i][b][j][a]  (SK_FULL units); a molecule's
// unit 0 starts its dressed factors, X = Y = [Co | Cv] (the t1 corrections are
// added by GEMMs).
__global__ void __launch_bounds__(NT) k_make_u(const CCMol *__restrict__ mols, const int *__restrict__ active,
                                               const int *__restrict__ start, int nmol)
{
    extern __shared__ double sm[];
    __shared__ int bi[64], bj[64];
    const Unit w = unit_of(mols, start, nmol, false, bi, bj);
    if (active && !active[w.mol]) return;
    const CCMol &m = mols[w.mol];
    if (w.u == 0) {
        for (int e = threadIdx.x; e < m.N * m.N; e += NT) { const double c = m.Cmo[e]; m.X[e] = c; m.Y[e] = c; }
        return;
    }
    const int o = m.o, v = m.v, nrows = w.nb * v;
    ROW_LANES(v)
    const double *__restrict__ t2 = m.t2;
    double *__restrict__ u = m.u;
#pragma unroll 4
    ROW_LOOP(nrows) {
        const int lb = row_ / v, a = row_ - lb * v;
        const double *src = t2 + pair_off(bi[lb], a, bj[lb], 0, o, v);
        double *srow = sm + (lb * v + a) * (v + 1);
        COL_LOOP(b, v) srow[b] = src[b];
    }
    __syncthreads();
#pragma unroll 4
    ROW_LOOP(nrows) {
        const int lb = row_ / v, a = row_ - lb * v;
        double *dst = u + pair_off(bi[lb], a, bj[lb], 0, o, v);
        const double *srow = sm + (lb * v + a) * (v + 1);
        COL_LOOP(b, v) dst[b] = 2.0 * srow[b] - sm[(lb * v + b) * (v + 1) + a];
    }
}

// Residual, Jacobi step and DIIS push of one unit (SK_UP units).
//   singles: d1 = r1 + r1b; t1 += s1 d1 / D1.
//   doubles of a block (i, j), i <= j: w = Omega2(ia, jb) assembled as
//     r2 + P + P pair-transposed, P_iajb = D_iajb + (E1 + E2)_iajb +
//     1/2 C_iajb + C_jaib (X2, Et and Cint, Cp), d2 = 2 w(ab) - w(ba)
//     (= w on a diagonal block, whose canonical element is the same for both);
//     g = 3 w ("2-1") or d2 ("1"); t2 += s2 g / D2 with the stored
//     reciprocal R2 = 1/D2 (stored_quotient).
// push = 1: (t, g) go into the ring slot count % nd and part gets the dots of
// g with every stored error vector. The error vector keeps the pair (ia, ib)
// of a diagonal block once (a <= b; the mirror element is stored as 0), so a
// plain dot is the reference's packed dot over (ia) <= (jb); t2 itself is
// written by k_amplitudes_energy. push = 0 (no DIIS): t1 and both halves of t2 are
// written here. part[0], part[1] = max|d1|, max|d2|.
__global__ void __launch_bounds__(NT) k_step_push(const CCMol *__restrict__ mols, const DiisMol *__restrict__ diis,
                                                  const int *__restrict__ active, const int *__restrict__ start,
                                                  int nmol, double s1, double s2, int proj, int push,
                                                  double *__restrict__ part)
{
    extern __shared__ double sm[];
    __shared__ int bi[64], bj[64];
    const Unit w = unit_of(mols, start, nmol, true, bi, bj);
    if (active && !active[w.mol]) return;
    const CCMol &m = mols[w.mol];
    const DiisMol &h = diis[w.mol];
    const int o = m.o, v = m.v, ov = o * v;
    double *P = part + (long long)blockIdx.x * HX_PART_STRIDE;
    const int cnt = push ? h.count[0] : 0;
    const int slot = push ? cnt % h.nd : 0, nvec = push ? min(cnt + 1, h.nd) : 0;
    double *__restrict__ t2 = m.t2;
    const double *__restrict__ X2 = m.X2;
    double *S = sm;                              // the assembled residual of the unit's blocks
    double mx = 0.0;
    long long hoff;
    const int nrows = w.nb * v;
    ROW_LANES(v)
    if (w.u == 0) {
        hoff = 0;
        for (int e = threadIdx.x; e < ov; e += NT) {
            const double d = m.r1[e] + m.r1b[e];
            mx = fmax(mx, fabs(d));
            const double t = m.t1[e] + s1 * d / m.D1[e];
            if (push) { h.Ht[(long long)slot * h.L + e] = t; h.He[(long long)slot * h.L + e] = d; }
            else m.t1[e] = t;
        }
    } else {
        hoff = ov + (long long)w.k0 * v * v;
        // S = r2 + (P + P[q][p]): element (a, b) of block (i, j) takes P[j][b][i][a],
        // read along a (coalesced) and added at the transposed tile position
        const double *__restrict__ Cp = m.Cp, *__restrict__ Et = m.Et, *__restrict__ E2 = m.Cint;
#pragma unroll 4
        ROW_LOOP(nrows) {
            const int lb = row_ / v, a = row_ - lb * v;
            const long long f = pair_off(bi[lb], a, bj[lb], 0, o, v), g = pair_off(bj[lb], a, bi[lb], 0, o, v);
            double *srow = S + (lb * v + a) * (v + 1);
            COL_LOOP(b, v) srow[b] = (X2[f + b] + (Et[f + b] + E2[f + b])) + fma(0.5, Cp[f + b], Cp[g + b]);
        }
        __syncthreads();
#pragma unroll 4
        ROW_LOOP(nrows) {
            const int lb = row_ / v, x = row_ - lb * v;              // x plays b, y plays a
            const long long f = pair_off(bj[lb], x, bi[lb], 0, o, v), g = pair_off(bi[lb], x, bj[lb], 0, o, v);
            COL_LOOP(y, v)
                S[(lb * v + y) * (v + 1) + x] += (X2[f + y] + (Et[f + y] + E2[f + y])) + fma(0.5, Cp[f + y], Cp[g + y]);
        }
        __syncthreads();
#pragma unroll 4
        ROW_LOOP(nrows) {
            const int lb = row_ / v, a = row_ - lb * v;
            const double *src = m.r2 + pair_off(bi[lb], a, bj[lb], 0, o, v);
            double *srow = S + (lb * v + a) * (v + 1);
            COL_LOOP(b, v) srow[b] = src[b] + srow[b];
        }
        __syncthreads();
        ROW_LOOP(nrows) {
            const int lb = row_ / v, a = row_ - lb * v, i = bi[lb], j = bj[lb];
            const double *srow = S + (lb * v + a) * (v + 1);
            const long long f0 = pair_off(i, a, j, 0, o, v);
            double *trow = t2 + f0;
            const double *Drow = m.D2 + f0, *Rrow = m.R2 + f0;
            const long long hrow = hoff + (long long)(lb * v + a) * v;
            COL_LOOP(b, v) {
                const double sab = srow[b], sba = S[(lb * v + b) * (v + 1) + a];
                double wv, d2;
                if (i < j) { wv = sab; d2 = 2.0 * sab - sba; }
                else { wv = a <= b ? sab : sba; d2 = wv; }
                mx = max_abs(mx, d2);
                const double g = proj == 1 ? d2 : 3.0 * wv, sg = s2 * g, R = Rrow[b];
                const double t = trow[b] + stored_quotient(sg, Drow[b], R);
                if (push) {
                    h.Ht[(long long)slot * h.L + hrow + b] = t;
                    // a diagonal block holds (ia, ib) and (ib, ia), the same pair: the
                    // error vector keeps it once (a <= b), so plain dots of stored error
                    // vectors are the reference's packed dots
                    h.He[(long long)slot * h.L + hrow + b] = (i == j && a > b) ? 0.0 : g;
                } else {
                    trow[b] = t;
                }
            }
        }
        __syncthreads();                         // (also makes the global writes above visible to the block)
        if (!push) {   // the mirror half: t2[j][b][i][a] = t2[i][a][j][b], a fastest (DIIS off only)
            ROW_LOOP(nrows) {
                const int lb = row_ / v, x = row_ - lb * v, i = bi[lb], j = bj[lb];   // x plays b
                if (i < j) {
                    double *dst = t2 + pair_off(j, x, i, 0, o, v);
                    COL_LOOP(y, v) dst[y] = t2[pair_off(i, y, j, x, o, v)];
                }
            }
        }
    }
    const double r = block_red(mx, true);
    if (threadIdx.x == 0) { P[0] = w.u == 0 ? r : 0.0; P[1] = w.u == 0 ? 0.0 : r; }
    // dots of the new error vector (just written, read back from L2) with every
    // stored one over the unit's contiguous stretch of the ring, eight stored
    // vectors per pass
    const int ne = w.u == 0 ? ov : w.nb * v * v;
    const double *En = h.He + (long long)slot * h.L + hoff;
    for (int k0 = 0; k0 < nvec; k0 += 8) {
        double acc[8] = {0.0, 0.0, 0.0, 0.0, 0.0, 0.0, 0.0, 0.0};
        const double *Ek[8];
#pragma unroll
        for (int q = 0; q < 8; ++q) Ek[q] = h.He + (long long)(k0 + q < nvec ? k0 + q : slot) * h.L + hoff;
#pragma unroll 2
        for (int e = threadIdx.x; e < ne; e += NT) {
            const double g = En[e];
#pragma unroll
            for (int q = 0; q < 8; ++q) acc[q] += g * Ek[q][e];
        }
        const double sum = block_sum8(acc);
        if (threadIdx.x < 8 && k0 + (int)threadIdx.x < nvec) P[2 + k0 + threadIdx.x] = sum;
    }
}

// ---------------------------------------------------------------- DIIS
// One block per molecule. The maxima of the units give res[0], res[1] (the
// reference's accuracy(1..2), before the step). gate[mol]: the DIIS step runs
// while max(|d1|,|d2|) >= gate[mol]. The reference stops mixing once the
// residual is below the convergence target (there the iteration ends); FP64
// iterations use that target, tensor-core iterations (which hand over rather
// than converge) their hand-over target. When it runs, the units' dots
// summed in a fixed order (strided per thread, then a fixed tree) form the
// Gram row of the new slot and the bordered system is solved by Gaussian
// elimination with partial pivoting; coef[HX_MAX_DIIS] = vectors to mix (1:
// none, t = the newest) and coef[HX_MAX_DIIS + 1] = the newest slot.
__global__ void __launch_bounds__(NT) k_diis_solve(const CCMol *__restrict__ mols, const DiisMol *__restrict__ diis,
                                                   const int *__restrict__ active, const int *__restrict__ start,
                                                   const double *gate, const double *__restrict__ part, int push)
{
    const int mol = blockIdx.x;
    if (active && !active[mol]) return;
    const CCMol &m = mols[mol];
    const int u0 = start[mol], u1 = start[mol + 1];
    __shared__ double ab[2];
    double a = 0.0, b = 0.0;
    for (int u = u0 + threadIdx.x; u < u1; u += NT) {
        a = fmax(a, part[(long long)u * HX_PART_STRIDE + 0]);
        b = fmax(b, part[(long long)u * HX_PART_STRIDE + 1]);
    }
    a = block_red(a, true);
    b = block_red(b, true);
    if (threadIdx.x == 0) { m.res[0] = a; m.res[1] = b; ab[0] = a; ab[1] = b; }
    __syncthreads();
    a = ab[0];
    b = ab[1];
    if (!push) return;
    const DiisMol &h = diis[mol];
    const int cnt = h.count[0];
    const int slot = cnt % h.nd, n = cnt + 1 < h.nd ? cnt + 1 : h.nd;
    if (!(fmax(a, b) >= gate[mol])) {                  // converged: the reference skips DIIS
        if (threadIdx.x == 0) { h.coef[HX_MAX_DIIS] = 1.0; h.coef[HX_MAX_DIIS + 1] = slot; }
        return;
    }
    __shared__ double g[HX_MAX_DIIS];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    for (int k = warp; k < n; k += NT / 32) {          // a warp per dot, no block barriers
        double s = 0.0;
        for (int u = u0 + lane; u < u1; u += 32) s += part[(long long)u * HX_PART_STRIDE + 2 + k];
        s = warp_sum(s);
        if (lane == 0) g[k] = s;
    }
    __syncthreads();
    for (int k = threadIdx.x; k < n; k += NT) {
        h.gram[slot * h.nd + k] = g[k];
        h.gram[k * h.nd + slot] = g[k];
    }
    if (threadIdx.x == 0) {
        h.count[0] = cnt + 1;
        h.coef[HX_MAX_DIIS + 1] = slot;
        h.coef[HX_MAX_DIIS] = 1.0;
    }
    if (n == 1) return;                                // newCCVectors(1) returns early
    // the bordered system [B 1; 1 0] c = e by Gaussian elimination with partial
    // pivoting in shared memory, the right-hand side as one more column, by one
    // warp (a lane per row, no block barriers): 21 pivots of a 21 x 21 system
    constexpr int MB = HX_MAX_DIIS + 1, LD = MB + 1 + (MB & 1);
    __shared__ double A[MB * LD];
    const int nb = n + 1;
    __syncthreads();
    for (int e = threadIdx.x; e < nb * (nb + 1); e += NT) {
        const int p = e / (nb + 1), q = e % (nb + 1);
        double val;
        if (q == nb) val = p == n ? 1.0 : 0.0;
        else if (p == n && q == n) val = 0.0;
        else if (p == n || q == n) val = 1.0;
        else val = (p == slot || q == slot) ? g[p == slot ? q : p] : h.gram[p * h.nd + q];
        A[p * LD + q] = val;
    }
    __syncthreads();
    if (warp != 0) return;
    for (int k = 0; k < nb; ++k) {
        // the first row of the largest magnitude, compared as bit patterns word by word
        // (two rows per lane at most; rows outside compare as zero)
        unsigned long long bb = 0;
        int br = k;
        for (int r = k + lane; r < nb; r += 32) {
            const unsigned long long x = (unsigned long long)__double_as_longlong(A[r * LD + k]) & 0x7FFFFFFFFFFFFFFFull;
            if (x > bb) { bb = x; br = r; }
        }
        const unsigned hi = __reduce_max_sync(0xffffffffu, (unsigned)(bb >> 32));
        const unsigned lo = __reduce_max_sync(0xffffffffu, (unsigned)(bb >> 32) == hi ? (unsigned)bb : 0u);
        const bool top = (unsigned)(bb >> 32) == hi && (unsigned)bb == lo;
        const int piv = (int)__reduce_min_sync(0xffffffffu, top && (hi | lo) ? (unsigned)br : (unsigned)nb);
        if (piv >= nb) return;                         // a zero column: singular, no mixing
        if (piv != k)
            for (int c = k + lane; c <= nb; c += 32) {
                const double t = A[k * LD + c];
                A[k * LD + c] = A[piv * LD + c];
                A[piv * LD + c] = t;
            }
        __syncwarp();
        const double d = A[k * LD + k];
        for (int r = k + 1 + lane; r < nb; r += 32) {
            const double f = A[r * LD + k] / d;
#pragma unroll 4
            for (int c = k + 1; c <= nb; ++c) A[r * LD + c] -= f * A[k * LD + c];
        }
        __syncwarp();
    }
    // back substitution by columns: once x_k is known every row above takes its share
    for (int k = nb - 1; k >= 0; --k) {
        const double xk = A[k * LD + nb] / A[k * LD + k];
        __syncwarp();
        for (int r = lane; r < k; r += 32) A[r * LD + nb] -= A[r * LD + k] * xk;
        if (lane == 0) A[k * LD + nb] = xk;
        __syncwarp();
    }
    bool ok = true;
    for (int k = lane; k < n; k += 32) ok = ok && isfinite(A[k * LD + nb]);
    if (!__all_sync(0xffffffffu, ok)) return;          // singular subspace: no mixing
    for (int k = lane; k < n; k += 32) h.coef[k] = A[k * LD + nb];
    if (lane == 0) h.coef[HX_MAX_DIIS] = (double)n;
}

// ---------------------------------------------------------------- amplitudes and energy
// energyCC r-ccsd of the unit: part[0] = sum F_ia t_ia (singles unit),
// part[1] = the unit's share of sum L (t2 + t1 t1), where element (a, b) of
// block (i, j), i <= j, counts twice when i < j (it and its mirror) and once
// on a diagonal block. With DIIS (from != 0) the amplitudes come from the
// ring -- the newest vector, or sum_k c_k Ht[k] in slot order -- and are
// written to t1 and both halves of t2; without, they are read from t1, t2.
__global__ void __launch_bounds__(NT) k_amplitudes_energy(const CCMol *__restrict__ mols,
                                                          const DiisMol *__restrict__ diis,
                                                          const int *__restrict__ active,
                                                          const int *__restrict__ start, int nmol, int from,
                                                          double *__restrict__ part)
{
    extern __shared__ double sm[];
    __shared__ int bi[64], bj[64];
    __shared__ double cf[HX_MAX_DIIS];
    const Unit w = unit_of(mols, start, nmol, true, bi, bj);
    if (active && !active[w.mol]) return;
    const CCMol &m = mols[w.mol];
    const DiisMol &h = diis[w.mol];
    const int o = m.o, v = m.v, n = m.N, ov = o * v;
    const int nmix = from ? (int)h.coef[HX_MAX_DIIS] : 0, slot = from ? (int)h.coef[HX_MAX_DIIS + 1] : 0;
    for (int k = threadIdx.x; k < nmix; k += NT) cf[k] = h.coef[k];
    __syncthreads();
    const double *__restrict__ Ht = h.Ht;
    const long long L = h.L;
    auto combine = [&](long long e) {
        if (nmix <= 1) return Ht[(long long)slot * L + e];
        double s = 0.0;
#pragma unroll 4
        for (int k = 0; k < nmix; ++k) s += cf[k] * Ht[(long long)k * L + e];
        return s;
    };
    double *P = part + (long long)blockIdx.x * HX_PART_STRIDE;
    double acc = 0.0;
    double *__restrict__ t2 = m.t2;
    if (w.u == 0) {
        for (int e = threadIdx.x; e < ov; e += NT) {
            const double t = from ? combine(e) : m.t1[e];
            if (from) m.t1[e] = t;
            acc += m.Fmo[(e / v) * n + o + e % v] * t;
        }
    } else {
        // this unit's t1 rows i and j (from the ring: t1 is being written by unit 0)
        double *T1 = sm + hx_unit_tile(o, v);            // [block][2][v]
        for (int e = threadIdx.x; e < w.nb * 2 * v; e += NT) {
            const int lb = e / (2 * v), r = e % (2 * v), a = r % v, row = r < v ? bi[lb] : bj[lb];
            T1[e] = from ? combine((long long)row * v + a) : m.t1[row * v + a];
        }
        __syncthreads();
        const int nrows = w.nb * v;
        ROW_LANES(v)
        const long long hoff = ov + (long long)w.k0 * v * v;
#pragma unroll 2
        ROW_LOOP(nrows) {
            const int lb = row_ / v, a = row_ - lb * v, i = bi[lb], j = bj[lb];
            const long long f0 = pair_off(i, a, j, 0, o, v);
            double *trow = t2 + f0;
            const double *Lrow = m.Lov + f0;
            const double t1a = T1[lb * 2 * v + a];
            const long long hrow = hoff + (long long)(lb * v + a) * v;
            double *srow = sm + (lb * v + a) * (v + 1);
            COL_LOOP(b, v) {
                double t;
                if (from) {
                    t = combine(hrow + b);
                    trow[b] = t;
                    srow[b] = t;
                } else {
                    t = trow[b];
                }
                const double s = Lrow[b] * (t + t1a * T1[lb * 2 * v + v + b]);
                acc += i < j ? 2.0 * s : s;
            }
        }
        if (from) {
            __syncthreads();
            ROW_LOOP(nrows) {
                const int lb = row_ / v, x = row_ - lb * v, i = bi[lb], j = bj[lb];   // x plays b
                if (i < j) {
                    double *dst = t2 + pair_off(j, x, i, 0, o, v);
                    COL_LOOP(y, v) dst[y] = sm[(lb * v + y) * (v + 1) + x];
                }
            }
        }
    }
    const double r = block_red(acc, false);
    // E = 2 sum F_ia t_ia + sum_(ia),(jb) L(ia,jb) (t2 + t1 t1)   (energyCC r-ccsd):
    // the molecule's last block sums the units' partials in a fixed order
    // (strided per thread, fixed tree); the counter wraps to zero for the next launch
    __shared__ bool last;
    const int u0 = start[w.mol], u1 = start[w.mol + 1];
    if (threadIdx.x == 0) {
        P[0] = w.u == 0 ? r : 0.0;
        P[1] = w.u == 0 ? 0.0 : r;
        __threadfence();
        last = atomicInc(h.done, (unsigned)(u1 - u0 - 1)) == (unsigned)(u1 - u0 - 1);
    }
    __syncthreads();
    if (!last) return;
    __threadfence();
    double x[2] = {0.0, 0.0};
    for (int u = u0 + threadIdx.x; u < u1; u += NT) {
        x[0] += __ldcg(part + (long long)u * HX_PART_STRIDE + 0);
        x[1] += __ldcg(part + (long long)u * HX_PART_STRIDE + 1);
    }
    block_sum_n<2>(x);
    if (threadIdx.x != 0) return;
    m.res[2] = 2.0 * x[0] + x[1] + m.eref;
    m.res[3] = m.eref;
    m.res[4] = 2.0 * x[0];
    m.res[5] = x[1];
}

// ---------------------------------------------------------------- amplitude layouts
// Between the reference's t1(o, v), t2(o, o, v, v) (column-major; a staging
// copy on the device) and the engine's t1 [i][a], t2 [i][a][j][b]: for fixed
// (j, a) an o x v transpose between i (contiguous in the column-major array)
// and b (contiguous in the pair layout), in 32 x 32 tiles through shared
// memory, so that both sides are read and written along their contiguous
// dimension. HBM bound: 32 bytes per element moved, 0.05 ms for 56^4 elements
// where the host's transpose took 20 ms. Block 0 also transposes t1.
constexpr int LT = 32;
template <bool TO_ENGINE>
__global__ void __launch_bounds__(256) k_layout(double *__restrict__ t1, double *__restrict__ t2,
                                                double *__restrict__ f1, double *__restrict__ f2, int o, int v)
{
    __shared__ double s[LT][LT + 1];
    const int ti = (o + LT - 1) / LT, tb = (v + LT - 1) / LT;
    unsigned x = blockIdx.x;
    const int b0 = (int)(x % tb) * LT;
    x /= tb;
    const int i0 = (int)(x % ti) * LT;
    x /= ti;
    const int j = (int)(x % o), a = (int)(x / o);
    const long long ov = (long long)o * v, vov = v * ov, oo = (long long)o * o, oov = oo * v;
    double *__restrict__ e = t2 + a * ov + (long long)j * v;                 // [i][.][.][b]
    double *__restrict__ f = f2 + (long long)j * o + a * oo;                 // (i, ., ., b)
    const int tx = threadIdx.x & 31, ty = threadIdx.x >> 5;
    for (int r = ty; r < LT; r += 8) {
        if (TO_ENGINE) {
            if (b0 + r < v && i0 + tx < o) s[tx][r] = f[i0 + tx + (b0 + r) * oov];
        } else {
            if (i0 + r < o && b0 + tx < v) s[r][tx] = e[(i0 + r) * vov + b0 + tx];
        }
    }
    __syncthreads();
    for (int r = ty; r < LT; r += 8) {
        if (TO_ENGINE) {
            if (i0 + r < o && b0 + tx < v) e[(i0 + r) * vov + b0 + tx] = s[r][tx];
        } else {
            if (b0 + r < v && i0 + tx < o) f[i0 + tx + (b0 + r) * oov] = s[tx][r];
        }
    }
    if (blockIdx.x == 0)
        for (int k = threadIdx.x; k < o * v; k += 256) {
            const int p = k / v + o * (k % v);
            if (TO_ENGINE) t1[k] = f1[p];
            else f1[p] = t1[k];
        }
}

// ---------------------------------------------------------------- Jacobian products
// The four points t +- h r, t +- 2 h r of each vector's stencil, into the
// amplitudes of molecules 4q .. 4q + 3 (blockIdx.z = q). t and r come as
// staging copies on the device, column-major (o, o, v, v) (order 0) or
// row-major [i][j][a][b] (order 1); tiles as k_layout's.
__device__ __forceinline__ double stage_at(const double *__restrict__ f, int order, int i, int j, int a, int b, int o, int v)
{
    return order ? f[(((long long)i * o + j) * v + a) * v + b]
                 : f[i + (long long)o * j + (long long)o * o * a + (long long)o * o * v * b];
}
__device__ __forceinline__ void stencil_points(double t, double r, double h, double (&x)[4])
{
    const double hr = h * r, h2 = hr + hr;
    x[0] = t + hr;
    x[1] = t - hr;
    x[2] = t + h2;
    x[3] = t - h2;
}
__global__ void __launch_bounds__(256) k_jacobian_points(const CCMol *__restrict__ mols, const double *__restrict__ t1s,
                                                         const double *__restrict__ t2s, int t_order,
                                                         const int *__restrict__ r_order, double h, int o, int v)
{
    __shared__ double st[LT][LT + 1], sr[LT][LT + 1];
    const int q = blockIdx.z, ti = (o + LT - 1) / LT, tb = (v + LT - 1) / LT, ro = r_order[q];
    unsigned x = blockIdx.x;
    const int b0 = (int)(x % tb) * LT;
    x /= tb;
    const int i0 = (int)(x % ti) * LT;
    x /= ti;
    const int j = (int)(x % o), a = (int)(x / o);
    const CCMol *m = mols + 4 * q;
    const double *r1s = m[0].U, *r2s = m[0].Cp;
    const int tx = threadIdx.x & 31, ty = threadIdx.x >> 5;
    // both into [i][b]: a column-major array is read along i, a row-major one along b
    for (int w = 0; w < 2; ++w) {
        const double *f = w ? r2s : t2s;
        const int order = w ? ro : t_order;
        double (*s)[LT + 1] = w ? sr : st;
        for (int y = ty; y < LT; y += 8) {
            const int i = order ? i0 + y : i0 + tx, b = order ? b0 + tx : b0 + y;
            if (i < o && b < v) s[i - i0][b - b0] = stage_at(f, order, i, j, a, b, o, v);
        }
    }
    __syncthreads();
    for (int y = ty; y < LT; y += 8) {
        const int i = i0 + y, b = b0 + tx;
        if (i >= o || b >= v) continue;
        double p[4];
        stencil_points(st[y][tx], sr[y][tx], h, p);
        const long long e = pair_off(i, a, j, b, o, v);
#pragma unroll
        for (int k = 0; k < 4; ++k) m[k].t2[e] = p[k];
    }
    if (blockIdx.x == 0)
        for (int e = threadIdx.x; e < o * v; e += 256) {
            const int f = e / v + o * (e % v);
            double p[4];
            stencil_points(t1s[t_order ? e : f], r1s[ro ? e : f], h, p);
            for (int k = 0; k < 4; ++k) m[k].t1[e] = p[k];
        }
}
// J r = [8 (W(+h) - W(-h)) - (W(+2h) - W(-2h))] / 12 h of the residuals W that
// the step left in the DIIS error slots (d1, and g = 3 W2 of the canonical
// blocks i <= j), row-major into U and X2 of molecule 4q. Block = one pair
// (i, j), i <= j, of vector blockIdx.y; both (i, j, a, b) and its mirror
// (j, i, b, a) are written, the transpose through shared memory.
__global__ void __launch_bounds__(256) k_jacobian_sum(const CCMol *__restrict__ mols, const DiisMol *__restrict__ diis, double h,
                                                      int o, int v)
{
    __shared__ double s[LT][LT + 1];
    const int q = blockIdx.y, ov = o * v;
    const CCMol &m = mols[4 * q];
    const double *E[4];
#pragma unroll
    for (int k = 0; k < 4; ++k) E[k] = diis[4 * q + k].He;
    auto sum = [&](long long e) { return 8.0 * (E[0][e] - E[1][e]) - (E[2][e] - E[3][e]); };
    int i, j;
    up_block(blockIdx.x, o, i, j);
    const long long base = ov + (long long)blockIdx.x * v * v;
    double *__restrict__ J2 = m.X2;
    const int tx = threadIdx.x & 31, ty = threadIdx.x >> 5;
    for (int a0 = 0; a0 < v; a0 += LT)
        for (int b0 = 0; b0 < v; b0 += LT) {
            __syncthreads();
            for (int y = ty; y < LT; y += 8) {
                const int a = a0 + y, b = b0 + tx;
                if (a >= v || b >= v) continue;
                const long long e = (i == j && a > b) ? base + (long long)b * v + a : base + (long long)a * v + b;
                const double d = sum(e) / (36.0 * h);
                s[y][tx] = d;
                J2[(((long long)i * o + j) * v + a) * v + b] = d;
            }
            __syncthreads();
            if (i < j)
                for (int y = ty; y < LT; y += 8) {
                    const int b = b0 + y, a = a0 + tx;
                    if (a < v && b < v) J2[(((long long)j * o + i) * v + b) * v + a] = s[tx][y];
                }
        }
    if (blockIdx.x == 0)
        for (int e = threadIdx.x; e < ov; e += 256) m.U[e] = sum(e) / (12.0 * h);
}

// ---------------------------------------------------------------- set-up
// Constants after SCF: denominators, ZDO vectors of the undressed ov space,
// and the reference guess (guessCC r-ccsd, mod_cc.f90:634-650) when asked.
__global__ void k_setup(EW_ARGS)
{
    EW_PROLOGUE
    const int n = m.N, o = m.o, v = m.v;
    const long long ov = (long long)o * v;
    EW_LOOP(e, ov + ov * ov + (long long)n * ov) {
        if (e < ov) {
            int i = (int)(e / v), a = (int)(e % v);
            m.D1[e] = m.Fmo[i * n + i] - m.Fmo[(o + a) * n + o + a];
        } else if (e < ov + ov * ov) {
            long long f = e - ov;
            int b = (int)(f % v);
            long long r = f / v;
            int j = (int)(r % o); r /= o;
            int a = (int)(r % v);
            int i = (int)(r / v);
            // grouped so that (ia),(jb) and (jb),(ia) round identically
            const double d = (m.Fmo[i * n + i] + m.Fmo[j * n + j]) - (m.Fmo[(o + a) * n + o + a] + m.Fmo[(o + b) * n + o + b]);
            m.D2[f] = d;
            m.R2[f] = 1.0 / d;
        } else {
            long long f = e - ov - ov * ov;
            int mu = (int)(f / ov), r = (int)(f % ov), k = r / v, c = r % v;
            m.Bov0[f] = m.Cmo[mu * n + k] * m.Cmo[mu * n + o + c];
        }
    }
}

// Lov = 2 gov - gov(ab swapped); t1, t2 = reference guess (when guess != 0)
__global__ void k_setup2(EW_ARGS, int guess)
{
    EW_PROLOGUE
    const int n = m.N, o = m.o, v = m.v;
    const long long ov = (long long)o * v;
    EW_LOOP(e, ov * ov) {
        int b = (int)(e % v);
        long long r = e / v;
        int j = (int)(r % o); r /= o;
        int a = (int)(r % v);
        int i = (int)(r / v);
        // canonical (upper-triangle) values: the guess and L are exactly pair-symmetric
        const long long p1 = (long long)i * v + a, q1 = (long long)j * v + b;
        const long long p2 = (long long)i * v + b, q2 = (long long)j * v + a;
        double g = m.gov[min(p1, q1) * ov + max(p1, q1)];
        double gx = m.gov[min(p2, q2) * ov + max(p2, q2)];
        double L = 2.0 * g - gx;
        m.Lov[e] = L;
        if (guess) m.t2[e] = L / m.D2[e];     // R(i,a,j,b) / (F_ii+F_jj-F_aa-F_bb)
        if (guess && e < ov) {
            int ii = (int)(e / v), aa = (int)(e % v);
            m.t1[e] = m.Fmo[ii * n + o + aa] / m.D1[e];
        }
    }
}
}  // namespace

// ---------------------------------------------------------------- launchers
#define LAUNCH_EW(kern, kind, ...)                                                                  \
    do {                                                                                            \
        if (S.blocks[kind] > 0)                                                                     \
            kern<<<(unsigned)S.blocks[kind], NT, 0, s>>>(m, act, S.start[kind], S.nmol, ##__VA_ARGS__); \
        hx_count_launches(1);                                                                       \
        cudaError_t e_ = cudaGetLastError();                                                        \
        if (e_ != cudaSuccess) return e_;                                                           \
    } while (0)

cudaError_t hx_ew_dress_fock(const CCMol *m, const int *act, const HxSched &S, cudaStream_t s)
{ LAUNCH_EW(k_dress_fock, SK_NN); return cudaSuccess; }
cudaError_t hx_ew_zdo_products(const CCMol *m, const int *act, const HxSched &S, cudaStream_t s)
{ LAUNCH_EW(k_zdo_products, SK_ZDO); return cudaSuccess; }
cudaError_t hx_ew_gamma_scale(const CCMol *m, const int *act, const HxSched &S, cudaStream_t s)
{ LAUNCH_EW(k_gamma_scale, SK_ONON); return cudaSuccess; }
cudaError_t hx_ew_setup(const CCMol *m, const int *act, const HxSched &S, cudaStream_t s)
{ LAUNCH_EW(k_setup, SK_SETUP); return cudaSuccess; }
cudaError_t hx_ew_setup2(const CCMol *m, const int *act, const HxSched &S, int guess, cudaStream_t s)
{ LAUNCH_EW(k_setup2, SK_PAIR, guess); return cudaSuccess; }

cudaError_t hx_layout(double *t1, double *t2, double *f1, double *f2, int o, int v, bool to_engine, cudaStream_t s)
{
    const unsigned g = (unsigned)o * v * ((o + LT - 1) / LT) * ((v + LT - 1) / LT);
    if (to_engine) k_layout<true><<<g, 256, 0, s>>>(t1, t2, f1, f2, o, v);
    else k_layout<false><<<g, 256, 0, s>>>(t1, t2, f1, f2, o, v);
    hx_count_launches(1);
    return cudaGetLastError();
}

cudaError_t hx_jacobian_points(const CCMol *m, int nvec, const double *t1, const double *t2, int t_order, const int *r_order,
                               double h, int o, int v, cudaStream_t s)
{
    const dim3 g((unsigned)o * v * ((o + LT - 1) / LT) * ((v + LT - 1) / LT), 1, (unsigned)nvec);
    k_jacobian_points<<<g, 256, 0, s>>>(m, t1, t2, t_order, r_order, h, o, v);
    hx_count_launches(1);
    return cudaGetLastError();
}
cudaError_t hx_jacobian_sum(const CCMol *m, const DiisMol *d, int nvec, double h, int o, int v, cudaStream_t s)
{
    k_jacobian_sum<<<dim3((unsigned)(o * (o + 1) / 2), (unsigned)nvec), 256, 0, s>>>(m, d, h, o, v);
    hx_count_launches(1);
    return cudaGetLastError();
}

// dynamic shared memory of the pair-unit kernels (bytes): the largest over the batch
size_t hx_unit_smem(const int *o, const int *v, int nmol, int kernel)
{
    long long mx = 0;
    for (int k = 0; k < nmol; ++k) {
        const long long t = hx_unit_tile(o[k], v[k]);
        long long need = t;                                                 // k_make_u
        if (kernel == 1) need = t;                                          // k_step_push
        if (kernel == 2) need = t + 2LL * hx_unit_blocks(v[k]) * v[k];      // k_amplitudes_energy
        mx = need > mx ? need : mx;
    }
    return (size_t)mx * sizeof(double);
}

// The attribute belongs to the kernel, not to a handle: it is only ever
// raised, so that a handle of small molecules does not take it from under one
// of large molecules made before.
cudaError_t hx_unit_kernels_init(size_t smem_max)
{
    static std::mutex mu;
    std::lock_guard<std::mutex> lock(mu);
    const void *kernels[] = {(const void *)k_make_u, (const void *)k_step_push, (const void *)k_amplitudes_energy};
    for (const void *k : kernels) {
        cudaFuncAttributes a;
        cudaError_t e = cudaFuncGetAttributes(&a, k);
        if (e == cudaSuccess && (size_t)a.maxDynamicSharedSizeBytes < smem_max)
            e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem_max);
        if (e != cudaSuccess) return e;
    }
    return cudaSuccess;
}

cudaError_t hx_ew_make_u(const CCMol *m, const int *act, const HxSched &S, size_t smem, cudaStream_t s)
{
    k_make_u<<<(unsigned)S.blocks[SK_FULL], NT, smem, s>>>(m, act, S.start[SK_FULL], S.nmol);
    hx_count_launches(1);
    return cudaGetLastError();
}

// stepCC + pushCCVectors + diisDotProduct + newCCVectors + energyCC of every active molecule
cudaError_t hx_tail(const CCMol *m, const DiisMol *h, const int *act, const HxSched &S, const size_t smem[2],
                    double s1, double s2, int proj, int use_diis, const double *gate, double *part, cudaStream_t s)
{
    k_step_push<<<(unsigned)S.blocks[SK_UP], NT, smem[0], s>>>(m, h, act, S.start[SK_UP], S.nmol, s1, s2, proj,
                                                               use_diis, part);
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return e;
    k_diis_solve<<<S.nmol, NT, 0, s>>>(m, h, act, S.start[SK_UP], gate, part, use_diis);
    if ((e = cudaGetLastError()) != cudaSuccess) return e;
    k_amplitudes_energy<<<(unsigned)S.blocks[SK_UP], NT, smem[1], s>>>(m, h, act, S.start[SK_UP], S.nmol, use_diis,
                                                                       part);
    hx_count_launches(3);
    return cudaGetLastError();
}

// energyCC of every (active) molecule from its current amplitudes
cudaError_t hx_energy(const CCMol *m, const DiisMol *h, const int *act, const HxSched &S, size_t smem, double *part,
                      cudaStream_t s)
{
    k_amplitudes_energy<<<(unsigned)S.blocks[SK_UP], NT, smem, s>>>(m, h, act, S.start[SK_UP], S.nmol, 0, part);
    hx_count_launches(1);
    return cudaGetLastError();
}
