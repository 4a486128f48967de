// PPP-RHF on the GPU in FP64: the whole SCF of a molecule in one launch, by a
// cluster of CTAs (one CTA up to kBlockN sites).
//
// Iteration of helios's SCF (src/methods/mod_scf.f90:106-136):
//   Fmin = (F R - R F) R,  R = 2D - 1          (prepareFmin :446-494)
//   accuracy = max|Fmin|
//   D -= (iter-step) Fmin;  F = fock(D)        (prepareFockian :417-442)
//   diagonalise F; D = aufbau(V); F = fock(D)
// with the generic iterator's stop rules (src/calculation/gIterator.f90:88-210).
// The guess diagonalises huckelCore (guessSCF :351-386) unless a density is given.
//
// Diagonalisation is a cyclic two-sided Jacobi method with the round-robin
// (circle) ordering, so the N/2 rotations of a round are disjoint and run in
// parallel. It works on A = V^T F V in the current orbital basis (warm start:
// the basis of the previous iteration already nearly diagonalises F) and
// accumulates the rotations into V. Eigenpairs are then sorted ascending, as
// the reference's tred4 returns them (src/modules/mod_math.f90:31-230).
//
// What bounds it: GB300's FP64 pipe (two multiply-adds per clock and SM) and
// the barrier of every Jacobi round. So
//  * a molecule is shared by a cluster of CTAs (16 or 8 SMs' FP64 pipes, the
//    cluster barrier instead of a grid-wide one); at most kBlockN sites run in
//    one CTA with every matrix in shared memory;
//  * a round is one pass: the rotated matrix is written to a second buffer, as
//    2 x 2 blocks J_k^T A J_l of its upper triangle, so a round has one barrier
//    and every CTA derives the next round's rotations from the finished matrix;
//  * the SCF iterations take the rotation angle in FP32 (a tangent within 1e-6
//    of the exact one leaves an off-diagonal 1e-6 of its size, which the
//    following sweeps remove: every diagonalisation ends at FP64's resolution);
//    its cosine is brought to FP64 by one third-order Newton step on
//    1/sqrt(1 + t^2), so the rotation is orthogonal to FP64. Against FP64 angles
//    the results are no less accurate (12 to 160 sites, after 1 to 10
//    iterations: density within 5e-14 of numpy's, 3e-13 with FP64 angles;
//    C^T C within 6e-14 of 1 at 160 sites, 3e-13). Diagonalising early
//    iterations to less (a millionth of their accuracy) saved 5 to 10 % of the
//    SCF and left 6e-10 in the orbitals of one that stops at its iteration limit;
//  * pairs far below FP64's resolution of the matrix are not rotated;
//  * V's rows stay in shared memory, and a round's matrix elements are fetched
//    while its angles are computed.
// Measured on whole calls, one CTA (a cooperative grid for one molecule above
// 64 sites) with three barriers a round before: a 38-site energy 88 -> 75 ms,
// 63 sites 182 -> 143 ms, 160 sites 1672 -> 1591 ms, a batch of 128 molecules
// of 8-64 sites 1077 -> 984 ms.
//
// The SCF body is written once over an execution context (BlockCtx, one CTA;
// ClusterCtx, a thread-block cluster).
#include <algorithm>
#include <cooperative_groups.h>
#include "hx_common.cuh"
#include "hx_plan.h"

namespace {
namespace cg = cooperative_groups;
constexpr int NT = 256;
constexpr int kBlockN = 24;      // largest molecule of the one-CTA, shared-memory form

// ---- execution contexts -------------------------------------------------
// two sums (or one maximum in a) over the CTA, valid in every thread
__device__ __forceinline__ void block_reduce(double &a, double &b, bool mx, double *sh)
{
    for (int o = 16; o > 0; o >>= 1) {
        const double x = __shfl_xor_sync(0xffffffffu, a, o), y = __shfl_xor_sync(0xffffffffu, b, o);
        a = mx ? fmax(a, x) : a + x;
        b += y;
    }
    const int wid = threadIdx.x >> 5;
    __syncthreads();
    if ((threadIdx.x & 31) == 0) { sh[wid] = a; sh[NT / 32 + wid] = b; }
    __syncthreads();
    a = sh[0];
    b = sh[NT / 32];
    for (int w = 1; w < NT / 32; ++w) { a = mx ? fmax(a, sh[w]) : a + sh[w]; b += sh[NT / 32 + w]; }
    __syncthreads();
}

struct BlockCtx {
    int tid, nt, rank = 0, size = 1;
    double *sh;          // 2 NT / 32 doubles of shared scratch
    __device__ explicit BlockCtx(double *s) : tid(threadIdx.x), nt(NT), sh(s) {}
    __device__ void sync() { __syncthreads(); }
    __device__ void reduce2(double &a, double &b, bool mx) { block_reduce(a, b, mx, sh); }
    __device__ static double ld(const double *p) { return *p; }
};

struct ClusterCtx {
    int tid, nt, rank, size;
    double *sh;          // shared scratch of this CTA
    double *gpart;       // 4 x cluster size global partials of this cluster
    int parity = 0;
    __device__ ClusterCtx(double *s, double *gp)
        : rank((int)cg::this_cluster().block_rank()), size((int)cg::this_cluster().num_blocks()), sh(s), gpart(gp)
    {
        tid = rank * NT + threadIdx.x;
        nt = size * NT;
    }
    __device__ void sync() { cg::this_cluster().sync(); }
    __device__ void reduce2(double &a, double &b, bool mx)
    {
        block_reduce(a, b, mx, sh);
        double *p = gpart + parity * 2 * size;          // two sets: the next reduction writes the other one
        parity ^= 1;
        if (threadIdx.x == 0) { __stcg(p + 2 * rank, a); __stcg(p + 2 * rank + 1, b); }
        sync();
        a = __ldcg(p);
        b = __ldcg(p + 1);
        for (int k = 1; k < size; ++k) {                // the same ordered sums in every thread
            const double x = __ldcg(p + 2 * k), y = __ldcg(p + 2 * k + 1);
            a = mx ? fmax(a, x) : a + x;
            b += y;
        }
    }
    // matrices another CTA of the cluster wrote are read from L2
    __device__ static double ld(const double *p) { return __ldcg(p); }
};

// C = op(A) op(B) for N x N row-major matrices (ta/tb: use the transpose).
template <class Ctx>
__device__ void mm(Ctx &c, double *C, const double *A, const double *B, int n, bool ta, bool tb, int kmax)
{
    for (int e = c.tid; e < n * n; e += c.nt) {
        int i = e / n, j = e % n;
        double s = 0.0;
        for (int k = 0; k < kmax; ++k) {
            double a = ta ? A[k * n + i] : A[i * n + k];
            double b = tb ? B[j * n + k] : B[k * n + j];
            s = fma(a, b, s);
        }
        C[e] = s;
    }
    c.sync();
}

// F = core - G o D + 2 diag(G diag D)
template <class Ctx>
__device__ void fock(Ctx &c, double *F, const double *core, const double *G, const double *D, int n)
{
    for (int e = c.tid; e < n * n; e += c.nt) {
        int i = e / n, j = e % n;
        double f = core[e] - G[e] * D[e];
        if (i == j) {
            double s = 0.0;
            for (int l = 0; l < n; ++l) s += G[i * n + l] * D[l * n + l];
            f += 2.0 * s;
        }
        F[e] = f;
    }
    c.sync();
}

// D = sum_{i<nocc} V[:,i] V[:,i]^T
template <class Ctx>
__device__ void density(Ctx &c, double *D, const double *V, int n, int nocc)
{
    for (int e = c.tid; e < n * n; e += c.nt) {
        int mu = e / n, nu = e % n;
        double s = 0.0;
        for (int i = 0; i < nocc; ++i) s = fma(V[mu * n + i], V[nu * n + i], s);
        D[e] = s;
    }
    c.sync();
}

// Pair k of round r in the circle ordering of np = n + (n & 1) players: p < q;
// q == n is the bye of an odd n.
__device__ __forceinline__ void circle_pair(int k, int r, int np, int &p, int &q)
{
    int x = k - 1 + r, y = np - 2 - k + r;
    if (x >= np - 1) x -= np - 1;
    if (y >= np - 1) y -= np - 1;
    p = k == 0 ? 0 : 1 + x;
    q = 1 + y;
    if (p > q) { const int t = p; p = q; q = t; }
}

// Rotation (c, s) that annihilates apq, the identity when |apq| <= thr. GUESS:
// in FP64 throughout. The diagonalisation from scratch turns by large angles
// whose choices between two nearly equal diagonal entries decide the orbitals'
// signs; with FP32 tangents one molecule in ten of 90-112 sites came out with
// other signs than the FP64 rotations give, and amplitudes follow those signs.
// The SCF iterations start from the last basis, turn by small angles and keep
// its signs: there the tangent is taken in FP32, and its cosine by one
// third-order Newton step (no sign differed in 60 such molecules).
template <bool GUESS>
__device__ __forceinline__ void rotation(double app, double aqq, double apq, double thr, double &c, double &s)
{
    c = 1.0;
    s = 0.0;
    if (!(fabs(apq) > thr)) return;
    if (GUESS) {
        const double theta = (aqq - app) / (2.0 * apq);
        const double t = fabs(theta) > 1e150 ? 0.5 / theta : (theta >= 0 ? 1.0 : -1.0) / (fabs(theta) + sqrt(theta * theta + 1.0));
        c = 1.0 / sqrt(t * t + 1.0);
        s = t * c;
        return;
    }
    const float den = (float)(apq + apq);
    if (den == 0.0f) return;
    const float theta = (float)(aqq - app) / den;
    const float m = fabsf(theta);
    const float tf = m > 1e9f ? 0.5f / theta : copysignf(1.0f / (m + sqrtf(m * m + 1.0f)), theta);
    const double t = (double)tf, x = fma(t, t, 1.0);
    const double y = (double)rsqrtf((float)x);          // within 1e-6 of 1 / sqrt(x)
    const double e = fma(-x * y, y, 1.0);               // 1 - x y^2
    c = fma(y * e, fma(0.375, e, 0.5), y);              // y (1 + e / 2 + 3 e^2 / 8): the error is of order e^3
    s = t * c;
}

// Item e of a round: the 2 x 2 block (k, l), k <= l, of the upper triangle of
// pairs (row k and row h - 1 - k folded into h + 1 items); false for the
// repeated half of the middle row.
__device__ __forceinline__ bool round_item(int e, int h, int &k, int &l)
{
    const int k0 = e / (h + 1), d = e - k0 * (h + 1);
    if (d < h - k0) { k = k0; l = k0 + d; return true; }
    k = h - 1 - k0;
    l = k + d - (h - k0);
    return k != k0;
}

// The elements of a block and where they sit (upper triangle) in round r.
struct Block2 {
    int i00, i01, i10, i11;
    bool hq, hv;                                         // (a bye has no second player)
    double a00, a01, a10, a11;
    template <class Ctx>
    __device__ __forceinline__ void load(const double *cur, int k, int l, int r, int np, int n)
    {
        int p, q, u, v;
        circle_pair(k, r, np, p, q);
        circle_pair(l, r, np, u, v);
        hq = q < n;
        hv = v < n;
        i00 = p < u ? p * n + u : u * n + p;
        i01 = p < v ? p * n + v : v * n + p;
        i10 = q < u ? q * n + u : u * n + q;
        i11 = q < v ? q * n + v : v * n + q;
        a00 = Ctx::ld(cur + i00);
        a01 = hv ? Ctx::ld(cur + i01) : 0.0;
        a10 = hq ? Ctx::ld(cur + i10) : 0.0;
        a11 = hq && hv ? Ctx::ld(cur + i11) : 0.0;
    }
    // J_k^T A J_l into nxt
    __device__ __forceinline__ void rotate(double *nxt, double ck, double sk, double cl, double sl, bool diag) const
    {
        double x00 = a00, x01 = a01, x10 = a10, x11 = a11;
        if (sl != 0.0) {
            x00 = cl * a00 - sl * a01; x01 = sl * a00 + cl * a01;
            x10 = cl * a10 - sl * a11; x11 = sl * a10 + cl * a11;
        }
        if (sk != 0.0) {
            const double y00 = x00, y01 = x01;
            x00 = ck * y00 - sk * x10; x01 = ck * y01 - sk * x11;
            x10 = sk * y00 + ck * x10; x11 = sk * y01 + ck * x11;
        }
        nxt[i00] = x00;
        if (hv) nxt[i01] = x01;
        if (hq && !diag) nxt[i10] = x10;
        if (hq && hv) nxt[i11] = x11;
    }
};

// Jacobi eigen-decomposition of the symmetric n x n matrix in A (upper
// triangle read; A and A2 are both overwritten) until its off-diagonal norm
// is FP64's 1e-15 of the matrix; rotations
// accumulate into V, this CTA's rows of it in the shared buffer vs. pc, ps,
// pd and rank_s are shared arrays of the CTA. A round's chain is: the pairs'
// entries from L2, their angles, the blocks, the barrier; the blocks' entries
// are fetched with the pairs' by the warps that do not compute angles.
template <bool GUESS, class Ctx>
__device__ void jacobi(Ctx &c, double *A, double *A2, double *V, double *E, double *vs, int n, double *pc, double *ps,
                       double *pd, int *rank_s)
{
    const int np = n + (n & 1), h = np / 2;
    const int nblk = ((h + 1) / 2) * (h + 1), step = c.size * NT;
    const int rows = (n + c.size - 1) / c.size, row0 = c.rank * rows, nrow = max(0, min(rows, n - row0));
    for (int e = threadIdx.x; e < nrow * n; e += NT) vs[e] = V[row0 * n + e];
    // items dealt out over the CTAs, within one to the last warps first
    const int first = c.rank + c.size * (NT - 1 - (int)threadIdx.x);
    int k1 = 0, l1 = 0;
    const bool has = first < nblk && round_item(first, h, k1, l1);
    double *cur = A, *nxt = A2;
    for (int sweep = 0; sweep < 40; ++sweep) {
        double off = 0.0, tot = 0.0;
        for (int e = c.tid; e < n * n; e += c.nt) {
            const int i = e / n, j = e - i * n;
            if (i > j) continue;
            const double x = c.ld(cur + e), a = x * x;
            if (i == j) tot += a; else off += a;
        }
        c.reduce2(off, tot, false);
        off += off;
        tot += off;
        const double goal = 1e-30 * tot;
        if (off <= goal || off < 1e-300) break;
        // all pairs at thr would leave off at a quarter of its bound
        const double thr = GUESS ? 1e-300 : 0.5 * sqrt(goal) / n;
        for (int r = 0; r < np - 1; ++r) {
            Block2 b;
            if (has) b.load<Ctx>(cur, k1, l1, r, np, n);
            for (int k = threadIdx.x; k < h; k += NT) {
                int p, q;
                double cc = 1.0, s = 0.0;
                circle_pair(k, r, np, p, q);
                if (q < n) rotation<GUESS>(c.ld(cur + p * n + p), c.ld(cur + q * n + q), c.ld(cur + p * n + q), thr, cc, s);
                pc[k] = cc;
                ps[k] = s;
            }
            __syncthreads();
            if (has) b.rotate(nxt, pc[k1], ps[k1], pc[l1], ps[l1], k1 == l1);
            for (int e = first + step; e < nblk; e += step) {
                int k, l;
                if (!round_item(e, h, k, l)) continue;
                b.load<Ctx>(cur, k, l, r, np, n);
                b.rotate(nxt, pc[k], ps[k], pc[l], ps[l], k == l);
            }
            // this CTA's rows of V: V <- V J
            for (int e = threadIdx.x; e < nrow * h; e += NT) {
                const int i = e / h, k = e - i * h;
                const double s = ps[k];
                if (s == 0.0) continue;                                // (a bye has s = 0)
                const double cs = pc[k];
                int p, q;
                circle_pair(k, r, np, p, q);
                double *row = vs + i * n;
                const double x = row[p], y = row[q];
                row[p] = cs * x - s * y;
                row[q] = s * x + cs * y;
            }
            c.sync();
            double *t = cur; cur = nxt; nxt = t;
        }
    }
    // sort ascending: rank each eigenvalue, permute V's columns
    for (int p = threadIdx.x; p < n; p += NT) pd[p] = c.ld(cur + p * n + p);
    __syncthreads();
    for (int p = threadIdx.x; p < n; p += NT) {
        const double ep = pd[p];
        int rank = 0;
        for (int q = 0; q < n; ++q) rank += (pd[q] < ep) || (pd[q] == ep && q < p);
        rank_s[p] = rank;
        if (c.rank == 0) E[rank] = ep;
    }
    __syncthreads();
    for (int e = threadIdx.x; e < nrow * n; e += NT) {
        const int i = e / n, p = e - i * n;
        V[(row0 + i) * n + rank_s[p]] = vs[e];
    }
    c.sync();
}

template <class Ctx>
__device__ void scf_body(Ctx &c, const ScfMol &m, const ScfParams &prm, double *vs, double *pc, double *ps, double *pd, int *rank_s)
{
    const int n = m.N, no = m.nocc, nn = n * n;
    double *F = m.F, *D = m.D, *V = m.V, *A = m.A, *W1 = m.W1, *W2 = m.W2;

    // guess
    if (m.D0) {
        for (int e = c.tid; e < nn; e += c.nt) D[e] = m.D0[e];
        for (int e = c.tid; e < nn; e += c.nt) V[e] = m.V0 ? m.V0[e] : (e / n == e % n);
        c.sync();
    } else {
        for (int e = c.tid; e < nn; e += c.nt) {
            A[e] = m.huckel[e];
            V[e] = (e / n == e % n) ? 1.0 : 0.0;
        }
        c.sync();
        jacobi<true>(c, A, W2, V, m.E, vs, n, pc, ps, pd, rank_s);
        density(c, D, V, n, no);
    }
    fock(c, F, m.core, m.G, D, n);

    int iteration = 0, successful = 1, status = 0;
    double current = 0.0;
    for (;;) {
        ++iteration;
        // W1 = F R, R = 2D - 1
        for (int e = c.tid; e < nn; e += c.nt) W2[e] = 2.0 * D[e] - (e / n == e % n);
        c.sync();
        mm(c, W1, F, W2, n, false, false, n);
        // A = W1 - W1^T  (F R - R F, both symmetric)
        for (int e = c.tid; e < nn; e += c.nt) A[e] = W1[e] - W1[(e % n) * n + e / n];
        c.sync();
        mm(c, W1, A, W2, n, false, false, n);           // Fmin
        double acc = 0.0, unused = 0.0;
        for (int e = c.tid; e < nn; e += c.nt) acc = fmax(acc, fabs(W1[e]));
        c.reduce2(acc, unused, true);
        for (int e = c.tid; e < nn; e += c.nt) D[e] -= prm.step * W1[e];
        c.sync();
        fock(c, F, m.core, m.G, D, n);
        // diagonalise F in the current basis: A = V^T F V
        mm(c, W1, F, V, n, false, false, n);
        mm(c, A, V, W1, n, true, false, n);
        jacobi<false>(c, A, W2, V, m.E, vs, n, pc, ps, pd, rank_s);
        density(c, D, V, n, no);
        fock(c, F, m.core, m.G, D, n);

        double previous = current;
        current = acc;
        if (current < previous) ++successful;
        if (!(current == current)) { status = HX_DIVERGED; break; }   // NaN
        if (current < prm.eps) { status = HX_CONVERGED; break; }
        if (prm.check_div && current > prm.divergence) { status = HX_DIVERGED; break; }
        if (iteration + 1 > prm.maxiter) { status = HX_FAILED_MAXITER; break; }
        if (prm.check_stag && iteration > prm.stag_after &&
            100.0 * successful / iteration <= prm.stag_pct) { status = HX_STAGNATED; break; }
    }
    // energy: Eel = sum D (core + F), Enuc = sum_{mu<nu} G   (energySCF :166-200)
    double eel = 0.0, enuc = 0.0;
    for (int e = c.tid; e < nn; e += c.nt) {
        eel += D[e] * (m.core[e] + F[e]);
        if (e / n < e % n) enuc += m.G[e];
    }
    c.reduce2(eel, enuc, false);
    if (c.tid == 0) {
        m.out[0] = eel + enuc;
        m.out[1] = eel;
        m.out[2] = enuc;
        m.out[3] = current;
        m.status[0] = status;
        m.status[1] = iteration;
    }
    // MO Fock (prepareFock('spatial'), mod_cc.f90:2336-2396): Fmo = V^T F V
    mm(c, W1, F, V, n, false, false, n);
    mm(c, m.Fmo, V, W1, n, true, false, n);
}

// One cluster per molecule; at most kBlockN sites: its first CTA alone, in
// shared memory.
__global__ void __launch_bounds__(NT) scf_kernel(const ScfMol *__restrict__ mols, ScfParams prm, double *gpart)
{
    __shared__ double sh[2 * NT / 32];
    __shared__ double pc[HX_MAX_MOL_N / 2], ps[HX_MAX_MOL_N / 2], pd[HX_MAX_MOL_N];
    __shared__ int rank_s[HX_MAX_MOL_N];
    extern __shared__ double dyn[];       // one CTA: seven matrices; a cluster: this CTA's rows of V
    const int cs = (int)cg::this_cluster().num_blocks(), mol = (int)blockIdx.x / cs;
    ScfMol m = mols[mol];
    if (m.N > kBlockN) {
        ClusterCtx c(sh, gpart + (long long)mol * 4 * cs);
        scf_body(c, m, prm, dyn, pc, ps, pd, rank_s);
        return;
    }
    if (cg::this_cluster().block_rank() != 0) return;
    BlockCtx c(sh);
    const ScfMol g = m;
    constexpr int NN = kBlockN * kBlockN;
    m.F = dyn; m.D = dyn + NN; m.V = dyn + 2 * NN; m.A = dyn + 3 * NN; m.W1 = dyn + 4 * NN; m.W2 = dyn + 5 * NN;
    scf_body(c, m, prm, dyn + 6 * NN, pc, ps, pd, rank_s);
    __syncthreads();
    for (int e = threadIdx.x; e < m.N * m.N; e += NT) { g.F[e] = m.F[e]; g.D[e] = m.D[e]; g.V[e] = m.V[e]; }
}
}  // namespace

// Cluster size: 16 CTAs (the non-portable size, where the device takes it)
// while every molecule's cluster has its SMs to itself; 8 while at most four
// CTAs share an SM; 4 for more molecules than that, whose reductions and
// cluster barriers then span half the CTAs (initialisation of 128 molecules of
// 8 to 64 sites: 65 ms with 8, 55 with 4). Molecules of at most kBlockN sites
// use one CTA of their cluster, so a launch of only such molecules takes
// clusters of one.
cudaError_t hx_scf_launch(const ScfMol *d_mols, int nmol, int nmax, const ScfParams &p, double *d_gpart,
                          cudaStream_t s)
{
    int cs = nmax <= kBlockN ? 1 : nmol * 16 <= HX_SCF_GRID_MAX ? 16 : nmol * 8 <= 4 * HX_SCF_GRID_MAX ? 8 : 4;
    cudaLaunchConfig_t cfg = {};
    cudaLaunchAttribute at[1];
    cfg.blockDim = dim3(NT);
    cfg.stream = s;
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    const int kMaxSmem = sizeof(double) * (HX_MAX_MOL_N / 4) * HX_MAX_MOL_N;     // 4 CTAs at the largest N
    cudaError_t ce = cudaFuncSetAttribute(scf_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kMaxSmem);
    if (ce != cudaSuccess) return ce;
    if (cs > 8) {
        int n = 0;
        cfg.dynamicSmemBytes = kMaxSmem;
        at[0].val.clusterDim.x = cs;
        cfg.gridDim = dim3((unsigned)cs);
        if (cudaFuncSetAttribute(scf_kernel, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) != cudaSuccess ||
            cudaOccupancyMaxActiveClusters(&n, scf_kernel, &cfg) != cudaSuccess || n < 1) {
            cudaGetLastError();
            cs = 8;
        }
    }
    // the smaller form's matrices, or the rows of V of the largest molecule
    const size_t rows_v = (size_t)((nmax + cs - 1) / cs) * nmax;
    cfg.dynamicSmemBytes = sizeof(double) * std::max<size_t>(7 * kBlockN * kBlockN, nmax > kBlockN ? rows_v : 0);
    at[0].val.clusterDim.x = cs;
    cfg.gridDim = dim3((unsigned)nmol * cs);
    hx_count_launches(1);
    return cudaLaunchKernelEx(&cfg, scf_kernel, d_mols, p, d_gpart);
}
