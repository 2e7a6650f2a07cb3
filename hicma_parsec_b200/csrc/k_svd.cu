// Batched small-core SVD and rank truncation, FP64.
//
// Replaces the SVD + truncation step inside HCORE_dgemm_qr_svd (the core
// R_U R_V^T of a recompression, call sites
// hicma_parsec/HiCMA_dpotrf_L_2flow.jdf:830-903,985-1058) and the rank rule of
// starsh_dense_dlrrsdd (STARSH_gen.jdf:162-171).
//
// QR-preconditioned one-sided Jacobi (Drmac and Veselic, "New fast and accurate
// Jacobi SVD algorithm", SIMAX 2008):
//   1. T = M^T with M = R_U R_V^T is formed on the FP64 tensor cores.
//   2. Householder QR with column pivoting, T P = Q R, with exact partial
//      column norms recomputed in the pass that applies a reflector.  It stops
//      at step k once the trailing block's Frobenius norm is below the
//      truncation floor, so only the leading k rows of R survive; k is about
//      the numerical rank, not K.  Columns stay where they are (the pivot order
//      is kept by the rows of R), so X = R^T (K x k) has the rows of M.
//   3. X is orthogonalised by one-sided (Hestenes) Jacobi, X J = W Sigma, in
//      round-robin tournament order.  The rotation angles come from the Gram
//      matrix G = X^T X: it is computed afresh by DMMA at the start of a sweep
//      and rotated along with X (G <- J^T G J), so a round needs no dot
//      products and no reductions.  A sweep is only run when the fresh G still
//      has a pair that is not orthogonal.  The rows of a pivoted R are graded,
//      so the columns of R^T are nearly orthogonal and few sweeps are needed.
//      G_ij carries an error of about K eps ||x_i|| ||x_j||, as a dot product
//      does, so the criterion |G_ij| <= tol sqrt(G_ii G_jj) keeps the relative
//      accuracy of one-sided Jacobi for the small singular values.
//   4. M = X Q^T, so the left singular vectors of M are U[:, q] = W[:, q] /
//      sigma.  Neither Q nor J is formed; the caller recovers
//      V Sigma = M^T U = R_V (R_U^T U) with GEMMs.
// The truncation threshold is absolute and the decision is FP64.
//
// Two kernels.  K <= SMALL_KMAX: one CTA per core, T in registers (four lanes
// a column) for the pivoted QR, then X and G in shared memory.  Wider cores:
// one thread-block cluster per core, T's columns dealt out over the shared
// memories of its CTAs for the pivoted QR, then block Jacobi on pairs of
// 16-column blocks, one pair per CTA and round (Gram product and the product
// with the accumulated rotations on DMMA, the rotations of the 32 x 32 Gram
// matrix in shared memory).
#include "core_layout.h"
#include "tlr_internal.h"

#include <algorithm>

#include <cooperative_groups.h>

namespace tlr {
namespace {

constexpr int SMALL_KMAX = 96;
constexpr int MAX_SWEEPS = 40;

__device__ __forceinline__ void dmma884(double (&d)[2], double a, double b) {
    asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0,%1}, {%2}, {%3}, {%0,%1};\n"
                 : "+d"(d[0]), "+d"(d[1])
                 : "d"(a), "d"(b));
}

__device__ __forceinline__ int tourney(int slot, int round, int kp) {
    if (slot == 0) return 0;
    int s = slot - 1 + round;
    if (s >= kp - 1) s -= kp - 1;
    return 1 + s;
}

template <int LP>
__device__ __forceinline__ double group_sum(double v) {
#pragma unroll
    for (int o = LP / 2; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}

// A pair of columns with squared norms aa, bb and dot product cc counts as
// orthogonal when |cc| <= tol sqrt(aa bb) (tol2 = tol^2), and columns at or
// below the truncation floor are left alone.  The values are first scaled by a
// power of two (exact) so that no square over- or underflows.
__device__ __forceinline__ bool pair_scaled(double &aa, double &bb, double &cc, double tau2, double tol2) {
    if (!(aa > tau2 && bb > tau2) || aa < 1e-290 || bb < 1e-290 || cc == 0.0) return false;
    const int e = (__double2hiint(fmax(aa, bb)) >> 20) & 0x7ff;
    const double sc = __hiloint2double((2046 - e) << 20, 0);
    aa *= sc;
    bb *= sc;
    cc *= sc;
    return cc * cc > tol2 * aa * bb;
}

// Rotation that makes the pair orthogonal: x' = cs x - sn y, y' = sn x + cs y.
// With h = sqrt((bb - aa)^2 + 4 cc^2): cs^2 = (1 + |bb - aa| / h) / 2 and
// sn cs = |cc| / h (the small angle).  cs = 1, sn = 0 where none is needed.
// On the critical path of a round: the test runs beside the rotation, and the
// scaling only where a square could over- or underflow.
__device__ __forceinline__ double2 pair_rotation(double aa, double bb, double cc, double tau2, double tol2) {
    bool need = aa > tau2 && bb > tau2 && cc * cc > tol2 * aa * bb;
    if (!(fmin(aa, bb) > 1e-120 && fmax(aa, bb) < 1e140)) need = pair_scaled(aa, bb, cc, tau2, tol2);
    const double d = bb - aa, c2x = cc + cc;
    const double rh = rsqrt(fma(d, d, c2x * c2x));
    const double c2 = fma(0.5 * fabs(d), rh, 0.5);
    const double rc = rsqrt(c2);
    return make_double2(need ? c2 * rc : 1.0, need ? copysign(cc, d * cc) * rh * rc : 0.0);
}

// G is symmetric: entry (x, y) of the lower triangle stored.
__device__ __forceinline__ int low(int x, int y, int ld) { return x > y ? x * ld + y : y * ld + x; }

// Blocks (I, J), I >= J, of G's lower triangle by pairs, in the order of a
// linear index (J of 16 bits above I of 16 bits).
__device__ __forceinline__ int tri_block(int q) {
    int i = 0;
    while ((i + 1) * (i + 2) / 2 <= q) ++i;
    return i | ((q - i * (i + 1) / 2) << 16);
}

// G <- J^T G J on the NB blocks blk[] of a thread (2 x 2 blocks of G at
// the pairs I and J, a | b << 16, rotations rot[]), all loaded before any is
// written, without branches.  A diagonal block belongs to one pair: the rotation
// makes its off-diagonal entry zero.
template <int NB>
__device__ __forceinline__ void rotate_blocks(double *G, int ld, const int (&blk)[NB], const double2 *rot,
                                              const int *pab) {
    double2 cr[NB], cc[NB];
    double gaa[NB], gab[NB], gba[NB], gbb[NB];
    int iaa[NB], iab[NB], iba[NB], ibb[NB];
#pragma unroll
    for (int q = 0; q < NB; ++q) {
        const int I = blk[q] & 0xffff, J = blk[q] >> 16;
        cr[q] = rot[I];
        cc[q] = rot[J];
        const int pi = pab[I], pj = pab[J];
        const int a0 = pi & 0xffff, b0 = pi >> 16, a1 = pj & 0xffff, b1 = pj >> 16;
        iaa[q] = low(a0, a1, ld);
        iab[q] = low(a0, b1, ld);
        iba[q] = low(b0, a1, ld);
        ibb[q] = low(b0, b1, ld);
        gaa[q] = G[iaa[q]];
        gab[q] = G[iab[q]];
        gba[q] = G[iba[q]];
        gbb[q] = G[ibb[q]];
    }
#pragma unroll
    for (int q = 0; q < NB; ++q) {
        const double u0 = cc[q].x * gaa[q] - cc[q].y * gab[q], u1 = cc[q].y * gaa[q] + cc[q].x * gab[q];
        const double v0 = cc[q].x * gba[q] - cc[q].y * gbb[q], v1 = cc[q].y * gba[q] + cc[q].x * gbb[q];
        const bool diag = (blk[q] & 0xffff) == blk[q] >> 16;
        G[iaa[q]] = cr[q].x * u0 - cr[q].y * v0;
        G[ibb[q]] = cr[q].y * u1 + cr[q].x * v1;
        // (on a diagonal block that needed no rotation the entry stays)
        const double vab = cr[q].x * u1 - cr[q].y * v1, vba = cr[q].y * u0 + cr[q].x * v0;
        const bool zero = diag && cr[q].y != 0.0;
        G[iab[q]] = zero ? 0.0 : vab;
        G[iba[q]] = zero ? 0.0 : vba;
    }
}

// Rotates the column pair ab (rotation r) in R rows of M from row c0 on, step rows
// apart (row-major, pitch ld), all loaded before any is written.
template <int R>
__device__ __forceinline__ void rotate_rows(double *M, int ld, int ab, double2 r, int c0, int step) {
    double *pa = M + c0 * ld + (ab & 0xffff), *pb = M + c0 * ld + (ab >> 16);
    double xa[R], xb[R];
#pragma unroll
    for (int q = 0; q < R; ++q) {
        xa[q] = pa[q * step * ld];
        xb[q] = pb[q * step * ld];
    }
#pragma unroll
    for (int q = 0; q < R; ++q) {
        pa[q * step * ld] = r.x * xa[q] - r.y * xb[q];
        pb[q * step * ld] = r.y * xa[q] + r.x * xb[q];
    }
}

// Truncation floor on squared norms: 1e-3 of the absolute threshold
// (recompression) or of tol * ||M||_F (generation, total = ||M||_F^2); zero in
// fixed-rank mode.
__device__ __forceinline__ double trunc_floor(const CoreParams &p, double total) {
    if (p.mode == 1) return 1e-6 * p.tol * p.tol * total;
    const double tau = p.fixed_rank <= 0 ? 1e-3 * p.tol : 0.0;
    return tau * tau;
}

// Rank of the core from its k singular values in decreasing order, sv(i), nge
// of them at or above p.tol; dropped: the squared mass below the truncation
// floor (generation).
template <class F>
__device__ __forceinline__ int core_rank(const CoreParams &p, int K, int k, double dropped, int nge, F sv) {
    int r;
    if (p.mode == 0) {
        r = p.fixed_rank > 0 ? min(p.fixed_rank, K) : nge;
        if (r > p.maxrank) {
            r = p.maxrank;
            if (p.overflow) atomicAdd(p.overflow, 1);
        }
        return r;
    }
    double total = dropped;
    for (int l = 0; l < k; ++l) total += sv(l) * sv(l);
    if (total == 0.0) return 0;
    const double thr = p.tol * p.tol * total;
    double tail = dropped;
    r = k;
    while (r > 0) {
        const double s2 = sv(r - 1) * sv(r - 1);
        if (tail + s2 > thr) break;
        tail += s2;
        --r;
    }
    return (2 * r < p.nb && r <= p.maxrank) ? r : -1;
}

// ------------------------------------------------------------ small cores --
// One CTA of 4 KM threads per core.  Pivoted QR: lane group of four per
// column, rows r = 4 q + sub in registers, so a reflector is applied with
// register FMAs and a two-level shuffle; every warp finds the pivot itself
// from the norms in shared memory, and the two barriers of a step are after
// the norms and after the pivot column is published.  Bound by the latency of
// those steps and of the Jacobi rounds; several CTAs share an SM.
// In a Jacobi round the first warps find the next round's rotations (about 600
// cycles of dependent FP64 operations) while the others rotate the rows of X; G is
// stored by its lower triangle with an odd pitch, since its blocks are read along
// rows and columns alike.  Latency of one core with k = 0.83 K: K = 32, 64, 80 107,
// 405, 791 us (145, 499, 1146 with the rotations found before both updates and G
// full with 4-way conflicts).  Against one CTA with dot products reduced over 8 or
// 16 lanes and two to three shuffles a value: the cores of the 60 x 60 tiles of
// 2700 2D workload (34,220 of K up to 100) 142 -> 74 ms, 20 x 20 tiles of 1350 90
// -> 33 ms.
template <int KM>
struct SmallCore {
    static constexpr int NT = 4 * KM;
    static constexpr int NW = NT / 32;
    static constexpr int P = KM + 4;          // pitch of X, == 4 mod 16: conflict-free DMMA fragments
    static constexpr int PG = KM + 1;         // pitch of G, odd: its rows and columns are read alike
    static constexpr int NT8 = KM / 8;
    static constexpr int NBLK = (KM / 2) * (KM / 2 + 1) / 2;   // 2 x 2 blocks of G's lower triangle
    static constexpr int BPT = (NBLK + NT - 1) / NT;           // of them a thread rotates
    static constexpr int XR = KM + 4 * NW;                     // rows of X: batches of four a warp
    // X, G and an idle entry, sig, hv, 2 x (cs, sn) of KM / 2 pairs and the idle pair
    static constexpr size_t doubles = (size_t)XR * P + (KM + 1) * PG + 1 + 2 * KM + 2 * (KM + 2);
    static constexpr size_t bytes = sizeof(double) * doubles + sizeof(int) * (2 * KM + 2);
};

template <int KM>
__global__ void __launch_bounds__(4 * KM) k_core_small(const CoreTask *__restrict__ tasks, CoreParams p) {
    using S = SmallCore<KM>;
    constexpr int NT = S::NT, NW = S::NW, P = S::P, PG = S::PG, NT8 = S::NT8;
    constexpr int Q = KM / 4;                 // rows a lane holds
    constexpr int NSLOT = (KM + 31) / 32;     // columns a lane scans for the pivot
    extern __shared__ __align__(16) double sm[];
    __shared__ int rank_sh;
    const CoreTask t = tasks[blockIdx.x];
    const int K = t.K;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int g = lane >> 2, tig = lane & 3;
    if (K <= 0) {
        if (tid == 0) {
            if (t.rank_out) *t.rank_out = 0;
            if (t.rank_task) *t.rank_task = 0;
        }
        return;
    }
    double *X = sm;                           // X(c, i) at c * P + i; T(r, c) at c * P + r before the QR
    double *G = X + S::XR * P;
    double *sig = G + (KM + 1) * PG + 1;      // keeps what follows 16-byte aligned: PG is odd
    double *hv = sig + KM;
    double2 *rot = (double2 *)(hv + KM);      // KM / 2 rotations of this and of the next round, an idle one each
    constexpr int RP = KM / 2 + 1;
    int *order = (int *)(rot + 2 * RP);
    int *pab = order + KM;                    // their column pairs, a | b << 16

    // 1. T = M^T: T(i, c) = sum_{l >= max(i, c)} RU(c, l) RV(i, l), the entries
    //    below the diagonals masked (RV may be a Householder-factored stack);
    //    warp w forms columns 8 w .. 8 w + 7.  RU null: M = RV^T, T = RV.
    if (t.RU) {
        double acc[NT8][2];
#pragma unroll
        for (int I = 0; I < NT8; ++I) acc[I][0] = acc[I][1] = 0.0;
        const int c = 8 * warp + g;
#pragma unroll 2
        for (int l0 = 8 * warp; l0 < K; l0 += 4) {
            const int l = l0 + tig;
            const double b = (c < K && l < K && l >= c) ? t.RU[(size_t)c + (size_t)l * t.ldru] : 0.0;
            double a[NT8];
#pragma unroll
            for (int I = 0; I < NT8; ++I) {
                const int i = 8 * I + g;
                a[I] = (i < K && l < K && l >= i) ? t.RV[(size_t)i + (size_t)l * t.ldrv] : 0.0;
            }
#pragma unroll
            for (int I = 0; I < NT8; ++I) dmma884(acc[I], a[I], b);
        }
#pragma unroll
        for (int I = 0; I < NT8; ++I)
#pragma unroll
            for (int e = 0; e < 2; ++e) X[(8 * warp + 2 * tig + e) * P + 8 * I + g] = acc[I][e];
    } else {
        for (int idx = tid; idx < KM * KM; idx += NT) {
            const int i = idx % KM, c = idx / KM;
            X[c * P + i] = (i <= c && c < K) ? t.RV[(size_t)i + (size_t)c * t.ldrv] : 0.0;
        }
    }
    __syncthreads();
    const int col = 8 * warp + g, sub = tig;
    double x[Q];
    double s2 = 0.0;
#pragma unroll
    for (int q = 0; q < Q; ++q) {
        x[q] = X[col * P + 4 * q + sub];
        s2 = fma(x[q], x[q], s2);
    }
    s2 = group_sum<4>(s2);
    if (sub == 0) sig[col] = s2;
    bool active = col < K;
    __syncthreads();
    double total = 0.0;
#pragma unroll
    for (int s = 0; s < NSLOT; ++s) total += lane + 32 * s < KM ? sig[lane + 32 * s] : 0.0;
    total = group_sum<32>(total);
    const double tau2 = trunc_floor(p, total);

    // 2. pivoted Householder QR of T, stopped when the trailing mass <= tau2
    unsigned done[NSLOT];                     // columns this lane scans that were pivots already
#pragma unroll
    for (int s = 0; s < NSLOT; ++s) done[s] = lane + 32 * s >= K;
    int k = K;
    double dropped = 0.0;
    for (int j = 0; j < K; ++j) {
        // pivot: the column of largest norm, by the upper half of the double
        // (20 bits of mantissa; the lowest index of equal ones)
        unsigned best = 0u;
        int bc = 0;
        double tr = 0.0;
#pragma unroll
        for (int s = 0; s < NSLOT; ++s) {
            if (!done[s]) {
                const double v = sig[lane + 32 * s];
                tr += v;
                const unsigned key = (unsigned)__double2hiint(v) + 1u;
                if (key > best) { best = key; bc = lane + 32 * s; }
            }
        }
        const unsigned top = __reduce_max_sync(0xffffffffu, best);
        int pc = __reduce_min_sync(0xffffffffu, best == top ? bc : KM);
        tr = group_sum<32>(tr);
        if (!(tr > tau2)) { k = j; dropped = tr; break; }    // the same in every warp
        pc = min(pc, KM - 1);
        const double n2 = sig[pc], sn = sqrt(n2);
        if ((pc & 31) == lane) {
#pragma unroll
            for (int s = 0; s < NSLOT; ++s)
                if (s == (pc >> 5)) done[s] = 1u;
        }
        if (col == pc) {
#pragma unroll
            for (int q = 0; q < Q; ++q) hv[4 * q + sub] = 4 * q + sub < j ? 0.0 : x[q];
        }
        __syncthreads();
        // H = I - v v^T / (n2 - alpha beta), v = x - beta e_j, beta = -sign(alpha) ||x||
        const double alpha = hv[j];
        const double beta = -copysign(sn, alpha);
        const double den = fma(-alpha, beta, n2);
        const double th = den > 0.0 ? 1.0 / den : 0.0;
        double v[Q], w0 = 0.0, w1 = 0.0;
#pragma unroll
        for (int q = 0; q < Q; ++q) {
            v[q] = hv[4 * q + sub];
            if (4 * q + sub == j) v[q] -= beta;
            if (q & 1) w1 = fma(v[q], x[q], w1);
            else w0 = fma(v[q], x[q], w0);
        }
        double w = group_sum<4>(w0 + w1) * th;
        if (!active) w = 0.0;
        double rj = 0.0, n0 = 0.0, n1 = 0.0;
#pragma unroll
        for (int q = 0; q < Q; ++q) {
            const int r = 4 * q + sub;
            x[q] = fma(-w, v[q], x[q]);
            if (r == j) rj = x[q];
            if (r > j) {
                if (q & 1) n1 = fma(x[q], x[q], n1);
                else n0 = fma(x[q], x[q], n0);
            }
        }
        const double nn = group_sum<4>(n0 + n1);
        // row j of R: beta at the pivot, zero at the earlier pivots
        if (sub == (j & 3)) X[col * P + j] = col == pc ? beta : (active ? rj : 0.0);
        if (col == pc) active = false;
        if (sub == 0) sig[col] = active ? nn : 0.0;
        __syncthreads();
    }

    // 3. one-sided Jacobi on the k columns of X = R^T
    const int kp = k + (k & 1), np = kp / 2, nk8 = (k + 7) >> 3;
    // the rounding of a K-term dot product is about K eps: a tighter threshold
    // would keep rotating noise and never converge
    const double tolj = 4.4e-16 * (double)(K > 16 ? K : 16), tol2 = tolj * tolj;
    int sweeps = 0;
    __syncthreads();
    // columns k .. 8 nk8 take part in the Gram tiles: zero
    for (int idx = tid; idx < KM * (8 * nk8 - k); idx += NT) X[(idx % KM) * P + k + idx / KM] = 0.0;
    __syncthreads();
    // the first warps find the rotations of the next round while the others
    // rotate the rows of X, lanes over pairs
    const int nwa = np > 32 && NW > 2 ? 2 : 1;
    const int L = np <= 8 ? 8 : np <= 16 ? 16 : 32;
    const int RS = 32 / L;                            // rows a warp takes at a time
    const int li = lane % L, lr = (warp - nwa) * RS + lane / L, rstep = (NW - nwa) * RS;
    int blk[S::BPT];                                  // this thread's blocks of G, -1: none
#pragma unroll
    for (int q = 0; q < S::BPT; ++q) {
        const int e = tid + q * NT;
        blk[q] = e < np * (np + 1) / 2 ? tri_block(e) : (KM / 2) | ((KM / 2) << 16);
    }
    // the idle pair of threads without a block: no rotation, of the idle entry
    if (tid < 2) {
        rot[tid * RP + KM / 2] = make_double2(1.0, 0.0);
        pab[tid * RP + KM / 2] = KM | (KM << 16);
        G[KM * PG + KM] = 0.0;
    }
    auto angles = [&](int round, int buf) {
        for (int pr = tid; pr < np; pr += 32 * nwa) {
            const int a = tourney(pr, round, kp), b = tourney(kp - 1 - pr, round, kp);
            rot[buf * RP + pr] = max(a, b) < k
                                           ? pair_rotation(G[a * PG + a], G[b * PG + b], G[low(a, b, PG)], tau2, tol2)
                                           : make_double2(1.0, 0.0);
            pab[buf * RP + pr] = a | (b << 16);
        }
    };
    while (k > 0) {
        // G = X^T X (rows past K are zero)
        for (int q = warp; q < nk8 * (nk8 + 1) / 2; q += NW) {
            int I = 0;
            while ((I + 1) * (I + 2) / 2 <= q) ++I;
            const int J = q - I * (I + 1) / 2;
            double a0[2] = {0.0, 0.0}, a1[2] = {0.0, 0.0};
            int c = 0;
            for (; c + 4 < K; c += 8) {
                const double *x0 = X + (c + tig) * P, *x1 = x0 + 4 * P;
                dmma884(a0, x0[8 * I + g], x0[8 * J + g]);
                dmma884(a1, x1[8 * I + g], x1[8 * J + g]);
            }
            if (c < K) dmma884(a0, X[(c + tig) * P + 8 * I + g], X[(c + tig) * P + 8 * J + g]);
#pragma unroll
            for (int e = 0; e < 2; ++e) G[(8 * I + g) * PG + 8 * J + 2 * tig + e] = a0[e] + a1[e];
        }
        __syncthreads();
        if (sweeps >= MAX_SWEEPS) break;
        int need = 0;
        for (int idx = tid; idx < k * k; idx += NT) {
            const int i = idx / k, jj = idx - i * k;
            if (jj < i) {
                double aa = G[i * PG + i], bb = G[jj * PG + jj], cc = G[i * PG + jj];
                need |= pair_scaled(aa, bb, cc, tau2, tol2);
            }
        }
        if (!__syncthreads_or(need)) break;
        ++sweeps;
        if (warp < nwa) angles(0, 0);
        __syncthreads();
        for (int round = 0; round < kp - 1; ++round) {
            const double2 *rr = rot + (round & 1) * RP;
            const int *pp = pab + (round & 1) * RP;
            rotate_blocks<S::BPT>(G, PG, blk, rr, pp);
            __syncthreads();
            if (warp < nwa) {
                if (round + 1 < kp - 1) angles(round + 1, (round + 1) & 1);
            } else {
                for (int I = li; I < np; I += L) {
                    const double2 r = rr[I];
                    const int ab = pp[I];
                    if (r.y == 0.0) continue;
                    // batches of four rows a warp; a last batch past K ends in X's padding
                    if (RS == 1)
                        for (int c = lr; c < K; c += 4 * rstep) rotate_rows<4>(X, P, ab, r, c, rstep);
                    else if (RS == 2)
                        for (int c = lr; c < K; c += 2 * rstep) rotate_rows<2>(X, P, ab, r, c, rstep);
                    else
                        for (int c = lr; c < K; c += rstep) rotate_rows<1>(X, P, ab, r, c, rstep);
                }
            }
            __syncthreads();
        }
    }

    // 4. singular values (from the fresh Gram matrix), descending order, rank
    for (int c = tid; c < k; c += NT) {
        sig[c] = sqrt(G[c * PG + c]);
        order[c] = c;
    }
    __syncthreads();
    const int nge = __syncthreads_count(tid < k && sig[tid] >= p.tol);
    for (int c = tid; c < k; c += NT) {
        const double sc = sig[c];
        int pos = 0;
        for (int l = 0; l < k; ++l) {
            const double sl = sig[l];
            pos += (sl > sc) || (sl == sc && l < c);
        }
        order[pos] = c;
    }
    __syncthreads();
    if (tid == 0) {
        const int r = core_rank(p, K, k, dropped, nge, [&](int i) { return sig[order[i]]; });
        rank_sh = r;
        if (t.rank_out) *t.rank_out = r;
        if (t.rank_task) *t.rank_task = r;
        if (p.sweeps) atomicAdd(p.sweeps, sweeps);
    }
    __syncthreads();
    // the r leading left singular vectors of M (consumers read rank columns);
    // past k the singular values are zero
    const int r = rank_sh;
    for (int i = warp; i < r; i += NW) {
        const int c = i < k ? order[i] : 0;
        const double s = i < k ? sig[c] : 0.0;
        const double is = s > 0.0 ? 1.0 / s : 0.0;
        for (int q = lane; q < K; q += 32) t.SU[(size_t)q + (size_t)i * K] = is > 0.0 ? X[q * P + c] * is : 0.0;
    }
}

// ------------------------------------------------------------- wide cores --
// One cluster of CS CTAs per core (CS from K, wide_cluster()).  The columns of
// T are dealt to the CTAs, c to CTA c mod CS: in its shared memory where they
// fit, else in the task's scratch.  A step of the pivoted QR has one cluster
// barrier: every CTA publishes its best column and its sum of norms to all
// others, then reads the pivot column from its owner's memory.  X lies in the
// task's scratch (column-major, ld K, read through L2 since other CTAs of the
// cluster write it), its columns in blocks of 16; a round of the block Jacobi
// pairs all blocks, and the CTA of a pair orthogonalises its 32 columns: Gram
// matrix, rotations of the Gram matrix with the rotations accumulated in J,
// then the columns times J.  Bound by the latency of the rounds: the 31
// rotation rounds of a pair problem take about as long as its two products.
// Pairs within a block are rotated once a sweep, pairs across two blocks in the
// round that brings the blocks together (16 rotation rounds of about 800 cycles).
// One core of K = 96, 256, 400: 0.52, 2.4, 9.0 ms.  Two launches of three cores and
// one of K about 650 (k about 430): 470 -> 32 ms against one warp per column pair
// reading its columns through L2.
__device__ __forceinline__ double ldg2(const double *p) { return __ldcg(p); }
__device__ __forceinline__ int ldg2(const int *p) { return __ldcg(p); }

struct WidePub {
    double norm, sum;
    int col, pad;
};

// HV: the pivot column is in shared memory (W_HV_SHARED)
template <bool HV>
__global__ void __launch_bounds__(W_CT) k_core_wide(const CoreTask *__restrict__ tasks, CoreParams p, int place) {
    namespace cg = cooperative_groups;
    cg::cluster_group cl = cg::this_cluster();
    extern __shared__ __align__(16) double sm[];
    __shared__ WidePub pub[2][W_CSMAX];
    __shared__ double2 rot[2][WP / 2];
    __shared__ int pab[2][WP / 2];
    __shared__ int rank_sh;
    const int CS = (int)cl.num_blocks(), crank = (int)cl.block_rank();
    const CoreTask t = tasks[blockIdx.x / CS];
    const int K = t.K;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int g = lane >> 2, tig = lane & 3;
    const int gw = crank * W_NW + warp, GW = CS * W_NW;
    const long long gt = (long long)crank * W_CT + tid, GT = (long long)CS * W_CT;
    if (K <= 0) {
        if (crank == 0 && tid == 0) {
            if (t.rank_out) *t.rank_out = 0;
            if (t.rank_task) *t.rank_task = 0;
        }
        return;
    }
    const bool t_in_smem = place & W_T_SHARED;
    const WideLayout L = wide_layout(K, CS, crank, place);
    double *X = t.work + L.X;
    double *sig = t.work + L.sig;
    int *rotf = (int *)(t.work + L.flags);    // [sweep]: a pair was rotated
    const int ncl = wide_ncl(K, CS), lcs = __ffs(CS) - 1;   // CS is a power of two
    double *sigl = sm + L.sigl;               // squared norms of the CTA's columns, -1 once pivots
    double *hv = (HV ? sm : t.work) + L.hv;   // the pivot column
    double *Tl = (t_in_smem ? sm : t.work) + L.T;   // the CTA's columns of T
    const int nc = crank < K ? (K - crank + CS - 1) / CS : 0;   // columns this CTA holds

    if (gt < 64) rotf[gt] = 0;
    // 1. the CTA's columns of T = M^T: T(i, c) = sum_{l >= max(i, c)} RU(c, l) RV(i, l);
    //    a warp takes eight local columns and up to eight 8-row tiles at a time
    if (t.RU) {
        const int ntr = (K + 7) >> 3, ntc = (nc + 7) >> 3, nrg = (ntr + 7) >> 3;
        for (int it = warp; it < ntc * nrg; it += W_NW) {
            const int jt = it % ntc, rg = it / ntc;
            const int q = 8 * jt + g, c = crank + CS * q;
            double acc[8][2];
#pragma unroll
            for (int I = 0; I < 8; ++I) acc[I][0] = acc[I][1] = 0.0;
            const int lb = max(crank + CS * 8 * jt, 64 * rg) & ~3;
#pragma unroll 2
            for (int l0 = lb; l0 < K; l0 += 4) {
                const int l = l0 + tig;
                const double b = (q < nc && l < K && l >= c) ? t.RU[(size_t)c + (size_t)l * t.ldru] : 0.0;
                double a[8];
#pragma unroll
                for (int I = 0; I < 8; ++I) {
                    const int i = 64 * rg + 8 * I + g;
                    a[I] = (l < K && l >= i) ? t.RV[(size_t)i + (size_t)l * t.ldrv] : 0.0;
                }
#pragma unroll
                for (int I = 0; I < 8; ++I) dmma884(acc[I], a[I], b);
            }
#pragma unroll
            for (int I = 0; I < 8; ++I)
#pragma unroll
                for (int e = 0; e < 2; ++e) {
                    const int i = 64 * rg + 8 * I + g, qq = 8 * jt + 2 * tig + e;
                    if (i < K && qq < nc) Tl[(size_t)qq * K + i] = acc[I][e];
                }
        }
    } else {
        for (int q = warp; q < nc; q += W_NW) {
            const int c = crank + CS * q;
            for (int i = lane; i < K; i += 32)
                Tl[(size_t)q * K + i] = i <= c ? t.RV[(size_t)i + (size_t)c * t.ldrv] : 0.0;
        }
    }
    __syncthreads();
    for (int q = warp; q < nc; q += W_NW) {
        double s2 = 0.0;
        for (int i = lane; i < K; i += 32) s2 = fma(Tl[(size_t)q * K + i], Tl[(size_t)q * K + i], s2);
        s2 = group_sum<32>(s2);
        if (lane == 0) sigl[q] = s2;
    }
    __syncthreads();

    // 2. pivoted Householder QR of T, stopped when the trailing mass <= tau2
    double tau2 = 0.0, dropped = 0.0;
    int k = K;
    for (int j = 0; j < K; ++j) {
        const int par = j & 1;
        if (warp == 0) {
            // the CTA's best column (by the upper half of the norm) and its sum of norms
            double tr = 0.0;
            unsigned best = 0u;
            int bq = 0x7fffffff;
            for (int q = lane; q < nc; q += 32) {
                const double v = sigl[q];
                if (v < 0.0) continue;
                tr += v;
                const unsigned key = (unsigned)__double2hiint(v) + 1u;
                if (key > best) { best = key; bq = q; }
            }
            const unsigned top = __reduce_max_sync(0xffffffffu, best);
            bq = __reduce_min_sync(0xffffffffu, best == top ? bq : 0x7fffffff);
            tr = group_sum<32>(tr);
            if (lane < CS) {
                WidePub *d = cl.map_shared_rank(&pub[par][crank], lane);
                d->norm = top ? sigl[bq] : -1.0;
                d->sum = tr;
                d->col = top ? crank + CS * bq : 0x7fffffff;
            }
        }
        cl.sync();
        // best of the CTAs: the same comparison in every warp of the cluster
        double tr = 0.0, n2 = -1.0;
        int pc = 0x7fffffff;
        {
            const WidePub e = pub[par][lane & (CS - 1)];
            tr = lane < CS ? e.sum : 0.0;
            const unsigned key = e.norm >= 0.0 || e.norm != e.norm ? (unsigned)__double2hiint(e.norm) + 1u : 0u;
            const unsigned top = __reduce_max_sync(0xffffffffu, key);
            pc = __reduce_min_sync(0xffffffffu, key == top ? e.col : 0x7fffffff);
            tr = group_sum<32>(tr);
        }
        if (j == 0) tau2 = trunc_floor(p, tr);
        if (!(tr > tau2) || pc >= K) { k = j; dropped = tr; break; }   // the same in every CTA
        // the pivot column, from its owner's memory (nothing writes it any more)
        const int owner = pc & (CS - 1), lp = pc >> lcs;
        n2 = pub[par][owner].norm;
        const double sn = sqrt(n2);
        if (t_in_smem) {
            const double *src = cl.map_shared_rank(Tl, owner) + (size_t)lp * K;
            for (int r = j + tid; r < K; r += W_CT) hv[r] = src[r];
        } else {
            const double *src = Tl + ((ptrdiff_t)(owner - crank) * ncl + lp) * K;
            for (int r = j + tid; r < K; r += W_CT) hv[r] = ldg2(src + r);
        }
        __syncthreads();
        const double alpha = hv[j];
        const double beta = -copysign(sn, alpha);
        const double den = fma(-alpha, beta, n2);
        const double th = den > 0.0 ? 1.0 / den : 0.0;
        // eight lanes a column, four columns a warp; row j apart (v_j = alpha - beta)
        const int gl = lane & 7;
        for (int q0 = 4 * warp; q0 < nc; q0 += 4 * W_NW) {
            const int q = q0 + (lane >> 3), c = crank + CS * q;
            const bool act = q < nc && c != pc && sigl[q] >= 0.0;
            double *tc = Tl + (size_t)q * K;
            double tj = act ? tc[j] : 0.0, w0 = 0.0, w1 = 0.0;
            int r = j + 1 + gl;
            if (act) {
#pragma unroll 2
                for (; r + 8 < K; r += 16) {
                    w0 = fma(hv[r], tc[r], w0);
                    w1 = fma(hv[r + 8], tc[r + 8], w1);
                }
                if (r < K) w0 = fma(hv[r], tc[r], w0);
            }
            double w = group_sum<8>(w0 + w1);
            w = fma(alpha - beta, tj, w) * th;
            double s0 = 0.0, s1 = 0.0;
            r = j + 1 + gl;
            if (act) {
#pragma unroll 2
                for (; r + 8 < K; r += 16) {
                    const double x0 = fma(-w, hv[r], tc[r]), x1 = fma(-w, hv[r + 8], tc[r + 8]);
                    tc[r] = x0;
                    tc[r + 8] = x1;
                    s0 = fma(x0, x0, s0);
                    s1 = fma(x1, x1, s1);
                }
                if (r < K) {
                    const double x0 = fma(-w, hv[r], tc[r]);
                    tc[r] = x0;
                    s0 = fma(x0, x0, s0);
                }
            }
            const double s2 = group_sum<8>(s0 + s1);
            __syncwarp();
            if (gl == 0 && q < nc) {
                // row j of R: beta at the pivot, zero at the earlier pivots
                X[(size_t)j * K + c] = c == pc ? beta : (act ? fma(-w, alpha - beta, tj) : 0.0);
                sigl[q] = act ? s2 : -1.0;
            }
        }
        __syncthreads();
    }
    if (!HV) cl.sync();                       // hv lies in columns that are zeroed now
    // blocks past k: zero columns
    const int nblk = max(2, (k + WB - 1) / WB), nbp = nblk + (nblk & 1);
    for (long long idx = (long long)k * K + gt; idx < (long long)nblk * WB * K && idx < (long long)K * (K + WP); idx += GT)
        X[idx] = 0.0;
    cl.sync();

    // 3. block Jacobi on the columns of X
    double *G = sm, *Jm = G + WP * WLD, *red = Jm + WP * WLD;   // the QR's shared memory is free
    const int gblk[1] = {tri_block(min(tid, WP / 2 * (WP / 2 + 1) / 2 - 1))};      // this thread's block of G
    const double tolj = 4.4e-16 * (double)(K > 16 ? K : 16), tol2 = tolj * tolj;
    int sweeps = 0;
    while (k > 1 && sweeps < MAX_SWEEPS) {
        for (int round = 0; round < nbp - 1; ++round) {
            for (int pr = crank; pr < nbp / 2; pr += CS) {
                const int ba = tourney(pr, round, nbp), bb = tourney(nbp - 1 - pr, round, nbp);
                if (max(ba, bb) >= nblk) continue;
                // local column m: block ba (m < 16) or bb
                auto colp = [&](int m) { return X + (size_t)((m < WB ? ba * WB : bb * WB - WB) + m) * K; };
                // Gram matrix: the warps take row quads in turn, then their partials are added in warp order
                double acc[W_TILES][2];
#pragma unroll
                for (int q = 0; q < W_TILES; ++q) acc[q][0] = acc[q][1] = 0.0;
                const double *cp0 = colp(g), *cp1 = colp(8 + g), *cp2 = colp(16 + g), *cp3 = colp(24 + g);
#pragma unroll 4
                for (int c0 = 4 * warp; c0 < K; c0 += 4 * W_NW) {
                    const int c = c0 + tig;
                    const bool in = c < K;
                    const double a0 = in ? ldg2(cp0 + c) : 0.0, a1 = in ? ldg2(cp1 + c) : 0.0;
                    const double a2 = in ? ldg2(cp2 + c) : 0.0, a3 = in ? ldg2(cp3 + c) : 0.0;
                    const double a[4] = {a0, a1, a2, a3};
                    int q = 0;
#pragma unroll
                    for (int I = 0; I < 4; ++I)
#pragma unroll
                        for (int J = 0; J <= I; ++J, ++q) dmma884(acc[q], a[I], a[J]);
                }
#pragma unroll
                for (int q = 0; q < W_TILES; ++q)
#pragma unroll
                    for (int e = 0; e < 2; ++e) red[(warp * W_TILES + q) * 64 + g * 8 + 2 * tig + e] = acc[q][e];
                __syncthreads();
                for (int idx = tid; idx < W_TILES * 64; idx += W_CT) {
                    double v = 0.0;
#pragma unroll
                    for (int w = 0; w < W_NW; ++w) v += red[w * W_TILES * 64 + idx];
                    const int q = idx >> 6, I = q >= 6 ? 3 : q >= 3 ? 2 : q >= 1 ? 1 : 0, J = q - I * (I + 1) / 2;
                    const int i = 8 * I + ((idx & 63) >> 3), jj = 8 * J + (idx & 7);
                    if (jj <= i) G[i * WGD + jj] = v;
                }
                for (int idx = tid; idx < WP * WP; idx += W_CT)
                    Jm[(idx >> 5) * WLD + (idx & 31)] = (idx >> 5) == (idx & 31) ? 1.0 : 0.0;
                __syncthreads();
                int need = 0;
                for (int idx = tid; idx < WP * WP; idx += W_CT) {
                    const int i = idx >> 5, jj = idx & 31;
                    if (jj < i) {
                        double va = G[i * WGD + i], vb = G[jj * WGD + jj], vc = G[i * WGD + jj];
                        need |= pair_scaled(va, vb, vc, tau2, tol2);
                    }
                }
                if (!__syncthreads_or(need)) continue;
                if (tid == 0) atomicExch(rotf + sweeps, 1);
                // rotations: every pair in the sweep's first round (each block is in one
                // problem then; with an odd number of blocks the one left out is in the
                // second round's), the pairs across the two blocks in the others; warp 0
                // finds the next round's while the other warps rotate J
                const bool full = round == 0 || (round == 1 && (nblk & 1));
                const int nr = full ? WP - 1 : WB;
                auto angles = [&](int rr) {
                    if (tid >= WP / 2) return;
                    const int a = full ? tourney(tid, rr, WP) : tid;
                    const int b = full ? tourney(WP - 1 - tid, rr, WP) : WB + ((tid + rr) & (WB - 1));
                    rot[rr & 1][tid] = pair_rotation(G[a * WGD + a], G[b * WGD + b], G[low(a, b, WGD)], tau2, tol2);
                    pab[rr & 1][tid] = a | (b << 16);
                };
                angles(0);
                __syncthreads();
                for (int rr = 0; rr < nr; ++rr) {
                    const double2 *rt = rot[rr & 1];
                    const int *pp = pab[rr & 1];
                    if (tid < WP / 2 * (WP / 2 + 1) / 2) rotate_blocks<1>(G, WGD, gblk, rt, pp);
                    __syncthreads();
                    if (warp == 0) {
                        if (rr + 1 < nr) angles(rr + 1);
                    } else {
                        const double2 r = rt[tid & 15];
                        // seven warps, two rows a warp: rows 0..27, then 28..31
                        const int c = 2 * (warp - 1) + (lane >> 4);
                        if (r.y != 0.0) {
                            rotate_rows<2>(Jm, WLD, pp[tid & 15], r, c, 2 * (W_NW - 1));
                            if (c < WP - 4 * (W_NW - 1)) rotate_rows<1>(Jm, WLD, pp[tid & 15], r, c + 4 * (W_NW - 1), 1);
                        }
                    }
                    __syncthreads();
                }
                // X <- X J on the pair's columns, eight rows at a time
                double jb[8][4];
#pragma unroll
                for (int k4 = 0; k4 < 8; ++k4)
#pragma unroll
                    for (int n = 0; n < 4; ++n) jb[k4][n] = Jm[(4 * k4 + tig) * WLD + 8 * n + g];
                for (int c0 = 8 * warp; c0 < K; c0 += 8 * W_NW) {
                    const int c = c0 + g;
                    double a[8], o[4][2];
#pragma unroll
                    for (int k4 = 0; k4 < 8; ++k4) a[k4] = c < K ? ldg2(colp(4 * k4 + tig) + c) : 0.0;
#pragma unroll
                    for (int n = 0; n < 4; ++n) o[n][0] = o[n][1] = 0.0;
#pragma unroll
                    for (int k4 = 0; k4 < 8; ++k4)
#pragma unroll
                        for (int n = 0; n < 4; ++n) dmma884(o[n], a[k4], jb[k4][n]);
                    if (c < K) {
#pragma unroll
                        for (int n = 0; n < 4; ++n) {
                            colp(8 * n + 2 * tig)[c] = o[n][0];
                            colp(8 * n + 2 * tig + 1)[c] = o[n][1];
                        }
                    }
                }
                __syncthreads();
            }
            cl.sync();
        }
        ++sweeps;
        if (!ldg2(rotf + sweeps - 1)) break;
    }

    // 4. singular values, descending order, rank, left singular vectors
    for (int c = gw; c < k; c += GW) {
        double s = 0.0;
        for (int r = lane; r < K; r += 32) { const double x = ldg2(X + (size_t)c * K + r); s = fma(x, x, s); }
        s = group_sum<32>(s);
        if (lane == 0) sig[c] = sqrt(s);
    }
    cl.sync();
    // every CTA orders them (in T's place, where that is free) and finds the rank (one
    // reports it)
    double *sg = (t_in_smem ? sm : t.work) + L.sort;
    int *order = (int *)(sg + K);
    int nge = 0;
    for (int c0 = 0; c0 < k; c0 += W_CT) {
        const int c = c0 + tid;
        if (c < k) {
            sg[c] = ldg2(sig + c);
            order[c] = c;
        }
        nge += __syncthreads_count(c < k && sg[c] >= p.tol);
    }
    __syncthreads();
    for (int c = tid; c < k; c += W_CT) {
        const double sc = sg[c];
        int pos = 0;
        for (int l = 0; l < k; ++l) {
            const double sl = sg[l];
            pos += (sl > sc) || (sl == sc && l < c);
        }
        order[pos] = c;
    }
    __syncthreads();
    if (tid == 0) {
        CoreParams q = p;
        if (crank != 0) q.overflow = nullptr;
        const int r = core_rank(q, K, k, dropped, nge, [&](int i) { return sg[order[i]]; });
        rank_sh = r;
        if (crank == 0) {
            if (t.rank_out) *t.rank_out = r;
            if (t.rank_task) *t.rank_task = r;
            if (p.sweeps) atomicAdd(p.sweeps, sweeps);
        }
    }
    __syncthreads();
    const int r = rank_sh;
    for (int i = gw; i < r; i += GW) {
        const int c = i < k ? order[i] : 0;
        const double s = i < k ? sg[c] : 0.0;
        for (int q = lane; q < K; q += 32)
            t.SU[(size_t)q + (size_t)i * K] = s > 0.0 ? ldg2(X + (size_t)c * K + q) / s : 0.0;
    }
}

template <int KM>
void launch_small(const CoreTask *d, int n, const CoreParams &p, cudaStream_t st) {
    using S = SmallCore<KM>;
    // per device and thread-safe: set on every launch (a host-side call, no synchronisation)
    cudaFuncSetAttribute(k_core_small<KM>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)S::bytes);
    k_core_small<KM><<<n, S::NT, S::bytes, st>>>(d, p);
}

}  // namespace

// One CTA beats a cluster at any width when the launch fills the device, but its
// latency grows with K (K = 80: 0.79 ms against 0.5 ms on four CTAs): cores of
// 65 to SMALL_KMAX columns take either kernel, so they bring scratch.
int core_smem_kmax() { return 64; }

size_t core_work_doubles(int K, size_t smem_limit) { return wide_work_doubles(K, std::min(smem_limit, W_SMEM_MAX)); }

int core_bucket(int K, bool cluster) {
    if (K <= 64) return K <= 16 ? 16 : K <= 32 ? 32 : K <= 48 ? 48 : 64;
    if (K <= SMALL_KMAX && !cluster) return K <= 80 ? 80 : SMALL_KMAX;
    return K <= W_EDGE1 ? W_EDGE1 : K <= W_EDGE2 ? W_EDGE2 : 1 << 30;
}
int core_one_cta_kmax() { return SMALL_KMAX; }

void launch_core_svd_batched(const CoreTask *d_tasks, int ntasks, int kmax, const CoreParams &p, bool cluster,
                             size_t smem_limit, cudaStream_t st) {
    if (ntasks <= 0) return;
    if (kmax <= 16) return launch_small<16>(d_tasks, ntasks, p, st);
    if (kmax <= 32) return launch_small<32>(d_tasks, ntasks, p, st);
    if (kmax <= 48) return launch_small<48>(d_tasks, ntasks, p, st);
    if (kmax <= 64) return launch_small<64>(d_tasks, ntasks, p, st);
    if (kmax <= 80 && !cluster) return launch_small<80>(d_tasks, ntasks, p, st);
    if (kmax <= SMALL_KMAX && !cluster) return launch_small<96>(d_tasks, ntasks, p, st);
    int cs = wide_cluster(kmax);
    for (;;) {
        const int place = wide_place(kmax, cs, std::min(smem_limit, W_SMEM_MAX));
        const size_t smem = wide_smem(kmax, cs, place);
        auto *kernel = place & W_HV_SHARED ? k_core_wide<true> : k_core_wide<false>;
        // the limit belongs to the function, for all threads of the process: always the same
        // value, so that a launch of another context never lowers it in between
        cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)W_SMEM_MAX);
        cudaFuncSetAttribute(kernel, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
        cudaLaunchConfig_t cfg = {};
        cfg.gridDim = dim3((unsigned)ntasks * cs);
        cfg.blockDim = dim3(W_CT);
        cfg.dynamicSmemBytes = smem;
        cfg.stream = st;
        cudaLaunchAttribute at[1];
        at[0].id = cudaLaunchAttributeClusterDimension;
        at[0].val.clusterDim.x = cs;
        at[0].val.clusterDim.y = 1;
        at[0].val.clusterDim.z = 1;
        cfg.attrs = at;
        cfg.numAttrs = 1;
        if (cs > 8) {
            // 16 CTAs need a GPC with that many SMs free: take 8 where none has them
            int n = 0;
            if (cudaOccupancyMaxActiveClusters(&n, kernel, &cfg) != cudaSuccess || n < 1) {
                cudaGetLastError();
                cs = 8;
                continue;
            }
        }
        cudaLaunchKernelEx(&cfg, kernel, d_tasks, p, place);
        return;
    }
}

}  // namespace tlr
