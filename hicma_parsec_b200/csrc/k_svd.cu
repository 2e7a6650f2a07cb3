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
#include "tlr_internal.h"

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
__device__ __forceinline__ bool pair_rotation(double aa, double bb, double cc, double tau2, double tol2, double &cs,
                                              double &sn) {
    cs = 1.0;
    sn = 0.0;
    if (!pair_scaled(aa, bb, cc, tau2, tol2)) return false;
    const double d = bb - aa;
    const double rh = rsqrt(fma(d, d, 4.0 * cc * cc));
    const double c2 = fma(0.5 * fabs(d), rh, 0.5);
    const double rc = rsqrt(c2);
    cs = c2 * rc;
    sn = copysign(1.0, d) * cc * rh * rc;
    return true;
}

// 2 x 2 block of G at rows (a0, b0) and columns (a1, b1): rotated by the row
// pair's (c0, s0) and the column pair's (c1, s1).
__device__ __forceinline__ void rotate_block(double *G, int ld, int a0, int b0, double c0, double s0, int a1, int b1,
                                             double c1, double s1, bool diag) {
    double *pa = G + a0 * ld, *pb = G + b0 * ld;
    const double gaa = pa[a1], gab = pa[b1], gba = pb[a1], gbb = pb[b1];
    const double u0 = c1 * gaa - s1 * gab, u1 = s1 * gaa + c1 * gab;
    const double v0 = c1 * gba - s1 * gbb, v1 = s1 * gba + c1 * gbb;
    pa[a1] = c0 * u0 - s0 * v0;
    pb[b1] = s0 * u1 + c0 * v1;
    // a diagonal block holds its own pair: the rotation made it zero
    pa[b1] = diag ? 0.0 : c0 * u1 - s0 * v1;
    pb[a1] = diag ? 0.0 : s0 * u0 + c0 * v0;
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
// Against one CTA with dot products reduced over 8 or 16 lanes and two to three
// shuffles a value (the form before): the cores of the 60 x 60 tiles of 2700 2D
// workload (34,220 of K up to 100) 142 -> 74 ms, 20 x 20 tiles of 1350 90 -> 33 ms.
template <int KM>
struct SmallCore {
    static constexpr int NT = 4 * KM;
    static constexpr int NW = NT / 32;
    static constexpr int P = KM + 4;          // == 4 mod 16: conflict-free DMMA fragments
    static constexpr int NT8 = KM / 8;
    static constexpr size_t doubles = 2 * (size_t)KM * P + 2 * KM + KM;   // X, G, sig, hv, (cs, sn)
    static constexpr size_t bytes = sizeof(double) * doubles + sizeof(int) * 2 * KM;
};

template <int KM>
__global__ void __launch_bounds__(4 * KM) k_core_small(const CoreTask *__restrict__ tasks, CoreParams p) {
    using S = SmallCore<KM>;
    constexpr int NT = S::NT, NW = S::NW, P = S::P, NT8 = S::NT8;
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
    double *G = X + KM * P;
    double *sig = G + KM * P;
    double *hv = sig + KM;
    double2 *rot = (double2 *)(hv + KM);      // KM / 2 rotations of a round
    int *order = (int *)(rot + KM / 2);
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
    // largest squared norm (scale of the pivot keys) and their sum
    double nmax = 0.0, total = 0.0;
#pragma unroll
    for (int s = 0; s < NSLOT; ++s) {
        const double v = lane + 32 * s < KM ? sig[lane + 32 * s] : 0.0;
        nmax = fmax(nmax, v);
        total += v;
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) nmax = fmax(nmax, __shfl_xor_sync(0xffffffffu, nmax, o));
    total = group_sum<32>(total);
    const double tau2 = trunc_floor(p, total);
    const double kscale = nmax > 1e-290 && nmax < 1e290 ? 1.0 / nmax : 1.0;

    // 2. pivoted Householder QR of T, stopped when the trailing mass <= tau2
    unsigned done[NSLOT];                     // columns this lane scans that were pivots already
#pragma unroll
    for (int s = 0; s < NSLOT; ++s) done[s] = lane + 32 * s >= K;
    int k = K;
    double dropped = 0.0;
    for (int j = 0; j < K; ++j) {
        // pivot: the column of largest norm (single-precision keys of the
        // scaled norms; the lowest index of equal ones)
        unsigned best = 0u;
        int bc = 0;
        double tr = 0.0;
#pragma unroll
        for (int s = 0; s < NSLOT; ++s) {
            if (!done[s]) {
                const double v = sig[lane + 32 * s];
                tr += v;
                const unsigned key = __float_as_uint((float)(v * kscale)) + 1u;
                if (key > best) { best = key; bc = lane + 32 * s; }
            }
        }
        const unsigned top = __reduce_max_sync(0xffffffffu, best);
        int pc = __reduce_min_sync(0xffffffffu, best == top ? bc : KM);
        tr = group_sum<32>(tr);
        if (!(tr > tau2)) { k = j; dropped = tr; break; }    // the same in every warp
        pc = min(pc, KM - 1);
        const double n2 = sig[pc];
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
        const double beta = -copysign(sqrt(n2), alpha);
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
    const int L = np <= 8 ? 8 : np <= 16 ? 16 : 32;   // lanes over pairs
    const int RS = 32 / L;                            // rows a warp takes at a time
    const int li = lane % L, lr = warp * RS + lane / L, rstep = NW * RS;
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
            for (int e = 0; e < 2; ++e) {
                const double v = a0[e] + a1[e];
                G[(8 * I + g) * P + 8 * J + 2 * tig + e] = v;
                G[(8 * J + 2 * tig + e) * P + 8 * I + g] = v;
            }
        }
        __syncthreads();
        if (sweeps >= MAX_SWEEPS) break;
        int need = 0;
        for (int idx = tid; idx < k * k; idx += NT) {
            const int i = idx / k, jj = idx - i * k;
            if (jj < i) {
                double aa = G[i * P + i], bb = G[jj * P + jj], cc = G[i * P + jj];
                need |= pair_scaled(aa, bb, cc, tau2, tol2);
            }
        }
        if (!__syncthreads_or(need)) break;
        ++sweeps;
        for (int round = 0; round < kp - 1; ++round) {
            for (int pr = tid; pr < np; pr += NT) {
                const int a = tourney(pr, round, kp), b = tourney(kp - 1 - pr, round, kp);
                double cs = 1.0, sn = 0.0;
                if (max(a, b) < k) pair_rotation(G[a * P + a], G[b * P + b], G[a * P + b], tau2, tol2, cs, sn);
                rot[pr] = make_double2(cs, sn);
                pab[pr] = a | (b << 16);
            }
            __syncthreads();
            for (int I = li; I < np; I += L) {
                const double2 ri = rot[I];
                const int ab = pab[I], a = ab & 0xffff, b = ab >> 16;
                for (int J = lr; J < np; J += rstep) {
                    const double2 rj = rot[J];
                    if (ri.y == 0.0 && rj.y == 0.0) continue;
                    const int abj = pab[J];
                    rotate_block(G, P, abj & 0xffff, abj >> 16, rj.x, rj.y, a, b, ri.x, ri.y, I == J);
                }
                if (ri.y != 0.0) {
                    for (int c = lr; c < K; c += rstep) {
                        const double xa = X[c * P + a], xb = X[c * P + b];
                        X[c * P + a] = ri.x * xa - ri.y * xb;
                        X[c * P + b] = ri.y * xa + ri.x * xb;
                    }
                }
            }
            __syncthreads();
        }
    }

    // 4. singular values (from the fresh Gram matrix), descending order, rank
    for (int c = tid; c < k; c += NT) {
        sig[c] = sqrt(G[c * P + c]);
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
// Two launches of three cores and one of K about 650 (k about 430): 470 -> 38 ms
// against one warp per column pair reading its columns through L2.
constexpr int WB = 16;                        // columns of a block
constexpr int WP = 2 * WB;                    // columns of a pair problem
constexpr int WLD = WP + 4;                   // pitch of its G and J
constexpr int W_CT = 256;
constexpr int W_NW = W_CT / 32;
constexpr int W_TILES = 10;                   // lower 8 x 8 tiles of the 32 x 32 Gram matrix
constexpr int W_CSMAX = 16;
constexpr size_t W_JACOBI_DOUBLES = 2 * WP * WLD + W_NW * W_TILES * 64;
constexpr size_t W_SMEM_MAX = 220 * 1024;

__device__ __forceinline__ double ldg2(const double *p) { return __ldcg(p); }
__device__ __forceinline__ int ldg2(const int *p) { return __ldcg(p); }

struct WidePub {
    double norm, sum;
    int col, pad;
};

// columns of T a CTA holds
__host__ __device__ __forceinline__ int wide_ncl(int K, int cs) { return (K + cs - 1) / cs; }

__global__ void __launch_bounds__(W_CT) k_core_wide(const CoreTask *__restrict__ tasks, CoreParams p, int t_in_smem) {
    namespace cg = cooperative_groups;
    cg::cluster_group cl = cg::this_cluster();
    extern __shared__ __align__(16) double sm[];
    __shared__ WidePub pub[2][W_CSMAX];
    __shared__ double2 rot[WP / 2];
    __shared__ int pab[WP / 2];
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
    // task scratch: X (K x (K + 32)), sigma, T when it does not fit, flags
    double *X = t.work;
    double *sig = X + (size_t)K * (K + WP);
    double *Tg = sig + K;
    int *rotf = (int *)(Tg + (size_t)K * (K + W_CSMAX));  // [sweep]: a pair was rotated
    const int ncl = wide_ncl(K, CS);
    double *hv = sm;                          // K
    double *sigl = hv + K;                    // ncl: squared norms of the CTA's columns, -1 once pivots
    double *Ts = sigl + ncl + ((K + ncl) & 1);
    const int nc = crank < K ? (K - crank + CS - 1) / CS : 0;   // columns this CTA holds
    double *Tl = t_in_smem ? Ts : Tg + (size_t)crank * ncl * K;

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
            double tr = 0.0, best = -1.0;
            int bc = 0x7fffffff;
            for (int q = lane; q < nc; q += 32) {
                const double v = sigl[q];
                if (v < 0.0) continue;
                tr += v;
                if (v > best) { best = v; bc = crank + CS * q; }
            }
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) {
                tr += __shfl_xor_sync(0xffffffffu, tr, o);
                const double ob = __shfl_xor_sync(0xffffffffu, best, o);
                const int oc = __shfl_xor_sync(0xffffffffu, bc, o);
                if (ob > best || (ob == best && oc < bc)) { best = ob; bc = oc; }
            }
            if (lane < CS) {
                WidePub *d = cl.map_shared_rank(&pub[par][crank], lane);
                d->norm = best;
                d->sum = tr;
                d->col = bc;
            }
        }
        cl.sync();
        double tr = 0.0, n2 = -1.0;
        int pc = 0x7fffffff;
        for (int r = 0; r < CS; ++r) {
            const double v = pub[par][r].norm;
            const int c = pub[par][r].col;
            tr += pub[par][r].sum;
            if (v > n2 || (v == n2 && c < pc)) { n2 = v; pc = c; }
        }
        if (j == 0) tau2 = trunc_floor(p, tr);
        if (!(tr > tau2) || pc >= K) { k = j; dropped = tr; break; }   // the same in every CTA
        // the pivot column, from its owner's memory (nothing writes it any more)
        const int owner = pc % CS, lp = pc / CS;
        if (t_in_smem) {
            const double *src = cl.map_shared_rank(Ts, owner) + (size_t)lp * K;
            for (int r = j + tid; r < K; r += W_CT) hv[r] = src[r];
        } else {
            const double *src = Tg + ((size_t)owner * ncl + lp) * K;
            for (int r = j + tid; r < K; r += W_CT) hv[r] = ldg2(src + r);
        }
        __syncthreads();
        const double alpha = hv[j];
        const double beta = -copysign(sqrt(n2), alpha);
        const double den = fma(-alpha, beta, n2);
        const double th = den > 0.0 ? 1.0 / den : 0.0;
        for (int q = warp; q < nc; q += W_NW) {
            const int c = crank + CS * q;
            const bool act = sigl[q] >= 0.0;
            double rj = 0.0;
            if (c == pc) {
                rj = beta;
            } else if (act) {
                double *tc = Tl + (size_t)q * K;
                double w = 0.0;
#pragma unroll 4
                for (int r = j + lane; r < K; r += 32) w = fma(r == j ? alpha - beta : hv[r], tc[r], w);
                w = group_sum<32>(w) * th;
                double s2 = 0.0;
#pragma unroll 4
                for (int r = j + lane; r < K; r += 32) {
                    const double x = fma(-w, r == j ? alpha - beta : hv[r], tc[r]);
                    tc[r] = x;
                    if (r == j) rj = x;
                    else s2 = fma(x, x, s2);
                }
                s2 = group_sum<32>(s2);
                if (lane == 0) sigl[q] = s2;
            }
            if (lane == 0) {
                X[(size_t)j * K + c] = rj;       // row j of R: zero at the earlier pivots
                if (c == pc) sigl[q] = -1.0;
            }
        }
        __syncthreads();
    }
    // blocks past k: zero columns
    const int nblk = max(2, (k + WB - 1) / WB), nbp = nblk + (nblk & 1);
    for (long long idx = (long long)k * K + gt; idx < (long long)nblk * WB * K && idx < (long long)K * (K + WP); idx += GT)
        X[idx] = 0.0;
    cl.sync();

    // 3. block Jacobi on the columns of X
    double *G = sm, *Jm = G + WP * WLD, *red = Jm + WP * WLD;   // the QR's shared memory is free
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
                    G[i * WLD + jj] = v;
                    G[jj * WLD + i] = v;
                }
                for (int idx = tid; idx < WP * WP; idx += W_CT)
                    Jm[(idx >> 5) * WLD + (idx & 31)] = (idx >> 5) == (idx & 31) ? 1.0 : 0.0;
                __syncthreads();
                int need = 0;
                for (int idx = tid; idx < WP * WP; idx += W_CT) {
                    const int i = idx >> 5, jj = idx & 31;
                    if (jj < i) {
                        double va = G[i * WLD + i], vb = G[jj * WLD + jj], vc = G[i * WLD + jj];
                        need |= pair_scaled(va, vb, vc, tau2, tol2);
                    }
                }
                if (!__syncthreads_or(need)) continue;
                if (tid == 0) atomicExch(rotf + sweeps, 1);
                for (int rr = 0; rr < WP - 1; ++rr) {
                    if (tid < WP / 2) {
                        const int a = tourney(tid, rr, WP), b = tourney(WP - 1 - tid, rr, WP);
                        double cs, sn;
                        pair_rotation(G[a * WLD + a], G[b * WLD + b], G[a * WLD + b], tau2, tol2, cs, sn);
                        rot[tid] = make_double2(cs, sn);
                        pab[tid] = a | (b << 16);
                    }
                    __syncthreads();
                    const int I = tid & 15, r0 = tid >> 4;
                    const double2 ri = rot[I], rj = rot[r0];
                    const int a = pab[I] & 0xffff, b = pab[I] >> 16;
                    if (ri.y != 0.0 || rj.y != 0.0)
                        rotate_block(G, WLD, pab[r0] & 0xffff, pab[r0] >> 16, rj.x, rj.y, a, b, ri.x, ri.y, I == r0);
                    if (ri.y != 0.0) {
#pragma unroll
                        for (int h = 0; h < 2; ++h) {
                            double *jr = Jm + (r0 + 16 * h) * WLD;
                            const double xa = jr[a], xb = jr[b];
                            jr[a] = ri.x * xa - ri.y * xb;
                            jr[b] = ri.y * xa + ri.x * xb;
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
    // every CTA orders them and finds the rank (one reports it)
    double *sg = sm;
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

size_t wide_smem(int K, int cs, bool t_in_smem) {
    const size_t ncl = wide_ncl(K, cs);
    const size_t qr = (size_t)K + ncl + 1 + (t_in_smem ? ncl * K : 0);
    return sizeof(double) * (qr > W_JACOBI_DOUBLES ? qr : W_JACOBI_DOUBLES);
}

// CTAs of a cluster: about one per pair problem of the Jacobi rounds (k / 32
// pairs, k about K / 2) and enough shared memory for T: 4 up to K = 160, 8 up
// to 448, then 16 (the non-portable maximum).
int wide_cluster(int K) { return K <= 160 ? 4 : K <= 448 ? 8 : W_CSMAX; }

}  // namespace

int core_smem_kmax() { return SMALL_KMAX; }

size_t core_work_doubles(int K) { return (size_t)K * (K + WP) + (size_t)K * (K + W_CSMAX) + (size_t)K + 64; }

int core_bucket(int K) {
    if (K <= 64) return K <= 16 ? 16 : K <= 32 ? 32 : K <= 48 ? 48 : 64;
    if (K <= SMALL_KMAX) return K <= 80 ? 80 : 96;
    return K <= 160 ? 160 : K <= 448 ? 448 : 1 << 30;
}

void launch_core_svd_batched(const CoreTask *d_tasks, int ntasks, int kmax, const CoreParams &p,
                             cudaStream_t st) {
    if (ntasks <= 0) return;
    if (kmax <= 16) return launch_small<16>(d_tasks, ntasks, p, st);
    if (kmax <= 32) return launch_small<32>(d_tasks, ntasks, p, st);
    if (kmax <= 48) return launch_small<48>(d_tasks, ntasks, p, st);
    if (kmax <= 64) return launch_small<64>(d_tasks, ntasks, p, st);
    if (kmax <= 80) return launch_small<80>(d_tasks, ntasks, p, st);
    if (kmax <= SMALL_KMAX) return launch_small<96>(d_tasks, ntasks, p, st);
    int cs = wide_cluster(kmax);
    for (;;) {
    // T in the cluster's shared memory where a CTA's share fits
        const bool in_smem = wide_smem(kmax, cs, true) <= W_SMEM_MAX;
        const size_t smem = wide_smem(kmax, cs, in_smem);
        cudaFuncSetAttribute(k_core_wide, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
        cudaFuncSetAttribute(k_core_wide, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
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
            if (cudaOccupancyMaxActiveClusters(&n, k_core_wide, &cfg) != cudaSuccess || n < 1) {
                cudaGetLastError();
                cs = 8;
                continue;
            }
        }
        cudaLaunchKernelEx(&cfg, k_core_wide, d_tasks, p, in_smem ? 1 : 0);
        return;
    }
}

}  // namespace tlr
