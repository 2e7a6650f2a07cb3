// Tile Cholesky and tile inverse in one persistent launch.
//
// Replaces HCORE_dpotrf on a diagonal tile (hicma_parsec/HiCMA_dpotrf_L_2flow.jdf
// :233-242) together with the inverse L^-1 that the panel solves of this
// engine apply as a GEMM.  The tile is split into 64 x 64 blocks, and a blocked
// left-looking algorithm becomes a list of tasks:
//   CHAIN        the critical path, run by one CTA from start to end: for each
//                block column j, Cholesky of A_jj and D_j = L_jj^-1, then
//                L_j+1,j = S_j+1,j D_j^T and S_j+1,j+1 -= L_j+1,j L_j+1,j^T,
//                the next diagonal block staying in shared memory
//   PRE(k)       S_k+1,{k,k+1} = A_k+1,{k,k+1} - sum_{j<k} L_k+1,j L_{k,k+1},j^T
//   LT(i,k)      L_{i,i+1},k = (A_{i,i+1},k - sum_{j<k} L_{i,i+1},j L_kj^T) D_k^T
//                                                               (i >= k + 2)
//   XT(i,p)      X_i,{2p,2p+1} = -D_i sum_{2p<=j<i} L_ij X_j,{2p,2p+1}
// where X = L^-1 is produced by block forward substitution.  A task keeps its
// 128 x 64 or 64 x 128 tile in the accumulators over all of its sum, reading
// each block once as it becomes final, so that the tile is read and written
// once and the waits overlap the products of the blocks before them.  The chain
// is the first task; the rest of the list is in a topological order and CTAs
// take tasks from it with an atomic ticket, so every task waits only on the
// chain or on tasks already held by running CTAs, and the chain waits only on
// tasks of earlier block columns, which the other CTAs take in list order: the
// kernel makes progress with two or more CTAs and needs no cooperative launch.  A CTA
// that waits holds its place on an SM, so beside the chain a second one has to become
// resident; it does when any block of another kernel ends.  Dependencies are per-block flags
// released with a fence after the block is written and acquired by one thread
// before the CTA reads (through L2: ld.global.cg).  Every wait is bounded; a wait
// that gives up sets the timeout flag and the abort flag, and every CTA leaves
// at its next wait or task.  A non-positive pivot sets the reference's INFO
// (k*NB + iinfo) and aborts the same way.  The block products run on the FP64
// tensor cores (mma.sync m8n8k4 f64).
// Bound by the chain (43 steps of about 24 us for a tile of 2700) when one CTA runs
// on every SM, by the DMMA rate of its CTAs below about 100.  Against one task per
// 64 x 64 x 64 block product (right-looking, C read and written for each of them, 20k
// cycles a product of which DMMA 4.1k): tile of 2700 with its inverse 2.00 -> 1.13 ms
// on 148 CTAs, 4.1 -> 1.67 ms on 64, 7.8 -> 3.05 ms on 32; tile of 1350 0.64 -> 0.54 ms.
#include "tlr_internal.h"

#include <map>
#include <mutex>
#include <vector>

namespace tlr {
namespace {

constexpr int TB = 64;          // block edge
constexpr int CP = TB + 4;      // shared pitch of the chain CTA's blocks (conflict-free DMMA fragments)
constexpr int NTH = 256;
constexpr int XLAG = 6;         // block columns by which the inverse's rows follow the factor's (0: 6 % slower, 2: 3 %)
constexpr long long SPIN_LIMIT = 1LL << 24;

enum { IT_CHAIN = 0, IT_PRE, IT_LT, IT_XT };
struct PItem {
    unsigned short type, i, k, pad;   // k: block column, or column pair of XT
};

struct PotrfParams {
    double *A;
    int lda, n, nblk;
    double *X;          // L^-1 (zeroed), or null
    int ldx;
    double *D;          // nblk x (64 x 64) block inverses when X is null
    const PItem *items;
    int nitems;
    int *cnt;           // [0] ticket [1] abort, then pdone, xdone (nblk^2 each), ddone, vpre (nblk each)
    int *info;
    int info_base;
    int *timeout;
    int v16;                // A and X are 16-byte aligned, with even leading dimensions
    long long spin_limit;   // polls before a wait gives up (SPIN_LIMIT in production)
};

__device__ __forceinline__ void dmma884(double (&d)[2], double a, double b) {
    asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0,%1}, {%2}, {%3}, {%0,%1};\n"
                 : "+d"(d[0]), "+d"(d[1])
                 : "d"(a), "d"(b));
}

__device__ __forceinline__ int ld_volatile(const int *p) { return *(const volatile int *)p; }

// thread 0 only: wait until *p >= v
__device__ bool wait_ge(const int *p, int v, const PotrfParams &P) {
    for (long long it = 0; it < P.spin_limit; ++it) {
        if (ld_volatile(p) >= v) {
            __threadfence();
            return true;
        }
        if (ld_volatile(P.cnt + 1)) return false;
        __nanosleep(it < 256 ? 32 : 256);
    }
    atomicExch(P.timeout, 1);
    atomicExch(P.cnt + 1, 1);
    return false;
}

__device__ __forceinline__ int bsz(int b, int n) { return min(TB, n - b * TB); }

// Flags of the task queue.
struct PFlags {
    int *pdone, *xdone, *ddone, *vpre;
    int nb;
    __device__ PFlags(const PotrfParams &P) : nb(P.nblk) {
        pdone = P.cnt + 8;
        xdone = pdone + nb * nb;
        ddone = xdone + nb * nb;
        vpre = ddone + nb;
    }
    __device__ int *p(int i, int j) const { return pdone + i * nb + j; }   // L_ij is final
    __device__ int *x(int i, int q) const { return xdone + i * nb + q; }   // X_i,{2q,2q+1} is final
};

// ------------------------------------------------------------ bulk tasks ----
// Inner step: 32 with cp.async (fewer barriers, against which one CTA per SM has
// nothing to run), 16 where the next step waits in registers.
template <bool V16>
__host__ __device__ constexpr int pk() { return V16 ? 32 : 16; }

// Flags (at most three) that release inner block j of a task.
struct JDeps {
    const int *a, *b, *c;
};
__device__ __forceinline__ bool deps_ready(const JDeps &d) {
    const int r = ld_volatile(d.a) & ld_volatile(d.b) & ld_volatile(d.c);
    if (r) __threadfence();
    return r;
}
__device__ bool deps_wait(const JDeps &d, const PotrfParams &P) {
    for (long long it = 0; it < P.spin_limit; ++it) {
        if (deps_ready(d)) return true;
        if (ld_volatile(P.cnt + 1)) return false;
        __nanosleep(it < 256 ? 32 : 256);
    }
    atomicExch(P.timeout, 1);
    atomicExch(P.cnt + 1, 1);
    return false;
}

// Warp-wide: how many of the inner blocks j, j + 1, ... below j1 are released (up
// to 32 looked at, so that a task with a backlog polls once for many blocks).
template <class Deps>
__device__ __forceinline__ int deps_count(int j, int j1, int lane, Deps deps) {
    bool r = false;
    if (j + lane < j1) {
        const JDeps d = deps(j + lane);
        r = ld_volatile(d.a) & ld_volatile(d.b) & ld_volatile(d.c);
    }
    const unsigned m = __ballot_sync(0xffffffffu, r);
    if (m & 1u) __threadfence();
    return m == 0xffffffffu ? 32 : __ffs(~m) - 1;
}

// bytes (16, 8 or 0) from gmem through L2, the rest of the 16 zero-filled
__device__ __forceinline__ void cp_async16(unsigned smem, const double *gmem, int bytes) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(smem), "l"(gmem), "r"(bytes));
}
// acc += A B over the inner blocks j0 <= j < j1 (64 each) for an MT x NL tile:
// A (rows x inner, mrows of them valid) column-major; B by op: BKC = false: B^T
// is stored (rows, column-major, nrows valid), true: B is stored (columns,
// contiguous along the inner dimension, nrows valid).  Eight warps of 32 x 32.
// Two shared stages: V16 (bases and leading dimensions 16-byte aligned) filled by
// cp.async through L2, otherwise with the next step's operands in registers
// (8-byte cp.async would go through L1, which may hold a neighbouring block's older
// rows).  The flags of a block are looked at when its first
// step comes up for loading, and waited for only when the products have caught up.
// Each block's 64-term sum is formed on its own before it is added: one running sum
// over up to 2700 terms rounds 2.3 times as far off (tile of 2700, 7.9e-14 against
// 3.4e-14).  A step's loads are issued in parts between its products: as one burst after the
// barrier they held up the fragment reads behind them (12.7k cycles a 128 x 64 x 64
// block against 8.2k of DMMA).  Returns false if a wait gave up or the run was
// aborted.
template <int MT, int NL, bool BKC, bool V16, class Deps>
__device__ bool acc_blocks(double *sm, double (&acc)[4][4][2], const PotrfParams &P, const double *A, int lda,
                           int mrows, const double *B, int ldb, int nrows, int j0, int j1, Deps deps) {
    constexpr int PK = pk<V16>(), PA = MT + 4, PB = BKC ? PK + 4 : NL + 4;
    constexpr int SA = PK * PA, SB = BKC ? NL * PB : PK * PB;
    constexpr int ST = 2, SPB = TB / PK;
    constexpr int W = V16 ? 2 : 1, QA = MT * PK / W / NTH, QB = NL * PK / W / NTH;
    __shared__ int poll_sh[2], wait_sh;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int g = lane >> 2, tig = lane & 3, wm = warp % (MT / 32), wn = warp / (MT / 32);
    if (j0 >= j1) return true;
    const int S = (j1 - j0) * SPB;
    double blk[4][4][2];                  // this block's sum
#pragma unroll
    for (int mi = 0; mi < 4; ++mi)
#pragma unroll
        for (int ni = 0; ni < 4; ++ni) blk[mi][ni][0] = blk[mi][ni][1] = 0.0;
    double ra[V16 ? 1 : QA], rb[V16 ? 1 : QB];
    const unsigned s0 = (unsigned)__cvta_generic_to_shared(sm);
    // part t of NP of step s's operands
    constexpr int NP = PK / 4;
    auto load_part = [&](int s, int t) {
        const int kb = j0 * TB + s * PK;
        const unsigned st = s0 + (unsigned)((s % ST) * (SA + SB) * sizeof(double));
#pragma unroll
        for (int q = 0; q < QA; ++q) {
            if (q < t * QA / NP || q >= (t + 1) * QA / NP) continue;
            const int e = tid + q * NTH, x = (e % (MT / W)) * W, kk = e / (MT / W);
            const double *src = A + x + (size_t)(kb + kk) * lda;
            if constexpr (V16) cp_async16(st + (unsigned)((kk * PA + x) * sizeof(double)), x < mrows ? src : A,
                                          x + 1 < mrows ? 16 : x < mrows ? 8 : 0);
            else ra[q] = x < mrows ? __ldcg(src) : 0.0;
        }
#pragma unroll
        for (int q = 0; q < QB; ++q) {
            if (q < t * QB / NP || q >= (t + 1) * QB / NP) continue;
            const int e = tid + q * NTH;
            if (BKC) {
                const int kk = (e % (PK / W)) * W, x = e / (PK / W);
                const double *src = B + kb + kk + (size_t)x * ldb;
                if constexpr (V16) cp_async16(st + (unsigned)((SA + x * PB + kk) * sizeof(double)), x < nrows ? src : B,
                                              x < nrows ? 16 : 0);
                else rb[q] = x < nrows ? __ldcg(src) : 0.0;
            } else {
                const int x = (e % (NL / W)) * W, kk = e / (NL / W);
                const double *src = B + x + (size_t)(kb + kk) * ldb;
                if constexpr (V16) cp_async16(st + (unsigned)((SA + kk * PB + x) * sizeof(double)), x < nrows ? src : B,
                                              x + 1 < nrows ? 16 : x < nrows ? 8 : 0);
                else rb[q] = x < nrows ? __ldcg(src) : 0.0;
            }
        }
    };
    auto load = [&](int s) {
#pragma unroll
        for (int t = 0; t < NP; ++t) load_part(s, t);
    };
    if (tid == 0) wait_sh = deps_wait(deps(j0), P);
    __syncthreads();
    if (!wait_sh) return false;
    int issued = 0, ready = j0 + 1;       // steps loaded or on their way; blocks known to be released
    load(issued++);
    for (int s = 0; s < S; ++s) {
        double *As = sm + (s % ST) * (SA + SB), *Bs = As + SA;
        if constexpr (V16) {
            asm volatile("cp.async.wait_all;\n" ::: "memory");
        } else {
#pragma unroll
            for (int q = 0; q < QA; ++q) {
                const int e = tid + q * NTH;
                As[(e / MT) * PA + e % MT] = ra[q];
            }
#pragma unroll
            for (int q = 0; q < QB; ++q) {
                const int e = tid + q * NTH;
                if (BKC) Bs[(e / PK) * PB + e % PK] = rb[q];
                else Bs[(e / NL) * PB + e % NL] = rb[q];
            }
        }
        // the step to load now starts a block not known to be released: look again
        const int jn = j0 + issued / SPB;
        const bool look = issued < S && jn >= ready;
        if (look && warp == 0) {
            const int n = deps_count(jn, j1, lane, deps);
            if (lane == 0) poll_sh[s & 1] = jn + n;
        }
        __syncthreads();                  // step s is in shared memory, step s - 1 has been read
        if (look) ready = poll_sh[s & 1];
        const bool now = issued < S && jn < ready;
        const double *pa = As + tig * PA + wm * 32 + g;
        const double *pb = BKC ? Bs + (wn * 32 + g) * PB + tig : Bs + tig * PB + wn * 32 + g;
#pragma unroll
        for (int k4 = 0; k4 < PK; k4 += 4) {
            double a[4], b[4];
#pragma unroll
            for (int mi = 0; mi < 4; ++mi) a[mi] = pa[k4 * PA + 8 * mi];
#pragma unroll
            for (int ni = 0; ni < 4; ++ni) b[ni] = BKC ? pb[8 * ni * PB + k4] : pb[k4 * PB + 8 * ni];
            if (now) load_part(issued, k4 / 4);
#pragma unroll
            for (int mi = 0; mi < 4; ++mi)
#pragma unroll
                for (int ni = 0; ni < 4; ++ni) dmma884(blk[mi][ni], a[mi], b[ni]);
        }
        if (s % SPB == SPB - 1) {
#pragma unroll
            for (int mi = 0; mi < 4; ++mi)
#pragma unroll
                for (int ni = 0; ni < 4; ++ni)
#pragma unroll
                    for (int e = 0; e < 2; ++e) {
                        acc[mi][ni][e] += blk[mi][ni][e];
                        blk[mi][ni][e] = 0.0;
                    }
        }
        if (now) ++issued;
        if (s + 1 < S && issued == s + 1) {
            if (tid == 0) wait_sh = deps_wait(deps(jn), P);
            __syncthreads();
            if (!wait_sh) return false;
            ready = jn + 1;
            load(issued++);
        }
    }
    return true;
}

// One bulk task; false if a wait gave up or the run was aborted.
// Not inlined, as the chain, so that each has the registers to itself.
template <bool V16>
__device__ __noinline__ bool run_bulk(double *sm, const PItem it, const PotrfParams &P) {
    __shared__ int d_sh;
    const PFlags F(P);
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int g = lane >> 2, tig = lane & 3;
    const int n = P.n, lda = P.lda, nb = P.nblk, i = it.i, k = it.k;
    auto Aij = [&](int r, int c) { return P.A + (size_t)r * TB + (size_t)c * TB * lda; };
    double acc[4][4][2];
    const bool lt = it.type == IT_LT;
    const int WMN = lt ? 4 : 2;               // warps down the tile
    const int wm = warp % WMN, wn = warp / WMN;
    auto row_of = [&](int mi) { return wm * 32 + 8 * mi + g; };
    auto col_of = [&](int ni, int e) { return wn * 32 + 8 * ni + 2 * tig + e; };
    if (it.type == IT_XT) {
        const int c0 = 2 * k;                 // first block column of the pair
#pragma unroll
        for (int mi = 0; mi < 4; ++mi)
#pragma unroll
            for (int ni = 0; ni < 4; ++ni) acc[mi][ni][0] = acc[mi][ni][1] = 0.0;
        const int mrows = bsz(i, n), ncols = min(2 * TB, i * TB - c0 * TB);   // columns left of the diagonal block
        auto deps = [&](int j) {
            return JDeps{F.p(i, j), j == c0 ? F.ddone + j : F.x(j, k), j <= c0 + 1 ? F.ddone + j : F.p(i, j)};
        };
        if (!acc_blocks<TB, 2 * TB, true, V16>(sm, acc, P, Aij(i, 0), lda, mrows, P.X + (size_t)c0 * TB * P.ldx, P.ldx, ncols,
                                          c0, i, deps))
            return false;
        // X = -D_i acc
        double *Ds = sm, *Ss = sm + TB * (TB + 4);
        if (tid == 0) d_sh = wait_ge(F.ddone + i, 1, P);
        __syncthreads();
        if (!d_sh) return false;
        const double *D = P.X + (size_t)i * TB + (size_t)i * TB * P.ldx;
#pragma unroll
        for (int q = 0; q < TB * TB / NTH; ++q) {
            const int e = tid + q * NTH, x = e % TB, kk = e / TB;
            Ds[kk * (TB + 4) + x] = x < mrows && kk < mrows ? __ldcg(D + x + (size_t)kk * P.ldx) : 0.0;
        }
#pragma unroll
        for (int mi = 0; mi < 4; ++mi)
#pragma unroll
            for (int ni = 0; ni < 4; ++ni)
#pragma unroll
                for (int e = 0; e < 2; ++e) {
                    Ss[col_of(ni, e) * (TB + 4) + row_of(mi)] = -acc[mi][ni][e];
                    acc[mi][ni][e] = 0.0;
                }
        __syncthreads();
        const int ke = wm * 32 + 32;          // D_i is lower triangular
        for (int k4 = 0; k4 < ke; k4 += 4) {
            double a[4], b[4];
#pragma unroll
            for (int mi = 0; mi < 4; ++mi) a[mi] = Ds[(k4 + tig) * (TB + 4) + row_of(mi)];
#pragma unroll
            for (int ni = 0; ni < 4; ++ni) b[ni] = Ss[(wn * 32 + 8 * ni + g) * (TB + 4) + k4 + tig];
#pragma unroll
            for (int mi = 0; mi < 4; ++mi)
#pragma unroll
                for (int ni = 0; ni < 4; ++ni) dmma884(acc[mi][ni], a[mi], b[ni]);
        }
        double *O = P.X + (size_t)i * TB + (size_t)c0 * TB * P.ldx;
#pragma unroll
        for (int mi = 0; mi < 4; ++mi)
#pragma unroll
            for (int ni = 0; ni < 4; ++ni)
#pragma unroll
                for (int e = 0; e < 2; ++e)
                    if (row_of(mi) < mrows && col_of(ni, e) < ncols)
                        O[row_of(mi) + (size_t)col_of(ni, e) * P.ldx] = acc[mi][ni][e];
        __syncthreads();
        if (tid == 0) {
            __threadfence();
            atomicExch(F.x(i, k), 1);
        }
        return true;
    }
    // rows of the tile: blocks i, i + 1 (LT) or block k + 1 (PRE); columns: block k (LT) or k, k + 1 (PRE)
    const int r0 = lt ? i : k + 1;
    const int mrows = min(lt ? 2 * TB : TB, n - r0 * TB), ncols = lt ? TB : min(2 * TB, n - k * TB);
    double *C = Aij(r0, k);
#pragma unroll
    for (int mi = 0; mi < 4; ++mi)
#pragma unroll
        for (int ni = 0; ni < 4; ++ni)
#pragma unroll
            for (int e = 0; e < 2; ++e)
                acc[mi][ni][e] = row_of(mi) < mrows && col_of(ni, e) < ncols
                                     ? -__ldcg(C + row_of(mi) + (size_t)col_of(ni, e) * lda) : 0.0;   // acc = sum - C
    if (!lt) {
        auto deps = [&](int j) { return JDeps{F.p(k + 1, j), F.p(k, j), F.p(k, j)}; };
        if (!acc_blocks<TB, 2 * TB, false, V16>(sm, acc, P, Aij(k + 1, 0), lda, mrows, Aij(k, 0), lda, ncols, 0, k, deps))
            return false;
#pragma unroll
        for (int mi = 0; mi < 4; ++mi)
#pragma unroll
            for (int ni = 0; ni < 4; ++ni)
#pragma unroll
                for (int e = 0; e < 2; ++e)
                    if (row_of(mi) < mrows && col_of(ni, e) < ncols)
                        C[row_of(mi) + (size_t)col_of(ni, e) * lda] = -acc[mi][ni][e];
        __syncthreads();
        if (tid == 0) {
            __threadfence();
            atomicExch(F.vpre + k, 1);
        }
        return true;
    }
    const bool two = i + 1 < nb;
    auto deps = [&](int j) { return JDeps{F.p(i, j), F.p(two ? i + 1 : i, j), F.p(k, j)}; };
    if (!acc_blocks<2 * TB, TB, false, V16>(sm, acc, P, Aij(i, 0), lda, mrows, Aij(k, 0), lda, TB, 0, k, deps)) return false;
    // L = -acc D_k^T
    double *Ss = sm, *Ds = sm + TB * (2 * TB + 4);
    if (tid == 0) d_sh = wait_ge(F.ddone + k, 1, P);
    __syncthreads();
    if (!d_sh) return false;
    const double *D = P.X ? P.X + (size_t)k * TB + (size_t)k * TB * P.ldx : P.D + (size_t)k * TB * TB;
    const int ldd = P.X ? P.ldx : TB;
#pragma unroll
    for (int q = 0; q < TB * TB / NTH; ++q) {
        const int e = tid + q * NTH, x = e % TB, kk = e / TB;
        Ds[kk * (TB + 4) + x] = __ldcg(D + x + (size_t)kk * ldd);
    }
#pragma unroll
    for (int mi = 0; mi < 4; ++mi)
#pragma unroll
        for (int ni = 0; ni < 4; ++ni)
#pragma unroll
            for (int e = 0; e < 2; ++e) {
                Ss[col_of(ni, e) * (2 * TB + 4) + row_of(mi)] = -acc[mi][ni][e];
                acc[mi][ni][e] = 0.0;
            }
    __syncthreads();
    const int ke = wn * 32 + 32;              // D_k^T is upper triangular
    for (int k4 = 0; k4 < ke; k4 += 4) {
        double a[4], b[4];
#pragma unroll
        for (int mi = 0; mi < 4; ++mi) a[mi] = Ss[(k4 + tig) * (2 * TB + 4) + row_of(mi)];
#pragma unroll
        for (int ni = 0; ni < 4; ++ni) b[ni] = Ds[(k4 + tig) * (TB + 4) + wn * 32 + 8 * ni + g];
#pragma unroll
        for (int mi = 0; mi < 4; ++mi)
#pragma unroll
            for (int ni = 0; ni < 4; ++ni) dmma884(acc[mi][ni], a[mi], b[ni]);
    }
#pragma unroll
    for (int mi = 0; mi < 4; ++mi)
#pragma unroll
        for (int ni = 0; ni < 4; ++ni)
#pragma unroll
            for (int e = 0; e < 2; ++e)
                if (row_of(mi) < mrows) C[row_of(mi) + (size_t)col_of(ni, e) * lda] = acc[mi][ni][e];
    __syncthreads();
    if (tid == 0) {
        __threadfence();
        atomicExch(F.p(i, k), 1);
        if (two) atomicExch(F.p(i + 1, k), 1);
    }
    return true;
}

// ------------------------------------------------------------ the chain ----
// The chain CTA keeps three 64 x 64 column-major blocks in shared memory
// (pitch CP): S (the diagonal block being factored), Xs (its inverse) and Pn
// (the panel block below it, and scratch of the inverse).  Blocks smaller
// than 64 are padded: with the identity on the diagonal of S, with zeros in
// Pn, so the padded parts factor to the identity and never reach the tile.
constexpr int CHAIN_SMEM_DOUBLES = 3 * TB * CP;
constexpr int SMEM_DOUBLES = 2 * (pk<true>() * (TB + 4) + 2 * TB * (pk<true>() + 4));   // two stages of an XT task
static_assert(SMEM_DOUBLES >= CHAIN_SMEM_DOUBLES, "the chain's blocks");
static_assert(SMEM_DOUBLES >= 2 * pk<true>() * (2 * TB + 4 + TB + 4), "two stages of an LT or PRE task");
static_assert(SMEM_DOUBLES >= TB * (2 * TB + 4) + TB * (TB + 4), "S and D of an LT task");
static_assert(SMEM_DOUBLES >= TB * (TB + 4) + 2 * TB * (TB + 4), "D and S of an XT task");

// M(r, c) = G(r, c) for r < rows, c < cols, else (r == c && pad_id); all of a
// thread's loads are issued before its shared stores.
__device__ __forceinline__ void load_frame(double *M, const double *G, int ld, int rows, int cols, bool pad_id) {
    const int tid = threadIdx.x;
    double v[(TB * TB) / NTH];
#pragma unroll
    for (int q = 0; q < (TB * TB) / NTH; ++q) {
        const int e = tid + q * NTH, r = e & (TB - 1), c = e >> 6;
        v[q] = (r < rows && c < cols) ? __ldcg(G + r + (size_t)c * ld) : ((pad_id && r == c) ? 1.0 : 0.0);
    }
#pragma unroll
    for (int q = 0; q < (TB * TB) / NTH; ++q) {
        const int e = tid + q * NTH;
        M[(e >> 6) * CP + (e & (TB - 1))] = v[q];
    }
}

// The 8-column panel p0..p0+7 of S on warps 0-2.  Every lane of the three
// warps factors the panel's 8 x 8 diagonal block itself, its lower part in
// registers, so the pivot chain has no shuffles (rsqrt(d) scales the column;
// the pivot is d * rsqrt(d), and the diagonal register keeps the reciprocal).
// The three warps meet once all of them have read the block; then lane 0 of
// warp 0 stores the factored block, warps 0 and 1 solve the rows below it (row p0+8+lane, row p0+40+lane), and lanes
// 0-7 of warp 2 write column `lane` of the block's inverse into Xs by forward
// substitution.  Returns the panel column of a non-positive pivot, or -1.
__device__ int chain_panel(double *S, double *Xs, int p0, int warp, int lane) {
    double d[8][8];   // d[r][c], c <= r
#pragma unroll
    for (int r = 0; r < 8; ++r)
#pragma unroll
        for (int c = 0; c <= r; ++c) d[r][c] = S[(p0 + c) * CP + p0 + r];
    asm volatile("bar.sync 1, 96;" ::: "memory");   // warps 0-2: the block is read before it is rewritten
    const bool store = warp == 0 && lane == 0;
#pragma unroll
    for (int c = 0; c < 8; ++c) {
        const double dc = d[c][c];
        if (!(dc > 0.0)) return c;          // the same on every lane
        const double inv = rsqrt(dc);
        d[c][c] = inv;
        if (store) S[(p0 + c) * CP + p0 + c] = dc * inv;
#pragma unroll
        for (int r = c + 1; r < 8; ++r) d[r][c] *= inv;
#pragma unroll
        for (int cc = c + 1; cc < 8; ++cc)
#pragma unroll
            for (int r = cc; r < 8; ++r) d[r][cc] = fma(-d[r][c], d[cc][c], d[r][cc]);
    }
    if (store) {
#pragma unroll
        for (int c = 0; c < 8; ++c)
#pragma unroll
            for (int r = c + 1; r < 8; ++r) S[(p0 + c) * CP + p0 + r] = d[r][c];
    }
    if (warp < 2) {
        const int row = p0 + 8 + 32 * warp + lane;
        if (row < TB) {
            double a[8];
#pragma unroll
            for (int c = 0; c < 8; ++c) a[c] = S[(p0 + c) * CP + row];
#pragma unroll
            for (int c = 0; c < 8; ++c) {
                a[c] *= d[c][c];
#pragma unroll
                for (int cc = c + 1; cc < 8; ++cc) a[cc] = fma(-a[c], d[cc][c], a[cc]);
            }
#pragma unroll
            for (int c = 0; c < 8; ++c) S[(p0 + c) * CP + row] = a[c];
        }
    } else if (lane < 8) {
        const int c = lane;
        double x[8];
#pragma unroll
        for (int r = 0; r < 8; ++r) {
            double s = 0.0;
#pragma unroll
            for (int l = 0; l < r; ++l)
                if (l >= c) s = fma(d[r][l], x[l], s);
            x[r] = r < c ? 0.0 : (r == c ? d[r][r] : -s * d[r][r]);
        }
#pragma unroll
        for (int r = 0; r < 8; ++r) Xs[(p0 + c) * CP + p0 + r] = x[r];
    }
    return -1;
}

// Cholesky of S in place and its inverse in Xs (its blocks above the diagonal are
// zero on entry and stay so; Pn is scratch).  Blocked by
// 8-column panels (chain_panel, which also inverts the panel's diagonal
// block), then every warp applies the panel's rank-8 update to the lower 8 x 8
// tiles of the trailing block on the tensor cores.  The inverse's diagonal
// blocks are then merged in pairs as X21 = -X22 (L21 X11) at widths 8, 16, 32.
// Returns the column (0..63) of a non-positive pivot, or -1.
__device__ int chain_diag(double *S, double *Xs, double *Pn, const int *flag, int *seen) {
    __shared__ int bad_sh;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int g = lane >> 2, tig = lane & 3;
    for (int p0 = 0; p0 < TB; p0 += 8) {
        if (warp < 3) {
            const int b = chain_panel(S, Xs, p0, warp, lane);
            if (warp == 0 && lane == 0) bad_sh = b < 0 ? -1 : p0 + b;
        }
        __syncthreads();
        if (bad_sh >= 0) return bad_sh;
        // rank-8 update of the trailing lower 8 x 8 tiles: warp w takes tile row w,
        // its tiles independent of each other
        if (8 * warp >= p0 + 8) {
            const int m0 = 8 * warp;
            double u[7][2];
            const double a0 = -S[(p0 + tig) * CP + m0 + g], a1 = -S[(p0 + 4 + tig) * CP + m0 + g];
#pragma unroll
            for (int c = 0; c < 7; ++c) {
                const int n0 = p0 + 8 + 8 * c;
                if (n0 <= m0) {
                    u[c][0] = S[(n0 + 2 * tig) * CP + m0 + g];
                    u[c][1] = S[(n0 + 2 * tig + 1) * CP + m0 + g];
                    dmma884(u[c], a0, S[(p0 + tig) * CP + n0 + g]);
                    dmma884(u[c], a1, S[(p0 + 4 + tig) * CP + n0 + g]);
                }
            }
#pragma unroll
            for (int c = 0; c < 7; ++c) {
                const int n0 = p0 + 8 + 8 * c;
                if (n0 <= m0) {
                    S[(n0 + 2 * tig) * CP + m0 + g] = u[c][0];
                    S[(n0 + 2 * tig + 1) * CP + m0 + g] = u[c][1];
                }
            }
        }
        __syncthreads();
    }
    if (tid == NTH - 1) {
        const int v = ld_volatile(flag);
        if (v) __threadfence();
        *seen = v;
    }
    for (int h = 8; h < TB; h *= 2) {
        const int hb = h / 8, tpp = hb * hb, nt = (TB / (2 * h)) * tpp;
        // T = L21 X11 into the frame position of X21 in Pn (X11 lower: k >= the column block)
        for (int t = warp; t < nt; t += NTH / 32) {
            const int s0 = (t / tpp) * 2 * h, ti = (t % tpp) % hb, tj = (t % tpp) / hb;
            const int m0 = s0 + h + 8 * ti, n0 = s0 + 8 * tj;
            // two accumulators: the trip count is even, and the chains interleave
            double acc[2] = {0.0, 0.0}, acd[2] = {0.0, 0.0};
            for (int k = s0 + 8 * tj; k < s0 + h; k += 8) {
                dmma884(acc, S[(k + tig) * CP + m0 + g], Xs[(n0 + g) * CP + k + tig]);
                dmma884(acd, S[(k + 4 + tig) * CP + m0 + g], Xs[(n0 + g) * CP + k + 4 + tig]);
            }
            Pn[(n0 + 2 * tig) * CP + m0 + g] = acc[0] + acd[0];
            Pn[(n0 + 2 * tig + 1) * CP + m0 + g] = acc[1] + acd[1];
        }
        __syncthreads();
        // X21 = -X22 T (X22 lower: k up to the row block)
        for (int t = warp; t < nt; t += NTH / 32) {
            const int s0 = (t / tpp) * 2 * h, ti = (t % tpp) % hb, tj = (t % tpp) / hb;
            const int m0 = s0 + h + 8 * ti, n0 = s0 + 8 * tj;
            double acc[2] = {0.0, 0.0}, acd[2] = {0.0, 0.0};
            for (int k = s0 + h; k < m0 + 8; k += 8) {
                dmma884(acc, -Xs[(k + tig) * CP + m0 + g], Pn[(n0 + g) * CP + k + tig]);
                dmma884(acd, -Xs[(k + 4 + tig) * CP + m0 + g], Pn[(n0 + g) * CP + k + 4 + tig]);
            }
            Xs[(n0 + 2 * tig) * CP + m0 + g] = acc[0] + acd[0];
            Xs[(n0 + 2 * tig + 1) * CP + m0 + g] = acc[1] + acd[1];
        }
        __syncthreads();
    }
    return -1;
}

// One warp's 32 x 16 tile (rows wm*32.., cols wn*16..) of C = alpha X Y^T
// over k in [0, kend), X and Y column-major in shared memory; acc holds C on
// entry (or zero).
__device__ __forceinline__ void chain_mm_nt(double (&acc)[4][2][2], const double *X, const double *Y, double alpha,
                                            int kend, int wm, int wn, int g, int tig) {
    for (int k = 0; k < kend; k += 4) {
        double a[4], b[2];
#pragma unroll
        for (int mi = 0; mi < 4; ++mi) a[mi] = alpha * X[(k + tig) * CP + wm * 32 + mi * 8 + g];
#pragma unroll
        for (int ni = 0; ni < 2; ++ni) b[ni] = Y[(k + tig) * CP + wn * 16 + ni * 8 + g];
#pragma unroll
        for (int mi = 0; mi < 4; ++mi)
#pragma unroll
            for (int ni = 0; ni < 2; ++ni) dmma884(acc[mi][ni], a[mi], b[ni]);
    }
}

// The critical path of the tile: for j = 0, 1, ...: factor the diagonal block
// held in S, write L_jj and D_j, release ddone(j); then L_j+1,j = A_j+1,j D_j^T
// (written, released as pdone(j+1, j)) and S = A_j+1,j+1 - L_j+1,j L_j+1,j^T,
// each after the block's updates from the earlier columns are in.  Returns
// false if a wait gave up or a pivot failed (the abort flag is then set).
__device__ __noinline__ bool run_chain(double *sm, const PotrfParams &P) {
    __shared__ int ok_c, pre_c;
    double *S = sm, *Xs = sm + TB * CP, *Pn = sm + 2 * TB * CP;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int g = lane >> 2, tig = lane & 3, wm = warp & 1, wn = warp >> 1;
    const int nb = P.nblk, n = P.n, lda = P.lda;
    const PFlags F(P);
    auto Ablk = [&](int r, int c) { return P.A + (size_t)r * TB + (size_t)c * TB * lda; };
    auto wait_all = [&](const int *p, int v) {
        if (tid == 0) ok_c = wait_ge(p, v, P);
        __syncthreads();
        return ok_c != 0;
    };
    load_frame(S, Ablk(0, 0), lda, bsz(0, n), bsz(0, n), true);
    for (int e = tid; e < TB * CP; e += NTH) Xs[e] = 0.0;
    __syncthreads();
    constexpr int FR = (TB * TB) / NTH;
    double fp[FR], fs[FR];                // the next panel and diagonal block, on their way
    for (int j = 0; j < nb; ++j) {
        const int jb = bsz(j, n);
        // an idle thread looks for S_j+1,{j,j+1} while the diagonal block is factored
        const int bad = chain_diag(S, Xs, Pn, F.vpre + j, &pre_c);
        if (bad >= 0) {
            if (tid == 0) {
                // a pivot of the padding is 1: bad < jb
                if (P.info) atomicCAS(P.info, 0, P.info_base + j * TB + bad + 1);
                atomicExch(P.cnt + 1, 1);
            }
            return false;
        }
        const int i = j + 1, ib = i < nb ? bsz(i, n) : 0;
        auto fetch = [&]() {
#pragma unroll
            for (int q = 0; q < FR; ++q) {
                const int e = tid + q * NTH, r = e & (TB - 1), c = e >> 6;
                fp[q] = r < ib ? __ldcg(Ablk(i, j) + r + (size_t)c * lda) : 0.0;
                fs[q] = r < ib && c < ib ? __ldcg(Ablk(i, i) + r + (size_t)c * lda) : (r == c ? 1.0 : 0.0);
            }
        };
        const bool early = i < nb && (j == 0 || pre_c);
        if (early) fetch();               // they cross the write-out of L_jj and D_j
        double *Dj = P.X ? P.X + (size_t)j * TB + (size_t)j * TB * P.ldx : P.D + (size_t)j * TB * TB;
        const int ldd = P.X ? P.ldx : TB;
        double *Ajj = Ablk(j, j);
#pragma unroll 4
        for (int q = 0; q < (TB * TB) / NTH; ++q) {
            const int e = tid + q * NTH, r = e & (TB - 1), c = e >> 6;
            if (r < jb && c < jb) {
                Ajj[r + (size_t)c * lda] = r >= c ? S[c * CP + r] : 0.0;
                Dj[r + (size_t)c * ldd] = r >= c ? Xs[c * CP + r] : 0.0;
            }
        }
        __syncthreads();
        if (tid == 0) {
            __threadfence();
            atomicExch(F.ddone + j, 1);
        }
        if (i >= nb) break;
        // L_ij = A_ij D_j^T (D_j^T upper: k stops at the warp's last column)
        if (!early) {
            if (!wait_all(F.vpre + j, 1)) return false;
            fetch();
        }
#pragma unroll
        for (int q = 0; q < FR; ++q) {
            const int e = tid + q * NTH;
            Pn[(e >> 6) * CP + (e & (TB - 1))] = fp[q];
            S[(e >> 6) * CP + (e & (TB - 1))] = fs[q];
        }
        __syncthreads();
        double acc[4][2][2];
#pragma unroll
        for (int a = 0; a < 4; ++a)
#pragma unroll
            for (int b = 0; b < 2; ++b) acc[a][b][0] = acc[a][b][1] = 0.0;
        chain_mm_nt(acc, Pn, Xs, 1.0, wn * 16 + 16, wm, wn, g, tig);
        __syncthreads();
        double *Aij = Ablk(i, j);
#pragma unroll
        for (int mi = 0; mi < 4; ++mi) {
            const int row = wm * 32 + mi * 8 + g;
#pragma unroll
            for (int ni = 0; ni < 2; ++ni)
#pragma unroll
                for (int e = 0; e < 2; ++e) {
                    const int col = wn * 16 + ni * 8 + 2 * tig + e;
                    Pn[col * CP + row] = acc[mi][ni][e];
                    if (row < ib) Aij[row + (size_t)col * lda] = acc[mi][ni][e];
                }
        }
        __syncthreads();
        // (a thread of a warp that is idle in the update below)
        if (tid == 4 * 32) {
            __threadfence();
            atomicExch(F.p(i, j), 1);
        }
        // S = S_ii - L_ij L_ij^T (lower tiles; the warps above the diagonal skip)
        if (wm * 32 + 31 >= wn * 16) {
#pragma unroll
            for (int mi = 0; mi < 4; ++mi)
#pragma unroll
                for (int ni = 0; ni < 2; ++ni)
#pragma unroll
                    for (int e = 0; e < 2; ++e)
                        acc[mi][ni][e] = S[(wn * 16 + ni * 8 + 2 * tig + e) * CP + wm * 32 + mi * 8 + g];
            chain_mm_nt(acc, Pn, Pn, -1.0, TB, wm, wn, g, tig);
#pragma unroll
            for (int mi = 0; mi < 4; ++mi)
#pragma unroll
                for (int ni = 0; ni < 2; ++ni)
#pragma unroll
                    for (int e = 0; e < 2; ++e)
                        S[(wn * 16 + ni * 8 + 2 * tig + e) * CP + wm * 32 + mi * 8 + g] = acc[mi][ni][e];
        }
        __syncthreads();
    }
    return true;
}

__global__ void __launch_bounds__(NTH, 1) k_potrf_tile(PotrfParams P) {
    extern __shared__ double sm[];
    __shared__ int item_sh;
    const int tid = threadIdx.x;
    for (;;) {
        if (tid == 0) {
            int t = -1;
            if (!ld_volatile(P.cnt + 1)) {
                t = atomicAdd(P.cnt, 1);
                if (t >= P.nitems) t = -1;
            }
            item_sh = t;
        }
        __syncthreads();
        const int t = item_sh;
        if (t < 0) break;
        const PItem it = P.items[t];
        if (!(it.type == IT_CHAIN ? run_chain(sm, P) : P.v16 ? run_bulk<true>(sm, it, P) : run_bulk<false>(sm, it, P)))
            break;
        __syncthreads();
    }
}

// The bulk tasks column by column: PRE(k), which the chain's step k waits on,
// LT(i,k), then the inverse's row k - XLAG, which the factorization does not wait
// on (a row of it is as much work as a column of L, so it may lag behind).
std::vector<PItem> build_items(int nblk, bool inv) {
    std::vector<PItem> v;
    auto add = [&](int t, int i, int k) { v.push_back(PItem{(unsigned short)t, (unsigned short)i, (unsigned short)k, 0}); };
    add(IT_CHAIN, 0, 0);
    for (int k = 0; k < nblk + XLAG; ++k) {
        if (k < nblk) {
            if (k > 0 && k + 1 < nblk) add(IT_PRE, 0, k);
            for (int i = k + 2; i < nblk; i += 2) add(IT_LT, i, k);
        }
        const int r = k - XLAG;
        if (inv && r >= 0)
            for (int p = 0; 2 * p < r; ++p) add(IT_XT, r, p);
    }
    return v;
}

struct ItemList {
    PItem *d = nullptr;
    int n = 0;
};
std::mutex g_items_mu;
std::map<std::pair<int, long long>, ItemList> g_items;   // (device, nblk*2 + inv)

const ItemList *get_items(int nblk, bool inv, cudaStream_t st) {
    int dev = 0;
    cudaGetDevice(&dev);
    std::lock_guard<std::mutex> lk(g_items_mu);
    auto key = std::make_pair(dev, (long long)nblk * 2 + (inv ? 1 : 0));
    auto f = g_items.find(key);
    if (f != g_items.end()) return &f->second;
    std::vector<PItem> h = build_items(nblk, inv);
    ItemList L;
    if (device_malloc((void **)&L.d, h.size() * sizeof(PItem))) return nullptr;
    // ordered on the launch stream and complete before the list is used (a
    // legacy-stream copy from pageable memory may land after the kernel reads it)
    if (cudaMemcpyAsync(L.d, h.data(), h.size() * sizeof(PItem), cudaMemcpyHostToDevice, st) != cudaSuccess ||
        cudaStreamSynchronize(st) != cudaSuccess) {
        cudaFree(L.d);
        return nullptr;
    }
    L.n = (int)h.size();
    return &(g_items[key] = L);
}

// Exercise of the bounded wait above, for tests: thread 0 of CTA b waits
// with wait_ge on the counter cnt[2 + b], which nothing sets, with limit
// limit0 (CTA 0) or limit1 (the others).  The first wait to run out sets the
// timeout and abort flags; the others then leave at their next poll.
__global__ void k_wait_probe(PotrfParams P, long long limit0, long long limit1) {
    if (threadIdx.x != 0) return;
    P.spin_limit = blockIdx.x == 0 ? limit0 : limit1;
    wait_ge(P.cnt + 2 + blockIdx.x, 1, P);
}

}  // namespace

int potrf_tile_max_n() { return 128 * TB; }

size_t potrf_tile_scratch_ints(int n) {
    const size_t nb = (size_t)(n + TB - 1) / TB;
    return 8 + 2 * nb * nb + 2 * nb;
}

// The caller provides cnt (potrf_tile_scratch_ints(n) ints, any content) and,
// when X is null, D (nblk * 64 * 64 doubles); X, when given, must be zeroed.
int launch_potrf_tile(double *A, int lda, int n, double *X, int ldx, double *D, int *cnt, int *info,
                      int info_base, int *timeout, int grid, cudaStream_t st) {
    const int nblk = (n + TB - 1) / TB;
    const ItemList *L = get_items(nblk, X != nullptr, st);
    if (!L) return -1;
    if (cudaMemsetAsync(cnt, 0, potrf_tile_scratch_ints(n) * sizeof(int), st) != cudaSuccess) return -1;
    const int smem = (int)sizeof(double) * SMEM_DOUBLES;
    // per device and thread-safe: set on every launch (a host-side call, no synchronisation)
    cudaFuncSetAttribute(k_potrf_tile, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
    const int v16 = (((size_t)A | (size_t)X) & 15) == 0 && ((lda | (X ? ldx : 0)) & 1) == 0;
    PotrfParams P{A, lda, n, nblk, X, ldx, D, L->d, L->n, cnt, info, info_base, timeout, v16, SPIN_LIMIT};
    // the chain waits on bulk tasks of earlier block columns, which only the
    // other CTAs take: with any bulk task in the list the launch has two CTAs
    // or more (they need not be resident at the same time)
    if (grid > L->n) grid = L->n;
    if (grid < 2) grid = L->n > 1 ? 2 : 1;
    k_potrf_tile<<<grid, NTH, smem, st>>>(P);
    return cudaGetLastError() == cudaSuccess ? 0 : -1;
}

// cnt: 2 + nblocks zeroed ints (abort flag at [1]); timeout: one zeroed int.
int launch_wait_probe(int *cnt, int *timeout, int nblocks, long long limit0, long long limit1, cudaStream_t st) {
    if (nblocks < 1 || nblocks > 64 || limit0 < 1 || limit1 < 1) return -1;
    PotrfParams P{};
    P.cnt = cnt;
    P.timeout = timeout;
    k_wait_probe<<<nblocks, 32, 0, st>>>(P, limit0, limit1);
    return cudaGetLastError() == cudaSuccess ? 0 : -1;
}

}  // namespace tlr
