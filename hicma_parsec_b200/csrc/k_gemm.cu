// Batched variable-size FP64 GEMM on the FP64 tensor cores (DMMA,
// mma.sync m8n8k4 f64) for sm_100a.  tcgen05 has no f64 kind, so FP64
// tensor-core work on Blackwell goes through DMMA.
//
// Replaces the CORE_dgemm / cblas_dgemm bodies of the reference task classes
// (hicma_parsec/HiCMA_dpotrf_L_2flow.jdf:704-708,717-728,745-778) and the
// products inside HCORE (low-rank SYRK/GEMM, QR/SVD recompression).
//
// CTA tile 64 x 64 x 16 (or 128 x 32 x 16 for outputs a rank wide), 4 warps
// (2 x 2 or 4 x 1, 32 x 32 each = 4 x 4 DMMA tiles).  Operands are staged in
// shared memory by cp.async in three stages with one barrier per 16-wide step,
// zero-filled at the edges: 16-byte copies where base and leading dimension
// allow, 8-byte ones otherwise.  An operand is stored along its contiguous
// dimension, [k][x] or [x][k], with a pitch == 4 mod 16 doubles, so that copies
// walk global memory and the DMMA fragment reads are free of bank conflicts in
// either form; the four op combinations are separate instances.  Bound by the
// DMMA rate (37 TFLOP/s) and by the last wave of CTAs.  Measured for C -= A op(B)
// on a B200, against two stages, two barriers, 8-byte copies and a pitch of 72
// (2-way conflicts): 2700^3 NT 22.8 -> 30.0, NN 20.8 -> 29.7, TN 17.4 -> 30.5
// TFLOP/s; 10800^3 27.5 -> 33.4, 23.6 -> 33.2, 20.1 -> 34.3; 1000^3 13 -> 23.
// Larger tiles (128 x 64, 128 x 128, 96 x 96) were slower at every size.
// A single product takes two stages and four CTAs an SM instead of three and three where
// waves of CTAs count more than the depth of the pipeline: k up to 128, or fewer waves
// and k up to 512, or one wave instead of two.  NT, three and four CTAs an SM: 24 x 24
// tiles, k = 16, 200, 1600 42, 75, 326 and 32, 61, 299 us; 32 x 32 tiles, k = 16, 400,
// 1600 54, 156, 453 and 43, 139, 458; 25 x 25 tiles (two waves either way), k = 16, 400
// 41, 106 and 40, 118.
// A batch is a list of tasks whose output tiles are flattened into one grid
// (prefix sums in tile_off).
#include "tlr_internal.h"

namespace tlr {
namespace {

constexpr int BM = 64, BN = 64, BK = 16, NT = 128;
constexpr int STAGES = 3;

__device__ __forceinline__ void dmma884(double (&d)[2], double a, double b) {
    asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0,%1}, {%2}, {%3}, {%0,%1};\n"
                 : "+d"(d[0]), "+d"(d[1])
                 : "d"(a), "d"(b));
}

__device__ __forceinline__ void cp_async8(unsigned smem, const double *gmem, bool pred) {
    const int sz = pred ? 8 : 0;
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;\n" ::"r"(smem), "l"(gmem), "r"(sz));
}
// bytes: 16, 8 or 0 read from gmem (16-byte aligned), the rest zero-filled
__device__ __forceinline__ void cp_async16(unsigned smem, const double *gmem, int bytes) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(smem), "l"(gmem), "r"(bytes));
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;\n" ::); }
template <int N>
__device__ __forceinline__ void cp_async_wait() {
    asm volatile("cp.async.wait_group %0;\n" ::"n"(N));
}

// Shared layout of an operand with BX outer rows: KC (contiguous along k in
// global memory) [x][BK + 4], else [k][BX + 4].
template <int BX, bool KC>
struct OpTile {
    static constexpr int P = KC ? BK + 4 : BX + 4;
    static constexpr int D = KC ? BX * P : BK * P;
};
template <int BX>
constexpr int op_doubles() { return OpTile<BX, true>::D > OpTile<BX, false>::D ? OpTile<BX, true>::D : OpTile<BX, false>::D; }
template <int BM_, int BN_, int ST = STAGES>
constexpr size_t gemm_smem() { return sizeof(double) * ST * (op_doubles<BM_>() + op_doubles<BN_>()); }

// Rows x0.. (below xe) and inner indices k0.. (below ke) of an operand into its stage.
template <int BX, bool KC, bool V16>
__device__ __forceinline__ void load_operand(double *sm, const double *X, int ld, int x0, int xe, int k0, int ke) {
    constexpr int P = OpTile<BX, KC>::P, INNER = KC ? BK : BX, W = V16 ? 2 : 1;
    const unsigned s0 = (unsigned)__cvta_generic_to_shared(sm);
    const int ei = KC ? ke : xe, eo = KC ? xe : ke;
#pragma unroll
    for (int q = 0; q < BX * BK / W / NT; ++q) {
        const int e = threadIdx.x + q * NT;
        const int in = (e % (INNER / W)) * W, ou = e / (INNER / W);
        const int gi = (KC ? k0 : x0) + in, go = (KC ? x0 : k0) + ou;
        const bool p = go < eo && gi < ei;
        const double *src = p ? X + (size_t)gi + (size_t)go * ld : X;
        const unsigned d = s0 + (unsigned)((ou * P + in) * sizeof(double));
        if (V16) cp_async16(d, src, p ? (gi + 1 < ei ? 16 : 8) : 0);
        else cp_async8(d, src, p);
    }
}

// One BM_ x BN_ output tile; four warps of 32 x 32 (2 x 2 for 64 x 64,
// 4 x 1 for the narrow 128 x 32 tile used when n is a rank).  AK / BKC: op(A) /
// op(B) is contiguous along the inner dimension (opA = 1, opB = 0).
template <int BM_, int BN_, int ST, bool AK, bool BKC, bool V16>
__device__ __forceinline__ void gemm_tile_op(double *sm, const GemmTask &t, int n, int i0, int j0) {
    using OA = OpTile<BM_, AK>;
    using OB = OpTile<BN_, BKC>;
    constexpr int WM = BM_ / 32;
    constexpr int SI = AK ? OA::P : 1, SKA = AK ? 1 : OA::P, SJ = BKC ? OB::P : 1, SKB = BKC ? 1 : OB::P;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int g = lane >> 2, tig = lane & 3;
    const int wm = warp % WM, wn = warp / WM;

    double acc[4][4][2];
#pragma unroll
    for (int a = 0; a < 4; ++a)
#pragma unroll
        for (int b = 0; b < 4; ++b) acc[a][b][0] = acc[a][b][1] = 0.0;

    // a triangular operand leaves the rest of the inner dimension zero for this tile
    int kend = t.k;
    if (t.tri == 1) kend = min(kend, i0 + BM_);
    else if (t.tri == 2) kend = min(kend, j0 + BN_);
    const int ktiles = (kend + BK - 1) / BK;
    auto load = [&](int s, int kt) {
        double *sa = sm + s * (OA::D + OB::D);
        load_operand<BM_, AK, V16>(sa, t.A, t.lda, i0, t.m, kt * BK, t.k);
        load_operand<BN_, BKC, V16>(sa + OA::D, t.B, t.ldb, j0, n, kt * BK, t.k);
    };
#pragma unroll
    for (int s = 0; s < ST - 1; ++s) {
        if (s < ktiles) load(s, s);
        cp_async_commit();
    }
    int s = 0;
    for (int kt = 0; kt < ktiles; ++kt) {
        cp_async_wait<ST - 2>();
        __syncthreads();   // the stage is complete, and the one loaded next is no longer read
        if (kt + ST - 1 < ktiles) load(s == 0 ? ST - 1 : s - 1, kt + ST - 1);
        cp_async_commit();
        const double *sa = sm + s * (OA::D + OB::D), *sb = sa + OA::D;
        const double *pa = sa + (wm * 32 + g) * SI + tig * SKA, *pb = sb + (wn * 32 + g) * SJ + tig * SKB;
#pragma unroll
        for (int k4 = 0; k4 < BK; k4 += 4) {
            double a[4], b[4];
#pragma unroll
            for (int mi = 0; mi < 4; ++mi) a[mi] = pa[mi * 8 * SI + k4 * SKA];
#pragma unroll
            for (int ni = 0; ni < 4; ++ni) b[ni] = pb[ni * 8 * SJ + k4 * SKB];
#pragma unroll
            for (int mi = 0; mi < 4; ++mi)
#pragma unroll
                for (int ni = 0; ni < 4; ++ni) dmma884(acc[mi][ni], a[mi], b[ni]);
        }
        s = s + 1 == ST ? 0 : s + 1;
    }

    const double alpha = t.alpha, beta = t.beta;
#pragma unroll
    for (int mi = 0; mi < 4; ++mi) {
        const int row = i0 + wm * 32 + mi * 8 + g;
        if (row >= t.m) continue;
#pragma unroll
        for (int ni = 0; ni < 4; ++ni) {
#pragma unroll
            for (int e = 0; e < 2; ++e) {
                const int col = j0 + wn * 32 + ni * 8 + tig * 2 + e;
                if (col >= n) continue;
                double *c = t.C + (size_t)row + (size_t)col * t.ldc;
                double v = alpha * acc[mi][ni][e];
                if (beta != 0.0) v += beta * (*c);
                *c = v;
            }
        }
    }
}

template <int BM_, int BN_, int ST = STAGES>
__device__ __forceinline__ void gemm_tile(double *sm, const GemmTask &t, int tm, int tn) {
    const int i0 = tm * BM_, j0 = tn * BN_;
    if (t.lower && j0 >= i0 + BM_) return;
    int n = t.n;
    if (t.n_dev) n = min(n, *t.n_dev);
    if (j0 >= n) return;
    const bool v16 = (((size_t)t.A | (size_t)t.B) & 15) == 0 && ((t.lda | t.ldb) & 1) == 0;
    switch ((t.opA ? 4 : 0) | (t.opB ? 2 : 0) | (v16 ? 1 : 0)) {
        case 0: gemm_tile_op<BM_, BN_, ST, false, true, false>(sm, t, n, i0, j0); break;
        case 1: gemm_tile_op<BM_, BN_, ST, false, true, true>(sm, t, n, i0, j0); break;
        case 2: gemm_tile_op<BM_, BN_, ST, false, false, false>(sm, t, n, i0, j0); break;
        case 3: gemm_tile_op<BM_, BN_, ST, false, false, true>(sm, t, n, i0, j0); break;
        case 4: gemm_tile_op<BM_, BN_, ST, true, true, false>(sm, t, n, i0, j0); break;
        case 5: gemm_tile_op<BM_, BN_, ST, true, true, true>(sm, t, n, i0, j0); break;
        case 6: gemm_tile_op<BM_, BN_, ST, true, false, false>(sm, t, n, i0, j0); break;
        default: gemm_tile_op<BM_, BN_, ST, true, false, true>(sm, t, n, i0, j0); break;
    }
}

// Task of output tile `bid`: the group table (after the ntasks + 1 prefix
// sums) names the task of the group's first tile; step forward from there.
__device__ __forceinline__ int task_of(const int *__restrict__ tile_off, int ntasks, int bid) {
    int lo = tile_off[ntasks + 1 + bid / GEMM_GROUP];
    while (lo + 1 < ntasks && tile_off[lo + 1] <= bid) ++lo;
    return lo;
}

template <int BM_, int BN_>
__global__ void __launch_bounds__(NT, 3) k_gemm_batched(const GemmTask *__restrict__ tasks,
                                                     const int *__restrict__ tile_off, int ntasks) {
    extern __shared__ __align__(16) double sm[];
    const int bid = blockIdx.x;
    const int lo = task_of(tile_off, ntasks, bid);
    const GemmTask t = tasks[lo];
    const int local = bid - tile_off[lo];
    gemm_tile<BM_, BN_>(sm, t, local % t.tiles_m, local / t.tiles_m);
}

template <int ST, int CTAS>
__global__ void __launch_bounds__(NT, CTAS) k_gemm_single(GemmTask t) {
    extern __shared__ __align__(16) double sm[];
    gemm_tile<BM, BN, ST>(sm, t, blockIdx.x, blockIdx.y);
}

template <int ST, int CTAS>
void launch_single(const GemmTask &t, dim3 grid, cudaStream_t st) {
    constexpr size_t smem = gemm_smem<BM, BN, ST>();
    if constexpr (smem > 48 * 1024)   // the limit without it
        cudaFuncSetAttribute(k_gemm_single<ST, CTAS>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    k_gemm_single<ST, CTAS><<<grid, NT, smem, st>>>(t);
}

// ---------------------------------------------------------------------------
// FP32 product path of the mixed-precision policy: operands are read in FP64,
// rounded to FP32 in shared memory and multiplied with FP32 FMAs (FP32
// accumulation); the result is scaled and written back in FP64.
constexpr int FB = 64, FK = 16;
__global__ void __launch_bounds__(256) k_sgemm_batched(const GemmTask *__restrict__ tasks,
                                                       const int *__restrict__ tile_off, int ntasks) {
    __shared__ float As[FK][FB + 4];
    __shared__ float Bs[FK][FB + 4];
    const int bid = blockIdx.x;
    const int lo = task_of(tile_off, ntasks, bid);
    GemmTask t = tasks[lo];
    const int local = bid - tile_off[lo];
    const int i0 = (local % t.tiles_m) * FB, j0 = (local / t.tiles_m) * FB;
    if (t.lower && j0 >= i0 + FB) return;
    if (t.n_dev) {
        const int nd = *t.n_dev;
        t.n = nd < t.n ? nd : t.n;
    }
    if (j0 >= t.n) return;
    const int tid = threadIdx.x, tx = tid & 15, ty = tid >> 4;
    float acc[4][4] = {};
    int kend = t.k;
    if (t.tri == 1) kend = min(kend, i0 + FB);
    else if (t.tri == 2) kend = min(kend, j0 + FB);
    for (int k0 = 0; k0 < kend; k0 += FK) {
        for (int e = tid; e < FB * FK; e += 256) {
            int i, kk;
            if (t.opA == 0) { i = e & (FB - 1); kk = e / FB; } else { kk = e & (FK - 1); i = e / FK; }
            const int gi = i0 + i, gk = k0 + kk;
            float v = 0.f;
            if (gi < t.m && gk < t.k)
                v = (float)((t.opA == 0) ? t.A[(size_t)gi + (size_t)gk * t.lda] : t.A[(size_t)gk + (size_t)gi * t.lda]);
            As[kk][i] = v;
            int j;
            if (t.opB == 0) { kk = e & (FK - 1); j = e / FK; } else { j = e & (FB - 1); kk = e / FB; }
            const int gj = j0 + j, gk2 = k0 + kk;
            float w = 0.f;
            if (gj < t.n && gk2 < t.k)
                w = (float)((t.opB == 0) ? t.B[(size_t)gk2 + (size_t)gj * t.ldb] : t.B[(size_t)gj + (size_t)gk2 * t.ldb]);
            Bs[kk][j] = w;
        }
        __syncthreads();
#pragma unroll
        for (int kk = 0; kk < FK; ++kk) {
            float a[4], b[4];
#pragma unroll
            for (int q = 0; q < 4; ++q) { a[q] = As[kk][tx + 16 * q]; b[q] = Bs[kk][ty + 16 * q]; }
#pragma unroll
            for (int p = 0; p < 4; ++p)
#pragma unroll
                for (int q = 0; q < 4; ++q) acc[p][q] = fmaf(a[p], b[q], acc[p][q]);
        }
        __syncthreads();
    }
#pragma unroll
    for (int p = 0; p < 4; ++p) {
        const int row = i0 + tx + 16 * p;
        if (row >= t.m) continue;
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            const int col = j0 + ty + 16 * q;
            if (col >= t.n) continue;
            double *c = t.C + (size_t)row + (size_t)col * t.ldc;
            double v = t.alpha * (double)acc[p][q];
            if (t.beta != 0.0) v += t.beta * (*c);
            *c = v;
        }
    }
}

__global__ void k_gemm_devcount(const GemmTask *__restrict__ tasks, int ntasks, double *acc) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= ntasks) return;
    const GemmTask t = tasks[i];
    if (!t.n_dev) return;
    const int nd = *t.n_dev;
    const double n = nd < t.n ? nd : t.n;
    if (n <= 0) return;
    atomicAdd(acc, 2.0 * t.m * n * t.k);
    atomicAdd(acc + 1, 8.0 * ((double)t.m * t.k + (double)t.k * n + (t.beta != 0.0 ? 2.0 : 1.0) * t.m * n));
}

}  // namespace

void launch_gemm_devcount(const GemmTask *d_tasks, int ntasks, double *acc, cudaStream_t st) {
    if (ntasks <= 0) return;
    k_gemm_devcount<<<(ntasks + 255) / 256, 256, 0, st>>>(d_tasks, ntasks, acc);
}

void launch_gemm_batched(const GemmTask *d_tasks, const int *d_tile_off, int ntasks, int total_tiles,
                         cudaStream_t st, bool fp32) {
    if (ntasks <= 0 || total_tiles <= 0) return;
    if (fp32)
        k_sgemm_batched<<<total_tiles, 256, 0, st>>>(d_tasks, d_tile_off, ntasks);
    else {
        // per device and thread-safe: set on every launch (a host-side call, no synchronisation)
        cudaFuncSetAttribute(k_gemm_batched<BM, BN>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)gemm_smem<BM, BN>());
        k_gemm_batched<BM, BN><<<total_tiles, NT, gemm_smem<BM, BN>(), st>>>(d_tasks, d_tile_off, ntasks);
    }
}

void launch_gemm_batched_narrow(const GemmTask *d_tasks, const int *d_tile_off, int ntasks, int total_tiles,
                                cudaStream_t st) {
    if (ntasks <= 0 || total_tiles <= 0) return;
    constexpr size_t smem = gemm_smem<GEMM_NARROW_M, GEMM_NARROW_N>();
    cudaFuncSetAttribute(k_gemm_batched<GEMM_NARROW_M, GEMM_NARROW_N>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    k_gemm_batched<GEMM_NARROW_M, GEMM_NARROW_N><<<total_tiles, NT, smem, st>>>(d_tasks, d_tile_off, ntasks);
}

void launch_gemm_single(const GemmTask &t, cudaStream_t st) {
    if (t.m <= 0 || t.n <= 0) return;
    dim3 grid((t.m + BM - 1) / BM, (t.n + BN - 1) / BN);
    if (t.k <= 128) return launch_single<2, 4>(t, grid, st);
    int dev = 0, nsm = 148;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev);
    const long long tiles = (long long)grid.x * grid.y;
    const long long waves3 = (tiles + 3 * nsm - 1) / (3 * nsm), waves4 = (tiles + 4 * nsm - 1) / (4 * nsm);
    if (waves4 < waves3 && (t.k <= 512 || waves4 == 1)) launch_single<2, 4>(t, grid, st);
    else launch_single<STAGES, 3>(t, grid, st);
}

}  // namespace tlr
