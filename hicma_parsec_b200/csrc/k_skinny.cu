// Products with few columns, C = alpha op(A) B + beta C (n = right-hand sides),
// of the triangular solves, FP64.
//
// The solves with a factor read every tile of it once per sweep and do little
// arithmetic on it, in a chain of NT steps, so what counts is how many bytes are
// in flight and how short a step is.  One CTA per 32 x 8 (or 32 x 32) block of
// C; its warps split the inner dimension in groups of 16 and read op(A) and B
// straight into DMMA fragments (mma.sync m8n8k4 f64, four quads of loads in
// flight per lane), then add their partials in warp order (deterministic).  A
// triangular A is read only where it has entries.  Two warps a CTA for inner
// dimensions up to 64 (the rank-wide factors); above, eight with 8 columns of C and
// four with 32.
// The batched GEMM used before walked a tile column's 2700-long inner dimension
// in one CTA (about 170 us a step).  Device time of a log-likelihood with the 36 x
// 36-tile factor of tile 2700: 41 -> 5 ms; a solve call of the 30 x 30-tile factor
// of tile 1350 with 1, 64 and 512 right-hand sides: 19 -> 2.4, 23 -> 12, 84 -> 71 ms,
// so every number of right-hand sides takes it.
#include "tlr_internal.h"

namespace tlr {
namespace {

__device__ __forceinline__ void dmma884(double (&d)[2], double a, double b) {
    asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0,%1}, {%2}, {%3}, {%0,%1};\n"
                 : "+d"(d[0]), "+d"(d[1])
                 : "d"(a), "d"(b));
}

template <int N8, int NW>
__global__ void __launch_bounds__(32 * NW) k_skinny(const SkinnyTask *__restrict__ tasks) {
    constexpr int BN = 8 * N8, U = 4;
    __shared__ double red[NW][32 * BN];
    const SkinnyTask t = tasks[blockIdx.y];
    const int nbi = (t.m + 31) / 32, nbj = (t.n + BN - 1) / BN;
    if ((int)blockIdx.x >= nbi * nbj) return;
    const int i0 = (int)(blockIdx.x % nbi) * 32, j0 = (int)(blockIdx.x / nbi) * BN;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, g = lane >> 2, tig = lane & 3;
    // a lower triangular A: op N ends at the block's last row, op T starts at its first
    const int kb = t.tri == 2 ? i0 & ~15 : 0, ke = t.tri == 1 ? min(t.k, i0 + 32) : t.k;
    double acc[4][N8][2];
#pragma unroll
    for (int a = 0; a < 4; ++a)
#pragma unroll
        for (int b = 0; b < N8; ++b) acc[a][b][0] = acc[a][b][1] = 0.0;
    const size_t sk = t.opA ? 1 : (size_t)t.lda, si = t.opA ? (size_t)t.lda : 1;
    const double *pa = t.A + (size_t)(i0 + g) * si, *pb = t.B + (size_t)(j0 + g) * t.ldb;
    bool ri[4], rj[N8];
#pragma unroll
    for (int q = 0; q < 4; ++q) ri[q] = i0 + 8 * q + g < t.m;
#pragma unroll
    for (int q = 0; q < N8; ++q) rj[q] = j0 + 8 * q + g < t.n;
    for (int k0 = kb + 16 * warp; k0 < ke; k0 += 16 * NW) {
        double a[U][4], b[U][N8];
#pragma unroll
        for (int u = 0; u < U; ++u) {
            const int k = k0 + 4 * u + tig;
            const bool in = k < ke;
#pragma unroll
            for (int q = 0; q < 4; ++q) a[u][q] = in && ri[q] ? __ldg(pa + (size_t)k * sk + (size_t)(8 * q) * si) : 0.0;
#pragma unroll
            for (int q = 0; q < N8; ++q) b[u][q] = in && rj[q] ? pb[(size_t)k + (size_t)(8 * q) * t.ldb] : 0.0;
        }
#pragma unroll
        for (int u = 0; u < U; ++u)
#pragma unroll
            for (int mi = 0; mi < 4; ++mi)
#pragma unroll
                for (int ni = 0; ni < N8; ++ni) dmma884(acc[mi][ni], a[u][mi], b[u][ni]);
    }
    // partials column by column, so that the sums go down the columns of C
#pragma unroll
    for (int mi = 0; mi < 4; ++mi)
#pragma unroll
        for (int ni = 0; ni < N8; ++ni)
#pragma unroll
            for (int e = 0; e < 2; ++e) red[warp][(8 * ni + 2 * tig + e) * 32 + 8 * mi + g] = acc[mi][ni][e];
    __syncthreads();
    for (int idx = threadIdx.x; idx < 32 * BN; idx += 32 * NW) {
        const int i = i0 + (idx & 31), j = j0 + (idx >> 5);
        if (i >= t.m || j >= t.n) continue;
        double s = 0.0;
#pragma unroll
        for (int w = 0; w < NW; ++w) s += red[w][idx];
        double *c = t.C + (size_t)i + (size_t)j * t.ldc;
        s *= t.alpha;
        if (t.beta != 0.0) s += t.beta * *c;
        *c = s;
    }
}

template <int N8>
void launch_n8(const SkinnyTask *d, int ntasks, int mmax, int nmax, int kmax, cudaStream_t st) {
    const dim3 grid((unsigned)(((mmax + 31) / 32) * ((nmax + 8 * N8 - 1) / (8 * N8))), (unsigned)ntasks);
    if (kmax <= 64) k_skinny<N8, 2><<<grid, 64, 0, st>>>(d);
    else k_skinny<N8, N8 == 1 ? 8 : 4><<<grid, N8 == 1 ? 256 : 128, 0, st>>>(d);
}

}  // namespace

void launch_skinny_batched(const SkinnyTask *d_tasks, int ntasks, int mmax, int nmax, int kmax, cudaStream_t st) {
    if (ntasks <= 0 || mmax <= 0 || nmax <= 0) return;
    if (nmax <= 8) launch_n8<1>(d_tasks, ntasks, mmax, nmax, kmax, st);
    else launch_n8<4>(d_tasks, ntasks, mmax, nmax, kmax, st);
}

}  // namespace tlr
