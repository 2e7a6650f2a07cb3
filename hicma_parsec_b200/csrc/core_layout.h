// Memory of the wide core SVD (k_core_wide): which part of it lies where in a CTA's
// dynamic shared memory and in the task's scratch.  Host code only needs a C++
// compiler, so that the arithmetic can be checked for every width.
#pragma once
#include <cstddef>

#ifdef __CUDACC__
#define TLR_HD __host__ __device__ __forceinline__
#else
#define TLR_HD inline
#endif

namespace tlr {

constexpr int WB = 16;                        // columns of a block
constexpr int WP = 2 * WB;                    // columns of a pair problem
constexpr int WLD = WP + 4;                   // pitch of its J (conflict-free DMMA fragments)
constexpr int WGD = WP + 1;                   // pitch of its G (rows and columns read alike)
constexpr int W_CT = 256;
constexpr int W_NW = W_CT / 32;
constexpr int W_TILES = 10;                   // lower 8 x 8 tiles of the 32 x 32 Gram matrix
constexpr int W_CSMAX = 16;
constexpr size_t W_JACOBI_DOUBLES = 2 * WP * WLD + W_NW * W_TILES * 64;
constexpr size_t W_SMEM_MAX = 220 * 1024;
enum { W_T_SHARED = 1, W_HV_SHARED = 2 };     // what of the pivoted QR is in shared memory

// columns of T a CTA holds
TLR_HD int wide_ncl(int K, int cs) { return (K + cs - 1) / cs; }

// Offsets in doubles.  Shared memory: sigl (ncl: squared norms of the CTA's columns),
// then, as `place` says, hv (K: the pivot column) and T (ncl x K).  Scratch of the task:
// X (K x (K + WP)), sig (K), T if it is here (K x (K + W_CSMAX), its columns by CTA), the
// rotation flags (64).  Without W_HV_SHARED, hv lies in X's columns past K, which are free until
// the QR is over.  The sorted values (K doubles and K ints) come last: over the CTA's T
// in shared memory, or over T in the scratch.
struct WideLayout {
    size_t sigl, hv, T, sort;                 // in shared memory, or in the scratch as `place` says
    size_t X, sig, flags;                     // in the scratch
};
TLR_HD WideLayout wide_layout(int K, int cs, int rank, int place) {
    const size_t k = (size_t)K, ncl = (size_t)wide_ncl(K, cs), r = (size_t)rank;
    WideLayout w;
    w.X = 0;
    w.sig = k * (k + WP);
    const size_t Tg = w.sig + k;
    w.flags = place & W_T_SHARED ? Tg : Tg + k * (k + W_CSMAX);
    w.sigl = 0;
    w.hv = place & W_HV_SHARED ? ncl : k * k + r * k;
    w.T = place & W_T_SHARED ? ncl + k + ((ncl + k) & 1) : Tg + r * ncl * k;
    w.sort = place & W_T_SHARED ? 0 : Tg + r * 2 * k;
    return w;
}

// Shared memory of a launch whose widest core has K columns (bytes): the pivoted QR's
// part, the Jacobi rounds' or the sorted values'.
TLR_HD size_t wide_smem(int K, int cs, int place) {
    const size_t k = (size_t)K, ncl = (size_t)wide_ncl(K, cs);
    const size_t qr = ncl + (place & W_HV_SHARED ? k + 1 : 0) + (place & W_T_SHARED ? ncl * k : 0);
    const size_t sort = place & W_T_SHARED ? k + (k + 1) / 2 : 0;
    size_t d = qr > sort ? qr : sort;
    if (d < W_JACOBI_DOUBLES) d = W_JACOBI_DOUBLES;
    return sizeof(double) * d;
}

// What fits `limit` bytes: T and the pivot column (K up to about 650), the pivot column
// alone (26,500), neither.
TLR_HD int wide_place(int K, int cs, size_t limit) {
    if (wide_smem(K, cs, W_T_SHARED | W_HV_SHARED) <= limit) return W_T_SHARED | W_HV_SHARED;
    return wide_smem(K, cs, W_HV_SHARED) <= limit ? W_HV_SHARED : 0;
}

// CTAs of a cluster: about one per pair problem of the Jacobi rounds (k / 32
// pairs, k about K / 2) and enough shared memory for T: 4 up to K = 160, 8 up
// to 448, then 16 (the non-portable maximum).
TLR_HD int wide_cluster(int K) { return K <= 160 ? 4 : K <= 448 ? 8 : W_CSMAX; }

// Launches hold cores of one of the widths up to 160, up to 448 and above.
constexpr int W_EDGE1 = 160, W_EDGE2 = 448;

// Scratch of a core (doubles) under a shared memory limit: without T where every launch
// that the core can be part of has it in shared memory.
TLR_HD size_t wide_work_doubles(int K, size_t limit) {
    const size_t k = (size_t)K;
    const int edge = K <= W_EDGE1 ? W_EDGE1 : W_EDGE2;
    const bool t_shared = K <= W_EDGE2 && (wide_place(edge, wide_cluster(edge), limit) & W_T_SHARED);
    return k * (k + WP) + k + 64 + (t_shared ? 0 : k * (k + W_CSMAX));
}

}  // namespace tlr
