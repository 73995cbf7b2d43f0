// qgrid.cu -- the displacement bins of the full-q-grid S(q,t), in a fixed
// order of summation.
//
// S(q) for every q of the N x N grid is the 2-D DFT of the bins
//   G(dr, dc) = sum over pairs (i, j) with (r_i - r_j, c_i - c_j) = (dr, dc)
//               mod N of  alpha C_ij - m_i . z_j
// (the single-q phase of llg_sqt_baseline.c:265-268 applied to every q).  The
// GEMM epilogues leave, for every tile (mb, nb) of bm x bn sites, the sums of
// that value along each diagonal d = r - c of the tile (r, c the local row and
// column), split by class: 0 when c_j <= c_i (i - j needs no column wrap),
// 1 otherwise.  Along a diagonal, i - j = delta is constant, so the column
// displacement is dc = delta mod N for both classes, and the row displacement
// is (delta - dc) / N in class 0 and one more in class 1.
//
// Tiles with the same key k = mb - (bn / bm) nb have the same i - j on each
// diagonal: delta = k bm + d.  So the bins follow in two fixed-order passes:
//   keys: ds[k][d][cls] = sum over the tiles of key k (slices of them, mb ascending)
//   bins: G(dr, dc) = sum over the (delta, cls) that land there (at most 4)
//         and over the keys whose tiles hold that delta (ascending)
// with no atomics: the bins repeat bit for bit.
#include <cuda_runtime.h>

#include "asd_internal.h"

namespace asd {
namespace {

__device__ __forceinline__ long floordiv(long a, long b) {  // b > 0
    long q = a / b;
    return (a % b != 0 && a < 0) ? q - 1 : q;
}

// A thread takes every KEY_SLICES-th tile of a key, and the slices are added in
// order: a key has up to min(num_m / R, num_n) tiles, a serial chain of L2 loads.
// At 100 x 100 (79 x 40 tiles) 25.7 -> 11.5 us against one thread a sum.
constexpr int KEY_X = 64, KEY_SLICES = 4;
__global__ void __launch_bounds__(KEY_X *KEY_SLICES)
    qgrid_keys_kernel(const float2 *__restrict__ tdiag, int num_m, int num_n, int bm, int bn,
                      const unsigned *__restrict__ top, double *__restrict__ ds) {
    pdl_begin();
    __shared__ double red[KEY_SLICES][KEY_X];
    const int x = threadIdx.x % KEY_X, slice = threadIdx.x / KEY_X;
    const double up = (double)(1L << grid_shift(top));
    const int R = bn / bm, nd = bm + bn - 1;
    const long nkeys = num_m + (long)R * (num_n - 1);
    const long n = nkeys * nd * 2, want = (long)blockIdx.x * KEY_X + x;
    const long idx = want < n ? want : n - 1;  // every thread reaches the barrier
    const long key = idx / (nd * 2);
    const int rem = (int)(idx - key * nd * 2);  // d index * 2 + class
    const long kp = key - (long)R * (num_n - 1);  // mb - R nb
    // tiles: mb = kp (mod R), 0 <= mb < num_m, 0 <= nb = (mb - kp) / R < num_n
    const long mb0 = kp >= 0 ? kp : ((kp % R) + R) % R;
    const long mb_end = kp + (long)R * num_n;  // nb < num_n
    // consecutive tiles of a key lie a constant distance apart
    const float2 *t = tdiag + (mb0 * num_n + (mb0 - kp) / R) * nd * 2 + rem;
    const long step = ((long)R * num_n + 1) * nd * 2, end = num_m < mb_end ? num_m : mb_end;
    double s = 0.0;
    t += slice * step;
#pragma unroll 4
    for (long mb = mb0 + slice * R; mb < end; mb += R * KEY_SLICES, t += step * KEY_SLICES)
        s += grid_value(*t);
    red[slice][x] = s;
    __syncthreads();
    if (slice || want >= n) return;
#pragma unroll
    for (int k = 1; k < KEY_SLICES; ++k) s += red[k][x];
    ds[idx] = s * up;
}

__global__ void qgrid_bins_kernel(const double *__restrict__ ds, int num_m, int num_n, int bm,
                                  int bn, int N, unsigned *top, double *__restrict__ G) {
    pdl_begin();
    if (blockIdx.x == 0 && threadIdx.x == 0) top[0] = 0;  // read by the kernels before
    const long b = (long)blockIdx.x * blockDim.x + threadIdx.x;
    if (b >= (long)N * N) return;
    const int R = bn / bm, nd = bm + bn - 1;
    const long kmin = -(long)R * (num_n - 1), kmax = num_m - 1;
    const int dy = (int)(b / N), dx = (int)(b % N);
    double s = 0.0;
    for (int cls = 0; cls < 2; ++cls)
        for (int w = 0; w < 2; ++w) {
            const long ry = w == 0 ? dy : dy - N;  // row displacement r_i - r_j
            if (ry <= -N) continue;
            const long delta = (long)N * ry + dx - (cls ? N : 0);  // i - j
            long k0 = -floordiv(-(delta - (bm - 1)), bm);          // ceil
            long k1 = floordiv(delta + bn - 1, bm);
            if (k0 < kmin) k0 = kmin;
            if (k1 > kmax) k1 = kmax;
            for (long k = k0; k <= k1; ++k) {
                const long d = delta - k * bm;  // in [-(bn - 1), bm - 1]
                s += ds[((k - kmin) * nd + (d + bn - 1)) * 2 + cls];
            }
        }
    G[b] = s;
}

}  // namespace

long qgrid_keys(int num_m, int num_n, int bm, int bn) {
    return num_m + (long)(bn / bm) * (num_n - 1);
}

cudaError_t launch_qgrid_bins(const float2 *tdiag, int num_m, int num_n, int bm, int bn, int lat_n,
                              unsigned *top, double *ds, double *G, cudaStream_t st) {
    if (bn % bm != 0) return cudaErrorInvalidValue;
    const long n1 = qgrid_keys(num_m, num_n, bm, bn) * (bm + bn - 1) * 2;
    const cudaError_t e = launch_pdl(qgrid_keys_kernel, (unsigned)((n1 + KEY_X - 1) / KEY_X),
                                     KEY_X * KEY_SLICES, 0, st, tdiag, num_m, num_n, bm, bn, top, ds);
    if (e != cudaSuccess) return e;
    const long n2 = (long)lat_n * lat_n;
    return launch_pdl(qgrid_bins_kernel, (unsigned)((n2 + 255) / 256), 256, 0, st, ds, num_m, num_n,
                      bm, bn, lat_n, top, G);
}

}  // namespace asd
