// phase_sum.cu -- S(q,t) at one q in FP64, as the sums the correlation GEMM
// factorises into.
//
// S(q,t) = (1/M) sum_ij u_i w_j (C_ij - m_i . z_j) with C = (1/nfile) A B^T
// (gemm/llg_sqt_mkl.c:378-423) is a bilinear form in the operands: summing
// over the sites first gives
//   S = (1/(M nfile)) sum_k F_k (G_k - Z_c(k)),
//   F_k = sum_i u_i A_ik,  G_k = sum_j w_j B_jk,  Z_c = (1/nfile) sum_f G_(f,c),
// 4 M K operations and one read of A instead of the 2 M^2 K of the product
// (the connected part, sum_c U_c W_c with U, W the sums of the replica means,
// is the Z term).  G and Z belong to the origin and are formed once per origin.
//
// phase_sum_kernel is bound by HBM: it reads A once (8 M K bytes), a thread
// per column pair (16-byte loads; one column and 8 bytes where K is odd), a
// block walking `rows` sites, 16 loads in flight.  phase_value_kernel sums the blocks' partials
// per column, forms the products and the final sum; its last block to finish
// adds the block sums.  Every sum runs in a fixed order.
//
// Measured on B200, one RK4 step, one S(q,t) and the spins' read-out at
// 128x128x500: 26.36 ms with the FP64 tensor-core GEMM (25.85 ms of it) that
// served the FP64 mode before, 0.548 ms with these sums; four S(q,t) and 20
// steps at 51x51x70: 1.150 -> 0.668 ms.  S(q,t) alone, 8 -> 16 loads in flight,
// 8 -> 16 slices and shorter chunks: 128x128x500 70 -> 40 us, 256x256x1000 294 ->
// 245 (6.4 TB/s), 100x100x240 23 -> 14, 64x64x100 17 -> 10.  Relative difference of the values
// 1.5e-16, their error against a 64-bit reference 1.7e-16 (before 2.2e-16).
#include "asd_internal.h"

namespace asd {
namespace {

constexpr int PS_THREADS = 128;
constexpr int PV_K = 32, PV_SLICES = 16;  // columns per value block, slices of the chunk sum

template <int VEC>
__global__ void __launch_bounds__(PS_THREADS) phase_sum_kernel(const double *__restrict__ A, long M,
                                                               int K,
                                                               const double2 *__restrict__ ph,
                                                               long rows,
                                                               double2 *__restrict__ Fpart) {
    pdl_begin();
    const int k = (blockIdx.x * PS_THREADS + threadIdx.x) * VEC;
    if (k >= K) return;
    const long i0 = (long)blockIdx.y * rows, i1 = min(M, i0 + rows);
    double re[VEC], im[VEC];
#pragma unroll
    for (int v = 0; v < VEC; ++v) re[v] = im[v] = 0.0;
    const double *p = A + i0 * K + k;
#pragma unroll 16
    for (long i = i0; i < i1; ++i, p += K) {
        double x[VEC];
        if (VEC == 2) {
            const double2 t = *reinterpret_cast<const double2 *>(p);
            x[0] = t.x;
            x[VEC - 1] = t.y;
        } else {
            x[0] = *p;
        }
        const double2 u = __ldg(ph + i);
#pragma unroll
        for (int v = 0; v < VEC; ++v) {
            re[v] += u.x * x[v];
            im[v] += u.y * x[v];
        }
    }
    double2 *o = Fpart + (long)blockIdx.y * K + k;
#pragma unroll
    for (int v = 0; v < VEC; ++v) o[v] = make_double2(re[v], im[v]);
}

// True in exactly one block of the grid, the last to arrive; its threads then
// see what every other block wrote before.  The counter wraps back to 0.
__device__ __forceinline__ bool last_block(unsigned *count) {
    __shared__ unsigned s_last;
    __threadfence();
    __syncthreads();
    if (threadIdx.x == 0) s_last = atomicInc(count, gridDim.x - 1) == gridDim.x - 1;
    __syncthreads();
    if (s_last) __threadfence();
    return s_last != 0;
}

// Sum of v over the block's 512 threads, a tree of fixed order.
__device__ __forceinline__ double2 block_sum(double2 v) {
    __shared__ double2 red[PV_K * PV_SLICES];
    red[threadIdx.x] = v;
    __syncthreads();
    for (int w = PV_K * PV_SLICES / 2; w > 0; w >>= 1) {
        if (threadIdx.x < w) {
            red[threadIdx.x].x += red[threadIdx.x + w].x;
            red[threadIdx.x].y += red[threadIdx.x + w].y;
        }
        __syncthreads();
    }
    const double2 r = red[0];
    __syncthreads();
    return r;
}

// F_k of 32 columns from the chunk partials: slice s adds chunks s, s + 16,
// ... and the slices are added in order; valid in the threads of slice 0.
__device__ __forceinline__ double2 column_sum(const double2 *__restrict__ Fpart, int nchunks, int K,
                                              int k) {
    __shared__ double2 red[PV_SLICES][PV_K];
    const int kl = threadIdx.x % PV_K, sl = threadIdx.x / PV_K;
    double2 f = make_double2(0.0, 0.0);
    if (k < K) {
#pragma unroll 16
        for (int c = sl; c < nchunks; c += PV_SLICES) {
            const double2 t = Fpart[(long)c * K + k];
            f.x += t.x;
            f.y += t.y;
        }
    }
    red[sl][kl] = f;
    __syncthreads();
    if (sl == 0) {
#pragma unroll
        for (int s = 1; s < PV_SLICES; ++s) {
            f.x += red[s][kl].x;
            f.y += red[s][kl].y;
        }
    }
    return f;
}

// G_k of the origin; the last block then forms Z_c = (1/nfile) sum_f G_(f,c).
__global__ void __launch_bounds__(PV_K *PV_SLICES) phase_origin_kernel(
    const double2 *__restrict__ Fpart, int nchunks, int K, int nfile, double2 *__restrict__ G,
    double2 *__restrict__ Z, unsigned *__restrict__ count) {
    pdl_begin();
    const int k = blockIdx.x * PV_K + threadIdx.x % PV_K;
    const double2 f = column_sum(Fpart, nchunks, K, k);
    if (threadIdx.x < PV_K && k < K) G[k] = f;
    if (!last_block(count)) return;
    for (int c = 0; c < 3; ++c) {
        double2 z = make_double2(0.0, 0.0);
        for (int r = threadIdx.x; r < nfile; r += PV_K * PV_SLICES) {
            const double2 g = __ldcg(G + 3L * r + c);
            z.x += g.x;
            z.y += g.y;
        }
        z = block_sum(z);
        if (threadIdx.x == 0) Z[c] = make_double2(z.x / nfile, z.y / nfile);
    }
}

// out = scale * sum_k F_k (G_k - Z_c(k)), or without Z where Z is null.
__global__ void __launch_bounds__(PV_K *PV_SLICES) phase_value_kernel(
    const double2 *__restrict__ Fpart, int nchunks, int K, const double2 *__restrict__ G,
    const double2 *__restrict__ Z, double scale, double2 *__restrict__ part,
    unsigned *__restrict__ count, double *__restrict__ out) {
    pdl_begin();
    const int k = blockIdx.x * PV_K + threadIdx.x % PV_K;
    const double2 f = column_sum(Fpart, nchunks, K, k);
    if (threadIdx.x < PV_K) {
        double re = 0.0, im = 0.0;
        if (k < K) {
            double2 g = G[k];
            if (Z) {
                const double2 z = Z[k % 3];
                g.x -= z.x;
                g.y -= z.y;
            }
            re = f.x * g.x - f.y * g.y;
            im = f.x * g.y + f.y * g.x;
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            re += __shfl_xor_sync(0xffffffffu, re, o);
            im += __shfl_xor_sync(0xffffffffu, im, o);
        }
        if (threadIdx.x == 0) part[blockIdx.x] = make_double2(re, im);
    }
    if (!last_block(count)) return;
    double2 s = make_double2(0.0, 0.0);
    for (int b = threadIdx.x; b < (int)gridDim.x; b += PV_K * PV_SLICES) {
        const double2 t = __ldcg(part + b);
        s.x += t.x;
        s.y += t.y;
    }
    s = block_sum(s);
    if (threadIdx.x == 0) {
        out[0] = s.x * scale;
        out[1] = s.y * scale;
    }
}

// Rows per chunk: 256, halved (down to 16) until the grid has at least six
// blocks per SM of a B200, so that the blocks' last round is a small part of the
// whole and small lattices still fill the GPU; doubled where the chunks would
// exceed the grid's y extent (N = 4096).  Measured with at least 2 / 4 / 6 / 9
// blocks per SM: 79 / 51 / 41 / 41 us at 128x128x500, 14 / 17 / 15 / 19 at
// 100x100x240 (more chunks cost the value kernel), 20 / 20 / 20 / 20 at 160x160x9.
int chunk_rows(long M, int K) {
    constexpr long kMinBlocks = 6 * 148;
    const int cols = PS_THREADS * (K % 2 == 0 ? 2 : 1);
    const long kb = (K + cols - 1) / cols;
    int rows = 256;
    while (rows > 16 && kb * ((M + rows - 1) / rows) < kMinBlocks) rows >>= 1;
    while ((M + rows - 1) / rows > 65535) rows <<= 1;
    return rows;
}

int chunks_for(long M, int K) { return (int)((M + chunk_rows(M, K) - 1) / chunk_rows(M, K)); }
int value_blocks(int K) { return (K + PV_K - 1) / PV_K; }

cudaError_t sum_columns(const double *A, long M, int K, const double2 *ph, const PhaseWork &w,
                        cudaStream_t st) {
    const int rows = chunk_rows(M, K);
    const int vec = (K % 2 == 0 && ((uintptr_t)A & 15) == 0) ? 2 : 1;
    const int cols = PS_THREADS * vec;
    const dim3 grid((unsigned)((K + cols - 1) / cols), (unsigned)chunks_for(M, K));
    return launch_pdl(vec == 2 ? phase_sum_kernel<2> : phase_sum_kernel<1>, grid, PS_THREADS, 0, st,
                      A, M, K, ph, rows, w.Fpart);
}

}  // namespace

size_t phase_work_bytes(long M, int K) {
    return ((size_t)chunks_for(M, K) * K + value_blocks(K) + 1) * sizeof(double2);
}

PhaseWork phase_work(void *p, long M, int K) {
    PhaseWork w;
    w.Fpart = static_cast<double2 *>(p);
    w.part = w.Fpart + (size_t)chunks_for(M, K) * K;
    w.count = reinterpret_cast<unsigned *>(w.part + value_blocks(K));
    return w;
}

cudaError_t launch_phase_origin(const double *B, long M, int K, int nfile, const double2 *wphase,
                                const PhaseWork &w, double2 *G, double2 *Z, cudaStream_t st) {
    cudaError_t e = sum_columns(B, M, K, wphase, w, st);
    if (e != cudaSuccess) return e;
    return launch_pdl(phase_origin_kernel, value_blocks(K), PV_K * PV_SLICES, 0, st, w.Fpart,
                      chunks_for(M, K), K, nfile, G, Z, w.count);
}

cudaError_t launch_phase_sum(const double *A, long M, int K, const double2 *uphase,
                             const PhaseWork &w, const double2 *G, const double2 *Z, double scale,
                             double *out, cudaStream_t st) {
    cudaError_t e = sum_columns(A, M, K, uphase, w, st);
    if (e != cudaSuccess) return e;
    return launch_pdl(phase_value_kernel, value_blocks(K), PV_K * PV_SLICES, 0, st, w.Fpart,
                      chunks_for(M, K), K, G, Z, scale, w.part, w.count, out);
}

}  // namespace asd
