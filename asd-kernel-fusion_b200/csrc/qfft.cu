// qfft.cu -- S(q,t) on the whole q grid in FP64, as 2-D Fourier transforms of
// the spins instead of the correlation product.
//
// At q = 2 pi (a, b) / N the connected correlation (gemm/llg_sqt_mkl.c:378-423
// with the phase of llg_sqt_baseline.c:265-268) is
//   S(q) = (1/(M nfile)) sum_k A~_k(q) conj(B~_k(q)),
// A~, B~ the 2-D transforms (kernel e^{-i q.r}) of column k of A - m and B - z,
// m and z the replica means at t and at the origin: sum_f (B - z) = 0, so
// subtracting m changes nothing but the rounding.  One complex transform serves
// both: with Z the transform of (A - m) + i (B - z), W = Z(-q),
//   A~ conj(B~) = (Z.x W.y + Z.y W.x) / 2 + (i/4) (|Z|^2 - |W|^2),
// whose rounding is that of the larger of |A~|^2 and |B~|^2.  So each operand is
// brought to the same size first, by a power of two from its largest component
// (read beside the means); the product is multiplied back at the end.  Spins of
// length 1 and 1e8 then have the relative error of equal ones (2e-9 without), and
// none overflow that the product does not.
// About 5 M log2(M) operations per column instead of 2 M^2.
//
// Columns go in chunks whose transform (16 M bytes a column) stays in L2, held
// in two buffers of the context's RK4 scratch (the caller leaves out the one that
// the one-launch step alternates with the state, as a captured call's replays may
// find the state in it) and, for the last blocks of a lattice whose columns make
// one chunk, in a small one of their own:
//   qfft_rows_kernel  a block takes one lattice row of KC columns, transforms
//                     along it in shared memory, writes X[r][b][columns]
//   qfft_cols_kernel  a block takes the lattice columns b and N - b of up to
//                     KC columns k, transforms both side by side, forms the
//                     product above for every a and adds it to its slice's
//                     sums over k
//   qfft_sum_kernel   sums the slices, scales, writes q and -q (conjugates)
// Both passes hold eight or more lines side by side (16 bytes each), so that
// eight neighbouring threads touch one 128-byte line in shared memory (and, KC
// = 8, in global memory) whatever the stride along the lattice: no bank
// conflicts for any radix.
// Stockham stages of radix 8, 4, 2, 3, 5 in registers; any other prime factor p
// as p-term sums from the twiddle table, so every N works.  Fixed order of
// summation everywhere: the grid repeats bit for bit.  The split modes' N x N
// displacement bins take the same transform (bins_dft_kernel).
//
// Bound by shared-memory traffic (each stage reads and writes 16 bytes a point)
// and, below about 64 x 64, by launch latency.  Measured on B200 against the FP64
// tensor-core GEMM with diagonal sums that served this before: 256x256x1000 831
// -> 6.55 ms, 128x128x500 26.9 -> 0.82 ms, 32x32x200 0.145 -> 0.026 ms; of these
// the scaling by magnitude 0.01, 0.015 and 0.0007 ms.
#include "asd_internal.h"

namespace asd {
namespace {

constexpr int MAX_STAGES = 12;
constexpr int MAX_THREADS = 256;
constexpr int MAX_SHARED_TW = 2048;  // column pass: longer twiddle tables stay in L2

struct FftPlan {
    int n;
    int stages;
    int radix[MAX_STAGES];
    int lk;   // log2 of the columns k held side by side, KC
    int lkc;  // the same in the column pass (of each of its two lines)
};

__device__ __forceinline__ double2 cadd(double2 a, double2 b) { return make_double2(a.x + b.x, a.y + b.y); }
__device__ __forceinline__ double2 csub(double2 a, double2 b) { return make_double2(a.x - b.x, a.y - b.y); }
__device__ __forceinline__ double2 cmul(double2 a, double2 b) {
    return make_double2(a.x * b.x - a.y * b.y, a.x * b.y + a.y * b.x);
}
// The caller's buffer holds doubles, on any boundary of eight bytes: two stores
// of eight bytes, never one of sixteen.
__device__ __forceinline__ void put(double *out, long i, double2 v) {
    out[2 * i] = v.x;
    out[2 * i + 1] = v.y;
}
__device__ __forceinline__ double2 mul_mi(double2 a) { return make_double2(a.y, -a.x); }  // -i a

// Forward transforms of length R in registers.
template <int R>
__device__ __forceinline__ void dft(double2 (&v)[R]);

template <>
__device__ __forceinline__ void dft<2>(double2 (&v)[2]) {
    const double2 t = v[0];
    v[0] = cadd(t, v[1]);
    v[1] = csub(t, v[1]);
}
template <>
__device__ __forceinline__ void dft<3>(double2 (&v)[3]) {
    constexpr double S3 = 0.86602540378443864676;  // sin(2 pi / 3)
    const double2 s = cadd(v[1], v[2]), d = csub(v[1], v[2]);
    const double2 m = make_double2(v[0].x - 0.5 * s.x, v[0].y - 0.5 * s.y);
    const double2 q = make_double2(S3 * d.y, -S3 * d.x);  // -i S3 d
    v[0] = cadd(v[0], s);
    v[1] = cadd(m, q);
    v[2] = csub(m, q);
}
template <>
__device__ __forceinline__ void dft<4>(double2 (&v)[4]) {
    const double2 a = cadd(v[0], v[2]), b = csub(v[0], v[2]);
    const double2 c = cadd(v[1], v[3]), d = mul_mi(csub(v[1], v[3]));
    v[0] = cadd(a, c);
    v[1] = cadd(b, d);
    v[2] = csub(a, c);
    v[3] = csub(b, d);
}
template <>
__device__ __forceinline__ void dft<5>(double2 (&v)[5]) {
    constexpr double C1 = 0.30901699437494742410, C2 = -0.80901699437494742410;  // cos(2 pi k / 5)
    constexpr double S1 = 0.95105651629515357212, S2 = 0.58778525229247312917;   // sin
    const double2 s1 = cadd(v[1], v[4]), d1 = csub(v[1], v[4]);
    const double2 s2 = cadd(v[2], v[3]), d2 = csub(v[2], v[3]);
    const double2 m1 = make_double2(v[0].x + C1 * s1.x + C2 * s2.x, v[0].y + C1 * s1.y + C2 * s2.y);
    const double2 m2 = make_double2(v[0].x + C2 * s1.x + C1 * s2.x, v[0].y + C2 * s1.y + C1 * s2.y);
    const double2 q1 = mul_mi(make_double2(S1 * d1.x + S2 * d2.x, S1 * d1.y + S2 * d2.y));
    const double2 q2 = mul_mi(make_double2(S2 * d1.x - S1 * d2.x, S2 * d1.y - S1 * d2.y));
    v[0] = cadd(v[0], cadd(s1, s2));
    v[1] = cadd(m1, q1);
    v[2] = cadd(m2, q2);
    v[3] = csub(m2, q2);
    v[4] = csub(m1, q1);
}
template <>
__device__ __forceinline__ void dft<8>(double2 (&v)[8]) {
    constexpr double H = 0.70710678118654752440;
    double2 e[4] = {v[0], v[2], v[4], v[6]}, o[4] = {v[1], v[3], v[5], v[7]};
    dft<4>(e);
    dft<4>(o);
    o[1] = make_double2(H * (o[1].x + o[1].y), H * (o[1].y - o[1].x));    // e^{-i pi / 4}
    o[2] = mul_mi(o[2]);
    o[3] = make_double2(H * (o[3].y - o[3].x), -H * (o[3].x + o[3].y));   // e^{-3 i pi / 4}
#pragma unroll
    for (int t = 0; t < 4; ++t) {
        v[t] = cadd(e[t], o[t]);
        v[t + 4] = csub(e[t], o[t]);
    }
}

// One Stockham stage on n points x 2^lk columns: Ns points are already
// combined; tw[j] = e^{-2 pi i j / n}.
template <int R>
__device__ __forceinline__ void stage(const double2 *in, double2 *out, const double2 *tw, int n,
                                      int Ns, int lk) {
    const int step = n / R, twu = step / Ns, total = step << lk, km = (1 << lk) - 1;
    for (int idx = threadIdx.x; idx < total; idx += blockDim.x) {
        const int k = idx & km, j = idx >> lk, jm = j % Ns;
        double2 v[R];
#pragma unroll
        for (int s = 0; s < R; ++s) v[s] = in[((j + s * step) << lk) + k];
        if (Ns > 1) {
#pragma unroll
            for (int s = 1; s < R; ++s) v[s] = cmul(v[s], tw[s * jm * twu]);
        }
        dft<R>(v);
        const int base = (j - jm) * R + jm;
#pragma unroll
        for (int t = 0; t < R; ++t) out[((base + t * Ns) << lk) + k] = v[t];
    }
}

// The same for any radix p, one output per thread.
__device__ __forceinline__ void stage_any(const double2 *in, double2 *out, const double2 *tw, int n,
                                          int p, int Ns, int lk) {
    const int step = n / p, twu = step / Ns, total = n << lk, km = (1 << lk) - 1;
    for (int idx = threadIdx.x; idx < total; idx += blockDim.x) {
        const int k = idx & km, o = idx >> lk;  // output position
        const int jm = o % Ns, q = o / Ns, t = q % p, j = (q / p) * Ns + jm;
        const int e = jm * twu + t * step;  // < n
        double2 acc = make_double2(0.0, 0.0);
        int w = 0;
        for (int s = 0; s < p; ++s) {
            const double2 x = in[((j + s * step) << lk) + k], c = tw[w];
            acc.x += x.x * c.x - x.y * c.y;
            acc.y += x.x * c.y + x.y * c.x;
            w += e;
            if (w >= n) w -= n;
        }
        out[(o << lk) + k] = acc;
    }
}

// Transforms `a` (n points x 2^lk columns); b is the other buffer.  Returns the
// one that holds the result; every thread is past its last write.
__device__ __forceinline__ double2 *transform(double2 *a, double2 *b, const double2 *tw,
                                              const FftPlan &p, int lk) {
    int Ns = 1;
    for (int s = 0; s < p.stages; ++s) {
        const int r = p.radix[s];
        if (r == 8) stage<8>(a, b, tw, p.n, Ns, lk);
        else if (r == 4) stage<4>(a, b, tw, p.n, Ns, lk);
        else if (r == 2) stage<2>(a, b, tw, p.n, Ns, lk);
        else if (r == 3) stage<3>(a, b, tw, p.n, Ns, lk);
        else if (r == 5) stage<5>(a, b, tw, p.n, Ns, lk);
        else stage_any(a, b, tw, p.n, r, Ns, lk);
        Ns *= r;
        double2 *t = a;
        a = b;
        b = t;
        __syncthreads();
    }
    return a;
}

// 2^(1023 - e) for the exponent field e of the largest magnitude (high word top),
// which brings it to [1, 2), and the inverse; 1 where it is subnormal or not finite.
// The inverse of a zero operand is 0: its product is, but for the rounding of the other.
__device__ __forceinline__ double to_unit(unsigned top) {
    const int e = (int)(top >> 20);
    return e == 0 || e == 0x7ff ? 1.0 : __hiloint2double((2046 - min(e, 2045)) << 20, 0);
}
__device__ __forceinline__ double from_unit(unsigned top) {
    const int e = (int)(top >> 20);
    if (top == 0) return 0.0;
    return e == 0 || e == 0x7ff ? 1.0 : __hiloint2double(min(e, 2045) << 20, 0);
}

__global__ void qfft_twiddle_kernel(int n, double2 *__restrict__ tw) {
    const int j = blockIdx.x * blockDim.x + threadIdx.x;
    if (j >= n) return;
    double sn, cs;
    sincospi(2.0 * (double)j / (double)n, &sn, &cs);
    tw[j] = make_double2(cs, -sn);
}

// The transforms of a chunk's blocks of KC columns: `per` blocks in each of the
// first two buffers, the rest in the third, each as [n][n][width] with width = the
// blocks there * KC.
struct Chunk {
    double2 *buf[3];
    int blocks, per;
    // column k of the chunk
    __device__ __forceinline__ double2 *at(int k, int lk, int &width) const {
        const int q = min(2, (k >> lk) / per), first = q * per;
        width = (q == 2 ? blocks - first : min(per, blocks - first)) << lk;
        return buf[q] + (k - (first << lk));
    }
};

// Block (kb, r): columns k0 + kb KC .. of lattice row r; columns at K and
// beyond are zero.
__global__ void __launch_bounds__(MAX_THREADS) qfft_rows_kernel(
    FftPlan p, const double *__restrict__ A, const double *__restrict__ B, int K, int k0, Chunk X,
    const double *__restrict__ m, const double *__restrict__ z, const unsigned *__restrict__ top,
    const double2 *__restrict__ tw) {
    pdl_begin();
    extern __shared__ __align__(16) double2 fsm[];
    const int n = p.n, kc = 1 << p.lk;
    double2 *b0 = fsm, *b1 = fsm + (n << p.lk), *stw = b1 + (n << p.lk);
    for (int j = threadIdx.x; j < n; j += blockDim.x) stw[j] = tw[j];
    const long r = blockIdx.y;
    const int kl = blockIdx.x * kc;  // within the chunk
    const double fa = to_unit(top[0]), fb = to_unit(top[1]);
    for (int idx = threadIdx.x; idx < (n << p.lk); idx += blockDim.x) {
        const int c = idx >> p.lk, k = k0 + kl + (idx & (kc - 1));
        double2 v = make_double2(0.0, 0.0);
        if (k < K) {
            const long site = r * n + c;
            v.x = (A[site * K + k] - m[site * 3 + k % 3]) * fa;
            v.y = (B[site * K + k] - z[site * 3 + k % 3]) * fb;
        }
        b0[idx] = v;
    }
    __syncthreads();
    const double2 *f = transform(b0, b1, stw, p, p.lk);
    int kw;
    double2 *o = X.at(kl, p.lk, kw);
    o += r * n * kw;
    for (int idx = threadIdx.x; idx < (n << p.lk); idx += blockDim.x)
        o[(long)(idx >> p.lk) * kw + (idx & (kc - 1))] = f[idx];
}

// Block (b, slice): frequencies (a, b) for every a, b <= n / 2; the slice's
// k blocks of this chunk.  add: onto the sums of the earlier chunks.
__global__ void __launch_bounds__(MAX_THREADS) qfft_cols_kernel(
    FftPlan p, Chunk X, const double2 *__restrict__ tw, int add, unsigned *top,
    double2 *__restrict__ part) {
    pdl_begin();
    if (blockIdx.x == 0 && blockIdx.y == 0 && threadIdx.x == 0) top[2] = top[0];
    extern __shared__ __align__(16) double2 fsm[];
    const int n = p.n, kc = 1 << p.lkc, lt = p.lkc + 1, len = n << p.lkc;
    double2 *b0 = fsm, *b1 = b0 + (n << lt), *sum = b1 + (n << lt), *stw = sum + n;
    const int b = blockIdx.x, mb = (b == 0) ? 0 : n - b;
    const bool copy_tw = n <= MAX_SHARED_TW;
    for (int j = threadIdx.x; j < n; j += blockDim.x) {
        if (copy_tw) stw[j] = tw[j];
        sum[j] = make_double2(0.0, 0.0);
    }
    const int nkb = X.blocks << (p.lk - p.lkc);
    for (int kb = blockIdx.y; kb < nkb; kb += gridDim.y) {
        int kw;
        const double2 *x = X.at(kb << p.lkc, p.lk, kw);
        __syncthreads();  // the previous block's products are formed
        // line b in columns 0 .. kc - 1, line n - b in kc .. 2 kc - 1
        for (int idx = threadIdx.x; idx < (n << lt); idx += blockDim.x) {
            const int r = idx >> lt, j = idx & (2 * kc - 1);
            b0[idx] = x[((long)r * n + (j < kc ? b : mb)) * kw + (j & (kc - 1))];
        }
        __syncthreads();
        const double2 *Z = transform(b0, b1, copy_tw ? stw : tw, p, lt);
        // whole warps: len is a multiple of kc, lanes of one a stay together
        for (int i0 = 0; i0 < len; i0 += blockDim.x) {
            const int idx = i0 + threadIdx.x, a = idx >> p.lkc, k = idx & (kc - 1);
            double re = 0.0, im = 0.0;
            if (idx < len) {
                const int ma = (a == 0) ? 0 : n - a;
                const double2 zv = Z[(a << lt) + k], w = Z[(ma << lt) + kc + k];
                re = 0.5 * (zv.x * w.y + zv.y * w.x);
                im = 0.25 * ((zv.x - w.x) * (zv.x + w.x) + (zv.y - w.y) * (zv.y + w.y));
            }
            for (int o = kc >> 1; o > 0; o >>= 1) {
                re += __shfl_xor_sync(0xffffffffu, re, o);
                im += __shfl_xor_sync(0xffffffffu, im, o);
            }
            if (idx < len && k == 0) {
                sum[a].x += re;
                sum[a].y += im;
            }
        }
    }
    __syncthreads();
    double2 *o = part + (long)blockIdx.y * n * (n / 2 + 1) + (long)b * n;
    for (int a = threadIdx.x; a < n; a += blockDim.x) {
        double2 v = sum[a];
        if (add) v = cadd(o[a], v);
        o[a] = v;
    }
}

// 16 frequencies a block, eight threads each: thread s adds slices s, s + 8, ...
// The state's magnitude, of which it reads the copy, is zero again for the next call.
__global__ void __launch_bounds__(128) qfft_sum_kernel(const double2 *__restrict__ part, int n,
                                                       int slices, double scale,
                                                       unsigned *top,
                                                       double *__restrict__ out) {
    pdl_begin();
    if (blockIdx.x == 0 && threadIdx.x == 0) top[0] = 0;
    __shared__ double2 red[8][16];
    const int tl = threadIdx.x & 15, sl = threadIdx.x >> 4;
    const long t = (long)blockIdx.x * 16 + tl;
    const long half = (long)n * (n / 2 + 1);
    double2 s = make_double2(0.0, 0.0);
    if (t < half) {
#pragma unroll 4
        for (int q = sl; q < slices; q += 8) s = cadd(s, part[q * half + t]);
    }
    red[sl][tl] = s;
    __syncthreads();
    if (sl != 0 || t >= half) return;
#pragma unroll
    for (int q = 1; q < 8; ++q) s = cadd(s, red[q][tl]);
    const int b = (int)(t / n), a = (int)(t - (long)b * n);
    const double fa = from_unit(top[2]), fb = from_unit(top[1]);
    s.x = s.x * scale * fa * fb;
    s.y = s.y * scale * fa * fb;
    put(out, (long)a * n + b, s);
    if (b > 0 && 2 * b != n) {  // -q: the displacement sums are real
        const int ma = (a == 0) ? 0 : n - a;
        put(out, (long)ma * n + (n - b), make_double2(s.x, -s.y));
    }
}

// One dimension of the 2-D transform of the displacement bins (split modes):
// a block transforms KC lines.  REAL: lines are rows of G [n][n], the result
// goes transposed to T [frequency][line]; else lines are rows of T, the result
// to out, scaled.
template <bool REAL>
__global__ void __launch_bounds__(MAX_THREADS) bins_dft_kernel(FftPlan p,
                                                               const double *__restrict__ G,
                                                               const double2 *__restrict__ T,
                                                               const double2 *__restrict__ tw,
                                                               double scale,
                                                               double *__restrict__ out) {
    pdl_begin();
    extern __shared__ __align__(16) double2 fsm[];
    const int n = p.n, kc = 1 << p.lk;
    double2 *b0 = fsm, *b1 = fsm + (n << p.lk), *stw = b1 + (n << p.lk);
    for (int j = threadIdx.x; j < n; j += blockDim.x) stw[j] = tw[j];
    const int l0 = blockIdx.x * kc;
    for (int idx = threadIdx.x; idx < (n << p.lk); idx += blockDim.x) {
        const int line = l0 + (idx & (kc - 1));
        const long e = (long)line * n + (idx >> p.lk);
        double2 v = make_double2(0.0, 0.0);
        if (line < n) v = REAL ? make_double2(G[e], 0.0) : T[e];
        b0[idx] = v;
    }
    __syncthreads();
    const double2 *f = transform(b0, b1, stw, p, p.lk);
    for (int idx = threadIdx.x; idx < (n << p.lk); idx += blockDim.x) {
        const int line = l0 + (idx & (kc - 1));
        if (line < n)
            put(out, (long)(idx >> p.lk) * n + line, make_double2(f[idx].x * scale, f[idx].y * scale));
    }
}

FftPlan make_plan(int n, int K) {
    FftPlan p{};
    p.n = n;
    int m = n;
    auto take = [&](int r) {
        while (m % r == 0 && p.stages < MAX_STAGES) {
            p.radix[p.stages++] = r;
            m /= r;
        }
    };
    take(8);
    take(4);
    take(2);
    take(3);
    take(5);
    for (int r = 7; m > 1; r += 2) take(r);
    // Columns side by side: 8, less where the two buffers do not leave room for
    // a second block on the SM or a scratch buffer (K doubles a site) holds no
    // block of them; in the column pass two lines lie side by side.
    auto fits = [&](int lines) { return (size_t)2 * n * lines * sizeof(double2) <= 104 * 1024; };
    p.lk = 3;
    while (p.lk > 0 && (!fits(1 << p.lk) || (2 << p.lk) > K)) --p.lk;
    p.lkc = p.lk;
    while (p.lkc > 0 && !fits(2 << p.lkc)) --p.lkc;
    return p;
}

size_t rows_smem(const FftPlan &p) { return ((size_t)2 * (p.n << p.lk) + p.n) * sizeof(double2); }
size_t cols_smem(const FftPlan &p) {
    return ((size_t)4 * (p.n << p.lkc) + (p.n <= MAX_SHARED_TW ? 2 : 1) * p.n) * sizeof(double2);
}

// Threads of a block: one per four points, whole warps, 64 to 256.
int threads_for(int points) {
    const int t = (points / 4 + 31) / 32 * 32;
    return t < 64 ? 64 : (t > MAX_THREADS ? MAX_THREADS : t);
}

struct Geometry {
    int per;     // blocks of KC columns a scratch buffer holds
    int blocks;  // blocks per chunk
    int own;     // of those, in the third buffer (0 to 2)
    int slices;  // sums over k kept apart
};

Geometry geometry(const FftPlan &p, int K) {
    const int kc = 1 << p.lk, all = (K + kc - 1) / kc;
    Geometry g;
    g.per = K / (2 * kc);
    long b = (48L << 20) / (16L * p.n * p.n * kc);  // the chunk's transform stays in L2
    if (b < 1) b = 1;
    // two buffers hold all blocks but the odd one or two: those, where that makes
    // one chunk of the lattice (32x32x200: 75 blocks of 8 columns, 37 a buffer)
    if (b >= all) b = all;
    else if (b > 2L * g.per) b = 2L * g.per;
    g.blocks = (int)b;
    g.own = g.blocks > 2 * g.per ? g.blocks - 2 * g.per : 0;
    const int lines = p.n / 2 + 1, nkb = g.blocks << (p.lk - p.lkc);
    g.slices = (8 * 148 + lines - 1) / lines;  // about eight blocks per SM
    if (g.slices > nkb) g.slices = nkb;
    return g;
}

}  // namespace

size_t qfft_work_bytes(int lat_n, int K) {
    const size_t n = (size_t)lat_n;
    const FftPlan p = make_plan(lat_n, K);
    const Geometry g = geometry(p, K);
    return (n + g.slices * n * (n / 2 + 1) + (n * n * g.own << p.lk)) * sizeof(double2);
}

cudaError_t launch_qfft_twiddles(int lat_n, void *work, cudaStream_t st) {
    qfft_twiddle_kernel<<<(lat_n + 127) / 128, 128, 0, st>>>(lat_n, static_cast<double2 *>(work));
    return cudaGetLastError();
}

int launch_qfft(const double *A, const double *B, int lat_n, int K, const double *m,
                const double *z, unsigned *top, double scale, void *work,
                double *const scratch[2], double *out, cudaStream_t st) {
    const FftPlan p = make_plan(lat_n, K);
    const Geometry g = geometry(p, K);
    double2 *tw = static_cast<double2 *>(work), *part = tw + lat_n;
    const long half = (long)lat_n * (lat_n / 2 + 1);
    const int rows_t = threads_for(p.n << p.lk), cols_t = threads_for(p.n << (p.lkc + 1));
    const int kc = 1 << p.lk, all = (K + kc - 1) / kc;
    ASD_CUDA_TRY(cudaFuncSetAttribute(qfft_rows_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                      (int)rows_smem(p)));
    ASD_CUDA_TRY(cudaFuncSetAttribute(qfft_cols_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                      (int)cols_smem(p)));
    int launches = 0;
    for (int b0 = 0; b0 < all; b0 += g.blocks) {
        Chunk X;
        for (int q = 0; q < 2; ++q) X.buf[q] = reinterpret_cast<double2 *>(scratch[q]);
        X.buf[2] = part + g.slices * half;
        X.blocks = all - b0 < g.blocks ? all - b0 : g.blocks;
        X.per = g.per;
        ASD_CUDA_TRY(launch_pdl(qfft_rows_kernel, dim3((unsigned)X.blocks, (unsigned)lat_n), rows_t,
                                rows_smem(p), st, p, A, B, K, b0 * kc, X, m, z, top, tw));
        // a last, shorter chunk still visits every slice (with no block it adds zero)
        ASD_CUDA_TRY(launch_pdl(qfft_cols_kernel,
                                dim3((unsigned)(lat_n / 2 + 1), (unsigned)g.slices), cols_t,
                                cols_smem(p), st, p, X, tw, b0 > 0, top, part));
        launches += 2;
    }
    ASD_CUDA_TRY(launch_pdl(qfft_sum_kernel, (unsigned)((half + 15) / 16), 128, 0, st, part, lat_n,
                            g.slices, scale, top, out));
    return launches + 1;
}

cudaError_t launch_bins_dft(const double *G, int lat_n, double scale, const double2 *tw, double2 *T,
                            double *out, cudaStream_t st) {
    const FftPlan p = make_plan(lat_n, 16);
    const int kc = 1 << p.lk, blocks = (lat_n + kc - 1) / kc, threads = threads_for(p.n << p.lk);
    const size_t smem = rows_smem(p);
    cudaError_t e;
    if ((e = cudaFuncSetAttribute(bins_dft_kernel<true>,
                                  cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem)) !=
            cudaSuccess ||
        (e = cudaFuncSetAttribute(bins_dft_kernel<false>,
                                  cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem)) !=
            cudaSuccess)
        return e;
    if ((e = launch_pdl(bins_dft_kernel<true>, blocks, threads, smem, st, p, G, nullptr, tw, 1.0,
                        reinterpret_cast<double *>(T))) != cudaSuccess)
        return e;
    return launch_pdl(bins_dft_kernel<false>, blocks, threads, smem, st, p, nullptr, T, tw, scale, out);
}

}  // namespace asd
