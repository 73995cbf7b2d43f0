// llg_kernels.cu -- RK4 time stepping of the LLG equation on the GPU, FP64.
//
// Arithmetic contract: every operation is an explicitly rounded FP64
// intrinsic (__dmul_rn, __dadd_rn, __dsub_rn, __ddiv_rn, __dsqrt_rn), in the
// order the reference writes it, so the compiler cannot contract a*b+c into
// an FMA.  With alpha = J2 = h = 0 the trajectory is therefore bit-identical
// to the reference's euler / runge_kutta / renormalisation built with
// -ffp-contract=off (llg_sqt_baseline.c:29-142, :298-309).
#include <cooperative_groups.h>

#include <algorithm>
#include <cmath>
#include <cstdlib>
#include <type_traits>

#include "asd_internal.h"

namespace asd {
namespace {

#include "llg_math.cuh"

// One fused RK4 stage, site-major layout.  Thread t handles replica
// f = t % nfile of site t / nfile, so a warp touches 32 consecutive 24-byte
// records (768 contiguous bytes) of each operand.  The combination order
// reproduces runge_kutta's final sum spin + k1/6 + k2/3 + k3/3 + k4/6
// evaluated left to right (llg_sqt_baseline.c:138), carried in acc.
//
// Thread mapping.  With fewer than 64 replicas, thread t is (site t / nc,
// replica t % nc).  With 64 or more (ngroups = ceil(nc / 32) groups of 32),
// block b takes a 2 x 4 patch of sites (one per warp) of replica group
// b % ngroups, lane = replica within the group: the warps of a block are
// lattice neighbours, so many of the input vectors a warp reads as
// neighbours are other warps' centres and hit in L1 instead of L2 (the block
// reads 20 distinct site vectors for 8 sites, 24 with J2, instead of 40 / 72).
// Measured on B200 against one thread per (site, replica) in order:
// 256x256x1000 with J2 5.21 vs 6.12-6.21 ms per step of four stages.
// At most 32 registers (8 blocks of 256 threads per SM): stage 4 with J2
// otherwise takes 34 and only 6 blocks fit.
template <int STAGE, bool J2, bool H, bool DAMP>
__global__ void __launch_bounds__(256, 8) llg_stage_kernel(LLGArgs a, const double *__restrict__ y,
                                                        const double *__restrict__ ys,
                                                        double *__restrict__ acc,
                                                        double *__restrict__ out, int ngroups) {
    pdl_begin();
    long site;
    int f;
    if (ngroups > 0) {
        const int g = (int)(blockIdx.x % ngroups);
        const long tile = blockIdx.x / ngroups;
        const int tcols = (a.N + 3) / 4;
        const int w = threadIdx.x >> 5;
        const int trow = (int)(tile / tcols) * 2 + (w >> 2), tcol = (int)(tile % tcols) * 4 + (w & 3);
        const int lf = g * 32 + (threadIdx.x & 31);
        if (trow >= a.N || tcol >= a.N || lf >= a.nc) return;
        site = (long)trow * a.N + tcol;
        f = a.f0 + lf;
    } else {
        const long t = (long)blockIdx.x * blockDim.x + threadIdx.x;
        if (t >= a.M * a.nc) return;
        site = t / a.nc;
        f = a.f0 + (int)(t - site * a.nc);
    }
    const int row = (int)(site / a.N), col = (int)(site - (long)row * a.N);
    const long sstride = 3L * a.nfile;
    const long off = 3L * f;
    const V3 d = llg_rhs<J2, H, DAMP>(ys, sstride, off, a.N, row, col, a);
    const long e = site * sstride + off;
    const double k0 = dm(d.x, a.dt), k1 = dm(d.y, a.dt), k2 = dm(d.z, a.dt);
    if (STAGE == 1) {
        const double y0 = y[e], y1 = y[e + 1], y2 = y[e + 2];
        out[e] = da(y0, half(k0));
        out[e + 1] = da(y1, half(k1));
        out[e + 2] = da(y2, half(k2));
        acc[e] = da(y0, div6(k0));
        acc[e + 1] = da(y1, div6(k1));
        acc[e + 2] = da(y2, div6(k2));
    } else if (STAGE == 2 || STAGE == 3) {
        const double y0 = y[e], y1 = y[e + 1], y2 = y[e + 2];
        if (STAGE == 2) {
            out[e] = da(y0, half(k0));
            out[e + 1] = da(y1, half(k1));
            out[e + 2] = da(y2, half(k2));
        } else {
            out[e] = da(y0, k0);
            out[e + 1] = da(y1, k1);
            out[e + 2] = da(y2, k2);
        }
        acc[e] = da(acc[e], div3(k0));
        acc[e + 1] = da(acc[e + 1], div3(k1));
        acc[e + 2] = da(acc[e + 2], div3(k2));
    } else {
        const double o0 = da(acc[e], div6(k0));
        const double o1 = da(acc[e + 1], div6(k1));
        const double o2 = da(acc[e + 2], div6(k2));
        // llg_sqt_baseline.c:301-308 / llg_sqt_fusion.c:353-360
        const double nrm = __dsqrt_rn(da(da(dm(o0, o0), dm(o1, o1)), dm(o2, o2)));
        out[e] = dq(dm(a.spin_len, o0), nrm);
        out[e + 1] = dq(dm(a.spin_len, o1), nrm);
        out[e + 2] = dq(dm(a.spin_len, o2), nrm);
    }
}

__device__ __forceinline__ V3 ld3(const double *p) { return V3{p[0], p[1], p[2]}; }

constexpr int kGroupedMinReplicas = 64;  // below: one thread per (site, replica) in order

template <int STAGE>
cudaError_t launch_stage_t(const LLGArgs &a, const double *y, const double *ys, double *acc,
                           double *out, cudaStream_t st) {
    if (a.f0 < 0 || a.nc < 1 || a.f0 + a.nc > a.nfile) return cudaErrorInvalidValue;
    const long total = a.M * a.nc;
    const int threads = 256;
    const int sel = (a.use_j2 ? 4 : 0) | (a.use_h ? 2 : 0) | (a.use_damp ? 1 : 0);
    // site-grouped mapping when the replica groups of 32 are mostly full
    const int ngroups = (a.nc >= kGroupedMinReplicas) ? (a.nc + 31) / 32 : 0;
    const long gblocks = (long)ngroups * ((a.N + 1) / 2) * ((a.N + 3) / 4);
    if (gblocks > 0x7fffffffL) return cudaErrorInvalidConfiguration;
    const unsigned blocks = ngroups > 0 ? (unsigned)gblocks
                                        : (unsigned)((total + threads - 1) / threads);
#define ASD_STAGE_CASE(S, J, Hh, D)                                                            \
    case S:                                                                                    \
        return launch_pdl(llg_stage_kernel<STAGE, J, Hh, D>, blocks, threads, 0, st, a, y, ys, \
                          acc, out, ngroups);
    switch (sel) {
        ASD_STAGE_CASE(0, false, false, false)
        ASD_STAGE_CASE(1, false, false, true)
        ASD_STAGE_CASE(2, false, true, false)
        ASD_STAGE_CASE(3, false, true, true)
        ASD_STAGE_CASE(4, true, false, false)
        ASD_STAGE_CASE(5, true, false, true)
        ASD_STAGE_CASE(6, true, true, false)
        ASD_STAGE_CASE(7, true, true, true)
    }
#undef ASD_STAGE_CASE
    return cudaErrorInvalidValue;
}

// ------------------------------------------------ row-streaming step
// One RK4 step per launch, streamed down the lattice.  The work is a set of
// columns of rows: a band of wc core columns (plus 4 halo columns each side,
// one per stage) for SF replicas, over all N rows.  A persistent grid of
// CTAs splits the band x replica-group x row space evenly, each CTA taking
// one contiguous run of rows that crosses at most a few (band, group)
// boundaries; every piece of a run is streamed on its own.
//
// A piece of rs rows (relative rows 0..rs+7: 4 halo rows above and below)
// is walked once, two phases per iteration j, separated by barriers:
//   phase A: stage 1 on row j-1 (y rows j-2..j), stage 3 on row j-4;
//   phase B: cp.async prefetch of y row j+1, stage 2 on row j-2, stage 4 on
//            row j-5 (renormalised, stored to DRAM).
// Each stage reads only rows written in an earlier phase, and the two stages
// of a phase are independent (twice the instruction-level parallelism of a
// stage-per-phase schedule, half the barriers).  Stage inputs live in rings
// of 3 rows, y in a ring of 5 rows, and the running RK4 combination of the
// five rows in flight in registers.  Halo work is (wc + 8) / wc in columns;
// DRAM traffic: y read once (the halo columns mostly from L2) and y_new
// written once, 48 bytes per site-step.  Per (site, replica) the arithmetic
// is the stage kernels' (bit-identical); with |J1| = 1 and the exact half and
// whole factors as FMAs 42 of 303 FP64 operations go (128x128x500 379 -> 364 us,
// 256x256x1000 with J2 3545 -> 3452 us).  Keeping y's own column in registers
// (12 shared loads fewer) spilled 160 bytes at the 96 registers that two CTAs of
// nine warps leave.
namespace stream {
constexpr int SF = 4;                  // replicas per CTA (96 contiguous bytes per site)
constexpr int WC_MAX = 64;             // core columns per band
constexpr int WT_MAX = WC_MAX + 8;     // columns held per row
constexpr int NT_MAX = WT_MAX * SF;    // threads per CTA at most (288)
constexpr int YR = 5;                  // rows of the y ring
constexpr int ROWS = YR + 3 * 3;       // row buffers in shared memory
constexpr int MIN_RUN = 16;            // fewest rows per CTA
}  // namespace stream

struct StreamGeom {
    int wc;   // core columns per band (a multiple of 8)
    int wt;   // wc + 8 columns held per row
    int nb;   // bands: ceil(N / wc)
    int ng;   // replica groups: ceil(nc / SF)
    int rw;   // doubles per row buffer: wt * SF * 3
    long run; // rows per CTA of the nb * ng * N rows of work
};

__device__ __forceinline__ void cp_async8(double *dst, const double *src) {
    const unsigned d = (unsigned)__cvta_generic_to_shared(dst);
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8;\n" ::"r"(d), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_async_commit() {
    asm volatile("cp.async.commit_group;\n" ::: "memory");
}
__device__ __forceinline__ void cp_async_wait_all() {
    asm volatile("cp.async.wait_group 0;\n" ::: "memory");
}


// Inputs of one stage at one (site, replica): the centre value, its
// neighbours in llg_rhs's order -- (row+1), (row-1), (col-1), (col+1), then
// the diagonals (+1,+1), (+1,-1), (-1,+1), (-1,-1) -- and the RK4 base y.
struct SIn {
    V3 s, nb[4], n2[4], yb;
};

// Loads record `me` of row buffer `mid` and its neighbours from the rows
// above (`up`, row-1) and below (`dn`, row+1); CS = doubles per column.
template <bool J2>
__device__ __forceinline__ void load_in(const double *up, const double *mid, const double *dn,
                                        int me, SIn &in) {
    constexpr int CS = stream::SF * 3;
    in.s = ld3(mid + me);
    in.nb[0] = ld3(dn + me);
    in.nb[1] = ld3(up + me);
    in.nb[2] = ld3(mid + me - CS);
    in.nb[3] = ld3(mid + me + CS);
    if (J2) {
        in.n2[0] = ld3(dn + me + CS);
        in.n2[1] = ld3(dn + me - CS);
        in.n2[2] = ld3(up + me + CS);
        in.n2[3] = ld3(up + me - CS);
    }
}

template <bool J2, bool H, bool DAMP, bool UNIT>
__global__ void __launch_bounds__(stream::NT_MAX, 2)
    llg_step_stream_kernel(LLGArgs a, StreamGeom g, const double *__restrict__ y,
                           double *__restrict__ yout) {
    pdl_begin();
    using namespace stream;
    extern __shared__ double ssm[];
    const int rw = g.rw;
    double *const ybuf = ssm;
    double *const s1 = ssm + YR * rw;
    double *const s2 = s1 + 3 * rw;
    double *const s3 = s2 + 3 * rw;
    const int N = a.N;
    const long K = 3L * a.nfile;
    const int tid = threadIdx.x;
    const int cl = tid / SF, fl = tid - cl * SF;
    const int me = tid * 3;  // == (cl * SF + fl) * 3
    const bool comp = cl >= 1 && cl <= g.wt - 2;
    const double dt = a.dt;

    const long total = (long)g.nb * g.ng * N;
    long b = (long)blockIdx.x * g.run;
    const long e = min(b + g.run, total);
    while (b < e) {
        // piece: rows [R0, R0 + rs) of work column u = band + nb * grp
        const long u = b / N;
        const int R0 = (int)(b - u * N);
        const int rs = (int)min((long)(N - R0), e - b);
        b += rs;
        const int band = (int)(u % g.nb), grp = (int)(u / g.nb);
        const int C0 = band * g.wc;
        const int fbase = a.f0 + grp * SF;
        const int nvalid = min(SF, a.f0 + a.nc - fbase);
        const int gcol = C0 + cl - 4;
        const bool store = cl >= 4 && cl < 4 + g.wc && gcol < N && fl < nvalid;
        const int J = rs + 9;  // iterations: stage 4 reaches relative row rs + 3 at j = rs + 8

        // A row buffer holds rw = 3 * blockDim.x doubles, so each thread
        // copies three of them per row: column c = x / 12 of the band
        // (periodic), value w = x % 12 of its 4 replicas x 3 components.
        // Their offsets within a lattice row are the same for every row of
        // the piece, so they are formed once here, not once per row.
        long goff[3];
        bool gval[3];
#pragma unroll
        for (int k = 0; k < 3; ++k) {
            const int x = tid + k * (int)blockDim.x;
            const int c = x / (SF * 3), w = x - c * (SF * 3);
            int gc = (C0 - 4 + c) % N;
            if (gc < 0) gc += N;
            gval[k] = w < 3 * nvalid;
            goff[k] = (long)gc * K + 3L * fbase + w;
        }
        const long row_stride = (long)N * K;
        // y row R0 - 4 + j (periodic) of this band and replica group -> y ring
        auto load_row = [&](int j, int slot) {  // slot = j % YR
            int gr = R0 - 4 + j;  // in [-4, N + 4): at most two wraps for N >= 3
            while (gr < 0) gr += N;
            while (gr >= N) gr -= N;
            const double *src = y + (long)gr * row_stride;
            double *dst = ybuf + slot * rw;
#pragma unroll
            for (int k = 0; k < 3; ++k) {
                const int x = tid + k * (int)blockDim.x;
                if (gval[k])
                    cp_async8(dst + x, src + goff[k]);
                else
                    dst[x] = 0.0;
            }
        };
        // Stage bodies on relative row r (in y slot r % 5, ring slot r % 3),
        // each split into its shared-memory loads (ld) and its arithmetic and
        // stores (st*), so that the two stages of a phase can issue all their
        // loads before either computes.  The callers pass the ring slots of
        // rows r - 1, r, r + 1 (and of the base row in the y ring, or -1):
        // the y slots are compile-time constants of the unrolled iteration,
        // the 3-row ring slots one of three rotations of a running j % 3.
        auto ld = [&](const double *ring, int su, int sm, int sd, int sb) {
            SIn in;
            load_in<J2>(ring + su * rw, ring + sm * rw, ring + sd * rw, me, in);
            if (sb >= 0) in.yb = ld3(ybuf + sb * rw + me);
            return in;
        };
        auto st1 = [&](const SIn &in, int r3, double *ac) {  // s1 = y + k/2, acc = y + k/6
            const V3 d = llg_rhs_vals<J2, H, DAMP, UNIT>(in.s, in.nb, in.n2, a);
            const double k0 = dm(d.x, dt), k1 = dm(d.y, dt), k2 = dm(d.z, dt);
            double *o = s1 + r3 * rw + me;
            o[0] = add_pow2(in.s.x, 0.5, k0);
            o[1] = add_pow2(in.s.y, 0.5, k1);
            o[2] = add_pow2(in.s.z, 0.5, k2);
            ac[0] = da(in.s.x, div6(k0));
            ac[1] = da(in.s.y, div6(k1));
            ac[2] = da(in.s.z, div6(k2));
        };
        auto st2 = [&](const SIn &in, int r3, double *ac) {  // s2 = y + k/2, acc += k/3
            const V3 d = llg_rhs_vals<J2, H, DAMP, UNIT>(in.s, in.nb, in.n2, a);
            const double k0 = dm(d.x, dt), k1 = dm(d.y, dt), k2 = dm(d.z, dt);
            double *o = s2 + r3 * rw + me;
            o[0] = add_pow2(in.yb.x, 0.5, k0);
            o[1] = add_pow2(in.yb.y, 0.5, k1);
            o[2] = add_pow2(in.yb.z, 0.5, k2);
            ac[0] = da(ac[0], div3(k0));
            ac[1] = da(ac[1], div3(k1));
            ac[2] = da(ac[2], div3(k2));
        };
        auto st3 = [&](const SIn &in, int r3, double *ac) {  // s3 = y + k, acc += k/3
            const V3 d = llg_rhs_vals<J2, H, DAMP, UNIT>(in.s, in.nb, in.n2, a);
            const double k0 = dm(d.x, dt), k1 = dm(d.y, dt), k2 = dm(d.z, dt);
            double *o = s3 + r3 * rw + me;
            o[0] = da(in.yb.x, k0);
            o[1] = da(in.yb.y, k1);
            o[2] = da(in.yb.z, k2);
            ac[0] = da(ac[0], div3(k0));
            ac[1] = da(ac[1], div3(k1));
            ac[2] = da(ac[2], div3(k2));
        };
        auto st4 = [&](const SIn &in, int r, const double *ac) {  // acc + k/6, renormalised
            const V3 d = llg_rhs_vals<J2, H, DAMP, UNIT>(in.s, in.nb, in.n2, a);
            const double k0 = dm(d.x, dt), k1 = dm(d.y, dt), k2 = dm(d.z, dt);
            const double o0 = da(ac[0], div6(k0));
            const double o1 = da(ac[1], div6(k1));
            const double o2 = da(ac[2], div6(k2));
            const double nrm = __dsqrt_rn(da(da(dm(o0, o0), dm(o1, o1)), dm(o2, o2)));
            if (store) {
                double *gp = yout + ((long)(R0 - 4 + r) * N + gcol) * K + 3L * (fbase + fl);
                gp[0] = dq(dm(a.spin_len, o0), nrm);
                gp[1] = dq(dm(a.spin_len, o1), nrm);
                gp[2] = dq(dm(a.spin_len, o2), nrm);
            }
        };

        double acc[5][3];  // row r's combination in acc[r % 5]
        __syncthreads();   // the previous piece is done with every buffer
        load_row(0, 0);
        cp_async_commit();
        // Iteration j with R = j % 5 known at compile time, so acc[] and the y
        // ring slots are static; m3 = j % 3 runs along, and the 3-row ring
        // slots of rows j - 1 .. j - 6 are its rotations (j-3, j-6: m3;
        // j-2, j-5: m3 + 1; j-1, j-4: m3 + 2, mod 3).  Valid rows: stage s on
        // relative rows s..rs+7-s.
        int m3 = 0;
        auto iter = [&](auto rc, int j) {
            constexpr int R = decltype(rc)::value;
            if (j >= J) return;  // uniform over the CTA
            const int a0 = m3, a1 = (m3 == 2) ? 0 : m3 + 1, a2 = (m3 == 0) ? 2 : m3 - 1;
            m3 = a1;
            cp_async_wait_all();
            __syncthreads();  // phase A: stage 1 on row j-1, stage 3 on row j-4
            if (comp) {
                const bool d1 = j >= 2 && j <= rs + 7, d3 = j >= 7;
                const int y_m2 = (j + 3) % 5, y_m1 = (j + 4) % 5, y_0 = j % 5, y_m4 = (j + 1) % 5;
                if (d1 && d3) {
                    const SIn i1 = ld(ybuf, y_m2, y_m1, y_0, -1), i3 = ld(s2, a1, a2, a0, y_m4);
                    st1(i1, a2, acc[(R + 4) % 5]);
                    st3(i3, a2, acc[(R + 1) % 5]);
                } else if (d1) {
                    st1(ld(ybuf, y_m2, y_m1, y_0, -1), a2, acc[(R + 4) % 5]);
                } else if (d3) {
                    st3(ld(s2, a1, a2, a0, y_m4), a2, acc[(R + 1) % 5]);
                }
            }
            __syncthreads();  // phase B: prefetch, stage 2 on row j-2, stage 4 on row j-5
            if (j + 1 <= rs + 7) load_row(j + 1, (R + 1) % 5);
            cp_async_commit();
            if (comp) {
                const bool d2 = j >= 4 && j <= rs + 7, d4 = j >= 9;
                const int y_m2 = (j + 3) % 5;
                if (d2 && d4) {
                    const SIn i2 = ld(s1, a0, a1, a2, y_m2), i4 = ld(s3, a0, a1, a2, -1);
                    st2(i2, a1, acc[(R + 3) % 5]);
                    st4(i4, j - 5, acc[R]);
                } else if (d2) {
                    st2(ld(s1, a0, a1, a2, y_m2), a1, acc[(R + 3) % 5]);
                } else if (d4) {
                    st4(ld(s3, a0, a1, a2, -1), j - 5, acc[R]);
                }
            }
        };
        for (int j0 = 0; j0 < J; j0 += 5) {
            iter(std::integral_constant<int, 0>{}, j0);
            iter(std::integral_constant<int, 1>{}, j0 + 1);
            iter(std::integral_constant<int, 2>{}, j0 + 2);
            iter(std::integral_constant<int, 3>{}, j0 + 3);
            iter(std::integral_constant<int, 4>{}, j0 + 4);
        }
    }
}

StreamGeom stream_geom(const LLGArgs &a) {
    using namespace stream;
    StreamGeom g;
    g.nb = (a.N + WC_MAX - 1) / WC_MAX;
    g.wc = ((a.N + g.nb - 1) / g.nb + 7) / 8 * 8;  // wt * SF is a whole number of warps
    g.wt = g.wc + 8;
    g.rw = g.wt * SF * 3;
    g.ng = (a.nc + SF - 1) / SF;
    g.run = 0;
    return g;
}

size_t stream_smem_bytes(const StreamGeom &g) {
    return (size_t)stream::ROWS * g.rw * sizeof(double);
}

template <bool J2, bool H, bool DAMP, bool UNIT>
cudaError_t launch_stream_t(const LLGArgs &a, const double *y, double *yout, cudaStream_t st) {
    using namespace stream;
    auto k = llg_step_stream_kernel<J2, H, DAMP, UNIT>;
    StreamGeom g = stream_geom(a);
    const int threads = g.wt * SF;
    const size_t smem = stream_smem_bytes(g);
    cudaError_t e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return e;
    int dev = 0, sms = 0, per_sm = 0;
    if ((e = cudaGetDevice(&dev)) != cudaSuccess) return e;
    if ((e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev)) != cudaSuccess)
        return e;
    if ((e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k, threads, smem)) !=
        cudaSuccess)
        return e;
    // One CTA per resident slot, each with an equal run of the rows of work
    // (at least MIN_RUN, so the 9-iteration fill of a piece stays small).
    const long total = (long)g.nb * g.ng * a.N;
    const long slots = (long)sms * (per_sm > 0 ? per_sm : 1);
    long run = (total + slots - 1) / slots;
    if (run < MIN_RUN) run = MIN_RUN;
    g.run = run;
    const long blocks = (total + run - 1) / run;
    if (blocks > 0x7fffffffL) return cudaErrorInvalidConfiguration;
    return launch_pdl(k, (unsigned)blocks, threads, smem, st, a, g, y, yout);
}

cudaError_t launch_stream(const LLGArgs &a, const double *y, double *yout, cudaStream_t st) {
    if (a.f0 < 0 || a.nc < 1 || a.f0 + a.nc > a.nfile) return cudaErrorInvalidValue;
    const int sel = (a.use_j2 ? 4 : 0) | (a.use_h ? 2 : 0) | (a.use_damp ? 1 : 0);
    const bool unit = a.J1 == 1.0 || a.J1 == -1.0;
#define ASD_STREAM_CASE(S, J, Hh, D)                                              \
    case S:                                                                       \
        return unit ? launch_stream_t<J, Hh, D, true>(a, y, yout, st)             \
                    : launch_stream_t<J, Hh, D, false>(a, y, yout, st);
    switch (sel) {
        ASD_STREAM_CASE(0, false, false, false)
        ASD_STREAM_CASE(1, false, false, true)
        ASD_STREAM_CASE(2, false, true, false)
        ASD_STREAM_CASE(3, false, true, true)
        ASD_STREAM_CASE(4, true, false, false)
        ASD_STREAM_CASE(5, true, false, true)
        ASD_STREAM_CASE(6, true, true, false)
        ASD_STREAM_CASE(7, true, true, true)
    }
#undef ASD_STREAM_CASE
    return cudaErrorInvalidValue;
}

// ------------------------------------------------- resident steps
// Any number of RK4 steps in one launch, one replica's whole lattice held on
// chip: a thread-block cluster of S CTAs (S = 1: a CTA) per replica, its rows
// split over the CTAs.  A CTA keeps the stage input and the stage output of its
// rows in shared memory (rows of 3 x W doubles, one halo row above and below,
// the two swapped after every stage); a thread owns up to RP consecutive rows of
// one column, whose running RK4 combination stays in registers and whose base
// values y lie in a planar scratch in L2, read and written by that thread alone.
// Walking down its column a thread reuses the two rows above from registers: 9
// shared loads per site and stage instead of 15 (21 instead of 27 with J2), all
// at compile-time offsets.  The first and last row of a CTA are also stored into
// the neighbouring CTAs' halo rows (distributed shared memory, or the same
// CTA's when S = 1), so one barrier ends a stage.  No redundant halo
// arithmetic, no traffic between steps.
//
// Up to 32 columns: CTAs of 256 threads with at most 4 rows each, three to an SM
// (85 registers); above, 512 threads with at most 8 rows, one to an SM (128).
namespace resident {
__host__ __device__ constexpr int threads(int W) { return W <= 32 ? 256 : 512; }
__host__ __device__ constexpr int rows_per_thread(int W) { return W <= 32 ? 4 : 8; }
__host__ __device__ constexpr int ctas_per_sm(int W) { return W <= 32 ? 3 : 1; }
}  // namespace resident

struct ResGeom {
    int s;       // CTAs per replica
    int rows;    // rows of the largest CTA
    int groups;  // row groups: threads / N
};

template <int W, bool J2, bool H, bool DAMP, bool UNIT, bool CL>
__global__ void __launch_bounds__(resident::threads(W), resident::ctas_per_sm(W))
    llg_resident_kernel(LLGArgs a, ResGeom g, const double *y, double *yout, double *scratch,
                        int nsteps) {
    pdl_begin();
    namespace cg = cooperative_groups;
    constexpr int RP = resident::rows_per_thread(W), WARPS = resident::threads(W) / 32;
    constexpr int RS = 3 * W;  // doubles per row
    extern __shared__ double rsm[];
    const int N = a.N, rank = CL ? (int)(blockIdx.x % g.s) : 0;
    const int lf = CL ? (int)(blockIdx.x / g.s) : (int)blockIdx.x;
    const int r0 = (int)((long)rank * N / g.s), nr = (int)((long)(rank + 1) * N / g.s) - r0;
    const int bs = (g.rows + 2) * RS;  // doubles per buffer
    const long K = 3L * a.nfile, off = 3L * (a.f0 + lf);
    double *ysc = scratch + (long)lf * 3 * a.M;  // [3][M]: this replica's y

    // every CTA's rows and halo rows of the initial state, a warp per row:
    // consecutive lanes take the components of a site, then the next site
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    for (int l = warp; l < nr + 2; l += WARPS) {
        int row = r0 - 1 + l;
        row = row < 0 ? row + N : (row >= N ? row - N : row);
        const double *src = y + (long)row * N * K + off;
        for (int x = lane; x < 3 * N; x += 32)
            cp_async8(rsm + l * RS + (x % 3) * W + x / 3, src + (long)(x / 3) * K + x % 3);
    }
    cp_async_commit();
    double *up_cta = rsm, *dn_cta = rsm;  // shared memory of the CTAs above and below
    int nr_up = nr;
    if (CL) {
        cg::cluster_group cluster = cg::this_cluster();
        const int ru = rank == 0 ? g.s - 1 : rank - 1, rd = rank + 1 == g.s ? 0 : rank + 1;
        up_cta = cluster.map_shared_rank(rsm, ru);
        dn_cta = cluster.map_shared_rank(rsm, rd);
        nr_up = (int)((long)(ru + 1) * N / g.s) - (int)((long)ru * N / g.s);
    }
    auto barrier = [&] {
        if (CL) cg::this_cluster().sync();
        else __syncthreads();
    };
    const int grp = threadIdx.x / N, col = threadIdx.x - grp * N;
    const int rp = (nr + g.groups - 1) / g.groups;      // <= RP
    const int first = grp * rp;                         // this thread's rows of the CTA
    const int cnt = grp < g.groups ? min(rp, nr - first) : 0;
    const int dl = col == 0 ? N - 1 : -1, dr = col == N - 1 ? 1 - N : 1;
    const int at0 = (first + 1) * RS + col;
    const long site0 = (long)(r0 + first) * N + col;
    // halo copies of the CTA's first and last row (only their owners use them)
    const bool owns_top = cnt > 0 && first == 0, owns_bot = cnt > 0 && first + cnt == nr;
    double *const halo_up = up_cta + (nr_up + 1) * RS + col, *const halo_dn = dn_cta + col;
    cp_async_wait_all();
    barrier();

    double acc[RP][3];
    // One stage, buffer `in` to buffer `out`; body(r, s, k) gives the output of
    // the thread's row r from its value s and k = dt f.
    auto walk = [&](int in, int out, auto body) {
        const double *const p = rsm + in * bs + at0, *const pl = p + dl, *const pr = p + dr;
        double *const o = rsm + out * bs + at0;
        const int ob = out * bs;
        auto at = [](const double *q) { return V3{q[0], q[W], q[2 * W]}; };
        V3 up, mid;
        if (cnt > 0) {
            up = at(p - RS);
            mid = at(p);
        }
#pragma unroll
        for (int r = 0; r < RP; ++r) {
            if (r < cnt) {
                const int q = r * RS;
                V3 nb[4], n2[4];
                nb[0] = at(p + q + RS);
                nb[1] = up;
                nb[2] = at(pl + q);
                nb[3] = at(pr + q);
                if (J2) {
                    n2[0] = at(pr + q + RS);
                    n2[1] = at(pl + q + RS);
                    n2[2] = at(pr + q - RS);
                    n2[3] = at(pl + q - RS);
                }
                const V3 d = llg_rhs_vals<J2, H, DAMP, UNIT>(mid, nb, n2, a);
                const V3 v = body(r, mid, V3{dm(d.x, a.dt), dm(d.y, a.dt), dm(d.z, a.dt)});
                o[q] = v.x;
                o[q + W] = v.y;
                o[q + 2 * W] = v.z;
                if (r == 0 && owns_top) {
                    halo_up[ob] = v.x;
                    halo_up[ob + W] = v.y;
                    halo_up[ob + 2 * W] = v.z;
                }
                if (owns_bot && r == cnt - 1) {
                    halo_dn[ob] = v.x;
                    halo_dn[ob + W] = v.y;
                    halo_dn[ob + 2 * W] = v.z;
                }
                up = mid;
                mid = nb[0];
            }
        }
    };
    for (int step = 0; step < nsteps; ++step) {
        // Stages 1 to 3: out = y + ck k; acc = y + k/6, then acc + k/3.  One copy
        // of the code: the divisors and their reciprocals (div6, div3) and the
        // factors 1/2 and 1 are uniform variables, the roundings the same.
#pragma unroll 1
        for (int st = 1; st <= 3; ++st) {
            const double ck = st == 3 ? 1.0 : 0.5, dd = st == 1 ? 6.0 : 3.0;
            const double inv = st == 1 ? 1.0 / 6.0 : 1.0 / 3.0;
            double *yp = ysc + site0;
            walk((st - 1) & 1, st & 1, [&](int r, const V3 &s, const V3 &k) {
                V3 yb = s;
                if (st > 1) {
                    yb = V3{yp[0], yp[a.M], yp[2 * a.M]};
                } else if (step == 0) {  // later steps: written by stage 4
                    yp[0] = s.x;
                    yp[a.M] = s.y;
                    yp[2 * a.M] = s.z;
                }
                yp += N;
                auto div = [&](double x) {
                    const double q = __dmul_rn(x, inv);
                    const double t = __fma_rn(q, dd, -x);
                    return __fma_rn(-t, inv, q);
                };
                const double bx = st == 1 ? yb.x : acc[r][0], by = st == 1 ? yb.y : acc[r][1],
                             bz = st == 1 ? yb.z : acc[r][2];
                acc[r][0] = da(bx, div(k.x));
                acc[r][1] = da(by, div(k.y));
                acc[r][2] = da(bz, div(k.z));
                return V3{add_pow2(yb.x, ck, k.x), add_pow2(yb.y, ck, k.y), add_pow2(yb.z, ck, k.z)};
            });
            barrier();
        }
        double *yp = ysc + site0;
        const bool more = step + 1 < nsteps;
        walk(1, 0, [&](int r, const V3 &, const V3 &k) {
            const double o0 = da(acc[r][0], div6(k.x));
            const double o1 = da(acc[r][1], div6(k.y));
            const double o2 = da(acc[r][2], div6(k.z));
            const double nrm = __dsqrt_rn(da(da(dm(o0, o0), dm(o1, o1)), dm(o2, o2)));
            const V3 v{dq(dm(a.spin_len, o0), nrm), dq(dm(a.spin_len, o1), nrm),
                       dq(dm(a.spin_len, o2), nrm)};
            if (more) {
                yp[0] = v.x;
                yp[a.M] = v.y;
                yp[2 * a.M] = v.z;
                yp += N;
            }
            return v;
        });
        barrier();  // also: no CTA leaves while another may store into its halo rows
    }
    for (int l = warp; l < nr; l += WARPS) {
        double *dst = yout + (long)(r0 + l) * N * K + off;
        const double *src = rsm + (l + 1) * RS;
        for (int x = lane; x < 3 * N; x += 32)
            dst[(long)(x / 3) * K + x % 3] = src[(x % 3) * W + x / 3];
    }
}

// Tiled transpose between [nfile][M][3] and [M][nfile][3] through shared
// memory: 32 sites x 32 replicas x 3 doubles per block.  Bound by HBM: a thread
// keeps one of a row's 96 doubles, so its 16 rows are a constant stride apart
// and all its loads are in flight at once; rows of 99 doubles (3 mod 16) make
// the transposed reads free of bank conflicts.  Measured on B200, site-major to
// AoS, against 256 threads with a division per element and rows of 97:
// 128x128x500 94 -> 63.5 us (6.2 TB/s), 256x256x1000 689 -> 502, 64x64x100 8.5 -> 6.2.
constexpr int TR_THREADS = 192, TR_ROWS = TR_THREADS / 96, TR_N = 32 / TR_ROWS;
template <bool TO_SITEMAJOR>
__global__ void __launch_bounds__(TR_THREADS) transpose_kernel(const double *__restrict__ src,
                                                               double *__restrict__ dst, long M,
                                                               int nfile, int fbeg, int nc) {
    pdl_begin();
    // The AoS side holds replicas [fbeg, fbeg + nc) as [nc][M][3]; the
    // site-major side is the whole [M][nfile][3] array.
    __shared__ double tile[32][32 * 3 + 3];
    const long s0 = (long)blockIdx.x * 32;
    const int l0 = blockIdx.y * 32;
    const int w = threadIdx.x % 96, r0 = threadIdx.x / 96, q = w / 3, c = w - 3 * q;
    const int ns = (int)min(32L, M - s0), nl = min(32, nc - l0);  // sites, replicas here
    // 96 contiguous doubles a row: sites of a replica, replicas of a site
    const long aos = ((long)l0 * M + s0) * 3 + w, sm = (s0 * nfile + fbeg + l0) * 3 + w;
    const long aos_row = 3 * M, sm_row = 3L * nfile;
    const double *p = src + (TO_SITEMAJOR ? aos : sm);
    double *o = dst + (TO_SITEMAJOR ? sm : aos);
    const long prow = TO_SITEMAJOR ? aos_row : sm_row, orow = TO_SITEMAJOR ? sm_row : aos_row;
    const int prows = q < (TO_SITEMAJOR ? ns : nl) ? (TO_SITEMAJOR ? nl : ns) : 0;
    const int orows = q < (TO_SITEMAJOR ? nl : ns) ? (TO_SITEMAJOR ? ns : nl) : 0;
    double x[TR_N];
#pragma unroll
    for (int t = 0; t < TR_N; ++t) {
        const int r = r0 + TR_ROWS * t;
        x[t] = r < prows ? p[r * prow] : 0.0;
    }
#pragma unroll
    for (int t = 0; t < TR_N; ++t) tile[r0 + TR_ROWS * t][w] = x[t];
    __syncthreads();
#pragma unroll
    for (int t = 0; t < TR_N; ++t) {
        const int r = r0 + TR_ROWS * t;
        if (r < orows) o[r * orow] = tile[q][r * 3 + c];
    }
}

// euler on the reference layout: thread t -> site t % M of replica t / M
// (the reference's loop order, llg_sqt_baseline.c:44-48), reference physics.
__global__ void __launch_bounds__(256) euler_aos_kernel(LLGArgs a, const double *__restrict__ y,
                                                        double *__restrict__ d) {
    const long t = (long)blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= a.M * a.nfile) return;
    const long f = t / a.M;
    const long site = t - f * a.M;
    const int row = (int)(site / a.N), col = (int)(site - (long)row * a.N);
    const V3 r = llg_rhs<false, false, false>(y, 3, f * a.M * 3, a.N, row, col, a);
    d[t * 3] = r.x;
    d[t * 3 + 1] = r.y;
    d[t * 3 + 2] = r.z;
}

// runge_kutta's element-wise loops (llg_sqt_baseline.c:104-139).
__global__ void rk_pass_kernel(int pass, long n, double dt, const double *__restrict__ spin,
                               double *__restrict__ cur, double *__restrict__ k,
                               const double *__restrict__ k1, const double *__restrict__ k2,
                               const double *__restrict__ k3) {
    const long j = (long)blockIdx.x * blockDim.x + threadIdx.x;
    if (j >= n) return;
    const double kk = dm(k[j], dt);
    k[j] = kk;
    if (pass == 1 || pass == 2) {
        cur[j] = da(spin[j], half(kk));
    } else if (pass == 3) {
        cur[j] = da(spin[j], kk);
    } else {
        double v = da(spin[j], dq(k1[j], 6.0));
        v = da(v, dq(k2[j], 3.0));
        v = da(v, dq(k3[j], 3.0));
        cur[j] = da(v, dq(kk, 6.0));
    }
}

__global__ void div_check_kernel(const double *__restrict__ x, long n, unsigned long long *bad) {
    for (long i = (long)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (long)gridDim.x * blockDim.x) {
        const double v = x[i];
        const bool ok3 = __double_as_longlong(div3(v)) == __double_as_longlong(__ddiv_rn(v, 3.0));
        const bool ok6 = __double_as_longlong(div6(v)) == __double_as_longlong(__ddiv_rn(v, 6.0));
        if (!ok3 || !ok6) atomicAdd(bad, 1ull);
    }
}

}  // namespace

cudaError_t launch_div_check(const double *x, long n, unsigned long long *bad, cudaStream_t st) {
    div_check_kernel<<<1184, 256, 0, st>>>(x, n, bad);
    return cudaGetLastError();
}

LLGArgs make_llg_args(const asd_params &p) {
    LLGArgs a;
    a.N = p.N;
    a.nfile = p.nfile;
    a.M = (long)p.N * p.N;
    a.J1 = p.J1;
    a.J2 = p.J2;
    a.hx = p.hx;
    a.hy = p.hy;
    a.hz = p.hz;
    a.alpha = p.alpha;
    a.g = 1.0 / (1.0 + p.alpha * p.alpha);
    a.dt = p.dt;
    a.spin_len = p.spin_len;
    a.use_j2 = p.J2 != 0.0;
    a.use_h = (p.hx != 0.0 || p.hy != 0.0 || p.hz != 0.0);
    a.use_damp = p.alpha != 0.0;
    a.f0 = 0;
    a.nc = p.nfile;
    return a;
}

cudaError_t launch_llg_stage(int stage, const LLGArgs &a, const double *y, const double *ys_in,
                             double *acc, double *ys_out, cudaStream_t st) {
    switch (stage) {
        case 1: return launch_stage_t<1>(a, y, ys_in, acc, ys_out, st);
        case 2: return launch_stage_t<2>(a, y, ys_in, acc, ys_out, st);
        case 3: return launch_stage_t<3>(a, y, ys_in, acc, ys_out, st);
        case 4: return launch_stage_t<4>(a, y, ys_in, acc, ys_out, st);
    }
    return cudaErrorInvalidValue;
}

// The geometry of the resident steps for lattice side N: rows of W doubles a
// component, the fewest CTAs per replica (1, 2, 4) whose threads cover the
// rows and whose two buffers fit shared memory; false if none does.
static bool resident_geom(int N, ResGeom &g, int &w, size_t &smem) {
    w = N <= 32 ? 32 : N <= 64 ? 64 : 128;
    if (N > w) return false;
    g.groups = resident::threads(w) / N;
    for (g.s = 1; g.s <= 4 && g.s <= N; g.s *= 2) {
        g.rows = (N + g.s - 1) / g.s;
        smem = (size_t)2 * 3 * (g.rows + 2) * w * sizeof(double);
        if ((g.rows + g.groups - 1) / g.groups <= resident::rows_per_thread(w) && smem <= 227 * 1024) return true;
    }
    return false;
}

template <int W, bool J2, bool H, bool DAMP, bool UNIT>
static cudaError_t launch_resident_t(const LLGArgs &a, const ResGeom &g, size_t smem,
                                     const double *y, double *yout, double *scratch, int nsteps,
                                     cudaStream_t st) {
    constexpr bool CL = W > 64;  // up to 64 columns one CTA holds a lattice
    auto k = llg_resident_kernel<W, J2, H, DAMP, UNIT, CL>;
    cudaError_t e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return e;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)((long)a.nc * g.s));
    cfg.blockDim = dim3(resident::threads(W));
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;  // as launch_pdl
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    attr[1].id = cudaLaunchAttributeClusterDimension;
    attr[1].val.clusterDim.x = (unsigned)g.s;
    attr[1].val.clusterDim.y = 1;
    attr[1].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = CL ? 2 : 1;
    return cudaLaunchKernelEx(&cfg, k, a, g, y, yout, scratch, nsteps);
}

template <int W>
static cudaError_t launch_resident_w(const LLGArgs &a, const ResGeom &g, size_t smem,
                                     const double *y, double *yout, double *scratch, int nsteps,
                                     cudaStream_t st) {
    const bool unit = a.J1 == 1.0 || a.J1 == -1.0;
    const int sel = (a.use_j2 ? 4 : 0) | (a.use_h ? 2 : 0) | (a.use_damp ? 1 : 0);
#define ASD_RES_CASE(S, J, Hh, D)                                                                 \
    case S:                                                                                       \
        return unit ? launch_resident_t<W, J, Hh, D, true>(a, g, smem, y, yout, scratch, nsteps,  \
                                                           st)                                    \
                    : launch_resident_t<W, J, Hh, D, false>(a, g, smem, y, yout, scratch, nsteps, \
                                                            st);
    switch (sel) {
        ASD_RES_CASE(0, false, false, false)
        ASD_RES_CASE(1, false, false, true)
        ASD_RES_CASE(2, false, true, false)
        ASD_RES_CASE(3, false, true, true)
        ASD_RES_CASE(4, true, false, false)
        ASD_RES_CASE(5, true, false, true)
        ASD_RES_CASE(6, true, true, false)
        ASD_RES_CASE(7, true, true, true)
    }
#undef ASD_RES_CASE
    return cudaErrorInvalidValue;
}

cudaError_t launch_llg_resident(const LLGArgs &a, const double *y, double *yout, double *scratch,
                                int nsteps, cudaStream_t st) {
    ResGeom g;
    int w = 0;
    size_t smem = 0;
    if (nsteps < 1 || a.f0 < 0 || a.nc < 1 || a.f0 + a.nc > a.nfile ||
        !resident_geom(a.N, g, w, smem))
        return cudaErrorInvalidValue;
    return w == 32   ? launch_resident_w<32>(a, g, smem, y, yout, scratch, nsteps, st)
           : w == 64 ? launch_resident_w<64>(a, g, smem, y, yout, scratch, nsteps, st)
                     : launch_resident_w<128>(a, g, smem, y, yout, scratch, nsteps, st);
}

// The three ways to step, compared by what each was measured to take on B200 (in
// us a step; within 10 % of the measurements near the crossings).  w =
// site-replicas, n = sites of a CTA:
//   stage kernels   9 + 0.065e-3 w (0.073 with J2): four launches, then HBM / L2
//   one-launch      rows per CTA + 9 iterations, for 72 columns 3.1 with two CTAs
//                   an SM and 1.8 with one (1.29 times that with J2)
//   resident        2.8 a launch, and per round of resident CTAs, q to an SM:
//                   2.3 + 3.7e-3 q n a step (clusters 6.3 + 3.9e-3 n; 1.35 times
//                   the part in n with J2), and 0.8 + 3.1e-3 q n once to load and
//                   store the lattice (1.9e-3 up to 32 columns)
// for 148 SMs, the same work a CTA on others (LLGArgs::sms).  Measured, stage kernels / one-launch / resident 1 step / resident 10 steps:
//   32x32x50    11.2 /  36 / 12.2 /  6.9     64x64x8     9.7 / 45 / 31.4 / 18.5
//   32x32x200   22   /  37 / 16.3 / 10.2     64x64x100  35.8 / 45 / 35.3 / 18.6
//   32x32x1000  70   /  67 / 51.9 / 31.5     12x12x1000 18   / 49 / 18.9 / 10.1
//   64x64x400   114  /  97 / 101  / 55.3     128x128x500 531 / 364 / 604 / 341
//   51x51x70    22   /  48 / 21.3 / 13.5     90x90x60   36.5 / 60
// and with J2, resident 1 / 4 steps a launch: 64x64x1000 298 / 268 / 278 / 189,
//   64x64x700   214  / 190 / 197  / 134      128x128x150 193 / 170 / -   / 151
static double stages_cost(const LLGArgs &a) {
    return 9.0 + (a.use_j2 ? 0.073e-3 : 0.065e-3) * (double)a.M * a.nc;
}

static double fused_cost(const LLGArgs &a) {
    const StreamGeom g = stream_geom(a);
    const long total = (long)g.nb * g.ng * a.N;
    const double run = std::max<double>(stream::MIN_RUN, total / (2.0 * a.sms));
    const double two = std::min(1.0, std::max(0.0, total / run / a.sms - 1.0));  // SMs with two
    const double iter = std::max(1.45 + 0.45 * two, (1.8 + 1.3 * two) * (g.wt + 24) / 96.0);
    return (run + 9.0) * iter * (a.use_j2 ? 1.29 : 1.0);
}

bool llg_fused_wins(const LLGArgs &a) { return fused_cost(a) < 0.95 * stages_cost(a); }

bool llg_resident_wins(const LLGArgs &a, int nsteps) {
    ResGeom g;
    int w = 0;
    size_t smem = 0;
    if (!resident_geom(a.N, g, w, smem)) return false;
    const double n = (double)g.rows * a.N;
    const bool cl = g.s > 1;
    const double base = cl ? 6.3 : 2.3, site = (cl ? 3.9e-3 : 3.7e-3) * (a.use_j2 ? 1.35 : 1.0);
    const double move = w <= 32 ? 1.9e-3 : 3.1e-3;
    auto round = [&](double q) { return nsteps * (base + site * q * n) + 0.8 + move * q * n; };
    // CTAs an SM takes in all (clusters of 4 fill about 140 of 148), and q at once
    const double per_sm = (double)a.nc * g.s / (cl ? a.sms * 140.0 / 148.0 : (double)a.sms);
    const int at_once = resident::ctas_per_sm(w);
    double res = 2.8;
    if (per_sm > 3.0 * at_once) {  // rounds blur into one another
        res += (per_sm / at_once + 0.3) * round(at_once);
    } else {
        for (int left = (int)std::ceil(per_sm); left > 0; left -= at_once)
            res += round(std::min(left, at_once));
    }
    return res < 0.95 * nsteps * std::min(stages_cost(a), fused_cost(a));
}

cudaError_t launch_llg_step_fused(const LLGArgs &a, const double *y, double *yout,
                                  cudaStream_t st) {
    return launch_stream(a, y, yout, st);
}

cudaError_t launch_aos_to_sitemajor_range(const double *aos, double *sm, long M, int nfile,
                                          int f0, int nc, cudaStream_t st) {
    if (f0 < 0 || nc < 1 || f0 + nc > nfile) return cudaErrorInvalidValue;
    dim3 grid((unsigned)((M + 31) / 32), (unsigned)((nc + 31) / 32));
    return launch_pdl(transpose_kernel<true>, grid, TR_THREADS, 0, st, aos, sm, M, nfile, f0, nc);
}

cudaError_t launch_sitemajor_to_aos_range(const double *sm, double *aos, long M, int nfile,
                                          int f0, int nc, cudaStream_t st) {
    if (f0 < 0 || nc < 1 || f0 + nc > nfile) return cudaErrorInvalidValue;
    dim3 grid((unsigned)((M + 31) / 32), (unsigned)((nc + 31) / 32));
    return launch_pdl(transpose_kernel<false>, grid, TR_THREADS, 0, st, sm, aos, M, nfile, f0, nc);
}

cudaError_t launch_aos_to_sitemajor(const double *aos, double *sm, long M, int nfile,
                                    cudaStream_t st) {
    return launch_aos_to_sitemajor_range(aos, sm, M, nfile, 0, nfile, st);
}

cudaError_t launch_sitemajor_to_aos(const double *sm, double *aos, long M, int nfile,
                                    cudaStream_t st) {
    return launch_sitemajor_to_aos_range(sm, aos, M, nfile, 0, nfile, st);
}

cudaError_t launch_euler_aos(const LLGArgs &a, const double *spin, double *deriv,
                             cudaStream_t st) {
    const long total = a.M * a.nfile;
    euler_aos_kernel<<<(unsigned)((total + 255) / 256), 256, 0, st>>>(a, spin, deriv);
    return cudaGetLastError();
}

cudaError_t launch_rk_pass(int pass, long n, double dt, const double *spin, double *cur,
                           double *k, const double *k1, const double *k2, const double *k3,
                           cudaStream_t st) {
    rk_pass_kernel<<<(unsigned)((n + 255) / 256), 256, 0, st>>>(pass, n, dt, spin, cur, k, k1,
                                                                 k2, k3);
    return cudaGetLastError();
}

}  // namespace asd

extern "C" int asd_check_const_division(const double *x, long n, unsigned long long *bad,
                                        void *stream) {
    using namespace asd;
    if (!x || !bad || n < 0) return fail(ASD_ERR_INVALID, "bad argument");
    ASD_CUDA_TRY(launch_div_check(x, n, bad, (cudaStream_t)stream));
    return ASD_OK;
}
