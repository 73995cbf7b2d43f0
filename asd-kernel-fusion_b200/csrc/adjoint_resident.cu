// adjoint_resident.cu -- the adjoint of a segment of RK4 steps in one launch, one
// replica's lattice held on one, two or four SMs (see adjoint.cu for the
// formulas and llg_kernels.cu for the resident forward steps it mirrors).
//
// A launch takes a segment between two checkpoints: it steps forward from the
// checkpoint keeping every state, then walks the steps back, each as
//   stages 1..3   recomputed; the stage state and its neighbour sums are kept
//   stage 4       recomputed; adjoint of the renormalisation, vector-Jacobian
//                 product at the stage-4 state, P into shared memory
//   3, 2, 1       gather of P (lam_s), product at that stage's state, new P
//   last          gather, lam of the step before; the next state is loaded
// Shared memory holds the two exchange buffers of the forward steps (a stage's
// input and output, then the P of consecutive stages) and the adjoint variables
// lam_v and lam_y; a thread owns up to RP rows of one column; what only it reads
// again (states of the segment, stage states, neighbour sums, lam) lies in a work
// space in L2 laid out by thread: per CTA and row of a thread, planes of THREADS
// doubles, so that every access is coalesced and at a fixed offset from one
// pointer.  Eight barriers a step instead of 9 to 13 launches that
// each read and write whole states.
//
// Bound by latency between shared memory, L2 and the cluster barriers (which wait
// for outstanding stores) at 16 warps an SM: at 64x64x100, two rounds of two CTAs a
// replica, shared memory moves 45 % of its wavefronts and the FP64 pipe is 39 % busy.
// Measured on B200, backward pass alone, us a step, kernel by
// kernel / resident: 64x64x100 144 / 97 (200 CTAs in two rounds), 64x64x74 112 /
// 50, 64x64x20 59 / 30, 48x48x300 223 / 161, 32x32x200 94 / 50, 12x12x500 54 / 37.
// With lam_v, lam_y and loc in registers and the walks unrolled, 1 KB of spills:
// 110 at 64x64x100; planar arrays per replica instead of by thread: 106.
#include <cooperative_groups.h>

#include <algorithm>

#include "asd_internal.h"

namespace asd {
namespace {

#include "llg_math.cuh"
#include "adjoint_math.cuh"

constexpr int THREADS = 512, RP = 4, W = 64, RS = 3 * W;
// Below, a CTA's threads would lie idle and the work space would be mostly padding.
constexpr int MIN_SIDE = 12;

__device__ __forceinline__ void cp_async8(double *dst, const double *src) {
    const unsigned d = (unsigned)__cvta_generic_to_shared(dst);
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8;\n" ::"r"(d), "l"(src) : "memory");
}

// The work space's planes of one row: vectors by role, three planes each.
enum Role { S2, S3, NN1, NN2, NN3, NNN1, NNN2, NNN3, LAMV, LAM, ROLES };
constexpr int PLANE = THREADS, VEC = 3 * PLANE;      // doubles
constexpr int ROW = ROLES * VEC, STATE_ROW = VEC;    // per row of a thread

__device__ __forceinline__ V3 pload(const double *p) { return V3{p[0], p[PLANE], p[2 * PLANE]}; }
__device__ __forceinline__ void pstore(double *p, const V3 &v) {
    p[0] = v.x;
    p[PLANE] = v.y;
    p[2 * PLANE] = v.z;
}

template <bool J2, bool DAMP, bool UNIT>
__global__ void __launch_bounds__(THREADS, 1)
    adjoint_segment_kernel(LLGArgs a, int S, int rows, int groups, int rpmax, AdjSegment q) {
    namespace cg = cooperative_groups;
    extern __shared__ double rsm[];
    __shared__ double2 gz[3];  // G_(f,c) - Z_c of this replica
    const int N = a.N, rank = (int)(blockIdx.x % S), f = (int)(blockIdx.x / S);
    const int r0 = (int)((long)rank * N / S), nr = (int)((long)(rank + 1) * N / S) - r0;
    const int bs = (rows + 2) * RS;
    const long K = 3L * a.nfile, off = 3L * f;
    double *const psum = rsm + 2 * bs;  // [NPAR][THREADS] derivative sums
    // [RP][3][THREADS]: the RK4 combination on the way forward, loc on the way
    // back; lam_y
    double *const accs = psum + NPAR * THREADS, *const lamy = accs + 3 * RP * THREADS;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    cg::cluster_group cluster = cg::this_cluster();
    const int ru = rank == 0 ? S - 1 : rank - 1, rd = rank + 1 == S ? 0 : rank + 1;
    const int nr_up = (int)((long)(ru + 1) * N / S) - (int)((long)ru * N / S);
    auto barrier = [&] {
        if (S > 1) cluster.sync();
        else __syncthreads();
    };

    // the checkpoint's rows and halo rows, a warp per row (site-major)
    for (int l = warp; l < nr + 2; l += THREADS / 32) {
        int row = r0 - 1 + l;
        row = row < 0 ? row + N : (row >= N ? row - N : row);
        const double *src = q.ck + (long)row * N * K + off;
        for (int x = lane; x < 3 * N; x += 32)
            cp_async8(rsm + l * RS + (x % 3) * W + x / 3, src + (long)(x / 3) * K + x % 3);
    }
    asm volatile("cp.async.commit_group;\n" ::: "memory");
#pragma unroll
    for (int p = 0; p < NPAR; ++p) psum[p * THREADS + tid] = 0.0;
    if (tid < 3) {
        const double2 g = q.G[off + tid], z = q.Z[tid];
        gz[tid] = make_double2(g.x - z.x, g.y - z.y);
    }

    const int grp = tid / N, col = tid - grp * N;
    const int rp = (nr + groups - 1) / groups, first = grp * rp;
    const int cnt = grp < groups ? min(rp, nr - first) : 0;
    const int dl = col == 0 ? N - 1 : -1, dr = col == N - 1 ? 1 - N : 1;
    const int at0 = (first + 1) * RS + col;
    const long site0 = (long)(r0 + first) * N + col;
    // this thread's work space, and its rows of state j of the segment
    double *const ws = q.work + (long)blockIdx.x * rpmax * ROW + tid;
    auto state = [&](int j) {
        return q.states + ((long)j * gridDim.x + blockIdx.x) * rpmax * STATE_ROW + tid;
    };
    const bool owns_top = cnt > 0 && first == 0, owns_bot = cnt > 0 && first + cnt == nr;
    double *const halo_up = cluster.map_shared_rank(rsm, ru) + (nr_up + 1) * RS + col;
    double *const halo_dn = cluster.map_shared_rank(rsm, rd) + col;
    asm volatile("cp.async.wait_group 0;\n" ::: "memory");
    barrier();

    auto at = [](const double *p) { return V3{p[0], p[W], p[2 * W]}; };
    // Row r's value into exchange buffer b, with the halo copies.
    auto put = [&](int b, int r, const V3 &v) {
        double *o = rsm + b * bs + at0 + r * RS;
        o[0] = v.x;
        o[W] = v.y;
        o[2 * W] = v.z;
        if (r == 0 && owns_top) {
            halo_up[b * bs] = v.x;
            halo_up[b * bs + W] = v.y;
            halo_up[b * bs + 2 * W] = v.z;
        }
        if (owns_bot && r == cnt - 1) {
            halo_dn[b * bs] = v.x;
            halo_dn[b * bs + W] = v.y;
            halo_dn[b * bs + 2 * W] = v.z;
        }
    };
    // The thread's rows of buffer b in order, with their neighbours: nearest in
    // the forward kernels' order, diagonal where DIAG.
    auto walk = [&](int b, auto diag, auto body) {
        constexpr bool DIAG = decltype(diag)::value;
        const double *const p = rsm + b * bs + at0, *const pl = p + dl, *const pr = p + dr;
        V3 up, mid;
        if (cnt > 0) {
            up = at(p - RS);
            mid = at(p);
        }
        // rolled: unrolled, the walks spill a kilobyte at 128 registers
#pragma unroll 1
        for (int r = 0; r < cnt; ++r) {
            V3 nb[4], n2[4];
            nb[0] = at(p + (r + 1) * RS);
            nb[1] = up;
            nb[2] = at(pl + r * RS);
            nb[3] = at(pr + r * RS);
            if (DIAG) {
                n2[0] = at(pr + (r + 1) * RS);
                n2[1] = at(pl + (r + 1) * RS);
                n2[2] = at(pr + (r - 1) * RS);
                n2[3] = at(pl + (r - 1) * RS);
            }
            body(r, mid, nb, n2);
            up = mid;
            mid = nb[0];
        }
    };
    auto mine = [&](double *p, int r) { return p + r * VEC + tid; };
    auto sum4 = [](const V3 (&n)[4]) { return vadd(vadd(n[0], n[1]), vadd(n[2], n[3])); };
    using TT = std::true_type;
    using JJ = std::integral_constant<bool, J2>;

    // Stages 1 to 3 of a step, buffer to buffer as in llg_resident_kernel; y at yp.
    // KEEP: the stage state and its neighbour sums go to the work space.
    auto stages = [&](double *yp, bool first_write, auto keep) {
        constexpr bool KEEP = decltype(keep)::value;
        using DD = std::integral_constant<bool, J2 || KEEP>;
#pragma unroll 1
        for (int st = 1; st <= 3; ++st) {
            const double ck = st == 3 ? 1.0 : 0.5, dd = st == 1 ? 6.0 : 3.0;
            const double inv = st == 1 ? 1.0 / 6.0 : 1.0 / 3.0;
            walk((st - 1) & 1, DD{}, [&](int r, const V3 &s, const V3(&nb)[4], const V3(&n2)[4]) {
                if (KEEP) {
                    double *w = ws + r * ROW;
                    if (st > 1) pstore(w + (S2 + st - 2) * VEC, s);
                    pstore(w + (NN1 + st - 1) * VEC, sum4(nb));
                    pstore(w + (NNN1 + st - 1) * VEC, sum4(n2));
                }
                const V3 d = llg_rhs_vals<J2, true, DAMP, UNIT>(s, nb, n2, a);
                const V3 k{dm(d.x, a.dt), dm(d.y, a.dt), dm(d.z, a.dt)};
                V3 yb = s;
                if (st > 1) yb = pload(yp + r * STATE_ROW);
                else if (first_write) pstore(yp + r * STATE_ROW, s);
                auto div = [&](double x) {
                    const double w = __dmul_rn(x, inv);
                    const double t = __fma_rn(w, dd, -x);
                    return __fma_rn(-t, inv, w);
                };
                double *ac = mine(accs, r);
                const V3 from = st == 1 ? yb : pload(ac);
                pstore(ac, V3{da(from.x, div(k.x)), da(from.y, div(k.y)),
                                       da(from.z, div(k.z))});
                put(st & 1, r, V3{add_pow2(yb.x, ck, k.x), add_pow2(yb.y, ck, k.y), add_pow2(yb.z, ck, k.z)});
            });
            barrier();
        }
    };

    // forward through the segment: states base .. base + len - 1
    for (int j = 1; j < q.len; ++j) {
        stages(state(j - 1), j == 1, std::false_type{});
        double *yn = state(j);
        walk(1, JJ{}, [&](int r, const V3 &s, const V3(&nb)[4], const V3(&n2)[4]) {
            const V3 d = llg_rhs_vals<J2, true, DAMP, UNIT>(s, nb, n2, a);
            const V3 ac = pload(mine(accs, r));
            const double o0 = da(ac.x, div6(dm(d.x, a.dt)));
            const double o1 = da(ac.y, div6(dm(d.y, a.dt)));
            const double o2 = da(ac.z, div6(dm(d.z, a.dt)));
            const double nrm = __dsqrt_rn(da(da(dm(o0, o0), dm(o1, o1)), dm(o2, o2)));
            const V3 v{dq(dm(a.spin_len, o0), nrm), dq(dm(a.spin_len, o1), nrm),
                       dq(dm(a.spin_len, o2), nrm)};
            pstore(yn + r * STATE_ROW, v);
            put(0, r, v);
        });
        barrier();
    }

    // backward; buffer 0 holds the state the step starts from
    for (int j = q.len; j >= 1; --j) {
        const int n = q.base + j;
        double *const y = state(j - 1);
        stages(y, q.len == 1, TT{});
        const bool eval = n % q.stride == 0 && n / q.stride <= q.E;
        const double2 cf = eval ? q.coef[n / q.stride - 1] : make_double2(0.0, 0.0);
        double part[NPAR];
        auto begin = [&] {
#pragma unroll
            for (int p = 0; p < NPAR; ++p) part[p] = 0.0;
        };
        auto end = [&] {
#pragma unroll
            for (int p = 0; p < NPAR; ++p) psum[p * THREADS + tid] += part[p];
            barrier();
        };
        // the product at state s with its neighbour sums: P to buffer b, loc kept
        auto product = [&](int r, const V3 &s, const V3 &nn, const V3 &nnn, const V3 &m, int b) {
            V3 P, l;
            vjp_vals(a, s, nn, nnn, m, P, l, part);
            pstore(mine(accs, r), l);
            put(b, r, P);
        };
        begin();
        walk(1, TT{}, [&](int r, const V3 &s, const V3(&nb)[4], const V3(&n2)[4]) {
            const long i = site0 + (long)r * N;
            const V3 d = llg_rhs_vals<J2, true, DAMP, UNIT>(s, nb, n2, a);
            const V3 ac = pload(mine(accs, r));
            const V3 v{da(ac.x, div6(dm(d.x, a.dt))), da(ac.y, div6(dm(d.y, a.dt))),
                       da(ac.z, div6(dm(d.z, a.dt)))};
            double *w = ws + r * ROW;
            V3 lam = (q.newest && j == q.len) ? v3(0.0, 0.0, 0.0) : pload(w + LAM * VEC);
            if (eval) {  // lam += Re(coef u_i (G - Z))
                const double2 u = __ldg(q.u + i);
                const double wr = cf.x * u.x - cf.y * u.y, wi = cf.x * u.y + cf.y * u.x;
                lam.x += wr * gz[0].x - wi * gz[0].y;
                lam.y += wr * gz[1].x - wi * gz[1].y;
                lam.z += wr * gz[2].x - wi * gz[2].y;
            }
            const double rn = sqrt(vdot(v, v));
            const V3 vh = vmul(1.0 / rn, v);
            const V3 lv = vmul(a.spin_len / rn, vsub(lam, vmul(vdot(vh, lam), vh)));
            pstore(w + LAMV * VEC, lv);
            pstore(mine(lamy, r), lv);
            product(r, s, sum4(nb), sum4(n2), vmul(a.dt / 6.0, lv), 0);
        });
        end();
        // lam_s = loc + the neighbours' P
        auto gather = [&](int r, const V3(&nb)[4], const V3(&n2)[4]) {
            V3 s = vadd(pload(mine(accs, r)), vmul(a.J1, sum4(nb)));
            if (J2) s = vadd(s, vmul(a.J2, sum4(n2)));
            return s;
        };
#pragma unroll 1
        for (int st = 3; st >= 1; --st) {
            const int b = (st + 1) & 1;  // P of stage st + 1
            const double cv = st == 1 ? 1.0 / 6.0 : 1.0 / 3.0, cs = st == 3 ? 1.0 : 0.5;
            begin();
            walk(b, JJ{}, [&](int r, const V3 &, const V3(&nb)[4], const V3(&n2)[4]) {
                const double *w = ws + r * ROW;
                const V3 s = pload(st == 1 ? y + r * STATE_ROW : w + (S2 + st - 2) * VEC);
                const V3 nn = pload(w + (NN1 + st - 1) * VEC), nnn = pload(w + (NNN1 + st - 1) * VEC);
                const V3 lv = pload(w + LAMV * VEC);
                const V3 ls = gather(r, nb, n2);
                double *ly = mine(lamy, r);
                pstore(ly, vadd(pload(ly), ls));
                product(r, s, nn, nnn, vmul(a.dt, vadd(vmul(cv, lv), vmul(cs, ls))), b ^ 1);
            });
            end();
        }
        // stage 1's P (buffer 1): lam of the step before; its state to buffer 0
        const double *ynext = j > 1 ? state(j - 2) : nullptr;
        walk(1, JJ{}, [&](int r, const V3 &, const V3(&nb)[4], const V3(&n2)[4]) {
            pstore(ws + r * ROW + LAM * VEC, vadd(pload(mine(lamy, r)), gather(r, nb, n2)));
            if (ynext) put(0, r, pload(ynext + r * STATE_ROW));
        });
        barrier();  // also: no CTA leaves while another may store into its halo rows
    }
    // derivative sums of the block, a tree of fixed order
    for (int w = THREADS / 2; w > 0; w >>= 1) {
        if (tid < w)
#pragma unroll
            for (int p = 0; p < NPAR; ++p) psum[p * THREADS + tid] += psum[p * THREADS + tid + w];
        __syncthreads();
    }
    if (tid < NPAR) q.bacc[(long)blockIdx.x * NPAR + tid] += psum[tid * THREADS];
}

size_t smem_bytes(int rows) {
    return ((size_t)2 * (rows + 2) * RS + (NPAR + 6 * RP) * THREADS) * sizeof(double);
}

// 1, 2 or 4 CTAs per replica (a CTA an SM; clusters of 4 find room on 132 of the
// 148 SMs), whichever is done first: a round of CTAs with n sites each took about
// 8 + 0.019 n us a step, 13 + 0.017 n where a cluster has to synchronise.  Measured
// with 1 / 2 / 4 (up to 33 replicas fit one round of 4, 74 one of 2):
//   16x16x16 10.2 / 14.1 / 13.7   20x20x16 15.4 / 15.6 / 14.6   24x24x37 19.4 / 17.1 / 29.2
//   32x32x16 24.6 / 19.2 / 16.1   32x32x80 24.8 / 37.3 / 45.9   48x48x33  -   / 32.3 / 23.4
//   48x48x74  -   / 33.1 / 67.6   64x64x33  -   / 47.8 / 29.6   64x64x90  -   / 95.3 / 86.4
bool geometry(const LLGArgs &a, int &S, int &rows, int &groups, int &rp) {
    const int N = a.N;
    if (N > W || N < MIN_SIDE) return false;
    groups = THREADS / N;
    double best = 0.0;
    S = 0;
    for (int s = 1; s <= 4; s *= 2) {
        const int rw = (N + s - 1) / s, r = (rw + groups - 1) / groups;
        if (r > RP || smem_bytes(rw) > 227 * 1024) continue;
        const long slots = std::max(1L, s == 4 ? a.sms * 132L / 148 : (long)a.sms);
        const long rounds = ((long)a.nfile * s + slots - 1) / slots;
        const double cost = rounds * (s == 1 ? 8.0 + 0.019 * rw * N : 13.0 + 0.017 * rw * N);
        if (S == 0 || cost < best) S = s, rows = rw, rp = r, best = cost;
    }
    return S > 0;
}

template <bool J2, bool DAMP, bool UNIT>
cudaError_t launch_t(const LLGArgs &a, int S, int rows, int groups, int rp, const AdjSegment &q,
                     cudaStream_t st) {
    auto k = adjoint_segment_kernel<J2, DAMP, UNIT>;
    const size_t smem = smem_bytes(rows);
    cudaError_t e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return e;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)((long)a.nfile * S));
    cfg.blockDim = dim3(THREADS);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = (unsigned)S;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, k, a, S, rows, groups, rp, q);
}

}  // namespace

int adjoint_resident_blocks(const LLGArgs &a) {
    int S, rows, groups, rp;
    return geometry(a, S, rows, groups, rp) ? a.nfile * S : 0;
}

size_t adjoint_resident_bytes(const LLGArgs &a, int states, size_t *work_bytes) {
    int S, rows, groups, rp;
    if (!geometry(a, S, rows, groups, rp)) return 0;
    const size_t cta_rows = (size_t)a.nfile * S * rp;
    *work_bytes = cta_rows * ROW * sizeof(double);
    return *work_bytes + cta_rows * STATE_ROW * sizeof(double) * states;
}

cudaError_t launch_adjoint_segment(const LLGArgs &a, const AdjSegment &q, cudaStream_t st) {
    int S, rows, groups, rp;
    if (!geometry(a, S, rows, groups, rp) || q.len < 1) return cudaErrorInvalidValue;
    const bool unit = a.J1 == 1.0 || a.J1 == -1.0;
    switch ((a.use_j2 ? 4 : 0) | (a.use_damp ? 2 : 0) | (unit ? 1 : 0)) {
        case 0: return launch_t<false, false, false>(a, S, rows, groups, rp, q, st);
        case 1: return launch_t<false, false, true>(a, S, rows, groups, rp, q, st);
        case 2: return launch_t<false, true, false>(a, S, rows, groups, rp, q, st);
        case 3: return launch_t<false, true, true>(a, S, rows, groups, rp, q, st);
        case 4: return launch_t<true, false, false>(a, S, rows, groups, rp, q, st);
        case 5: return launch_t<true, false, true>(a, S, rows, groups, rp, q, st);
        case 6: return launch_t<true, true, false>(a, S, rows, groups, rp, q, st);
        default: return launch_t<true, true, true>(a, S, rows, groups, rp, q, st);
    }
}

}  // namespace asd
