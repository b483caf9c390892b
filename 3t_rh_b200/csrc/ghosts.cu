// Ghost-node update of one RK stage (ghost.rs:199-268 update_values_parallel,
// bc1.rs:609-928 set_ghost_point_value with precomputed GhostBC data), in one
// launch. Cheap ghosts (ReflectiveWall, ZerothOrder, Periodic, Constant,
// TimeDependent) take six threads each at its start.
// k_ghosts, heavy ghosts on persistent warps, two ghosts at a time per warp, one
// on each half-warp. A ghost's tables (the rows of S_r and w, d; 9.7 KB)
// arrive in shared memory by a bulk copy (cp.async.bulk, completion on an
// mbarrier). One table buffer per half-warp: once step 3 has read the rows
// (and d is in registers) the next pair's copies are issued into the same
// buffers, so the table stream overlaps steps 4-6.
// Per ghost:
//   1. L, R and lambda at the nearest fluid node, rotated to the (normal,
//      tangential) frame (bc1.rs:294-312): for the warp's next 30 ghosts at
//      once, one per lane (on the lanes of one ghost its six rows, three kinds
//      of code, took a quarter of the pair's time), staged in the table buffers
//      and kept in global scratch until the ghost's turn; they and the E_r
//      stencil states (E_0..E_4, 55 nodes, four per lane) are loaded while the
//      pair before is processed, the fetches spread over the steps so that none
//      waits on another;
//   2. lanes spread over the 55 stencil nodes: rotate the momentum and
//      project on the six characteristic fields (bc1.rs:209-219);
//   3. the 70 dot products with the stencil data, all six fields at once, four
//      rows of one order per lane (ghost_rows.cuh): the 55 rows of S_0..S_4,
//      each then stored over the data as its beta term d_c,a (S_r d_c)_a, and
//      the 15 rows w_{r,k}, V^(k)_{c,r} = w_{r,k} . d_c (bc1.rs:221-244);
//      orders 1 and 0 by (row, field);
//   4. lanes (c, r): beta_{c,r} = the sum of its row terms in order and
//      alpha = d_r / (eps + beta)^q;
//   5. lanes (c, r): the weight alpha_r / sum(alpha); lanes (k, c): V^(k)_c =
//      the weighted sum of V_r (bc1.rs:247-252);
//   6. FarField rows, R products, the Wall's two 6x6 LU solves (a column per
//      lane), Outflow's LODI row and the Taylor sum on lanes (bc1.rs:691-923).
// The per-k loop of the reference (bc1.rs:673-675) recomputes steps 2-4
// unchanged; they are done once. Every sum keeps the reference's order, so
// the no-contraction build reproduces the reference's values.
#include <algorithm>

#include "common.cuh"
#include "kernels.cuh"
#include "physics.cuh"
#include "ghost_rows.cuh"
#include "mbar.cuh"
#include "per_device.h"

namespace rh3t {

#ifdef RH3T_EXACT
constexpr bool kExactG = true;
#else
constexpr bool kExactG = false;
#endif

constexpr int GH_WARPS = 8; // one block per SM

struct GhostSlot { // one ghost: half a warp
    double rec[GH_COPY];   // the tables (the next ones are copied in during step 4)
    double LR[GH_LR];      // this ghost's L, R, lambda
    double D[56][6];       // characteristic data d_c at stencil node a, row d_row(a); then d_c,a (S_r d_c)_a; then u
    double alpha[6][5];    // alpha, then the weights
    double V[6][15];       // [c][r (r + 1) / 2 + k], k <= r
    double v[5][6];        // V^(k)_c
    double ui[6], vinf[6]; // FarField state, and L of it
    GhostRec cur;          // this ghost's GhostRec (copied in while the pair before it ran)
};
struct GhostWarp {
    GhostSlot g[2];
    unsigned long long bar, pad;
};
static_assert(sizeof(GhostSlot) % 16 == 0 && sizeof(GhostWarp) % 16 == 0, "tables stay 16-byte aligned");
static_assert(GH_COPY * 8 % 16 == 0 && GH_REC * 8 % 16 == 0 && 2 * GR_CHUNKS == GH_D, "record layout");
constexpr int GH_SMEM = GH_WARPS * (int)sizeof(GhostWarp);
static_assert(GH_SMEM <= 232448, "one block per SM");
constexpr int GH_LR_R = 36, GH_LR_LAM = 72; // of a slot's LR
constexpr int CHUNK = 15; // pairs whose L, R and lambda are formed together: 78 x 15 values in a slot's rec
static_assert(78 * CHUNK <= GH_COPY, "a chunk's L, R, lambda fit in the table buffer");

// ---------------------------------------------------------------- bulk copy
// one thread: expect the tables of two ghosts on bar, then copy them global ->
// shared (16-byte aligned addresses, sizes a multiple of 16). The buffers are
// reused: the proxy fence orders the warp's earlier reads of them (generic
// proxy, made visible to this thread by the __syncwarp before every call)
// before the copies' writes (async proxy).
__device__ __forceinline__ void bulk_copy(void* dst, const void* src, uint32_t bytes, unsigned long long* bar) {
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
                     smem_u32(dst)),
                 "l"(src), "r"(bytes), "r"(smem_u32(bar))
                 : "memory");
}
__device__ __forceinline__ void load_tables(GhostWarp& W, const double* __restrict__ hrec, int heavy0, int heavy1) {
    constexpr uint32_t bytes = GH_COPY * 8;
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(&W.bar)), "r"(2 * bytes)
                 : "memory");
    bulk_copy(W.g[0].rec, hrec + (size_t)heavy0 * GH_REC, bytes, &W.bar);
    bulk_copy(W.g[1].rec, hrec + (size_t)heavy1 * GH_REC, bytes, &W.bar);
}

// a / b for operands of any sign, correctly rounded (divrn.cuh: |b| > 0 there)
__device__ __forceinline__ double quot_any(double a, double b) {
    const double m = fabs(b);
    if (den_near(m) && num_near(a)) return div_near(b < 0.0 ? -a : a, recip_near(m));
    return div_ieee(a, b);
}

// bc1.rs:467-469 solve6 with LAPACK getrf/getrs semantics (first-maximum
// pivots, multipliers by the pivot's reciprocal), on one half-warp: lane k < 6
// holds column k of A in a, lane 6 the right-hand side, which is eliminated with
// the columns (the same products in the same order as a forward substitution
// after the factorisation). The solution is left in lane 6's a; returns false on
// every lane if a pivot is zero. m: the half's lanes, h: its first lane
__device__ __forceinline__ bool solve6(double a[6], int l, unsigned m, int h) {
#pragma unroll
    for (int j = 0; j < 6; ++j) {
        int p = j;
        double mx = fabs(a[j]), pv = a[j];
#pragma unroll
        for (int i = j + 1; i < 6; ++i)
            if (fabs(a[i]) > mx) { mx = fabs(a[i]); pv = a[i]; p = i; }
        p = __shfl_sync(m, p, h + j);
        pv = __shfl_sync(m, pv, h + j);
        if (pv == 0.0) return false;
#pragma unroll
        for (int i = j + 1; i < 6; ++i)
            if (p == i) { const double t = a[j]; a[j] = a[i]; a[i] = t; }
        if (j == 5) break;
        const double rcp = quot_any(1.0, pv);
#pragma unroll
        for (int i = j + 1; i < 6; ++i) {
            const double f = __shfl_sync(m, a[i], h + j) * rcp;
            if (l == j) a[i] = f;
            else if (l > j) a[i] -= f * a[j];
        }
    }
#pragma unroll
    for (int k = 5; k >= 0; --k) {
        const double d = __shfl_sync(m, a[k], h + k);
        const double x = quot_any(a[k], d);
#pragma unroll
        for (int i = 0; i < k; ++i) {
            const double f = __shfl_sync(m, a[i], h + k);
            if (l == 6) a[i] -= x * f;
        }
        if (l == 6) a[k] = x;
    }
    return true;
}

// Wall (bc1.rs:691-756): u_0 and u_1 from the two ILW systems; Outflow
// (bc1.rs:760-828): u_1 with the LODI row. On the half-warp (m, h as above) of
// a ghost whose u_k = R v_k are in u. Returns false when an ILW system is
// singular. (On one lane, with the systems in local memory, it took most of a
// Wall ghost's time: 47 us for the 1,344 Wall ghosts of a double Mach stage.)
__device__ __noinline__ bool wall_outflow_rows(const Inst& I, const GhostRec& Rg, const double* LR,
                                               const double (*v)[6], double (*u)[6], int l, unsigned m, int h) {
    const DevParams& P = I.P;
    const double ge = P.gamma_e - 1.0, gi = P.gamma_i - 1.0, gr = P.gamma_r - 1.0;
    if (Rg.kind == BC_WALL) {
        const double gt = gi + ge + gr;
        double a[6];
        a[0] = l == 1 ? 1.0 : 0.0;
#pragma unroll
        for (int i = 1; i < 6; ++i) a[i] = l < 6 ? LR[6 * i + l] : (l == 6 ? v[0][i] : 0.0);
        if (!solve6(a, l, m, h)) return false;
        const double u1 = __shfl_sync(m, a[0], h + 6), u3 = __shfl_sync(m, a[2], h + 6);
        if (l == 6)
#pragma unroll
            for (int k = 0; k < 6; ++k) u[0][k] = a[k];
        const double q0 = -gt * sqd(u3) / (6.0 * sqd(u1)), q2 = gt * u3 / (6.0 * u1);
        a[0] = l == 0 ? q0 : (l == 2 ? q2 : (l == 3 ? -ge : (l == 4 ? -gi : (l == 5 ? -gr : 0.0))));
#pragma unroll
        for (int i = 1; i < 6; ++i) a[i] = l < 6 ? LR[6 * i + l] : (l == 6 ? v[1][i] : 0.0);
        if (!solve6(a, l, m, h)) return false;
        if (l == 6)
#pragma unroll
            for (int k = 0; k < 6; ++k) u[1][k] = a[k];
        return true;
    }
    // Outflow
    const DevBC& bc = I.bcs[Rg.bc];
    const double rho0 = u[0][0];
    const double un0 = u[0][1] / rho0, ut0 = u[0][2] / rho0;
    const double w2 = un0 * un0 + ut0 * ut0;
    const double ee1 = u[0][3] / rho0 - w2 / 6.0, ei1 = u[0][4] / rho0 - w2 / 6.0, er1 = u[0][5] / rho0 - w2 / 6.0;
    const double p0 = rho0 * (ge * ee1 + gi * ei1 + gr * er1);
    const double a2 = P.gamma_e * ge * ee1 + P.gamma_i * gi * ei1 + P.gamma_r * gr * er1;
    const double a = sqrt(a2);
    const double lambda1 = un0 - a;
    double r0 = v[1][0];
    if (lambda1 < 0.0) {
        const double m_local = fabs(un0 / a);
        const double l1 = bc.sigma * (1.0 - sqd(m_local)) * a / bc.l_domain * (p0 - bc.p_inf);
        r0 = l1 / lambda1;
    }
    if (l < 6) {
        const double* Rc = LR + GH_LR_R;
        double acc = 0.0;
#pragma unroll
        for (int j = 0; j < 6; ++j) acc += Rc[6 * j + l] * (j == 0 ? r0 : v[1][j]);
        u[1][l] = acc;
    }
    return true;
}

// ---------------------------------------------------------------- cheap ghosts
__device__ __forceinline__ void cheap_ghost(const Inst& I, const GhostRec& Rg, int c, int stage) {
    double* buf = const_cast<double*>(stage_src(I, stage));
    const long long plane = I.plane;
    const DevBC& bc = I.bcs[Rg.bc];
    double val;
    if (Rg.kind == BC_CONSTANT) {
        val = bc.state[c]; // bc1.rs:631-633
    } else if (Rg.kind == BC_TIME_DEPENDENT) {
        const double xs = bc.td_x0 + bc.td_speed * I.sc->t_stage[stage]; // bc1.rs:634-636, init.rs:61-65
        val = Rg.p0x <= xs ? bc.td_left[c] : bc.td_right[c];
    } else if (Rg.kind == BC_REFLECTIVE_WALL) {
        double s[6]; // bc1.rs:930-1037
        load6(buf, plane, Rg.src, s);
        const double mom_n = s[1] * Rg.nx + s[2] * Rg.ny;
        val = c == 1 ? s[1] - 2.0 * mom_n * Rg.nx : (c == 2 ? s[2] - 2.0 * mom_n * Rg.ny : s[c]);
    } else {
        val = buf[c * plane + Rg.src]; // ZerothOrder bc1.rs:471-545, Periodic bc1.rs:547-607
    }
    if (!isfinite(val)) report(I, 1 + 2 * stage, 2, (unsigned)Rg.gid);
    buf[c * plane + Rg.node] = val;
}

// ---------------------------------------------------------------- heavy ghosts
// L, R and lambda of a Roe state: LR[6c + k] = L[c][k], LR[36 + 6c + i] =
// R[i][c], LR[72 + c] = lambda_c, value e at LR[e * CHUNK]
__device__ __forceinline__ void store_lr(double* LR, int row, const double Lr[6], const double Rr[6], const Roe& q) {
#pragma unroll
    for (int k = 0; k < 6; ++k) {
        LR[(6 * row + k) * CHUNK] = Lr[k];
        LR[(GH_LR_R + 6 * k + row) * CHUNK] = Rr[k];
    }
    LR[(GH_LR_LAM + row) * CHUNK] = row == 0 ? q.u - q.cs : (row == 5 ? q.u + q.cs : q.u);
}
// states outside the branch-free quotients' range (divrn.cuh)
static __device__ __noinline__ void lr_each(const Roe* q, const DevParams& P, double* LR) {
#pragma unroll 1
    for (int row = 0; row < 6; ++row) {
        double Lr[6], Rr[6];
        l_row<0>(row, *q, P, Lr);
        r_row<0, false>(row, *q, RecipN{1.0, 1.0, 0.0}, P, Rr);
        store_lr(LR, row, Lr, Rr, *q);
    }
}

// A double whose quotients take the branch-free form: the FMA build forms the
// rows by the templates of physics.cuh over it, which contract as over double
struct NearD {
    double v;
    __device__ __forceinline__ NearD() {}
    __device__ __forceinline__ NearD(double x) : v(x) {}
};
__device__ __forceinline__ NearD operator-(NearD a) { return -a.v; }
__device__ __forceinline__ NearD operator+(NearD a, NearD b) { return a.v + b.v; }
__device__ __forceinline__ NearD operator-(NearD a, NearD b) { return a.v - b.v; }
__device__ __forceinline__ NearD operator*(NearD a, NearD b) { return a.v * b.v; }
__device__ __forceinline__ NearD operator/(NearD a, NearD b) { return div_near(a.v, recip_near(b.v)); }
__device__ __forceinline__ NearD quot3(NearD x) { return div3_near(x.v); }
__device__ __forceinline__ NearD quot6(NearD x) { return div6_near(x.v); }
// the entries of L with a tiny velocity in the numerator
static __device__ __noinline__ void lr_velocity(const Roe* q, const DevParams& P, double* LR) {
#pragma unroll 1
    for (int row = 0; row < 6; ++row) {
        if (row == 4) continue;
        const LVel l = l_row_velocity<0>(row, *q, P, false);
        if (row == 0 || row == 5) LR[6 * row * CHUNK] = l.l0;
        LR[(6 * row + 1) * CHUNK] = l.l1;
        LR[(6 * row + 2) * CHUNK] = l.l2;
    }
}

// L, R and lambda at the nearest fluid node of heavy ghost Rg in its (normal,
// tangential) frame (bc1.rs:294-312)
__device__ __forceinline__ void local_lr(const Inst& I, const GhostRec& Rg, int stage, double* LR) {
    const DevParams& P = I.P;
    double s[6];
    load6(stage_src(I, stage), I.plane, Rg.src, s);
    const double mom_n = s[1] * Rg.nx + s[2] * Rg.ny;
    const double mom_t = -s[1] * Rg.ny + s[2] * Rg.nx;
    const double q6[6] = {s[0], mom_n, mom_t, s[3], s[4], s[5]};
    const Prim d1 = prim_from_state(q6, P);
    const double rt = sqrt(q6[0]);
    const Roe q = roe_average_sqrt(rt, d1, rt, d1, P);
    const double gi = P.gamma_i - 1.0, ge = P.gamma_e - 1.0, gr = P.gamma_r - 1.0;
    const double gt = gi + ge + gr;
    RoeDivN rd;
    const int mode = near_gammas(P) && den_mid_near(gt) ? near_face(q, gt, rd) : FACE_GENERAL;
    if (mode > 0) {
        if (!kExactG) {
            const RoeT<NearD> n = {q.u, q.v, q.w2, q.ee, q.ei, q.er, q.cs2, q.cs, q.he, q.hi, q.hr, q.b, q.den};
#pragma unroll
            for (int row = 0; row < 6; ++row) {
                NearD Lr[6], Rc[6], lam;
                l_row<0>(row, n, P, Lr);
                r_col<0>(row, n, P, Rc, lam);
#pragma unroll
                for (int k = 0; k < 6; ++k) {
                    LR[(6 * row + k) * CHUNK] = Lr[k].v;
                    LR[(GH_LR_R + 6 * row + k) * CHUNK] = Rc[k].v;
                }
                LR[(GH_LR_LAM + row) * CHUNK] = lam.v;
            }
            if (mode == FACE_VELOCITY) {
                const Roe t = q;
                lr_velocity(&t, P, LR);
            }
            return;
        }
        rd.scale();
        const RecipN rgt = recip_near(gt);
#pragma unroll
        for (int row = 0; row < 6; ++row) {
            double Lr[6], Rr[6];
            const double gl = row == 1 ? ge : (row == 2 ? gi : gr); // of an energy row of L (1-3)
            const double gk = row == 3 ? ge : (row == 4 ? gi : gr); // of an energy row of R (3-5)
            l_row<0>(row, q, rd, row >= 1 && row <= 3 ? div_near(gl, rgt) : 0.0, P, Lr);
            r_row<0, true>(row, q, row >= 3 ? recip_near(6.0 * gk) : rgt, P, Rr);
            store_lr(LR, row, Lr, Rr, q);
        }
        if (mode == FACE_VELOCITY) {
            const Roe t = q;
            lr_velocity(&t, P, LR);
        }
    } else {
        const Roe t = q;
        lr_each(&t, P, LR);
    }
}

// x + y . (d of one stencil node): one term of four rows for all six fields
__device__ __forceinline__ void four_rows(double acc[4][6], const double2 x01, const double2 x23, const double* D) {
    double d[6];
    load_d6(D, d);
    const double x[4] = {x01.x, x01.y, x23.x, x23.y};
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int c = 0; c < 6; ++c) acc[i][c] += x[i] * d[c];
}

// a / b: IEEE quotients of positive operands, branch-free where they are in range
__device__ __forceinline__ double quot_pos(double a, double b) {
    if (a > 0.0 && num_near(a) && den_near(b)) return div_once(a, b);
    return div_ieee(a, b);
}

// alpha = d_r / x^q, x = eps + beta (bc1.rs:241)
__device__ __forceinline__ double alpha_of(double dr, double x, double weno_q) {
    double xq;
    if (!kExactG && weno_q == 10.0) { // four products (within a few ulp) in the FMA build
        const double x2 = x * x, x4 = x2 * x2, x8 = x4 * x4;
        xq = x8 * x2;
    } else {
        xq = pow_q(x, weno_q); // correctly rounded, as the reference's powf
    }
    return quot_pos(dr, xq);
}

// the 30 (c, r) tasks of steps 4 and 5 on 16 lanes in two rounds, the long
// sums (orders 4 and 3) in the first: a hex digit per lane; lanes 14 and 15
// have one task
constexpr unsigned long long kTaskC[2] = {0x3210543210543210ull, 0x0054321054321054ull};
constexpr unsigned long long kTaskR[2] = {0x2222333333444444ull, 0x0000000011111122ull};
__device__ __forceinline__ int task_digit(unsigned long long k, int l) { return (int)(k >> (4 * l)) & 15; }

// What a launch does: all of the update in one, unless a table makes the order of
// its parts matter (launch_ghosts)
enum { GH_PART_ALL = 0, GH_PART_LR = 1, GH_PART_REST = 2 };

// Warps take the heavy ghosts in turn, two at a time (half-warps 0 and 1; an
// odd last ghost runs on both halves and is written by the first). What the
// next pair needs is fetched in four places, so that no load waits on the one
// before it: its GhostRecs (slot, instance) at the top, its stencil
// indices after step 3, its stencil states, L, R, lambda and error flags after
// step 4, its tables once step 3 has read this pair's.
//
// Bound by latency and by the L1 / shared-memory data pipe (55% busy; FP64 pipe
// 40%). Four rows a lane halve the loads of the data against two rows a lane and
// one ghost a warp, two ghosts a warp give every serial step (4-6) two chains
// to interleave, and nothing on a pair's path waits for a global load. 24 batch
// instances (84,000 ghosts), a stage: 348 us against 425 us for a preparation
// kernel and one ghost a warp on 12 warps a SM (FMA build 293 us against 426);
// 1024 x 8 planar shock, where one pass is all latency: 18 us against 34 us.
// Tables read from L2 by the lanes instead of bulk copies: 1.32 ms a step of the
// 24 instances against 1.23 ms at that point, with 12 warps (168 registers,
// spills) 1.73 ms; stencil indices fetched before step 3: 1.15 against 1.06 ms.
__global__ void __launch_bounds__(GH_WARPS * 32, 1) k_ghosts(const Inst* __restrict__ insts,
                                                             const GhostRec* __restrict__ heavy, int nh,
                                                             const GhostRec* __restrict__ cheap, int nc,
                                                             const double* __restrict__ hrec, double* lrbuf, int stage,
                                                             int part) {
    extern __shared__ __align__(128) unsigned char gh_smem[];
    const int lane = threadIdx.x & 31, half = lane >> 4, l = lane & 15, warp = threadIdx.x >> 5;
    GhostWarp& W = reinterpret_cast<GhostWarp*>(gh_smem)[warp];
    GhostSlot& G = W.g[half];
    const int npair = (nh + 1) >> 1, stride = gridDim.x * GH_WARPS;
    // cheap ghosts, six threads each, on the warps that come last in the order of the pairs first
    for (int t = ((GH_WARPS - 1 - warp) * gridDim.x + blockIdx.x) * 32 + lane; t < 6 * nc;
         t += gridDim.x * GH_WARPS * 32) {
        const int c = t % 6;
        const GhostRec Rg = cheap[t / 6];
        const Inst& I = insts[Rg.inst];
        if (!has_error(I)) cheap_ghost(I, Rg, c, stage);
    }
    const int first = blockIdx.x + gridDim.x * warp; // pairs spread over the SMs first
    if (first >= npair) return;                      // warp-uniform
    // this lane's four rows of step 3
    const int ord = l < 7 || l == 15 ? 4 : (l < 12 ? 3 : 2);
    const int quad = l < 7 ? l : (l == 15 ? 7 : (l < 12 ? l - 7 : l - 12));
    const int ord_m = (ord + 1) * (ord + 1);
    // tasks (c, r) of steps 4 and 5
    const int c0 = task_digit(kTaskC[0], l), r0 = task_digit(kTaskR[0], l);
    const int c1 = task_digit(kTaskC[1], l), r1 = task_digit(kTaskR[1], l);
    // task (row, three fields) of orders 1 (rows 0-3 of S, 4-5 w) and 0 (row 6 S, 7 w)
    const int lrow = l >> 1, lc = 3 * (l & 1);
    constexpr int kRecWords = (int)(sizeof(GhostRec) / 8);
    static_assert(sizeof(GhostRec) % 8 == 0 && kRecWords <= 16, "GhostRec copied as words by half a warp");

    if (lane == 0) {
        mbar_init(&W.bar, 1);
        mbar_fence_init();
    }
    // per pair, loaded while the pair before it runs
    double s[4][6], lr[5], ui_l, eps, weno_q;
    double* out_p; // component l (< 6) of the ghost node
    bool skip, n_skip = false;
    int it = 0;
    for (int i0 = first; i0 < npair; i0 += CHUNK * stride) {
    // ---- 1. L, R, lambda of the chunk's ghosts, one per lane, staged in the
    // table buffer and stored by half-warps
    if (part != GH_PART_REST) {
        if (l < CHUNK && i0 + l * stride < npair) {
            const GhostRec Rg = heavy[min(2 * (i0 + l * stride) + half, nh - 1)];
            local_lr(insts[Rg.inst], Rg, stage, G.rec + l);
        }
        __syncwarp();
        for (int t = 0; t < CHUNK && i0 + t * stride < npair; ++t) {
            double* o = lrbuf + (size_t)min(2 * (i0 + t * stride) + half, nh - 1) * GH_LR;
#pragma unroll
            for (int j = 0; j < 5; ++j)
                if (l + 16 * j < 78) o[l + 16 * j] = G.rec[(l + 16 * j) * CHUNK + t];
        }
        __syncwarp();
        if (part == GH_PART_LR) continue;
    }
    // the chunk's first pair
    {
        const GhostRec& R0 = heavy[min(2 * i0 + half, nh - 1)];
        const int slot = __ldg(&R0.heavy);
        const int slot1 = __shfl_sync(0xffffffffu, slot, 16);
        if (lane == 0) load_tables(W, hrec, slot, slot1);
        const Inst& I = insts[__ldg(&R0.inst)];
        const int32_t* st = reinterpret_cast<const int32_t*>(hrec + (size_t)slot * GH_REC + GH_ST);
        const double* buf = stage_src(I, stage);
#pragma unroll
        for (int j = 0; j < 4; ++j)
            if (l + 16 * j < 55) load6(buf, I.plane, __ldg(&st[l + 16 * j]), s[j]);
#pragma unroll
        for (int j = 0; j < 5; ++j) lr[j] = __ldcg(lrbuf + (size_t)min(2 * i0 + half, nh - 1) * GH_LR + l + 16 * j);
        ui_l = l < 6 ? I.bcs[__ldg(&R0.bc)].state[l] : 0.0;
        eps = I.P.eps;
        weno_q = I.P.weno_q;
        out_p = const_cast<double*>(buf) + (l < 6 ? l : 0) * I.plane + __ldg(&R0.node);
        skip = has_error(I);
        if (l < kRecWords)
            reinterpret_cast<unsigned long long*>(&G.cur)[l] =
                __ldg(reinterpret_cast<const unsigned long long*>(&R0) + l);
        __syncwarp();
    }
    for (int t = 0, i = i0; t < CHUNK && i < npair; ++t, ++it, i += stride) {
        const bool more = t + 1 < CHUNK && i + stride < npair; // warp-uniform
        int n_heavy = 0, n_inst = 0, n_bc = 0, n_node = 0;
        unsigned long long nword = 0;
        if (more) {
            const GhostRec* R = heavy + min(2 * (i + stride) + half, nh - 1);
            n_heavy = __ldg(&R->heavy);
            n_inst = __ldg(&R->inst);
            n_bc = __ldg(&R->bc);
            n_node = __ldg(&R->node);
            if (l < kRecWords) nword = __ldg(reinterpret_cast<const unsigned long long*>(R) + l);
        }
#pragma unroll
        for (int j = 0; j < 5; ++j) G.LR[l + 16 * j] = lr[j];
        if (l < 6) G.ui[l] = ui_l;
        const double nx = G.cur.nx, ny = G.cur.ny;
        const int kind = G.cur.kind;
        const Inst& I = insts[G.cur.inst];
        const bool write = !skip && 2 * i + half < nh;
        const double* L = G.LR;
        const double* Rc = G.LR + GH_LR_R;
        const double* lam = G.LR + GH_LR_LAM;
        __syncwarp();
        // ---- 2. characteristic data of the 55 stencil nodes
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const double mn = s[j][1] * nx + s[j][2] * ny, mt = -s[j][1] * ny + s[j][2] * nx;
            s[j][1] = mn;
            s[j][2] = mt;
        }
#pragma unroll
        for (int c = 0; c < 6; c += 2) {
            const double2* q = reinterpret_cast<const double2*>(L + 6 * c);
            const double2 a0 = q[0], a1 = q[1], a2 = q[2], b0 = q[3], b1 = q[4], b2 = q[5];
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                const double* u = s[j];
                const double d0 = a0.x * u[0] + a0.y * u[1] + a1.x * u[2] + a1.y * u[3] + a2.x * u[4] + a2.y * u[5];
                const double d1 = b0.x * u[0] + b0.y * u[1] + b1.x * u[2] + b1.y * u[3] + b2.x * u[4] + b2.y * u[5];
                if (l + 16 * j < 55) *reinterpret_cast<double2*>(&G.D[d_row(l + 16 * j)][c]) = make_double2(d0, d1);
            }
        }
        if (l < 6) { // the FarField state in characteristic variables (bc1.rs:839-846)
            const double uinf[6] = {G.ui[0], G.ui[1] * nx + G.ui[2] * ny, -G.ui[1] * ny + G.ui[2] * nx,
                                    G.ui[3], G.ui[4], G.ui[5]};
            double a = 0.0;
#pragma unroll
            for (int j = 0; j < 6; ++j) a += L[6 * l + j] * uinf[j];
            G.vinf[l] = a;
        }
        const bool ok_copy = __all_sync(0xffffffffu, mbar_wait(&W.bar, (uint32_t)(it & 1)));
        if (!ok_copy) {
            if (l == 0 && write) report(I, 1 + 2 * stage, MBAR_TIMEOUT_CODE, (unsigned)G.cur.gid);
            (void)mbar_wait(&W.bar, (uint32_t)(it & 1)); // (once more: they write this block's shared memory)
            return;
        }
        __syncwarp();
        // ---- 3. the 70 rows: orders 4, 3 and 2
        double acc[4][6];
#pragma unroll
        for (int q = 0; q < 4; ++q)
#pragma unroll
            for (int c = 0; c < 6; ++c) acc[q][c] = 0.0;
        {
            const double2* rows = reinterpret_cast<const double2*>(G.rec);
            const double* D = &G.D[kDOff[ord]][0];
            // (lane 15 has one pair: its second chunk is a neighbour's and goes unused)
#pragma unroll 3
            for (int b = 0; b < 9; ++b) four_rows(acc, rows[31 * b + l], rows[31 * b + 16 + l], D + 6 * b);
            if (ord >= 3) {
                const double2* p = rows + GR_SEG1 + (l == 15 ? 12 : l);
                const double2* p2 = rows + GR_SEG1 + 13 + l;
#pragma unroll
                for (int b = 0; b < 7; ++b) four_rows(acc, p[25 * b], p2[25 * b], D + 54 + 6 * b);
            }
            if (ord == 4) {
                const double2* p = rows + GR_SEG2 + (l == 15 ? 7 : l);
                const double2* p2 = rows + GR_SEG2 + 8 + l;
#pragma unroll 3
                for (int b = 0; b < 9; ++b) four_rows(acc, p[15 * b], p2[15 * b], D + 96 + 6 * b);
            }
        }
        double low[3] = {0.0, 0.0, 0.0};
#pragma unroll
        for (int b = 0; b < 4; ++b) {
            const double* d = &G.D[lrow < 6 ? 1 + b : 0][lc];
            if (lrow < 6 || b == 0)
#pragma unroll
                for (int c = 0; c < 3; ++c)
                    low[c] += G.rec[lrow < 6 ? row_place(1, lrow, b) : 2 * GR_ORDER0 + lrow - 6] * d[c];
        }
        const double dr0 = G.rec[GH_D + r0], dr1 = G.rec[GH_D + r1];
        // the next pair's stencil indices, state buffer, error flag and BC table
        int st[4] = {0, 0, 0, 0};
        if (more) {
            const int32_t* q = reinterpret_cast<const int32_t*>(hrec + (size_t)n_heavy * GH_REC + GH_ST);
#pragma unroll
            for (int j = 0; j < 4; ++j)
                if (l + 16 * j < 55) st[j] = __ldg(&q[l + 16 * j]);
        }
        const Inst& In = insts[n_inst];
        const double* nbuf = stage_src(In, stage);
        const long long nplane = In.plane;
        const DevError* nerr = In.err;
        const DevBC* nbcs = In.bcs;
        const double n_eps = In.P.eps, n_weno_q = In.P.weno_q;
        const int n_heavy1 = __shfl_sync(0xffffffffu, n_heavy, 16);
        __syncwarp();
        // the tables are not read below: bring in the next pair's
        if (lane == 0 && more) load_tables(W, hrec, n_heavy, n_heavy1);
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            const int R = quad_row(ord, quad, q);
            if (R < ord_m) {
                double* Dr = &G.D[kDOff[ord] + R][0];
                double d[6], p[6];
                load_d6(Dr, d);
#pragma unroll
                for (int c = 0; c < 6; ++c) p[c] = d[c] * acc[q][c];
                store_d6(Dr, p);
            } else if (R - ord_m <= ord) {
#pragma unroll
                for (int c = 0; c < 6; ++c) G.V[c][ord * (ord + 1) / 2 + R - ord_m] = acc[q][c];
            }
        }
#pragma unroll
        for (int c = 0; c < 3; ++c) {
            const int row = lrow == 6 ? 0 : 1 + lrow;
            if (lrow < 4 || lrow == 6) G.D[row][lc + c] = G.D[row][lc + c] * low[c];
            else G.V[lc + c][lrow == 7 ? 0 : lrow - 3] = low[c];
        }
        __syncwarp();
        // ---- 4. beta_{c,r} = sum_a d_a (S d)_a in order, alpha = d_r / (eps + beta)^q
        {
            double b0 = 0.0, b1 = 0.0;
            const int m0 = (r0 + 1) * (r0 + 1), m1 = (r1 + 1) * (r1 + 1);
            const double *q0 = &G.D[kDOff[r0]][c0], *q1 = &G.D[kDOff[r1]][c1];
#pragma unroll
            for (int a = 0; a < 9; ++a) {
                b0 += q0[6 * a];
                if (a < m1) b1 += q1[6 * a];
            }
#pragma unroll 8
            for (int a = 9; a < m0; ++a) b0 += q0[6 * a];
            const double al0 = alpha_of(dr0, eps + b0, weno_q), al1 = alpha_of(dr1, eps + b1, weno_q);
            G.alpha[c0][r0] = al0;
            if (l < 14) G.alpha[c1][r1] = al1;
        }
        // the next pair's stencil states, L, R, lambda (used in its step 2), FarField states and error flags
        if (more) {
#pragma unroll
            for (int j = 0; j < 4; ++j)
                if (l + 16 * j < 55) load6(nbuf, nplane, st[j], s[j]);
#pragma unroll
            for (int j = 0; j < 5; ++j)
                lr[j] = __ldcg(lrbuf + (size_t)min(2 * (i + stride) + half, nh - 1) * GH_LR + l + 16 * j);
            if (l < 6) ui_l = nbcs[n_bc].state[l];
            n_skip = nerr->key != ~0ull;
        }
        __syncwarp();
        // ---- 5. nonlinear weights (bc1.rs:247-252); V^(k)_r = 0 for k > r
        {
            auto weight = [&](int c, int r) {
                double asum = 0.0;
#pragma unroll
                for (int q = 0; q < 5; ++q) asum += G.alpha[c][q];
                return quot_pos(G.alpha[c][r], asum);
            };
            const double w0 = weight(c0, r0), w1 = weight(c1, r1);
            __syncwarp();
            G.alpha[c0][r0] = w0;
            if (l < 14) G.alpha[c1][r1] = w1;
        }
        __syncwarp();
#pragma unroll
        for (int j = 0; j < 2; ++j) {
            const int t = l + 16 * j, k = t / 6, c = t - 6 * (t / 6);
            if (t < 30) {
                double res = 0.0;
#pragma unroll
                for (int r = 0; r < 5; ++r) res += G.alpha[c][r] * (k <= r ? G.V[c][r * (r + 1) / 2 + k] : 0.0);
                G.v[k][c] = res;
            }
        }
        __syncwarp();
        // ---- 6. BC rows, R products, Taylor expansion (bc1.rs:690-924)
        double(*u)[6] = reinterpret_cast<double(*)[6]>(&G.D[0][0]); // D is dead here
        const bool far = kind == BC_FAR_FIELD;
        {
            double a[2] = {0.0, 0.0};
#pragma unroll
            for (int m = 0; m < 6; ++m) {
                const bool in = far && lam[m] < 0.0;
                const double vi = G.vinf[m];
#pragma unroll
                for (int j = 0; j < 2; ++j) {
                    const int t = l + 16 * j < 30 ? l + 16 * j : 29, k = t / 6, q = t - 6 * (t / 6);
                    const double x = in ? (k == 0 ? vi : 0.0) : G.v[k][m];
                    a[j] += Rc[6 * m + q] * x;
                }
            }
#pragma unroll
            for (int j = 0; j < 2; ++j) {
                const int t = l + 16 * j;
                if (t < 30) u[t / 6][t - 6 * (t / 6)] = a[j];
            }
        }
        __syncwarp();
        bool ok = true;
        if (!far) ok = wall_outflow_rows(I, G.cur, G.LR, G.v, u, l, 0xffffu << (16 * half), 16 * half);
        __syncwarp();
        double g = 0.0;
        if (l < 6) {
            g = u[0][l];
            double coef = 1.0;
            const double dist = G.cur.dist;
#pragma unroll
            for (int k = 1; k <= 4; ++k) {
                coef *= k == 3 ? div3_rn(dist) : dist / (double)k;
                g = g + coef * u[k][l];
            }
        }
        const double mn = __shfl_sync(0xffffffffu, g, (lane & 16) + 1), mt = __shfl_sync(0xffffffffu, g, (lane & 16) + 2);
        if (write) {
            if (!ok) {
                if (l == 0) report(I, 1 + 2 * stage, 3, (unsigned)G.cur.gid);
            } else if (l < 6) {
                const double out = l == 1 ? mn * nx - mt * ny : (l == 2 ? mn * ny + mt * nx : g);
                *out_p = out;
                if (!isfinite(out)) report(I, 1 + 2 * stage, 2, (unsigned)G.cur.gid);
            }
        }
        __syncwarp();
        if (l < kRecWords) reinterpret_cast<unsigned long long*>(&G.cur)[l] = nword;
        skip = n_skip;
        eps = n_eps;
        weno_q = n_weno_q;
        out_p = const_cast<double*>(nbuf) + (l < 6 ? l : 0) * nplane + n_node;
        __syncwarp();
    }
    }
}

void launch_ghosts(cudaStream_t s, const Inst* insts, const GhostRec* heavy, int nh, const GhostRec* cheap, int nc,
                   const double* hrec, double* lrbuf, int stage, bool ordered) {
    if (nh + nc <= 0) return;
    static OncePerDevice attributes;
    int dev = 0;
    cudaGetDevice(&dev);
    const int sms = multiprocessors(dev);
    attributes(dev, [] {
        return cudaFuncSetAttribute(k_ghosts, cudaFuncAttributeMaxDynamicSharedMemorySize, GH_SMEM) == cudaSuccess;
    });
    auto launch = [&](int h, int c, int part) {
        const int n = std::max((h + 1) / 2, (6 * c + GH_WARPS * 32 - 1) / (GH_WARPS * 32));
        if (n > 0)
            k_ghosts<<<std::min(n, sms), GH_WARPS * 32, GH_SMEM, s>>>(insts, heavy, h, cheap, c, hrec, lrbuf,
                                                                                 stage, part);
    };
    if (!ordered) {
        launch(nh, nc, GH_PART_ALL);
        return;
    }
    launch(nh, 0, GH_PART_LR);
    launch(0, nc, GH_PART_ALL);
    launch(nh, 0, GH_PART_REST);
}

int ghost_launches(int nh, int nc, bool ordered) {
    if (!ordered) return nh + nc > 0 ? 1 : 0;
    return (nh > 0 ? 2 : 0) + (nc > 0 ? 1 : 0);
}

// one warp: the ghost update's bounded wait on a fresh mbarrier whose phase
// completes (arrive: one arrival, no bytes expected) or never does; out[0] =
// 1 when the wait gave up
__global__ void k_wait_check(int arrive, int* out) {
    __shared__ unsigned long long bar;
    const int lane = threadIdx.x & 31;
    if (lane == 0) {
        mbar_init(&bar, 1);
        mbar_fence_init();
        if (arrive)
            mbar_arrive(&bar);
    }
    __syncwarp();
    const bool ok = __all_sync(0xffffffffu, mbar_wait(&bar, 0u));
    if (lane == 0) out[0] = ok ? 0 : 1;
}

} // namespace rh3t

extern "C" int rh3t_wait_check(int32_t device, int32_t arrive, int32_t* timed_out) {
    if (!timed_out) return 7; // RH3T_ERR_INVALID_ARGUMENT
    int ndev = 0;
    if (cudaGetDeviceCount(&ndev) != cudaSuccess || device < 0 || device >= ndev) return 10; // RH3T_ERR_NO_DEVICE
    if (cudaSetDevice(device) != cudaSuccess) return 8;
    int* d = nullptr;
    if (cudaMalloc(&d, sizeof(int)) != cudaSuccess) return 8;
    int h = -1;
    rh3t::k_wait_check<<<1, 32>>>(arrive ? 1 : 0, d);
    cudaError_t e = cudaGetLastError();
    if (e == cudaSuccess) e = cudaMemcpy(&h, d, sizeof(int), cudaMemcpyDeviceToHost);
    cudaFree(d);
    if (e != cudaSuccess) return 8; // RH3T_ERR_CUDA
    *timed_out = h;
    return 0;
}
