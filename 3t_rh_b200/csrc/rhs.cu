// Cell right-hand side fused with the SSP-RK3 stage update (main.rs:251-349):
// flux differences, the non-conservative x/y terms (noncon.rs:288-332), the
// exchange source (source.rs:7-21) and the diffusion differences, then
// u' = a u + b v + c dt rhs with the admissibility check (main.rs:22-33).
//
// A block covers TI x TJ = 256 cells (shape chosen per tile) in three phases:
//   1. the pressures, the transport velocities and the pressure differences
//      2 p_k - p_l - p_m of the nodes within reach of the 9-point non-conservative
//      stencils (the tile plus a 4-node halo, corners excluded) go to shared
//      memory once; the reference's access-table gathers (main.rs:276-277)
//      evaluate them once per use, 17 times per node. A 16 x 16 tile has 512 such
//      nodes, two a thread, and a thread loads both before it uses either;
//   2. the jumps of the three differences at every interface of the tile: the
//      reference forms those at a cell's left and right (lower and upper)
//      interface in each of the two cells they belong to (noncon.rs:259-285). The
//      tile's far edges go one difference to a thread, three to seven warps, instead of
//      three to each thread of the two warps that the others then wait for;
//   3. one cell per thread.
// Bound by latency (24 face fluxes and the stage inputs a cell) and the FP64
// pipe. Forming a jump once, and quotients without a branch each (divrn.cuh), take
// away a third of the FP64 operations and the registers that held two 9-point
// windows, so three blocks fit an SM instead of two. Per stage, 24 batch instances
// 98 us (both windows a cell: 153 us; node loop over the whole halo and far edges on
// two warps: 105 us), the 961 x 3841 half-cylinder 288 us (453 us; 312 us). Two blocks
// of 119 registers were 25% slower, four of 64 (spills) 16%; the face fluxes
// loaded ahead of phases 1 or 2, or prefetched to L2, gave nothing.
//
// mode 0 writes the rhs (6 planes of nx*ny, i*ny+j, instance k at
// rhs_out + 6*cell_off) for l(); mode 1 applies the stage update of `stage`;
// mode 2 does both, the rhs into padded planes at rhs_out + aoff (the
// adjoint's record of the forward stages).
#include <algorithm>

#include "common.cuh"
#include "kernels.cuh"
#include "per_device.h"
#include "physics.cuh"

namespace rh3t {

#ifdef RH3T_EXACT
constexpr bool kExactR = true;
#else
constexpr bool kExactR = false;
#endif
constexpr int RHS_BLOCKS = 3; // per SM: 80 registers
static_assert(RHS_THREADS == 1 << 8, "log2 TI = 8 - lg");

// divisors shared by every cell of an instance: 60 dx, dx, 60 dy, dy
// (noncon.rs:26-44, 315-331), 6 cve, 6 cvi, a_rad (state.rs:245-276)
constexpr int RHS_NR = 7;
__device__ __forceinline__ double rhs_divisor(const Inst& I, int k) {
    switch (k) {
    case 0: return 60.0 * I.dx;
    case 1: return I.dx;
    case 2: return 60.0 * I.dy;
    case 3: return I.dy;
    case 4: return 6.0 * I.P.cve;
    case 5: return 6.0 * I.P.cvi;
    default: return I.P.a_rad;
    }
}
// sR: the two parts of their reciprocals
__device__ __forceinline__ RecipN rhs_recip(const Inst& I, const double* sR, int k) {
    return {rhs_divisor(I, k), sR[k], sR[RHS_NR + k]};
}

// Shared memory of a tile of shape lg: p_e, p_i, p_r, u, v and the three
// differences per node, the jumps per x and y interface, the reciprocals
__host__ __device__ __forceinline__ int rhs_nodes(int lg) { return ((RHS_THREADS >> lg) + 8) * ((1 << lg) + 8); }
__host__ __device__ __forceinline__ int rhs_xfaces(int lg) { return RHS_THREADS + (1 << lg); }
__host__ __device__ __forceinline__ int rhs_yfaces(int lg) { return RHS_THREADS + (RHS_THREADS >> lg); }
int rhs_smem(int lg) { return 8 * (8 * rhs_nodes(lg) + 3 * (rhs_xfaces(lg) + rhs_yfaces(lg)) + 2 * RHS_NR); }

// jumps of the three differences (planes of npt nodes) over the 8 nodes from p
// at stride st (noncon.rs:259-285)
__device__ __forceinline__ void jumps(const double* sN, int npt, int p, int st, double* out, int stride) {
#pragma unroll
    for (int c = 0; c < 3; ++c) {
        double a[8];
#pragma unroll
        for (int q = 0; q < 8; ++q) a[q] = sN[c * npt + p + q * st];
        out[c * stride] = jump8(a);
    }
}

__global__ void __launch_bounds__(RHS_THREADS, RHS_BLOCKS) k_rhs_stage(const Inst* __restrict__ insts, const Tile* __restrict__ tiles,
                                                   int nt, int stage, int mode, double* __restrict__ rhs_out) {
    extern __shared__ double rhs_mem[];
    if (blockIdx.x >= nt) return;
    const Tile t = tiles[blockIdx.x];
    const Inst& I = insts[t.inst];
    if (has_error(I)) return;
    const DevParams& P = I.P;
    const long long plane = I.plane;
    const double* __restrict__ src = stage_src(I, stage);
    const int nx = I.nx, ny = I.ny;
    const int TJ = 1 << t.lg, TI = RHS_THREADS >> t.lg;
    const int HJ = TJ + 8, NPT = (TI + 8) * HJ, nfx = rhs_xfaces(t.lg), nfy = rhs_yfaces(t.lg);
    double* sP = rhs_mem;            // [5][NPT] p_e, p_i, p_r, u, v
    double* sN = sP + 5 * NPT;       // [3][NPT] 2 p_e - p_i - p_r, 2 p_i - p_e - p_r, 2 p_r - p_e - p_i
    double* sX = sN + 3 * NPT;       // [3][nfx] jumps at x interface (a, tj): a * TJ + tj
    double* sY = sX + 3 * nfx;       // [3][nfy] jumps at y interface (ti, b): ti * (TJ + 1) + b
    double* sR = sY + 3 * nfy;       // [2][RHS_NR] reciprocals of the instance's divisors
    if (threadIdx.x < RHS_NR) {
        const RecipN r = recip_near(rhs_divisor(I, threadIdx.x));
        sR[threadIdx.x] = r.y;
        sR[RHS_NR + threadIdx.x] = r.yl;
    }
    // ---- 1. stage node primitives (tile + 4-node cross halo)
    const int mid = (TI + 8) << t.lg, nodes = mid + 8 * TI;
    auto place = [&](int q, int& hi, int& hj) {
        const int r = q - mid;
        hi = r < 0 ? q >> t.lg : 4 + (r >> 3);
        hj = r < 0 ? 4 + (q & (TJ - 1)) : (r & 7) + (r & 4 ? TJ : 0);
        const int i = t.i - 4 + hi, j = t.j0 - 4 + hj;
        return q < nodes && i >= -RH3T_PAD && i < nx + RH3T_PAD && j >= -RH3T_PAD && j < ny + RH3T_PAD;
    };
    auto put = [&](int p, const double* s) {
        const Prim d = kExactR ? prim_from_state(s, P) : fastm::prim(s, P);
        sP[p] = d.pe; sP[NPT + p] = d.pi; sP[2 * NPT + p] = d.pr; sP[3 * NPT + p] = d.u; sP[4 * NPT + p] = d.v;
        sN[p] = 2.0 * d.pe - d.pi - d.pr;
        sN[NPT + p] = 2.0 * d.pi - d.pe - d.pr;
        sN[2 * NPT + p] = 2.0 * d.pr - d.pe - d.pi;
    };
    for (int q = threadIdx.x; q < nodes; q += 2 * RHS_THREADS) {
        int h0, j0, h1, j1;
        const bool a = place(q, h0, j0), b = place(q + RHS_THREADS, h1, j1);
        double s[6], z[6];
        if (a) load6(src, plane, node_of(I, t.i - 4 + h0, t.j0 - 4 + j0), s);
        if (b) load6(src, plane, node_of(I, t.i - 4 + h1, t.j0 - 4 + j1), z);
        if (a) put(h0 * HJ + j0, s);
        if (b) put(h1 * HJ + j1, z);
    }
    __syncthreads();
    const int ti = threadIdx.x >> t.lg, tj = threadIdx.x & (TJ - 1);
    // ---- 2. jumps: this cell's left and lower interfaces, then the tile's far edges
    jumps(sN, NPT, ti * HJ + tj + 4, HJ, sX + threadIdx.x, nfx);
    jumps(sN, NPT, (ti + 4) * HJ + tj, 1, sY + ti * (TJ + 1) + tj, nfy);
    if (threadIdx.x < 3 * (TJ + TI)) {
        const int e = threadIdx.x - 3 * TJ;
        const bool x = e < 0;
        const int lg = x ? t.lg : 8 - t.lg, q = x ? threadIdx.x : e, c = q >> lg, k = q & ((1 << lg) - 1);
        const double* a = sN + c * NPT + (x ? TI * HJ + k + 4 : (k + 4) * HJ + TJ);
        const int st = x ? HJ : 1;
        double w[8];
#pragma unroll
        for (int m = 0; m < 8; ++m) w[m] = a[m * st];
        *(x ? sX + c * nfx + TI * TJ + k : sY + c * nfy + k * (TJ + 1) + TJ) = jump8(w);
    }
    __syncthreads();
    // ---- 3. this thread's cell
    const int i = t.i + ti, j = t.j0 + tj;
    if (i >= nx || j >= ny) return;
    const long long n = node_of(I, i, j);
    if (!I.mask[n]) return;
    const double dx = I.dx, dy = I.dy;
    const long long fpx = (long long)(nx + 1) * ny, fix = (long long)i * ny + j;
    const long long fpy = (long long)nx * (ny + 1), fiy = (long long)i * (ny + 1) + j;
    double rhs[6];
    const double sx = 1.0 / dx, sy = 1.0 / dy;
#pragma unroll
    for (int c = 0; c < 6; ++c) {
        const double fl = I.fx[c * fpx + fix], fr = I.fx[c * fpx + fix + ny];
        const double fb = I.fy[c * fpy + fiy], ft = I.fy[c * fpy + fiy + 1];
        rhs[c] = -(fr - fl) * sx + -(ft - fb) * sy;
    }
    double ncx[3], ncy[3];
    const double* c0 = sP + (ti + 4) * HJ + (tj + 4);
    {
        const int ix = threadIdx.x, iy = ti * (TJ + 1) + tj;
        double jm[3], jp[3];
#pragma unroll
        for (int c = 0; c < 3; ++c) { jm[c] = sX[c * nfx + ix]; jp[c] = sX[c * nfx + ix + TJ]; }
        if (kExactR) {
            DivGroup dv;
            noncon_by(c0, c0 + NPT, c0 + 2 * NPT, c0 + 3 * NPT, HJ, jm, jp, rhs_recip(I, sR, 0), rhs_recip(I, sR, 1), dv,
                      ncx);
            if (!(dv.ok & den_near(60.0 * dx) & den_mid_near(dx))) {
                const double a[3] = {jm[0], jm[1], jm[2]}, b[3] = {jp[0], jp[1], jp[2]};
                double o[3];
                noncon_each(c0, c0 + NPT, c0 + 2 * NPT, c0 + 3 * NPT, HJ, a, b, dx, o);
#pragma unroll
                for (int c = 0; c < 3; ++c) ncx[c] = o[c];
            }
        } else {
            fastm::noncon(c0, c0 + NPT, c0 + 2 * NPT, c0 + 3 * NPT, HJ, jm, jp, 1.0 / (60.0 * dx), 1.0 / dx, ncx);
        }
#pragma unroll
        for (int c = 0; c < 3; ++c) { jm[c] = sY[c * nfy + iy]; jp[c] = sY[c * nfy + iy + 1]; }
        if (kExactR) {
            DivGroup dv;
            noncon_by(c0, c0 + NPT, c0 + 2 * NPT, c0 + 4 * NPT, 1, jm, jp, rhs_recip(I, sR, 2), rhs_recip(I, sR, 3), dv,
                      ncy);
            if (!(dv.ok & den_near(60.0 * dy) & den_mid_near(dy))) {
                const double a[3] = {jm[0], jm[1], jm[2]}, b[3] = {jp[0], jp[1], jp[2]};
                double o[3];
                noncon_each(c0, c0 + NPT, c0 + 2 * NPT, c0 + 4 * NPT, 1, a, b, dy, o);
#pragma unroll
                for (int c = 0; c < 3; ++c) ncy[c] = o[c];
            }
        } else {
            fastm::noncon(c0, c0 + NPT, c0 + 2 * NPT, c0 + 4 * NPT, 1, jm, jp, 1.0 / (60.0 * dy), 1.0 / dy, ncy);
        }
    }
#pragma unroll
    for (int k = 0; k < 3; ++k) rhs[3 + k] = rhs[3 + k] + ncx[k] + ncy[k];
    if (I.source) {
        double s[6];
        load6(src, plane, n, s);
        double te, ti_, tr;
        temps_from_state(s, P, rhs_recip(I, sR, 4), rhs_recip(I, sR, 5), rhs_recip(I, sR, 6),
                         den_near(6.0 * P.cve) & den_near(6.0 * P.cvi) & den_near(P.a_rad), te, ti_, tr);
        const double so[3] = {-P.omega_ei * (te - ti_) - P.omega_er * (pow4d(te) - pow4d(tr)),
                              P.omega_ei * (te - ti_), P.omega_er * (pow4d(te) - pow4d(tr))};
#pragma unroll
        for (int k = 0; k < 3; ++k) rhs[3 + k] = rhs[3 + k] + so[k];
    }
    if (I.diffusion) {
        const double cx = -1.0 / (dx * dx), cy = -1.0 / (dy * dy);
#pragma unroll
        for (int k = 0; k < 3; ++k) {
            const double a = I.dfx[k * fpx + fix], b = I.dfx[k * fpx + fix + ny];
            const double c2 = I.dfy[k * fpy + fiy], d2 = I.dfy[k * fpy + fiy + 1];
            rhs[3 + k] = rhs[3 + k] + ((-(b - a) * cx) + (-(d2 - c2) * cy));
        }
    }
    if (mode == 0) {
        const long long ln = (long long)i * ny + j, lp = (long long)nx * ny;
        double* __restrict__ ro = rhs_out + 6 * I.cell_off;
#pragma unroll
        for (int c = 0; c < 6; ++c) ro[c * lp + ln] = rhs[c];
        return;
    }
    if (mode == 2) {
        double* __restrict__ ro = rhs_out + I.aoff;
#pragma unroll
        for (int c = 0; c < 6; ++c) ro[c * plane + n] = rhs[c];
    }
    const DevScalars& sc = *I.sc;
    double v[6];
    if (stage == 0) {
        const double coef = sc.coef[0];
#pragma unroll
        for (int c = 0; c < 6; ++c) v[c] = I.U[c * plane + n] + rhs[c] * coef;
#pragma unroll
        for (int c = 0; c < 6; ++c) I.A[c * plane + n] = v[c];
    } else if (stage == 1) {
        const double coef = sc.coef[1];
#pragma unroll
        for (int c = 0; c < 6; ++c) v[c] = I.U[c * plane + n] * 0.75 + I.A[c * plane + n] * 0.25 + rhs[c] * coef;
#pragma unroll
        for (int c = 0; c < 6; ++c) I.B[c * plane + n] = v[c];
    } else {
        const double coef = sc.coef[2];
        const double wb = 1.0 / 3.0, wa = 2.0 / 3.0;
#pragma unroll
        for (int c = 0; c < 6; ++c) v[c] = I.U[c * plane + n] * wb + I.B[c * plane + n] * wa + rhs[c] * coef;
#pragma unroll
        for (int c = 0; c < 6; ++c) I.U[c * plane + n] = v[c];
    }
    bool ok = isfinite(v[0]) && isfinite(v[1]) && isfinite(v[2]) && isfinite(v[3]) && isfinite(v[4]) &&
              isfinite(v[5]) && v[0] > 0.0;
    if (ok) { // main.rs:24-33
        // an energy e > rho w2 / 6 beyond any rounding passes without the exact
        // quotients: y is 1 / rho to 2^-39, the products below to 2^-37
        double y;
        asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(v[0]));
        y = __fma_rn(y, __fma_rn(-v[0], y, 1.0), y);
        const double ux = v[1] * y, uy = v[2] * y, e = fmin(fmin(v[3], v[4]), v[5]) * y;
        if (!(e > (ux * ux + uy * uy) * (1.0 / 6.0) * (1.0 + 1e-9) + 1e-290)) {
            const Recip r0 = recip(v[0]); // the five quotients by rho through one reciprocal (IEEE quotients)
            const double qx = div_rn(v[1], r0), qy = div_rn(v[2], r0);
            const double k = div6_rn(qx * qx + qy * qy);
            ok = !(div_rn(v[3], r0) - k <= 0.0 || div_rn(v[4], r0) - k <= 0.0 || div_rn(v[5], r0) - k <= 0.0);
        }
    }
    if (!ok) report(I, 2 + 2 * stage, 1, (unsigned)((long long)i * ny + j));
}

void launch_rhs_stage(cudaStream_t s, const Inst* insts, const Tile* tc, int nt, int stage, int mode, double* rhs,
                      int smem) {
    if (nt <= 0) return;
    static OncePerDevice attributes;
    int dev = 0;
    cudaGetDevice(&dev);
    attributes(dev, [] {
        int most = 0;
        for (int lg = RHS_LG_MIN; lg <= RHS_LG_MAX; ++lg) most = std::max(most, rhs_smem(lg));
        return cudaFuncSetAttribute(k_rhs_stage, cudaFuncAttributeMaxDynamicSharedMemorySize, most) == cudaSuccess;
    });
    k_rhs_stage<<<nt, RHS_THREADS, smem, s>>>(insts, tc, nt, stage, mode, rhs);
}

} // namespace rh3t
