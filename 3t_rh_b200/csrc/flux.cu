// Interface fluxes (main.rs:165-246: weno.rs:685-802 reconstruction_fast per
// x and y face, plus diffusion.rs:27-50 when diffusion is on).
//
// A block of two warps covers 64 faces (a TI x TJ tile, shape chosen per
// tile), one face per thread (small launches: up to three threads, each with
// two or three of the characteristic fields):
//   1. staging: the tile's stencil points (x faces: (TI + 5) x TJ points,
//      y faces: TI x (TJ + 5)) with their primitives and physical flux go to
//      shared memory once (the reference evaluates them once per face, six
//      times per point);
//   2. face: each thread forms its face's Roe state from the staged
//      primitives of its points 3 and 2;
//   3. characteristic pass: field by field (warp-uniform code), the row of
//      L, the projections and the two WENO5 reconstructions of f+ and f-;
//   4. output pass: (R g)_k = sum_c R[k][c] g_c in the reference's summation
//      order (weno.rs:793, 834-843), plus the diffusion flux for k >= 3.
//
// Bound by the FP64 pipe (65-72% busy in the no-contraction build; a loop of
// independent FMAs reaches 92%), at about 2,850 FP64 operations a face. A face
// per thread instead of a field per warp: nothing but the staged points
// crosses threads, so the two warps meet one barrier of equal work (with six
// warps each on other fields the barriers were the top stall, 2.1-2.6 warps per
// issued instruction), and the quotients a face's rows share are formed once.
// 8 blocks of 128 registers: 10 blocks of 96 spill (3% slower), 6 blocks of 150
// 4% slower. Without a branch per quotient (divrn.cuh), in this form and in one launch
// the fluxes of 24 batch instances take 1.25 ms a step instead of 2.08 ms, of the
// 961 x 3841 half-cylinder 4.75 ms instead of 7.44 ms (same bits); FMA build
// 0.89 ms instead of 1.17 ms. (A face whose state is out of the branch-free form's
// range, physics.cuh near_face: the general form, face by face.)
//
// RH3T_EXACT selects the reference's expressions; otherwise the fastm forms
// (shared reciprocals, one division per WENO5) are used.
#include <algorithm>

#include "common.cuh"
#include "kernels.cuh"
#include "physics.cuh"

namespace rh3t {

#ifdef RH3T_EXACT
constexpr bool kExact = true;
#else
constexpr bool kExact = false;
#endif

// Shared memory of a block, sized for the launch's largest tile (npt points):
//   pt: per point seven double2: the state (rho, mx) (my, ee) (ei, er), the
//       physical flux, (u, v). 112 bytes: the 16-byte loads of consecutive
//       points fall in different banks;
//   E:  per point e_e, e_i, e_r, sqrt(rho), for the Roe averages; then G, the
//       six g_c of a face;
//   Q:  per face the Roe state u v w2 ee ei er cs2 cs he hi hr b den, then
//       the reciprocals the L rows divide by: no-contraction build
//       (recip_near, both parts) of den, b, gt cs2; FMA build 1/cs2, 1/b;
//   T:  per point te, ti, tr (launches with a diffusive instance);
//   gkgt, y6: no-contraction build, gk / gt and the reciprocal of 6 gk (both
//       parts) for gk = ge, gi, gr;
//   act: per face near_face's answer (launches with several thread groups a tile).
constexpr int NQ = kExact ? 19 : 15, PT = 7;
struct FluxShared {
    double2* pt;
    double *E, *G, *Q, *T, *gkgt, *y6;
    int* act;
    int npt;
};
__host__ __device__ __forceinline__ int flux_e_doubles(int npt) {
    return 4 * npt > 6 * FLUX_FACES ? 4 * npt : 6 * FLUX_FACES;
}
__host__ __device__ __forceinline__ int flux_smem(int npt, bool diffusion) {
    return npt * PT * 16 + 8 * (flux_e_doubles(npt) + NQ * FLUX_FACES + 10 + FLUX_FACES / 2 + (diffusion ? 3 * npt : 0));
}
__device__ __forceinline__ FluxShared flux_shared(unsigned char* smem, int npt) {
    FluxShared S;
    S.npt = npt;
    S.pt = reinterpret_cast<double2*>(smem);
    S.Q = reinterpret_cast<double*>(S.pt + npt * PT);
    S.gkgt = S.Q + NQ * FLUX_FACES;
    S.y6 = S.gkgt + 3;
    S.act = reinterpret_cast<int*>(S.gkgt + 10);
    S.E = S.gkgt + 10 + FLUX_FACES / 2;
    S.G = S.E;
    S.T = S.E + flux_e_doubles(npt);
    return S;
}

// face f of the tile -> face (i, j), first stencil point p0 and point stride
template <int DIR>
__device__ __forceinline__ void face_index(const Tile& t, int f, int& i, int& j, int& p0, int& ps) {
    const int r = f >> t.lg, cc = f & ((1 << t.lg) - 1);
    i = t.i + r;
    j = t.j0 + cc;
    if (DIR == 0) { p0 = f; ps = 1 << t.lg; }
    else { p0 = r * ((1 << t.lg) + 5) + cc; ps = 1; }
}

// Qf: the face's column of Q (stride FLUX_FACES)
__device__ __forceinline__ void load_q(const double* Qf, Roe& q) {
    constexpr int F = FLUX_FACES;
    q.u = Qf[0]; q.v = Qf[F]; q.w2 = Qf[2 * F]; q.ee = Qf[3 * F]; q.ei = Qf[4 * F]; q.er = Qf[5 * F];
    q.cs2 = Qf[6 * F]; q.cs = Qf[7 * F]; q.he = Qf[8 * F]; q.hi = Qf[9 * F]; q.hr = Qf[10 * F]; q.b = Qf[11 * F];
    q.den = Qf[12 * F];
}

template <int DIR> __device__ __forceinline__ double char_speed(int c, const Roe& q) {
    const double vel = DIR == 0 ? q.u : q.v;
    return fabs(c == 0 ? vel - q.cs : (c == 5 ? vel + q.cs : vel));
}

// f+ and f- of field c at the six points (weno.rs:760-780): L . f, L . u and
// the Lax-Friedrichs split with speed a. pf: the face's first point, ps the
// point stride in double2
__device__ __forceinline__ void split_fluxes(const double2* pf, int ps, const double Lc[6], double a, double fp[6],
                                             double fm[6]) {
#pragma unroll
    for (int k = 0; k < 6; ++k) {
        const double2* p = pf + k * ps;
        const double2 u01 = p[0], u23 = p[1], u45 = p[2];
        const double2 f01 = p[3], f23 = p[4], f45 = p[5];
        const double cf = Lc[0] * f01.x + Lc[1] * f01.y + Lc[2] * f23.x + Lc[3] * f23.y + Lc[4] * f45.x +
                          Lc[5] * f45.y;
        const double cs = Lc[0] * u01.x + Lc[1] * u01.y + Lc[2] * u23.x + Lc[3] * u23.y + Lc[4] * u45.x +
                          Lc[5] * u45.y;
        fp[k] = 0.5 * (cf + a * cs);
        fm[k] = 0.5 * (cf - a * cs);
    }
}

// the same for the transverse field, whose row of L is (-w, 0, 1, 0, 0, 0), w
// the transverse velocity, with the 1 at the transverse momentum
// (finite data: the four products by 0 add zeros)
template <int DIR>
__device__ __forceinline__ void split_transverse(const double2* pf, int ps, double w, double a, double fp[6],
                                                 double fm[6]) {
#pragma unroll
    for (int k = 0; k < 6; ++k) {
        const double2* p = pf + k * ps;
        const double cf = DIR == 0 ? -w * p[3].x + p[4].x : -w * p[3].x + p[3].y;
        const double cs = DIR == 0 ? -w * p[0].x + p[1].x : -w * p[0].x + p[0].y;
        fp[k] = 0.5 * (cf + a * cs);
        fm[k] = 0.5 * (cf - a * cs);
    }
}

// index of an energy row's gk (0 for the other rows, which do not use it)
template <int DIR> __device__ __forceinline__ int energy_index(int c) {
    const int mode = row_mode<DIR>(c);
    return mode < 2 || mode == 5 ? 0 : mode - 2;
}

// Quotients with a test and a fallback each (divrn.cuh), out of line: faces
// with operands outside the branch-free form's range
template <int DIR>
static __device__ __noinline__ double char_flux_each(const double2* pf, int ps, const double* Qf, const DevParams& P,
                                                     int c, double gkgt) {
    Roe q;
    double Lc[6], fp[6], fm[6];
    load_q(Qf, q);
    l_row<DIR>(c, q, roe_div(q, P), gkgt, P, Lc);
    split_fluxes(pf, ps, Lc, char_speed<DIR>(c, q), fp, fm);
    double r0 = 0.0, r1 = 0.0;
#pragma unroll 1
    for (int s = 0; s < 2; ++s) {
        const bool m = s != 0;
        const double w = weno5(m ? fm[5] : fp[0], m ? fm[4] : fp[1], m ? fm[3] : fp[2], m ? fm[2] : fp[3],
                               m ? fm[1] : fp[4], P.eps);
        if (m) r1 = w;
        else r0 = w;
    }
    return r0 + r1;
}

// entries 0 to 2 of the row of L, for a face with a tiny velocity
template <int DIR>
static __device__ __noinline__ LVel char_row_velocity(const double* Qf, const DevParams& P, int c, bool square) {
    Roe q;
    load_q(Qf, q);
    return l_row_velocity<DIR>(c, q, P, square);
}

// g_c; mode: near_face's answer, not FACE_GENERAL; lo: weno_window
template <int DIR>
__device__ __forceinline__ double char_flux(const double2* pf, int ps, const double* Qf, const DevParams& P, int c,
                                            const double* gkgt, int mode, unsigned lo) {
    Roe q;
    load_q(Qf, q);
    double Lc[6], fp[6], fm[6];
    const double a = char_speed<DIR>(c, q);
    if (row_mode<DIR>(c) == 1) {
        split_transverse<DIR>(pf, ps, DIR == 0 ? q.v : q.u, a, fp, fm);
    } else if (kExact) {
        RoeDivN rd;
        const double gt = (P.gamma_i - 1.0) + (P.gamma_e - 1.0) + (P.gamma_r - 1.0);
        rd.den = {q.den, Qf[13 * FLUX_FACES], Qf[14 * FLUX_FACES]};
        rd.b = {q.b, Qf[15 * FLUX_FACES], Qf[16 * FLUX_FACES]};
        rd.cg = {gt * q.cs2, Qf[17 * FLUX_FACES], Qf[18 * FLUX_FACES]};
        rd.scale();
        l_row<DIR>(c, q, rd, gkgt[energy_index<DIR>(c)], P, Lc);
        if (mode != FACE_NEAR) {
            const LVel l = char_row_velocity<DIR>(Qf, P, c, mode == FACE_SQUARE);
            if (c == 0 || c == 5 || mode == FACE_SQUARE) Lc[0] = l.l0;
            Lc[1] = l.l1;
            Lc[2] = l.l2;
        }
        split_fluxes(pf, ps, Lc, a, fp, fm);
    } else {
        fastm::l_row<DIR>(c, q, Qf[13 * FLUX_FACES], Qf[14 * FLUX_FACES], P, Lc);
        split_fluxes(pf, ps, Lc, a, fp, fm);
    }
    if (!kExact)
        return fastm::weno5(fp[0], fp[1], fp[2], fp[3], fp[4], P.eps) +
               fastm::weno5(fm[5], fm[4], fm[3], fm[2], fm[1], P.eps);
    bool near = true;
    const double r0 = weno5_near(fp[0], fp[1], fp[2], fp[3], fp[4], P.eps, lo, near);
    const double r1 = weno5_near(fm[5], fm[4], fm[3], fm[2], fm[1], P.eps, lo, near);
    return near ? r0 + r1 : char_flux_each<DIR>(pf, ps, Qf, P, c, gkgt[energy_index<DIR>(c)]);
}

// The diffusion terms (off in most runs) are out of line: their code stays
// out of the instruction cache of runs without diffusion.
// diffusion.rs:27-50: component 3 <- Te, 4 <- Ti, 5 <- Tr^4 (m3 = 0, 1, 2); T:
// the temperature at the face's first point, ps the point stride
static __device__ __noinline__ void diffusion_out(const double* T, int ps, const DevParams& P, int m3, double* out) {
    double v[6];
#pragma unroll
    for (int m = 0; m < 6; ++m) {
        const double x = T[m * ps];
        v[m] = m3 == 2 ? pow4d(x) : x;
    }
    const double kap = m3 == 0 ? P.kappa_e : (m3 == 1 ? P.kappa_i : P.kappa_r);
    const double term = kap * (2.0 * v[5] - 25.0 * v[4] + 245.0 * v[3] - 245.0 * v[2] + 25.0 * v[1] - 2.0 * v[0]);
    *out = term / 180.0;
}

// temperatures of a staged point
static __device__ __noinline__ void stage_temps(const double2* p, const DevParams& P, double* T, int npt) {
    const double s[6] = {p[0].x, p[0].y, p[1].x, p[1].y, p[2].x, p[2].y};
    temps_from_state(s, P, T[0], T[npt], T[2 * npt]);
}

// (R g)_k in the reference's summation order (weno.rs:793, 834-843); Gf: the
// face's column of G
template <int DIR, bool NEAR>
__device__ __forceinline__ double r_dot(const Roe& q, const double* Gf, const double* y6, const DevParams& P, int k) {
    double Rr[6];
    RecipN r6k = {1.0, 1.0, 0.0};
    if (NEAR && k >= 3) {
        const double gk = (k == 3 ? P.gamma_e : (k == 4 ? P.gamma_i : P.gamma_r)) - 1.0;
        r6k = {6.0 * gk, y6[k - 3], y6[k]};
    }
    r_row<DIR, NEAR>(k, q, r6k, P, Rr);
    constexpr int F = FLUX_FACES;
    return Rr[0] * Gf[0] + Rr[1] * Gf[F] + Rr[2] * Gf[2 * F] + Rr[3] * Gf[3 * F] + Rr[4] * Gf[4 * F] +
           Rr[5] * Gf[5 * F];
}
template <int DIR>
static __device__ __noinline__ double r_dot_each(const double* Qf, const double* Gf, const DevParams& P, int k) {
    Roe q;
    load_q(Qf, q);
    return r_dot<DIR, false>(q, Gf, nullptr, P, k);
}

// Field `m` of group `g` when NG groups of 64 threads share a tile's six fields
// (each group about the same work: x faces: fields 1-3 energy, 0 and 5
// acoustic, 4 transverse; y faces 2-4, 0 and 5, 1), a hex digit each
template <int DIR, int NG> __device__ __forceinline__ int group_field(int g, int m) {
    constexpr unsigned long long x = NG == 1 ? 0x543210ull : (NG == 2 ? 0x350421ull : 0x435201ull);
    constexpr unsigned long long y = NG == 1 ? 0x543210ull : (NG == 2 ? 0x450132ull : 0x145302ull);
    return (int)((DIR == 0 ? x : y) >> (4 * (g * (6 / NG) + m))) & 15;
}

template <int DIR, int NG>
__device__ __forceinline__ void flux_tile(const Inst& I, const Tile& t, int stage, const FluxShared& S) {
    const DevParams& P = I.P;
    const double* __restrict__ buf = stage_src(I, stage);
    const long long plane = I.plane;
    const int nx = I.nx, ny = I.ny, npt = S.npt;
    const int cols = 1 << t.lg, rows = FLUX_FACES >> t.lg;
    const int np = DIR == 0 ? (rows + 5) * cols : rows * (cols + 5);
    const bool diff = I.diffusion != 0;
    if (kExact && threadIdx.x < 3) {
        const int k = threadIdx.x;
        const double gi = P.gamma_i - 1.0, ge = P.gamma_e - 1.0, gr = P.gamma_r - 1.0;
        const double gk = k == 0 ? ge : (k == 1 ? gi : gr);
        S.gkgt[k] = __ddiv_rn(gk, gi + ge + gr);
        const RecipN r = recip_near(6.0 * gk);
        S.y6[k] = r.y;
        S.y6[3 + k] = r.yl;
    }
    // ---- 1. staging: state, primitives and physical flux of every point
    for (int p = threadIdx.x; p < np; p += FLUX_FACES * NG) {
        int pi, pj;
        if (DIR == 0) { pi = t.i - 3 + (p >> t.lg); pj = t.j0 + (p & (cols - 1)); }
        else { const int r = p / (cols + 5); pi = t.i + r; pj = t.j0 - 3 + (p - r * (cols + 5)); }
        double s[6] = {1.0, 0.0, 0.0, 1.0, 1.0, 1.0};
        if (pi >= -RH3T_PAD && pi < nx + RH3T_PAD && pj >= -RH3T_PAD && pj < ny + RH3T_PAD)
            load6(buf, plane, node_of(I, pi, pj), s);
        const Prim d = kExact ? prim_from_state(s, P) : fastm::prim(s, P);
        double f[6];
        phys_flux<DIR>(s, d, f);
        double2* q = S.pt + PT * p;
#pragma unroll
        for (int k = 0; k < 3; ++k) {
            q[k] = make_double2(s[2 * k], s[2 * k + 1]);
            q[3 + k] = make_double2(f[2 * k], f[2 * k + 1]);
        }
        q[6] = make_double2(d.u, d.v);
        S.E[p] = d.e_e; S.E[npt + p] = d.e_i; S.E[2 * npt + p] = d.e_r; S.E[3 * npt + p] = sqrt(s[0]);
        if (diff) stage_temps(q, P, S.T + p, npt);
    }
    // ---- 2. this thread's face (its Roe state by the first group)
    const int f = NG == 1 ? threadIdx.x : threadIdx.x & (FLUX_FACES - 1), g = NG == 1 ? 0 : threadIdx.x / FLUX_FACES;
    int i, j, p0, ps;
    face_index<DIR>(t, f, i, j, p0, ps);
    bool valid = DIR == 0 ? (i <= nx && j < ny) : (i < nx && j <= ny);
    if (valid) {
        const uint8_t m0 = I.mask[node_of(I, i, j)];
        const uint8_t m1 = DIR == 0 ? I.mask[node_of(I, i - 1, j)] : I.mask[node_of(I, i, j - 1)];
        valid = (m0 | m1) != 0;
    }
    __syncthreads();
    double* Qf = S.Q + f;
    int near = FACE_NEAR; // near_face's answer
    if (valid && g == 0) {
        // points[3] and points[2] of the face: the staged primitives (the
        // same functions of the same states as a fresh evaluation)
        const int p3 = p0 + 3 * ps, p2 = p0 + 2 * ps;
        const double2 v3 = S.pt[PT * p3 + 6], v2 = S.pt[PT * p2 + 6];
        Prim d3, d2;
        d3.u = v3.x; d3.v = v3.y; d3.e_e = S.E[p3]; d3.e_i = S.E[npt + p3]; d3.e_r = S.E[2 * npt + p3];
        d2.u = v2.x; d2.v = v2.y; d2.e_e = S.E[p2]; d2.e_i = S.E[npt + p2]; d2.e_r = S.E[2 * npt + p2];
        const double rho3 = S.E[3 * npt + p3], rho2 = S.E[3 * npt + p2];
        Roe q;
        double y[6];
        if (kExact) {
            q = roe_average_sqrt(rho3, d3, rho2, d2, P);
            RoeDivN rd;
            const double gt = (P.gamma_i - 1.0) + (P.gamma_e - 1.0) + (P.gamma_r - 1.0);
            near = near_gammas(P) && near_eps(P) ? near_face(q, gt, rd) : FACE_GENERAL;
            y[0] = rd.den.y; y[1] = rd.den.yl; y[2] = rd.b.y; y[3] = rd.b.yl; y[4] = rd.cg.y; y[5] = rd.cg.yl;
        } else {
            const double a6[6] = {rho3, d3.u, d3.v, d3.e_e, d3.e_i, d3.e_r};
            const double b6[6] = {rho2, d2.u, d2.v, d2.e_e, d2.e_i, d2.e_r};
            q = fastm::roe(a6, b6, P);
            y[0] = 1.0 / q.cs2;
            y[1] = 1.0 / q.b;
        }
        const double qv[13] = {q.u, q.v, q.w2, q.ee, q.ei, q.er, q.cs2, q.cs, q.he, q.hi, q.hr, q.b, q.den};
#pragma unroll
        for (int k = 0; k < 13; ++k) Qf[k * FLUX_FACES] = qv[k];
#pragma unroll
        for (int k = 13; k < NQ; ++k) Qf[k * FLUX_FACES] = y[k - 13];
    }
    if (NG > 1 && g == 0) S.act[f] = near;
    __syncthreads(); // E is read; G takes its place
    if (NG == 1 && !valid) return;
    if (NG > 1) near = S.act[f];
    // ---- 3. characteristic pass (a loop, not unrolled: one copy of its code
    // stays within the instruction cache)
    double* Gf = S.G + f;
    const unsigned lo = kExact ? weno_window(P.eps) : 0u;
    const double2* pf = S.pt + PT * p0;
    // (a face in the general form: a loop of its own with one thread a face; in the loop
    // of all with several, where its registers spill: NG 2 64 B of stores against 0)
    if (kExact && NG == 1 && near == FACE_GENERAL) {
#pragma unroll 1
        for (int c = 0; c < 6; ++c)
            Gf[c * FLUX_FACES] = char_flux_each<DIR>(pf, PT * ps, Qf, P, c, S.gkgt[energy_index<DIR>(c)]);
    } else if (NG == 1 || valid) {
#pragma unroll 1
        for (int m = 0; m < 6 / NG; ++m) {
            const int c = NG == 1 ? m : group_field<DIR, NG>(g, m);
            Gf[c * FLUX_FACES] = kExact && NG > 1 && near == FACE_GENERAL
                                     ? char_flux_each<DIR>(pf, PT * ps, Qf, P, c, S.gkgt[energy_index<DIR>(c)])
                                     : char_flux<DIR>(pf, PT * ps, Qf, P, c, S.gkgt, near, lo);
        }
    }
    if (NG > 1) {
        __syncthreads();
        if (!valid) return;
    }
    // ---- 4. output pass
    long long fplane, fidx;
    double *fo, *dfo;
    if (DIR == 0) { fplane = (long long)(nx + 1) * ny; fidx = (long long)i * ny + j; fo = I.fx; dfo = I.dfx; }
    else { fplane = (long long)nx * (ny + 1); fidx = (long long)i * (ny + 1) + j; fo = I.fy; dfo = I.dfy; }
    if (!kExact || near > 0) {
        Roe q;
        load_q(Qf, q);
#pragma unroll
        for (int k = 0; k < 6; ++k)
            if (NG == 1 || k % NG == g) fo[k * fplane + fidx] = r_dot<DIR, kExact>(q, Gf, S.y6, P, k);
    } else {
#pragma unroll 1
        for (int k = g; k < 6; k += NG) fo[k * fplane + fidx] = r_dot_each<DIR>(Qf, Gf, P, k);
    }
    if (diff)
#pragma unroll 1
        for (int m = g; m < 3; m += NG) diffusion_out(S.T + m * npt + p0, ps, P, m, dfo + m * fplane + fidx);
}

constexpr int FLUX_NG3 = 2 * 148, FLUX_NG2 = 4 * 148; // tiles up to which 3 and 2 groups share a tile
// blocks per SM (FMA build: bounds of 12, 80 registers, 2% faster than of 8; shared
// memory admits 9 blocks of default tiles, 7 with an x tile of 4 x 16)
constexpr int FLUX_MIN_BLOCKS = kExact ? 8 : 12;
// x faces (blocks [0, ntx)), then y faces: in one launch the y tiles fill the
// SMs that the last x tiles leave idle (121 x 481: two launches of 0.8 waves each
// took 42 us, one takes 31 us).
// NG groups of 64 threads share a tile where the launch has too few tiles to
// fill the SMs: at one thread a face a small launch is one face's serial chain
// (about 14 cycles an FP64 operation at a warp or two per scheduler). Three
// groups while the tiles fit two blocks of 192 threads a SM, two while they fit
// four of 128, one beyond (a step's fluxes, one / two / three groups: 31x121, 128
// tiles, 48 / 40 / 40 us; 512x8 planar shock, 193 tiles, 53 / 48 / 45; 61x241, 492
// tiles, 59 / 57 / 61; 1024x8, 385 tiles, 64 / 56 / 63; 75x297, 717 tiles, 69 / 69 /
// 74; 121x481, 1937 tiles, 118 / 118 / 140).
template <int NG>
__global__ void __launch_bounds__(FLUX_FACES * NG, NG == 1 ? FLUX_MIN_BLOCKS : (NG == 2 ? 4 : 2)) k_flux(
    const Inst* __restrict__ insts, const Tile* __restrict__ tx, int ntx, const Tile* __restrict__ ty, int stage,
    int npx, int npy) {
    extern __shared__ __align__(16) unsigned char flux_mem[];
    const bool x = (int)blockIdx.x < ntx;
    const Tile t = x ? tx[blockIdx.x] : ty[blockIdx.x - ntx];
    const Inst& I = insts[t.inst];
    if (has_error(I)) return;
    if (x) flux_tile<0, NG>(I, t, stage, flux_shared(flux_mem, npx));
    else flux_tile<1, NG>(I, t, stage, flux_shared(flux_mem, npy));
}

int flux_points(int dir, int lg) {
    const int cols = 1 << lg, rows = FLUX_FACES >> lg;
    return dir == 0 ? (rows + 5) * cols : rows * (cols + 5);
}

void launch_flux(cudaStream_t s, const Inst* insts, const Tile* tx, int ntx, const Tile* ty, int nty, int stage,
                 const FluxSize& z) {
    if (ntx + nty <= 0) return;
    const int np = std::max(ntx > 0 ? z.npx : 0, nty > 0 ? z.npy : 0);
    const int n = ntx + nty, smem = flux_smem(np, z.diffusion);
    // (FMA build: one instantiation, since another might contract other sums, and
    // an instance's result must not depend on what else the launch holds)
    if constexpr (kExact) {
        if (n <= FLUX_NG3) {
            k_flux<3><<<n, 3 * FLUX_FACES, smem, s>>>(insts, tx, ntx, ty, stage, z.npx, z.npy);
            return;
        }
        if (n <= FLUX_NG2) {
            k_flux<2><<<n, 2 * FLUX_FACES, smem, s>>>(insts, tx, ntx, ty, stage, z.npx, z.npy);
            return;
        }
    }
    k_flux<1><<<n, FLUX_FACES, smem, s>>>(insts, tx, ntx, ty, stage, z.npx, z.npy);
}

int flux_launches(int ntx, int nty) { return ntx + nty > 0 ? 1 : 0; }

} // namespace rh3t
