// sweep_core.cuh -- the fused directional sweep kernel: one launch per x/y/z
// sweep of an SSPRK stage (src/ssprk.cpp:1000-1025, 1218-1272).  Included by
// sweep_kernels.cu (single-domain launches) and ensemble_sweep.cu (batched
// ensembles); each translation unit instantiates the shapes it launches.
//
// The reference runs a sweep as six all-line kernels with workspaces in
// memory (qx, ux, ax, Fx and the 7x7 L and R per interface: ~18 GB at 256^3).
// Here a warp owns NL neighbouring lines and marches along the sweep in
// chunks of W = 32 / NL cells, one new cell and one interface per lane; HBM
// sees only the stage input, the RK base, the stage output and the two CT
// flux arrays.
//
// One chunk (interfaces fb .. fb+W-1 of each line; interface f sits between
// padded cells f+2 and f+3, its WENO stencil is cells f .. f+5,
// src/ssprk.cpp:861-865; the chunk's new cells are fb+5 .. fb+W+4):
//   load   the new cells' 8 conserved variables arrive by a TMA tensor load
//          issued one chunk ahead, the update's read operand by one issued at
//          the chunk's start.  The variable permutation of the y/z sweeps
//          (src/ssprk.cpp:1054-1061, 1145-1152) is applied on reading.
//   cell   primitives with floors (458-516), eigenvalues and fluxes (538-595)
//          of the lane's cell, and its differences (F, q_proj) to the cell
//          before (by shuffle) into the warp's shared-memory window, which
//          still holds the last cells of the chunk before.
//   face   everything of the lane's interface in registers: arithmetic-mean
//          state and eigen-system (610-660), projection of the 5 cell
//          differences of the stencil, LLF split and WENO5-JS of the seven
//          fields (841-937), back-projection (941-943), CT terms (967-994).
//   update -dtdl (F^_{i+1/2} - F^_{i-1/2}) (949-965) and the stage
//          accumulation (405-431, 1067-1096, 1158-1187) of the cell left of
//          the interface; the flux before comes from the neighbouring lane.
//
// Why this form.  The sweep is bound by the FP64 pipe (~1,350 FP64
// instructions per zone; 220 bytes).  A form with one block per tile and the
// seven fields on seven threads spent more than half of its issue slots on
// other instructions, and waited at six block barriers per tile.  Here the
// warps share nothing, so there is no block barrier; one lane forms all
// seven fields, so the eigenvectors' common parts are formed once (see
// project below) and no 7x7 matrix exists in any form; and the only work done
// twice is one interface and five cells per segment end.
//
// Bit-for-bit reproducibility: the arithmetic is written with explicit fma
// calls and these translation units are compiled with -fmad=false, so every
// instantiation (single domain, ensemble member, label collection, any NL and
// segment length) computes the same bits.
//
// Precision: the kernel is a template on the working type R of the
// eigen-system, projection and WENO arithmetic.  R = double is the plain
// method.  R = float is the mixed-precision method: primitives, cell fluxes,
// the physical central flux F_i, the back-projected interface flux sum, the
// CT terms and the stage update stay FP64; the FP32 part only carries the
// characteristic upwind corrections, computed from cell differences that are
// formed in FP64 and then rounded.
#pragma once

#include "fp_ops.cuh"
#include "how_internal.cuh"
#include "router.cuh"
#include "tma.cuh"
#include "tmem.cuh"

#include <type_traits>

namespace how {

namespace {

using how::fm;   // (beside the overloads for pairs)
using how::near_recip;

// Two FP32 values that take the same operations: of a cell difference the
// flux's and the state's part, of a field pair the minus and the plus field.
// One packed instruction (add, sub, mul and fma.rn.f32x2) does both, rounded as
// the two alone: the mixed sweep is bound by its instructions' issue (192^3
// sweep 0.86 -> 0.76 ms).
struct PairF { unsigned long long v; };

__device__ __forceinline__ PairF make_pair(float a, float b) {
    PairF r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r.v) : "f"(a), "f"(b));
    return r;
}
__device__ __forceinline__ PairF both(float s) { return make_pair(s, s); }
__device__ __forceinline__ PairF from_mem(float2 m) { return make_pair(m.x, m.y); }
__device__ __forceinline__ void split(PairF p, float& a, float& b) { asm("mov.b64 {%0, %1}, %2;" : "=f"(a), "=f"(b) : "l"(p.v)); }
__device__ __forceinline__ PairF operator+(PairF x, PairF y) {
    PairF r;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r.v) : "l"(x.v), "l"(y.v));
    return r;
}
__device__ __forceinline__ PairF operator-(PairF x, PairF y) {
    PairF r;
    asm("sub.rn.f32x2 %0, %1, %2;" : "=l"(r.v) : "l"(x.v), "l"(y.v));
    return r;
}
__device__ __forceinline__ PairF operator*(PairF x, PairF y) {
    PairF r;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r.v) : "l"(x.v), "l"(y.v));
    return r;
}
__device__ __forceinline__ PairF fm(PairF x, PairF y, PairF z) {
    PairF r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r.v) : "l"(x.v), "l"(y.v), "l"(z.v));
    return r;
}
__device__ __forceinline__ PairF near_recip(PairF x) {
    float a, b;
    split(x, a, b);
    return make_pair(near_recip(a), near_recip(b));
}

// The window's cell differences: FP64 keeps the rows of the flux's and the
// state's differences apart (D + 7 rows), FP32 as pairs.
template <typename R> struct Diff;
template <> struct Diff<double> { using T = double; static constexpr int rows = 14; };
template <> struct Diff<float> { using T = float2; static constexpr int rows = 7; };

__host__ __device__ constexpr int align_up(int x, int a) { return (x + a - 1) / a * a; }

// One warp's shared memory.  Window arrays are [row][column], a column per
// (cell, line) with the lines fastest: the first H cells are the last of the
// chunk before, the other 32 columns are the lanes' new cells.  Consecutive
// lanes read consecutive columns at every stencil offset, so no access has a
// bank conflict, and the offset is an immediate.
template <int DIR, int NL, typename R, int MODE>
struct WarpMem {
    static constexpr int W = 32 / NL;                 // cells (and interfaces) per line and chunk
    // the x sweep's operand tile starts one cell early: its innermost TMA
    // coordinate has to be even, and the raw tile's start fb+5 is
    static constexpr int TO = DIR == 0 ? W + 2 : W;
    // cells of history: differences 4, |lambda| 5, primitives and fluxes 3,
    // and 4 for the three primitives the four-point CT average reads
    static constexpr int HD = 4, HL = 5, HP = 3, HB = 4;
    static constexpr int CD = HD * NL + 32, CL = HL * NL + 32, CP = HP * NL + 32, CB = HB * NL + 32;
    static constexpr int NCF = MODE == 3 ? 5 : MODE != 0 ? 2 : 0;   // routing values per cell, FP32
    static constexpr int bRaw = 0;                                  // [8][...] raw conserved of the new cells
    static constexpr int bOp = bRaw + 8 * 8 * 32;                   // [8][...] update operand
    static constexpr int bP = align_up(bOp + 8 * 8 * NL * TO, 128); // [5][CP] rho vx By Bz H
    static constexpr int bF = bP + 8 * 5 * CP;                      // [7][CP] cell fluxes
    static constexpr int bB = align_up(bF + 8 * 7 * CP, 16);        // [3][CB] vy vz Bx
    static constexpr int bU = bB + 8 * 3 * CB;                      // [4][NL] M, E of the last cell before
    static constexpr int bX = bU + 8 * 4 * NL;                      // [7][NL] interface flux before
    static constexpr int bBar = bX + 8 * 7 * NL;                    // 2 mbarriers: raw, operand
    static constexpr int bS = bBar + 16;                            // [32] the lanes' offsets (see spot)
    static constexpr int bD = align_up(bS + 8 * 32, 16);              // [14][CD] differences of (F, q), R (Diff)
    static constexpr int bL = align_up(bD + (int)sizeof(R) * 14 * CD, 16);   // [7][CL] |lambda|, R
    static constexpr int bC = align_up(bL + (int)sizeof(R) * 7 * CL, 16);    // [NCF][CL] FP32
    static constexpr int bytes = align_up(bC + 4 * NCF * CL, 128);
    static constexpr uint32_t raw_bytes = 8u * 8 * 32;
    static constexpr uint32_t op_bytes = 8u * 8 * NL * TO;
    static_assert(HL * NL <= 32, "the window shift moves at most one column per lane");
};

// The move of a window array's last COLS columns to its front, in two steps so
// that a warp issues every load before the first store (the compiler cannot
// rule out that they alias): 16-byte moves where the rows allow it, a power of
// two of lanes per row.
template <typename T, int ROWS, int PITCH, int COLS>
struct MoveBack {
    static constexpr bool VEC = PITCH * sizeof(T) % 16 == 0 && COLS * sizeof(T) % 16 == 0;
    static constexpr int E = VEC ? 16 / (int)sizeof(T) : 1;
    static constexpr int per_row(int n) { int p = 1; while (p < n) p *= 2; return p; }
    static constexpr int PER = per_row(COLS / E), RPI = 32 / PER, N = (ROWS + RPI - 1) / RPI;
    using V = std::conditional_t<VEC, float4, T>;
    V v[N];
    static __device__ __forceinline__ bool mine(int i, int lane) {
        return i * RPI + lane / PER < ROWS && lane % PER < COLS / E;
    }
    // s: the array's first row and column
    __device__ __forceinline__ void load(const T* s, int lane) {
        const T* at = s + lane / PER * PITCH + lane % PER * E + 32;
#pragma unroll
        for (int i = 0; i < N; ++i)
            if (mine(i, lane)) v[i] = *reinterpret_cast<const V*>(at + i * RPI * PITCH);
    }
    __device__ __forceinline__ void store(T* s, int lane) const {
        T* at = s + lane / PER * PITCH + lane % PER * E;
#pragma unroll
        for (int i = 0; i < N; ++i)
            if (mine(i, lane)) *reinterpret_cast<V*>(at + i * RPI * PITCH) = v[i];
    }
};

// One half of the WENO5-JS split (src/ssprk.cpp:883-937) from its four
// arguments (twice the LLF-split differences; see weno_flux).  With t = a - b,
// b - c, c - d the indicators are
//   13 t^2 + 3 (a - 3 b)^2 = 16 t^2 - 12 b t + 12 b^2,    the same with (b + c),
//   13 t^2 + 3 (3 c - d)^2 = 16 t^2 + 12 c t + 12 c^2,
// and a common factor cancels from the weights, so they are formed as a twelfth
// of that, eps with them, in eleven operations for the three (no term cancels
// by more than a fifth: the least value over t is 13/16 b^2).
//   w0 = P / D, w2 = 3 Q / D with e_k = (eps + IS_k)^2, P = e1 e2, Q = e0 e1,
//   D = P + 6 e0 e2 + 3 Q;  X0, X1: the two second differences.
// (V: a value or a pair of them; k: both() of a constant.  The differences are
// taken with the signs that need no negation: X1m = -X1.)
template <typename V>
struct WenoHalf { V e0, e1, e2, X0, X1m; };

template <typename V, typename K>
__device__ __forceinline__ WenoHalf<V> weno_half(V a, V b, V c, V d, K k) {
    const V g = k(4.0 / 3.0), eps = k(4.0e-10 / 12.0);
    const V t0 = b - a, t2 = c - b, t4 = c - d;   // -t, -t, t above
    const V bb = fm(b, b, eps), cc = fm(c, c, eps);
    const V d0 = fm(t0, fm(g, t0, b), bb), d1 = fm(t2, fm(g, t2, b), bb), d2 = fm(t4, fm(g, t4, c), cc);
    return WenoHalf<V>{d0 * d0, d1 * d1, d2 * d2, t2 - t0, t2 + t4};
}

// Characteristic WENO5-JS/LLF flux of one field (src/ssprk.cpp:883-937) from
// the projected cell differences f_k = L.(F_{k+1} - F_k), q_k = L.(q_{k+1} - q_k),
// k = 0..4 over the 6-cell stencil, and the stencil's largest |lambda|.
//
// Restated, not transcribed:
//  * the fourth-order central part (-F1 + 7F2 + 7F3 - F4)/12 equals
//    F2 + (f1 + 6 f2 - f3)/12; its F2 share is added back in physical
//    space after the back-projection (R L = I), so only the correction is
//    returned;
//  * the LLF-split arguments 0.5 (f +- amx q) are used without the 0.5:
//    doubling a, b, c, d quadruples every smoothness indicator, so with
//    eps -> 4 eps the nonlinear weights are unchanged and the 0.5 moves onto
//    the linear combination (1/3 -> 1/6, 1/6 -> 1/12);
//  * FP64: a half's weighted second differences are w / 6 - X1 / 24 with
//    w = (P / D) X0 + 1.5 (Q / D) X1.  FP32 keeps the weights c_k / e_k (the
//    products of e_k would underflow) with fast reciprocals.
template <bool DEV>
__device__ __forceinline__ double weno_flux(const double* f, const double* q, double amx, double* dev) {
    auto k = [](double c) { return c; };
    const WenoHalf<double> p = weno_half(fm(amx, q[0], f[0]), fm(amx, q[1], f[1]), fm(amx, q[2], f[2]),
                                         fm(amx, q[3], f[3]), k);
    const WenoHalf<double> m = weno_half(fm(-amx, q[4], f[4]), fm(-amx, q[3], f[3]), fm(-amx, q[2], f[2]),
                                         fm(-amx, q[1], f[1]), k);
    const double Pp = p.e1 * p.e2, Qp = p.e0 * p.e1, Dp = fm(6.0, p.e0 * p.e2, fm(3.0, Qp, Pp));
    const double Pm = m.e1 * m.e2, Qm = m.e0 * m.e1, Dm = fm(6.0, m.e0 * m.e2, fm(3.0, Qm, Pm));
    // (the weights before their products with X: P X would overflow first)
    const double ip = near_recip(Dp), im = near_recip(Dm);
    const double wp = fm(-1.5, (Qp * ip) * p.X1m, (Pp * ip) * p.X0), wm = fm(-1.5, (Qm * im) * m.X1m, (Pm * im) * m.X0);
    if constexpr (DEV) {
        // largest departure of the nonlinear weights from the linear (0.1, 0.6, 0.3)
        const double w0p = Pp / Dp, w2p = 3.0 * Qp / Dp, w0m = Pm / Dm, w2m = 3.0 * Qm / Dm;
        double d = fmax(fabs(w0p - 0.1), fabs(w2p - 0.3));
        d = fmax(d, fabs(1.0 - w0p - w2p - 0.6));
        d = fmax(d, fmax(fabs(w0m - 0.1), fabs(w2m - 0.3)));
        *dev = fmax(d, fabs(1.0 - w0m - w2m - 0.6));
    }
    const double c = fm(6.0, f[2], f[1]) - f[3];
    return fm(1.0 / 6.0, wm - wp, fm(1.0 / 12.0, c, (1.0 / 24.0) * (m.X1m - p.X1m)));
}

// FP32, of one field (V = float) or two side by side (V = PairF)
template <typename V, typename K>
__device__ __forceinline__ V weno_flux32(const V* f, const V* q, V amx, V minus_amx, K k) {
    const WenoHalf<V> p = weno_half(fm(amx, q[0], f[0]), fm(amx, q[1], f[1]), fm(amx, q[2], f[2]),
                                    fm(amx, q[3], f[3]), k);
    const WenoHalf<V> m = weno_half(fm(minus_amx, q[4], f[4]), fm(minus_amx, q[3], f[3]), fm(minus_amx, q[2], f[2]),
                                    fm(minus_amx, q[1], f[1]), k);
    // twelve times a half's weighted second differences, 2 w0 X0 + (w2 - 1/2) X1
    auto part = [&](const WenoHalf<V>& h) {
        const V a0 = near_recip(h.e0), a1 = k(6.0) * near_recip(h.e1), a2 = k(-3.0) * near_recip(h.e2);
        const V is = near_recip(a0 + a1 - a2);
        return fm((a0 * is) * h.X0, k(2.0), fm(a2, is, k(0.5)) * h.X1m);
    };
    const V c = fm(k(6.0), f[2], f[1]) - f[3];
    return k(1.0 / 12.0) * (c - part(p) + part(m));
}

// Component-wise fifth-order upwind flux with the linear weights
// (0.1, 0.6, 0.3) and the stencil's largest |lambda| as Lax-Friedrichs speed:
// the cheap flux a router sends smooth interfaces to.  f_k, q_k are the
// physical cell differences of one component over the stencil; returns the
// correction to the central F_i (the same form as weno_flux with constant
// weights, whose second differences then add up to one fifth-order stencil).
template <typename R>
__device__ __forceinline__ R linear_flux(const R* f, const R* q, R amx) {
    const R cf = fm(R(7), f[1] - f[3], fm(R(30), f[2], f[4] - f[0]));
    const R cq = fm(R(6), q[2], fm(R(-4), q[1] + q[3], q[0] + q[4]));
    return fm(-amx, cq, cf) * R(1.0 / 60.0);
}

__device__ __forceinline__ constexpr int perm_of(int dir, int v) {
    // line variable v -> conserved index (x: identity; y: rho,My,Mz,Mx,By,Bz,Bx,E;
    // z: rho,Mz,Mx,My,Bz,Bx,By,E)
    return dir == 0 ? v
         : dir == 1 ? (v == 1 ? 2 : v == 2 ? 3 : v == 3 ? 1 : v == 4 ? 5 : v == 5 ? 6 : v == 6 ? 4 : v)
                    : (v == 1 ? 3 : v == 2 ? 1 : v == 3 ? 2 : v == 4 ? 6 : v == 5 ? 4 : v == 6 ? 5 : v);
}

// the inverse: the line variable of a conserved index (the y and z
// permutations are each other's inverses)
__device__ __forceinline__ constexpr int line_var(int dir, int gv) { return perm_of(dir == 0 ? 0 : 3 - dir, gv); }

// A cell: primit (src/ssprk.cpp:479-512) with v from the unfloored density and
// floors on rho and p with E recomputed; eigenst centre fluxes (561-593) with
// the floored values; the eigenvalues in the working type R: FP64 for the plain
// method, FP32 in the mixed one (where they feed only the FP32 characteristic
// part).  Primitives and speeds are formed in the reference's own operations
// and order: where the transverse field vanishes, sqrt(lf^2 - c^2) turns their
// last bit into 1e-8.
template <typename R>
struct CellValues {
    double rho, vx, vy, vz, EE, HH, F[7];
    R lam[7];      // |lambda_m|: every reader takes the magnitude (the LLF speeds)
    float cf[5];   // the routing features' values (MODE 1-3)
};

template <int MODE, typename R>
__device__ __forceinline__ void cell_values(const double* q, double gam, double rhomin, double pgmin, CellValues<R>& o) {
    const double Mx = q[1], My = q[2], Mz = q[3], Bx = q[4], By = q[5], Bz = q[6], gm1 = gam - 1.0;
    double rho = q[0], EE = q[7];
    double irho = recip(rho);
    const double vx = quot(Mx, rho, irho), vy = quot(My, rho, irho), vz = quot(Mz, rho, irho);
    const double vv2 = vx * vx + vy * vy + vz * vz;
    const double BB2 = Bx * Bx + By * By + Bz * Bz;
    double pg = gm1 * (EE - 0.5 * (rho * vv2 + BB2));
    const bool low = rho < rhomin || pg < pgmin;
    if (low) {
        rho = fmax(rhomin, rho);
        pg = fmax(pgmin, pg);
        EE = quot(pg, gm1, recip(gm1)) + 0.5 * (rho * vv2 + BB2);
        irho = recip(rho);
    }
    o.rho = rho; o.vx = vx; o.vy = vy; o.vz = vz; o.EE = EE;
    o.HH = quot(EE + pg, rho, irho);
    const double pt = fm(0.5, BB2, pg);
    const double vdB = fm(vz, Bz, fm(vy, By, vx * Bx));
    o.F[0] = rho * vx;                 // DD (floored) * vx
    o.F[1] = fm(Mx, vx, fm(-Bx, Bx, pt));
    o.F[2] = fm(My, vx, -(Bx * By));
    o.F[3] = fm(Mz, vx, -(Bx * Bz));
    o.F[4] = fm(By, vx, -(Bx * vy));
    o.F[5] = fm(Bz, vx, -(Bx * vz));
    o.F[6] = fm(EE + pt, vx, -(Bx * vdB));
    R bbn2, bnx2, cs2;
    if constexpr (std::is_same<R, double>::value) {
        bbn2 = quot(BB2, rho, irho);
        bnx2 = quot(Bx * Bx, rho, irho);
        cs2 = gam * fabs(quot(pg, rho, irho));
    } else {
        const R irR = R(irho);
        bbn2 = R(BB2) * irR;
        bnx2 = R(Bx * Bx) * irR;
        cs2 = R(gam) * fabs(R(pg) * irR);
    }
    const R bc = bbn2 + cs2;
    const R rt = root(bc * bc - R(4) * bnx2 * cs2);
    const R lf = root(R(0.5) * (bc + rt));
    const R la = root(bnx2);
    const R ls = root(R(0.5) * (bc - rt));
    const R vxR = R(vx);
    o.lam[0] = fabs(vxR - lf); o.lam[1] = fabs(vxR - la); o.lam[2] = fabs(vxR - ls); o.lam[3] = fabs(vxR);
    o.lam[4] = fabs(vxR + ls); o.lam[5] = fabs(vxR + la); o.lam[6] = fabs(vxR + lf);
    if constexpr (MODE != 0) {
        // (the guard needs density and pressure only)
        o.cf[0] = (float)rho; o.cf[1] = (float)pg;
        if constexpr (MODE == 3) { o.cf[2] = sqrtf((float)BB2); o.cf[3] = sqrtf((float)vv2); o.cf[4] = (float)lf; }
    }
}

// Values per lane to tensor memory, and TIMES groups of N, STEP values apart,
// from it
__device__ __forceinline__ void put_five(uint32_t at, const double* v) {
    uint32_t w[10];
#pragma unroll
    for (int i = 0; i < 5; ++i) { w[2 * i] = (uint32_t)__double2loint(v[i]); w[2 * i + 1] = (uint32_t)__double2hiint(v[i]); }
    tmem_store<8>(at, w);
    tmem_store<2>(at + 8, w + 8);
}
__device__ __forceinline__ void put_ten(uint32_t at, const float* v) {
    uint32_t w[10];
#pragma unroll
    for (int i = 0; i < 10; ++i) w[i] = (uint32_t)__float_as_int(v[i]);
    tmem_store<8>(at, w);
    tmem_store<2>(at + 8, w + 8);
}
template <int N, int TIMES, int STEP> __device__ __forceinline__ void get_values(uint32_t at, double* v) {
    uint32_t w[2 * N * TIMES];
#pragma unroll
    for (int i = 0; i < TIMES; ++i) tmem_load<2 * N>(at + 2 * STEP * i, w + 2 * N * i);
    tmem_wait_loads<2 * N * TIMES>(w);
#pragma unroll
    for (int i = 0; i < N * TIMES; ++i) v[i] = __hiloint2double((int)w[2 * i + 1], (int)w[2 * i]);
}
template <int N, int TIMES, int STEP> __device__ __forceinline__ void get_values(uint32_t at, float* v) {
    uint32_t w[N * TIMES];
#pragma unroll
    for (int i = 0; i < TIMES; ++i) tmem_load<N>(at + STEP * i, w + N * i);
    tmem_wait_loads<N * TIMES>(w);
#pragma unroll
    for (int i = 0; i < N * TIMES; ++i) v[i] = __int_as_float((int)w[i]);
}

// The interface between the first two cells of the window at P (the lane's
// column): eigen-system, projection, WENO5 of the seven fields and
// back-projection.  out: the upwind correction to the left cell's flux.
// before_back runs before the back-projection.
template <typename R>
struct FaceValues {
    R out[7];
    R rho, hvv, bbn2;    // of the mean state (label collection)
    float departure;     // largest departure of the nonlinear weights (label collection)
};

template <int NL, int CP, int CB, int CD, int CL, int MODE, typename R, typename Before>
__device__ __forceinline__ void face_values(const double* sP, const double* sB, const typename Diff<R>::T* sD, const R* sL,
                                            uint32_t tm, R gamR,
                                            R gam2, FaceValues<R>& o, Before before_back) {
    if constexpr (MODE == 3) o.departure = 0.0f;
    const R gam0 = R(1) - gamR;
    // eigen-system of the arithmetic mean of the two cells'
    // primitives (src/ssprk.cpp:610-660)
    auto mean = [&](const double* s) { return R(0.5 * (s[0] + s[NL])); };
    const R rho = mean(sP), vx = mean(sP + CP), By = mean(sP + 2 * CP), Bz = mean(sP + 3 * CP);
    const R HH = mean(sP + 4 * CP);
    const R vy = mean(sB + NL), vz = mean(sB + CB + NL), Bx = mean(sB + 2 * CB + NL);
    const R vv2 = vx * vx + vy * vy + vz * vz;
    const R BB2 = Bx * Bx + By * By + Bz * Bz;
    R bbn2, bnx2;
    const R isqr = root_inverse(rho);
    if constexpr (std::is_same<R, double>::value) {
        const double irho = recip(rho);
        bbn2 = quot(BB2, rho, irho);
        bnx2 = quot(Bx * Bx, rho, irho);
    } else {
        const R irho = isqr * isqr;
        bbn2 = BB2 * irho;
        bnx2 = Bx * Bx * irho;
    }
    const R cs2 = (gamR - R(1)) * (HH - R(0.5) * (vv2 + bbn2));
    const R cs = root(cs2);
    const R bc = bbn2 + cs2;
    const R rt = root(bc * bc - R(4) * bnx2 * cs2);
    const R lf = root(R(0.5) * (bc + rt));
    const R ls = root(R(0.5) * (bc - rt));
    const R Bt2 = By * By + Bz * Bz;
    const bool some = Bt2 >= R(1.0e-30);
    const R ib = root_inverse(Bt2), h = R(0.70710678118654752440);
    const R bty = some ? By * ib : h, btz = some ? Bz * ib : h;
    const R df = lf * lf - ls * ls;
    const bool wide = df >= R(1.0e-30);
    const R idf = root_inverse(df);
    const R af = wide ? root(cs2 - ls * ls) * idf : R(1), as = wide ? root(lf * lf - cs2) * idf : R(1);
    const R hvv = R(0.5) * vv2, sqr = rho * isqr;
    R ics2;
    if constexpr (std::is_same<R, double>::value) ics2 = recip(cs2);
    else ics2 = near_recip(cs2);
    const R sgnB = (Bx >= R(0)) ? R(1) : R(-1);
    const R btv = fm(bty, vy, btz * vz);

    // Left eigenvectors (src/ssprk.cpp:662-726) applied to the
    // stencil's differences.  The four magnetosonic rows are
    // even +- odd combinations of four products with D that do
    // not depend on the field,
    //   e = (-v^2/2, v, B_t, -1).D    b = beta.(D4, D5)
    //   x = D1 - vx D0                t = beta.(D2, D3) - beta.v D0
    // with coefficients below for the fast and the slow pair; the
    // entropy row is D0 + s e, and the two Alfven rows are even
    // +- odd in (beta x) the transverse momenta and fields.
    // (The reference turns the fast or slow rows and columns by
    // sgn(B_t), src/ssprk.cpp:789-818; the field's flux is odd in
    // its row, so the sign cancels exactly from row and column.)
    auto speed = [&](int m) -> R {   // the stencil's largest |lambda_m|
        const R* sm = sL + m * CL;
        R amx = sm[0];
#pragma unroll
        for (int k = 1; k < 6; ++k) amx = larger(amx, sm[k * NL]);
        return amx;
    };
    const R hn = R(0.5) * ics2;   // the rows' normalisation
    const R cen = -gam0 * ics2;
    // Three pairs of fields: fast (0, 6), slow (2, 4), Alfven (1, 5), and the
    // entropy field.  The differences are read once for the magnetosonic and
    // entropy fields; their products (50 values a lane) wait in tensor memory
    // for the loop over the pairs, whose two WENO fluxes are then the only copy
    // of that code but one.  Held in registers the products leave room for 8
    // warps per SM instead of 12, and unroll the loop past the instruction
    // caches; formed again for each pair they cost 120 FP64 operations and 70
    // shared-memory loads more.  The Alfven pair shares no product.
    R F0, F1, F2, F3, F4, F5, F6;
    {
        if constexpr (std::is_same<R, double>::value) {
            const double cef = hn * gam0 * af, cbf = hn * cs * as * sqr, cxf = hn * lf * af, ctf = -hn * as * ls * sgnB;
            const double ces = hn * gam0 * as, cbs = -hn * cs * af * sqr, cxs = hn * ls * as, cts = hn * af * lf * sgnB;
#pragma unroll 1
            for (int h = 0; h < 2; ++h)   // fluxes, states
#pragma unroll
                for (int k = 0; k < 5; ++k) {
                    const double* D = sD + (7 * h) * CD + k * NL;
                    const double D0 = D[0], D1 = D[CD], D2 = D[2 * CD], D3 = D[3 * CD], D4 = D[4 * CD], D5 = D[5 * CD];
                    const double e = fm(-hvv, D0, fm(vx, D1, fm(vy, D2, fm(vz, D3, fm(By, D4, fm(Bz, D5, -D[6 * CD]))))));
                    const double b = fm(bty, D4, btz * D5);
                    const double x = fm(-vx, D0, D1);
                    const double t = fm(bty, D2, fm(btz, D3, -btv * D0));
                    const double fe = fm(cef, e, cbf * b), fo = fm(cxf, x, ctf * t);
                    const double se = fm(ces, e, cbs * b), so = fm(cxs, x, cts * t);
                    const double v[5] = {fe - fo, fe + fo, se - so, se + so, fm(cen, e, D0)};
                    put_five(tm + (h * 5 + k) * 10, v);
                }
        } else {
            using P = PairF;
            const P cef = both(-hn * gam0 * af), cbf = both(hn * cs * as * sqr), cxf = both(hn * lf * af),
                    ctf = both(-hn * as * ls * sgnB);
            const P ces = both(-hn * gam0 * as), cbs = both(-hn * cs * af * sqr), cxs = both(hn * ls * as),
                    cts = both(hn * af * lf * sgnB);
            const P cen_ = both(-cen), h2 = both(hvv), nvx = both(-vx), nvy = both(-vy), nvz = both(-vz), nBy = both(-By),
                    nBz = both(-Bz), by = both(bty), bz = both(btz), nbv = both(-btv);
#pragma unroll
            for (int k = 0; k < 5; ++k) {
                const auto* D = sD + k * NL;
                const P D0 = from_mem(D[0]), D1 = from_mem(D[CD]), D2 = from_mem(D[2 * CD]), D3 = from_mem(D[3 * CD]),
                        D4 = from_mem(D[4 * CD]), D5 = from_mem(D[5 * CD]), D6 = from_mem(D[6 * CD]);
                const P ne = fm(h2, D0, fm(nvx, D1, fm(nvy, D2, fm(nvz, D3, fm(nBy, D4, fm(nBz, D5, D6))))));   // -e
                const P b = fm(by, D4, bz * D5);
                const P x = fm(nvx, D0, D1);
                const P t = fm(by, D2, fm(bz, D3, nbv * D0));
                R v[10], ef, eq, of, oq;   // per pair: flux minus, plus, state minus, plus; then the entropy field's
                split(fm(cef, ne, cbf * b), ef, eq);
                split(fm(cxf, x, ctf * t), of, oq);
                v[0] = ef - of; v[1] = ef + of; v[2] = eq - oq; v[3] = eq + oq;
                split(fm(ces, ne, cbs * b), ef, eq);
                split(fm(cxs, x, cts * t), of, oq);
                v[4] = ef - of; v[5] = ef + of; v[6] = eq - oq; v[7] = eq + oq;
                split(fm(cen_, ne, D0), v[8], v[9]);
                put_ten(tm + k * 10, v);
            }
        }
        tmem_wait_stores();
    }
#pragma unroll 1
    for (int pair = 0; pair < 3; ++pair) {
        R w[20];   // per difference: flux minus, plus, state minus, plus
        if (pair < 2) {
            if constexpr (std::is_same<R, double>::value) {
                double v[20];   // [flux, state][difference][minus, plus]
                get_values<2, 10, 5>(tm + pair * 4, v);
#pragma unroll
                for (int k = 0; k < 5; ++k) {
                    w[4 * k] = v[2 * k]; w[4 * k + 1] = v[2 * k + 1];
                    w[4 * k + 2] = v[10 + 2 * k]; w[4 * k + 3] = v[11 + 2 * k];
                }
            } else {
                get_values<4, 5, 10>(tm + pair * 4, w);
            }
        } else if constexpr (std::is_same<R, double>::value) {
            const double cv = 0.5 * fm(btz, vy, -(bty * vz)), cy = 0.5 * bty, cz = 0.5 * btz;
            const double cm = sgnB * sqr, cby = cm * cy, cbz = cm * cz;
#pragma unroll
            for (int h = 0; h < 2; ++h)
#pragma unroll
                for (int k = 0; k < 5; ++k) {
                    const double* D = sD + (7 * h) * CD + k * NL;
                    const double ev = fm(cv, D[0], fm(cy, D[3 * CD], -(cz * D[2 * CD])));
                    const double od = fm(cbz, D[4 * CD], -(cby * D[5 * CD]));
                    w[4 * k + 2 * h] = ev - od;
                    w[4 * k + 2 * h + 1] = ev + od;
                }
        } else {
            using P = PairF;
            const R cz = R(0.5) * btz, cm = sgnB * sqr;
            const P cv = both(R(0.5) * fm(btz, vy, -(bty * vz))), cy = both(R(0.5) * bty), ncz = both(-cz);
            const P cbz = both(cm * cz), ncby = both(-cm * (R(0.5) * bty));
#pragma unroll
            for (int k = 0; k < 5; ++k) {
                const auto* D = sD + k * NL;
                const P ev = fm(cv, from_mem(D[0]), fm(cy, from_mem(D[3 * CD]), ncz * from_mem(D[2 * CD])));
                const P od = fm(cbz, from_mem(D[4 * CD]), ncby * from_mem(D[5 * CD]));
                R ef, eq, of, oq;
                split(ev, ef, eq);
                split(od, of, oq);
                w[4 * k] = ef - of; w[4 * k + 1] = ef + of; w[4 * k + 2] = eq - oq; w[4 * k + 3] = eq + oq;
            }
        }
        const int m = pair == 0 ? 0 : 3 - pair;   // 0, 2, 1
        R lo, hi;
        if constexpr (std::is_same<R, double>::value) {
            double f[5], q[5], d = 0.0;
#pragma unroll
            for (int k = 0; k < 5; ++k) { f[k] = w[4 * k]; q[k] = w[4 * k + 2]; }
            lo = weno_flux<MODE == 3>(f, q, speed(m), &d);
            if constexpr (MODE == 3) o.departure = fmaxf(o.departure, (float)d);
#pragma unroll
            for (int k = 0; k < 5; ++k) { f[k] = w[4 * k + 1]; q[k] = w[4 * k + 3]; }
            hi = weno_flux<MODE == 3>(f, q, speed(6 - m), &d);
            if constexpr (MODE == 3) o.departure = fmaxf(o.departure, (float)d);
        } else {
            PairF f[5], q[5];
#pragma unroll
            for (int k = 0; k < 5; ++k) { f[k] = make_pair(w[4 * k], w[4 * k + 1]); q[k] = make_pair(w[4 * k + 2], w[4 * k + 3]); }
            const float s0 = speed(m), s1 = speed(6 - m);
            split(weno_flux32(f, q, make_pair(s0, s1), make_pair(-s0, -s1), [](double c) { return both((float)c); }), lo, hi);
        }
        if (pair == 0) { F0 = lo; F6 = hi; }
        else if (pair == 1) { F2 = lo; F4 = hi; }
        else { F1 = lo; F5 = hi; }
    }
    {
        R w[10];
        const R s = speed(3);
        if constexpr (std::is_same<R, double>::value) {
            double d = 0.0;
            get_values<1, 10, 5>(tm + 8, w);
            F3 = weno_flux<MODE == 3>(w, w + 5, s, &d);
            if constexpr (MODE == 3) o.departure = fmaxf(o.departure, (float)d);
        } else {
            float f[5], q[5];
            get_values<2, 5, 10>(tm + 8, w);
#pragma unroll
            for (int k = 0; k < 5; ++k) { f[k] = w[2 * k]; q[k] = w[2 * k + 1]; }
            F3 = weno_flux32(f, q, s, -s, [](double c) { return (float)c; });
        }
    }

    before_back();
    // Right eigenvectors (src/ssprk.cpp:729-787) by the same
    // symmetry: sums and differences of the paired fields
    const R fs = af * (F0 + F6), ss = as * (F2 + F4);
    const R fd = af * lf * (F6 - F0), sd = as * ls * (F4 - F2);
    const R w = sgnB * fm(as * ls, F0 - F6, (af * lf) * (F4 - F2));
    const R u = F1 + F5, du = sgnB * isqr * (F1 - F5);
    const R bq = cs * isqr * fm(as, F0 + F6, -af * (F2 + F4));
    R* out = o.out;
    out[0] = fs + ss + F3;
    out[1] = fm(vx, out[0], fd + sd);
    out[2] = fm(vy, out[0], fm(bty, w, -(btz * u)));
    out[3] = fm(vz, out[0], fm(btz, w, bty * u));
    out[4] = fm(bty, bq, -(btz * du));
    out[5] = fm(btz, bq, bty * du);
    const R gc = gam2 * cs2;
    out[6] = fm(hvv, out[0], fm(lf * lf - gc, fs, fm(ls * ls - gc, ss, fm(vx, fd + sd,
                fm(btv, w, fm(bty, vz, -(btz * vy)) * u)))));
    if constexpr (MODE == 3) { o.rho = rho; o.hvv = hvv; o.bbn2 = bbn2; }
}

constexpr uint32_t kWaitLimit = 1u << 26;   // bounded TMA wait (~seconds), then flag and skip

// How a direction's lines are cut into work items (one warp each).  Lines of
// the x sweep start at j = 3; lines of the y/z sweeps are NL consecutive i
// from a multiple of NL (masked ghost lines at the ends), so that a tile row
// is a whole 32-byte sector for NL = 4 and the innermost TMA coordinate is
// even.  A segment of `chunks` chunks advances chunks * W - ov cells: its
// first interface repeats the segment before's last (ov = 1; in x ov = 2 and
// the first interface is -1, which keeps the raw tiles' x even).
template <int DIR, int NL>
struct Cut {
    static constexpr int W = 32 / NL, ov = DIR == 0 ? 2 : 1, f0 = DIR == 0 ? -1 : 0, line0 = DIR == 0 ? 3 : 0;
    int n, nt1, nt2, groups, segs;
    __host__ __device__ Cut(const Grid& g, int chunks) {
        n = DIR == 0 ? g.nx : DIR == 1 ? g.ny : g.nz;
        nt1 = DIR == 0 ? g.ny : g.nx;
        nt2 = DIR == 2 ? g.ny : g.nz;
        groups = (3 + nt1 - line0 + NL - 1) / NL;
        const int step = chunks * W - ov;
        segs = (n + step - 1) / step;
    }
    __host__ __device__ long long items() const { return (long long)groups * segs * nt2; }
};

template <bool FIRST, typename A, typename B>
__device__ __forceinline__ auto& either(A& a, B& b) {
    if constexpr (FIRST) return a; else return b;
}

// MODE 0: plain method.  1: learned routing (network + guard).  2: guard-only
// routing (the ablation).  3: plain method that also records features and
// nonlinear-weight labels of sampled tiles for training.
//
// ENS: one launch advances this sweep for every member of a batched
// ensemble; the global item index runs over the members' items in order, and
// each item reads its member's arguments from the ensemble table.
template <int DIR, int NL, int WPB, typename R, int MINB, int MODE, bool ENS = false>
__global__ void __launch_bounds__(32 * WPB, MINB) k_sweep(const __grid_constant__ SweepArgs a0) {
    static_assert(!ENS || MODE == 0, "ensembles run the plain method");
    static_assert(MODE != 3 || std::is_same<R, double>::value, "labels are recorded by the FP64 method");
    constexpr bool ROUTED = MODE == 1 || MODE == 2;
    using M = WarpMem<DIR, NL, R, MODE>;
    using CUT = Cut<DIR, NL>;
    constexpr int W = M::W, CD = M::CD, CL = M::CL, CP = M::CP, CB = M::CB;
    constexpr unsigned ALL = 0xffffffffu;
    extern __shared__ __align__(128) unsigned char smem_raw[];
    const int lane = threadIdx.x & 31, warp = __shfl_sync(ALL, threadIdx.x >> 5, 0);   // (uniform in the warp)
    const int l = lane % NL, j = lane / NL;   // the lane's line and its place along the chunk
    // TMA destinations need 128-byte alignment: align the carve-up base
    unsigned char* sm = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(smem_raw) + 127) & ~uintptr_t(127)) +
                        warp * M::bytes;
    const double* sRaw = reinterpret_cast<const double*>(sm + M::bRaw);
    const double* sOp = reinterpret_cast<const double*>(sm + M::bOp);
    // window arrays, at the lane's column: the cell s places after the first
    // of the window is s * NL further (a new cell is H * NL further)
    double* sP = reinterpret_cast<double*>(sm + M::bP) + lane;
    double* sB = reinterpret_cast<double*>(sm + M::bB) + lane;
    double* sF = reinterpret_cast<double*>(sm + M::bF) + lane;
    using DT = typename Diff<R>::T;
    DT* sD = reinterpret_cast<DT*>(sm + M::bD) + lane;
    R* sL = reinterpret_cast<R*>(sm + M::bL) + lane;
    float* sC = reinterpret_cast<float*>(sm + M::bC) + lane;
    double* sU = reinterpret_cast<double*>(sm + M::bU) + l;
    double* sX = reinterpret_cast<double*>(sm + M::bX) + l;
    uint64_t* bars = reinterpret_cast<uint64_t*>(sm + M::bBar);
    volatile long long* sSpot = reinterpret_cast<long long*>(sm + M::bS) + lane;

    // tensor memory: a warp reaches lanes 32 (warp % 4) on, and the warps that
    // share them take columns of their own.  (The runtime's occupancy calculator
    // answers one block per SM for this kernel with blocks of four warps too, whose
    // registers and shared memory allow more, and a sweep then takes 4.1 ms: the
    // block holds all of the SM's warps.)
    static_assert(WPB % 4 == 0, "blocks of whole tensor memory lanes");
    constexpr int kValues = 50, kPer = (kValues * (int)sizeof(R) / 4 + 3) / 4 * 4;   // columns per warp
    constexpr int kUsed = WPB / 4 * kPer, kColumns = kUsed <= 128 ? 128 : kUsed <= 256 ? 256 : 512;
    static_assert(kUsed <= 512, "tensor memory has 512 columns");
    __shared__ uint32_t s_tmem;
    if (warp == 0) tmem_alloc<kColumns>(&s_tmem);
    __syncthreads();
    const uint32_t tm = s_tmem + ((uint32_t)(32 * (warp % 4)) << 16) + (uint32_t)(warp / 4 * kPer);

    // component r's k-th difference of the lane's stencil, flux and state
    [[maybe_unused]] auto diff_at = [&](int r, int k, R& f, R& q) {
        if constexpr (std::is_same<R, double>::value) { f = sD[r * CD + k * NL]; q = sD[(7 + r) * CD + k * NL]; }
        else { const float2 d = sD[r * CD + k * NL]; f = d.x; q = d.y; }
    };

    // One place of the march: a chunk (first interface fb) of an item's segment
    // (last chunk's first interface fend, first owned interface lo; the chunk
    // before the first, with the five cells before the first interface, has no
    // interface yet).  FP64 at 12 warps keeps it in shared memory and reads it
    // again where it is used: held across a chunk it takes 15 of 168 registers
    // (256^3 sweep 2.55 ms with it, 2.45 without; the mixed method has them to
    // spare, 0.76 against 0.79 ms at 192^3).
    struct Place { int fb, fend, lo, t1_0, t2, item; const SweepArgs* a; };
    constexpr bool FREE_REGS = sizeof(R) == 4 || WPB <= 8;
    __shared__ Place s_place[FREE_REGS ? 1 : WPB];
    Place r_place;
    volatile Place& m_place = s_place[FREE_REGS ? 0 : warp];
    auto& here = either<FREE_REGS>(r_place, m_place);
    auto first_chunk = [](int lo, int fb) { return fb >= lo - CUT::ov; };   // an interface chunk
    auto member_of = [&](long long item) -> int {
        int lo = 0, hi = a0.ens_n - 1;   // last member whose first item is <= item
        while (lo < hi) {
            const int mid = (lo + hi + 1) >> 1;
            if (a0.ens_tile_start[mid] <= item) lo = mid; else hi = mid - 1;
        }
        return lo;
    };
    // (a sweep has fewer than 2^31 items)
    const int nitems = ENS ? (int)a0.ens_tile_start[a0.ens_n] : (int)CUT(a0.g, a0.seg_chunks).items();
    // the item's first place; items of members that are not stepping are skipped whole
    auto enter = [&](int item) -> Place {
        const int chunks = a0.seg_chunks, stride = (int)gridDim.x * WPB;
        Place p{0, 0, 0, 0, 0, item, &a0};
        int li = item;
        if constexpr (ENS) {
            while (item < nitems) {
                const int m = member_of(item);
                if (a0.ens_active[m]) {
                    p.a = a0.ens_tab + ((long long)m * a0.ens_stride + a0.ens_off + a0.ens_par[m]);
                    li = item - (int)a0.ens_tile_start[m];
                    break;
                }
                const int end = (int)a0.ens_tile_start[m + 1];
                item += (end - item + stride - 1) / stride * stride;
            }
            p.item = item;
        }
        if (item >= nitems) return p;
        const CUT c(p.a->g, chunks);
        // line groups fastest: neighbouring lines are worked on at the same time
        const unsigned u = (unsigned)li, r = u / (unsigned)c.groups;
        p.t1_0 = CUT::line0 + NL * (int)(u - r * (unsigned)c.groups);
        const unsigned seg = r / (unsigned)c.nt2;
        p.t2 = 3 + (int)(r - seg * (unsigned)c.nt2);
        const int fa = CUT::f0 + (int)seg * (chunks * W - CUT::ov), all = (c.n - fa) / W;   // chunk of the last interface n
        p.lo = seg == 0 ? 0 : fa + CUT::ov;
        p.fb = fa - W;
        p.fend = fa + (all < chunks - 1 ? all : chunks - 1) * W;
        return p;
    };

    if (lane == 0) {
        mbar_init(&bars[0], 1);
        mbar_init(&bars[1], 1);
        fence_barrier_init();
    }
    __syncwarp();
    bool issued = true;            // lane 0's view
    unsigned par = 0u, pend = 0u;  // per barrier: phase parity, copy in flight (lane 0's view)
    // TMA loads (lane 0): the new cells of a place (which == 0), or the update
    // operand of its chunk (which == 1): cells fb+2 .. fb+W+1
    auto issue = [&](int which, const SweepArgs* a, int fb, int t1_0, int t2) -> bool {
        const int along = which == 0 ? fb + 5 : DIR == 0 ? fb + 1 : fb + 2;
        const int c0 = DIR == 0 ? along : t1_0;
        const int c1 = DIR == 0 ? t1_0 : DIR == 1 ? along : t2;
        const int c2 = DIR == 2 ? along : t2;
        if (c0 & 1) {   // never issue a misaligned tensor copy
            atomicOr(a->status, HOW_STATUS_TMA_ALIGN);
            return false;
        }
        pend |= 1u << which;
        mbar_arrive_expect_tx(&bars[which], which == 0 ? M::raw_bytes : M::op_bytes);
        tma_load_4d(sm + (which == 0 ? M::bRaw : M::bOp), which == 0 ? &a->tm_in : &a->tm_out, &bars[which], c0, c1, c2,
                    0);
        return true;
    };
    // the lanes' tile waits are bounded (a failure-detection test can make
    // them give up at once); on expiry the warp leaves, lane 0 after a
    // bounded wait for its copies in flight
    const uint32_t wait_limit = a0.wait_expire ? 0u : kWaitLimit;
    auto arrived = [&](int which) -> bool {
        const bool ok = issued && mbar_wait_bounded(&bars[which], (par >> which) & 1u, wait_limit);
        if (__all_sync(ALL, ok)) {
            par ^= 1u << which;
            pend &= ~(1u << which);
            return true;
        }
        if (lane == 0) {
            atomicOr(a0.status, HOW_STATUS_TMA_TIMEOUT);
            for (int b = 0; b < 2; ++b)
                if ((pend >> b) & 1u) mbar_wait_bounded(&bars[b], (par >> b) & 1u, kWaitLimit);
        }
        return false;
    };

    // optional per-phase cycle accounting of lane 0 (prof != nullptr), summed
    // in shared memory and added to the counters at the end
    __shared__ unsigned long long s_prof[WPB][12];
    const bool timed = a0.prof != nullptr && lane == 0;
    if (timed)
        for (int k = 0; k < 12; ++k) s_prof[warp][k] = 0ull;
    __shared__ unsigned s_clock[WPB];
    if (timed) s_clock[warp] = (unsigned)clock();
    auto mark = [&](int ph) {
        if (a0.prof != nullptr && lane == 0) {
            s_prof[warp][ph] += (unsigned)clock() - s_clock[warp];
            if (ph == 10) ++s_prof[warp][11];   // chunks
            s_clock[warp] = (unsigned)clock();
        }
    };
    unsigned n_full = 0, n_cheap = 0;   // routed interfaces of this warp

    {
        // (items go to all blocks before a block gets a second one)
        const Place p = enter(warp * (int)gridDim.x + (int)blockIdx.x);
        if constexpr (FREE_REGS) r_place = p;
        else if (lane == 0) s_place[warp] = p;
        if (lane == 0) {
            if (p.item < nitems) issued = issue(0, p.a, p.fb, p.t1_0, p.t2);
        }
        __syncwarp();
    }
    while (here.item < nitems) {
        const SweepArgs& a = ENS ? *here.a : a0;
        const Grid& g = a.g;
        const int n = DIR == 0 ? g.nx : DIR == 1 ? g.ny : g.nz;
        const int nt1 = DIR == 0 ? g.ny : g.nx;
        const double gam = a.gam, gm1 = gam - 1.0;
        // where the lane is: its face, its line, and whether its segment owns
        // the face (all from its second, in the x sweep third, interface on,
        // and face 0)
        struct Spot { int f, t1, t2; bool owned; };
        auto spot = [&]() -> Spot {
            Spot o;
            o.f = here.fb + j; o.t1 = here.t1_0 + l; o.t2 = here.t2;
            o.owned = o.t1 >= 3 && o.t1 <= nt1 + 2 && o.f <= n && o.f >= here.lo;
            return o;
        };
        // an owned face's offset (and that of the cell left of it), for the
        // stores: doubled, odd where the cell is the line's own (f >= 1); -1
        // for a face the lane does not own
        [[maybe_unused]] long long r_spot;
        {
            const Spot o = spot();
            const long long at = DIR == 0 ? g.idx(o.f + 2, o.t1, o.t2)
                               : DIR == 1 ? g.idx(o.t1, o.f + 2, o.t2) : g.idx(o.t1, o.t2, o.f + 2);
            const long long code = o.owned ? 2 * at + (o.f >= 1 ? 1 : 0) : -1;
            if constexpr (FREE_REGS) r_spot = code; else *sSpot = code;
        }
        auto spot_code = [&]() -> long long { if constexpr (FREE_REGS) return r_spot; else return *sSpot; };

        // -------------------------------------------------------------- load
        if (!arrived(0)) break;   // results void; host sees the status
        double q[8];
#pragma unroll
        for (int v = 0; v < 8; ++v) {
            const int gv = perm_of(DIR, v);
            q[v] = DIR == 0 ? sRaw[(gv * NL + l) * W + j] : sRaw[gv * 32 + lane];
        }
        __syncwarp();   // every read of the raw tile, and of the window's new columns, is done
        const bool faces = first_chunk(here.lo, here.fb);
        {
            const int fb = here.fb, t1_0 = here.t1_0, t2 = here.t2;
            if (fb < here.fend) {
                if (lane == 0) {
                    fence_proxy_async_smem();
                    if (faces) issued = issue(1, &a, fb, t1_0, t2) && issued;
                    issued = issue(0, &a, fb + W, t1_0, t2) && issued;
                }
            } else {
                const Place nx = enter(here.item + (int)gridDim.x * WPB);
                if (lane == 0) {
                    fence_proxy_async_smem();
                    if (faces) issued = issue(1, &a, fb, t1_0, t2) && issued;
                    if (nx.item < nitems) issued = issue(0, nx.a, nx.fb, nx.t1_0, nx.t2) && issued;
                }
            }
        }
        // MODE 1: the routing pass's decisions of the lane's face and its two
        // neighbours along the sweep (decisions formed once per step stay
        // valid while a feature moves by up to one cell)
        bool flagged = false;
        if constexpr (MODE == 1) {
            const Spot o = spot();
            if (faces && o.t1 >= 3 && o.t1 <= nt1 + 2) {
                const unsigned char* d = a.route_next + route_line(g, DIR, o.t1, o.t2) + (o.f + 2);
                unsigned any = 0u;
#pragma unroll
                for (int s = -1; s <= 1; ++s)
                    if (o.f + s >= 0 && o.f + s <= n) any |= d[s];
                flagged = any != 0u;
            }
        }
        mark(0);

        // -------------------------------------------------------------- cell
        CellValues<R> cv;
        cell_values<MODE>(q, gam, a.rhomin, a.pgmin, cv);
        {
            constexpr int nP = M::HP * NL, nB = M::HB * NL, nD = M::HD * NL, nL = M::HL * NL;
            const double By = q[5], Bz = q[6];
            sP[0 * CP + nP] = cv.rho; sP[1 * CP + nP] = cv.vx; sP[2 * CP + nP] = By; sP[3 * CP + nP] = Bz;
            sP[4 * CP + nP] = cv.HH;
            sB[0 * CB + nB] = cv.vy; sB[1 * CB + nB] = cv.vz; sB[2 * CB + nB] = q[4];
#pragma unroll
            for (int r = 0; r < 7; ++r) sF[r * CP + nP] = cv.F[r];
#pragma unroll
            for (int m = 0; m < 7; ++m) sL[m * CL + nL] = cv.lam[m];
            if constexpr (MODE != 0) {
#pragma unroll
                for (int r = 0; r < M::NCF; ++r) sC[r * CL + nL] = cv.cf[r];
            }
            // differences of (F, q_proj) to the cell before, formed in FP64
            // and stored in the working type.  The cell before: from the
            // window, but momentum and energy from the neighbouring lane (or
            // what the last lanes of the chunk before left)
            double u[4] = {q[1], q[2], q[3], cv.EE}, before[14];
#pragma unroll
            for (int v = 0; v < 4; ++v) {
                const double up = __shfl_up_sync(ALL, u[v], NL);
                before[v == 3 ? 13 : 8 + v] = j == 0 ? sU[v * NL] : up;
            }
            __syncwarp();
#pragma unroll
            for (int r = 0; r < 7; ++r) before[r] = sF[r * CP + nP - NL];
            before[7] = sP[0 * CP + nP - NL]; before[11] = sP[2 * CP + nP - NL]; before[12] = sP[3 * CP + nP - NL];
            const double now[14] = {cv.F[0], cv.F[1], cv.F[2], cv.F[3], cv.F[4], cv.F[5], cv.F[6],
                                    cv.rho, q[1], q[2], q[3], By, Bz, cv.EE};
#pragma unroll
            for (int v = 0; v < 7; ++v) {
                const R d = R(now[v] - before[v]), e = R(now[7 + v] - before[7 + v]);
                if constexpr (std::is_same<R, double>::value) { sD[v * CD + nD] = d; sD[(7 + v) * CD + nD] = e; }
                else sD[v * CD + nD] = make_float2(d, e);
            }
            if (j == W - 1) {
#pragma unroll
                for (int v = 0; v < 4; ++v) sU[v * NL] = u[v];
            }
            __syncwarp();
        }
        mark(1);

        if (faces) {
            // ---------------------------------------------------------- face
            double fl[7];   // the interface's flux, rows rho, Mx, My, Mz, By, Bz, E of the line frame
            bool full = true;
            if constexpr (ROUTED) {
                float rr[6], pp[6];
#pragma unroll
                for (int s = 0; s < 6; ++s) { rr[s] = sC[s * NL]; pp[s] = sC[CL + s * NL]; }
                // the hard guard on this stage's state, whatever the stage
                // the network's decisions were formed at
                full = flagged || router_guard_rp(rr, pp, (float)a.rhomin, (float)a.pgmin, a.guard_jump, a.guard_floor);
                const Spot o = spot();
                const unsigned mf = __ballot_sync(ALL, o.owned && full), mc = __ballot_sync(ALL, o.owned && !full);
                n_full += __popc(mf);
                n_cheap += __popc(mc);
                if constexpr (MODE == 2) {
                    if (o.owned) a.route_next[route_line(g, DIR, o.t1, o.t2) + (o.f + 2)] = (unsigned char)(full ? 1 : 0);
                }
            }
            // the stage input of the cell left of the interface, which the
            // first sweep of a stage combines with the RK base (issued before
            // the back-projection, used at the update)
            // (with this stage's dt / d, per member in an ensemble)
            double prev[8], dtdl;
            auto load_prev = [&] {
                dtdl = *a.dtdl;
                const long long code = spot_code();
                if (a.mode == 1 && (code & 1) && code > 0) {
                    const double* in = a.qprev + (code >> 1);
#pragma unroll
                    for (int gv = 0; gv < 8; ++gv, in += g.fs) prev[line_var(DIR, gv)] = *in;
                }
            };
            float lab_w = 0.0f, lab_f = 0.0f;   // MODE 3: largest weight and flux departures

            // a warp takes the full path when one of its faces does (shocks
            // are surfaces: its 32 faces are neighbours), the linear one when
            // one of its faces does; a face keeps the result of its own
            if (!ROUTED || __any_sync(ALL, full)) {
                FaceValues<R> fv;
                face_values<NL, CP, CB, CD, CL, MODE>(sP, sB, sD, sL, tm, R(gam), R(a.gam2), fv, load_prev);
                if constexpr (MODE == 3) lab_w = fv.departure;
#pragma unroll
                for (int r = 0; r < 7; ++r) {
                    fl[r] = (double)fv.out[r] + sF[r * CP];
                    if constexpr (MODE == 3) {
                        // label collection: what routing this face to the cheap
                        // flux would change -- dt/dx |F_full - F_linear| for this
                        // component, relative to the local size of its conserved
                        // variable (density; rho (|v| + c) for momentum; sqrt(rho) c
                        // for the field; the total energy), with
                        // c^2 = (gam p + B^2) / rho at the mean state
                        R amx = larger(sL[0], sL[6 * CL]), dF[5], dq[5];
#pragma unroll
                        for (int k = 1; k < 6; ++k) amx = larger(amx, larger(sL[k * NL], sL[6 * CL + k * NL]));
#pragma unroll
                        for (int k = 0; k < 5; ++k) diff_at(r, k, dF[k], dq[k]);
                        const double lin = (double)linear_flux(dF, dq, amx);
                        const double rho = fv.rho, v2 = 2.0 * fv.hvv, b2 = fv.bbn2 * fv.rho;
                        const double pg = 0.5 * ((double)sC[CL + 2 * NL] + (double)sC[CL + 3 * NL]);
                        const double c = sqrt((gam * pg + b2) / rho);
                        const double scale = r == 0 ? rho
                                           : r < 4 ? rho * (sqrt(v2) + c)
                                           : r < 6 ? sqrt(rho) * c
                                           : pg / gm1 + 0.5 * rho * v2 + 0.5 * b2;
                        lab_f = fmaxf(lab_f, (float)(dtdl * fabs((double)fv.out[r] - lin) / scale));
                    }
                }
            }
            if constexpr (ROUTED) {
                if (__all_sync(ALL, !full)) load_prev();   // (the full path was skipped)
                if (__any_sync(ALL, !full)) {
                    // Lax-Friedrichs speed of the linear flux: the stencil's largest |lambda|
                    R amx = larger(sL[0], sL[6 * CL]);
#pragma unroll
                    for (int k = 1; k < 6; ++k) amx = larger(amx, larger(sL[k * NL], sL[6 * CL + k * NL]));
#pragma unroll
                    for (int r = 0; r < 7; ++r) {
                        R dF[5], dq[5];
#pragma unroll
                        for (int k = 0; k < 5; ++k) diff_at(r, k, dF[k], dq[k]);
                        const double lin = (double)linear_flux(dF, dq, amx) + sF[r * CP];
                        fl[r] = full ? fl[r] : lin;
                    }
                }
            }
            if constexpr (MODE == 3) {
                // the records of owned faces of the sampled tiles (a hash of
                // the index of the tile of 32 faces, 1 line in x and 2 lines
                // x 16 faces in y and z, so the sample does not alias with the
                // grid nor depend on how the sweep is cut)
                const Spot o = spot();
                if (o.owned) {
                    const int f = o.f, t1 = o.t1;
                    a.route_next[route_line(g, DIR, t1, o.t2) + (f + 2)] = 0;
                    constexpr int TL = DIR == 0 ? 1 : 2, TT = 32 / TL;
                    const int ntx = (n + TT - 1) / TT;
                    const int nty = DIR == 0 ? nt1 : (nt1 + 1 + TL - 1) / TL;
                    const int tx = f / TT < ntx ? f / TT : ntx - 1, ty = DIR == 0 ? t1 - 3 : (t1 - 2) / TL;
                    const long long tile = ((long long)(o.t2 - 3) * nty + ty) * ntx + tx;
                    const unsigned long long hs = (unsigned long long)tile * 0x9E3779B97F4A7C15ull;
                    if ((unsigned int)(hs >> 32) % a.collect_every == 0u) {
                        StencilCell sc[6];
#pragma unroll
                        for (int s = 0; s < 6; ++s)
                            sc[s] = StencilCell{sC[s * NL], sC[CL + s * NL], sC[2 * CL + s * NL], sC[3 * CL + s * NL],
                                                sC[4 * CL + s * NL]};
                        // the prior-stage feature is held at 0: fed back from the
                        // network's own decisions it locked smooth flows at full WENO
                        float ft[kRouterNF];
                        bool flat;
                        router_features(sc, 0.0f, (float)a.rhomin, (float)a.pgmin, a.guard_jump, a.guard_floor, ft, &flat);
                        const unsigned int slot = atomicAdd(a.collect_n, 1u);
                        if (slot < a.collect_cap) {
                            float* rec = a.collect + 8ull * slot;
#pragma unroll
                            for (int k = 0; k < 6; ++k) rec[k] = ft[k];
                            rec[6] = lab_w;
                            rec[7] = lab_f;
                        }
                    }
                }
            }
            mark(8);

            // CT terms (src/ssprk.cpp:973-993): flux plus the mean of B_n v_t
            // over the two cells
            const long long code = spot_code();
            if (code >= 0) {
#pragma unroll
                for (int c = 0; c < 2; ++c) {
                    const double* v = sB + c * CB + NL;       // v_t1 or v_t2 of cell f+2
                    const double* b = sB + 2 * CB + NL;       // B_n
                    const double x1 = b[0] * v[0], x2 = b[NL] * v[NL];
                    double avg;
                    if (a.ct4) {
                        // fourth-order midpoint value (-1, 9, 9, -1) / 16 over cells f+1 .. f+4
                        avg = fm(9.0, x1 + x2, -(b[-NL] * v[-NL] + b[2 * NL] * v[2 * NL])) * 0.0625;
                    } else {
                        // the reference's two-point form (-0, 9, 9, -0) / 18
                        avg = quot(fm(9.0, x1, 9.0 * x2), 18.0, 1.0 / 18.0);
                    }
                    (c == 0 ? a.cta : a.ctb)[code >> 1] = fl[4 + c] + avg;
                }
            }
            mark(9);

            // -------------------------------------------------------- update
            double dfl[7];
#pragma unroll
            for (int r = 0; r < 7; ++r) {
                const double up = __shfl_up_sync(ALL, fl[r], NL);
                dfl[r] = fl[r] - (j == 0 ? sX[r * NL] : up);
            }
            if (!arrived(1)) break;
            // cell f+2, between this interface and the one before
            if (code >= 0 && (code & 1)) {
                double* out = a.qout + (code >> 1);
#pragma unroll
                for (int gv = 0; gv < 8; ++gv, out += g.fs) {
                    const int v = line_var(DIR, gv);
                    const double cur = DIR == 0 ? sOp[(gv * NL + l) * M::TO + j + 1] : sOp[gv * 32 + lane];
                    double w = a.mode == 1 ? fm(a.k3, prev[v], a.k1 * cur) : cur;
                    // (the flux rows skip line variable 4, the normal B)
                    if (v != 4) w = fm(-dtdl, dfl[v < 4 ? v : v - 1], w);
                    if (v != 4 || a.mode != 0) *out = w;
                }
            }
            __syncwarp();   // every read of the operand tile and of sX is done
            if (j == W - 1) {
#pragma unroll
                for (int r = 0; r < 7; ++r) sX[r * NL] = fl[r];
            }
        }
        // the window's last cells become the history of the next chunk
        __syncwarp();
        {
            MoveBack<double, 12, CP, M::HP * NL> pf;   // P and F rows are adjacent
            MoveBack<double, 3, CB, M::HB * NL> vb;
            MoveBack<DT, Diff<R>::rows, CD, M::HD * NL> d;
            MoveBack<R, 7, CL, M::HL * NL> e;
            pf.load(sP - lane, lane); vb.load(sB - lane, lane); d.load(sD - lane, lane); e.load(sL - lane, lane);
            if constexpr (MODE != 0) {
                MoveBack<float, M::NCF, CL, M::HL * NL> c;
                c.load(sC - lane, lane);
                c.store(sC - lane, lane);
            }
            pf.store(sP - lane, lane); vb.store(sB - lane, lane); d.store(sD - lane, lane); e.store(sL - lane, lane);
        }
        // the next place (in shared memory: read by all before lane 0 writes it,
        // and written before the others read it)
        if constexpr (FREE_REGS) {
            if (here.fb < here.fend) here.fb += W;
            else r_place = enter(here.item + (int)gridDim.x * WPB);
        } else if (here.fb < here.fend) {
            __syncwarp();
            if (lane == 0) here.fb = here.fb + W;
        } else {
            const Place nx = enter(here.item + (int)gridDim.x * WPB);
            __syncwarp();
            if (lane == 0) s_place[warp] = nx;
        }
        __syncwarp();
        mark(10);
    }
    if (timed)
        for (int k = 0; k < 12; ++k) atomicAdd(a0.prof + k, s_prof[warp][k]);
    __syncthreads();   // every warp is done with its tensor memory
    if (warp == 0) tmem_free<kColumns>(s_tmem);
    if constexpr (ROUTED) {
        if (lane == 0) {
            if (n_full) atomicAdd(&a0.route_count[0], (unsigned long long)n_full);
            if (n_cheap) atomicAdd(&a0.route_count[1], (unsigned long long)n_cheap);
        }
    }
}

}  // namespace
}  // namespace how
