// physics.cuh -- pointwise ideal-MHD physics on the device (FP64).
//
// Each function keeps the operation order of the reference Fortran routine
// it cites, so that a build without FMA contraction (--fmad=false) rounds
// exactly like the reference's arithmetic statement by statement.  Fortran
// MAX/MIN become fmax/fmin (the non-NaN argument wins).
#pragma once

#include <cstdint>

namespace hosono {

// variable indices, src/definitions.f90:18-35 (0-based)
enum : int { DENS = 0, MOMX = 1, MOMY = 2, MOMZ = 3, ENER = 4, MAGX = 5, MAGY = 6, MAGZ = 7 };
enum : int { VELX = 1, VELY = 2, VELZ = 3, PRES = 4, EINT = 8, GAMM = 9 };
enum : int { XDIR = 0, YDIR = 1 };
enum : int { NORTH = 0, SOUTH = 1, EAST = 2, WEST = 3 };
constexpr int NCONS = 8;
constexpr int NPRIM = 10;

struct Phys {
    double gamma;
    double small_pressure;
    double small_density;
    double small_b;  // sim_smallB (eigen_beta_T only)
    int force_hydro;
};

// sim_forceHydro as a run-time flag (FH = -1) or as a compile-time constant
// (FH = 0: MHD, 1: hydro), for kernels instantiated per mode.  The
// expressions are the same either way; with a constant the compiler drops
// the other mode's branch and keeps the magnetic field of an MHD state in
// the registers of the conserved variables.
template <int FH>
__device__ __forceinline__ bool hydro(const Phys& s) {
    return FH < 0 ? s.force_hydro != 0 : FH != 0;
}

// src/eos.f90:9-26 (pressure floor)
__device__ __forceinline__ double eos_pres(const Phys& s, double dens, double eint) {
    double pres = (s.gamma - 1.0) * dens * eint;
    if (pres < s.small_pressure) pres = s.small_pressure;
    return pres;
}

// src/convert.f90:198-234
__device__ __forceinline__ void cons2prim(const Phys& s, const double* U, double* V) {
    double Bp;
    if (s.force_hydro)
        Bp = 0.0;
    else
        Bp = 0.5 * (U[MAGX] * U[MAGX] + U[MAGY] * U[MAGY] + U[MAGZ] * U[MAGZ]);
    const double density = U[DENS];
    const double velx = U[MOMX] / density;
    const double vely = U[MOMY] / density;
    const double velz = U[MOMZ] / density;
    const double eint = (U[ENER] - Bp) / density - 0.5 * (velx * velx + vely * vely + velz * velz);
    V[DENS] = density;
    V[VELX] = velx;
    V[VELY] = vely;
    V[VELZ] = velz;
    if (s.force_hydro) {
        V[MAGX] = 0.0;
        V[MAGY] = 0.0;
        V[MAGZ] = 0.0;
    } else {
        V[MAGX] = U[MAGX];
        V[MAGY] = U[MAGY];
        V[MAGZ] = U[MAGZ];
    }
    V[PRES] = eos_pres(s, density, eint);
    V[EINT] = eint;
    V[GAMM] = s.gamma;
}

// src/convert.f90:236-254 (not floored; SUM starts from zero)
template <int FH = -1>
__device__ __forceinline__ double cons2pres(const Phys& s, const double* U) {
    double Bp;
    if (hydro<FH>(s))
        Bp = 0.0;
    else
        Bp = 0.5 * ((0.0 + U[MAGX] * U[MAGX]) + U[MAGY] * U[MAGY] + U[MAGZ] * U[MAGZ]);
    const double msq = (0.0 + U[MOMX] * U[MOMX]) + U[MOMY] * U[MOMY] + U[MOMZ] * U[MOMZ];
    return (s.gamma - 1.0) * (U[ENER] - Bp - 0.5 * msq / U[DENS]);
}

// src/detect.f90:250-265 (CAD) and :238-248 (PAD): both finite (not NaN,
// not infinite) and both > 0, i.e. each bit pattern is a positive, nonzero,
// finite double (tested on the integer pipes)
__device__ __forceinline__ bool positive_finite(double x) {
    const unsigned long long u = (unsigned long long)__double_as_longlong(x);
    return u - 1ull < 0x7fefffffffffffffull;  // u in [1, 0x7fefffffffffffff]
}
__device__ __forceinline__ bool admissible(double dens, double pres) {
    return positive_finite(dens) && positive_finite(pres);
}

// src/eigen.f90:305-321 (Ryu & Jones 1995, eqs. 2.18-2.19)
__device__ __forceinline__ double c_fs(double gam, double rho, double p, double BB, double B_N, double pm) {
    double c = (gam * p + BB) / rho;
    c = 0.5 * (c + pm * sqrt(c * c - 4.0 * gam * p * (B_N * B_N) / (rho * rho)));
    return sqrt(fmax(1.0e-14, c));
}

__device__ __forceinline__ double dot3(double a0, double a1, double a2, double b0, double b1, double b2) {
    return (0.0 + a0 * b0) + a1 * b1 + a2 * b2;
}

// ---- division by shared denominators.  Most quotients of the Riemann solver
// come in groups with one denominator (the density of a side, sR - sL, the
// HLL density, sK - sStar).  SharedRecip holds b, y = RN(1/b) (__drcp_rn,
// correctly rounded) and z, the rest of 1/b rounded, so y + z is 1/b to twice
// the precision; shared_quot then takes each quotient in four operations:
// q0 = fma(a, y, a*z) is within one ulp of a/b, and by Markstein's theorem
// (P. Markstein, "Computation of elementary functions on the IBM RISC
// System/6000 processor", IBM J. Res. Dev. 34(1), 1990; a reciprocal kept in
// two parts: N. Brisebarre, J.-M. Muller, S. K. Raina, "Accelerating correctly
// rounded floating-point division when the divisor is known in advance", IEEE
// Trans. Comput. 53(8), 2004) the remainder r = a - b*q0 is exact and
// RN(q0 + r*y) = RN(a/b): the same bits as '/', whose sign a zero quotient
// takes from the operands (tests/div_check.cu compares the two on the GPU).
// Without a*z, q0 = RN(a*y) is up to two ulps off and takes a second
// correction per quotient.  The proof assumes no overflow, underflow or
// subnormal on the way, which the operand ranges of GroupDiv guarantee.  A zero
// quotient is +0; with_sign gives it the operands' sign, which the solver does
// not need: no expression of it tells the zeros apart.
struct SharedRecip {
    double b, y, z;
};
__device__ __forceinline__ SharedRecip shared_recip(double b) {
    const double y = __drcp_rn(b);
    return SharedRecip{b, y, fma(-b, y, 1.0) * y};
}
__device__ __forceinline__ double shared_quot(double a, const SharedRecip& r) {
    const double q0 = fma(a, r.y, a * r.z);
    return fma(fma(-r.b, q0, a), r.y, q0);
}
__device__ __forceinline__ double with_sign(double q, double a, double b) {
    const int sign = (__double2hiint(a) ^ __double2hiint(b)) & (int)0x80000000;
    return __hiloint2double((__double2hiint(q) & 0x7fffffff) | sign, __double2loint(q));
}
// Quotients with their operand ranges watched: |b| in [2^DLO, 2^(DHI+1)), a
// zero or |a| in [2^NLO, 2^(NHI+1)).  The smallest and largest exponents seen
// are kept as integer keys (the magnitude's high word, one bit for the rest),
// four integer instructions a numerator, and compared once.
template <int NLO, int NHI, int DLO, int DHI>
struct GroupDiv {
    unsigned nmin = ~0u, nmax = 0u, dmin = ~0u, dmax = 0u;
    __device__ __forceinline__ SharedRecip recip(double b) {
        watch(b);
        return shared_recip(b);
    }
    // a value that has to lie in the denominators' range
    __device__ __forceinline__ void watch(double b) {
        const unsigned k = (unsigned)__double2hiint(b) << 1;
        dmin = min(dmin, k);
        dmax = max(dmax, k);
    }
    __device__ __forceinline__ double div(double a, const SharedRecip& r) {
        const unsigned k = ((unsigned)__double2hiint(a) << 1) + min((unsigned)__double2loint(a), 1u);
        nmin = min(nmin, k - 1u);  // a zero wraps to the top
        nmax = max(nmax, k);
        return shared_quot(a, r);
    }
    __device__ __forceinline__ bool ok() const {
        return nmin >= ((1023u + NLO) << 21) - 1u && nmax < ((1024u + NHI) << 21) && dmin >= ((1023u + DLO) << 21) &&
               dmax < ((1024u + DHI) << 21);
    }
};
// The solver's ranges: b in [2^-100, 2^101) and a down to 2^-860 keep every
// intermediate normal (the quotient above 2^-962, the remainder a multiple of
// 2^-965); momenta ahead of a front fall off by orders of magnitude a cell, so
// the numerators' range is the wide one.  Below 2^301 they keep every product
// of the solver finite, which the terms it leaves out need: zero times a
// finite value.
typedef GroupDiv<-860, 300, -100, 100> SolverDiv;
// one quotient at a time over a symmetric range, as tests/div_check.cu drives it
struct SharedRecipDiv {
    GroupDiv<-500, 500, -500, 500> g;
    bool ok = true;
    __device__ __forceinline__ SharedRecip recip(double b) { return g.recip(b); }
    __device__ __forceinline__ double div(double a, const SharedRecip& r) {
        const double q = g.div(a, r);
        ok = g.ok();
        return with_sign(q, a, r.b);
    }
};

// CAD and PAD of a state by its density, |m|^2 and |B|^2 (each summed x, y, z
// from zero) and energy: admissible(rho, cons2pres).  Nearly every state is
// seen to pass without cons2pres's division: rho * (E - Bp) exceeds 0.5 |m|^2
// by more than its rounding (a margin of 2^-40), with every term far from
// overflow and underflow.
__device__ __forceinline__ bool state_admissible(const Phys& s, double rho, double msq, double bsq, double E) {
    const double Bp = s.force_hydro ? 0.0 : 0.5 * bsq;
    const double e = E - Bp;
    if (rho > 1e-100 && rho < 1e100 && e > 1e-100 && e < 1e100 && e * rho > 0.5 * msq * (1.0 + 0x1p-40) &&
        s.gamma > 1.001 && s.gamma < 1000.0)
        return true;
    return admissible(rho, (s.gamma - 1.0) * (E - Bp - 0.5 * msq / rho));
}
// pressure (floored) and in-plane velocity of a state as cons2prim gives them
// (convert.f90:198-234), its four quotients by the density on one reciprocal
__device__ __forceinline__ double prim_pres(const Phys& s, const double* U, double& vx, double& vy) {
    double Bp = 0.0;
    if (!s.force_hydro) Bp = 0.5 * (U[MAGX] * U[MAGX] + U[MAGY] * U[MAGY] + U[MAGZ] * U[MAGZ]);
    const double EB = s.force_hydro ? U[ENER] : U[ENER] - Bp;
    SolverDiv g;
    const SharedRecip r = g.recip(U[DENS]);
    vx = g.div(U[MOMX], r);
    vy = g.div(U[MOMY], r);
    double vz = g.div(U[MOMZ], r), q = g.div(EB, r);
    if (!g.ok()) {
        vx = U[MOMX] / U[DENS];
        vy = U[MOMY] / U[DENS];
        vz = U[MOMZ] / U[DENS];
        q = EB / U[DENS];
    }
    return eos_pres(s, U[DENS], q - 0.5 * (vx * vx + vy * vy + vz * vz));
}

// ---- src/riemannSolver.f90:68-221 (HLLC for MHD, Li 2005) in face
// coordinates: N the normal, T the other in-plane component, Z out of plane.
// A y-face is the x-face of the state with x and y exchanged, bit for bit:
// the solver's sums over components are of two commuted in-plane terms, then
// the z term, so no expression's rounding changes.
enum : int { MOMN = 1, MOMT = 2, MOMZ_ = 3, MAGN = 5, MAGT = 6, MAGZ_ = 7 };

// The solver with IEEE division, statement by statement: for the operands the
// shared-denominator form does not take, and hydro runs whose conserved
// state carries a field.  What the chosen branch does not read is not
// computed.
template <int FH>
struct IeeeSide {
    double rho, v[3], p, b[3];
};
template <int FH>
__device__ __forceinline__ void ieee_prim(const Phys& s, const double* U, IeeeSide<FH>& V) {
    double Bp;
    if (hydro<FH>(s))
        Bp = 0.0;
    else
        Bp = 0.5 * (U[5] * U[5] + U[6] * U[6] + U[7] * U[7]);
    V.rho = U[DENS];
    for (int k = 0; k < 3; k++) {
        V.v[k] = U[1 + k] / V.rho;
        V.b[k] = hydro<FH>(s) ? 0.0 : U[5 + k];
    }
    const double eint = (U[ENER] - Bp) / V.rho - 0.5 * (V.v[0] * V.v[0] + V.v[1] * V.v[1] + V.v[2] * V.v[2]);
    V.p = eos_pres(s, V.rho, eint);
}
// fast magnetosonic speed of one side or of the average state (eigen.f90:257-303)
__device__ __forceinline__ double side_cf(const Phys& s, double rho0, double p0, double bN, double bT, double bZ) {
    const double rho = fmax(rho0, s.small_density);
    const double p = fmax(p0, s.small_pressure);
    const double BB = bN * bN + bT * bT + bZ * bZ;
    return c_fs(s.gamma, rho, p, BB, bN, +1.0);
}
// cons2flux (convert.f90:28-92)
template <int FH>
__device__ __forceinline__ void ieee_flux(const Phys& s, const double* U, const IeeeSide<FH>& V, double* F) {
    double Bp = 0.0;
    if (!hydro<FH>(s)) Bp = 0.5 * (U[5] * U[5] + U[6] * U[6] + U[7] * U[7]);
    const double Ptot = V.p + Bp;
    F[DENS] = U[MOMN];
    F[MOMN] = U[MOMN] * U[MOMN] / V.rho + Ptot;
    F[MOMT] = U[MOMN] * V.v[1];
    F[MOMZ_] = U[MOMN] * V.v[2];
    F[ENER] = (U[ENER] + Ptot) * V.v[0];
    F[MAGN] = F[MAGT] = F[MAGZ_] = 0.0;
    if (!hydro<FH>(s)) {
        F[MOMN] = F[MOMN] - V.b[0] * V.b[0];
        F[MOMT] = F[MOMT] - V.b[1] * V.b[0];
        F[MOMZ_] = F[MOMZ_] - V.b[2] * V.b[0];
        F[MAGT] = V.v[0] * V.b[1] - V.v[1] * V.b[0];
        F[MAGZ_] = V.v[0] * V.b[2] - V.v[2] * V.b[0];
        F[ENER] = F[ENER] - V.b[0] * (V.v[0] * V.b[0] + V.v[1] * V.b[1] + V.v[2] * V.b[2]);
    }
}
template <int FH>
__device__ __forceinline__ void ieee_solve(const Phys& s, const double* uL, const double* uR, double* flux) {
    IeeeSide<FH> L, R;
    ieee_prim<FH>(s, uL, L);
    ieee_prim<FH>(s, uR, R);
    // eigenvalues 1 and 7 of L, R and the arithmetic average (riemannSolver.f90:84-96)
    const double vNA = (L.v[0] + R.v[0]) / 2.0;
    const double cfA = side_cf(s, (L.rho + R.rho) / 2.0, (L.p + R.p) / 2.0, (L.b[0] + R.b[0]) / 2.0,
                               (L.b[1] + R.b[1]) / 2.0, (L.b[2] + R.b[2]) / 2.0);
    const double sL = fmin(L.v[0] - side_cf(s, L.rho, L.p, L.b[0], L.b[1], L.b[2]), vNA - cfA);
    const double sR = fmax(vNA + cfA, R.v[0] + side_cf(s, R.rho, R.p, R.b[0], R.b[1], R.b[2]));
    const double pTotL = L.p + 0.5 * dot3(L.b[0], L.b[1], L.b[2], L.b[0], L.b[1], L.b[2]);
    const double pTotR = R.p + 0.5 * dot3(R.b[0], R.b[1], R.b[2], R.b[0], R.b[1], R.b[2]);
    const double dL = sL - L.v[0], dR = sR - R.v[0];
    const double sStr = (uR[MOMN] * dR - uL[MOMN] * dL + pTotL - pTotR - L.b[0] * L.b[0] + R.b[0] * R.b[0]) /
                        (R.rho * dR - L.rho * dL);
    // final choice (riemannSolver.f90:189-219): fL if 0 < sL; left star state
    // if sL <= 0 < sStr; right star state if sStr <= 0 <= sR; fR otherwise.
    const int side = 0.0 < sL ? 0 : (sL <= 0.0) && (0.0 < sStr) ? 1 : (sStr <= 0.0) && (0.0 <= sR) ? 2 : 3;
    double fL[NCONS], fR[NCONS], uHLL[NCONS], uStr[NCONS];
    ieee_flux<FH>(s, uL, L, fL);
    ieee_flux<FH>(s, uR, R, fR);
    if (side == 0 || side == 3) {
        for (int v = 0; v < NCONS; v++) flux[v] = side == 0 ? fL[v] : fR[v];
        return;
    }
    for (int v = 0; v < NCONS; v++) uHLL[v] = (sR * uR[v] - sL * uL[v] + fL[v] - fR[v]) / (sR - sL);
    const double magDotVelHLL = dot3(uHLL[5], uHLL[6], uHLL[7], uHLL[1] / uHLL[0], uHLL[2] / uHLL[0], uHLL[3] / uHLL[0]);
    const double pStr = L.rho * dL * (sStr - L.v[0]) + pTotL - L.b[0] * L.b[0] + uHLL[MAGN] * uHLL[MAGN];
    const bool left = side == 1;
    const IeeeSide<FH>& K = left ? L : R;
    const double* uK = left ? uL : uR;
    const double sK = left ? sL : sR, dK = left ? dL : dR, pTotK = left ? pTotL : pTotR;
    const double magDotVelK = dot3(K.b[0], K.b[1], K.b[2], K.v[0], K.v[1], K.v[2]);
    uStr[DENS] = K.rho * dK / (sK - sStr);
    uStr[MOMN] = uStr[DENS] * sStr;
    uStr[MOMT] = uStr[DENS] * K.v[1] - (uHLL[MAGN] * uHLL[MAGT] - K.b[0] * K.b[1]) / (sK - sStr);
    uStr[MOMZ_] = uStr[DENS] * K.v[2] - (uHLL[MAGN] * uHLL[MAGZ_] - K.b[0] * K.b[2]) / (sK - sStr);
    uStr[MAGN] = uHLL[MAGN];
    uStr[MAGT] = uHLL[MAGT];
    uStr[MAGZ_] = uHLL[MAGZ_];
    uStr[ENER] = uK[ENER] * dK + pStr * sStr - pTotK * K.v[0] - uHLL[MAGN] * magDotVelHLL + K.b[0] * magDotVelK;
    uStr[ENER] = uStr[ENER] / (sK - sStr);
    for (int v = 0; v < NCONS; v++) flux[v] = (left ? fL[v] : fR[v]) + sK * (uStr[v] - uK[v]);
}
// out of line and by value: a pointer to the caller's states would keep them
// in local memory on the common path too
struct Cons8 {
    double v[NCONS];
};
template <int FH>
static __device__ __noinline__ Cons8 hllc_ieee(Phys s, Cons8 uL, Cons8 uR) {
    Cons8 F;
    ieee_solve<FH>(s, uL.v, uR.v, F.v);
    return F;
}

// What a solve may leave out, because its terms are zeros (bits: a sum with
// them, and a product kept under another sum, has the same value without):
// out-of-plane momentum and field of a planar flow, the field of a hydro run.
// SOLVE_HYDRO_FIELD: a hydro run whose conserved state carries a field, which
// the solver reads in its HLL state (IEEE form only).
enum : int { SOLVE_MHD = 0, SOLVE_MHD_PLANAR = 1, SOLVE_HYDRO = 2, SOLVE_HYDRO_PLANAR = 3, SOLVE_HYDRO_FIELD = 4 };
template <int MODE>
struct Solve {
    static constexpr bool H = MODE >= SOLVE_HYDRO;            // hydro: no field
    static constexpr bool Z = (MODE & 1) == 0;                // out-of-plane momentum
    static constexpr bool BZ = MODE == SOLVE_MHD;             // out-of-plane field
    static constexpr bool LEFT = MODE != SOLVE_MHD && MODE != SOLVE_HYDRO_FIELD;  // it leaves some out
    static constexpr __host__ __device__ bool var(int v) {   // state variables it reads
        return MODE == SOLVE_HYDRO_FIELD || v < 3 || v == ENER || (v == MOMZ_ && Z) || (!H && (v == MAGN || v == MAGT)) || (BZ && v == MAGZ_);
    }
};
template <int MODE>
struct FaceSide {
    double rho, vN, vT, vZ, p, bN, bT, bZ, Bp, cf;
    SharedRecip r;
};
// the primitive variables of one side (cons2prim, convert.f90:198-234), its
// fast speed; returns CAD and PAD on its density and cons2pres
// (convert.f90:236-254, not floored).  A density below the floor that
// eigen.f90 applies goes to the IEEE form.
template <int MODE>
__device__ __forceinline__ bool side_eval(const Phys& s, const double* U, FaceSide<MODE>& V, SolverDiv& g, bool& floored) {
    typedef Solve<MODE> S;
    V.rho = U[DENS];
    V.r = g.recip(V.rho);
    floored = floored || V.rho < s.small_density;
    double BB = 0.0;
    V.Bp = V.bN = V.bT = V.bZ = 0.0;
    if (!S::H) {
        V.bN = U[MAGN];
        V.bT = U[MAGT];
        BB = V.bN * V.bN + V.bT * V.bT;
        if (S::BZ) {
            V.bZ = U[MAGZ_];
            BB = BB + V.bZ * V.bZ;
        }
        V.Bp = 0.5 * BB;
    }
    const double EB = S::H ? U[ENER] : U[ENER] - V.Bp;
    double msq = U[MOMN] * U[MOMN] + U[MOMT] * U[MOMT];
    if (S::Z) msq = msq + U[MOMZ_] * U[MOMZ_];
    const bool adm = admissible(V.rho, (s.gamma - 1.0) * (EB - g.div(0.5 * msq, V.r)));
    V.vN = g.div(U[MOMN], V.r);
    V.vT = g.div(U[MOMT], V.r);
    V.vZ = S::Z ? g.div(U[MOMZ_], V.r) : 0.0;
    double vsq = V.vN * V.vN + V.vT * V.vT;
    if (S::Z) vsq = vsq + V.vZ * V.vZ;
    V.p = eos_pres(s, V.rho, g.div(EB, V.r) - 0.5 * vsq);
    // c_fs (eigen.f90:305-321) of the floored state, whose floors hold here
    if (S::H) {
        // the discriminant is c*c, whose root is c (rounding to nearest, no
        // overflow or underflow: c is watched), and 0.5*(c + c) = c
        const double c = g.div(s.gamma * V.p, V.r);
        g.watch(c);
        V.cf = sqrt(fmax(1.0e-14, c));
    } else {
        const double c = g.div(s.gamma * V.p + BB, V.r);
        V.cf = sqrt(fmax(1.0e-14,
                         0.5 * (c + sqrt(c * c - 4.0 * s.gamma * V.p * (V.bN * V.bN) / (V.rho * V.rho)))));
    }
    return adm;
}
// the flux of one side (cons2flux, convert.f90:28-92) without the energy
template <int MODE>
__device__ __forceinline__ void side_flux(const double* U, const FaceSide<MODE>& V, double* F, SolverDiv& g) {
    typedef Solve<MODE> S;
    const double Ptot = V.p + V.Bp;
    F[DENS] = U[MOMN];
    F[MOMN] = g.div(U[MOMN] * U[MOMN], V.r) + Ptot;
    F[MOMT] = U[MOMN] * V.vT;
    if (S::Z) F[MOMZ_] = U[MOMN] * V.vZ;
    if (!S::H) {
        F[MOMN] = F[MOMN] - V.bN * V.bN;
        F[MOMT] = F[MOMT] - V.bT * V.bN;
        if (S::Z) F[MOMZ_] = F[MOMZ_] - V.bZ * V.bN;
        F[MAGT] = V.vN * V.bT - V.vT * V.bN;
        if (S::BZ) F[MAGZ_] = V.vN * V.bZ - V.vZ * V.bN;
    }
}
// HLLC in face coordinates with shared denominators; false when an operand
// left their range (flux is then not to be used).  The variables the mode
// leaves out are not read and not written.  admL, admR: CAD and PAD of the
// sides.
template <int MODE>
__device__ __forceinline__ bool face_solve(const Phys& s, const double* uL, const double* uR, double* flux,
                                           bool& admL, bool& admR) {
    typedef Solve<MODE> S;
    SolverDiv g;
    bool floored = false;
    FaceSide<MODE> L, R;
    admL = side_eval<MODE>(s, uL, L, g, floored);
    admR = side_eval<MODE>(s, uR, R, g, floored);
    // eigenvalues 1 and 7 of L, R and the arithmetic average (riemannSolver.f90:84-96)
    double cfA;
    {
        const double rho = (L.rho + R.rho) / 2.0, p = (L.p + R.p) / 2.0;
        if (S::H) {
            const double c = s.gamma * p / rho;
            g.watch(c);
            cfA = sqrt(fmax(1.0e-14, c));
        } else {
            const double bN = (L.bN + R.bN) / 2.0, bT = (L.bT + R.bT) / 2.0;
            double BB = bN * bN + bT * bT;
            if (S::BZ) {
                const double bZ = (L.bZ + R.bZ) / 2.0;
                BB = BB + bZ * bZ;
            }
            cfA = c_fs(s.gamma, rho, p, BB, bN, +1.0);
        }
    }
    const double vNA = (L.vN + R.vN) / 2.0;
    const double sL = fmin(L.vN - L.cf, vNA - cfA);
    const double sR = fmax(vNA + cfA, R.vN + R.cf);
    const double pTotL = L.p + L.Bp, pTotR = R.p + R.Bp;
    const double dL = sL - L.vN, dR = sR - R.vN;
    double num = uR[MOMN] * dR - uL[MOMN] * dL + pTotL - pTotR;
    if (!S::H) num = num - L.bN * L.bN + R.bN * R.bN;
    const double sStr = num / (R.rho * dR - L.rho * dL);
    // final choice (riemannSolver.f90:189-219): fL if 0 < sL; left star state
    // if sL <= 0 < sStr; right star state if sStr <= 0 <= sR; fR otherwise.
    const bool left = 0.0 < sL || ((sL <= 0.0) && (0.0 < sStr));
    const bool star = !(0.0 < sL) && (left || ((sStr <= 0.0) && (0.0 <= sR)));
    double fL[NCONS], fR[NCONS];
    side_flux<MODE>(uL, L, fL, g);
    side_flux<MODE>(uR, R, fR, g);
    // the chosen side
    const double vNK = left ? L.vN : R.vN, pTotK = left ? pTotL : pTotR, bNK = left ? L.bN : R.bN;
    const double eK = left ? uL[ENER] : uR[ENER];
    double bDotV = 0.0;  // of the chosen side
    double fE = (eK + pTotK) * vNK;
    if (!S::H) {
        const double vTK = left ? L.vT : R.vT, bTK = left ? L.bT : R.bT;
        bDotV = vNK * bNK + vTK * bTK;
        if (S::BZ) bDotV = bDotV + (left ? L.vZ : R.vZ) * (left ? L.bZ : R.bZ);
        fE = fE - bNK * bDotV;
    }
#pragma unroll
    for (int v = 0; v < NCONS; v++)
        if (S::var(v)) flux[v] = v == ENER ? fE : v == MAGN ? 0.0 : left ? fL[v] : fR[v];
    if (star) {
        const double sK = left ? sL : sR, dK = left ? dL : dR;
        const double rhoK = left ? L.rho : R.rho, vTK = left ? L.vT : R.vT;
        const SharedRecip rK = g.recip(sK - sStr);
        double uStr[NCONS];
        uStr[DENS] = g.div(rhoK * dK, rK);
        uStr[MOMN] = uStr[DENS] * sStr;
        uStr[MOMT] = uStr[DENS] * vTK;
        if (S::Z) uStr[MOMZ_] = uStr[DENS] * (left ? L.vZ : R.vZ);
        double pStr = L.rho * dL * (sStr - L.vN) + pTotL;
        if (S::H) {
            // without a field the HLL state enters no other term, and its
            // products with it are zeros where its velocity is finite: where
            // its density is not lost to rounding (a side beyond Mach 2^53)
            g.watch(sR - sL);
            floored = floored || !(sR * uR[DENS] - sL * uL[DENS] + fL[DENS] - fR[DENS] > 0x1p-300);
            uStr[ENER] = g.div(eK * dK + pStr * sStr - pTotK * vNK, rK);
        } else {
            double uHLL[NCONS];
            const SharedRecip rS = g.recip(sR - sL);
#pragma unroll
            for (int v = 0; v < NCONS; v++)
                if (S::var(v) && v != ENER)
                    uHLL[v] = v == MAGN ? g.div(sR * uR[v] - sL * uL[v] + 0.0, rS)
                                        : g.div(sR * uR[v] - sL * uL[v] + fL[v] - fR[v], rS);
            const SharedRecip rH = g.recip(uHLL[DENS]);
            double bvH = 0.0 + uHLL[MAGN] * g.div(uHLL[MOMN], rH);
            bvH = bvH + uHLL[MAGT] * g.div(uHLL[MOMT], rH);
            if (S::BZ) bvH = bvH + uHLL[MAGZ_] * g.div(uHLL[MOMZ_], rH);
            const double bTK = left ? L.bT : R.bT;
            pStr = pStr - L.bN * L.bN + uHLL[MAGN] * uHLL[MAGN];
            uStr[MOMT] = uStr[MOMT] - g.div(uHLL[MAGN] * uHLL[MAGT] - bNK * bTK, rK);
            if (S::BZ)
                uStr[MOMZ_] = uStr[MOMZ_] - g.div(uHLL[MAGN] * uHLL[MAGZ_] - bNK * (left ? L.bZ : R.bZ), rK);
            uStr[MAGN] = uHLL[MAGN];
            uStr[MAGT] = uHLL[MAGT];
            if (S::BZ) uStr[MAGZ_] = uHLL[MAGZ_];
            uStr[ENER] = g.div(eK * dK + pStr * sStr - pTotK * vNK - uHLL[MAGN] * bvH + bNK * (0.0 + bDotV), rK);
        }
#pragma unroll
        for (int v = 0; v < NCONS; v++)
            if (S::var(v)) flux[v] = flux[v] + sK * (uStr[v] - (left ? uL[v] : uR[v]));
    }
    return g.ok() && !floored;
}
// CAD and PAD of a state whose left-out variables are zeros
template <int MODE>
__device__ __forceinline__ bool state_adm(const Phys& s, const double* u) {
    double U[NCONS];
#pragma unroll
    for (int v = 0; v < NCONS; v++) U[v] = Solve<MODE>::var(v) ? u[v] : 0.0;
    return admissible(U[DENS], cons2pres<Solve<MODE>::H ? 1 : 0>(s, U));
}
// a mode's solve, the IEEE form where it has to be; that form's eight fluxes go
// to `all`, for a left-out variable's flux is NaN where a speed or a product of
// the solve is infinite (zero times infinity, zero by zero)
template <int MODE, class All>
__device__ __forceinline__ void face_flux(const Phys& s, const double* uL, const double* uR, double* F, bool& admL,
                                          bool& admR, All&& all) {
    bool done = false;
    if (MODE != SOLVE_HYDRO_FIELD) done = face_solve<MODE>(s, uL, uR, F, admL, admR);
    if (!done) {
        Cons8 a, b;
#pragma unroll
        for (int v = 0; v < NCONS; v++) {
            a.v[v] = Solve<MODE>::var(v) ? uL[v] : 0.0;
            b.v[v] = Solve<MODE>::var(v) ? uR[v] : 0.0;
        }
        const Cons8 f = hllc_ieee<Solve<MODE>::H ? 1 : 0>(s, a, b);
#pragma unroll
        for (int v = 0; v < NCONS; v++)
            if (Solve<MODE>::var(v)) F[v] = f.v[v];
        all(f);
        admL = state_adm<MODE>(s, uL);
        admR = state_adm<MODE>(s, uR);
    }
}
__device__ __forceinline__ bool bits_zero(double a) {
    return (((unsigned)__double2hiint(a) << 1) | (unsigned)__double2loint(a)) == 0u;
}
// in face coordinates, hydro flag at run time; admL, admR: CAD and PAD of the sides
__device__ __forceinline__ void hllc_face(const Phys& s, const double* uL, const double* uR, double* F, bool& admL,
                                          bool& admR) {
    auto whole = [](const Cons8&) {};  // the mode's own variables are all there are
    if (!s.force_hydro) {
        face_flux<SOLVE_MHD>(s, uL, uR, F, admL, admR, whole);
        return;
    }
    bool field = false;
#pragma unroll
    for (int v = MAGN; v <= MAGZ_; v++) field = field || !bits_zero(uL[v]) || !bits_zero(uR[v]);
    if (field) {
        face_flux<SOLVE_HYDRO_FIELD>(s, uL, uR, F, admL, admR, whole);
        return;
    }
    F[MAGN] = F[MAGT] = F[MAGZ_] = 0.0;
    face_flux<SOLVE_HYDRO>(s, uL, uR, F, admL, admR, [&](const Cons8& f) {
        F[MAGN] = f.v[MAGN];
        F[MAGT] = f.v[MAGT];
        F[MAGZ_] = f.v[MAGZ_];
    });
}
// in grid coordinates: a y-face exchanges x and y on the way in and out
__device__ __forceinline__ void hllc(const Phys& s, const double* uL, const double* uR, int dir, double* flux) {
    const bool x = dir == XDIR;
    double a[NCONS], b[NCONS], F[NCONS];
#pragma unroll
    for (int v = 0; v < NCONS; v++) {
        const int t = v == MOMX ? MOMY : v == MOMY ? MOMX : v == MAGX ? MAGY : v == MAGY ? MAGX : v;
        a[v] = x ? uL[v] : uL[t];
        b[v] = x ? uR[v] : uR[t];
    }
    bool al, ar;
    hllc_face(s, a, b, F, al, ar);
#pragma unroll
    for (int v = 0; v < NCONS; v++) {
        const int t = v == MOMX ? MOMY : v == MOMY ? MOMX : v == MAGX ? MAGY : v == MAGY ? MAGX : v;
        flux[v] = x ? F[v] : F[t];
    }
}


// ----------------------------------------------------------------------
// eigen_vecsFromPrim (src/eigen.f90:20-255) with eigen_alpha_fs (:323-349)
// and eigen_beta_T (:351-371): the left and right eigenvectors of the 7 MHD
// waves, in primitive or (cons) conserved variables.  Not on the time-step
// path (no .par option of the reference uses it); exposed by
// hosono_gpu_eigenvecs.  Statement order of the reference; MATMUL as sums
// over k ascending from zero.
// alpha_f for pm = +1, alpha_s for pm = -1
__device__ __forceinline__ double eigen_alpha_fs(double c_f, double c_s, double a, double BB, double B_N, double pm) {
    double BB_T = BB - B_N * B_N;
    (void)BB_T;  // computed by the reference, unused
    double cf2_minus_cs2 = c_f * c_f - c_s * c_s;
    double alpha;
    if (cf2_minus_cs2 > 1.0e-14) {
        alpha = 0.5 * (cf2_minus_cs2) + pm * (a * a - 0.5 * (c_f * c_f + c_s * c_s));
        alpha = alpha / (cf2_minus_cs2);
    } else if (pm > 0) {
        alpha = 1.0;
    } else {
        alpha = 0.0;
    }
    alpha = fmin(1.0, fmax(0.0, alpha));
    return sqrt(alpha);
}
// src/eigen.f90:351-371
__device__ __forceinline__ double eigen_beta_T(double B_T1, double B_T2, double smallB) {
    double BB_T = B_T1 * B_T1 + B_T2 * B_T2;
    if (BB_T < smallB * smallB) return copysign(1.0, B_T1) / sqrt(2.0);
    return B_T1 / sqrt(fmax(BB_T, 1.0e-30));
}
// src/eigen.f90:20-255: right eigenvectors (columns of R) and left
// eigenvectors (columns of L) of the 7 MHD waves in direction dir, 8x8
// column-major with the variable index as the row; cons: converted to
// conserved variables by dU/dV and dV/dU (MATMUL as k-ascending sums from 0)
__device__ inline void eigen_vecs(const Phys& s, const double* V, int dir, bool cons, double* Lm, double* Rm) {
    const int vN = dir == XDIR ? VELX : VELY, vT1 = dir == XDIR ? VELY : VELX, vT2 = VELZ;
    const int bN = dir == XDIR ? MAGX : MAGY, bT1 = dir == XDIR ? MAGY : MAGX, bT2 = MAGZ;
#define R(r, c) Rm[(r) + NCONS * ((c) - 1)]
#define L(r, c) Lm[(r) + NCONS * ((c) - 1)]
    const double rho = fmax(V[DENS], s.small_density);
    const double velN = V[vN], velT1 = V[vT1], velT2 = V[vT2];
    const double B_N = V[bN], B_T1 = V[bT1], B_T2 = V[bT2];
    const double p = fmax(V[PRES], s.small_pressure);
    const double gam = V[GAMM];
    const double BB = B_N * B_N + B_T1 * B_T1 + B_T2 * B_T2;
    const double c_f = c_fs(gam, rho, p, BB, B_N, +1.0);
    const double c_s = c_fs(gam, rho, p, BB, B_N, -1.0);
    const double a = sqrt(gam * p / rho);
    const double alpha_f = eigen_alpha_fs(c_f, c_s, a, BB, B_N, +1.0);
    const double alpha_s = eigen_alpha_fs(c_f, c_s, a, BB, B_N, -1.0);
    const double beta_T1 = eigen_beta_T(B_T1, B_T2, s.small_b);
    const double beta_T2 = eigen_beta_T(B_T2, B_T1, s.small_b);
    const double sgnBn = copysign(1.0, B_N);
    const double sr = sqrt(rho);
    for (int k = 0; k < NCONS * NCONS; k++) Rm[k] = Lm[k] = 0.0;
    R(DENS, 1) = alpha_f * rho;
    R(vN, 1) = -alpha_f * c_f;
    R(vT1, 1) = alpha_s * c_s * beta_T1 * sgnBn;
    R(vT2, 1) = alpha_s * c_s * beta_T2 * sgnBn;
    R(bT1, 1) = alpha_s * sr * a * beta_T1;
    R(bT2, 1) = alpha_s * sr * a * beta_T2;
    R(PRES, 1) = alpha_f * rho * (a * a);
    R(vT1, 2) = -beta_T2;
    R(vT2, 2) = beta_T1;
    R(bT1, 2) = -sr * beta_T2 * sgnBn;
    R(bT2, 2) = sr * beta_T1 * sgnBn;
    R(DENS, 3) = alpha_s * rho;
    R(vN, 3) = -alpha_s * c_s;
    R(vT1, 3) = -alpha_f * c_f * beta_T1 * sgnBn;
    R(vT2, 3) = -alpha_f * c_f * beta_T2 * sgnBn;
    R(bT1, 3) = -alpha_f * sr * a * beta_T1;
    R(bT2, 3) = -alpha_f * sr * a * beta_T2;
    R(PRES, 3) = alpha_s * rho * (a * a);
    R(DENS, 4) = 1.0;
    R(DENS, 5) = alpha_s * rho;
    R(vN, 5) = alpha_s * c_s;
    R(vT1, 5) = alpha_f * c_f * beta_T1 * sgnBn;
    R(vT2, 5) = alpha_f * c_f * beta_T2 * sgnBn;
    R(bT1, 5) = -alpha_f * sr * a * beta_T1;
    R(bT2, 5) = -alpha_f * sr * a * beta_T2;
    R(PRES, 5) = alpha_s * rho * (a * a);
    R(vT1, 6) = beta_T2;
    R(vT2, 6) = -beta_T1;
    R(bT1, 6) = -sr * beta_T2 * sgnBn;
    R(bT2, 6) = sr * beta_T1 * sgnBn;
    R(DENS, 7) = alpha_f * rho;
    R(vN, 7) = alpha_f * c_f;
    R(vT1, 7) = -alpha_s * c_s * beta_T1 * sgnBn;
    R(vT2, 7) = -alpha_s * c_s * beta_T2 * sgnBn;
    R(bT1, 7) = alpha_s * sr * a * beta_T1;
    R(bT2, 7) = alpha_s * sr * a * beta_T2;
    R(PRES, 7) = alpha_f * rho * (a * a);
    const double h = 1 / (2 * (a * a));
    L(vN, 1) = h * (-alpha_f * c_f);
    L(vT1, 1) = h * (alpha_s * c_s * beta_T1 * sgnBn);
    L(vT2, 1) = h * (alpha_s * c_s * beta_T2 * sgnBn);
    L(bT1, 1) = h * (alpha_s * a * beta_T1 / sr);
    L(bT2, 1) = h * (alpha_s * a * beta_T2 / sr);
    L(PRES, 1) = h * (alpha_f / rho);
    L(vT1, 2) = 0.5 * (-beta_T2);
    L(vT2, 2) = 0.5 * (beta_T1);
    L(bT1, 2) = 0.5 * (-beta_T2 * sgnBn / sr);
    L(bT2, 2) = 0.5 * (beta_T1 * sgnBn / sr);
    L(vN, 3) = h * (-alpha_s * c_s);
    L(vT1, 3) = h * (-alpha_f * c_f * beta_T1 * sgnBn);
    L(vT2, 3) = h * (-alpha_f * c_f * beta_T2 * sgnBn);
    L(bT1, 3) = h * (-alpha_f * a * beta_T1 / sr);
    L(bT2, 3) = h * (-alpha_f * a * beta_T2 / sr);
    L(PRES, 3) = h * (alpha_s / rho);
    L(DENS, 4) = 1.0;
    L(PRES, 4) = -1 / (a * a);
    L(vN, 5) = h * (alpha_s * c_s);
    L(vT1, 5) = h * (alpha_f * c_f * beta_T1 * sgnBn);
    L(vT2, 5) = h * (alpha_f * c_f * beta_T2 * sgnBn);
    L(bT1, 5) = h * (-alpha_f * a * beta_T1 / sr);
    L(bT2, 5) = h * (-alpha_f * a * beta_T2 / sr);
    L(PRES, 5) = h * (alpha_s / rho);
    L(vT1, 6) = 0.5 * (beta_T2);
    L(vT2, 6) = 0.5 * (-beta_T1);
    L(bT1, 6) = 0.5 * (-beta_T2 * sgnBn / sr);
    L(bT2, 6) = 0.5 * (beta_T1 * sgnBn / sr);
    L(vN, 7) = h * (alpha_f * c_f);
    L(vT1, 7) = h * (-alpha_s * c_s * beta_T1 * sgnBn);
    L(vT2, 7) = h * (-alpha_s * c_s * beta_T2 * sgnBn);
    L(bT1, 7) = h * (alpha_s * a * beta_T1 / sr);
    L(bT2, 7) = h * (alpha_s * a * beta_T2 / sr);
    L(PRES, 7) = h * (alpha_f / rho);
    if (!cons) {
#undef R
#undef L
        return;
    }
#undef R
#undef L
    const double k = 1.0 - gam;
    double dUdV[NCONS * NCONS] = {}, dVdU[NCONS * NCONS] = {};
#define A(r, c) dUdV[(r) + NCONS * (c)]
#define Bm(r, c) dVdU[(r) + NCONS * (c)]
    A(DENS, DENS) = 1.0;
    A(VELX, DENS) = V[VELX];
    A(VELY, DENS) = V[VELY];
    A(VELZ, DENS) = V[VELZ];
    A(PRES, DENS) = 0.5 * (velN * velN + velT1 * velT1 + velT2 * velT2);
    A(VELX, VELX) = rho;
    A(PRES, VELX) = rho * V[VELX];
    A(VELY, VELY) = rho;
    A(PRES, VELY) = rho * V[VELY];
    A(VELZ, VELZ) = rho;
    A(PRES, VELZ) = rho * V[VELZ];
    A(MAGX, MAGX) = 1.0;
    A(PRES, MAGX) = V[MAGX];
    A(MAGY, MAGY) = 1.0;
    A(PRES, MAGY) = V[MAGY];
    A(MAGZ, MAGZ) = 1.0;
    A(PRES, MAGZ) = V[MAGZ];
    A(PRES, PRES) = -1 / k;
    Bm(DENS, DENS) = 1.0;
    Bm(VELX, DENS) = -V[VELX] / rho;
    Bm(VELY, DENS) = -V[VELY] / rho;
    Bm(VELZ, DENS) = -V[VELZ] / rho;
    Bm(PRES, DENS) = -k * A(PRES, DENS);
    Bm(VELX, VELX) = 1 / rho;
    Bm(PRES, VELX) = k * V[VELX];
    Bm(VELY, VELY) = 1 / rho;
    Bm(PRES, VELY) = k * V[VELY];
    Bm(VELZ, VELZ) = 1 / rho;
    Bm(PRES, VELZ) = k * V[VELZ];
    Bm(MAGX, MAGX) = 1.0;
    Bm(PRES, MAGX) = k * V[MAGX];
    Bm(MAGY, MAGY) = 1.0;
    Bm(PRES, MAGY) = k * V[MAGY];
    Bm(MAGZ, MAGZ) = 1.0;
    Bm(PRES, MAGZ) = k * V[MAGZ];
    Bm(PRES, PRES) = -k;
    double Rc[NCONS * NCONS], Lc[NCONS * NCONS];
    for (int j = 0; j < NCONS; j++)
        for (int i = 0; i < NCONS; i++) {
            double r = 0.0, l = 0.0;
            for (int q = 0; q < NCONS; q++) {
                r = r + A(i, q) * Rm[q + NCONS * j];
                l = l + Bm(q, i) * Lm[q + NCONS * j];
            }
            Rc[i + NCONS * j] = r;
            Lc[i + NCONS * j] = l;
        }
#undef A
#undef Bm
    for (int q = 0; q < NCONS * NCONS; q++) {
        Rm[q] = Rc[q];
        Lm[q] = Lc[q];
    }
}

}  // namespace hosono
