// flux_fp64.cuh -- the reference's face physics in FP64, operation for
// operation. Included only by translation units built with -fmad=false, so
// that no multiply-add is contracted and every result is the IEEE-rounded
// value the reference's Fortran produces without FMA:
//   cell_prims_fp64, roe_flux_prim_fp64
//                      flux_2d_module.F90:63-182 (flux_roe_2d)
//   residual_rate      solver_residual_subgrid_2d_module.F90 (-R / volume)
//   bc_flux_fp64       bc_2d_module.F90:14-75 + flux_2d_module.F90:13-60
//   cfl_candidate_fp64 solver_time_step_2d_module.F90:106-116
// gamma = 1.4 and gm1 = 0.4 are hard-coded exactly as there; the flux's
// pressure uses (gamma - 1) = 0.3999999999999999, its sound speed 0.4.
#pragma once

namespace amrgpu {

// ---- division and square root without branches
//
// An IEEE division or square root is an approximation, its refinement and a
// range check that branches to a slow path. A face flux holds eleven of
// them, and behind those branches the compiler can neither interleave
// independent ones nor share work between quotients of one divisor: the
// stage kernels waited on that chain (FP64 pipe 41-45% busy). The functions
// below return the same bits from fused multiply-adds alone, for operands
// whose ranges are checked once per cell:
//   recip_rn     RN(1/b): the approximation y0, two factors of Goldschmidt's
//                product y0 (1 + e) (1 + e^2), e = 1 - b y0 (R. E. Goldschmidt,
//                "Applications of division by convergence", MIT, 1964), then
//                y + y (1 - b y), which rounds correctly for every mantissa
//                but all ones (P. Markstein, "Computation of elementary
//                functions on the IBM RISC System/6000 processor", 1990).
//                Markstein's step wants a y within one last place: next to a
//                rounding boundary the product is one of the two doubles
//                around 1/b (its two roundings are half a place each, and the
//                doubles beyond are one and a half away). All ones ends on
//                the tie 1/2, one last place too low, and is set
//   quotient_by  RN(a/b) from y = RN(1/b): q = RN(a y), then
//                RN(q + y RN(a - b q)) (Markstein; N. Brisebarre,
//                J.-M. Muller and S. K. Raina, "Accelerating correctly
//                rounded floating-point division when the divisor is known
//                in advance", 2004)
//   sqrt_rn      RN(sqrt(x)): two coupled Goldschmidt steps for g = sqrt(x)
//                and h = 1 / (2 sqrt(x)), then g + h (x - g g). The sum is
//                within 2^-51 last places of the root, and a root lies that
//                close to a rounding boundary only for mantissas with
//                x = k^2 + k + c, |c| <= 4 (in last places), which are
//                among those checked
// test_gpu_fp64_ops.py calls the three and finds no bit different from IEEE
// in 5 x 2^30 random operands, the 4096 mantissas at each end of the binade,
// the roots' mantissas with |c| <= 4000 and 20,000 quotients within 2^-103 of
// a boundary, out to both ends of the stated ranges.
//
// Ranges: a cell record is marked (sign bit of its sqrt(rho), see
// cell_prims_fp64) unless rho lies in [2^-110, 2^110), rho E / rho in
// [2^-80, 2^80), and each velocity is in [2^-160, 2^100) or its momentum
// zero: the density's unit is free (1e-33 .. 1e33: CGS and SI, interstellar
// gas too), for the flux depends on it by a factor only. From unmarked
// states and a normal of length [2^-100, 2^100) whose components are zero or
// at least 2^-100 of it, every divisor of the flux lies in [2^-301, 2^251),
// every radicand in [2^-300, 2^220), every numerator is zero or in
// [2^-840, 2^514) and every quotient zero or in [2^-943, 2^637) (all values
// are whole multiples of their operands' last places, so a difference is
// zero or no smaller than those), and so nothing under- or overflows on the
// way; or the flux is NaN either way (a negative or zero square under a
// root). Everything else takes the IEEE operations.
__device__ __forceinline__ bool hi_outside(double x, int lo_exp, int hi_exp)
{
    // the biased exponent field: NaN, infinities, zero and (x as given, not
    // |x|) negative values are outside
    return (unsigned)(__double2hiint(x) - ((1023 + lo_exp) << 20)) >= (unsigned)((hi_exp - lo_exp) << 20);
}

// |x| neither zero nor in [2^lo_exp, 2^hi_exp)
__device__ __forceinline__ bool abs_outside_or_zero(double x, int lo_exp, int hi_exp)
{
    const unsigned h = (unsigned)__double2hiint(x) & 0x7fffffffu;
    return (h | (unsigned)__double2loint(x)) != 0u &&
           h - (unsigned)((1023 + lo_exp) << 20) >= (unsigned)((hi_exp - lo_exp) << 20);
}

// m not zero and |x| not in [2^lo_exp, 2^hi_exp). (A product of tests, not a
// chain of branches: 1024^2 RK3 250.0 us per step with &&, 247.7 us.)
__device__ __forceinline__ bool abs_outside_unless_zero(double x, double m, int lo_exp, int hi_exp)
{
    const unsigned h = (unsigned)__double2hiint(x) & 0x7fffffffu;
    return (m != 0.0) & (h - (unsigned)((1023 + lo_exp) << 20) >= (unsigned)((hi_exp - lo_exp) << 20));
}

// RN(1/b), |b| in [2^-500, 2^500]
__device__ __forceinline__ double recip_rn(double b)
{
    double y;
    asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(b));
    double e = __fma_rn(-b, y, 1.0);
    y = __fma_rn(y, e, y);
    e = e * e;
    y = __fma_rn(y, e, y);
    e = __fma_rn(-b, y, 1.0);
    y = __fma_rn(y, e, y);
    const unsigned ones = (unsigned)__double2loint(b) & ((unsigned)__double2hiint(b) | 0xfff00000u);
    return __hiloint2double(__double2hiint(y), ones == 0xffffffffu ? 1 : __double2loint(y));
}

// RN(sqrt(x)), x in [2^-500, 2^500]
__device__ __forceinline__ double sqrt_rn(double x)
{
    double y;
    asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(x));
    double g = x * y, h = 0.5 * y;
    double r = __fma_rn(-g, h, 0.5);
    g = __fma_rn(g, r, g);
    h = __fma_rn(h, r, h);
    r = __fma_rn(-g, h, 0.5);
    g = __fma_rn(g, r, g);
    h = __fma_rn(h, r, h);
    return __fma_rn(__fma_rn(-g, g, x), h, g);
}

// RN(a/b) from y = RN(1/b): a zero or |a| in [2^-850, 2^700], |b| in
// [2^-320, 2^320], |a/b| in [2^-950, 2^950]
__device__ __forceinline__ double quotient_by(double a, double b, double y)
{
    const double q = a * y;
    return __fma_rn(__fma_rn(-b, q, a), y, q);
}

// q[f] = (r[f] / vol) * -1.0, the residual of one cell: each r[f] zero or in
// [2^-700, 2^700) and vol in [2^-200, 2^200), else IEEE divisions.
__device__ __forceinline__ void residual_rate(const double r[4], double vol, double k[4])
{
    const double y = recip_rn(vol);
    bool odd = hi_outside(vol, -200, 200);
#pragma unroll
    for (int f = 0; f < 4; ++f) odd |= abs_outside_or_zero(r[f], -700, 700);
    if (__builtin_expect(odd, 0)) {
#pragma unroll
        for (int f = 0; f < 4; ++f) k[f] = (r[f] / vol) * -1.0;
    } else {
#pragma unroll
        for (int f = 0; f < 4; ++f) k[f] = quotient_by(r[f], vol, y) * -1.0;
    }
}

// Per-cell primitive record shared by the four faces of a cell:
// [0] rho [1] rho*u [2] rho*v [3] rho*E [4] u [5] v [6] p [7] H [8] sqrt(rho),
// each computed by exactly the expression flux_roe_2d uses
// (flux_2d_module.F90:93-99, 113-118), so reusing them is bit-exact. The
// sign bit of [8] marks a state outside the ranges of quotient_by's use (the
// root itself is never negative; its readers take the absolute value).
__device__ __forceinline__ void cell_prims_fp64(const double q[4], double P[9])
{
    const double gamma = 1.4;
    const double half = 0.5;
    double rho = q[0];
    bool odd = hi_outside(rho, -110, 110);
    double oneOrho = recip_rn(rho), sr = sqrt_rn(rho);
    if (__builtin_expect(odd, 0)) {
        oneOrho = 1.0 / rho;
        sr = sqrt(rho);
    }
    double u = q[1] * oneOrho;
    double v = q[2] * oneOrho;
    double E = q[3] * oneOrho;
    // (a velocity may underflow to zero where its momentum is not)
    odd = odd | hi_outside(E, -80, 80) | abs_outside_unless_zero(u, q[1], -160, 100) |
          abs_outside_unless_zero(v, q[2], -160, 100);
    double p = (gamma - 1.0) * (q[3] - half * rho * (u * u + v * v));
    P[0] = q[0];
    P[1] = q[1];
    P[2] = q[2];
    P[3] = q[3];
    P[4] = u;
    P[5] = v;
    P[6] = p;
    P[7] = E + p * oneOrho;
    // (the bit itself: the negative of a NaN keeps no sign)
    P[8] = __hiloint2double(__double2hiint(sr) | (odd ? (int)0x80000000 : 0), __double2loint(sr));
}

// The operations of the flux: IEEE, or the branch-free ones above.
struct IeeeOps {
    __device__ static __forceinline__ double recip(double b) { return 1.0 / b; }
    __device__ static __forceinline__ double root(double x) { return sqrt(x); }
    __device__ static __forceinline__ double over(double a, double b, double) { return a / b; }
};
struct FastOps {
    __device__ static __forceinline__ double recip(double b) { return recip_rn(b); }
    __device__ static __forceinline__ double root(double x) { return sqrt_rn(x); }
    __device__ static __forceinline__ double over(double a, double b, double y) { return quotient_by(a, b, y); }
};

// flux_roe_2d on primitive records, unit normal (nx, ny) and length mag.
// AXIS: the normal is +x (nx = 1, ny = 0), and the terms that are zero then
// are left out: a value plus or minus zero is the value. Only a zero's sign
// can differ, which no residual keeps (the sums start at +0). For a +y
// normal the caller swaps the two momenta and velocities: every expression
// below maps onto itself then, the sums of two products included.
template <bool AXIS, class O>
__device__ __forceinline__ void roe_flux_ops(const double *L, const double *R, double nx, double ny, double mag,
                                             double flux[4])
{
    const double gm1 = 0.4;
    const double half = 0.5;
    const double rhol = L[0], ul = L[4], vl = L[5], pl = L[6], Hl = L[7], srl = fabs(L[8]);
    const double rhor = R[0], ur = R[4], vr = R[5], pr = R[6], Hr = R[7], srr = fabs(R[8]);
    const double unl = AXIS ? ul : ul * nx + vl * ny;
    const double unr = AXIS ? ur : ur * nx + vr * ny;
    const double oneOroe_fact = O::recip(srl + srr);
    const double rhobar = O::root(rhol * rhor);
    const double ubar = (ul * srl + ur * srr) * oneOroe_fact;
    const double vbar = (vl * srl + vr * srr) * oneOroe_fact;
    const double Hbar = (Hl * srl + Hr * srr) * oneOroe_fact;
    const double abar = O::root(gm1 * (Hbar - half * (ubar * ubar + vbar * vbar)));
    const double unbar = AXIS ? ubar : ubar * nx + vbar * ny;
    const double Mnbar = O::over(unbar, abar, O::recip(abar));
    const double eigp = unbar + abar;
    const double eigm = unbar - abar;
    const double eigp_max = unr + abar;
    const double eigm_min = unl - abar;
    const double b1 = (eigp > 0.0 || eigp_max > 0.0) ? ((eigp > eigp_max) ? eigp : eigp_max) : 0.0;
    const double b2 = (eigm < 0.0 || eigm_min < 0.0) ? ((eigm < eigm_min) ? eigm : eigm_min) : 0.0;
    const double db = b1 - b2;
    const double y = O::recip(db);
    const double aa = abar * abar;
    const double delta1 = (rhor - rhol) - O::over(pr - pl, aa, O::recip(aa));
    const double Mcoeff = O::recip(1.0 + fabs(Mnbar));
    const double bcoeff = O::over(b1 * b2, db, y);
    const double bM = bcoeff * Mcoeff;
    double fluxl, fluxr, disp;

    fluxl = AXIS ? L[1] : L[1] * nx + L[2] * ny;
    fluxr = AXIS ? R[1] : R[1] * nx + R[2] * ny;
    disp = bcoeff * (rhor - rhol) - bM * delta1;
    flux[0] = (O::over(b1 * fluxl - b2 * fluxr, db, y) + disp) * mag;

    fluxl = AXIS ? L[1] * ul + pl : (L[1] * ul + pl) * nx + (L[2] * ul) * ny;
    fluxr = AXIS ? R[1] * ur + pr : (R[1] * ur + pr) * nx + (R[2] * ur) * ny;
    disp = bcoeff * (R[1] - L[1]) -
           bM * (AXIS ? delta1 * ubar : delta1 * ubar + rhobar * (ur - ul - nx * (unr - unl)));
    flux[1] = (O::over(b1 * fluxl - b2 * fluxr, db, y) + disp) * mag;

    fluxl = AXIS ? L[1] * vl : (L[1] * vl) * nx + (L[2] * vl + pl) * ny;
    fluxr = AXIS ? R[1] * vr : (R[1] * vr) * nx + (R[2] * vr + pr) * ny;
    disp = bcoeff * (R[2] - L[2]) -
           bM * (delta1 * vbar + rhobar * (AXIS ? vr - vl : vr - vl - ny * (unr - unl)));
    flux[2] = (O::over(b1 * fluxl - b2 * fluxr, db, y) + disp) * mag;

    fluxl = (L[3] + pl) * unl;
    fluxr = (R[3] + pr) * unr;
    disp = bcoeff * (rhor * Hr - rhol * Hl) - bM * (delta1 * Hbar + rhobar * (Hr - Hl));
    flux[3] = (O::over(b1 * fluxl - b2 * fluxr, db, y) + disp) * mag;
}

// Any normal and any states: called, not inlined (one copy per call site
// would crowd the instruction cache and spill). On a domain whose width and
// corner are powers of two or whole numbers no interior normal is off its
// axis; on any other (width 0.7, corner 0.1) rounding of the nodes tilts a
// quarter to a third of them, so that nearly every row has one and its warp
// comes here: 1024^2 RK3 takes 312 us per step there against 249 us (380 and
// 356 us with every division and root IEEE's own). Records and flux in
// (x, y) components; by value: as scalars they cost the callers 20-60 bytes
// more spills a thread.
struct Flux4 {
    double v[4];
};
struct Record9 {
    double v[9];
};
static __device__ __noinline__ Flux4 roe_flux_any(Record9 L, Record9 R, double n0, double n1)
{
    Flux4 f;
    double mag, nx, ny;
    bool odd = (__double2hiint(L.v[8]) | __double2hiint(R.v[8])) < 0;
    // For an axis-aligned normal (one component exactly zero) |n| =
    // sqrt(n0*n0) is |n0| exactly in IEEE round-to-nearest and n0/|n0| = +-1,
    // n1/|n0| = n1 (a signed zero), so the shortcut returns the same bits as
    // the general path.
    const double nn = n0 * n0 + n1 * n1;
    if (n1 == 0.0 && fabs(n0) > 1e-150) {
        mag = fabs(n0);
        nx = n0 > 0.0 ? 1.0 : -1.0;
        ny = n1;
    } else if (n0 == 0.0 && fabs(n1) > 1e-150) {
        mag = fabs(n1);
        nx = n0;
        ny = n1 > 0.0 ? 1.0 : -1.0;
    } else if (hi_outside(nn, -200, 200) || abs_outside_or_zero(n0, -300, 300) || abs_outside_or_zero(n1, -300, 300)) {
        mag = sqrt(nn);
        nx = n0 / mag;
        ny = n1 / mag;
        odd = true;
    } else {
        mag = sqrt_rn(nn);
        const double y = recip_rn(mag);
        nx = quotient_by(n0, mag, y);
        ny = quotient_by(n1, mag, y);
        odd |= !(fmin(fabs(nx), fabs(ny)) >= 0x1p-100);
    }
    odd |= hi_outside(mag, -100, 100);
    if (odd) roe_flux_ops<false, IeeeOps>(L.v, R.v, nx, ny, mag, f.v);
    else roe_flux_ops<false, FastOps>(L.v, R.v, nx, ny, mag, f.v);
    return f;
}

// flux_roe_2d on primitive records for the face normal (n0, n1). DIR = 0 / 1:
// the normal is meant along +x / +y (a cell face of a rectangle; rounding of
// its nodes may still tilt it); 2: either, decided per lane.
template <int DIR>
__device__ __forceinline__ void roe_flux_prim_fp64(const double *L, const double *R, double n0, double n1,
                                                   double flux[4])
{
    const bool swap = DIR == 2 ? n0 == 0.0 : DIR == 1;
    const double along = swap ? n1 : n0, across = swap ? n0 : n1;
    // out of range: NaN, negative and tiny lengths too
    const bool odd = ((__double2hiint(L[8]) | __double2hiint(R[8])) < 0) || across != 0.0 ||
                     hi_outside(along, -100, 100);
    // for the whole warp: lanes on both paths would run one after the other
    if (__builtin_expect(__any_sync(__activemask(), odd), 0)) {
        Record9 l, r;
#pragma unroll
        for (int c = 0; c < 9; ++c) {
            l.v[c] = L[c];
            r.v[c] = R[c];
        }
        const Flux4 f = roe_flux_any(l, r, n0, n1);
#pragma unroll
        for (int c = 0; c < 4; ++c) flux[c] = f.v[c];
    } else {
        const double A[9] = {L[0], swap ? L[2] : L[1], swap ? L[1] : L[2], L[3], swap ? L[5] : L[4],
                             swap ? L[4] : L[5], L[6], L[7], L[8]};
        const double B[9] = {R[0], swap ? R[2] : R[1], swap ? R[1] : R[2], R[3], swap ? R[5] : R[4],
                             swap ? R[4] : R[5], R[6], R[7], R[8]};
        double f[4];
        roe_flux_ops<true, FastOps>(A, B, 1.0, 0.0, along, f);
        flux[0] = f[0];
        flux[1] = swap ? f[2] : f[1];
        flux[2] = swap ? f[1] : f[2];
        flux[3] = f[3];
    }
}

// Boundary face: ghost state of bc_2d, then the physical flux F.n of
// flux_bc_2d. bc 3 (extension, no reference counterpart): prescribed state
// qin, used for supersonic inflow.
__device__ __forceinline__ void bc_flux_fp64(int bc, const double q[4], double n0, double n1,
                                             const double qin[4], double flux[4])
{
    const double gamma = 1.4;
    double qb[4];
    double rho = q[0];
    double oneOrho = 1.0 / rho;
    double u = q[1] * oneOrho;
    double v = q[2] * oneOrho;
    if (bc == 1) {
        double mag = sqrt(n0 * n0 + n1 * n1);
        double nx = n0 / mag;
        double ny = n1 / mag;
        double U_dot_n = u * nx + v * ny;
        double ub = u - U_dot_n * nx;
        double vb = v - U_dot_n * ny;
        qb[0] = q[0];
        qb[1] = q[0] * ub;
        qb[2] = q[0] * vb;
        qb[3] = q[3];
    } else if (bc == 2) {
        qb[0] = q[0];
        qb[1] = 0.0;
        qb[2] = 0.0;
        qb[3] = q[3] - 0.5 * rho * (u * u + v * v);
    } else if (bc == 3) {
        qb[0] = qin[0]; qb[1] = qin[1]; qb[2] = qin[2]; qb[3] = qin[3];
    } else {
        qb[0] = q[0]; qb[1] = q[1]; qb[2] = q[2]; qb[3] = q[3];
    }
    // flux_native_2d
    double r = qb[0];
    double oor = 1.0 / r;
    double ub2 = qb[1] * oor;
    double vb2 = qb[2] * oor;
    double p = (gamma - 1.0) * (qb[3] - 0.5 * r * (ub2 * ub2 + vb2 * vb2));
    double fx0 = qb[1], fx1 = qb[1] * ub2 + p, fx2 = qb[1] * vb2, fx3 = ub2 * (qb[3] + p);
    double fy0 = qb[2], fy1 = qb[2] * ub2, fy2 = qb[2] * vb2 + p, fy3 = vb2 * (qb[3] + p);
    flux[0] = fx0 * n0 + fy0 * n1;
    flux[1] = fx1 * n0 + fy1 * n1;
    flux[2] = fx2 * n0 + fy2 * n1;
    flux[3] = fx3 * n0 + fy3 * n1;
}

// One cell's CFL step candidate: cfl*sqrt(volume)/(|V| + c).
__device__ __forceinline__ double cfl_candidate_fp64(const double q[4], double volume, double cfl)
{
    const double gamma = 1.4;
    const double gm1 = 0.4;
    double oneOrho = 1.0 / q[0];
    double u = q[1] * oneOrho;
    double v = q[2] * oneOrho;
    double V2 = u * u + v * v;
    double pOverRho = gm1 * (q[3] * oneOrho - 0.5 * V2);
    double c = sqrt(gamma * pOverRho);
    double eig = sqrt(V2) + c;
    return cfl * sqrt(volume) / eig;
}

}  // namespace amrgpu
