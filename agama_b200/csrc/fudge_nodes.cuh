// The Staeckel fudge from the node form of the splines: actions with angles and frequencies.
//
// An angle is the integral from a turning point to the star, whose distance from the turning point
// enters as a square root: next to it (one star in 1e5 lies within 1e-10 of the range) a change of
// the limit in its last bits moves the angle by 1e-7 and more.  The phases of the angles therefore
// keep one arithmetic inside the radial grid to the last bit, that of the node form, and with it their own
// text of phase 1 (a text shared with the cells' form compiles to other contractions of multiply and
// add); the actions alone are smooth in the limits and take the cells (fudge.cuh).  Beyond the grid the
// expansions are one inline loop (axisPowerLaw), which moves the angles of orbits that get there by
// rounding (1e-11 relative for 7 % of the stars about a grid of 0.3 to 6 scale radii).
#pragma once
#include "fudge.cuh"
#include "multipole_force.cuh"

namespace agb {

/// the fudge's auxiliary function F(tau) and the integrals of motion of one point
struct FudgeFunction {
    const MultipoleView* M;
    double lambda, nu, D2;          // point in prolate spheroidal coordinates (Delta^2 = D2)
    double E, Lz, I3, flambda, fnu;
    double Ilam, Inu, L2h;          // I3 - fnu, I3 - flambda and Lz^2 / 2, formed once (derive())

    /// the terms of F that do not depend on tau, from the integrals of motion (the same
    /// operations as in F itself, so the same bits)
    __device__ void derive() { Ilam = I3 - fnu; Inu = I3 - flambda; L2h = Lz * Lz / 2; }

    /// F(tau) and optionally F', F'' (src/actions_staeckel.cpp:202-252); INL: the potential
    /// evaluation inlined at this call site instead of the shared out-of-line copy
    template<bool DER, bool DER2, bool INL = false>
    __device__ void eval(double tau, double* val, double* der, double* der2) const
    {
        double lam, n, mult, I;
        if(tau >= D2) { lam = tau; n = fabs(nu); mult = lam - n; I = Ilam; }
        else          { lam = lambda; n = tau; mult = n - lam; I = Inu; }
        // prolate spheroidal -> cylindrical (src/coord.cpp:266-291)
        const double absnu = fabs(n), sgn = n >= 0 ? 1 : -1;
        const double lmd = lam - D2, nmd = absnu - D2;
        if(nmd > 0 || lmd < 0) {
            *val = NAN; if(DER) *der = NAN; if(DER2) *der2 = NAN;
            return;
        }
        const double R = sqrt(lmd * (1 - absnu / D2));
        const double z = sqrt(lam * absnu / D2) * sgn;
        double Phi;
        CylDerivs g; CylHess h;
        if(INL)      evalMultipoleCyl<DER2 ? 6 : DER ? 3 : 1, EVAL_AXI>(*M, R, z, 0, &Phi, &g, &h);
        else if(DER2) evalMultipoleCylCall<6, EVAL_AXI>(*M, R, z, 0, &Phi, &g, &h);
        else if(DER) evalMultipoleCylCall<3, EVAL_AXI>(*M, R, z, 0, &Phi, &g, &h);
        else         evalMultipoleCylCall<1, EVAL_AXI>(*M, R, z, 0, &Phi, &g, &h);
        const double tmd = tau - D2;
        *val = (tmd != 0 ? (E * tau - I - Phi * mult) * tmd : 0) - L2h * tau;
        if(DER || DER2) {
            // dR/dtau, dz/dtau along the coordinate that tau moves (lambda or nu): only that pair
            // is divided out
            const bool lbranch = tau >= D2;
            double dRdt, dzdt;
            if(lbranch) { dRdt = 0.5 * R / lmd; dzdt = 0.5 * z / lam; }
            else        { dRdt = 0.5 * R / nmd * sgn; dzdt = 0.5 * z / n; }
            const double dPhidtau = g.dR * dRdt + g.dz * dzdt;
            if(DER)
                *der = E * (tau + tmd) - L2h - I - (mult + tmd) * Phi -
                       (tmd != 0 ? tmd * mult * dPhidtau : 0);
            if(DER2) {
                double d2;
                if(lbranch) {
                    const double d2Rdl2 = -0.25 * R / pow2(lmd), d2zdl2 = -0.25 * z / pow2(lam);
                    d2 = h.dR2 * pow2(dRdt) + h.dz2 * pow2(dzdt) + 2 * h.dRdz * dRdt * dzdt +
                         g.dR * d2Rdl2 + g.dz * d2zdl2;
                } else {
                    const double d2Rdn2 = -0.25 * R / pow2(nmd), d2zdn2 = -0.25 * z / pow2(n);
                    d2 = h.dR2 * pow2(dRdt) + h.dz2 * pow2(dzdt) + 2 * h.dRdz * dRdt * dzdt +
                         g.dR * d2Rdn2 + g.dz * d2zdn2;
                }
                *der2 = 2 * (E - Phi - (mult + tmd) * dPhidtau) - tmd * mult * d2;
            }
        }
    }
    __device__ double value(double tau) const { double v; eval<false, false, true>(tau, &v, nullptr, nullptr); return v; }
};

/** The point's F(tau) from its record.  The azimuth given to the potential is 0: the fudge takes
    only axisymmetric potentials, whose coefficients (and so the index sets of their splines and
    asymptotes) have m = 0 alone, and their evaluators never read the azimuth; a constant leaves
    the register free for the searches (the record keeps the point's azimuth for the angles). */
__device__ __forceinline__ void loadFudgeFunction(const MultipoleView& M, const FudgeRecord& r, FudgeFunction& f)
{
    f.M = &M;
    f.lambda = r.lambda; f.nu = r.nu; f.D2 = r.D2;
    f.E = r.E; f.Lz = r.Lz; f.I3 = r.I3; f.flambda = r.flambda; f.fnu = r.fnu;
    f.derive();
}

/// the root functions of the integration limits (as limitRootEval of the cells' form)
__device__ __forceinline__ void limitRootEval(const FudgeFunction& f, int kind, double u0, double x,
    double* v, double* d)
{
    const bool semiInf = kind == ROOT_LAMBDA_MAX;
    double duds = 1, tau = x;
    if(semiInf) tau = unscaleSemiInf(u0, x, &duds);
    const bool far = semiInf && tau > 1e100;
    double fval = 0, fder = 0;
    if(!far) f.eval<true, false, true>(tau, &fval, &fder, nullptr);
    if(!semiInf) { *v = fval; *d = fder; }
    else if(far) { *v = f.E; *d = NAN; }
    else {
        *v = fval / pow2(tau);
        *d = (fder - 2 * fval / tau) / pow2(tau) * duds;
    }
}

/// F(tau) of one branch (FudgeFunction::eval, to the bit inside the radial grid) in a potential with cells, without
/// calls; D2inv = 1 / D2
static __device__ __forceinline__ double branchValue(const FudgeFunction& f, double D2inv, double tau)
{
    const MultipoleView& M = *f.M;
    const bool lambda = tau >= f.D2;
    const double lam = lambda ? tau : f.lambda, n = lambda ? fabs(f.nu) : tau;
    const double mult = lambda ? lam - n : n - lam, I = lambda ? f.Ilam : f.Inu;
    const double absnu = fabs(n), lmd = lam - f.D2, nmd = absnu - f.D2;
    if(nmd > 0 || lmd < 0) return NAN;
    // coordinates that leave the range of normal numbers take the library's roots
    const double R2 = lmd * (1 - quotient(absnu, f.D2, D2inv)), z2 = quotient(lam * absnu, f.D2, D2inv);
    const bool usual = R2 > 1e-200 && R2 < 1e200 && z2 > 1e-200 && z2 < 1e200;
    const double R = usual ? squareRoot(R2) : sqrt(R2), z = (usual ? squareRoot(z2) : sqrt(z2)) * (n >= 0 ? 1 : -1);
    const double rsq = sumProducts(z, z, R, R);
    const double Phi = inCells(M, rsq) ? valueInterp2d(M, R, z) : axisPowerLaw<false>(rsq < M.rInnerSq ? M.inner : M.outer, R, z, rsq, nullptr, nullptr);
    const double tmd = tau - f.D2;
    return fma(-f.L2h, tau, tmd != 0 ? fma(-Phi, mult, fma(f.E, tau, -I)) * tmd : 0);
}

/// the same with F'(tau)
static __device__ __forceinline__ void branchSlope(const FudgeFunction& f, double D2inv, double tau, double* val, double* der)
{
    const MultipoleView& M = *f.M;
    const bool lambda = tau >= f.D2;
    const double lam = lambda ? tau : f.lambda, n = lambda ? fabs(f.nu) : tau;
    const double mult = lambda ? lam - n : n - lam, I = lambda ? f.Ilam : f.Inu;
    const double absnu = fabs(n), lmd = lam - f.D2, nmd = absnu - f.D2;
    if(nmd > 0 || lmd < 0) { *val = *der = NAN; return; }
    const double R2 = lmd * (1 - quotient(absnu, f.D2, D2inv)), z2 = quotient(lam * absnu, f.D2, D2inv);
    const bool usual = R2 > 1e-200 && R2 < 1e200 && z2 > 1e-200 && z2 < 1e200;
    const double sgn = n >= 0 ? 1 : -1;
    const double R = usual ? squareRoot(R2) : sqrt(R2), z = (usual ? squareRoot(z2) : sqrt(z2)) * sgn;
    double Phi;
    CylDerivs g;
    const double rsq = sumProducts(R, R, z, z);     // (the value alone adds them the other way round)
    if(inCells(M, rsq)) forceInterp2d<EVAL_AXI, 1, false>(M, R, z, rsq, 0, &Phi, &g);
    else                Phi = axisPowerLaw<true>(rsq < M.rInnerSq ? M.inner : M.outer, R, z, rsq, &g.dR, &g.dz);
    const double tmd = tau - f.D2;
    *val = fma(-f.L2h, tau, tmd != 0 ? fma(-Phi, mult, fma(f.E, tau, -I)) * tmd : 0);
    // dR/dtau, dz/dtau along the coordinate that tau moves
    const double dR = lambda ? lmd : nmd, dz = lambda ? lam : n;
    double dRdt, dzdt;
    if(usual) { dRdt = quotient(0.5 * R, dR, reciprocal(dR)); dzdt = quotient(0.5 * z, dz, reciprocal(dz)); }
    else      { dRdt = 0.5 * R / dR; dzdt = 0.5 * z / dz; }
    if(!lambda) dRdt *= sgn;
    const double dPhidtau = sumProducts(g.dR, dRdt, g.dz, dzdt);
    *der = fma(-(mult + tmd), Phi, fma(f.E, tau + tmd, -f.L2h) - I) - (tmd != 0 ? tmd * mult * dPhidtau : 0);
}

/// limitRootEval of a potential with cells
static __device__ __forceinline__ void limitRootSegments(const FudgeFunction& f, double D2inv, int kind, double u0, double x,
    double* v, double* d)
{
    const bool semiInf = kind == ROOT_LAMBDA_MAX;
    double duds = 1, tau = x;
    if(semiInf) {       // unscaleSemiInf (u0 > Delta^2 > 0; x = 1 gives NaN: far)
        const double w = 1 - x, w2 = pow2(w);
        tau = u0 * exp(quotient(x, w, reciprocal(w)));
        duds = quotient(tau, w2, reciprocal(w2));
    }
    const bool far = semiInf && !(tau <= 1e100);
    double fval = 0, fder = 0;
    if(!far) branchSlope(f, D2inv, tau, &fval, &fder);
    if(!semiInf) { *v = fval; *d = fder; }
    else if(far) { *v = f.E; *d = NAN; }
    else {
        const double tau2 = pow2(tau), y2 = reciprocal(tau2);
        *v = quotient(fval, tau2, y2);
        *d = quotient(fder - quotient(2 * fval, tau, reciprocal(tau)), tau2, y2) * duds;
    }
}

/** Integration limits of the lambda and nu motions (findIntegrationLimitsAxisym,
    src/actions_staeckel.cpp:360-483), part 1: every decision up to the three root searches, whose
    brackets go into the record; limits that need no root are stored directly (NaN otherwise).
    ends receives F and F' at the ends of the plain brackets (FudgeEnds), which the
    root searches then take instead of evaluating them: at lambda_pos from the evaluation above,
    at Delta^2 and |nu| from the same evaluation of F as the searches would make. */
static __device__ void nodeLimitsSetup(const FudgeFunction& fnc, FudgeRecord& rec, FudgeEnds* ends)
{
    const double delta = fnc.D2;
    const double f_zero = fnc.value(0);
    double f_lambda, df_lambda, d2f_lambda;
    fnc.eval<true, true>(fnc.lambda, &f_lambda, &df_lambda, &d2f_lambda);
    double nu_max = NAN, lambda_min = NAN, lambda_max = NAN;
    double nu_upper = delta, lambda_lower = delta;
    int roots = 0;
    if(fnc.Lz == 0) {
        const double dminus = delta * (1 - 1e-15), dplus = delta * (1 + 1e-15);
        if(fnc.value(dminus) < 0) {
            if(f_zero > 0) nu_upper = dminus;
            else nu_max = 0;
        } else
            nu_max = delta;
        if(fnc.value(dplus) < 0) lambda_lower = dplus;
        else lambda_min = delta;
    }
    if(!isFinite(nu_max)) {
        if(f_zero > 0) roots |= ROOT_NU_MAX;           // falls back to |nu| if no root is found
        else nu_max = fabs(fnc.nu);
    }
    double lambda_pos = fnc.lambda, f_pos = f_lambda, df_pos = df_lambda;
    const double dxToRoot = -f_lambda / df_lambda;
    if(f_lambda <= 0 || fabs(dxToRoot) < fnc.lambda * FUDGE_MINIMUM_RANGE) {
        if(df_lambda >= 0) lambda_min = fnc.lambda;
        if(df_lambda <= 0) {
            lambda_max = fnc.lambda;
            if(fnc.lambda == delta) lambda_min = delta;
        }
        bool nearShell = d2f_lambda < 0 &&
            pow2(df_lambda) - 2 * f_lambda * d2f_lambda - pow2(fnc.lambda * FUDGE_MINIMUM_RANGE * d2f_lambda) < 0;
        const double safeOffset = fmin(0.5 * fabs(df_lambda / d2f_lambda), fnc.lambda * FUDGE_MINIMUM_RANGE);
        lambda_pos += fmax(dxToRoot, safeOffset) * (df_lambda >= 0 ? 1 : -1);
        double f_lp, df_lp, d2f_lp;
        fnc.eval<true, true>(lambda_pos, &f_lp, &df_lp, &d2f_lp);
        f_pos = f_lp; df_pos = df_lp;
        nearShell |= d2f_lp < 0 &&
            pow2(df_lp) - 2 * f_lp * d2f_lp - pow2(fnc.lambda * FUDGE_MINIMUM_RANGE * d2f_lp) < 0;
        if(nearShell || f_lp < 0)
            lambda_min = lambda_max = fnc.lambda;
    }
    if(!isFinite(lambda_min)) roots |= ROOT_LAMBDA_MIN;
    if(!isFinite(lambda_max)) roots |= ROOT_LAMBDA_MAX;
    rec.nuMax = nu_max; rec.lambdaMin = lambda_min; rec.lambdaMax = lambda_max;
    rec.nuUpper = nu_upper; rec.lambdaLower = lambda_lower; rec.lambdaPos = lambda_pos;
    rec.roots = roots;
    ends->fPos = f_pos; ends->dfPos = df_pos;
    ends->fD2 = ends->dfD2 = ends->fNu = ends->dfNu = NAN;
    if(((roots & ROOT_NU_MAX) && nu_upper == delta) || ((roots & ROOT_LAMBDA_MIN) && lambda_lower == delta))
        fnc.eval<true, false>(delta, &ends->fD2, &ends->dfD2, nullptr);
    if(roots & ROOT_NU_MAX)
        fnc.eval<true, false>(fabs(fnc.nu), &ends->fNu, &ends->dfNu, nullptr);
}

/** Phase 1 of the actions of one point (R, z, phi, vR, vz, vphi) for focal distance fd
    (evalAxisymFudge, src/actions_staeckel.cpp:683-693: fd <= 0 falls back to max(R,1)*1e-4);
    Phi is the potential at the point.  Writes Jphi into act[2]; for a point without actions
    (unbound, or lambda = nu = Delta^2) also NaN into act[0..1] and marks the record invalid.
    Otherwise the record holds the integrals of motion (findIntegralsOfMotionAxisymFudge,
    :176-195) and the limits and root brackets of nodeLimitsSetup (ends: as there). */
static __device__ void nodePrepare(const MultipoleView& M, const double* pc, double Phi, double fd,
    FudgeRecord& rec, double* act, FudgeEnds* ends)
{
    const double R = pc[0], z = pc[1], phi = pc[2], vR = pc[3], vz = pc[4], vphi = pc[5];
    if(fd <= 0) fd = fmax(R, 1.) * 1e-4;
    const double D2 = fd * fd;
    const double Lz = R * vphi;
    act[2] = Lz;
    rec.valid = 0;
    rec.roots = 0;
    // cylindrical -> prolate spheroidal (src/coord.cpp:294-338) and velocities (:525-531)
    const double R2 = R * R, z2 = z * z, signz = z >= 0 ? 1 : -1;
    const double sum = R2 + z2 + D2, dif = R2 + z2 - D2;
    double sqD = sqrt(pow2(dif) + 4 * R2 * D2);
    if(z2 == 0) sqD = sum;
    if(R2 == 0) sqD = fabs(dif);
    double lmd, dmn;
    if(dif >= 0) { lmd = 0.5 * (sqD + dif); dmn = R2 > 0 ? D2 * R2 / lmd : 0; }
    else         { dmn = 0.5 * (sqD - dif); lmd = D2 * R2 / dmn; }
    const double lambda = D2 + lmd;
    double absnu = 2 * D2 / (sum + sqD) * z2;
    if(absnu * 2 > D2) absnu = D2 - dmn; else dmn = D2 - absnu;
    if(sqD == 0) { act[0] = act[1] = NAN; return; }   // lambda = nu = Delta^2: undefined
    FudgeFunction fnc;
    fnc.M = &M;
    fnc.lambda = lambda;
    fnc.nu = absnu * signz;
    fnc.D2 = D2;
    double Phi0;
    CylDerivs g; CylHess h;
    evalMultipoleCylCall<1, EVAL_AXI>(M, sqrt(lambda - D2), 0, 0, &Phi0, &g, &h);
    const double Ekin = 0.5 * (vR * vR + vz * vz + vphi * vphi);
    fnc.E = Phi + Ekin;
    fnc.Lz = Lz;
    fnc.flambda = -lambda * Phi0;
    fnc.fnu = fnc.flambda + Phi * (lambda - absnu);
    fnc.I3 = lambda * (Phi - Phi0) + 0.5 * (pow2(z * vphi) + pow2(R * vz - z * vR) + pow2(vz) * D2);
    fnc.derive();
    if(!isFinite(fnc.E + fnc.I3 + fnc.Lz) || fnc.E >= 0) { act[0] = act[1] = NAN; return; }
    rec.lambda = fnc.lambda; rec.nu = fnc.nu; rec.D2 = D2; rec.E = fnc.E; rec.Lz = Lz; rec.I3 = fnc.I3;
    rec.flambda = fnc.flambda; rec.fnu = fnc.fnu; rec.phi = phi;
    nodeLimitsSetup(fnc, rec, ends);
    // velocities in prolate spheroidal coordinates (src/coord.cpp:317-322, :525-531)
    const double lambdadot = R * 2 * lambda / sqD * vR + z * 2 * lmd / sqD * vz;
    const double nudot = R * 2 * -absnu / sqD * signz * vR + z * 2 * dmn / sqD * signz * vz;
    rec.valid = REC_VALID | (lambdadot >= 0 ? REC_LDOT_POS : 0) | (nudot * fnc.nu >= 0 ? REC_NDOT_NU_POS : 0) |
        (nudot < 0 ? REC_NUDOT_NEG : 0);
}

/** Inverse of the cubic end-point scaling (math::scale of ScalingCub, src/math_core.cpp:370-386):
    s in [0, 1] with u = ul (1-s)^2 (1+2s) + ur s^2 (3-2s).  On the nearer half, w = s^2 (3 - 2s) is
    a depressed cubic in y = s - 1/2 whose trigonometric root s = 1/2 + cos((acos(1 - 2w) - 2pi)/3)
    is polished by three Newton steps; u outside [ul, ur] gives NaN, as in the reference. */
static __device__ double scaleCubInverse(double ul, double ur, double u)
{
    if(u == ul) return 0;
    if(u == ur) return 1;
    const double half = 0.5 * (ul + ur);
    if(u == half) return 0.5;
    const double w = u < half ? (u - ul) / (ur - ul) : (ur - u) / (ur - ul);
    double s = 0.5 + cos((acos(1 - 2 * w) - 2 * M_PI) / 3);
    for(int i = 0; i < 3; i++)
        s -= (s * s * (3 - 2 * s) - w) / (6 * s * (1 - s));
    return u < half ? s : 1 - s;
}

/// the integrals over one branch of a point that its angles and frequencies need: those of the inverse
/// momentum and (over the full range) of the momentum
struct BranchSums { double e, i3, lz, act; };

/// the branch integrals of a point, in the order of the tasks of angleIntegralKernel
enum { BRANCH_LAMBDA = 0, BRANCH_NU = 1, BRANCH_LAMBDA_PART = 2, BRANCH_NU_PART = 3, NUM_BRANCHES = 4 };

/// what the branch integrals of a point share: dF/dtau at nu_max and the scaled positions of the point
/// within its ranges (the upper ends of the partial integrals)
struct AngleSetup { double dfdnuMax, yl, yn; };

static __device__ AngleSetup fudgeAngleSetup(const MultipoleView& M, const FudgeRecord& rec, bool parts)
{
    FudgeFunction fnc;
    loadFudgeFunction(M, rec, fnc);
    const FudgeLimits lim = fudgeLimitsFinish(rec);
    AngleSetup a{ 0, 0, 0 };
    double unused;
    fnc.eval<true, false>(lim.nu_max, &unused, &a.dfdnuMax, nullptr);
    if(parts) {
        a.yl = scaleCubInverse(lim.lambda_min, lim.lambda_max, rec.lambda);
        a.yn = lim.nu_max == 0 ? 0 : scaleCubInverse(0, lim.nu_max, fabs(rec.nu));
    }
    return a;
}

/// one node (abscissa x, weight w) of a branch integral over the scaled interval [0, y] of [lo, hi]
/// (integrateGL(ScaledIntegrand<ScalingCub>, 0, y, N), src/math_core.cpp:1191-1205) added to its sums: the three
/// integrands of AxisymIntegrand::value with p in the denominator (n = -1), from one F(tau):
/// (tau-Delta^2)^-1 [E], (tau-Delta^2)^-1 tau^-1 [I3], (tau-Delta^2)^-2 with the singular part at nu_max
/// removed [Lz] (src/actions_staeckel.cpp:276-299), and p itself.  The quotients are rounded from shared
/// reciprocals; where one of them has no finite value its term is left out in either case.
/// CELLS: the potential has cells (2-D splines).
template<bool CELLS>
static __device__ __forceinline__ void addBranchNode(const FudgeFunction& fnc, double D2inv, double x, double w,
    double lo, double hi, double y, double nuMax, double dfdnuMax, BranchSums& sum)
{
    const double s = y * x;
    const double duds = (hi - lo) * 6 * s * (1 - s);
    const double tau = sumProducts(hi * pow2(s), 3 - 2 * s, lo * pow2(1 - s), 1 + 2 * s);
    const double ft = CELLS ? branchValue(fnc, D2inv, tau) : fnc.value(tau);
    const double tmd = tau - fnc.D2, tmd2 = pow2(tmd), den = 2 * tmd2 * tau;
    const double p2 = quotient(ft, den, reciprocal(den));
    if(p2 < 0) return;
    const double root = squareRoot(p2), r = reciprocal(root), tmdInv = reciprocal(tmd);
    double v = quotient(r, tmd, tmdInv);
    if(isFinite(v)) sum.e = fma(w, v * duds, sum.e);
    v = quotient(v, tau, reciprocal(tau));
    if(isFinite(v)) sum.i3 = fma(w, v * duds, sum.i3);
    v = quotient(r, tmd2, reciprocal(tmd2));
    if(tmd < 0) v += sqrt(2 * nuMax / dfdnuMax / (tau - nuMax)) / tmd;
    if(isFinite(v)) sum.lz = fma(w, v * duds, sum.lz);
    if(isFinite(root)) sum.act = fma(w, root * duds, sum.act);
}

/// 2 pi wrap of an angle into [0, 2 pi) (math::wrapAngle, src/math_core.cpp:149-157; NaN -> 0)
static __device__ __forceinline__ double wrapAngle(double x)
{
    x -= 2 * M_PI * floor(1 / (2 * M_PI) * x);
    return x >= 0 && x < 2 * M_PI ? x : 0;
}

/** Actions, frequencies and angles of a prepared point whose roots are found (evalAxisym,
    src/actions_staeckel.cpp:645-670): computeActions (:604-619), computeActionDerivatives
    (:489-527), computeIntDerivatives (:532-560), computeGenFuncDerivatives (:566-600) and
    computeAngles (:624-636), from the sums of its branch integrals (scaled by the upper ends of their
    intervals).  ang / freq may be null. */
static __device__ void fudgeAnglesFrequencies(const MultipoleView& M, const FudgeRecord& rec, const AngleSetup& setup,
    const BranchSums* sums, double* act, double* ang, double* freq)
{
    const FudgeLimits lim = fudgeLimitsFinish(rec);
    const double D2 = rec.D2, Lz = rec.Lz, dfdnuMax = setup.dfdnuMax;
    BranchSums L = sums[BRANCH_LAMBDA];
    const BranchSums N = sums[BRANCH_NU];
    act[0] = L.act / M_PI;
    act[1] = N.act / M_PI * 2;
    if(lim.lambda_min == lim.lambda_max) {      // limitingIntegralValue, :307-323
        const double tau = lim.lambda_min, tmd = tau - D2;
        FudgeFunction fnc;
        loadFudgeFunction(M, rec, fnc);
        double d2, v0;
        fnc.eval<false, true>(tau, &v0, nullptr, &d2);
        const double base = 2 * M_PI * sqrt(-tau / d2) * fabs(tmd);
        L.e = base / tmd;
        L.i3 = base / tmd / tau;
        L.lz = base / pow2(tmd);
    }
    const double dJrdE = L.e / (4 * M_PI), dJzdE = N.e / (2 * M_PI);
    const double dJrdI3 = -L.i3 / (4 * M_PI), dJzdI3 = -N.i3 / (2 * M_PI);
    const double dJrdLz = -Lz * L.lz / (4 * M_PI);
    const double dmn = D2 - lim.nu_max;
    const double singpart = 2 * sqrt(-2 * lim.nu_max / dfdnuMax / dmn) * atan(sqrt(lim.nu_max / dmn));
    const double dJzdLz = -Lz * (N.lz + singpart) / (2 * M_PI);
    // inverse matrix: frequencies and the derivatives of I3 over the actions
    double Or, Oz, Ophi, dI3dJr, dI3dJz, dI3dJphi;
    const double det = sumProducts(dJrdE, dJzdI3, -dJrdI3, dJzdE);
    if(lim.nu_max == 0 || det == 0) {
        Or = 1 / dJrdE;
        Ophi = -dJrdLz / dJrdE;
        dI3dJr = dI3dJz = dI3dJphi = Oz = 0;
    } else {
        Or = dJzdI3 / det;
        Oz = -dJrdI3 / det;
        Ophi = sumProducts(dJrdI3, dJzdLz, -dJrdLz, dJzdI3) / det;
        dI3dJr = -dJzdE / det;
        dI3dJz = dJrdE / det;
        dI3dJphi = -sumProducts(dJrdE, dJzdLz, -dJrdLz, dJzdE) / det;
    }
    if(freq) { freq[0] = Or; freq[1] = Oz; freq[2] = Ophi; }
    if(!ang) return;
    // derivatives of the generating function over (E, I3, Lz): integrals up to the point
    const double signl = rec.valid & REC_LDOT_POS ? 1 : -1, signn = rec.valid & REC_NDOT_NU_POS ? 1 : -1;
    const double absnu = fabs(rec.nu);
    const BranchSums Lp = sums[BRANCH_LAMBDA_PART], Np = sums[BRANCH_NU_PART];
    const double dSdE = signl * Lp.e / 4 + signn * Np.e / 4;
    const double dSdI3 = signl * -Lp.i3 / 4 + signn * -Np.i3 / 4;
    const double singS = 2 * sqrt(-2 * lim.nu_max / dfdnuMax / dmn) *
        (atan(sqrt(lim.nu_max / dmn)) - atan(sqrt((lim.nu_max - absnu) / dmn)));
    const double dSdLz = Lz == 0 ? 0 : rec.phi + signl * -Lz * Lp.lz / 4 + signn * -Lz * (Np.lz + singS) / 4;
    const bool addPi = (rec.valid & REC_NUDOT_NEG) && Lz != 0;
    ang[0] = wrapAngle(sumProducts(dSdE, Or, dSdI3, dI3dJr) + dSdLz * 0);
    ang[1] = wrapAngle(sumProducts(dSdE, Oz, dSdI3, dI3dJz) + dSdLz * 0 + M_PI * addPi);
    ang[2] = wrapAngle(sumProducts(dSdE, Ophi, dSdI3, dI3dJphi) + dSdLz * 1);
}

}  // namespace agb
