// Axisymmetric Staeckel-fudge actions on the device (one phase-space point per thread).
//
// Reference: src/actions_staeckel.cpp -- findIntegralsOfMotionAxisymFudge (:176-195),
// AxisymFunctionFudge::evalDeriv (:202-252), AxisymIntegrand (:276-299),
// AxisymScaledForRootfinder (:329-354), findIntegrationLimitsAxisym (:360-483),
// computeActions (:604-619), evalAxisym (:645-670), evalAxisymFudge (:683-693) and
// ActionFinderAxisymFudge::eval (:954-979); prolate spheroidal coordinates from src/coord.cpp
// (:266-338, :525-531); L_circ(E) from potential::Interpolator (src/potential_utils.cpp:872-980).
#pragma once
#include "multipole_cells.cuh"
#include "fudge_types.h"

namespace agb {

constexpr int FUDGE_INTEGR_ORDER = 10;           // src/actions_staeckel.cpp:21
constexpr double FUDGE_ACCURACY_RANGE = 1e-6;    // src/actions_staeckel.cpp:35
constexpr double FUDGE_MINIMUM_RANGE = 1e-10;    // src/actions_staeckel.cpp:38

/// QuinticSpline::evalDeriv (src/math_spline.cpp:1405-1429): linear extrapolation outside
__device__ __forceinline__ void spline1d(const Spline1dView& S, double x, double* f, double* df, double* d2f)
{
    const int n = S.n;
    const double* xv = S.t;
    const double* fv = S.t + n;
    const double* f1 = S.t + 2 * n;
    const double* f2 = S.t + 3 * n;
    if(n == 0 || x != x) { *f = NAN; if(df) *df = NAN; if(d2f) *d2f = NAN; return; }
    const int i = binSearch(x, xv, n);
    if(i < 0 || i >= n - 1) {
        const int e = i < 0 ? 0 : n - 1;
        const double d = ldg(f1 + e);
        *f = ldg(fv + e) + (d == 0 ? 0 : d * (x - ldg(xv + e)));
        if(df) *df = d;
        if(d2f) *d2f = 0;
        return;
    }
    const double fl[1] = { ldg(fv + i) }, fh[1] = { ldg(fv + i + 1) }, d1l[1] = { ldg(f1 + i) },
        d1h[1] = { ldg(f1 + i + 1) }, d2l[1] = { ldg(f2 + i) }, d2h[1] = { ldg(f2 + i + 1) };
    quinticSegment<1>(x, ldg(xv + i), ldg(xv + i + 1), fl, fh, d1l, d1h, d2l, d2h, f, df, d2f);
}

/// potential::Interpolator::evalDeriv (src/potential_utils.cpp:872-911): Phi(R), dPhi/dR, d2Phi/dR2
static __device__ __forceinline__ void interpPhi(const FudgeTables& F, double R, double* val, double* der, double* der2)
{
    const double logR = log(R);
    if(logR > ldg(F.PhiofR.t + F.PhiofR.n - 1) && F.coefOut != 0) {
        const double Rs = exp(logR * F.slopeOut);
        const double Phi = (-F.massOut + (F.slopeOut == -1 ? logR : (R * Rs - 1) / (F.slopeOut + 1)) * F.coefOut) / R;
        *val = Phi;
        *der = (-Phi + F.coefOut * Rs) / R;
        *der2 = (2 * Phi + F.coefOut * Rs * (F.slopeOut - 2)) / pow2(R);
        return;
    }
    double s, d1, d2;
    spline1d(F.PhiofR, logR, &s, &d1, &d2);
    const double ex = exp(s), E = 1 / (F.iInvPhi0 - ex), dE = E * E * ex, d2E = E * dE * (F.iInvPhi0 + ex);
    *val = E;
    *der = dE * d1 / R;
    *der2 = (dE * (d2 - d1) + d2E * d1 * d1) / pow2(R);
}

/// potential::Interpolator::L_circ (src/potential_utils.cpp:954-980)
static __device__ __forceinline__ double interpLcirc(const FudgeTables& F, double E)
{
    if(!(E >= 1. / F.iInvPhi0 && E <= 0))
        return NAN;
    const double scaledE = log(F.iInvPhi0 - 1 / E);
    double logL;
    spline1d(F.LofE, scaledE, &logL, nullptr, nullptr);
    double Lcirc = exp(logL);
    if(scaledE > ldg(F.LofE.t + F.LofE.n - 1)) {   // large-radius correction
        double logR;
        spline1d(F.RofL, logL, &logR, nullptr, nullptr);
        const double Rc = exp(logR);
        double Phi, dPhi, d2Phi;
        interpPhi(F, Rc, &Phi, &dPhi, &d2Phi);
        const double Ec = Phi + 0.5 * Rc * dPhi;
        const double denom = 1 - 0.5 * (Ec - E) * (Rc * d2Phi - dPhi) / ((Rc * d2Phi + 3 * dPhi) * Rc * dPhi);
        Lcirc = clip(sqrt(Rc * dPhi) * (Rc - (Ec - E) / (dPhi * denom)), 0.75 * Lcirc, 1.25 * Lcirc);
    }
    return Lcirc;
}

/// bilinear Delta(xi, chi) (LinearInterpolator2d::evalDeriv, src/math_spline.cpp:2152-2190)
static __device__ __forceinline__ double deltaLookup(const FudgeTables& F, double x, double y)
{
    const int nx = F.nE, ny = F.nL;
    const int xi = binSearch(x, F.gridE, nx), yi = binSearch(y, F.gridL, ny);
    if(xi < 0 || xi >= nx - 1 || yi < 0 || yi >= ny - 1)
        return NAN;
    const double* f = F.delta + static_cast<size_t>(xi) * ny + yi;
    const double zll = ldg(f), zlu = ldg(f + 1), zul = ldg(f + ny), zuu = ldg(f + ny + 1);
    const double xl = ldg(F.gridE + xi), yl = ldg(F.gridL + yi);
    const double t = (x - xl) / (ldg(F.gridE + xi + 1) - xl), u = (y - yl) / (ldg(F.gridL + yi + 1) - yl);
    const double T = 1 - t, U = 1 - u;
    return T * (U * zll + u * zlu) + t * (U * zul + u * zuu);
}

/** An axisymmetric asymptotic expansion (evalPowerLaw) at (R, z): the potential, and with DER its derivatives
    over ln r and over the latitude.  One loop over l with the Legendre recurrence, inline. */
template<bool DER>
__device__ __forceinline__ void powerLawAxi(const PowerLawView& A, double rsq, double R, double z, double* Phi, double* px,
    double* ppsi)
{
    const double dlogr = 0.5 * log(rsq / A.r0sq);
    const int lmax = (A.inner && rsq < A.r0sq * 1e-16) || (!A.inner && rsq > A.r0sq * 1e16) ? 0 : A.ind.lmax;
    const double rinv = rsq > 0 ? 1 / sqrt(rsq) : 0, ct = z * rinv, st = R * rinv;
    double sum = 0, sumr = 0, sumt = 0, P = 1, Pm1 = 0, dP = 0, dPm1 = 0;  // Legendre P_l and dP_l / d(ct)
    for(int l = 0; l <= lmax; l++) {
        if(l > 0) {
            const double p = ((2 * l - 1) * ct * P - (l - 1) * Pm1) / l;
            const double d = DER ? dPm1 + (2 * l - 1) * P : 0;
            Pm1 = P; P = p;
            dPm1 = dP; dP = d;
        }
        if(l % A.ind.step) continue;
        const int c = HarmIndices::index(l, 0);
        const double s = ldg(A.S + c), u = ldg(A.U + c), w = ldg(A.W + c), v = A.inner ? l : -l - 1;
        const double rv = v != 0 ? exp(dlogr * v) : 1;
        const double rs = s != v ? (s != 0 && u != 0 ? exp(dlogr * s) : 1) : rv;
        const double urs = u * rs * (s != v || u == 0 ? 1 : dlogr), wrv = w * rv;
        const double qr2 = v == 0 ? A.Q * rsq / A.r0sq : 0, norm = lmax == 0 ? 1 : sqrt(2 * l + 1.);
        sum += (urs + wrv + qr2) * (norm * P);
        if(DER) {
            sumr += (urs * s + wrv * v + (s != v ? 0 : u * rs) + 2 * qr2) * (norm * P);
            sumt += (urs + wrv + qr2) * (norm * dP);
        }
    }
    *Phi = sum;
    if(DER) { *px = sumr; *ppsi = sumt * st; }      // d(ct) / dpsi = cos(psi) = sin(theta)
}

/** The fudge's auxiliary function F(tau) along one of the two coordinates of a point (the other one
    stays at its value there); AxisymFunctionFudge::evalDeriv, src/actions_staeckel.cpp:202-252, with
    prolate spheroidal -> cylindrical coordinates from src/coord.cpp:266-291.

    What does not depend on tau is formed once: with (lambda, nu) the point and D2 = Delta^2,

        lambda branch (tau = lambda > D2):  R = c1 sqrt(tau - D2),  z = c2 sqrt(tau),
                                            r^2 = (tau - D2) + nu
        nu branch     (tau = nu < D2):      R = c1 sqrt(D2 - tau),  z = c2 sqrt(tau),
                                            r^2 = tau + (lambda - D2)

    and the derivative along the branch needs no gradient in (R, z): with x = ln r and the latitude
    psi (tau_spline = tan(psi / 2)), dx/dtau = 1 / (2 r^2) and dpsi/dtau = K / (2 r^2 sqrt(|tau - D2| tau)),
    K = -sqrt(nu (D2 - nu)) or +sqrt(lambda (lambda - D2)), i.e. -+ D2 c1 c2, with the reciprocal
    roots that R and z are formed from.  One evaluation takes three reciprocal square roots, one
    reciprocal and a logarithm beside the cell, and with log scaling a second reciprocal and an
    exponential (before: three square roots and five to seven divisions, and the gradient's
    transformation). */
struct FudgeBranch {
    double E, I, L2h, D2;       // I: I3 - fnu (lambda branch) or I3 - flambda; L2h = Lz^2 / 2
    double mo, ro, c1, c2;      // tau - mo multiplies Phi; r^2 = (tau - D2 or tau) + ro
    bool lam;

    /// the branch's constants from the point's record (nu enters by its absolute value)
    __device__ void set(bool lambdaBranch, double lambda, double nu, double D2_, double E_, double Lz, double I3,
        double flambda, double fnu)
    {
        lam = lambdaBranch;
        E = E_; D2 = D2_; L2h = Lz * Lz / 2;
        I = lam ? I3 - fnu : I3 - flambda;
        const double n = fabs(nu), lmd = lambda - D2, inv = rcpNormal(D2);
        mo = lam ? n : lambda;
        ro = lam ? n : lmd;
        // D2 - n is exact near the axis and 0 on it (|z| > Delta), where 1 - n * inv is the rounding of the
        // reciprocal, of either sign
        c1 = NormalArithmetic::root((lam ? fmax(D2 - n, 0.) : lmd) * inv);
        c2 = NormalArithmetic::root((lam ? n : lambda) * inv);
    }

    /// F(tau), and with DER its derivative.  CELLS: the potential has cells (2-D splines), and beyond them
    /// the asymptotic expansions are evaluated inline: with a call there the registers saved around it cost the
    /// searches and integrals their hot path (370 B of spills)
    template<bool DER, bool CELLS>
    __device__ __forceinline__ void eval(const MultipoleView& M, double tau, double* val, double* der) const
    {
        const double tmd = tau - D2;
        const double u = fmax(lam ? tmd : -tmd, 0.), rsq = (lam ? tmd : tau) + ro;
        // zeros are kept out of the reciprocal roots: u -> 0 and tau -> 0 give R = 0 and z = 0
        const double iu = rsqrtNormal(fmax(u, 1e-280)), it = rsqrtNormal(fmax(tau, 1e-280));
        const double R = c1 * (u * iu), z = c2 * (tau * it);
        double Phi, px = 0, ppsi = 0, r2inv;        // Phi, dPhi/dln r, dPhi/dpsi
        if(inCells(M, rsq)) {
            const double rinv = rsqrtNormal(rsq), logr = 0.5 * log(rsq);
            const double y = fmin(z * rcpNormal(fma(rsq, rinv, R)), 1.);
            r2inv = rinv * rinv;
            double xl, xh, xi, yl, yh, yi;
            const int ix = gridCell(M.gridR, logr, &xl, &xh, &xi), iy = gridCell(M.gridTau, y, &yl, &yh, &yi);
            double P, dummy;
            cellPolynomial<DER ? 3 : 1>(M.cells + (static_cast<size_t>(ix) * (M.nt - 1) + iy) * CELL_COEFS,
                (logr - xl) * xi, (y - cellAnchor(yl, yh)) * yi, &P, &px, &ppsi, &dummy, &dummy, &dummy);
            if(DER) { px *= xi; ppsi *= yi * fma(0.5 * y, y, 0.5); }
            Phi = P;
            if(M.logScaling) {
                const double ex = exp(P);
                Phi = rcpNormal(M.invPhi0 - ex);
                if(DER) { const double d = Phi * Phi * ex; px *= d; ppsi *= d; }
            }
        } else if(CELLS) {
            r2inv = 1 / rsq;
            powerLawAxi<DER>(rsq < M.rInnerSq ? M.inner : M.outer, rsq, R, z, &Phi, &px, &ppsi);
        } else {
            BeyondCells b;
            evalBeyondCells<DER ? 3 : 1>(M, R, z, 0, &b);
            Phi = b.pot;
            r2inv = 1 / rsq;
            if(DER) { px = R * b.g.dR + z * b.g.dz; ppsi = R * b.g.dz - z * b.g.dR; }
        }
        const double mult = tau - mo;
        *val = (E * tau - I - Phi * mult) * tmd - L2h * tau;
        if(DER) {
            const double K = D2 * (c1 * c2);
            const double dPhi = 0.5 * r2inv * (px + (lam ? -K : K) * (ppsi * iu * it));
            *der = E * (tau + tmd) - L2h - I - (mult + tmd) * Phi - (tmd != 0 ? tmd * mult * dPhi : 0);
        }
    }
    template<bool CELLS>
    __device__ __forceinline__ double value(const MultipoleView& M, double tau) const
    {
        double v;
        eval<false, CELLS>(M, tau, &v, nullptr);
        return v;
    }
};

/// F, F' and F'' on the lambda branch from the potential, its gradient and Hessian at (R, z >= 0)
__device__ __forceinline__ void fudgeSecond(double E, double I, double L2h, double D2, double mo, double tau, double R,
    double z, double Phi, const CylDerivs& g, const CylHess& h, double* val, double* der, double* der2)
{
    const double tmd = tau - D2, mult = tau - mo;
    const double dRdt = 0.5 * R / tmd, dzdt = 0.5 * z / tau;
    const double dPhi = g.dR * dRdt + g.dz * dzdt;
    const double d2 = h.dR2 * pow2(dRdt) + h.dz2 * pow2(dzdt) + 2 * h.dRdz * dRdt * dzdt -
        0.25 * (g.dR * R / pow2(tmd) + g.dz * z / pow2(tau));
    *val = (tmd != 0 ? (E * tau - I - Phi * mult) * tmd : 0) - L2h * tau;
    *der = E * (tau + tmd) - L2h - I - (mult + tmd) * Phi - (tmd != 0 ? tmd * mult * dPhi : 0);
    *der2 = 2 * (E - Phi - (mult + tmd) * dPhi) - tmd * mult * d2;
}

/// the same at any tau of the lambda branch, evaluating the potential there (rare: out of line)
static __device__ __noinline__ void fudgeSecondAt(const MultipoleView& M, const FudgeBranch& f, double tau,
    double* val, double* der, double* der2)
{
    const double R = f.c1 * sqrt(fmax(tau - f.D2, 0.)), z = f.c2 * sqrt(tau);
    double Phi;
    CylDerivs g; CylHess h;
    evalCellsCyl<6, EVAL_AXI>(M, R, z, 0, &Phi, &g, &h);
    fudgeSecond(f.E, f.I, f.L2h, f.D2, f.mo, tau, R, z, Phi, g, h, val, der, der2);
}

/// F(tau) out of line, for the rare single values of phase 1 and the angles
static __device__ __noinline__ double fudgeValueAt(const MultipoleView& M, const FudgeBranch& f, double tau)
{
    return f.value<false>(M, tau);
}

/// State of one point between the phases of the action computation: the point in prolate
/// spheroidal coordinates, its integrals of motion, the integration limits known so far and the
/// brackets of the roots still to be found.  One 128-byte record per point.
struct __align__(16) FudgeRecord {
    double lambda, nu, D2, E, Lz, I3, flambda, fnu, phi;
    double lambdaMin, lambdaMax, nuMax;     // nu_min is always 0
    double nuUpper;                         // nu_max root bracket: [|nu|, nuUpper]
    double lambdaLower, lambdaPos;          // lambda_min root in [lambdaLower, lambdaPos];
                                            // lambda_max root in [lambdaPos, inf)
    int roots;                              // ROOT_* bits of the roots still to be found
    int valid;                              // 0: the point has no integrals to do; otherwise
                                            // REC_VALID | the REC_* direction-of-motion bits
};

/// bits of FudgeRecord::valid: the point has integrals to do, and the signs of its motion in
/// prolate spheroidal coordinates that the angles need (lambdadot >= 0, nudot * nu >= 0, nudot < 0)
enum { REC_VALID = 1, REC_LDOT_POS = 2, REC_NDOT_NU_POS = 4, REC_NUDOT_NEG = 8 };
static_assert(sizeof(FudgeRecord) == 128, "FudgeRecord is one 128-byte line");

enum { ROOT_NU_MAX = 1, ROOT_LAMBDA_MIN = 2, ROOT_LAMBDA_MAX = 4 };

/// F and F' at the ends of the plain root brackets that phase 1 evaluates once for the searches of
/// phase 2: lambda_pos (shared by the lambda_min and lambda_max brackets), Delta^2 (the upper end
/// of the nu_max bracket and the lower end of the lambda_min one) and |nu| (the lower end of the
/// nu_max bracket); NaN where not evaluated
struct FudgeEnds { double fPos, dfPos, fD2, dfD2, fNu, dfNu; };

/** The root functions of the three integration limits behind one evaluation site: F(tau) and F'(tau)
    for nu_max and lambda_min; with semiInf (lambda_max) F(tau)/tau^2 on
    [u0, inf) mapped to s in [0, 1] by the semi-infinite scaling, AxisymScaledForRootfinder inside
    ScaledFnc<ScalingSemiInf>, src/actions_staeckel.cpp:329-354, src/math_core.h:214-232). */
template<bool CELLS>
__device__ __forceinline__ void limitRootEval(const MultipoleView& M, const FudgeBranch& f, bool semiInf, double u0,
    double x, double* v, double* d)
{
    double duds = 1, tau = x;
    if(semiInf) {       // unscaleSemiInf with one reciprocal (x = 1 gives NaN: far)
        const double w = rcpNormal(1 - x);
        tau = u0 * exp(x * w);
        duds = tau * w * w;
    }
    const bool far = semiInf && !(tau <= 1e100);
    double fval = 0, fder = 0;
    if(!far) f.eval<true, CELLS>(M, tau, &fval, &fder);
    if(!semiInf) { *v = fval; *d = fder; }
    else if(far) { *v = f.E; *d = NAN; }
    else {
        const double it = rcpNormal(tau), it2 = it * it;
        *v = fval * it2;
        *d = (fder - 2 * fval * it) * it2 * duds;
    }
}

/// the branch of a record along which one of its limits is searched or one of its actions integrated
__device__ __forceinline__ void loadFudgeBranch(const FudgeRecord& r, bool lambdaBranch, FudgeBranch& f)
{
    f.set(lambdaBranch, r.lambda, r.nu, r.D2, r.E, r.Lz, r.I3, r.flambda, r.fnu);
}

/// the potential of the cells in the equatorial plane or on the axis at squared radius rsq (inCells)
__device__ __forceinline__ double cellsOnAxes(const MultipoleView& M, double rsq, int axis)
{
    const double logr = 0.5 * log(rsq);
    double xl, xh, xi, yl, yh, yi, Phi, dummy;
    const int ix = gridCell(M.gridR, logr, &xl, &xh, &xi), iy = gridCell(M.gridTau, axis, &yl, &yh, &yi);
    cellPolynomial<1>(M.cells + (static_cast<size_t>(ix) * (M.nt - 1) + iy) * CELL_COEFS, (logr - xl) * xi,
        (axis - cellAnchor(yl, yh)) * yi, &Phi, &dummy, &dummy, &dummy, &dummy, &dummy);
    return M.logScaling ? rcpNormal(M.invPhi0 - exp(Phi)) : Phi;
}

/// the same at any radius
__device__ __forceinline__ double potentialOnAxes(const MultipoleView& M, double rsq, int axis)
{
    if(inCells(M, rsq)) return cellsOnAxes(M, rsq, axis);
    const double r = sqrt(rsq);
    BeyondCells b;
    evalBeyondCells<1>(M, axis ? 0 : r, axis ? r : 0, 0, &b);
    return b.pot;
}

/** What phase 1 needs of the potential, from the cells: one evaluation with the Hessian at the point
    (R, |z|) gives F of both branches there up to F'', the value at (lambda, nu = 0) gives the
    integrals of motion and F(0), and the value on the axis F' at Delta^2.  (The node form evaluates
    the potential six times.)  The same struct is the evaluator of fudgeLimitsSetup.
    FAST: for points inside the cells, without calls; `rare` is set where something else is needed. */
template<bool FAST>
struct CellPoint {
    bool rare = false;
    double R, z, Phi, Phi0;
    CylDerivs g;
    CylHess h;
    const MultipoleView* view;
    const FudgeRecord* rec;
    __device__ __forceinline__ void locate(const MultipoleView& M, double R_, double z_)
    {
        view = &M;
        R = R_; z = fabs(z_);
        // (axisymmetric: no azimuth)
        if(FAST) evalCells<6, EVAL_AXI>(M, R, z, 1, 0, &Phi, &g, &h);
        else     evalCellsCyl<6, EVAL_AXI>(M, R, z, 0, &Phi, &g, &h);
    }
    __device__ double onAxes(double rsq, int axis)
    {
        if(!FAST) return potentialOnAxes(*view, rsq, axis);
        if(inCells(*view, rsq)) return cellsOnAxes(*view, rsq, axis);
        const double r = sqrt(rsq);
        double v, unused;
        powerLawAxi<false>(rsq < view->rInnerSq ? view->inner : view->outer, rsq, axis ? 0 : r, axis ? r : 0, &v, &unused,
            &unused);
        return v;
    }
    __device__ double equatorial(double rsq) { return Phi0 = onAxes(rsq, 0); }
    __device__ FudgeBranch branch(bool lambdaBranch) const
    {
        FudgeBranch f;
        loadFudgeBranch(*rec, lambdaBranch, f);
        return f;
    }
    // F(0): the potential at (lambda, nu = 0)
    __device__ double zero() const { return ((rec->I3 - rec->flambda) - Phi0 * rec->lambda) * rec->D2; }
    __device__ void second(double* v, double* d, double* d2) const
    {
        fudgeSecond(rec->E, rec->I3 - rec->fnu, rec->Lz * rec->Lz / 2, rec->D2, fabs(rec->nu), rec->lambda, R, z, Phi,
            g, h, v, d, d2);
    }
    __device__ void secondAt(double tau, double* v, double* d, double* d2)
    {
        if(FAST) { rare = true; *v = *d = *d2 = NAN; }
        else fudgeSecondAt(*view, branch(true), tau, v, d, d2);
    }
    __device__ double valueAt(bool lambdaBranch, double tau)
    {
        if(FAST) { rare = true; return NAN; }
        return fudgeValueAt(*view, branch(lambdaBranch), tau);
    }
    __device__ double nuValue(double tau) { return valueAt(false, tau); }
    __device__ double lambdaValue(double tau) { return valueAt(true, tau); }
    // at Delta^2, on the axis (R = 0, z = sqrt(nu)): F needs no potential, F' its value alone
    __device__ void endD2(double* v, double* d)
    {
        const double n = fabs(rec->nu), D2 = rec->D2, L2h = rec->Lz * rec->Lz / 2;
        *v = -L2h * D2;
        *d = rec->E * D2 - L2h - (rec->I3 - rec->fnu) - (D2 - n) * onAxes(n, 1);
    }
    // at |nu|, on the nu branch: the point itself
    __device__ void endNu(double* v, double* d) const
    {
        const double n = fabs(rec->nu), tmd = n - rec->D2, mult = n - rec->lambda, L2h = rec->Lz * rec->Lz / 2;
        const double I = rec->I3 - rec->flambda, dPhi = 0.5 * (g.dR * R / tmd + g.dz * z / n);
        *v = (tmd != 0 ? (rec->E * n - I - Phi * mult) * tmd : 0) - L2h * n;
        *d = rec->E * (n + tmd) - L2h - I - (mult + tmd) * Phi - (tmd != 0 ? tmd * mult * dPhi : 0);
    }
};

/** Integration limits of the lambda and nu motions (findIntegrationLimitsAxisym,
    src/actions_staeckel.cpp:360-483), part 1: every decision up to the three root searches, whose
    brackets go into the record; limits that need no root are stored directly (NaN otherwise).
    ends receives F and F' at the ends of the plain brackets (FudgeEnds), which the
    root searches then take instead of evaluating them. */
template<bool FAST>
static __device__ __forceinline__ void fudgeLimitsSetup(CellPoint<FAST>& fnc, FudgeRecord& rec, FudgeEnds* ends)
{
    const double delta = rec.D2, lambda = rec.lambda;
    const double f_zero = fnc.zero();
    double f_lambda, df_lambda, d2f_lambda;
    fnc.second(&f_lambda, &df_lambda, &d2f_lambda);
    double nu_max = NAN, lambda_min = NAN, lambda_max = NAN;
    double nu_upper = delta, lambda_lower = delta;
    int roots = 0;
    if(rec.Lz == 0) {
        const double dminus = delta * (1 - 1e-15), dplus = delta * (1 + 1e-15);
        if(fnc.nuValue(dminus) < 0) {
            if(f_zero > 0) nu_upper = dminus;
            else nu_max = 0;
        } else
            nu_max = delta;
        if(fnc.lambdaValue(dplus) < 0) lambda_lower = dplus;
        else lambda_min = delta;
    }
    if(!isFinite(nu_max)) {
        if(f_zero > 0) roots |= ROOT_NU_MAX;           // falls back to |nu| if no root is found
        else nu_max = fabs(rec.nu);
    }
    double lambda_pos = lambda, f_pos = f_lambda, df_pos = df_lambda;
    const double dxToRoot = -f_lambda / df_lambda;
    if(f_lambda <= 0 || fabs(dxToRoot) < lambda * FUDGE_MINIMUM_RANGE) {
        if(df_lambda >= 0) lambda_min = lambda;
        if(df_lambda <= 0) {
            lambda_max = lambda;
            if(lambda == delta) lambda_min = delta;
        }
        bool nearShell = d2f_lambda < 0 &&
            pow2(df_lambda) - 2 * f_lambda * d2f_lambda - pow2(lambda * FUDGE_MINIMUM_RANGE * d2f_lambda) < 0;
        const double safeOffset = fmin(0.5 * fabs(df_lambda / d2f_lambda), lambda * FUDGE_MINIMUM_RANGE);
        lambda_pos += fmax(dxToRoot, safeOffset) * (df_lambda >= 0 ? 1 : -1);
        double f_lp, df_lp, d2f_lp;
        fnc.secondAt(lambda_pos, &f_lp, &df_lp, &d2f_lp);
        f_pos = f_lp; df_pos = df_lp;
        nearShell |= d2f_lp < 0 &&
            pow2(df_lp) - 2 * f_lp * d2f_lp - pow2(lambda * FUDGE_MINIMUM_RANGE * d2f_lp) < 0;
        if(nearShell || f_lp < 0)
            lambda_min = lambda_max = lambda;
    }
    if(!isFinite(lambda_min)) roots |= ROOT_LAMBDA_MIN;
    if(!isFinite(lambda_max)) roots |= ROOT_LAMBDA_MAX;
    rec.nuMax = nu_max; rec.lambdaMin = lambda_min; rec.lambdaMax = lambda_max;
    rec.nuUpper = nu_upper; rec.lambdaLower = lambda_lower; rec.lambdaPos = lambda_pos;
    rec.roots = roots;
    ends->fPos = f_pos; ends->dfPos = df_pos;
    ends->fD2 = ends->dfD2 = ends->fNu = ends->dfNu = NAN;
    if(((roots & ROOT_NU_MAX) && nu_upper == delta) || ((roots & ROOT_LAMBDA_MIN) && lambda_lower == delta))
        fnc.endD2(&ends->fD2, &ends->dfD2);
    if(roots & ROOT_NU_MAX)
        fnc.endNu(&ends->fNu, &ends->dfNu);
}

struct FudgeLimits { double lambda_min, lambda_max, nu_max; int order; };

/** Part 3 (part 2 is the root searches: RootSearch driven by limitRootEval): the final checks of
    the limits and the Gauss-Legendre order of both integrals. */
static __device__ FudgeLimits fudgeLimitsFinish(const FudgeRecord& rec)
{
    const double delta = rec.D2;
    FudgeLimits lim{ rec.lambdaMin, rec.lambdaMax, rec.nuMax, 0 };
    if(!(lim.nu_max >= delta * FUDGE_MINIMUM_RANGE))
        lim.nu_max = 0;
    if(!(lim.lambda_max - lim.lambda_min >= delta * FUDGE_MINIMUM_RANGE))
        lim.lambda_min = lim.lambda_max = rec.lambda;
    const double ratio = sqrt((lim.lambda_min - delta) / (lim.lambda_max - delta));
    if(ratio == 0) lim.order = GL_MAX_ORDER;
    else {
        int e;
        frexp(ratio, &e);
        lim.order = min(GL_MAX_ORDER, FUDGE_INTEGR_ORDER - e);
    }
    return lim;
}

/** One node of the momentum integral of sqrt(p^2(tau)) over [lo, hi] with the cubic end-point
    stretch (integrateGL of ScaledIntegrand<ScalingCub>(AxisymIntegrand), src/math_core.cpp:1191-1205,
    src/actions_staeckel.cpp:276-299) at tau = lo + (hi - lo) s^2 (3 - 2 s): the integrand alone (the
    node's weight and du/ds / (hi - lo) come tabulated). */
template<bool CELLS>
__device__ __forceinline__ double fudgeMomentum(const MultipoleView& M, const FudgeBranch& f, double tau)
{
    const double tmd = tau - f.D2;
    const double p2 = f.value<CELLS>(M, tau) * rcpNormal(2 * pow2(tmd) * tau);
    // p^2 < 0, NaN or infinite (a node on an end of the interval): no contribution
    return p2 > 1e-280 && p2 < INFINITY ? p2 * rsqrtNormal(p2) : 0;
}

/** The same node with the integrand's arithmetic in FP32 (the mixed-precision form of the action
    quadrature): F(tau) and the point tau come from FP64 (the potential and the cancellation in
    F stay FP64), then p = sqrt(F / (2 tau)) / |tau - D2| is FP32 (the square root through the hardware
    reciprocal square root); the caller accumulates the weighted terms with compensation. */
template<bool CELLS>
__device__ __forceinline__ float fudgeMomentum32(const MultipoleView& M, const FudgeBranch& f, double tau)
{
    const double F = f.value<CELLS>(M, tau), tmd64 = tau - f.D2;
    // p = sqrt(F / (2 tau)) / |tau - D2|: the square root before the division by (tau - D2)^2
    // keeps every FP32 intermediate in range for tau up to ~1e18 (the product (tau - D2)^2 tau
    // overflows FP32 already at tau ~ 1e12, where loosely bound orbits reach); a value of F
    // beyond the FP32 range takes the FP64 form
    if(!(fabs(F) < 1e37)) {
        const double p2 = F / (2 * pow2(tmd64) * tau), v = p2 < 0 ? 0 : sqrt(p2);
        return isFinite(v) ? static_cast<float>(v) : 0.f;
    }
    const float tmd = static_cast<float>(tmd64), t = static_cast<float>(tau);
    const float q = static_cast<float>(F) / (2.f * t);
    const float v = q > 0.f ? q * rsqrtf(q) / fabsf(tmd) : 0.f;
    return v < INFINITY ? v : 0.f;
}

/** Phase 1 of the actions of one point (R, z, phi, vR, vz, vphi) for focal distance fd
    (evalAxisymFudge, src/actions_staeckel.cpp:683-693: fd <= 0 falls back to max(R,1)*1e-4);
    p has been located at the point.  Writes Jphi into act[2]; for a point without actions
    (unbound, or lambda = nu = Delta^2) also NaN into act[0..1] and marks the record invalid.
    Otherwise the record holds the integrals of motion (findIntegralsOfMotionAxisymFudge,
    :176-195) and the limits and root brackets of fudgeLimitsSetup (ends: as there). */
template<bool FAST>
static __device__ __forceinline__ void fudgePrepare(const double* pc, CellPoint<FAST>& p, double fd,
    FudgeRecord& rec, double* act, FudgeEnds* ends)
{
    const double Phi = p.Phi;
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
    const double Phi0 = p.equatorial(lambda - D2);
    const double Ekin = 0.5 * (vR * vR + vz * vz + vphi * vphi);
    rec.lambda = lambda; rec.nu = absnu * signz; rec.D2 = D2; rec.E = Phi + Ekin; rec.Lz = Lz; rec.phi = phi;
    rec.flambda = -lambda * Phi0;
    rec.fnu = rec.flambda + Phi * (lambda - absnu);
    rec.I3 = lambda * (Phi - Phi0) + 0.5 * (pow2(z * vphi) + pow2(R * vz - z * vR) + pow2(vz) * D2);
    if(!isFinite(rec.E + rec.I3 + rec.Lz) || rec.E >= 0) { act[0] = act[1] = NAN; return; }
    p.rec = &rec;
    fudgeLimitsSetup(p, rec, ends);
    // velocities in prolate spheroidal coordinates (src/coord.cpp:317-322, :525-531)
    const double lambdadot = R * 2 * lambda / sqD * vR + z * 2 * lmd / sqD * vz;
    const double nudot = R * 2 * -absnu / sqD * signz * vR + z * 2 * dmn / sqD * signz * vz;
    rec.valid = REC_VALID | (lambdadot >= 0 ? REC_LDOT_POS : 0) | (nudot * rec.nu >= 0 ? REC_NDOT_NU_POS : 0) |
        (nudot < 0 ? REC_NUDOT_NEG : 0);
}

/// Cartesian posvel -> cylindrical (R, z, phi, vR, vz, vphi); reference src/coord.cpp:476-484; without
/// AZIMUTH phi is left 0 (only the angles need it)
template<bool AZIMUTH>
__device__ __forceinline__ void carToCylPosVel(const double* w, double* pc)
{
    const double R = sqrt(w[0] * w[0] + w[1] * w[1]);
    if(R == 0) {
        pc[0] = 0; pc[1] = w[2]; pc[2] = AZIMUTH ? atan2(w[4], w[3]) : 0;
        pc[3] = sqrt(w[3] * w[3] + w[4] * w[4]); pc[4] = w[5]; pc[5] = 0;
        return;
    }
    const double c = w[0] / R, s = w[1] / R;
    pc[0] = R; pc[1] = w[2]; pc[2] = AZIMUTH ? atan2(w[1], w[0]) : 0;
    pc[3] = w[3] * c + w[4] * s;
    pc[4] = w[5];
    pc[5] = -w[3] * s + w[4] * c;
}

/** focal distance of the action finder at a point with potential Phi: E, Lz -> Lcirc(E) ->
    (xi, chi) -> Delta; reference ActionFinderAxisymFudge::eval steps 0-1,
    src/actions_staeckel.cpp:957-977 */
static __device__ __forceinline__ double finderFocalDistance(const FudgeTables& F, const double* pc, double Phi)
{
    const double E = Phi + 0.5 * (pc[3] * pc[3] + pc[4] * pc[4] + pc[5] * pc[5]);
    const double Lz = pc[0] * pc[5];
    const double Lcirc = interpLcirc(F, E);
    const double xi = clip(log(F.invPhi0 - 1 / E), ldg(F.gridE), ldg(F.gridE + F.nE - 1));
    const double Lzrel = clip(fabs(Lz) / Lcirc, 0., 1.);
    const double chi = scaleCub(0, 1, Lzrel);
    return fmax(0., deltaLookup(F, xi, chi));
}

/// inputs of the bracket predictor: the point's (R, z, vR, vz, vphi) with E and Lz in
/// scale-free form -- ln r, |z| / r, velocities over the escape speed sqrt(-2 Phi) (so
/// that E = Phi (1 - v^2 / v_esc^2) and Lz = R vphi follow), ln(Delta / r); symmetric
/// under z -> -z and Lz -> -Lz like the limits themselves
__device__ __forceinline__ void bracketFeatures(const double* pc, double Phi, double delta, float* out)
{
    const double r = fmax(sqrt(pc[0] * pc[0] + pc[1] * pc[1]), 1e-300), vesc = sqrt(fmax(-2 * Phi, 1e-300));
    const float f[6] = { static_cast<float>(log(r)), static_cast<float>(fabs(pc[1]) / r),
        static_cast<float>(pc[3] / vesc), static_cast<float>((pc[1] >= 0 ? pc[4] : -pc[4]) / vesc),
        static_cast<float>(fabs(pc[5]) / vesc), static_cast<float>(log(fmax(delta, 1e-300) / r)) };
    for(int k = 0; k < 6; k++) out[k] = f[k];
}

}  // namespace agb
