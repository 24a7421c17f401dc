// The force of a Multipole potential for the orbit integration, from the node form of its splines.
//
// An orbit's end point is not determined by 64-bit arithmetic beyond some periods (a change of 1e-16 in
// the start of an isotropic sample of orbits moves their end points by 1e-9 to 1e-5 of their norm
// within ten), so this path keeps the arithmetic of the evaluation to the bit: the same operations
// as evalMultipoleCar, arranged for a short instruction stream, with the contractions of a sum of two
// products (which of them is rounded) written out where the compiler could choose.  One evaluation
// at a time per lane decides how long an orbit takes, and its cost is the number of instructions
// it issues.
#pragma once
#include "multipole_cells.cuh"

namespace agb {

/// a b + c d with c d rounded
__device__ __forceinline__ double sumProducts(double a, double b, double c, double d) { return fma(a, b, __dmul_rn(c, d)); }

/// a / b correctly rounded from y = 1 / b correctly rounded (Markstein 1990: a quotient estimate within
/// one unit in the last place, its exact remainder by a fused multiply-add, and y give the rounded
/// quotient; the first step brings a y to such an estimate).  For a and b well inside the range of
/// normal numbers, a = 0 included.
__device__ __forceinline__ double quotient(double a, double b, double y)
{
    const double q0 = a * y, q1 = fma(fma(-b, q0, a), y, q0);
    return fma(fma(-b, q1, a), y, q1);
}

/// 1 / b correctly rounded, for b well inside the range of normal numbers (the same step); the one exception
/// is a b whose fraction is of ones alone, left a unit low where the approximation is (Markstein's; its
/// quotients are right all the same)
__device__ __forceinline__ double reciprocal(double b)
{
    const double y = rcpNormal(b);
    return fma(fma(-b, y, 1.0), y, y);
}

/// sqrt(a) correctly rounded, for a > 0 well inside the range of normal numbers: the root estimate a y
/// corrected by its exact remainder (Markstein)
__device__ __forceinline__ double squareRoot(double a)
{
    const double y = rsqrtNormal(a), g = a * y;
    return fma(fma(-g, g, a), 0.5 * y, g);
}

/// the divisions and roots of the root searches, correctly rounded without the library's slow paths (for operands
/// outside the range of normal numbers a quotient is NaN where the library gives 0, NaN or an infinity: the
/// searches refuse such steps alike)
struct RoundedArithmetic {
    static __device__ __forceinline__ double quotient(double a, double b) { return agb::quotient(a, b, reciprocal(b)); }
    static __device__ __forceinline__ double root(double a) { return a > 1e-280 ? squareRoot(a) : sqrt(a); }
};

/// the basis of a quintic segment at one point (quinticSegmentR): f = fl + bf d0 + dx f1l + b1 d1 + e f2l + b2 d2,
/// f' = bfp d0 + f1l + b1p d1 + dx f2l + b2p d2
struct SegmentBasis {
    double bf, dx, b1, e, b2, bfp, b1p, b2p;
    __device__ __forceinline__ SegmentBasis(double x, double xl, double xh, double hi)
    {
        dx = x - xl;
        const double h = xh - xl, h2 = h * h, t = dx * hi, t2 = t * t, t3 = t * t2, omt = t * (1 - t);
        e = 0.5 * dx * dx;
        bf = t3 * (10 - t * (15 - 6 * t));
        b1 = t3 * (1 - t * 0.5) * h;
        b2 = t3 * (1 - t * (1.25 - 0.5 * t)) * h2;
        bfp = 30 * omt * hi * omt;
        b1p = t2 * (3 - t * 2);
        b2p = t2 * (3 - t * (5 - 2.5 * t)) * h;
    }
    __device__ __forceinline__ double value(double fl, double f1l, double f2l, double d0, double d1, double d2) const
    {
        return fma(b2, d2, fma(e, f2l, fma(b1, d1, fma(dx, f1l, fma(bf, d0, fl)))));
    }
    __device__ __forceinline__ double slope(double f1l, double f2l, double d0, double d1, double d2) const
    {
        return fma(b2p, d2, fma(dx, f2l, fma(b1p, d1, fma(bfp, d0, f1l))));
    }
};

/** The values (and with SLOPE the tau derivatives) of the six functions of a cell at a tau within it
    (MultipoleView::segments): what depends on the table alone -- the three defects of each segment, a
    quarter of the arithmetic of spline2dCell -- is tabulated, by the same operations.  At the cell's upper
    tau node (the last one of the grid, on the axis) they are the node values, without round-off; node:
    the spline node (xlow, yupp), row: the distance to (xupp, yupp).  F[0] and F[1] are relative to off.
    (The upper ln r node is never met: the last one lies beyond the switch to the outer expansion.) */
template<bool SLOPE>
__device__ __forceinline__ void cellSegments(const double* __restrict__ c, const double* node, size_t row, bool upper,
    const SegmentBasis& y, double* F, double* G, double* off)
{
    if(upper) {
        const int val[3] = { 0, 1, 3 }, dy[3] = { 2, 4, 6 };
        *off = ldg(node);
#pragma unroll
        for(int p = 0; p < 3; p++) {
            F[2 * p] = p == 0 ? 0 : ldg(node + val[p]);
            F[2 * p + 1] = p == 0 ? ldg(node + row) - *off : ldg(node + row + val[p]);
            if(SLOPE) { G[2 * p] = ldg(node + dy[p]); G[2 * p + 1] = ldg(node + row + dy[p]); }
        }
        return;
    }
#pragma unroll
    for(int p = 0; p < 6; p += 2) {
        double w[12];
        ldg4(c + 6 * p, w);
        ldg4(c + 6 * p + 4, w + 4);
        ldg4(c + 6 * p + 8, w + 8);
        if(p == 0) { *off = w[0]; w[0] = 0; }
#pragma unroll
        for(int a = 0; a < 2; a++) {
            const double* s = w + 6 * a;
            F[p + a] = y.value(s[0], s[1], s[2], s[3], s[4], s[5]);
            if(SLOPE) G[p + a] = y.slope(s[1], s[2], s[3], s[4], s[5]);
        }
    }
}

/// the defects of the segment in ln r from its six values (quinticSegmentR), hx: its width
__device__ __forceinline__ void segmentDefects(const double* f, double hx, double* d)
{
    d[0] = fma(-(0.5 * hx), f[3] + f[2], f[1] - f[0]);
    d[1] = fma(-(0.5 * hx), f[5] + f[4], f[3] - f[2]);
    d[2] = f[5] - f[4];
}

/// spline2dCell for value and gradient from the cell's segments
__device__ __forceinline__ void segmentCell(const double* __restrict__ c, const double* node, size_t row, bool upper,
    const SegmentBasis& x, double hx, const SegmentBasis& y, double* z, double* zx, double* zy)
{
    double F[6], G[6], off, d[3];
    cellSegments<true>(c, node, row, upper, y, F, G, &off);
    segmentDefects(F, hx, d);
    *z = x.value(F[0], F[2], F[4], d[0], d[1], d[2]) + off;
    *zx = x.slope(F[2], F[4], d[0], d[1], d[2]);
    segmentDefects(G, hx, d);
    *zy = x.value(G[0], G[2], G[4], d[0], d[1], d[2]);
}

/** evalInterp2dFast for value and gradient with the harmonics taken one after the other: each one is
    evaluated, scaled and added to the Fourier sums (m = 0 first, then by ascending m), and the
    cosine and sine of m phi follow by the same multiple-angle recurrence up to |m| (begun anew where |m|
    falls), so nothing is kept per harmonic.
    G > 1: the lanes of a group take G harmonics at a time, one each, and every lane adds all of them
    in the same order from the lane that evaluated it, so every G gives the same bits.
    MIXED: the m != 0 harmonics from the FP32 table.  rsq: R^2 + z^2, rounded as the caller wants it. */
template<int KIND, int G, bool MIXED>
__device__ __forceinline__ void forceInterp2d(const MultipoleView& M, double R, double z, double rsq, double phi, double* pot,
    CylDerivs* g)
{
    const int gl = G > 1 ? static_cast<int>(threadIdx.x % G) : 0;
    const unsigned gmask = G > 1 ? groupMask<G>() : 0u;
    const double r = squareRoot(rsq), logr = log(r), rpRinv = reciprocal(r + fabs(R));
    const double tau = R == 0 ? signOf(z) : z * rpRinv;
    const bool inside = logr >= M.gridR.x0 && logr <= M.gridR.xEnd && tau >= M.gridTau.x0 && tau <= M.gridTau.xEnd;
    double xl, xh, yl, yh, xhi, yhi;
    const int xs = gridCell(M.gridR, logr, &xl, &xh, &xhi), ys = gridCell(M.gridTau, tau, &yl, &yh, &yhi);
    const bool upper = tau == yh;
    const SegmentBasis bx(logr, xl, xh, xhi), by(tau, yl, yh, yhi);
    const size_t slotStride = static_cast<size_t>(M.nr) * M.nt * NODE_STRIDE;
    const size_t segmentStride = static_cast<size_t>(M.nr - 1) * (M.nt - 1) * CELL_COEFS;
    const double* segments = M.segments + (static_cast<size_t>(xs) * (M.nt - 1) + ys) * CELL_COEFS;
    const double* nodes = M.spl2d + (static_cast<size_t>(xs) * M.nt + ys + 1) * NODE_STRIDE;
    auto cell = [&](int s, double* P, double* Dr, double* Dt) {
        const int slot = M.fastSlot[s];
        if(MIXED && s > 0) {    // m != 0 (angular) harmonics in FP32, the radial m = 0 one in FP64
            double rr, rt, tt;
            spline2dCell32<3>(M.spl2d32 + slot * slotStride, M.nt, xs, ys, logr, xl, xh, tau, yl, yh,
                P, Dr, Dt, &rr, &rt, &tt);
        } else
            segmentCell(segments + slot * segmentStride, nodes + slot * slotStride, static_cast<size_t>(M.nt) * NODE_STRIDE,
                upper, bx, xh - xl, by, P, Dr, Dt);
        if(!inside) *P = *Dr = *Dt = NAN;
    };
    const int numHarm = KIND == EVAL_AXI ? 1 : M.nFast;
    double P0, Dr0, Dt0;            // the m = 0 harmonic, as it enters the sums
    double Pv = 0, Drv = 0, Dtv = 0;    // this lane's harmonic of the current round
    SphDerivs gs;
    double s1 = 0, c1 = 1, sh = 0, ch = 1;
    if(KIND != EVAL_AXI && numHarm > 1) {
        sincos(phi, &s1, &c1);
        sincos(0.5 * phi, &sh, &ch);
    }
    const double alpha = 2 * sh * sh, beta = s1;
    double cp = 1, sp = 0;
    int k = 0;
    for(int base = 0; base < numHarm; base += G) {
        const int s = base + gl;
        if(s < numHarm) cell(s, &Pv, &Drv, &Dtv);
        if(base == 0) {
            P0 = Pv; Dr0 = Drv; Dt0 = Dtv;
            if(G > 1) {
                P0 = __shfl_sync(gmask, P0, 0, G); Dr0 = __shfl_sync(gmask, Dr0, 0, G); Dt0 = __shfl_sync(gmask, Dt0, 0, G);
            }
            if(M.logScaling) {
                const double ex = exp(P0), val = reciprocal(M.invPhi0 - ex);
                P0 = val;
                const double dPdX = val * val * ex;
                Dr0 *= dPdX;
                Dt0 *= dPdX;
            }
            *pot = P0;
            gs.dr = Dr0; gs.dt = Dt0; gs.dphi = 0;
        }
        if(M.logScaling && s > 0) {
            Drv = sumProducts(Drv, P0, Pv, Dr0);
            Dtv = sumProducts(Dtv, P0, Pv, Dt0);
            Pv *= P0;
        }
        if(KIND != EVAL_AXI) {
#pragma unroll
            for(int q = 0; q < G; q++) {
                if(base + q == 0) continue;
                if(base + q >= numHarm) break;
                const int m = M.fastM[base + q], absm = m < 0 ? -m : m;
                if(absm < k) { cp = 1; sp = 0; k = 0; }
                for(; k < absm; k++) {
                    const double c = cp - sumProducts(alpha, cp, beta, sp);
                    const double sv = sp - (k == 1 ? sumProducts(-beta, cp, alpha, sp) : sumProducts(alpha, sp, -beta, cp));
                    cp = c;
                    sp = sv;
                }
                double P = Pv, Dr = Drv, Dt = Dtv;
                if(G > 1) {
                    P = __shfl_sync(gmask, P, q, G); Dr = __shfl_sync(gmask, Dr, q, G); Dt = __shfl_sync(gmask, Dt, q, G);
                }
                const double tr = m > 0 ? cp : sp;
                const double dtr = m > 0 ? -m * sp : -m * cp;
                *pot += P * tr;
                gs.dr += Dr * tr;
                gs.dt += Dt * tr;
                gs.dphi += P * dtr;
            }
        }
    }
    const double rinv = reciprocal(r), r2inv = rinv * rinv;
    const double drdR = R * r2inv, drdz = z * r2inv, dtdR = -tau * rinv, dtdz = rinv - rpRinv;
    g->dR = sumProducts(gs.dr, drdR, gs.dt, dtdR);
    g->dz = sumProducts(gs.dr, drdz, gs.dt, dtdz);
    g->dphi = gs.dphi;
}

/** evalPowerLaw for value and gradient and expansions with cosine terms only (lmax > 2 or one harmonic):
    the terms are summed as they come.  A lane beyond the grid holds its whole warp in this path, so its
    length counts (4500 instructions an evaluation of a triaxial expansion of lmax 6 before): the powers
    (r/r0)^v are formed once per l instead of once per term, those of terms with amplitude 0 not at all, the
    derivatives of the Legendre functions only for the l in use, the ratios of their normalisations are
    tabulated, and the divisions by sin(theta) and by l - m share their reciprocals (quotient). */
__device__ __forceinline__ void powerLawTerms(const PowerLawView& A, double R, double z, double phi, double* pot,
    CylDerivs* g)
{
    const HarmIndices& ind = A.ind;
    const double rsq = sumProducts(z, z, R, R), dlogr = log(rsq / A.r0sq) * 0.5;
    const int lmax = (A.inner && rsq < A.r0sq * 1e-16) || (!A.inner && rsq > A.r0sq * 1e16) ? 0 : ind.lmax;
    double rv[LMAX_MAX + 1];
    for(int l = 0; l <= lmax; l += ind.step) {
        const double v = A.inner ? l : -l - 1;
        rv[l] = v != 0 ? exp(dlogr * v) : 1;
    }
    // Phi_lm(r) = U (r/r0)^s [ln(r/r0) if s == v] + W (r/r0)^v [+ Q (r/r0)^2]; derivative in ln r
    auto coef = [&](int l, int m, double* C, double* dC) {
        const int c = HarmIndices::index(l, m);
        const double s = ldg(A.S + c), u = ldg(A.U + c), w = ldg(A.W + c), v = A.inner ? l : -l - 1;
        const double rs = s != v ? (s != 0 && u != 0 ? exp(dlogr * s) : 1) : rv[l];
        const double urs = u * rs * (s != v || u == 0 ? 1 : dlogr);
        const double wrv = w * rv[l];
        const double qr2 = v == 0 ? A.Q * rsq / A.r0sq : 0;
        *C = __dadd_rn(urs, wrv) + qr2;
        *dC = sumProducts(wrv, v, urs, s) + (s != v ? 0 : u * rs) + qr2 * 2;
    };
    if(lmax == 0) {
        double C0, dC0 = 0;
        coef(0, 0, &C0, &dC0);
        *pot = C0;
        const double rsqinv = rsq > 0 ? 1 / rsq : 0;
        const double Rr2 = rsq < INFINITY ? R * rsqinv : 0, zr2 = rsq < INFINITY ? z * rsqinv : 0;
        g->dR = dC0 * Rr2; g->dz = dC0 * zr2; g->dphi = 0;
        return;
    }
    const double tau = z == 0 ? 0 : z / (sqrt(sumProducts(z, z, R, R)) + R);
    const double ct = 2 * tau / (1 + tau * tau), st = (1 - tau * tau) / (1 + tau * tau);
    const double EPS = 1e-8, stInv = 1 / st;
    double s1 = 0, c1 = 1, sh = 0, ch = 1;
    if(ind.mmax > 0) {
        sincos(phi, &s1, &c1);
        sincos(0.5 * phi, &sh, &ch);
    }
    const double alpha = 2 * sh * sh, beta = s1;
    double cp = 1, sp = 0, val = 0, gr = 0, gt = 0, gp = 0;
    for(int m = 0; m <= ind.mmax; m++) {
        if(m > 0) {
            const double c = cp - sumProducts(alpha, cp, beta, sp), sv = sp - sumProducts(alpha, sp, -beta, cp);
            cp = c;
            sp = sv;
        }
        const int lmin = ind.lmin(m);
        if(lmin > lmax) continue;
        const double mul = m == 0 ? 2 * SQRT_PI : 2 * SQRT_PI * M_SQRT2;
        // P_m^m and its derivative (legendreArray)
        double prefact = PMM_NORM_DEV[m], P, dP;
        if(m == 0) { P = prefact; dP = 0; }
        else if(m == 1) { P = -st * prefact; dP = -ct * prefact; }
        else {
            double sinm2 = 1, base = st;
            for(int e = m - 2; ; ) {
                if(e % 2) sinm2 *= base;
                e >>= 1;
                base *= base;
                if(!e) break;
            }
            P = PMM_COEF_DEV[m] * sinm2 * (st * st);
            dP = m * PMM_COEF_DEV[m] * sinm2 * st * ct;
        }
        double Cm = 0, dCm = 0, tCm = 0;
        auto add = [&](int l) {
            double C, dC;
            coef(l, m, &C, &dC);
            Cm = fma(P * C, mul, Cm);
            dCm = fma(P * dC, mul, dCm);
            tCm = fma(dP * C, mul, tCm);
        };
        if(lmin == m) add(m);
        double Plm1 = P / prefact, Plm = ct * (2 * m + 1) * Plm1, Plm2 = 0;
        for(int l = m + 1; l <= lmax; l++) {
            if(l > m + 1) {
                const double num = sumProducts(ct * (2 * l - 1), Plm1, -(l + m - 1), Plm2), d = l - m;
                Plm = quotient(num, d, 1 / d);
            }
            prefact *= ldg(A.norm + m * (LMAX_MAX + 1) + l);
            if(l >= lmin && (l - lmin) % ind.step == 0) {
                P = Plm * prefact;
                double dPlm = 0;
                if(st >= EPS || (m > 2 && st > 0))
                    dPlm = quotient(sumProducts(l * ct, Plm, -(l + m), Plm1), st, stInv);
                else if(m == 0)
                    dPlm = -l * (l + 1) / 2 * st * (ct > 0 || l % 2 == 1 ? 1 : -1);
                else if(m == 1)
                    dPlm = -l * (l + 1) / 2 * (ct > 0 || l % 2 == 0 ? 1 : -1);
                else if(m == 2)
                    dPlm = l * (l + 1) * (l + 2) * (l - 1) / 4 * st * (ct > 0 || l % 2 == 1 ? 1 : -1);
                dP = prefact * dPlm;
                add(l);
            }
            Plm2 = Plm1;
            Plm1 = Plm;
        }
        if(m == 0) { val = Cm; gr = dCm; gt = tCm; }
        else {
            val = fma(Cm, cp, val);
            gr = fma(dCm, cp, gr);
            gt = fma(tCm, cp, gt);
            gp = fma(Cm, -m * sp, gp);
        }
    }
    *pot = val;
    const double r2inv = 1 / sumProducts(z, z, R, R);
    const double drdR = R * r2inv, drdz = z * r2inv;
    g->dR = sumProducts(gr, drdR, gt, drdz);
    g->dz = sumProducts(gr, drdz, gt, -drdR);
    g->dphi = gp;
}

/// the potential alone of an axisymmetric expansion at (R, z) inside its 2-D splines, to the bit that of
/// evalInterp2dFast
__device__ __forceinline__ double valueInterp2d(const MultipoleView& M, double R, double z)
{
    const double r = squareRoot(sumProducts(z, z, R, R)), logr = log(r), rpRinv = reciprocal(r + fabs(R));
    const double tau = R == 0 ? signOf(z) : z * rpRinv;
    const bool inside = logr >= M.gridR.x0 && logr <= M.gridR.xEnd && tau >= M.gridTau.x0 && tau <= M.gridTau.xEnd;
    double xl, xh, yl, yh, xhi, yhi, F[6], off, d[3];
    const int xs = gridCell(M.gridR, logr, &xl, &xh, &xhi), ys = gridCell(M.gridTau, tau, &yl, &yh, &yhi);
    const SegmentBasis x(logr, xl, xh, xhi), y(tau, yl, yh, yhi);
    const size_t slot = M.fastSlot[0];
    cellSegments<false>(M.segments + ((slot * (M.nr - 1) + xs) * (M.nt - 1) + ys) * CELL_COEFS,
        M.spl2d + ((slot * M.nr + xs) * M.nt + ys + 1) * NODE_STRIDE, static_cast<size_t>(M.nt) * NODE_STRIDE, tau == yh, y,
        F, nullptr, &off);
    segmentDefects(F, xh - xl, d);
    double P = x.value(F[0], F[2], F[4], d[0], d[1], d[2]) + off;
    if(!inside) P = NAN;
    if(M.logScaling) P = reciprocal(M.invPhi0 - exp(P));
    return P;
}

/// an axisymmetric asymptotic expansion (evalPowerLaw), with SLOPE its gradient over R and z: one short
/// loop, inline; rsq: R^2 + z^2, rounded as the caller wants it.  The same sums, but not to the bit:
/// the contractions of evalPowerLaw are the compiler's, and expansions of lmax 2 take the recurrence
/// here and a closed form there.
template<bool SLOPE>
__device__ __forceinline__ double axisPowerLaw(const PowerLawView& A, double R, double z, double rsq, double* gR, double* gz)
{
    const HarmIndices& ind = A.ind;
    const double dlogr = log(rsq / A.r0sq) * 0.5;
    const int lmax = (A.inner && rsq < A.r0sq * 1e-16) || (!A.inner && rsq > A.r0sq * 1e16) ? 0 : ind.lmax;
    const double tau = z == 0 ? 0 : z / (sqrt(rsq) + R);
    const double ct = 2 * tau / (1 + tau * tau), st = SLOPE ? (1 - tau * tau) / (1 + tau * tau) : 0, stInv = SLOPE ? 1 / st : 0;
    double prefact = PMM_NORM_DEV[0], sum = 0, sumr = 0, sumt = 0, Plm1 = 1, Plm = 1, Plm2 = 0;
    for(int l = 0; l <= lmax; l++) {
        if(l == 1) Plm = ct * Plm1;
        else if(l > 1) {
            const double num = sumProducts(ct * (2 * l - 1), Plm1, -(l - 1), Plm2), d = l;
            Plm = quotient(num, d, 1 / d);
        }
        if(l > 0) prefact *= ldg(A.norm + l);
        if(l % ind.step == 0) {
            const int c = HarmIndices::index(l, 0);
            const double s = ldg(A.S + c), u = ldg(A.U + c), w = ldg(A.W + c), v = A.inner ? l : -l - 1;
            const double rv = v != 0 ? exp(dlogr * v) : 1;
            const double rs = s != v ? (s != 0 && u != 0 ? exp(dlogr * s) : 1) : rv;
            const double urs = u * rs * (s != v || u == 0 ? 1 : dlogr), wrv = w * rv;
            const double qr2 = v == 0 ? A.Q * rsq / A.r0sq : 0;
            const double C = __dadd_rn(urs, wrv) + qr2;
            double dC = 0;
            if(SLOPE) dC = sumProducts(wrv, v, urs, s) + (s != v ? 0 : u * rs) + qr2 * 2;
            if(lmax == 0) {
                if(SLOPE) {
                    const double rsqinv = rsq > 0 ? 1 / rsq : 0;
                    *gR = dC * (rsq < INFINITY ? R * rsqinv : 0);
                    *gz = dC * (rsq < INFINITY ? z * rsqinv : 0);
                }
                return C;
            }
            const double P = Plm * prefact;
            sum = fma(P * C, 2 * SQRT_PI, sum);
            if(SLOPE) {
                sumr = fma(P * dC, 2 * SQRT_PI, sumr);
                const double dPlm = l == 0 ? 0 :
                    st >= 1e-8 ? quotient(sumProducts(l * ct, Plm, -l, Plm1), st, stInv) :
                    -l * (l + 1) / 2 * st * (ct > 0 || l % 2 == 1 ? 1 : -1);
                sumt = fma(prefact * dPlm * C, 2 * SQRT_PI, sumt);
            }
        }
        Plm2 = Plm1;
        Plm1 = Plm;
    }
    if(SLOPE) {
        const double r2inv = 1 / rsq, drdR = R * r2inv, drdz = z * r2inv;
        *gR = sumProducts(sumr, drdR, sumt, drdz);
        *gz = sumProducts(sumr, drdz, sumt, -drdR);
    }
    return sum;
}

/// beyond the 2-D splines: asymptotic expansions (and 1-D splines); out of line
static __device__ __noinline__ void forceBeyond(const MultipoleView& M, double R, double z, double phi, double* pot, CylDerivs* g)
{
    const double rsq = sumProducts(R, R, z, z);
    CylHess h;
    if(rsq < M.rInnerSq || rsq > M.rOuterSq) {
        const PowerLawView& A = rsq < M.rInnerSq ? M.inner : M.outer;
        if(A.ind.mmin() == 0 && (A.ind.lmax != 2 || A.ind.step != 2))
            powerLawTerms(A, R, z, phi, pot, g);
        else
            evalPowerLaw<3>(A, R, z, phi, pot, g, &h);
    } else if(M.is2d)
        evalInterp2d<3>(M, R, z, phi, pot, g, &h);      // (2-D splines without cells)
    else
        evalInterp1d<3>(M, R, z, phi, pot, g, &h);
}

/** Potential and its gradient at a Cartesian point (evalMultipoleCar for value and gradient) */
template<int KIND, int G, bool MIXED>
__device__ __forceinline__ void evalForceCar(const MultipoleView& M, double x, double y, double z, double* pot, double* grad)
{
    // (squares that leave the range of normal numbers take the library's root and divisions)
    const double R2 = sumProducts(x, x, y, y);
    const bool usual = R2 > 1e-200 && R2 < 1e200;
    const double R = usual ? squareRoot(R2) : sqrt(R2);
    // a potential with only m = 0 terms (its splines and both asymptotes): its evaluators neither
    // read the azimuth nor give a phi derivative (exactly 0), so neither atan2 nor the azimuth's
    // derivatives are formed (the results are the same bits)
    const bool noAzimuth = KIND == EVAL_AXI && M.ind.mmax == 0 && M.inner.ind.mmax == 0 && M.outer.ind.mmax == 0;
    double phi;
    double dRdx, dRdy, dphidx = 0, dphidy = 0;
    if(R == 0) {
        phi = 0; dRdx = dRdy = dphidx = dphidy = 1;
    } else {
        const double Rinv = usual ? reciprocal(R) : 0;
        const double cphi = usual ? quotient(x, R, Rinv) : x / R, sphi = usual ? quotient(y, R, Rinv) : y / R;
        dRdx = cphi; dRdy = sphi;
        if(!noAzimuth) {
            dphidx = usual ? quotient(-sphi, R, Rinv) : -sphi / R;
            dphidy = usual ? quotient(cphi, R, Rinv) : cphi / R;
        }
        phi = noAzimuth ? 0 : atan2(y, x);
    }
    CylDerivs g;
    const double rsq = sumProducts(R, R, z, z);
    if(KIND == EVAL_GENERAL) {
        CylHess h;
        evalMultipoleCyl<3, KIND>(M, R, z, phi, pot, &g, &h);
    } else if(inCells(M, rsq))
        forceInterp2d<KIND, G, MIXED>(M, R, z, sumProducts(z, z, R, R), phi, pot, &g);
    else {      // (results of this branch's own: the common ones stay in registers)
        double p;
        CylDerivs d;
        forceBeyond(M, R, z, phi, &p, &d);
        *pot = p;
        g = d;
    }
    grad[0] = noAzimuth ? g.dR * dRdx : sumProducts(g.dR, dRdx, g.dphi, dphidx);
    grad[1] = noAzimuth ? g.dR * dRdy : sumProducts(g.dR, dRdy, g.dphi, dphidy);
    grad[2] = g.dz;
}

}  // namespace agb
