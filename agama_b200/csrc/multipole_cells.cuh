// Device evaluation of the Multipole potential from the coefficients of its spline cells.
//
// A cell of a 2-D quintic spline is a polynomial of degree 5 in each of the two positions within
// the cell, s = (ln r - its lower node) / width and t = (tau - the anchor node) / width.  The node
// form (multipole_eval.cuh) gathers the 4 x 9 node values of the cell and forms the Hermite basis, six
// segments in one direction and up to three in the other at every point: ~180 FP64 instructions for
// value and gradient, with all 36 values and twelve or more intermediates live.  Here the same
// polynomial is a Horner sum over its 36 monomial coefficients (nine 32-byte loads of one contiguous
// run): 35 multiply-adds for the value, 68 with the gradient, two rows of six at a time and only the
// running sums live, which is what lets the kernels keep more warps on an SM.  Both forms are the
// same polynomial; their results differ by rounding (the cells' coefficients are formed from the same
// node data).
//
// Callers whose results must not move in the last bits have the node form's arithmetic: orbits (chaotic
// ones amplify a rounding difference without bound) and angles from the segments of the same cells
// (multipole_force.cuh), the construction of the action finder (its grids come from differences of second
// derivatives) from the node form itself.
#pragma once
#include "multipole_eval.cuh"

namespace agb {

/// 1 / b for |b| well inside the range of normal numbers (no zeros, infinities or subnormals: they
/// give NaN): the hardware approximation refined by one step of third-order Newton (Householder)
/// iteration, y + y (e + e^2) with e = 1 - b y
__device__ __forceinline__ double rcpNormal(double b)
{
    double y;
    asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(b));
    const double e = fma(-b, y, 1.0);
    return fma(y, fma(e, e, e), y);
}

/// 1 / sqrt(a) for a > 0 well inside the range of normal numbers, by the same kind of step:
/// y + y (e / 2 + 3 e^2 / 8) with e = 1 - a y^2
__device__ __forceinline__ double rsqrtNormal(double a)
{
    double y;
    asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(a));
    const double e = fma(-(a * y), y, 1.0);
    return fma(y * e, fma(0.375, e, 0.5), y);
}

/// the arithmetic of root searches whose steps may move at the level of rounding
struct NormalArithmetic {
    static __device__ __forceinline__ double quotient(double a, double b)
    {
        const double y = rcpNormal(b), q = a * y;
        return fma(fma(-b, q, a), y, q);
    }
    static __device__ __forceinline__ double root(double a) { return a > 1e-280 ? a * rsqrtNormal(a) : a >= 0 ? 0 : NAN; }
};

/// four consecutive doubles, 32-byte aligned, in one load: a lane's cell lies in lines of its own, and
/// the L1's cost of a load is the number of different lines its lanes touch, so the width halves it
__device__ __forceinline__ void ldg4(const double* p, double* v)
{
    asm("ld.global.nc.v4.f64 {%0, %1, %2, %3}, [%4];" : "=d"(v[0]), "=d"(v[1]), "=d"(v[2]), "=d"(v[3]) : "l"(p));
}

/// findCell from device tables: index, nodes and reciprocal width of the cell
__device__ __forceinline__ int gridCell(const GridView& g, double x, double* xl, double* xh, double* invH)
{
    GridNode lo, hi;
    const int k = findCell(g, x, &lo, &hi, [&](int i) { const double2 v = ldg2(&g.cell[i].x); return GridNode{ v.x, v.y }; },
        [&](int b) { return __ldg(g.lut + b); });
    *xl = lo.x; *xh = hi.x; *invH = lo.invH;
    return k;
}

/// the node of a tau cell [yl, yh] about which its polynomial is expanded: the one nearer the pole
/// (the upper node in the upper half of the grid, the lower node below)
__device__ __forceinline__ double cellAnchor(double yl, double yh) { return yl + yh > 0 ? yh : yl; }

/** The polynomial of one cell at (s, t): value p, and by NQ the derivatives over s and t (3) and the
    second ones (6).  c: CELL_COEFS coefficients, 32-byte aligned (288 bytes a cell). */
template<int NQ>
__device__ __forceinline__ void cellPolynomial(const double* __restrict__ c, double s, double t,
    double* p, double* ps, double* pt, double* pss, double* pst, double* ptt)
{
    double v = 0, vs = 0, vt = 0, vss = 0, vst = 0, vtt = 0;
#pragma unroll
    for(int i = 4; i >= 0; i -= 2) {
        double w[12];       // rows i and i + 1
        ldg4(c + 6 * i, w);
        ldg4(c + 6 * i + 4, w + 4);
        ldg4(c + 6 * i + 8, w + 8);
#pragma unroll
        for(int k = 1; k >= 0; k--) {
            const double* a = w + 6 * k;
            // one row: sum over the powers of t, its first and (half the) second derivative
            double q = fma(a[5], t, a[4]), qt = a[5], qtt = 0;
            if(NQ == 6) qtt = a[5];
            if(NQ >= 3) qt = fma(qt, t, q);
            q = fma(q, t, a[3]);
            if(NQ == 6) qtt = fma(qtt, t, qt);
            if(NQ >= 3) qt = fma(qt, t, q);
            q = fma(q, t, a[2]);
            if(NQ == 6) qtt = fma(qtt, t, qt);
            if(NQ >= 3) qt = fma(qt, t, q);
            q = fma(q, t, a[1]);
            if(NQ == 6) qtt = fma(qtt, t, qt);
            if(NQ >= 3) qt = fma(qt, t, q);
            q = fma(q, t, a[0]);
            const int row = i + k;
            if(row == 5) { v = q; vt = qt; vtt = qtt; }
            else {
                if(NQ == 6) {
                    vss = row == 4 ? 0 : row == 3 ? vs : fma(vss, s, vs);
                    vst = row == 4 ? vt : fma(vst, s, vt);
                    vtt = fma(vtt, s, qtt);
                }
                if(NQ >= 3) { vs = row == 4 ? v : fma(vs, s, v); vt = fma(vt, s, qt); }
                v = fma(v, s, q);
            }
        }
    }
    *p = v;
    if(NQ >= 3) { *ps = vs; *pt = vt; }
    if(NQ == 6) { *pss = 2 * vss; *pst = vst; *ptt = 2 * vtt; }
}

/// value, gradient and Hessian of an evaluation out of line
struct BeyondCells { double pot; CylDerivs g; CylHess h; };

/// the rare places: the asymptotic expansions beyond the radial grid, the 1-D splines of lmax <= 2
/// and 2-D splines without cells; out of line so that the callers' registers and
/// instruction stream are those of the cells (the callers copy from a result of this branch's own: one
/// whose address left the common path would keep the common results in local memory)
template<int NQ>
__device__ __noinline__ void evalBeyondCells(const MultipoleView& M, double R, double z, double phi, BeyondCells* r)
{
    const double rsq = R * R + z * z;
    if(rsq < M.rInnerSq)      evalPowerLaw<NQ>(M.inner, R, z, phi, &r->pot, &r->g, &r->h);
    else if(rsq > M.rOuterSq) evalPowerLaw<NQ>(M.outer, R, z, phi, &r->pot, &r->g, &r->h);
    else if(M.is2d)           evalInterp2d<NQ>(M, R, z, phi, &r->pot, &r->g, &r->h);
    else                      evalInterp1d<NQ>(M, R, z, phi, &r->pot, &r->g, &r->h);
}

/** The 2-D spline evaluation (MultipoleInterp2d::evalCyl, src/potential_multipole.cpp:1969-2080) from
    the cells: the harmonics are taken one after the other (m = 0 first, then by ascending m), each
    scaled and added to the Fourier sums at once, with cos and sin of m phi carried along by
    rotations from cos and sin of phi.  KIND: EVAL_AXI (one harmonic) or EVAL_FAST. */
template<int NQ, int KIND>
__device__ __forceinline__ void evalCells(const MultipoleView& M, double R, double z, double cphi, double sphi,
    double* pot, CylDerivs* g, CylHess* h)
{
    const double rsq = R * R + z * z, logr = 0.5 * log(rsq);
    const double rinv = rsqrtNormal(rsq), r = rsq * rinv, rpRinv = rcpNormal(r + fabs(R));
    const double tau = R == 0 ? signOf(z) : fmin(fmax(z * rpRinv, -1.), 1.);
    const bool inside = logr >= M.gridR.x0 && logr <= M.gridR.xEnd && tau >= M.gridTau.x0 && tau <= M.gridTau.xEnd;
    double xl, xh, xi, yl, yh, yi;
    const int ix = gridCell(M.gridR, logr, &xl, &xh, &xi), iy = gridCell(M.gridTau, tau, &yl, &yh, &yi);
    const double s = (logr - xl) * xi, t = (tau - cellAnchor(yl, yh)) * yi;
    const size_t slotStride = static_cast<size_t>(M.nr - 1) * (M.nt - 1) * CELL_COEFS;
    const double* cell = M.cells + (static_cast<size_t>(ix) * (M.nt - 1) + iy) * CELL_COEFS;
    double P0, x0, y0, xx0 = 0, xy0 = 0, yy0 = 0;       // the m = 0 harmonic and its derivatives
    cellPolynomial<NQ>(cell + M.fastSlot[0] * slotStride, s, t, &P0, &x0, &y0, &xx0, &xy0, &yy0);
    if(!inside) P0 = NAN;
    if(NQ >= 3) { x0 *= xi; y0 *= yi; }
    if(NQ == 6) { xx0 *= xi * xi; xy0 *= xi * yi; yy0 *= yi * yi; }
    if(M.logScaling) {
        const double ex = exp(P0), val = rcpNormal(M.invPhi0 - ex);
        if(NQ >= 3) {
            const double dPdX = val * val * ex;
            if(NQ == 6) {
                const double d2PdX2 = dPdX * val * (M.invPhi0 + ex);
                xx0 = dPdX * xx0 + d2PdX2 * x0 * x0;
                yy0 = dPdX * yy0 + d2PdX2 * y0 * y0;
                xy0 = dPdX * xy0 + d2PdX2 * x0 * y0;
            }
            x0 *= dPdX;
            y0 *= dPdX;
        }
        P0 = val;
    }
    double Phi = P0;
    SphDerivs gs{ x0, y0, 0 };
    SphHess hs{ xx0, yy0, 0, xy0, 0, 0 };
    if(KIND == EVAL_FAST) {
        double cm = 1, sm = 0;
        int k = 0;
        for(int q = 1; q < M.nFast; q++) {
            const int m = M.fastM[q], absm = m < 0 ? -m : m;
            if(absm < k) { cm = 1; sm = 0; k = 0; }
            for(; k < absm; k++) {
                const double c = cm * cphi - sm * sphi;
                sm = sm * cphi + cm * sphi;
                cm = c;
            }
            double P, x, y, xx = 0, xy = 0, yy = 0;
            cellPolynomial<NQ>(cell + M.fastSlot[q] * slotStride, s, t, &P, &x, &y, &xx, &xy, &yy);
            if(NQ >= 3) { x *= xi; y *= yi; }
            if(NQ == 6) { xx *= xi * xi; xy *= xi * yi; yy *= yi * yi; }
            if(M.logScaling) {
                if(NQ == 6) {
                    xx = xx * P0 + P * xx0 + 2 * x * x0;
                    yy = yy * P0 + P * yy0 + 2 * y * y0;
                    xy = xy * P0 + P * xy0 + x * y0 + y * x0;
                }
                if(NQ >= 3) { x = x * P0 + P * x0; y = y * P0 + P * y0; }
                P *= P0;
            }
            const double tr = m > 0 ? cm : sm, dtr = m > 0 ? -m * sm : -m * cm;
            Phi += P * tr;
            if(NQ >= 3) { gs.dr += x * tr; gs.dt += y * tr; gs.dphi += P * dtr; }
            if(NQ == 6) {
                hs.dr2 += xx * tr; hs.drdt += xy * tr; hs.dt2 += yy * tr;
                hs.drdphi += x * dtr; hs.dtdphi += y * dtr; hs.dphi2 -= m * m * (P * tr);
            }
        }
    }
    *pot = Phi;
    if(NQ == 1) return;
    const double r2inv = rinv * rinv;
    const double drdR = R * r2inv, drdz = z * r2inv, dtdR = -tau * rinv, dtdz = rinv - rpRinv;
    g->dR = gs.dr * drdR + gs.dt * dtdR;
    g->dz = gs.dr * drdz + gs.dt * dtdz;
    g->dphi = gs.dphi;
    if(NQ == 6) {
        const double d2rdR2 = drdz * drdz - drdR * drdR, d2rdRdz = -2 * drdR * drdz, d2rdz2 = -d2rdR2;
        const double d2tdR2 = z * r2inv * rinv;
        const double d2tdRdz = dtdR * dtdR - drdR * drdR * r * rpRinv;
        const double d2tdz2 = -d2tdR2 - dtdR * rpRinv;
        h->dR2 = (hs.dr2 * drdR + hs.drdt * dtdR) * drdR + (hs.drdt * drdR + hs.dt2 * dtdR) * dtdR +
                 gs.dr * d2rdR2 + gs.dt * d2tdR2;
        h->dRdz = (hs.dr2 * drdz + hs.drdt * dtdz) * drdR + (hs.drdt * drdz + hs.dt2 * dtdz) * dtdR +
                  gs.dr * d2rdRdz + gs.dt * d2tdRdz;
        h->dz2 = (hs.dr2 * drdz + hs.drdt * dtdz) * drdz + (hs.drdt * drdz + hs.dt2 * dtdz) * dtdz +
                 gs.dr * d2rdz2 + gs.dt * d2tdz2;
        h->dRdphi = hs.drdphi * drdR + hs.dtdphi * dtdR;
        h->dzdphi = hs.drdphi * drdz + hs.dtdphi * dtdz;
        h->dphi2 = hs.dphi2;
    }
}

/// inside the radial range of the cells (evalMultipoleCyl's choice of the interpolator; NaN is too)
__device__ __forceinline__ bool inCells(const MultipoleView& M, double rsq)
{
    return !(rsq < M.rInnerSq) && !(rsq > M.rOuterSq) && M.cells;
}

/// Multipole::evalCyl (src/potential_multipole.cpp:1538-1548); KIND EVAL_GENERAL keeps the node form
template<int NQ, int KIND>
__device__ __forceinline__ void evalCellsCyl(const MultipoleView& M, double R, double z, double phi,
    double* pot, CylDerivs* g, CylHess* h)
{
    if(KIND == EVAL_GENERAL) { evalMultipoleCyl<NQ, KIND>(M, R, z, phi, pot, g, h); return; }
    if(inCells(M, R * R + z * z)) {
        double sphi = 0, cphi = 1;
        if(KIND == EVAL_FAST) sincos(phi, &sphi, &cphi);
        evalCells<NQ, KIND>(M, R, z, cphi, sphi, pot, g, h);
    } else {        // (a result of this branch's own, whose address the calls in it take)
        double p;
        CylDerivs d; CylHess dd;
        evalMultipoleCyl<NQ, KIND>(M, R, z, phi, &p, &d, &dd);
        *pot = p;
        if(NQ >= 3) *g = d;
        if(NQ == 6) *h = dd;
    }
}

/** Evaluation at a Cartesian point with gradient (and Hessian xx,yy,zz,xy,yz,zx) in Cartesian
    coordinates, as evalMultipoleCar: the azimuth enters only through its cosine and
    sine, x / R and y / R, so neither atan2 nor sincos is formed.  False for a point beyond the cells
    (nothing evaluated). */
template<int NQ, int KIND>
__device__ __forceinline__ bool evalCellsCar(const MultipoleView& M, double x, double y, double z,
    double* pot, double* grad, double* hess)
{
    const double R2 = x * x + y * y, R = sqrt(R2);
    if(!inCells(M, R * R + z * z)) return false;
    const bool axis = R == 0;
    const double Rinv = axis ? 0 : 1 / R, c = x * Rinv, s = y * Rinv;
    CylDerivs g; CylHess h;
    evalCells<NQ, KIND>(M, R, z, axis ? 1 : c, s, pot, &g, &h);
    if(NQ == 1) return true;
    // on the axis the transformation is degenerate: the derivatives of R and phi are given as 1
    const double dRdx = axis ? 1 : c, dRdy = axis ? 1 : s, dphidx = axis ? 1 : -s * Rinv, dphidy = axis ? 1 : c * Rinv;
    grad[0] = g.dR * dRdx + g.dphi * dphidx;
    grad[1] = g.dR * dRdy + g.dphi * dphidy;
    grad[2] = g.dz;
    if(NQ == 6) {
        double d2Rdx2 = 1, d2Rdy2 = 1, d2Rdxdy = 1, d2phidx2 = 1, d2phidy2 = 1, d2phidxdy = 1;
        if(!axis) {
            d2Rdx2 = s * s * Rinv; d2Rdy2 = c * c * Rinv; d2Rdxdy = -s * c * Rinv;
            // (factor by factor: the square of 1 / R overflows where the factor before it can be 0)
            d2phidx2 = 2 * s * c * Rinv * Rinv; d2phidy2 = -d2phidx2; d2phidxdy = (s * s - c * c) * Rinv * Rinv;
        }
        hess[0] = (h.dR2 * dRdx + h.dRdphi * dphidx) * dRdx + (h.dRdphi * dRdx + h.dphi2 * dphidx) * dphidx +
                  g.dR * d2Rdx2 + g.dphi * d2phidx2;                                         // xx
        hess[1] = (h.dR2 * dRdy + h.dRdphi * dphidy) * dRdy + (h.dRdphi * dRdy + h.dphi2 * dphidy) * dphidy +
                  g.dR * d2Rdy2 + g.dphi * d2phidy2;                                         // yy
        hess[2] = h.dz2;                                                                      // zz
        hess[3] = (h.dR2 * dRdy + h.dRdphi * dphidy) * dRdx + (h.dRdphi * dRdy + h.dphi2 * dphidy) * dphidx +
                  g.dR * d2Rdxdy + g.dphi * d2phidxdy;                                       // xy
        hess[4] = h.dRdz * dRdy + h.dzdphi * dphidy;                                          // yz
        hess[5] = h.dRdz * dRdx + h.dzdphi * dphidx;                                          // zx
    }
    return true;
}

}  // namespace agb
