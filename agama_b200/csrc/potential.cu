// Multipole potential on the device: table upload and the batched evaluation kernel.
#include "runtime.h"
#include "multipole_cells.cuh"

namespace agb {

namespace {
thread_local std::string g_error;

/// Blocks of 128 per SM that the registers are cut for: points beyond the radial grid wait for the
/// logarithms and powers of the expansions, and the cells for their loads, so more warps are worth some
/// spilled registers.  Potential alone at 6 / 8 blocks: 54.0 / 51.5 us inside the grid, 99 / 88 beyond it (1e6 points,
/// disk potential); value and gradient at 5 / 6: 58.0 / 56.0, 123 / 115; with the Hessian at 3 / 4: 76 / 73, 236 / 199.
/// Potentials without cells take the compiler's own choice (96 and 166 registers; 1e6 points of one with 17
/// harmonics, potential alone: 436 us, 461 at 6 blocks, 517 at one) but for value and gradient, at 4 blocks
/// (4e5 points at its choice of 164 registers / 5 / 4 blocks: 17 harmonics inside the grid 270 / 266 / 250, inside and beyond it
/// 1205 / 967 / 1017, a lopsided l <= 2 potential 226 / 232 / 216).
constexpr int minBlocks(int nq, int kind)
{
    return kind == EVAL_GENERAL ? (nq == 3 ? 4 : 0) : nq == 1 ? 8 : nq == 3 ? 6 : 4;
}

/// One point per thread; 128 threads per block.  NQ = 1 (potential), 3 (+gradient), 6 (+Hessian);
/// KIND = spline evaluator matching the potential (EvalKind).  Bound by the L1: each lane reads its own
/// cells, nine 32-byte loads a harmonic at one data-stage cycle per lane (60 % of its rate at 2e6
/// points of the triaxial lmax 6 potential, value and gradient: 543 us from the node form at 168
/// registers, 410 from the cells with 16-byte loads at 80 registers, 330 with 32-byte loads, 305 with the
/// sign applied here instead of in a pass of its own, 298 with the expansions inline; Hessian and density of 4e5
/// points of the bar potential: 295 -> 161 us).
/// gradSign, hessSign: 1, or -1 for the acceleration and its derivatives.
template<int NQ, int KIND>
__global__ void __launch_bounds__(128, minBlocks(NQ, KIND)) evalPotentialKernel(const __grid_constant__ MultipoleView M, long n,
    const double* __restrict__ pos, double* __restrict__ phi, double* __restrict__ grad,
    double* __restrict__ hess, double gradSign, double hessSign)
{
    const long i = blockIdx.x * static_cast<long>(blockDim.x) + threadIdx.x;
    if(i >= n) return;
    const double x = pos[3 * i], y = pos[3 * i + 1], z = pos[3 * i + 2];
    auto store = [&](double p, const double* g, const double* h) {
        if(phi) phi[i] = p;
        if(NQ >= 3 && grad)
            for(int k = 0; k < 3; k++) grad[3 * i + k] = gradSign * g[k];
        if(NQ == 6 && hess)
            for(int k = 0; k < 6; k++) hess[6 * i + k] = hessSign * h[k];
    };
    double p, g[3], h[6];
    if constexpr(KIND == EVAL_GENERAL)
        evalMultipoleCar<NQ, KIND>(M, x, y, z, &p, g, h);
    else if(!evalCellsCar<NQ, KIND>(M, x, y, z, &p, g, h)) {
        double pb, gb[3], hb[6];    // (variables of the rare path's own, whose calls take their addresses)
        evalMultipoleCar<NQ, KIND>(M, x, y, z, &pb, gb, hb);
        store(pb, gb, hb);
        return;
    }
    store(p, g, h);
}

/// the same at n cylindrical points (R, z, phi), derivatives in cylindrical coordinates
/// (dR, dz, dphi; dR2, dz2, dphi2, dRdz, dzdphi, dRdphi) straight from the evaluator, as the
/// reference's BasePotentialCyl::evalCyl returns them (no round trip through Cartesian
/// derivatives, which loses the phi derivatives to cancellation at large R)
template<int NQ, int KIND>
__global__ void __launch_bounds__(128, minBlocks(NQ, KIND)) evalPotentialCylKernel(const __grid_constant__ MultipoleView M, long n,
    const double* __restrict__ pos, double* __restrict__ phi, double* __restrict__ grad,
    double* __restrict__ hess)
{
    const long i = blockIdx.x * static_cast<long>(blockDim.x) + threadIdx.x;
    if(i >= n) return;
    double p;
    CylDerivs g; CylHess h;
    evalCellsCyl<NQ, KIND>(M, pos[3 * i], pos[3 * i + 1], pos[3 * i + 2], &p, &g, &h);
    if(phi) phi[i] = p;
    if(NQ >= 3 && grad) { grad[3 * i] = g.dR; grad[3 * i + 1] = g.dz; grad[3 * i + 2] = g.dphi; }
    if(NQ == 6 && hess) {
        hess[6 * i] = h.dR2; hess[6 * i + 1] = h.dz2; hess[6 * i + 2] = h.dphi2;
        hess[6 * i + 3] = h.dRdz; hess[6 * i + 4] = h.dzdphi; hess[6 * i + 5] = h.dRdphi;
    }
}

/** The coefficients of the 2-D splines cell by cell (MultipoleView::cells) from the node values: one
    cell per thread.  Both directions take the Hermite data (value, first and second derivative in
    units of the cell width) of the two ends to the six monomial coefficients; the values are taken
    relative to one corner, as the node form does, so that c_00 alone carries the offset.  Cells of
    the upper half of the tau grid are expanded about their upper node (cellAnchor): towards either
    pole the m != 0 harmonics vanish with a power of the distance from it, which only an expansion
    about the pole's own node gives without cancellation (and gives exactly 0 on the axis). */
__global__ void cellCoefsKernel(int numSlots, int nr, int nt, const GridNode* __restrict__ gr,
    const GridNode* __restrict__ gt, const double* __restrict__ nodes, double* __restrict__ cells)
{
    const long k = blockIdx.x * static_cast<long>(blockDim.x) + threadIdx.x;
    const long perSlot = static_cast<long>(nr - 1) * (nt - 1);
    if(k >= numSlots * perSlot) return;
    const int slot = static_cast<int>(k / perSlot), rem = static_cast<int>(k % perSlot);
    const int xi = rem / (nt - 1), yi = rem % (nt - 1);
    const double hx = gr[xi + 1].x - gr[xi].x, hy = gt[yi + 1].x - gt[yi].x;
    auto hermite = [](double v0, double g0, double s0, double v1, double g1, double s1, double* c, int stride) {
        const double A = v1 - v0 - g0 - 0.5 * s0, B = g1 - g0 - s0, C = s1 - s0;
        c[0] = v0;
        c[stride] = g0;
        c[2 * stride] = 0.5 * s0;
        c[3 * stride] = 10 * A - 4 * B + 0.5 * C;
        c[4 * stride] = -15 * A + 7 * B - C;
        c[5 * stride] = 6 * A - 3 * B + 0.5 * C;
    };
    // node layout: 0 f, 1 fx, 2 fy, 3 fxx, 4 fxy, 5 fyy, 6 fxxy, 7 fxyy, 8 fxxyy
    const int val[3] = { 0, 1, 3 }, dy[3] = { 2, 4, 6 }, dyy[3] = { 5, 7, 8 };
    const double* ll = nodes + ((static_cast<size_t>(slot) * nr + xi) * nt + yi) * NODE_STRIDE;
    const double off = cellAnchor(gt[yi].x, gt[yi + 1].x) != gt[yi].x ? ll[NODE_STRIDE] : ll[0];
    double G[2][3][6];       // [x node][x derivative][power of t]
    const bool upper = cellAnchor(gt[yi].x, gt[yi + 1].x) != gt[yi].x;
    const double w = upper ? -hy : hy;      // from the anchor to the other end
    for(int a = 0; a < 2; a++) {
        const double* lo = ll + a * static_cast<size_t>(nt) * NODE_STRIDE;
        const double* up = lo + NODE_STRIDE;
        const double* base = upper ? up : lo;
        const double* other = upper ? lo : up;
        double sx = 1;
        for(int p = 0; p < 3; p++) {
            const double o = p == 0 ? off : 0;
            hermite((base[val[p]] - o) * sx, base[dy[p]] * w * sx, base[dyy[p]] * w * w * sx,
                    (other[val[p]] - o) * sx, other[dy[p]] * w * sx, other[dyy[p]] * w * w * sx, G[a][p], 1);
            if(upper)       // powers of the distance below the upper node -> powers of t in [-1, 0]
                for(int j = 1; j < 6; j += 2) G[a][p][j] = -G[a][p][j];
            sx *= hx;
        }
    }
    double* c = cells + k * CELL_COEFS;
    for(int j = 0; j < 6; j++)
        hermite(G[0][0][j], G[0][1][j], G[0][2][j], G[1][0][j], G[1][1][j], G[1][2][j], c + j, 6);
    c[0] += off;
}

/// the segments of the 2-D splines cell by cell (MultipoleView::segments): one cell per thread; the
/// defects by the operations of quinticSegmentR
__global__ void cellSegmentsKernel(int numSlots, int nr, int nt, const GridNode* __restrict__ gt,
    const double* __restrict__ nodes, double* __restrict__ segments)
{
    const long k = blockIdx.x * static_cast<long>(blockDim.x) + threadIdx.x;
    const long perSlot = static_cast<long>(nr - 1) * (nt - 1);
    if(k >= numSlots * perSlot) return;
    const int slot = static_cast<int>(k / perSlot), rem = static_cast<int>(k % perSlot);
    const int xi = rem / (nt - 1), yi = rem % (nt - 1);
    const double h = gt[yi + 1].x - gt[yi].x;
    const double* low = nodes + ((static_cast<size_t>(slot) * nr + xi) * nt + yi) * NODE_STRIDE;
    const double off = low[0];
    // node layout: 0 f, 1 fx, 2 fy, 3 fxx, 4 fxy, 5 fyy, 6 fxxy, 7 fxyy, 8 fxxyy
    const int val[3] = { 0, 1, 3 }, dy[3] = { 2, 4, 6 }, dyy[3] = { 5, 7, 8 };
    for(int p = 0; p < 3; p++)
        for(int a = 0; a < 2; a++) {
            const double* lo = low + a * static_cast<size_t>(nt) * NODE_STRIDE;
            const double* up = lo + NODE_STRIDE;
            const double o = p == 0 ? off : 0;
            const double fl = lo[val[p]] - o, fh = up[val[p]] - o;
            const double f1l = lo[dy[p]], f1h = up[dy[p]], f2l = lo[dyy[p]], f2h = up[dyy[p]];
            double* s = segments + k * CELL_COEFS + (2 * p + a) * 6;
            s[0] = p == 0 && a == 0 ? off : fl;
            s[1] = f1l;
            s[2] = f2l;
            s[3] = fma(-(0.5 * h), f1h + f1l, fh - fl);
            s[4] = fma(-(0.5 * h), f2h + f2l, f1h - f1l);
            s[5] = f2h - f2l;
        }
}
}  // namespace

void setError(const std::string& msg) { g_error = msg; }
const char* lastError() { return g_error.c_str(); }

void requireDevice()
{
    int count = 0;
    cudaError_t e = cudaGetDeviceCount(&count);
    if(e != cudaSuccess || count == 0)
        throw std::runtime_error("no CUDA device available: the B200 engine has no CPU fallback");
}

void launchEvalPotential(const MultipoleView& M, long n, const double* pos, double* phi,
    double* grad, double* hess, cudaStream_t stream, bool cylindrical, double gradSign, double hessSign)
{
    if(n <= 0) return;
    const int block = 128;
    const long grid = (n + block - 1) / block;
    const int nq = hess ? 6 : grad ? 3 : 1, kind = evalKindOf(M);
#define AGB_LAUNCH(NQ_, K_) \
    (cylindrical ? evalPotentialCylKernel<NQ_, K_><<<grid, block, 0, stream>>>(M, n, pos, phi, grad, hess) \
                 : evalPotentialKernel<NQ_, K_><<<grid, block, 0, stream>>>(M, n, pos, phi, grad, hess, gradSign, hessSign))
    if(kind == EVAL_AXI)       { if(nq == 6) AGB_LAUNCH(6, EVAL_AXI);     else if(nq == 3) AGB_LAUNCH(3, EVAL_AXI);     else AGB_LAUNCH(1, EVAL_AXI); }
    else if(kind == EVAL_FAST) { if(nq == 6) AGB_LAUNCH(6, EVAL_FAST);    else if(nq == 3) AGB_LAUNCH(3, EVAL_FAST);    else AGB_LAUNCH(1, EVAL_FAST); }
    else                       { if(nq == 6) AGB_LAUNCH(6, EVAL_GENERAL); else if(nq == 3) AGB_LAUNCH(3, EVAL_GENERAL); else AGB_LAUNCH(1, EVAL_GENERAL); }
#undef AGB_LAUNCH
    AGB_CUDA(cudaGetLastError());
}

DevicePotential* createDevicePotential(const std::vector<double>& radii,
    const std::vector<std::vector<double>>& Phi, const std::vector<std::vector<double>>& dPhi)
{
    requireDevice();
    DevicePotential* P = new DevicePotential;
    try {
        AGB_CUDA(cudaGetDevice(&P->device));
        P->host = buildMultipole(radii, Phi, dPhi);
        const MultipoleHost& H = P->host;
        P->lnr.upload(H.lnr);
        P->tau.upload(H.tau);
        // reciprocal interval widths (IEEE division on the host and on the device give the same
        // correctly rounded value, so the spline segments built from them are bit-identical)
        auto invWidths = [](const std::vector<double>& g) {
            std::vector<double> w(g.size() > 1 ? g.size() - 1 : 1, 0.0);
            for(size_t k = 0; k + 1 < g.size(); k++) w[k] = 1 / (g[k + 1] - g[k]);
            return w;
        };
        P->lnrInvH.upload(invWidths(H.lnr));
        P->tauInvH.upload(invWidths(H.tau));
        P->spl2d.upload(H.spl2d);
        P->spl2d32.upload(std::vector<float>(H.spl2d.begin(), H.spl2d.end()));
        P->spl1d.upload(H.spl1d);
        P->innerS.upload(H.inner.S); P->innerU.upload(H.inner.U); P->innerW.upload(H.inner.W);
        P->outerS.upload(H.outer.S); P->outerU.upload(H.outer.U); P->outerW.upload(H.outer.W);
        MultipoleView& V = P->view;
        V.ind = H.ind;
        V.is2d = H.is2d;
        // switching radii (reference src/potential_multipole.cpp:1538-1548, GRID_SAFETY_FACTOR = eps^(1/3))
        const double gsf = 6.0554544523933395e-06;
        V.rInnerSq = pow2(H.radii.front() * (1 + gsf));
        V.rOuterSq = pow2(H.radii.back() * (1 - gsf));
        V.nr = static_cast<int>(H.lnr.size());
        V.lnr = P->lnr.ptr;
        V.nt = static_cast<int>(H.tau.size());
        V.tau = P->tau.ptr;
        V.lnrInvH = P->lnrInvH.ptr;
        V.tauInvH = P->tauInvH.ptr;
        auto guessScale = [](const std::vector<double>& g) {
            return g.size() > 1 ? static_cast<double>(g.size() - 1) / (g.back() - g.front()) : 0.0;
        };
        V.lnrScale = guessScale(H.lnr);
        V.tauScale = guessScale(H.tau);
        for(int i = 0; i < 2 * LMAX_MAX + 1; i++) V.splSlot[i] = H.splSlot[i];
        V.spl2d = P->spl2d.ptr;
        V.spl2d32 = P->spl2d32.ptr;
        V.spl1d = P->spl1d.ptr;
        V.logScaling = H.logScaling;
        V.invPhi0 = H.invPhi0;
        V.inner.ind = H.inner.ind; V.inner.r0sq = H.inner.r0sq; V.inner.inner = 1; V.inner.Q = H.inner.Q;
        V.inner.S = P->innerS.ptr; V.inner.U = P->innerU.ptr; V.inner.W = P->innerW.ptr;
        V.outer.ind = H.outer.ind; V.outer.r0sq = H.outer.r0sq; V.outer.inner = 0; V.outer.Q = H.outer.Q;
        V.outer.S = P->outerS.ptr; V.outer.U = P->outerU.ptr; V.outer.W = P->outerW.ptr;
        std::vector<double> norm((LMAX_MAX + 1) * (LMAX_MAX + 1), 1.);
        for(int m = 0; m <= LMAX_MAX; m++)
            for(int l = m + 1; l <= LMAX_MAX; l++)
                norm[m * (LMAX_MAX + 1) + l] = sqrt((2 * l + 1.) / (2 * l - 1.) * (l - m) / (l + m));
        P->legendreNorm.upload(norm);
        V.inner.norm = V.outer.norm = P->legendreNorm.ptr;
        P->axisymmetric = (H.ind.sym & SYM_AXISYMMETRIC) == SYM_AXISYMMETRIC;
        // register-resident evaluator: m = 0 first, then ascending m
        V.nFast = 0;
        if(H.is2d && H.splSlot[H.ind.mmax] >= 0) {
            std::vector<int> ms(1, 0);
            for(int m = -H.ind.mmax; m <= H.ind.mmax; m++)
                if(m != 0 && H.splSlot[m + H.ind.mmax] >= 0) ms.push_back(m);
            if(static_cast<int>(ms.size()) <= FAST_MAX_HARMONICS) {
                V.nFast = static_cast<int>(ms.size());
                for(int s = 0; s < V.nFast; s++) { V.fastM[s] = ms[s]; V.fastSlot[s] = H.splSlot[ms[s] + H.ind.mmax]; }
            }
        }
        for(int s = V.nFast; s < FAST_MAX_HARMONICS; s++) { V.fastM[s] = 0; V.fastSlot[s] = 0; }
        if(H.is2d) {
            auto gridView = [](const std::vector<double>& g, DevBuf<GridNode>& cell, DevBuf<int>& lut) {
                std::vector<GridNode> c;
                std::vector<int> l;
                GridView v;
                makeGridTables(g, &c, &l, &v);
                cell.upload(c);
                lut.upload(l);
                v.cell = cell.ptr;
                v.lut = lut.ptr;
                return v;
            };
            if(H.lnr.size() < 2 || H.tau.size() < 2)
                throw std::invalid_argument("Multipole: the grids need at least 2 nodes");
            V.gridR = gridView(H.lnr, P->gridCellR, P->gridLutR);
            V.gridTau = gridView(H.tau, P->gridCellTau, P->gridLutTau);
            // squares of radii outside the range of normal numbers stay with the node form
            if(V.nFast > 0 && V.rInnerSq > 1e-280 && V.rOuterSq < 1e280) {
                const long count = static_cast<long>(H.numSlots) * (V.nr - 1) * (V.nt - 1);
                P->cells.alloc(count * CELL_COEFS);
                cellCoefsKernel<<<(count + 127) / 128, 128>>>(H.numSlots, V.nr, V.nt, V.gridR.cell, V.gridTau.cell,
                    V.spl2d, P->cells.ptr);
                P->segments.alloc(count * CELL_COEFS);
                cellSegmentsKernel<<<(count + 127) / 128, 128>>>(H.numSlots, V.nr, V.nt, V.gridTau.cell, V.spl2d,
                    P->segments.ptr);
                AGB_CUDA(cudaGetLastError());
                AGB_CUDA(cudaStreamSynchronize(nullptr));
            }
        } else
            V.gridR = V.gridTau = GridView{};
        V.cells = P->cells.ptr;
        V.segments = P->segments.ptr;
    } catch(...) {
        delete P;
        throw;
    }
    return P;
}

}  // namespace agb
