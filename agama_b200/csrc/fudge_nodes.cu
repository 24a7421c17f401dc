// Phase 1 of the Staeckel fudge from the node form of the splines (fudge_nodes.cuh), in its own
// compilation unit: its results keep their bits, which a unit shared with the cells' form would not
// guarantee.
#include "runtime.h"
#include "fudge_nodes.cuh"
#include "fudge_phases.h"

namespace agb {

namespace {

constexpr int PREPARE_BLOCK = 128;

/// one point per thread, as fudgePrepareKernel; also the focal distance used (fdOut)
template<bool FINDER>
__global__ void __launch_bounds__(PREPARE_BLOCK, 5) nodePrepareKernel(const __grid_constant__ MultipoleView M,
    const __grid_constant__ FudgeTables F, long n, const double* __restrict__ posvel, const double* __restrict__ fd,
    double fd0, FudgeRecord* __restrict__ rec, double* __restrict__ act, double* __restrict__ fdOut,
    int* __restrict__ iters, float* __restrict__ features, FudgeEnds* __restrict__ ends)
{
    const long i = blockIdx.x * static_cast<long>(blockDim.x) + threadIdx.x;
    if(i >= n) return;
    double w[6], pc[6];
    for(int c = 0; c < 6; c++) w[c] = posvel[6 * i + c];
    carToCylPosVel<true>(w, pc);
    double Phi;
    CylDerivs g; CylHess h;
    evalMultipoleCylCall<1, EVAL_AXI>(M, pc[0], pc[1], 0, &Phi, &g, &h);   // axisymmetric: no azimuth
    const double delta = FINDER ? finderFocalDistance(F, pc, Phi) : (fd ? fd[i] : fd0);
    FudgeRecord r;
    double a[3];
    FudgeEnds e;
    nodePrepare(M, pc, Phi, delta, r, a, &e);
    rec[i] = r;
    if(r.valid) ends[i] = e;
    act[3 * i + 2] = a[2];
    if(!r.valid) { act[3 * i] = a[0]; act[3 * i + 1] = a[1]; }
    if(fdOut) fdOut[i] = delta;
    if(iters) iters[i] = 0;
    if(features) bracketFeatures(pc, Phi, delta, features + 6 * i);
}

}  // namespace

void launchNodePrepare(bool finder, const MultipoleView& M, const FudgeTables& F, long n, const double* posvel,
    const double* fd, double fd0, FudgeRecord* rec, double* act, double* fdOut, int* iters, float* features,
    FudgeEnds* ends, cudaStream_t stream)
{
    if(n <= 0) return;
    (finder ? nodePrepareKernel<true> : nodePrepareKernel<false>)<<<(n + PREPARE_BLOCK - 1) / PREPARE_BLOCK, PREPARE_BLOCK,
        0, stream>>>(M, F, n, posvel, fd, fd0, rec, act, fdOut, iters, features, ends);
    AGB_CUDA(cudaGetLastError());
}

}  // namespace agb
