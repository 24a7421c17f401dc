// Phase 3 of the Staeckel-fudge actions: the Gauss-Legendre action integrals.  In its own
// compilation unit so that its register budget does not constrain the other phases (what the
// kernels for potentials without cells call out of line is compiled once per unit).
#include "runtime.h"
#include "fudge.cuh"
#include "fudge_phases.h"
#include <algorithm>
#include <map>
#include <mutex>

namespace agb {

namespace {

constexpr int INTEGRAL_BLOCK = 128;
constexpr int WARPS_PER_BLOCK = INTEGRAL_BLOCK / 32;
constexpr unsigned FULL_MASK = 0xffffffffu;

/// the integrals a warp works on at a time (Jr and Jz of up to 16 points): the constants of F, the
/// interval and the rule of each, and a ring of the last nodes' terms
struct WarpIntegrals {
    double E[32], I[32], L2h[32], D2[32], mo[32], ro[32], c1[32], c2[32], lo[32], width[32];
    const double* rule[32];
    int start[32];              // index of the integral's first node among those of the warp
    double term[128];
};

/** Phase 3: the action integrals (computeActions, src/actions_staeckel.cpp:604-619: Jr = I_lambda / pi,
    Jz = 2 I_nu / pi), taken from one work counter by a persistent grid of warps.  A warp claims
    `points` consecutive points (at most 16), each lane prepares one of their integrals (Jr in the
    lower lanes, Jz in the upper ones), and then the nodes of all of them, laid end to end, are
    evaluated 32 at a time.  Neighbouring lanes are thus neighbouring nodes of one orbit and lie in
    the same one to three cells of the spline table: the L1 serves a load by the number of
    different lines its lanes touch, and with one integral per lane it was the bound (85 % of its
    rate, 25 lines per load).  The terms of an integral are added up by the lane that prepared it, in
    the order of the nodes, when its last one is done, so the result does not depend on which
    integrals share a warp.
    MIXED: the integrand's arithmetic after F(tau) in FP32 (fudgeMomentum32) and the weighted
    terms summed in FP32 with a compensation term (Kahan), converted to FP64 at the end.
    CELLS: the potential has cells.
    Bound by the latency of its FP64 chains and of the L1: 1e6 disk points at 3 / 4 / 5 / 6 / 7 / 8 blocks per
    SM 687 / 580 / 508 / 484 / 471 / 470 us, 7e5 halo points 716 / 630 / 550 / 533 / 528 / 533. */
template<bool MIXED, bool CELLS>
__global__ void __launch_bounds__(INTEGRAL_BLOCK, 7) fudgeIntegralKernel(const __grid_constant__ MultipoleView M,
    const __grid_constant__ GLRules gl, long n, int points, const FudgeRecord* __restrict__ rec,
    double* __restrict__ act, unsigned long long* __restrict__ counter)
{
    __shared__ WarpIntegrals shared[WARPS_PER_BLOCK];
    WarpIntegrals& W = shared[threadIdx.x / 32];
    const int lane = threadIdx.x & 31;
    const unsigned below = (1u << lane) - 1;
    const int which = lane >= points;
    while(true) {
        unsigned long long claimed = 0;
        if(lane == 0) claimed = atomicAdd(counter, static_cast<unsigned long long>(points));
        const long first = static_cast<long>(__shfl_sync(FULL_MASK, claimed, 0));
        if(first >= n) break;
        const long point = first + lane - which * points;
        const FudgeRecord* r = rec + point;
        const bool mine = lane < 2 * points && point < n && r->valid;
        // this lane's integral: its constants into the slot of its rank among the warp's integrals
        const unsigned all = __ballot_sync(FULL_MASK, mine);
        const int slot = __popc(all & below);
        int count = 0;
        double width = 0;
        if(mine) {
            FudgeBranch f;
            loadFudgeBranch(*r, which == 0, f);
            const FudgeLimits lim = fudgeLimitsFinish(*r);
            const double lo = which == 0 ? lim.lambda_min : 0;
            width = (which == 0 ? lim.lambda_max : lim.nu_max) - lo;
            count = lim.order < 1 ? 1 : lim.order;
            while(gl.offset[count] < 0) count++;
            W.E[slot] = f.E; W.I[slot] = f.I; W.L2h[slot] = f.L2h; W.D2[slot] = f.D2;
            W.mo[slot] = f.mo; W.ro[slot] = f.ro; W.c1[slot] = f.c1; W.c2[slot] = f.c2;
            W.lo[slot] = lo; W.width[slot] = width;
            W.rule[slot] = gl.cubic + 2 * gl.offset[count];
        }
        int end = count;
#pragma unroll
        for(int d = 1; d < 32; d *= 2) {
            const int v = __shfl_up_sync(FULL_MASK, end, d);
            if(lane >= d) end += v;
        }
        const int total = __shfl_sync(FULL_MASK, end, 31), start = end - count;
        if(mine) W.start[slot] = start;
        const unsigned lambdaSlots = __popc(all & ((1u << points) - 1));
        __syncwarp();
        for(int base = 0; base < total; base += 32) {
            // the integral of node base + lane: those begun before this chunk, and those that begin in
            // it at or before this lane
            const int before = __popc(__ballot_sync(FULL_MASK, mine && start < base));
            const unsigned begins = __reduce_or_sync(FULL_MASK, mine && start >= base && start < base + 32 ?
                1u << (start - base) : 0u);
            const int j = before + __popc(begins & (below | (1u << lane))) - 1, node = base + lane;
            if(node < total) {
                FudgeBranch f;
                f.E = W.E[j]; f.I = W.I[j]; f.L2h = W.L2h[j]; f.D2 = W.D2[j];
                f.mo = W.mo[j]; f.ro = W.ro[j]; f.c1 = W.c1[j]; f.c2 = W.c2[j];
                f.lam = j < static_cast<int>(lambdaSlots);
                const double2 g = ldg2(W.rule[j] + 2 * (node - W.start[j]));
                const double tau = fma(W.width[j], g.x, W.lo[j]);
                W.term[node & 127] = MIXED ? static_cast<double>(static_cast<float>(g.y) * fudgeMomentum32<CELLS>(M, f, tau))
                                           : g.y * fudgeMomentum<CELLS>(M, f, tau);
            }
            __syncwarp();
            if(mine && end > base && end <= base + 32) {        // (at most 40 + 32 nodes back: in the ring)
                double sum = 0;
                if(MIXED) {
                    float sum32 = 0.f, comp32 = 0.f;
                    for(int k = start; k < end; k++) {
                        const float y = static_cast<float>(W.term[k & 127]) - comp32, t = sum32 + y;
                        comp32 = (t - sum32) - y;
                        sum32 = t;
                    }
                    sum = static_cast<double>(sum32) - static_cast<double>(comp32);
                } else
                    for(int k = start; k < end; k++) sum += W.term[k & 127];
                sum *= width;
                act[3 * point + which] = which == 0 ? sum / M_PI : sum / M_PI * 2;
            }
            __syncwarp();
        }
    }
}

/// resident blocks of the integral kernel on the current device (cached per device and variant)
template<bool MIXED, bool CELLS>
int integralGridSize()
{
    static std::mutex mutex;
    static std::map<int, int> cache;
    int dev;
    AGB_CUDA(cudaGetDevice(&dev));
    std::lock_guard<std::mutex> lock(mutex);
    auto it = cache.find(dev);
    if(it != cache.end()) return it->second;
    int sms = 0, perSM = 0;
    AGB_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
    AGB_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&perSM, fudgeIntegralKernel<MIXED, CELLS>, INTEGRAL_BLOCK, 0));
    const int grid = std::max(1, sms * std::max(1, perSM));
    cache[dev] = grid;
    return grid;
}

}  // namespace

namespace {
template<bool MIXED, bool CELLS>
void launchIntegrals(const MultipoleView& M, const GLRules& gl, long n, const FudgeRecord* rec, double* act,
    unsigned long long* counter, cudaStream_t stream)
{
    const long resident = integralGridSize<MIXED, CELLS>();
    // 16 points a claim, fewer where that would leave warps without any
    int points = 16;
    while(points > 1 && n < points * resident * WARPS_PER_BLOCK) points /= 2;
    const long claims = (n + points - 1) / points;
    const long grid = std::min(resident, (claims + WARPS_PER_BLOCK - 1) / WARPS_PER_BLOCK);
    fudgeIntegralKernel<MIXED, CELLS><<<grid, INTEGRAL_BLOCK, 0, stream>>>(M, gl, n, points, rec, act, counter);
    AGB_CUDA(cudaGetLastError());
}
}  // namespace

void launchFudgeIntegrals(const MultipoleView& M, const GLRules& gl, long n, const FudgeRecord* rec, double* act,
    unsigned long long* counter, bool mixed, cudaStream_t stream)
{
    if(n <= 0) return;
    AGB_CUDA(cudaMemsetAsync(counter, 0, sizeof(unsigned long long), stream));
    auto launch = M.cells ? (mixed ? launchIntegrals<true, true> : launchIntegrals<false, true>)
                          : (mixed ? launchIntegrals<true, false> : launchIntegrals<false, false>);
    launch(M, gl, n, rec, act, counter, stream);
}

}  // namespace agb
