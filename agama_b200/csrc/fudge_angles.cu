// Phase 3 of the Staeckel-fudge computation when angles or frequencies are requested: the branch
// integrals of each prepared point, and from them its actions, frequencies and angles.
#include "runtime.h"
#include "fudge_nodes.cuh"
#include "fudge_phases.h"
#include <algorithm>
#include <map>
#include <mutex>

namespace agb {

namespace {

constexpr int ANGLE_BLOCK = 128;
constexpr unsigned FULL_MASK = 0xffffffffu;

/// dF/dtau at nu_max and the scaled positions of each point (AngleSetup), one point per thread
__global__ void __launch_bounds__(ANGLE_BLOCK, 4) angleSetupKernel(const __grid_constant__ MultipoleView M, long n,
    bool parts, const FudgeRecord* __restrict__ rec, AngleSetup* __restrict__ setup)
{
    const long i = blockIdx.x * static_cast<long>(blockDim.x) + threadIdx.x;
    if(i >= n || !rec[i].valid) return;
    setup[i] = fudgeAngleSetup(M, rec[i], parts);
}

/** The branch integrals (task t = branch * n + i for point i) drained from one work counter by a
    persistent grid: a lane adds one node of its integral per step and takes the next task as soon as
    its last node is added, so integrals of different orders (10 to 40 nodes) keep every lane busy and
    the batch ends evenly.  (One point per thread ran its four integrals in turn: 22 of 32 lanes active,
    and 1e5 points were 1.3 waves of blocks; 702 us.)  The nodes of an integral are added in
    order.  CELLS: the potential has cells (2-D splines): evaluated without calls. */
template<bool CELLS>
__global__ void __launch_bounds__(ANGLE_BLOCK, 4) angleIntegralKernel(const __grid_constant__ MultipoleView M,
    const __grid_constant__ GLRules gl, long n, int branches, const FudgeRecord* __restrict__ rec,
    const AngleSetup* __restrict__ setup, BranchSums* __restrict__ sums, unsigned long long* __restrict__ counter)
{
    const long total = branches * n;
    const unsigned lane = threadIdx.x & 31;
    bool busy = false, drained = false;
    long point = 0;
    int branch = 0, node = 0, numNodes = 0;
    double lo = 0, hi = 0, y = 1, nuMax = 0, dfdnuMax = 0, D2inv = 0;
    const double* x = nullptr;
    const double* w = nullptr;
    BranchSums sum{ 0, 0, 0, 0 };
    FudgeFunction fnc{};
    while(true) {
        while(true) {
            const unsigned need = __ballot_sync(FULL_MASK, !busy && !drained);
            if(!need) break;
            const int leader = __ffs(need) - 1;
            unsigned long long base = 0;
            if(static_cast<int>(lane) == leader) base = atomicAdd(counter, static_cast<unsigned long long>(__popc(need)));
            base = __shfl_sync(FULL_MASK, base, leader);
            if(!busy && !drained) {
                const long t = static_cast<long>(base) + __popc(need & ((1u << lane) - 1));
                if(t >= total) drained = true;
                else {
                    branch = t >= 2 * n ? (t >= 3 * n ? 3 : 2) : t >= n ? 1 : 0;
                    point = t - branch * n;
                    const FudgeRecord& r = rec[point];
                    if(r.valid) {
                        loadFudgeFunction(M, r, fnc);
                        const FudgeLimits lim = fudgeLimitsFinish(r);
                        const AngleSetup a = setup[point];
                        const bool lambda = branch == BRANCH_LAMBDA || branch == BRANCH_LAMBDA_PART;
                        lo = lambda ? lim.lambda_min : 0;
                        hi = lambda ? lim.lambda_max : lim.nu_max;
                        y = branch == BRANCH_LAMBDA_PART ? a.yl : branch == BRANCH_NU_PART ? a.yn : 1;
                        nuMax = lim.nu_max;
                        dfdnuMax = a.dfdnuMax;
                        D2inv = 1 / r.D2;
                        int N = lim.order < 1 ? 1 : lim.order;
                        while(gl.offset[N] < 0) N++;
                        x = gl.nodes + gl.offset[N];
                        w = gl.weights + gl.offset[N];
                        numNodes = N;
                        node = 0;
                        sum = BranchSums{ 0, 0, 0, 0 };
                        busy = y != 0;
                        if(!busy) sums[branch * n + point] = sum;
                    }
                }
            }
        }
        if(!__any_sync(FULL_MASK, busy)) break;
        if(busy) {
            addBranchNode<CELLS>(fnc, D2inv, ldg(x + node), ldg(w + node), lo, hi, y, nuMax, dfdnuMax, sum);
            if(++node == numNodes) {
                busy = false;
                sum.e *= y; sum.i3 *= y; sum.lz *= y; sum.act *= y;
                sums[branch * n + point] = sum;
            }
        }
    }
}

/// actions, frequencies and angles of each point from its branch integrals, one point per thread
__global__ void __launch_bounds__(ANGLE_BLOCK, 4) angleFinishKernel(const __grid_constant__ MultipoleView M, long n,
    const FudgeRecord* __restrict__ rec, const AngleSetup* __restrict__ setup, const BranchSums* __restrict__ sums,
    double* __restrict__ act, double* __restrict__ ang, double* __restrict__ freq)
{
    const long i = blockIdx.x * static_cast<long>(blockDim.x) + threadIdx.x;
    if(i >= n) return;
    const FudgeRecord r = rec[i];
    if(!r.valid) {          // no actions (set by phase 1): angles and frequencies are NaN too
        for(int k = 0; k < 3; k++) {
            if(ang) ang[3 * i + k] = NAN;
            if(freq) freq[3 * i + k] = NAN;
        }
        return;
    }
    BranchSums s[NUM_BRANCHES];
    for(int b = 0; b < (ang ? NUM_BRANCHES : 2); b++) s[b] = sums[b * n + i];
    double a[2];
    fudgeAnglesFrequencies(M, r, setup[i], s, a, ang ? ang + 3 * i : nullptr, freq ? freq + 3 * i : nullptr);
    act[3 * i] = a[0];
    act[3 * i + 1] = a[1];
}

/// resident blocks of the integral kernel on the current device (cached per device and variant)
template<bool CELLS>
int angleGridSize()
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
    AGB_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&perSM, angleIntegralKernel<CELLS>, ANGLE_BLOCK, 0));
    const int grid = std::max(1, sms * std::max(1, perSM));
    cache[dev] = grid;
    return grid;
}

}  // namespace

size_t angleScratchBytes(long n) { return n * (sizeof(AngleSetup) + NUM_BRANCHES * sizeof(BranchSums)); }

void launchFudgeAngles(const MultipoleView& M, const GLRules& gl, long n, const FudgeRecord* rec, double* act,
    double* ang, double* freq, void* scratch, unsigned long long* counter, cudaStream_t stream)
{
    if(n <= 0) return;
    BranchSums* sums = static_cast<BranchSums*>(scratch);
    AngleSetup* setup = reinterpret_cast<AngleSetup*>(sums + NUM_BRANCHES * n);
    const int branches = ang ? NUM_BRANCHES : 2;
    const long points = (n + ANGLE_BLOCK - 1) / ANGLE_BLOCK;
    angleSetupKernel<<<points, ANGLE_BLOCK, 0, stream>>>(M, n, ang != nullptr, rec, setup);
    AGB_CUDA(cudaGetLastError());
    AGB_CUDA(cudaMemsetAsync(counter, 0, sizeof(unsigned long long), stream));
    const bool cells = M.cells;
    const long grid = std::min<long>(cells ? angleGridSize<true>() : angleGridSize<false>(),
        (branches * n + ANGLE_BLOCK - 1) / ANGLE_BLOCK);
    (cells ? angleIntegralKernel<true> : angleIntegralKernel<false>)<<<grid, ANGLE_BLOCK, 0, stream>>>(M, gl, n, branches, rec, setup, sums, counter);
    AGB_CUDA(cudaGetLastError());
    angleFinishKernel<<<points, ANGLE_BLOCK, 0, stream>>>(M, n, rec, setup, sums, act, ang, freq);
    AGB_CUDA(cudaGetLastError());
}

}  // namespace agb
