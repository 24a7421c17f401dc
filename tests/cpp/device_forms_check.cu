// Device check of the arithmetic and of the forms of the potential that the engine's kernels share, each
// against what it stands for:
//   quotient, reciprocal, squareRoot (multipole_force.cuh) against the correctly rounded / and sqrt,
//   rcpNormal, rsqrtNormal, NormalArithmetic (multipole_cells.cuh) in units in the last place,
//   evalForceCar and valueInterp2d (segments) against the node form inside the radial grid,
//   powerLawTerms, axisPowerLaw and powerLawAxi against evalPowerLaw beyond it.
// Operands: random exponents, and fractions that are random, short, next to 1 and next to 2.
// Usage: device_forms_check <coefficient file> ...; prints "name count maximum" lines.
#include "runtime.h"
#include "fudge_nodes.cuh"
#include <cstdio>
#include <string>

using namespace agb;

namespace {

enum { RECIPROCAL, RECIPROCAL_ONES, QUOTIENT, QUOTIENT_ONES, ROOT, RCP, RSQRT, NORMAL_QUOTIENT, NORMAL_ROOT,
       FORCE, VALUE, TERMS, AXIS, AXIS_SLOPE, BRANCH, BRANCH_SLOPE, NUM_CHECKS };
const char* const NAMES[NUM_CHECKS] = { "reciprocal", "reciprocal_ones", "quotient", "quotient_ones", "root", "rcp", "rsqrt",
    "normal_quotient", "normal_root", "force", "value", "terms", "axis", "axis_slope", "branch", "branch_slope" };

/// number of values that differ, the largest difference (times 2^10, rounded up): in units in the last place of the
/// correct value, or of 2^-52 times the scale of the forms
struct Result { unsigned long long differ, most; };

struct Random {
    unsigned long long s;
    __device__ unsigned long long next()        // splitmix64 (Steele, Lea and Flood 2014)
    {
        unsigned long long z = s += 0x9E3779B97F4A7C15ull;
        z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
        z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
        return z ^ (z >> 31);
    }
    __device__ double uniform() { return (next() >> 11) * 0x1p-53; }
    __device__ double operand(int exponents)
    {
        const unsigned long long one = 0xFFFFFFFFFFFFFull, m = next();
        const int e = static_cast<int>(next() % (2 * exponents + 1)) - exponents, kind = next() % 8;
        const unsigned long long f = kind == 0 ? m & (one << 20) & one : kind == 1 ? m % 4096 : kind == 2 ? one - m % 4096 : m & one;
        return __longlong_as_double(static_cast<long long>(static_cast<unsigned long long>(1023 + e) << 52 | f));
    }
};

__device__ void note(Result* r, int check, bool same, double difference)
{
    if(same) return;
    atomicAdd(&r[check].differ, 1ull);
    atomicMax(&r[check].most, static_cast<unsigned long long>(fmin(ceil(difference * 0x1p10), 1e18)));
}

/// got against the correctly rounded `want`, in units in the last place of `want`
__device__ void noteUlps(Result* r, int check, double got, double want)
{
    const double ulp = __longlong_as_double(__double_as_longlong(want) + 1) - want;
    note(r, check, got == want, fabs(got - want) / ulp);
}

/// the same function value relative to a scale (NaN alike is the same)
__device__ void noteScaled(Result* r, int check, double got, double want, double scale)
{
    const bool same = got == want || (got != got && want != want);
    note(r, check, same, got == got && want == want ? fabs(got - want) / scale * 0x1p52 : 1e12);
}

__global__ void arithmeticKernel(long n, int exponents, Result* r)
{
    const long i = blockIdx.x * static_cast<long>(blockDim.x) + threadIdx.x;
    if(i >= n) return;
    Random rnd{ 77 + i * 1000003ull };
    const double a = rnd.operand(exponents), b = rnd.operand(exponents);
    const bool ones = (__double_as_longlong(b) & 0xFFFFFFFFFFFFFll) == 0xFFFFFFFFFFFFFll;
    noteUlps(r, ones ? RECIPROCAL_ONES : RECIPROCAL, reciprocal(b), 1 / b);
    noteUlps(r, ones ? QUOTIENT_ONES : QUOTIENT, quotient(a, b, reciprocal(b)), a / b);
    noteUlps(r, ROOT, squareRoot(a), sqrt(a));
    noteUlps(r, RCP, rcpNormal(b), 1 / b);
    noteUlps(r, RSQRT, rsqrtNormal(a), 1 / sqrt(a));
    noteUlps(r, NORMAL_QUOTIENT, NormalArithmetic::quotient(a, b), a / b);
    noteUlps(r, NORMAL_ROOT, NormalArithmetic::root(a), sqrt(a));
}

template<int KIND>
__global__ void formsKernel(const __grid_constant__ MultipoleView M, long n, Result* r)
{
    const long i = blockIdx.x * static_cast<long>(blockDim.x) + threadIdx.x;
    if(i >= n) return;
    Random rnd{ 99 + i * 1000003ull };
    // radii from a tenth of the inner to ten times the outer one; on the axis, in the planes, next to either, and at nodes
    const double lo = log(M.rInnerSq) / 2 - 2.3, hi = log(M.rOuterSq) / 2 + 2.3;
    const int special = static_cast<int>(rnd.next() % 12);
    double rad = exp(lo + (hi - lo) * rnd.uniform()), ct = 2 * rnd.uniform() - 1;
    const double azimuth = 2 * M_PI * rnd.uniform();
    if(special == 0) ct = ct < 0 ? -1 : 1;
    if(special == 1) ct = 0;
    if(special == 2) ct *= 1e-9;
    if(special == 3) ct = ct < 0 ? -1 + 1e-12 : 1 - 1e-12;
    if(special == 4) rad = exp(M.lnr[rnd.next() % M.nr]);
    double R = rad * sqrt((1 - ct) * (1 + ct)), z = rad * ct;
    if(special == 5) R = fabs(z);
    double sa, ca;
    sincos(azimuth, &sa, &ca);
    double x = R * ca, y = R * sa;
    if(special == 6) { x = R; y = 0; }
    if(special == 7) { x = 0; y = -R; }
    const double rsq = x * x + y * y + z * z;
    double p1, g1[3], p2, g2[3], h[6];
    evalForceCar<KIND, 1, false>(M, x, y, z, &p1, g1);
    evalMultipoleCar<3, KIND>(M, x, y, z, &p2, g2, h);
    const bool inside = rsq >= M.rInnerSq * (1 + 1e-9) && rsq <= M.rOuterSq * (1 - 1e-9);
    const int check = inside ? FORCE : TERMS;
    const double scale = fabs(p2) / sqrt(rsq);
    noteScaled(r, check, p1, p2, fabs(p2));
    for(int k = 0; k < 3; k++) noteScaled(r, check, g1[k], g2[k], scale);
    if(KIND != EVAL_AXI) return;
    R = sqrt(x * x + y * y);
    const double rsq2 = R * R + z * z;
    CylDerivs g; CylHess hh;
    if(inside) {
        evalMultipoleCyl<1, KIND>(M, R, z, 0, &p2, &g, &hh);
        noteScaled(r, VALUE, valueInterp2d(M, R, z), p2, fabs(p2));
        return;
    }
    const PowerLawView& A = rsq2 < M.rInnerSq ? M.inner : M.outer;
    if(!(rsq2 < M.rInnerSq || rsq2 > M.rOuterSq)) return;
    double gR, gz, px, ppsi;
    evalPowerLaw<3>(A, R, z, 0, &p2, &g, &hh);
    noteScaled(r, AXIS, axisPowerLaw<false>(A, R, z, rsq2, nullptr, nullptr), p2, fabs(p2));
    noteScaled(r, AXIS, axisPowerLaw<true>(A, R, z, rsq2, &gR, &gz), p2, fabs(p2));
    noteScaled(r, AXIS_SLOPE, gR, g.dR, scale);
    noteScaled(r, AXIS_SLOPE, gz, g.dz, scale);
    powerLawAxi<true>(A, rsq2, R, z, &p1, &px, &ppsi);
    noteScaled(r, BRANCH, p1, p2, fabs(p2));
    noteScaled(r, BRANCH_SLOPE, px, R * g.dR + z * g.dz, fabs(p2));
    noteScaled(r, BRANCH_SLOPE, ppsi, R * g.dz - z * g.dR, fabs(p2));
}

}  // namespace

int main(int argc, char** argv)
{
    Result* r;
    if(cudaMallocManaged(&r, NUM_CHECKS * sizeof(Result)) != cudaSuccess) return 3;
    auto print = [&](const char* what) {
        if(cudaDeviceSynchronize() != cudaSuccess) { std::printf("error %s\n", cudaGetErrorString(cudaGetLastError())); std::exit(2); }
        for(int c = 0; c < NUM_CHECKS; c++) std::printf("%s %s %llu %.3g\n", what, NAMES[c], r[c].differ, r[c].most * 0x1p-10);
        for(int c = 0; c < NUM_CHECKS; c++) r[c] = Result{ 0, 0 };
    };
    for(int c = 0; c < NUM_CHECKS; c++) r[c] = Result{ 0, 0 };
    const long n = 1L << 24;
    for(int e : { 0, 2, 60, 300 }) {
        arithmeticKernel<<<n / 256, 256>>>(n, e, r);
        print(("arithmetic" + std::to_string(e)).c_str());
    }
    for(int f = 1; f < argc; f++) {
        std::vector<double> radii;
        std::vector<std::vector<double>> Phi, dPhi;
        readMultipoleCoefFile(argv[f], radii, Phi, dPhi);
        DevicePotential* p = createDevicePotential(radii, Phi, dPhi);
        const long m = 1L << 20;
        if(evalKindOf(p->view) == EVAL_AXI) formsKernel<EVAL_AXI><<<m / 128, 128>>>(p->view, m, r);
        else                                formsKernel<EVAL_FAST><<<m / 128, 128>>>(p->view, m, r);
        print(("forms" + std::to_string(f)).c_str());
        delete p;
    }
    return 0;
}
