// sweepCurrent and trace rows of one ionic model.  Compiled once per model with
// -DCFG_MODEL=<namespace> and without FMA contraction, so that every algebraic
// rounds as the reference's computeVariables does.
#include <cuda_runtime.h>

#include "ionic_kernels.cuh"

#define CFG_STR2(x) #x
#define CFG_STR(x) CFG_STR2(x)
#define CFG_CAT3_(a, b, c) a##b##c
#define CFG_CAT3(a, b, c) CFG_CAT3_(a, b, c)
#include CFG_STR(models/CFG_MODEL.cuh)

using M = cfg::CFG_MODEL::Model;

// ---------------------------------------------------------------- sweepCurrent
// <Model>::sweepCurrent (e.g. TNNP.C:208-272): the states of one cell with
// state 0 clamped to V = vmin + (vmax - vmin) i / (npts - 1), the first
// variables function at VOI = 0, one thread per voltage.  Row i of `out` is
// [states | algebraic | rates] (2 NS + NA doubles).
// With clamp = 0 the states are taken as they are (one row: the variables
// of a cell at model time t, as a trace row of ionicModelIO::write holds).
template <bool SV>
__global__ void sweep_kernel(const double* y0, const double* C, int tissue, cfg::CfgStimulus stim,
                             double vmin, double vmax, int npts, double t, int clamp, double* out)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= npts) return;
    constexpr int NS = M::NS, NA = M::NA;
    double y[NS];
    for (int k = 0; k < NS; ++k) y[k] = y0[k];
    if (clamp) {
        const double denom = double(npts - 1);
        y[0] = vmin + (vmax - vmin) * double(i) / denom;
    }
    double A[NA > 0 ? NA : 1] = {};
    double R[NS] = {};
    const cfg::ConstView<double> K{C};
    M::template all_variables<double, SV>(t, cfg::ArrayView<double>{y}, K, A, R, tissue, stim);
    double* row = out + (long long)i * (2 * NS + NA);
    for (int k = 0; k < NS; ++k) row[k] = y[k];
    for (int k = 0; k < NA; ++k) row[NS + k] = A[k];
    for (int k = 0; k < NS; ++k) row[NS + NA + k] = R[k];
}

extern "C" cudaError_t CFG_CAT3(cfg_ionic_sweep_, CFG_MODEL, )(
    const double* y0, const double* C, int tissue, int solve_vm, const cfg::CfgStimulus& stim,
    double vmin, double vmax, int npts, double t, int clamp, double* out, cudaStream_t s)
{
    if (npts <= 0) return cudaSuccess;
    const int block = 64;
    const unsigned grid = unsigned((npts + block - 1) / block);
    if (solve_vm)
        sweep_kernel<true><<<grid, block, 0, s>>>(y0, C, tissue, stim, vmin, vmax, npts, t, clamp,
                                                  out);
    else
        sweep_kernel<false><<<grid, block, 0, s>>>(y0, C, tissue, stim, vmin, vmax, npts, t, clamp,
                                                   out);
    return cudaGetLastError();
}
