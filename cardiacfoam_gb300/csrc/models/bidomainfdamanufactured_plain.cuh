// Generated by cardiacfoam_gb300.cellml2cuda from src/ionicModels/bidomainFDAManufactured/bidomainFDAManufactured_2014.H: the right-hand
// sides of the plain FP64 form (see cellml2cuda/emit_plain.py).  Regenerate with
// `python -m cardiacfoam_gb300.cellml2cuda` instead of editing.
#pragma once
#include "bidomainfdamanufactured.cuh"

namespace cfg { namespace bidomainfdamanufactured { namespace plain {

// rhs() of the common header
template <bool SOLVE_VM, class YS, class KS>
__device__ __forceinline__ double rhs(double t, const YS& Y, const KS& K, double* dydt, int tissue, const CfgStimulus& stim)
{
    using R = double;
    (void)tissue; (void)K; (void)stim; (void)t;
    const R y_BidomainV = Y(S_BidomainV);
    const R y_BidomainU1 = Y(S_BidomainU1);
    const R y_BidomainU2 = Y(S_BidomainU2);
    const R y_BidomainU3 = Y(S_BidomainU3);
    dydt[S_BidomainV] = R(0.0);
    dydt[S_BidomainU1] = cfg_fma(cfg_ipow<2>(((y_BidomainU1 + y_BidomainU3) - y_BidomainV)), cfg_ipow<2>(y_BidomainU2), (((R(0.5) * ((y_BidomainU1 + y_BidomainU3) - y_BidomainV)) * cfg_ipow<2>(y_BidomainU2)) * (y_BidomainV - y_BidomainU3)));
    dydt[S_BidomainU2] = ((-((y_BidomainU1 + y_BidomainU3) - y_BidomainV)) * cfg_ipow<3>(y_BidomainU2));
    dydt[S_BidomainU3] = R(0.0);
    R a_BidomainIion = cfg_fma(((((-R(0.5)) * K(C_BidomainCm)) * ((y_BidomainU1 + y_BidomainU3) - y_BidomainV)) * cfg_ipow<2>(y_BidomainU2)), (y_BidomainV - y_BidomainU3), cfg_cdiv<KS>((K(C_BidomainBeta) * (y_BidomainV - y_BidomainU3)), K(C_BidomainChi)));
    return a_BidomainIion;
}

// hoist() and rhs_tissue() of the common header; a slot read only as a divisor
// holds its reciprocal too
template <class KS>
__device__ __forceinline__ void hoist(double y_BidomainV, const KS& K, int tissue, CfgSlot* H)
{
    using R = double;
    (void)tissue; (void)K; (void)H; (void)y_BidomainV;
}
template <class YS, class KS, class HS>
__device__ __forceinline__ double rhs_tissue(const YS& Y, const KS& K, const HS& H, double* dydt, int tissue)
{
    using R = double;
    (void)H;
    return rhs<false>(0.0, Y, K, dydt, tissue, CfgStimulus{});
}
// States whose tissue-mode rate is a - b y with a and b functions of state 0 and
// constants alone (bit i = state i): b of each, and their rates alone.
constexpr unsigned long long LIN_MASK = 0x0ull;
template <class KS, class HS>
__device__ __forceinline__ void gate_decay(double y_BidomainV, const KS& K, const HS& H, int tissue, double* b)
{
    using R = double;
    (void)tissue; (void)K; (void)H; (void)b; (void)y_BidomainV;
}
template <class YS, class KS, class HS>
__device__ __forceinline__ void gate_rates(const YS& Y, const KS& K, const HS& H, int tissue, double* d)
{
    using R = double;
    (void)tissue; (void)K; (void)H; (void)d; (void)Y;
}
// Warp of state i where four warps share a cell's step (tissue mode; split.py).
CFG_HD constexpr int part_tissue(int i)
{
    constexpr signed char part[NS] = {0, 1, 2, 3};
    return part[i];
}
// Warp of state i where four warps share a cell's step (Vm a state; split.py).
CFG_HD constexpr int part_sv(int i)
{
    constexpr signed char part[NS] = {3, 1, 2, 3};
    return part[i];
}

// the model's traits with these right-hand sides
struct Model : bidomainfdamanufactured::Model {
    static constexpr unsigned long long LIN_MASK = plain::LIN_MASK;
    template <bool SV, class YS, class KS>
    __device__ static __forceinline__ double rates(double t, const YS& Y, const KS& K, double* dydt, int tissue, const CfgStimulus& st) { return plain::rhs<SV>(t, Y, K, dydt, tissue, st); }
    template <class KS>
    __device__ static __forceinline__ void hoist_vm(double v, const KS& K, int tissue, CfgSlot* H) { plain::hoist(v, K, tissue, H); }
    template <class YS, class KS, class HS>
    __device__ static __forceinline__ double rates_tissue(const YS& Y, const KS& K, const HS& H, double* dydt, int tissue) { return plain::rhs_tissue(Y, K, H, dydt, tissue); }
    template <class KS, class HS>
    __device__ static __forceinline__ void decay(double v, const KS& K, const HS& H, int tissue, double* b) { plain::gate_decay(v, K, H, tissue, b); }
    template <class YS, class KS, class HS>
    __device__ static __forceinline__ void slopes(const YS& Y, const KS& K, const HS& H, int tissue, double* d) { plain::gate_rates(Y, K, H, tissue, d); }
    CFG_HD static constexpr int part_tissue(int i) { return plain::part_tissue(i); }
    CFG_HD static constexpr int part_sv(int i) { return plain::part_sv(i); }
};

} } }  // namespace cfg::bidomainfdamanufactured::plain
