// Generated by cardiacfoam_gb300.cellml2cuda from src/ionicModels/AlievPanfilov/AlievPanfilov_1996.H: the right-hand
// sides of the plain FP64 form (see cellml2cuda/emit_plain.py).  Regenerate with
// `python -m cardiacfoam_gb300.cellml2cuda` instead of editing.
#pragma once
#include "alievpanfilov.cuh"

namespace cfg { namespace alievpanfilov { namespace plain {

// rhs() of the common header
template <bool SOLVE_VM, class YS, class KS>
__device__ __forceinline__ double rhs(double t, const YS& Y, const KS& K, double* dydt, int tissue, const CfgStimulus& stim)
{
    using R = double;
    (void)tissue; (void)K; (void)stim; (void)t;
    const R y_u = Y(S_u);
    const R y_recovery_r = Y(S_recovery_r);
    R a_AV_eps = (K(C_AC_epsilon) + ((K(C_AC_mu1) * y_recovery_r) / (K(C_AC_mu2) + y_u)));
    dydt[S_recovery_r] = (a_AV_eps * cfg_fma(-(K(C_AC_k) * y_u), (y_u - (K(C_AC_a) + R(1.0))), (-y_recovery_r)));
    R a_Iion_cm = cfg_fma(((K(C_AC_k) * y_u) * (y_u - K(C_AC_a))), (y_u - R(1.0)), (y_recovery_r * y_u));
    R a_Istim = (SOLVE_VM ? R(cfg_stimulus_current<double>(t, stim)) : R(0));
    if (SOLVE_VM) {
        dydt[S_u] = ((-a_Iion_cm) - a_Istim);
    }
    return a_Iion_cm;
}

// hoist() and rhs_tissue() of the common header; a slot read only as a divisor
// holds its reciprocal too
template <class KS>
__device__ __forceinline__ void hoist(double y_u, const KS& K, int tissue, CfgSlot* H)
{
    using R = double;
    (void)tissue; (void)K; (void)H; (void)y_u;
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
__device__ __forceinline__ void gate_decay(double y_u, const KS& K, const HS& H, int tissue, double* b)
{
    using R = double;
    (void)tissue; (void)K; (void)H; (void)b; (void)y_u;
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
    constexpr signed char part[NS] = {0, 1};
    return part[i];
}
// Warp of state i where four warps share a cell's step (Vm a state; split.py).
CFG_HD constexpr int part_sv(int i)
{
    constexpr signed char part[NS] = {2, 1};
    return part[i];
}

// the model's traits with these right-hand sides
struct Model : alievpanfilov::Model {
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

} } }  // namespace cfg::alievpanfilov::plain
