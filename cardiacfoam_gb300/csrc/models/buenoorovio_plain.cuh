// Generated by cardiacfoam_gb300.cellml2cuda from src/ionicModels/BuenoOrovio/BuenoOrovio_2008.H: the right-hand
// sides of the plain FP64 form (see cellml2cuda/emit_plain.py).  Regenerate with
// `python -m cardiacfoam_gb300.cellml2cuda` instead of editing.
#pragma once
#include "buenoorovio.cuh"

namespace cfg { namespace buenoorovio { namespace plain {

// rhs() of the common header
template <bool SOLVE_VM, class YS, class KS>
__device__ __forceinline__ double rhs(double t, const YS& Y, const KS& K, double* dydt, int tissue, const CfgStimulus& stim)
{
    using R = double;
    (void)tissue; (void)K; (void)stim; (void)t;
    const R y_u = Y(S_u);
    const R y_v = Y(S_v);
    const R y_w = Y(S_w);
    const R y_s = Y(S_s);
    R a_tauSo = (K(C_tauSo1) + cfg_cdiv<KS>(((K(C_tauSo2) - K(C_tauSo1)) * (R(1.0) + cfg_tanh((K(C_kSo) * (y_u - K(C_uSo)))))), R(2.0)));
    R a_tauO = cfg_fma((R(1.0) - (((y_u - K(C_thetaO))) > R(0) ? 1 : 0)), K(C_tauO1), ((((y_u - K(C_thetaO))) > R(0) ? 1 : 0) * K(C_tauO2)));
    R a_Jfi = cfg_cdiv<KS>(((((-y_v) * (((y_u - K(C_thetaV))) > R(0) ? 1 : 0)) * (y_u - K(C_thetaV))) * (K(C_uU) - y_u)), K(C_tauFi));
    R a_Jso = ((((y_u - K(C_uO)) * (R(1.0) - (((y_u - K(C_thetaW))) > R(0) ? 1 : 0))) / a_tauO) + ((((y_u - K(C_thetaW))) > R(0) ? 1 : 0) / a_tauSo));
    R a_Jsi = cfg_cdiv<KS>((((-(((y_u - K(C_thetaW))) > R(0) ? 1 : 0)) * y_w) * y_s), K(C_tauSi));
    R a_Jion = ((a_Jfi + a_Jso) + a_Jsi);
    R a_tauVMinus = cfg_fma((R(1.0) - (((y_u - K(C_thetaVMinus))) > R(0) ? 1 : 0)), K(C_tauV1Minus), ((((y_u - K(C_thetaVMinus))) > R(0) ? 1 : 0) * K(C_tauV2Minus)));
    R a_tauWMinus = (K(C_tauW1Minus) + cfg_cdiv<KS>(((K(C_tauW2Minus) - K(C_tauW1Minus)) * (R(1.0) + cfg_tanh((K(C_kWMinus) * (y_u - K(C_uWMinus)))))), R(2.0)));
    R a_tauS = cfg_fma((R(1.0) - (((y_u - K(C_thetaW))) > R(0) ? 1 : 0)), K(C_tauS1), ((((y_u - K(C_thetaW))) > R(0) ? 1 : 0) * K(C_tauS2)));
    R a_vInfty = (((K(C_thetaVMinus) - y_u)) > R(0) ? 1 : 0);
    R a_wInfty = cfg_fma((R(1.0) - (((y_u - K(C_thetaO))) > R(0) ? 1 : 0)), (R(1.0) - cfg_cdiv<KS>(y_u, K(C_tauWInfty))), ((((y_u - K(C_thetaO))) > R(0) ? 1 : 0) * K(C_wInftyStar)));
    dydt[S_v] = ((((R(1.0) - (((y_u - K(C_thetaV))) > R(0) ? 1 : 0)) * (a_vInfty - y_v)) / a_tauVMinus) - cfg_cdiv<KS>(((((y_u - K(C_thetaV))) > R(0) ? 1 : 0) * y_v), K(C_tauVPlus)));
    dydt[S_w] = ((((R(1.0) - (((y_u - K(C_thetaW))) > R(0) ? 1 : 0)) * (a_wInfty - y_w)) / a_tauWMinus) - cfg_cdiv<KS>(((((y_u - K(C_thetaW))) > R(0) ? 1 : 0) * y_w), K(C_tauWPlus)));
    dydt[S_s] = ((cfg_cdiv<KS>((R(1.0) + cfg_tanh((K(C_kS) * (y_u - K(C_uS))))), R(2.0)) - y_s) / a_tauS);
    R a_Istim = (SOLVE_VM ? R(cfg_stimulus_current<double>(t, stim)) : R(0));
    if (SOLVE_VM) {
        dydt[S_u] = ((-a_Jion) - a_Istim);
    }
    return a_Jion;
}

// hoist() and rhs_tissue() of the common header; a slot read only as a divisor
// holds its reciprocal too
template <class KS>
__device__ __forceinline__ void hoist(double y_u, const KS& K, int tissue, CfgSlot* H)
{
    using R = double;
    (void)tissue; (void)K; (void)H; (void)y_u;
    R a_tauSo = (K(C_tauSo1) + cfg_cdiv<KS>(((K(C_tauSo2) - K(C_tauSo1)) * (R(1.0) + cfg_tanh((K(C_kSo) * (y_u - K(C_uSo)))))), R(2.0)));
    R a_tauO = cfg_fma((R(1.0) - (((y_u - K(C_thetaO))) > R(0) ? 1 : 0)), K(C_tauO1), ((((y_u - K(C_thetaO))) > R(0) ? 1 : 0) * K(C_tauO2)));
    R a_Jso = ((((y_u - K(C_uO)) * (R(1.0) - (((y_u - K(C_thetaW))) > R(0) ? 1 : 0))) / a_tauO) + ((((y_u - K(C_thetaW))) > R(0) ? 1 : 0) / a_tauSo));
    R a_tauVMinus = cfg_fma((R(1.0) - (((y_u - K(C_thetaVMinus))) > R(0) ? 1 : 0)), K(C_tauV1Minus), ((((y_u - K(C_thetaVMinus))) > R(0) ? 1 : 0) * K(C_tauV2Minus)));
    R a_tauWMinus = (K(C_tauW1Minus) + cfg_cdiv<KS>(((K(C_tauW2Minus) - K(C_tauW1Minus)) * (R(1.0) + cfg_tanh((K(C_kWMinus) * (y_u - K(C_uWMinus)))))), R(2.0)));
    R a_tauS = cfg_fma((R(1.0) - (((y_u - K(C_thetaW))) > R(0) ? 1 : 0)), K(C_tauS1), ((((y_u - K(C_thetaW))) > R(0) ? 1 : 0) * K(C_tauS2)));
    R a_vInfty = (((K(C_thetaVMinus) - y_u)) > R(0) ? 1 : 0);
    R a_wInfty = cfg_fma((R(1.0) - (((y_u - K(C_thetaO))) > R(0) ? 1 : 0)), (R(1.0) - cfg_cdiv<KS>(y_u, K(C_tauWInfty))), ((((y_u - K(C_thetaO))) > R(0) ? 1 : 0) * K(C_wInftyStar)));
    H[H_Jso] = a_Jso;
    H[H_vInfty] = a_vInfty;
    H[H_tauVMinus] = CfgSlot::divisor(a_tauVMinus);
    H[H_wInfty] = a_wInfty;
    H[H_tauWMinus] = CfgSlot::divisor(a_tauWMinus);
    H[H_tauS] = CfgSlot::divisor(a_tauS);
    H[6] = cfg_cdiv<KS>((R(1.0) + cfg_tanh((K(C_kS) * (y_u - K(C_uS))))), R(2.0));
}
template <class YS, class KS, class HS>
__device__ __forceinline__ double rhs_tissue(const YS& Y, const KS& K, const HS& H, double* dydt, int tissue)
{
    using R = double;
    constexpr bool SOLVE_VM = false;
    constexpr double t = 0.0;
    const CfgStimulus stim{};
    (void)tissue; (void)K; (void)H; (void)t; (void)stim;
    const R y_u = Y(S_u);
    const R y_v = Y(S_v);
    const R y_w = Y(S_w);
    const R y_s = Y(S_s);
    R a_Jfi = cfg_cdiv<KS>(((((-y_v) * (((y_u - K(C_thetaV))) > R(0) ? 1 : 0)) * (y_u - K(C_thetaV))) * (K(C_uU) - y_u)), K(C_tauFi));
    R a_Jsi = cfg_cdiv<KS>((((-(((y_u - K(C_thetaW))) > R(0) ? 1 : 0)) * y_w) * y_s), K(C_tauSi));
    R a_Jion = ((a_Jfi + H(H_Jso)) + a_Jsi);
    dydt[S_v] = (cfg_hdiv(((R(1.0) - (((y_u - K(C_thetaV))) > R(0) ? 1 : 0)) * (H(H_vInfty) - y_v)), H(H_tauVMinus)) - cfg_cdiv<KS>(((((y_u - K(C_thetaV))) > R(0) ? 1 : 0) * y_v), K(C_tauVPlus)));
    dydt[S_w] = (cfg_hdiv(((R(1.0) - (((y_u - K(C_thetaW))) > R(0) ? 1 : 0)) * (H(H_wInfty) - y_w)), H(H_tauWMinus)) - cfg_cdiv<KS>(((((y_u - K(C_thetaW))) > R(0) ? 1 : 0) * y_w), K(C_tauWPlus)));
    dydt[S_s] = cfg_hdiv((H(6) - y_s), H(H_tauS));
    R a_Istim = (SOLVE_VM ? R(cfg_stimulus_current<double>(t, stim)) : R(0));
    if (SOLVE_VM) {
        dydt[S_u] = ((-a_Jion) - a_Istim);
    }
    return a_Jion;
}
// States whose tissue-mode rate is a - b y with a and b functions of state 0 and
// constants alone (bit i = state i): b of each, and their rates alone.
constexpr unsigned long long LIN_MASK = 0xeull;
template <class KS, class HS>
__device__ __forceinline__ void gate_decay(double y_u, const KS& K, const HS& H, int tissue, double* b)
{
    using R = double;
    (void)tissue; (void)K; (void)H; (void)b; (void)y_u;
    b[S_v] = (-(cfg_hdiv(((-R(1.0)) * (R(1.0) - (((y_u - K(C_thetaV))) > R(0) ? 1 : 0))), H(H_tauVMinus)) - cfg_cdiv<KS>((((y_u - K(C_thetaV))) > R(0) ? 1 : 0), K(C_tauVPlus))));
    b[S_w] = (-(cfg_hdiv(((-R(1.0)) * (R(1.0) - (((y_u - K(C_thetaW))) > R(0) ? 1 : 0))), H(H_tauWMinus)) - cfg_cdiv<KS>((((y_u - K(C_thetaW))) > R(0) ? 1 : 0), K(C_tauWPlus))));
    b[S_s] = cfg_hdiv(R(1.0), H(H_tauS));
}
template <class YS, class KS, class HS>
__device__ __forceinline__ void gate_rates(const YS& Y, const KS& K, const HS& H, int tissue, double* d)
{
    using R = double;
    (void)tissue; (void)K; (void)H; (void)d; (void)Y;
    const R y_u = Y(S_u);
    const R y_v = Y(S_v);
    const R y_w = Y(S_w);
    const R y_s = Y(S_s);
    d[S_v] = (cfg_hdiv(((R(1.0) - (((y_u - K(C_thetaV))) > R(0) ? 1 : 0)) * (H(H_vInfty) - y_v)), H(H_tauVMinus)) - cfg_cdiv<KS>(((((y_u - K(C_thetaV))) > R(0) ? 1 : 0) * y_v), K(C_tauVPlus)));
    d[S_w] = (cfg_hdiv(((R(1.0) - (((y_u - K(C_thetaW))) > R(0) ? 1 : 0)) * (H(H_wInfty) - y_w)), H(H_tauWMinus)) - cfg_cdiv<KS>(((((y_u - K(C_thetaW))) > R(0) ? 1 : 0) * y_w), K(C_tauWPlus)));
    d[S_s] = cfg_hdiv((H(6) - y_s), H(H_tauS));
}
// Warp of state i where four warps share a cell's step (tissue mode; split.py).
CFG_HD constexpr int part_tissue(int i)
{
    constexpr signed char part[NS] = {0, 3, 1, 2};
    return part[i];
}
// Warp of state i where four warps share a cell's step (Vm a state; split.py).
CFG_HD constexpr int part_sv(int i)
{
    constexpr signed char part[NS] = {1, 0, 2, 3};
    return part[i];
}

// the model's traits with these right-hand sides
struct Model : buenoorovio::Model {
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

} } }  // namespace cfg::buenoorovio::plain
