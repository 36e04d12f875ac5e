// Generated by cardiacfoam_gb300.cellml2cuda from src/ionicModels/TNNP/TNNP_2004.H: the right-hand
// sides of the plain FP64 form (see cellml2cuda/emit_plain.py).  Regenerate with
// `python -m cardiacfoam_gb300.cellml2cuda` instead of editing.
#pragma once
#include "tnnp.cuh"

namespace cfg { namespace tnnp { namespace plain {

// rhs() of the common header
template <bool SOLVE_VM, class YS, class KS>
__device__ __forceinline__ double rhs(double t, const YS& Y, const KS& K, double* dydt, int tissue, const CfgStimulus& stim)
{
    using R = double;
    (void)tissue; (void)K; (void)stim; (void)t;
    const R y_V = Y(S_V);
    const R y_K_i = Y(S_K_i);
    const R y_Na_i = Y(S_Na_i);
    const R y_Ca_i = Y(S_Ca_i);
    const R y_Xr1 = Y(S_Xr1);
    const R y_Xr2 = Y(S_Xr2);
    const R y_Xs = Y(S_Xs);
    const R y_m = Y(S_m);
    const R y_h = Y(S_h);
    const R y_j = Y(S_j);
    const R y_d = Y(S_d);
    const R y_f = Y(S_f);
    const R y_fCa = Y(S_fCa);
    const R y_s = Y(S_s);
    const R y_r = Y(S_r);
    const R y_Ca_SR = Y(S_Ca_SR);
    const R y_g = Y(S_g);
    R a_m_inf = (R(1.00000) / cfg_ipow<2>((R(1.00000) + cfg_exp(cfg_cdiv<KS>(((-R(56.8600)) - y_V), R(9.03000))))));
    R a_alpha_m = (R(1.00000) / (R(1.00000) + cfg_exp(cfg_cdiv<KS>(((-R(60.0000)) - y_V), R(5.00000)))));
    R a_beta_m = ((R(0.100000) / (R(1.00000) + cfg_exp(cfg_cdiv<KS>((y_V + R(35.0000)), R(5.00000))))) + (R(0.100000) / (R(1.00000) + cfg_exp(cfg_cdiv<KS>((y_V - R(50.0000)), R(200.000))))));
    R a_tau_m = ((R(1.00000) * a_alpha_m) * a_beta_m);
    dydt[S_m] = ((a_m_inf - y_m) / a_tau_m);
    R a_h_inf = (R(1.00000) / cfg_ipow<2>((R(1.00000) + cfg_exp(cfg_cdiv<KS>((y_V + R(71.5500)), R(7.43000))))));
    R a_alpha_h = ((y_V < (-R(40.0000))) ? (R(0.0570000) * cfg_exp(cfg_cdiv<KS>((-(y_V + R(80.0000))), R(6.80000)))) : R(0.00000));
    R a_beta_h = ((y_V < (-R(40.0000))) ? cfg_fma(R(2.70000), cfg_exp((R(0.0790000) * y_V)), (R(310000.) * cfg_exp((R(0.348500) * y_V)))) : (R(0.770000) / (R(0.130000) * (R(1.00000) + cfg_exp(cfg_cdiv<KS>((y_V + R(10.6600)), (-R(11.1000))))))));
    R a_tau_h = (R(1.00000) / (a_alpha_h + a_beta_h));
    dydt[S_h] = ((a_h_inf - y_h) / a_tau_h);
    R a_j_inf = (R(1.00000) / cfg_ipow<2>((R(1.00000) + cfg_exp(cfg_cdiv<KS>((y_V + R(71.5500)), R(7.43000))))));
    R a_alpha_j = ((y_V < (-R(40.0000))) ? (cfg_cdiv<KS>((cfg_fma((-R(25428.0)), cfg_exp((R(0.244400) * y_V)), -(R(6.94800e-06) * cfg_exp(((-R(0.0439100)) * y_V)))) * (y_V + R(37.7800))), R(1.00000)) / (R(1.00000) + cfg_exp((R(0.311000) * (y_V + R(79.2300)))))) : R(0.00000));
    R a_beta_j = ((y_V < (-R(40.0000))) ? ((R(0.0242400) * cfg_exp(((-R(0.0105200)) * y_V))) / (R(1.00000) + cfg_exp(((-R(0.137800)) * (y_V + R(40.1400)))))) : ((R(0.600000) * cfg_exp((R(0.0570000) * y_V))) / (R(1.00000) + cfg_exp(((-R(0.100000)) * (y_V + R(32.0000)))))));
    R a_tau_j = (R(1.00000) / (a_alpha_j + a_beta_j));
    dydt[S_j] = ((a_j_inf - y_j) / a_tau_j);
    R a_d_inf = (R(1.00000) / (R(1.00000) + cfg_exp(cfg_cdiv<KS>(((-R(5.00000)) - y_V), R(7.50000)))));
    R a_alpha_d = ((R(1.40000) / (R(1.00000) + cfg_exp(cfg_cdiv<KS>(((-R(35.0000)) - y_V), R(13.0000))))) + R(0.250000));
    R a_gama_fCa = (R(1.40000) / (R(1.00000) + cfg_exp(cfg_cdiv<KS>((y_V + R(5.00000)), R(5.00000)))));
    R a_gamma_d = (R(1.00000) / (R(1.00000) + cfg_exp(cfg_cdiv<KS>((R(50.0000) - y_V), R(20.0000)))));
    R a_tau_d = cfg_fma((R(1.00000) * a_alpha_d), a_gama_fCa, a_gamma_d);
    dydt[S_d] = ((a_d_inf - y_d) / a_tau_d);
    R a_f_inf = (R(1.00000) / (R(1.00000) + cfg_exp(cfg_cdiv<KS>((y_V + R(20.0000)), R(7.00000)))));
    R a_tau_f = (cfg_fma(R(1125.00), cfg_exp(cfg_cdiv<KS>((-cfg_ipow<2>((y_V + R(27.0000)))), R(240.000))), R(80.0000)) + (R(165.000) / (R(1.00000) + cfg_exp(cfg_cdiv<KS>((R(25.0000) - y_V), R(10.0000))))));
    dydt[S_f] = ((a_f_inf - y_f) / a_tau_f);
    R a_alpha_fCa = (R(1.00000) / (R(1.00000) + cfg_ipow<8>(cfg_cdiv<KS>(y_Ca_i, R(0.000325000)))));
    R a_beta_fCa = (R(0.100000) / (R(1.00000) + cfg_exp(cfg_cdiv<KS>((y_Ca_i - R(0.000500000)), R(0.000100000)))));
    R a_beta_d = (R(0.200000) / (R(1.00000) + cfg_exp(cfg_cdiv<KS>((y_Ca_i - R(0.000750000)), R(0.000800000)))));
    R a_fCa_inf = cfg_cdiv<KS>((((a_alpha_fCa + a_beta_fCa) + a_beta_d) + R(0.230000)), R(1.46000));
    R a_d_fCa = cfg_cdiv<KS>((a_fCa_inf - y_fCa), K(C_tau_fCa));
    dydt[S_fCa] = (((a_fCa_inf > y_fCa) && (y_V > (-R(60.0000)))) ? R(0.00000) : a_d_fCa);
    R a_s_inf = ((tissue == 1) ? (R(1.00000) / (R(1.00000) + cfg_exp(cfg_cdiv<KS>((y_V + R(20.0000)), R(5.00000))))) : (R(1.10000) / (R(1.00000) + cfg_exp(cfg_cdiv<KS>((y_V + R(28.0000)), R(6.00000))))));
    R a_tau_s = ((tissue == 1) ? (cfg_fma(R(85.0000), cfg_exp(cfg_cdiv<KS>((-cfg_ipow<2>((y_V + R(45.0000)))), R(320.000))), (R(5.00000) / (R(1.00000) + cfg_exp(cfg_cdiv<KS>((y_V - R(20.0000)), R(5.00000)))))) + R(3.00000)) : cfg_fma(R(1000.0000), cfg_exp(cfg_cdiv<KS>((-cfg_ipow<2>((y_V + R(67.0000)))), R(1000.000))), R(8.00000)));
    dydt[S_s] = ((a_s_inf - y_s) / a_tau_s);
    R a_r_inf = (R(1.00000) / (R(1.00000) + cfg_exp(cfg_cdiv<KS>((R(20.0000) - y_V), R(6.00000)))));
    R a_tau_r = cfg_fma(R(9.50000), cfg_exp(cfg_cdiv<KS>((-cfg_ipow<2>((y_V + R(40.0000)))), R(1800.00))), R(0.800000));
    dydt[S_r] = ((a_r_inf - y_r) / a_tau_r);
    R a_xr1_inf = (R(1.00000) / (R(1.00000) + cfg_exp(cfg_cdiv<KS>(((-R(26.0000)) - y_V), R(7.00000)))));
    R a_alpha_xr1 = (R(450.000) / (R(1.00000) + cfg_exp(cfg_cdiv<KS>(((-R(45.0000)) - y_V), R(10.0000)))));
    R a_beta_xr1 = (R(6.00000) / (R(1.00000) + cfg_exp(cfg_cdiv<KS>((y_V + R(30.0000)), R(11.5000)))));
    R a_tau_xr1 = ((R(1.00000) * a_alpha_xr1) * a_beta_xr1);
    dydt[S_Xr1] = ((a_xr1_inf - y_Xr1) / a_tau_xr1);
    R a_xr2_inf = (R(1.00000) / (R(1.00000) + cfg_exp(cfg_cdiv<KS>((y_V + R(88.0000)), R(24.0000)))));
    R a_alpha_xr2 = (R(3.00000) / (R(1.00000) + cfg_exp(cfg_cdiv<KS>(((-R(60.0000)) - y_V), R(20.0000)))));
    R a_beta_xr2 = (R(1.12000) / (R(1.00000) + cfg_exp(cfg_cdiv<KS>((y_V - R(60.0000)), R(20.0000)))));
    R a_tau_xr2 = ((R(1.00000) * a_alpha_xr2) * a_beta_xr2);
    dydt[S_Xr2] = ((a_xr2_inf - y_Xr2) / a_tau_xr2);
    R a_xs_inf = (R(1.00000) / (R(1.00000) + cfg_exp(cfg_cdiv<KS>(((-R(5.00000)) - y_V), R(14.0000)))));
    R a_alpha_xs = (R(1100.00) / cfg_sqrt((R(1.00000) + cfg_exp(cfg_cdiv<KS>(((-R(10.0000)) - y_V), R(6.00000))))));
    R a_beta_xs = (R(1.00000) / (R(1.00000) + cfg_exp(cfg_cdiv<KS>((y_V - R(60.0000)), R(20.0000)))));
    R a_tau_xs = ((R(1.00000) * a_alpha_xs) * a_beta_xs);
    dydt[S_Xs] = ((a_xs_inf - y_Xs) / a_tau_xs);
    R a_g_inf = ((y_Ca_i < R(0.000350000)) ? (R(1.00000) / (R(1.00000) + cfg_ipow<6>(cfg_cdiv<KS>(y_Ca_i, R(0.000350000))))) : (R(1.00000) / (R(1.00000) + cfg_ipow<16>(cfg_cdiv<KS>(y_Ca_i, R(0.000350000))))));
    R a_d_g = cfg_cdiv<KS>((a_g_inf - y_g), K(C_tau_g));
    dydt[S_g] = (((a_g_inf > y_g) && (y_V > (-R(60.0000)))) ? R(0.00000) : a_d_g);
    R a_i_NaK = (((((K(C_P_NaK) * K(C_K_o)) / (K(C_K_o) + K(C_K_mk))) * y_Na_i) / (y_Na_i + K(C_K_mNa))) / cfg_fma(R(0.0353000), cfg_exp(cfg_cdiv<KS>(((-y_V) * K(C_F)), (K(C_R) * K(C_T)))), cfg_fma(R(0.124500), cfg_exp(cfg_cdiv<KS>((((-R(0.100000)) * y_V) * K(C_F)), (K(C_R) * K(C_T)))), R(1.00000))));
    R a_E_Na = (((K(C_R) * K(C_T)) / K(C_F)) * cfg_log((K(C_Na_o) / y_Na_i)));
    R a_i_Na = ((((K(C_g_Na) * cfg_ipow<3>(y_m)) * y_h) * y_j) * (y_V - a_E_Na));
    R a_i_b_Na = (K(C_g_bNa) * (y_V - a_E_Na));
    R a_i_NaCa = ((K(C_K_NaCa) * cfg_fma((cfg_exp(cfg_cdiv<KS>(((K(C_gamma_NCX) * y_V) * K(C_F)), (K(C_R) * K(C_T)))) * cfg_ipow<3>(y_Na_i)), K(C_Ca_o), -(((cfg_exp(cfg_cdiv<KS>((((K(C_gamma_NCX) - R(1.00000)) * y_V) * K(C_F)), (K(C_R) * K(C_T)))) * cfg_ipow<3>(K(C_Na_o))) * y_Ca_i) * K(C_alpha_NCX)))) / (((cfg_ipow<3>(K(C_Km_Nai)) + cfg_ipow<3>(K(C_Na_o))) * (K(C_Km_Ca) + K(C_Ca_o))) * cfg_fma(K(C_K_sat), cfg_exp(cfg_cdiv<KS>((((K(C_gamma_NCX) - R(1.00000)) * y_V) * K(C_F)), (K(C_R) * K(C_T)))), R(1.00000))));
    dydt[S_Na_i] = cfg_cdiv<KS>(((-cfg_fma(R(3.00000), a_i_NaCa, cfg_fma(R(3.00000), a_i_NaK, (a_i_Na + a_i_b_Na)))) * K(C_Cm)), (K(C_V_c) * K(C_F)));
    R a_E_K = (((K(C_R) * K(C_T)) / K(C_F)) * cfg_log((K(C_K_o) / y_K_i)));
    R a_alpha_K1 = (R(0.100000) / (R(1.00000) + cfg_exp((R(0.0600000) * ((y_V - a_E_K) - R(200.000))))));
    R a_beta_K1 = (cfg_fma(R(3.00000), cfg_exp((R(0.000200000) * ((y_V - a_E_K) + R(100.000)))), (R(1.00000) * cfg_exp((R(0.100000) * ((y_V - a_E_K) - R(10.0000)))))) / (R(1.00000) + cfg_exp(((-R(0.500000)) * (y_V - a_E_K)))));
    R a_xK1_inf = (a_alpha_K1 / (a_alpha_K1 + a_beta_K1));
    R a_i_K1 = (((K(C_g_K1) * a_xK1_inf) * cfg_sqrt((K(C_K_o) / R(5.40000)))) * (y_V - a_E_K));
    R a_i_to = (((K(C_g_to) * y_r) * y_s) * (y_V - a_E_K));
    R a_i_Kr = ((((K(C_g_Kr) * cfg_sqrt((K(C_K_o) / R(5.40000)))) * y_Xr1) * y_Xr2) * (y_V - a_E_K));
    R a_E_Ks = (((K(C_R) * K(C_T)) / K(C_F)) * cfg_log(((K(C_K_o) + (K(C_P_kna) * K(C_Na_o))) / cfg_fma(K(C_P_kna), y_Na_i, y_K_i))));
    R a_i_Ks = ((K(C_g_Ks) * cfg_ipow<2>(y_Xs)) * (y_V - a_E_Ks));
    R a_i_CaL = ((cfg_cdiv<KS>(((((((K(C_g_CaL) * y_d) * y_f) * y_fCa) * R(4.00000)) * y_V) * cfg_ipow<2>(K(C_F))), (K(C_R) * K(C_T))) * cfg_fma(y_Ca_i, cfg_exp(cfg_cdiv<KS>(((R(2.00000) * y_V) * K(C_F)), (K(C_R) * K(C_T)))), -(R(0.341000) * K(C_Ca_o)))) / cfg_expm1(cfg_cdiv<KS>(((R(2.00000) * y_V) * K(C_F)), (K(C_R) * K(C_T)))));
    R a_E_Ca = ((((R(0.500000) * K(C_R)) * K(C_T)) / K(C_F)) * cfg_log((K(C_Ca_o) / y_Ca_i)));
    R a_i_b_Ca = (K(C_g_bCa) * (y_V - a_E_Ca));
    R a_i_p_K = ((K(C_g_pK) * (y_V - a_E_K)) / (R(1.00000) + cfg_exp(cfg_cdiv<KS>((R(25.0000) - y_V), R(5.98000)))));
    R a_i_p_Ca = ((K(C_g_pCa) * y_Ca_i) / (y_Ca_i + K(C_K_pCa)));
    R a_Iion_cm = (((((((((((a_i_K1 + a_i_to) + a_i_Kr) + a_i_Ks) + a_i_CaL) + a_i_NaK) + a_i_Na) + a_i_b_Na) + a_i_NaCa) + a_i_b_Ca) + a_i_p_K) + a_i_p_Ca);
    R a_Istim = (SOLVE_VM ? R(cfg_stimulus_current<double>(t, stim)) : R(0));
    dydt[S_V] = R(0.0);
    if (SOLVE_VM) {
        dydt[S_V] = ((-a_Iion_cm) - a_Istim);
    }
    dydt[S_K_i] = cfg_cdiv<KS>(((-cfg_fma(-R(2.00000), a_i_NaK, (((((a_i_K1 + a_i_to) + a_i_Kr) + a_i_Ks) + a_i_p_K) + a_Istim))) * K(C_Cm)), (K(C_V_c) * K(C_F)));
    R a_i_rel = (((((K(C_a_rel) * cfg_ipow<2>(y_Ca_SR)) / (cfg_ipow<2>(K(C_b_rel)) + cfg_ipow<2>(y_Ca_SR))) + K(C_c_rel)) * y_d) * y_g);
    R a_i_up = (K(C_Vmax_up) / (R(1.00000) + (cfg_ipow<2>(K(C_K_up)) / cfg_ipow<2>(y_Ca_i))));
    R a_i_leak = (K(C_V_leak) * (y_Ca_SR - y_Ca_i));
    R a_ddt_Ca_i_total = ((cfg_fma(cfg_cdiv<KS>((-cfg_fma(-R(2.00000), a_i_NaCa, ((a_i_CaL + a_i_b_Ca) + a_i_p_Ca))), ((R(2.00000) * K(C_V_c)) * K(C_F))), K(C_Cm), a_i_leak) - a_i_up) + a_i_rel);
    R a_f_JCa_i_free = (R(1.00000) / (R(1.00000) + ((K(C_Buf_c) * K(C_K_buf_c)) / cfg_ipow<2>((y_Ca_i + K(C_K_buf_c))))));
    dydt[S_Ca_i] = (a_ddt_Ca_i_total * a_f_JCa_i_free);
    R a_ddt_Ca_sr_total = ((K(C_V_c) / K(C_V_sr)) * (a_i_up - (a_i_rel + a_i_leak)));
    R a_f_JCa_sr_free = (R(1.00000) / (R(1.00000) + ((K(C_Buf_sr) * K(C_K_buf_sr)) / cfg_ipow<2>((y_Ca_SR + K(C_K_buf_sr))))));
    dydt[S_Ca_SR] = (a_ddt_Ca_sr_total * a_f_JCa_sr_free);
    return a_Iion_cm;
}

// hoist() and rhs_tissue() of the common header; a slot read only as a divisor
// holds its reciprocal too
template <class KS>
__device__ __forceinline__ void hoist(double y_V, const KS& K, int tissue, CfgSlot* H)
{
    using R = double;
    (void)tissue; (void)K; (void)H; (void)y_V;
    R a_m_inf = (R(1.00000) / cfg_ipow<2>((R(1.00000) + cfg_exp(cfg_cdiv<KS>(((-R(56.8600)) - y_V), R(9.03000))))));
    R a_alpha_m = (R(1.00000) / (R(1.00000) + cfg_exp(cfg_cdiv<KS>(((-R(60.0000)) - y_V), R(5.00000)))));
    R a_beta_m = ((R(0.100000) / (R(1.00000) + cfg_exp(cfg_cdiv<KS>((y_V + R(35.0000)), R(5.00000))))) + (R(0.100000) / (R(1.00000) + cfg_exp(cfg_cdiv<KS>((y_V - R(50.0000)), R(200.000))))));
    R a_tau_m = ((R(1.00000) * a_alpha_m) * a_beta_m);
    R a_h_inf = (R(1.00000) / cfg_ipow<2>((R(1.00000) + cfg_exp(cfg_cdiv<KS>((y_V + R(71.5500)), R(7.43000))))));
    R a_alpha_h = ((y_V < (-R(40.0000))) ? (R(0.0570000) * cfg_exp(cfg_cdiv<KS>((-(y_V + R(80.0000))), R(6.80000)))) : R(0.00000));
    R a_beta_h = ((y_V < (-R(40.0000))) ? cfg_fma(R(2.70000), cfg_exp((R(0.0790000) * y_V)), (R(310000.) * cfg_exp((R(0.348500) * y_V)))) : (R(0.770000) / (R(0.130000) * (R(1.00000) + cfg_exp(cfg_cdiv<KS>((y_V + R(10.6600)), (-R(11.1000))))))));
    R a_tau_h = (R(1.00000) / (a_alpha_h + a_beta_h));
    R a_j_inf = (R(1.00000) / cfg_ipow<2>((R(1.00000) + cfg_exp(cfg_cdiv<KS>((y_V + R(71.5500)), R(7.43000))))));
    R a_alpha_j = ((y_V < (-R(40.0000))) ? (cfg_cdiv<KS>((cfg_fma((-R(25428.0)), cfg_exp((R(0.244400) * y_V)), -(R(6.94800e-06) * cfg_exp(((-R(0.0439100)) * y_V)))) * (y_V + R(37.7800))), R(1.00000)) / (R(1.00000) + cfg_exp((R(0.311000) * (y_V + R(79.2300)))))) : R(0.00000));
    R a_beta_j = ((y_V < (-R(40.0000))) ? ((R(0.0242400) * cfg_exp(((-R(0.0105200)) * y_V))) / (R(1.00000) + cfg_exp(((-R(0.137800)) * (y_V + R(40.1400)))))) : ((R(0.600000) * cfg_exp((R(0.0570000) * y_V))) / (R(1.00000) + cfg_exp(((-R(0.100000)) * (y_V + R(32.0000)))))));
    R a_tau_j = (R(1.00000) / (a_alpha_j + a_beta_j));
    R a_d_inf = (R(1.00000) / (R(1.00000) + cfg_exp(cfg_cdiv<KS>(((-R(5.00000)) - y_V), R(7.50000)))));
    R a_alpha_d = ((R(1.40000) / (R(1.00000) + cfg_exp(cfg_cdiv<KS>(((-R(35.0000)) - y_V), R(13.0000))))) + R(0.250000));
    R a_gama_fCa = (R(1.40000) / (R(1.00000) + cfg_exp(cfg_cdiv<KS>((y_V + R(5.00000)), R(5.00000)))));
    R a_gamma_d = (R(1.00000) / (R(1.00000) + cfg_exp(cfg_cdiv<KS>((R(50.0000) - y_V), R(20.0000)))));
    R a_tau_d = cfg_fma((R(1.00000) * a_alpha_d), a_gama_fCa, a_gamma_d);
    R a_f_inf = (R(1.00000) / (R(1.00000) + cfg_exp(cfg_cdiv<KS>((y_V + R(20.0000)), R(7.00000)))));
    R a_tau_f = (cfg_fma(R(1125.00), cfg_exp(cfg_cdiv<KS>((-cfg_ipow<2>((y_V + R(27.0000)))), R(240.000))), R(80.0000)) + (R(165.000) / (R(1.00000) + cfg_exp(cfg_cdiv<KS>((R(25.0000) - y_V), R(10.0000))))));
    R a_s_inf = ((tissue == 1) ? (R(1.00000) / (R(1.00000) + cfg_exp(cfg_cdiv<KS>((y_V + R(20.0000)), R(5.00000))))) : (R(1.10000) / (R(1.00000) + cfg_exp(cfg_cdiv<KS>((y_V + R(28.0000)), R(6.00000))))));
    R a_tau_s = ((tissue == 1) ? (cfg_fma(R(85.0000), cfg_exp(cfg_cdiv<KS>((-cfg_ipow<2>((y_V + R(45.0000)))), R(320.000))), (R(5.00000) / (R(1.00000) + cfg_exp(cfg_cdiv<KS>((y_V - R(20.0000)), R(5.00000)))))) + R(3.00000)) : cfg_fma(R(1000.0000), cfg_exp(cfg_cdiv<KS>((-cfg_ipow<2>((y_V + R(67.0000)))), R(1000.000))), R(8.00000)));
    R a_r_inf = (R(1.00000) / (R(1.00000) + cfg_exp(cfg_cdiv<KS>((R(20.0000) - y_V), R(6.00000)))));
    R a_tau_r = cfg_fma(R(9.50000), cfg_exp(cfg_cdiv<KS>((-cfg_ipow<2>((y_V + R(40.0000)))), R(1800.00))), R(0.800000));
    R a_xr1_inf = (R(1.00000) / (R(1.00000) + cfg_exp(cfg_cdiv<KS>(((-R(26.0000)) - y_V), R(7.00000)))));
    R a_alpha_xr1 = (R(450.000) / (R(1.00000) + cfg_exp(cfg_cdiv<KS>(((-R(45.0000)) - y_V), R(10.0000)))));
    R a_beta_xr1 = (R(6.00000) / (R(1.00000) + cfg_exp(cfg_cdiv<KS>((y_V + R(30.0000)), R(11.5000)))));
    R a_tau_xr1 = ((R(1.00000) * a_alpha_xr1) * a_beta_xr1);
    R a_xr2_inf = (R(1.00000) / (R(1.00000) + cfg_exp(cfg_cdiv<KS>((y_V + R(88.0000)), R(24.0000)))));
    R a_alpha_xr2 = (R(3.00000) / (R(1.00000) + cfg_exp(cfg_cdiv<KS>(((-R(60.0000)) - y_V), R(20.0000)))));
    R a_beta_xr2 = (R(1.12000) / (R(1.00000) + cfg_exp(cfg_cdiv<KS>((y_V - R(60.0000)), R(20.0000)))));
    R a_tau_xr2 = ((R(1.00000) * a_alpha_xr2) * a_beta_xr2);
    R a_xs_inf = (R(1.00000) / (R(1.00000) + cfg_exp(cfg_cdiv<KS>(((-R(5.00000)) - y_V), R(14.0000)))));
    R a_alpha_xs = (R(1100.00) / cfg_sqrt((R(1.00000) + cfg_exp(cfg_cdiv<KS>(((-R(10.0000)) - y_V), R(6.00000))))));
    R a_beta_xs = (R(1.00000) / (R(1.00000) + cfg_exp(cfg_cdiv<KS>((y_V - R(60.0000)), R(20.0000)))));
    R a_tau_xs = ((R(1.00000) * a_alpha_xs) * a_beta_xs);
    H[H_m_inf] = a_m_inf;
    H[H_tau_m] = CfgSlot::divisor(a_tau_m);
    H[H_h_inf] = a_h_inf;
    H[H_tau_h] = CfgSlot::divisor(a_tau_h);
    H[H_j_inf] = a_j_inf;
    H[H_tau_j] = CfgSlot::divisor(a_tau_j);
    H[H_d_inf] = a_d_inf;
    H[H_tau_d] = CfgSlot::divisor(a_tau_d);
    H[H_f_inf] = a_f_inf;
    H[H_tau_f] = CfgSlot::divisor(a_tau_f);
    H[H_s_inf] = a_s_inf;
    H[H_tau_s] = CfgSlot::divisor(a_tau_s);
    H[H_r_inf] = a_r_inf;
    H[H_tau_r] = CfgSlot::divisor(a_tau_r);
    H[H_xr1_inf] = a_xr1_inf;
    H[H_tau_xr1] = CfgSlot::divisor(a_tau_xr1);
    H[H_xr2_inf] = a_xr2_inf;
    H[H_tau_xr2] = CfgSlot::divisor(a_tau_xr2);
    H[H_xs_inf] = a_xs_inf;
    H[H_tau_xs] = CfgSlot::divisor(a_tau_xs);
    H[20] = CfgSlot::divisor(cfg_fma(R(0.0353000), cfg_exp(cfg_cdiv<KS>(((-y_V) * K(C_F)), (K(C_R) * K(C_T)))), cfg_fma(R(0.124500), cfg_exp(cfg_cdiv<KS>((((-R(0.100000)) * y_V) * K(C_F)), (K(C_R) * K(C_T)))), R(1.00000))));
    H[21] = CfgSlot::divisor((((cfg_ipow<3>(K(C_Km_Nai)) + cfg_ipow<3>(K(C_Na_o))) * (K(C_Km_Ca) + K(C_Ca_o))) * cfg_fma(K(C_K_sat), cfg_exp(cfg_cdiv<KS>((((K(C_gamma_NCX) - R(1.00000)) * y_V) * K(C_F)), (K(C_R) * K(C_T)))), R(1.00000))));
    H[22] = cfg_exp(cfg_cdiv<KS>(((K(C_gamma_NCX) * y_V) * K(C_F)), (K(C_R) * K(C_T))));
    H[23] = (cfg_exp(cfg_cdiv<KS>((((K(C_gamma_NCX) - R(1.00000)) * y_V) * K(C_F)), (K(C_R) * K(C_T)))) * cfg_ipow<3>(K(C_Na_o)));
    H[24] = cfg_sqrt((K(C_K_o) / R(5.40000)));
    H[25] = (K(C_g_Kr) * cfg_sqrt((K(C_K_o) / R(5.40000))));
    H[26] = CfgSlot::divisor(cfg_expm1(cfg_cdiv<KS>(((R(2.00000) * y_V) * K(C_F)), (K(C_R) * K(C_T)))));
    H[27] = cfg_exp(cfg_cdiv<KS>(((R(2.00000) * y_V) * K(C_F)), (K(C_R) * K(C_T))));
    H[28] = CfgSlot::divisor((R(1.00000) + cfg_exp(cfg_cdiv<KS>((R(25.0000) - y_V), R(5.98000)))));
}
template <class YS, class KS, class HS>
__device__ __forceinline__ double rhs_tissue(const YS& Y, const KS& K, const HS& H, double* dydt, int tissue)
{
    using R = double;
    constexpr bool SOLVE_VM = false;
    constexpr double t = 0.0;
    const CfgStimulus stim{};
    (void)tissue; (void)K; (void)H; (void)t; (void)stim;
    const R y_V = Y(S_V);
    const R y_K_i = Y(S_K_i);
    const R y_Na_i = Y(S_Na_i);
    const R y_Ca_i = Y(S_Ca_i);
    const R y_Xr1 = Y(S_Xr1);
    const R y_Xr2 = Y(S_Xr2);
    const R y_Xs = Y(S_Xs);
    const R y_m = Y(S_m);
    const R y_h = Y(S_h);
    const R y_j = Y(S_j);
    const R y_d = Y(S_d);
    const R y_f = Y(S_f);
    const R y_fCa = Y(S_fCa);
    const R y_s = Y(S_s);
    const R y_r = Y(S_r);
    const R y_Ca_SR = Y(S_Ca_SR);
    const R y_g = Y(S_g);
    dydt[S_m] = cfg_hdiv((H(H_m_inf) - y_m), H(H_tau_m));
    dydt[S_h] = cfg_hdiv((H(H_h_inf) - y_h), H(H_tau_h));
    dydt[S_j] = cfg_hdiv((H(H_j_inf) - y_j), H(H_tau_j));
    dydt[S_d] = cfg_hdiv((H(H_d_inf) - y_d), H(H_tau_d));
    dydt[S_f] = cfg_hdiv((H(H_f_inf) - y_f), H(H_tau_f));
    R a_alpha_fCa = (R(1.00000) / (R(1.00000) + cfg_ipow<8>(cfg_cdiv<KS>(y_Ca_i, R(0.000325000)))));
    R a_beta_fCa = (R(0.100000) / (R(1.00000) + cfg_exp(cfg_cdiv<KS>((y_Ca_i - R(0.000500000)), R(0.000100000)))));
    R a_beta_d = (R(0.200000) / (R(1.00000) + cfg_exp(cfg_cdiv<KS>((y_Ca_i - R(0.000750000)), R(0.000800000)))));
    R a_fCa_inf = cfg_cdiv<KS>((((a_alpha_fCa + a_beta_fCa) + a_beta_d) + R(0.230000)), R(1.46000));
    R a_d_fCa = cfg_cdiv<KS>((a_fCa_inf - y_fCa), K(C_tau_fCa));
    dydt[S_fCa] = (((a_fCa_inf > y_fCa) && (y_V > (-R(60.0000)))) ? R(0.00000) : a_d_fCa);
    dydt[S_s] = cfg_hdiv((H(H_s_inf) - y_s), H(H_tau_s));
    dydt[S_r] = cfg_hdiv((H(H_r_inf) - y_r), H(H_tau_r));
    dydt[S_Xr1] = cfg_hdiv((H(H_xr1_inf) - y_Xr1), H(H_tau_xr1));
    dydt[S_Xr2] = cfg_hdiv((H(H_xr2_inf) - y_Xr2), H(H_tau_xr2));
    dydt[S_Xs] = cfg_hdiv((H(H_xs_inf) - y_Xs), H(H_tau_xs));
    R a_g_inf = ((y_Ca_i < R(0.000350000)) ? (R(1.00000) / (R(1.00000) + cfg_ipow<6>(cfg_cdiv<KS>(y_Ca_i, R(0.000350000))))) : (R(1.00000) / (R(1.00000) + cfg_ipow<16>(cfg_cdiv<KS>(y_Ca_i, R(0.000350000))))));
    R a_d_g = cfg_cdiv<KS>((a_g_inf - y_g), K(C_tau_g));
    dydt[S_g] = (((a_g_inf > y_g) && (y_V > (-R(60.0000)))) ? R(0.00000) : a_d_g);
    R a_i_NaK = cfg_hdiv(((((K(C_P_NaK) * K(C_K_o)) / (K(C_K_o) + K(C_K_mk))) * y_Na_i) / (y_Na_i + K(C_K_mNa))), H(20));
    R a_E_Na = (((K(C_R) * K(C_T)) / K(C_F)) * cfg_log((K(C_Na_o) / y_Na_i)));
    R a_i_Na = ((((K(C_g_Na) * cfg_ipow<3>(y_m)) * y_h) * y_j) * (y_V - a_E_Na));
    R a_i_b_Na = (K(C_g_bNa) * (y_V - a_E_Na));
    R a_i_NaCa = cfg_hdiv((K(C_K_NaCa) * cfg_fma((H(22) * cfg_ipow<3>(y_Na_i)), K(C_Ca_o), -((H(23) * y_Ca_i) * K(C_alpha_NCX)))), H(21));
    dydt[S_Na_i] = cfg_cdiv<KS>(((-cfg_fma(R(3.00000), a_i_NaCa, cfg_fma(R(3.00000), a_i_NaK, (a_i_Na + a_i_b_Na)))) * K(C_Cm)), (K(C_V_c) * K(C_F)));
    R a_E_K = (((K(C_R) * K(C_T)) / K(C_F)) * cfg_log((K(C_K_o) / y_K_i)));
    R a_alpha_K1 = (R(0.100000) / (R(1.00000) + cfg_exp((R(0.0600000) * ((y_V - a_E_K) - R(200.000))))));
    R a_beta_K1 = (cfg_fma(R(3.00000), cfg_exp((R(0.000200000) * ((y_V - a_E_K) + R(100.000)))), (R(1.00000) * cfg_exp((R(0.100000) * ((y_V - a_E_K) - R(10.0000)))))) / (R(1.00000) + cfg_exp(((-R(0.500000)) * (y_V - a_E_K)))));
    R a_xK1_inf = (a_alpha_K1 / (a_alpha_K1 + a_beta_K1));
    R a_i_K1 = (((K(C_g_K1) * a_xK1_inf) * H(24)) * (y_V - a_E_K));
    R a_i_to = (((K(C_g_to) * y_r) * y_s) * (y_V - a_E_K));
    R a_i_Kr = (((H(25) * y_Xr1) * y_Xr2) * (y_V - a_E_K));
    R a_E_Ks = (((K(C_R) * K(C_T)) / K(C_F)) * cfg_log(((K(C_K_o) + (K(C_P_kna) * K(C_Na_o))) / cfg_fma(K(C_P_kna), y_Na_i, y_K_i))));
    R a_i_Ks = ((K(C_g_Ks) * cfg_ipow<2>(y_Xs)) * (y_V - a_E_Ks));
    R a_i_CaL = cfg_hdiv((cfg_cdiv<KS>(((((((K(C_g_CaL) * y_d) * y_f) * y_fCa) * R(4.00000)) * y_V) * cfg_ipow<2>(K(C_F))), (K(C_R) * K(C_T))) * cfg_fma(y_Ca_i, H(27), -(R(0.341000) * K(C_Ca_o)))), H(26));
    R a_E_Ca = ((((R(0.500000) * K(C_R)) * K(C_T)) / K(C_F)) * cfg_log((K(C_Ca_o) / y_Ca_i)));
    R a_i_b_Ca = (K(C_g_bCa) * (y_V - a_E_Ca));
    R a_i_p_K = cfg_hdiv((K(C_g_pK) * (y_V - a_E_K)), H(28));
    R a_i_p_Ca = ((K(C_g_pCa) * y_Ca_i) / (y_Ca_i + K(C_K_pCa)));
    R a_Iion_cm = (((((((((((a_i_K1 + a_i_to) + a_i_Kr) + a_i_Ks) + a_i_CaL) + a_i_NaK) + a_i_Na) + a_i_b_Na) + a_i_NaCa) + a_i_b_Ca) + a_i_p_K) + a_i_p_Ca);
    R a_Istim = (SOLVE_VM ? R(cfg_stimulus_current<double>(t, stim)) : R(0));
    dydt[S_V] = R(0.0);
    if (SOLVE_VM) {
        dydt[S_V] = ((-a_Iion_cm) - a_Istim);
    }
    dydt[S_K_i] = cfg_cdiv<KS>(((-cfg_fma(-R(2.00000), a_i_NaK, (((((a_i_K1 + a_i_to) + a_i_Kr) + a_i_Ks) + a_i_p_K) + a_Istim))) * K(C_Cm)), (K(C_V_c) * K(C_F)));
    R a_i_rel = (((((K(C_a_rel) * cfg_ipow<2>(y_Ca_SR)) / (cfg_ipow<2>(K(C_b_rel)) + cfg_ipow<2>(y_Ca_SR))) + K(C_c_rel)) * y_d) * y_g);
    R a_i_up = (K(C_Vmax_up) / (R(1.00000) + (cfg_ipow<2>(K(C_K_up)) / cfg_ipow<2>(y_Ca_i))));
    R a_i_leak = (K(C_V_leak) * (y_Ca_SR - y_Ca_i));
    R a_ddt_Ca_i_total = ((cfg_fma(cfg_cdiv<KS>((-cfg_fma(-R(2.00000), a_i_NaCa, ((a_i_CaL + a_i_b_Ca) + a_i_p_Ca))), ((R(2.00000) * K(C_V_c)) * K(C_F))), K(C_Cm), a_i_leak) - a_i_up) + a_i_rel);
    R a_f_JCa_i_free = (R(1.00000) / (R(1.00000) + ((K(C_Buf_c) * K(C_K_buf_c)) / cfg_ipow<2>((y_Ca_i + K(C_K_buf_c))))));
    dydt[S_Ca_i] = (a_ddt_Ca_i_total * a_f_JCa_i_free);
    R a_ddt_Ca_sr_total = ((K(C_V_c) / K(C_V_sr)) * (a_i_up - (a_i_rel + a_i_leak)));
    R a_f_JCa_sr_free = (R(1.00000) / (R(1.00000) + ((K(C_Buf_sr) * K(C_K_buf_sr)) / cfg_ipow<2>((y_Ca_SR + K(C_K_buf_sr))))));
    dydt[S_Ca_SR] = (a_ddt_Ca_sr_total * a_f_JCa_sr_free);
    return a_Iion_cm;
}
// States whose tissue-mode rate is a - b y with a and b functions of state 0 and
// constants alone (bit i = state i): b of each, and their rates alone.
constexpr unsigned long long LIN_MASK = 0x6ff0ull;
template <class KS, class HS>
__device__ __forceinline__ void gate_decay(double y_V, const KS& K, const HS& H, int tissue, double* b)
{
    using R = double;
    (void)tissue; (void)K; (void)H; (void)b; (void)y_V;
    b[S_Xr1] = cfg_hdiv(R(1.0), H(H_tau_xr1));
    b[S_Xr2] = cfg_hdiv(R(1.0), H(H_tau_xr2));
    b[S_Xs] = cfg_hdiv(R(1.0), H(H_tau_xs));
    b[S_m] = cfg_hdiv(R(1.0), H(H_tau_m));
    b[S_h] = cfg_hdiv(R(1.0), H(H_tau_h));
    b[S_j] = cfg_hdiv(R(1.0), H(H_tau_j));
    b[S_d] = cfg_hdiv(R(1.0), H(H_tau_d));
    b[S_f] = cfg_hdiv(R(1.0), H(H_tau_f));
    b[S_s] = cfg_hdiv(R(1.0), H(H_tau_s));
    b[S_r] = cfg_hdiv(R(1.0), H(H_tau_r));
}
template <class YS, class KS, class HS>
__device__ __forceinline__ void gate_rates(const YS& Y, const KS& K, const HS& H, int tissue, double* d)
{
    using R = double;
    (void)tissue; (void)K; (void)H; (void)d; (void)Y;
    const R y_Xr1 = Y(S_Xr1);
    const R y_Xr2 = Y(S_Xr2);
    const R y_Xs = Y(S_Xs);
    const R y_m = Y(S_m);
    const R y_h = Y(S_h);
    const R y_j = Y(S_j);
    const R y_d = Y(S_d);
    const R y_f = Y(S_f);
    const R y_s = Y(S_s);
    const R y_r = Y(S_r);
    d[S_m] = cfg_hdiv((H(H_m_inf) - y_m), H(H_tau_m));
    d[S_h] = cfg_hdiv((H(H_h_inf) - y_h), H(H_tau_h));
    d[S_j] = cfg_hdiv((H(H_j_inf) - y_j), H(H_tau_j));
    d[S_d] = cfg_hdiv((H(H_d_inf) - y_d), H(H_tau_d));
    d[S_f] = cfg_hdiv((H(H_f_inf) - y_f), H(H_tau_f));
    d[S_s] = cfg_hdiv((H(H_s_inf) - y_s), H(H_tau_s));
    d[S_r] = cfg_hdiv((H(H_r_inf) - y_r), H(H_tau_r));
    d[S_Xr1] = cfg_hdiv((H(H_xr1_inf) - y_Xr1), H(H_tau_xr1));
    d[S_Xr2] = cfg_hdiv((H(H_xr2_inf) - y_Xr2), H(H_tau_xr2));
    d[S_Xs] = cfg_hdiv((H(H_xs_inf) - y_Xs), H(H_tau_xs));
}
// Warp of state i where four warps share a cell's step (tissue mode; split.py).
CFG_HD constexpr int part_tissue(int i)
{
    constexpr signed char part[NS] = {0, 1, 3, 2, 2, 3, 2, 1, 3, 3, 0, 1, 0, 0, 2, 0, 3};
    return part[i];
}
// Warp of state i where four warps share a cell's step (Vm a state; split.py).
CFG_HD constexpr int part_sv(int i)
{
    constexpr signed char part[NS] = {1, 1, 1, 2, 0, 3, 2, 2, 3, 0, 0, 1, 3, 3, 3, 2, 0};
    return part[i];
}

// the model's traits with these right-hand sides
struct Model : tnnp::Model {
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

} } }  // namespace cfg::tnnp::plain
