// Ionic update kernels: one thread per cell, state in SoA arrays, the whole
// per-cell ODE solve of a PDE step held in registers / thread-local memory.
//
// Reference behaviour reproduced (per cell, <Model>::solveODE, e.g.
// src/ionicModels/TNNP/TNNP.C:114-179):
//   STATES[0] <- Vm mapped to model units; step <- min(step, dt_model);
//   ODESolver::solve(tStart, tEnd, STATES, step) with RKF45;
//   computeVariables(tEnd); Im = scale * ALGEBRAIC[Iion].
// The RKF45 step control restates OpenFOAM's ODESolver/adaptiveSolver
// (truncated last step, persistent per-cell step, safeScale/minScale/
// maxScale/alphaInc/alphaDec); the tableau is Fehlberg's.
//
// This file holds the plain form: every operation in FP64, right-hand sides
// and sums in the reference's evaluation order with explicit multiply-adds,
// the linear gates of a tissue step in closed form.  The mixed form is in
// ionic_mixed.cuh.
#pragma once

#include <type_traits>

#include "ionic_common.cuh"
#include "linear_gates.cuh"
#include "../../include/cardiac_gpu.h"

// resident 128-thread blocks per SM the ionic kernels are compiled for
// (register budget 65536 / (128 * blocks))
#ifndef CFG_IONIC_MIN_BLOCKS
#define CFG_IONIC_MIN_BLOCKS 2
#endif
// unroll factor of the FP64 batch's loops over the states (stage sums,
// 5th-order update, error norm); 1 keeps the kernel's instruction footprint
// close to one copy of the model body
#ifndef CFG_IONIC_STATE_UNROLL
#define CFG_IONIC_STATE_UNROLL 1
#endif


namespace cfg {

constexpr int kStateUnroll = CFG_IONIC_STATE_UNROLL;

struct IonicLaunch {
    long long n;                     // cells (and the stride of the state arrays)
    long long first, count;          // state slots [first, first + count) of this launch
    const int* perm;                 // [n] cell of each state slot, or null (slot = cell)
    int cells_per_thread;            // slots per thread (grid-stride), chosen by the launcher
    double t0, dt;                   // PDE step [s] (used when t_dev is null)
    const double* t_dev;             // device time of the step start [s], or null
    int tissue;                      // uniform tissue flag (when tissue_cell is null)
    const unsigned char* tissue_cell;
    const double* scales;            // [6][scale_stride] conductance scales, or null
    long long scale_stride;
    CfgStimulus stim;                // single-cell protocol (tissue runs: none)
    OdeSettings ode;
    const double* vm;                // [n] membrane potential [V] (tissue mode)
    double* im;                      // [n] ionic current [V/s]
    double* yw;                      // wide states  [NW][n] (all states in the plain form)
    float* yn;                       // narrow states [NN][n] (mixed form only)
    double* step;                    // [n] persistent ODE step [model time units]
    int* status;                     // CFG_ERR_* bits, OR-ed
    unsigned long long* rhs_evals;   // optional counter of RHS evaluations
    double* fail_record;             // optional [8]: first failing cell (see IonicFailure)
};

// Record of the first cell whose ODE solve failed: [0] cell, [1] reason
// (1 = maxSteps, 2 = step underflow), [2] x, [3] dx, [4] worst state,
// [5] its normalised error, [6] that state's value, [7] substeps taken.
struct IonicFailure {
    int reason = 0;
    double x = 0, dx = 0, err = 0, value = 0;
    int worst = -1;
    long long steps = 0;
};

template <class R>
struct ArrayView {
    const R* a;
    CFG_D __forceinline__ R operator()(int i) const { return a[i]; }
};

// constants computed at run time (per-cell tissue or conductance scales)
template <class R>
struct ConstView {
    static constexpr bool kFolded = false;
    const double* c;
    CFG_D __forceinline__ R operator()(int i) const { return R(c[i]); }
};

// constants of one uniform tissue, known at compile time
template <class R, class M, int T>
struct ConstFold {
    static constexpr bool kFolded = true;
    CFG_D __forceinline__ R operator()(int i) const { return R(M::template constant<T>(i)); }
};

template <unsigned long long MASK>
CFG_D __forceinline__ constexpr bool is_wide(int i) { return (MASK >> i) & 1ull; }

template <class M, bool FP64>
struct Layout {
    // index of state i inside the wide or the narrow array
    static CFG_HD constexpr int slot(int i)
    {
        int k = 0;
        for (int j = 0; j < i; ++j)
            if (FP64 || ((M::WIDE_MASK >> j) & 1ull) == ((M::WIDE_MASK >> i) & 1ull)) ++k;
        return k;
    }
    static CFG_HD constexpr int n_wide()
    {
        int k = 0;
        for (int j = 0; j < M::NS; ++j)
            if (FP64 || ((M::WIDE_MASK >> j) & 1ull)) ++k;
        return k;
    }
    static CFG_HD constexpr int n_narrow() { return M::NS - n_wide(); }
};

template <int MAP>
CFG_D __forceinline__ double vm_to_state0(double vm)
{
    if constexpr (MAP == CFG_VM_ALIEV) return (vm * 1000.0 + 80) / 100;
    else if constexpr (MAP == CFG_VM_BUENO) return (vm * 1000.0 + 84) / 85.7;
    else if constexpr (MAP == CFG_VM_IDENTITY) return vm;
    else return vm * 1000.0;
}

// model time of the step: TNNP.C:122-123 (t*1000), AlievPanfilov.C:107-108
template <class M>
CFG_D __forceinline__ void model_times(double t0, double dt, double& ts, double& te, double& dtm)
{
    if constexpr (M::TIME_SCALE == 1000.0) {
        // model time in seconds (monodomainFDAManufactured.C:96-97)
        ts = t0;
        te = t0 + dt;
        dtm = dt;
    } else if constexpr (M::TIME_SCALE == 1.0) {
        ts = t0 * 1000;
        te = (t0 + dt) * 1000;
        dtm = dt * 1000.0;
    } else {
        ts = t0 * 1000.0 / M::TIME_SCALE;
        te = (t0 + dt) * 1000.0 / M::TIME_SCALE;
        dtm = dt * 1000.0 / M::TIME_SCALE;
    }
}

// Step-control arithmetic that must round exactly as written (no FMA
// contraction, which the mixed-form build enables): the end-of-interval test
// relies on x - xEnd being exactly zero when x has landed on xEnd.
CFG_D __forceinline__ double exact_add(double a, double b) { return __dadd_rn(a, b); }
CFG_D __forceinline__ double exact_sub(double a, double b) { return __dsub_rn(a, b); }
CFG_D __forceinline__ double exact_mul(double a, double b) { return __dmul_rn(a, b); }

// Stage table of the Fehlberg tableau for the stage loop (row s: a_s,j).
static __constant__ double kRkfA[6][5] = {
    {0, 0, 0, 0, 0},
    {rkf::a21, 0, 0, 0, 0},
    {rkf::a31, rkf::a32, 0, 0, 0},
    {rkf::a41, rkf::a42, rkf::a43, 0, 0},
    {rkf::a51, rkf::a52, rkf::a53, rkf::a54, 0},
    {rkf::a61, rkf::a62, rkf::a63, rkf::a64, rkf::a65},
};
static __constant__ double kRkfC[6] = {0.0, rkf::c2, rkf::c3, rkf::c4, rkf::c5, rkf::c6};

// Mixed form: multiple of the FP32 unit round-off charged to each stage
// derivative in the error test (model right-hand sides lose a few tens of
// ulps through exp/log/division chains).
constexpr double kFp32NoiseUlps = 64.0;


// The larger of two magnitudes by their bits (an FP64 comparison takes the FP64
// pipe); NaN if one is.
CFG_D __forceinline__ double larger_magnitude(double a, double b)
{
    const double p = fabs(a), q = fabs(b);
    return __double_as_longlong(p) > __double_as_longlong(q) ? p : q;
}

// One right-hand-side evaluation with Vm among the states.  Not inlined: the
// stage loop and the final current evaluation share one copy of the (large)
// model body, which keeps the kernel's instruction footprint to a single
// model instance.
template <class M, class KS>
__device__ __noinline__ double rhs_eval(double t, const double* y, const KS* K, double* dydt,
                                        int tissue, const CfgStimulus* st)
{
    return M::template rates<true>(t, ArrayView<double>{y}, *K, dydt, tissue, *st);
}

// Storage of the per-cell membrane-potential-only values (at least one
// element, so that models without any still compile).
template <class M, class R>
struct Hoisted {
    R v[M::NH > 0 ? M::NH : 1];
};

// ODESolver::solve(xStart, xEnd, y, dxTry) with adaptiveSolver::solve and
// RKF45::solve inside, Vm among the states.  The six right-hand-side
// evaluations of a trial step (dydx0 and stages 2..6) run through one loop, so
// the model body is instantiated once.  Stage sums are accumulated left to
// right exactly as the host code writes them.  Returns accepted substeps, or -1
// on maxSteps overflow / step underflow.
template <class M, class KS>
CFG_D __forceinline__ long long rkf45_solve(double xs, double xe, double (&y)[M::NS],
                                            double& dx_try, double (*k)[M::NS], const KS& K,
                                            int tissue, const CfgStimulus& st,
                                            const OdeSettings& s, unsigned& evals,
                                            IonicFailure* why)
{
    using namespace rkf;
    constexpr int NS = M::NS;
    double step_dx = dx_try;
    bool last = false;
    double x = xs;
    double yt[NS];             // stage input, then y5
    for (long long n = 0; n < s.max_steps; ++n) {
        const double dx_try0 = step_dx;
        {
            const double xn = exact_add(x, step_dx);
            if (exact_mul(exact_sub(xn, xe), exact_sub(xn, xs)) > 0) {
                last = true;
                step_dx = exact_sub(xe, x);
            }
        }
        // --- adaptiveSolver::solve(odes, x, y, dxTry)
        double dx = step_dx;
        double err;
        int worst = -1;
        int s0 = 0;   // dydx0 is evaluated once per adaptive step
        for (;;) {
#pragma unroll 1
            for (int sg = s0; sg < 6; ++sg) {
                if (sg == 0) {
#pragma unroll kStateUnroll
                    for (int i = 0; i < NS; ++i) yt[i] = y[i];
                } else if (sg == 1) {
#pragma unroll kStateUnroll
                    for (int i = 0; i < NS; ++i) yt[i] = y[i] + a21 * dx * k[0][i];
                } else {
#pragma unroll kStateUnroll
                    for (int i = 0; i < NS; ++i) {
                        double acc = kRkfA[sg][0] * k[0][i];
                        for (int j = 1; j < sg; ++j) acc += kRkfA[sg][j] * k[j][i];
                        yt[i] = y[i] + dx * acc;
                    }
                }
                rhs_eval<M, KS>(x + kRkfC[sg] * dx, yt, &K, k[sg], tissue, &st);
                evals += 1;
            }
            s0 = 1;
            // 5th-order solution and the embedded error (RKF45::solve), then
            // ODESolver::normalizeError
            ErrorNorm norm;
#pragma unroll kStateUnroll
            for (int i = 0; i < NS; ++i) {
                yt[i] = y[i] + dx * (b1 * k[0][i] + b3 * k[2][i] + b4 * k[3][i]
                                     + b5 * k[4][i] + b6 * k[5][i]);
                const double e_i = dx * (e1 * k[0][i] + e3 * k[2][i] + e4 * k[3][i]
                                         + e5 * k[4][i] + e6 * k[5][i]);
                norm.take(fabs(e_i), s.abs_tol + s.rel_tol * larger_magnitude(y[i], yt[i]), i);
            }
            err = norm.value();
            worst = norm.state;
            if (!(err > 1)) break;
            double scale = s.safe_scale * pow(err, -s.alpha_dec);
            if (scale < s.min_scale) scale = s.min_scale;
            dx *= scale;
            if (dx < 1e-300) {
                *why = IonicFailure{2, x, dx, err, worst >= 0 ? y[worst] : 0.0, worst, n};
                return -1;
            }
        }
        why->x = x; why->dx = dx; why->err = err; why->worst = worst; why->steps = n;
        x = exact_add(x, dx);
#pragma unroll kStateUnroll
        for (int i = 0; i < NS; ++i) y[i] = yt[i];
        if (err > s.inc_threshold) {
            double scale = s.safe_scale * pow(err, -s.alpha_inc);
            if (scale > s.max_scale) scale = s.max_scale;
            step_dx = scale * dx;
        } else {
            step_dx = s.safe_scale * s.max_scale * dx;
        }
        // --- back in ODESolver::solve
        if (exact_mul(exact_sub(x, xe), exact_sub(xe, xs)) >= 0) {
            if (n > 0 && last) step_dx = dx_try0;
            dx_try = step_dx;
            return n + 1;
        }
    }
    why->reason = 1;
    why->value = why->worst >= 0 ? y[why->worst] : 0.0;
    return -1;
}

// The plain form's step of 32 cells (a tile) by W warps.
//
// What bounds it: GB300 issues one FP64 instruction per SM partition (a
// quarter of an SM) every 64 clocks, however many of its 32 lanes are active,
// and one warp alone keeps a partition's FP64 unit at 90 % (456 us for a tile
// of ORd, 928 us for two tiles on one partition).  The time of a step is
// therefore the number of FP64 instructions of a tile times the number of
// tiles on the fullest partition, and three things set it:
//
//   * the linear gates of a tissue step follow their closed form
//     (linear_gates.cuh): 15 multiply-adds for a gate's five stage values,
//     where its stage sums and slopes cost about 85, and the error norm takes
//     one division per trial instead of one per state (ErrorNorm);
//   * the stages, trials and substeps of a lane are one loop, so the lanes of
//     a warp that need different numbers of them meet at the right-hand side;
//   * where the tiles do not fill the partitions, four warps share a tile
//     (W = 4): each integrates a part of the states (M::part_*, chosen by
//     the emitter so that the parts cost the same) and evaluates only the
//     statements their rates need; the stage inputs cross in shared memory,
//     one block barrier per stage.  Warp 0 takes the step control's decisions
//     and publishes them, so every warp follows the same path.
//
// Stage sums are accumulated left to right as the host code writes them, with
// explicit multiply-adds (and no contraction by the compiler), and the error
// norm is the largest ratio exactly, so that a cell's result does not depend on
// the launch shape.
template <class M, bool SV>
struct StepSplit {
    using T = TissueSplit<M>;
    static constexpr bool lin(int i) { return !SV && T::lin(i); }
    static constexpr bool moves(int i) { return SV || i > 0; }
    static constexpr bool rest(int i) { return moves(i) && !lin(i); }
    static constexpr bool any_rest()
    {
        for (int i = 0; i < M::NS; ++i)
            if (rest(i)) return true;
        return false;
    }
};

// The states of part P of W and their stage slots.
template <class M, bool SV, int W, int P>
struct StepPart {
    using S = StepSplit<M, SV>;
    static constexpr bool own(int i)
    {
        return W == 1 || (SV ? M::part_sv(i) : M::part_tissue(i)) == P;
    }
    // index of state n among this part's states with stage slots
    static constexpr int slot(int n)
    {
        int k = 0;
        for (int j = 0; j < n; ++j) k += (S::rest(j) && own(j)) ? 1 : 0;
        return k;
    }
    static constexpr int NK = slot(M::NS), NKA = NK > 0 ? NK : 1;
};

template <int NS, int W>
struct StepShared {
    double y[2][NS][32];    // stage inputs of a tile, double buffered
    double err[W][32];      // error norm of each part, and its state
    int worst[W][32];
    double step[32];        // decision: next step, the norm, its state, accept
    double norm[32];
    int norm_state[32], accept[32];
};
template <int NS>
struct StepShared<NS, 1> {};

template <int W>
CFG_D __forceinline__ void tile_sync()
{
    if constexpr (W > 1) asm volatile("bar.sync 1, %0;" ::"n"(32 * W) : "memory");
}

template <int NS>
CFG_D __forceinline__ double value_at(const double (&y)[NS], int i)
{
    double v = 0.0;
#pragma unroll
    for (int k = 0; k < NS; ++k)
        if (k == i) v = y[k];
    return v;
}

struct SharedState {
    const double* a;   // [NS][32], at this lane
    CFG_D __forceinline__ double operator()(int i) const { return a[32 * i]; }
};

// The right-hand side of a step, at time t and the states of a view.
template <class M, bool SV, class KS>
struct StepRates {
    const KS& K;
    const CfgSlot* H;
    int tissue;
    const CfgStimulus& stim;
    template <class YS>
    CFG_D __forceinline__ double operator()(double t, const YS& y, double* d) const
    {
        if constexpr (SV)
            return M::template rates<true>(t, y, K, d, tissue, stim);
        else
            return M::rates_tissue(y, K, ArrayView<CfgSlot>{H}, d, tissue);
    }
};

// Part P of a tile's step; lanes with live = false repeat another cell and
// store nothing.
template <class M, bool SV, int W, int P, class KS>
CFG_D __forceinline__ void fp64_tile(const IonicLaunch& p, const KS& K, int tissue, long long c,
                                     bool live, StepShared<M::NS, W>& sh, unsigned& evals)
{
    using namespace rkf;
    using S = StepSplit<M, SV>;
    using L = Layout<M, true>;
    using Q = StepPart<M, SV, W, P>;
    constexpr int NS = M::NS;
    constexpr unsigned kFull = 0xffffffffu;
    const int lane = threadIdx.x & 31;
    const OdeSettings& s = p.ode;
    const long long cell = p.perm ? p.perm[c] : c;
    const double t0 = p.t_dev ? p.t_dev[0] : p.t0;
    double xs, xe, dtm;
    model_times<M>(t0, p.dt, xs, xe, dtm);
    double y[NS], yt[NS];      // states; stage inputs, then y5
#pragma unroll
    for (int i = 0; i < NS; ++i)
        if (Q::own(i) || (i == 0 && !SV)) y[i] = p.yw[(long long)L::slot(i) * p.n + c];
    if constexpr (!SV) y[0] = vm_to_state0<M::VM_MAP>(p.vm[cell]);
    double step = p.step[c];
    if (dtm < step) step = dtm;   // step = min(step, dt_model)

    CfgSlot H[M::NH > 0 ? M::NH : 1];   // values of the membrane potential alone
    double decay[NS], hk[NS];     // of the gates: coefficient, dx k1
    if constexpr (!SV) {
        M::hoist_vm(y[0], K, tissue, H);
        M::decay(y[0], K, ArrayView<CfgSlot>{H}, tissue, decay);
    }
    const StepRates<M, SV, KS> rates{K, H, tissue, p.stim};
    double k[6][Q::NKA];
    double x = xs, step_dx = step, dx = 0.0, dx_try0 = 0.0, err = 0.0;
    bool last = false, begin = true, new_try = true, done = false;
    int sg = 0, worst = -1, buf = 0, reason = 0;
    long long n = 0;
    double fail_x = 0.0, fail_dx = 0.0;   // as ODESolver reports a failure
    long long fail_steps = 0;
    for (;;) {
        if (!done && begin) {
            begin = false;
            if (n >= s.max_steps) {
                reason = 1;
                done = true;
            } else {
                dx_try0 = step_dx;
                const double xn = exact_add(x, step_dx);
                if (exact_mul(exact_sub(xn, xe), exact_sub(xn, xs)) > 0) {
                    last = true;
                    step_dx = exact_sub(xe, x);
                }
                dx = step_dx;
                sg = 0;
                new_try = true;
            }
        }
        if (__all_sync(kFull, done)) break;
        if (new_try) {
            new_try = false;
            if constexpr (!SV) {
                // the gates' slopes at the substep's start
                double d[NS];
                M::slopes(ArrayView<double>{y}, K, ArrayView<CfgSlot>{H}, tissue, d);
#pragma unroll
                for (int i = 1; i < NS; ++i)
                    if (S::lin(i) && Q::own(i)) hk[i] = dx * d[i];
            }
        }
        if constexpr (S::any_rest()) {
            // stage inputs: the gates y + hk q_sg(-dx decay), the rest y + dx sum a k
            const auto gates = [&](auto poly) {
#pragma unroll
                for (int i = 1; i < NS; ++i)
                    if (S::lin(i) && Q::own(i))
                        yt[i] = lingate::fma_r(hk[i], poly(-dx * decay[i]), y[i]);
            };
            if (sg == 0) {
#pragma unroll
                for (int i = 0; i < NS; ++i)
                    if (S::moves(i) && Q::own(i)) yt[i] = y[i];
            } else {
                switch (sg) {
                case 1: gates([](double z) { return lingate::stage_poly<1, double>(z); }); break;
                case 2: gates([](double z) { return lingate::stage_poly<2, double>(z); }); break;
                case 3: gates([](double z) { return lingate::stage_poly<3, double>(z); }); break;
                case 4: gates([](double z) { return lingate::stage_poly<4, double>(z); }); break;
                default: gates([](double z) { return lingate::stage_poly<5, double>(z); }); break;
                }
#pragma unroll
                for (int i = 0; i < NS; ++i)
                    if (S::rest(i) && Q::own(i)) {
                        const int e = Q::slot(i);
                        double acc = kRkfA[sg][0] * k[0][e];
#pragma unroll 1
                        for (int j = 1; j < sg; ++j) acc = cfg_fma(kRkfA[sg][j], k[j][e], acc);
                        yt[i] = cfg_fma(dx, acc, y[i]);
                    }
            }
            const double t = SV ? x + kRkfC[sg] * dx : 0.0;
            double d[NS] = {};
            if constexpr (W > 1) {
#pragma unroll
                for (int i = 0; i < NS; ++i) {
                    if (S::moves(i) && Q::own(i)) sh.y[buf][i][lane] = yt[i];
                    if (i == 0 && !SV && P == 0) sh.y[buf][0][lane] = y[0];
                }
                tile_sync<W>();
                (void)rates(t, SharedState{&sh.y[buf][0][lane]}, d);
                buf ^= 1;
            } else {
                if constexpr (!SV) yt[0] = y[0];
                (void)rates(t, ArrayView<double>{yt}, d);
            }
#pragma unroll
            for (int i = 0; i < NS; ++i)
                if (S::rest(i) && Q::own(i)) k[sg][Q::slot(i)] = d[i];
            if (!done && live && P == 0) ++evals;
        } else {
            if (!done && live) evals += unsigned(6 - sg);   // the closed form's stages
            sg = 5;
        }
        const bool at_end = !done && sg == 5;
        if (__any_sync(kFull, at_end)) {
            // 5th-order solution and the embedded error (RKF45::solve), then
            // ODESolver::normalizeError
            ErrorNorm norm;
            if (at_end) {
#pragma unroll
                for (int i = 0; i < NS; ++i) {
                    if (!(S::moves(i) && Q::own(i))) continue;
                    double e_i;
                    if (S::lin(i)) {
                        const double z = -dx * decay[i];
                        yt[i] = lingate::fma_r(hk[i], lingate::increment_poly<double>(z), y[i]);
                        e_i = hk[i] * lingate::error_poly<double>(z);
                    } else {
                        const int j = Q::slot(i);
                        const double k1 = k[0][j], k3 = k[2][j], k4 = k[3][j], k5 = k[4][j],
                                     k6 = k[5][j];
                        yt[i] = cfg_fma(dx, cfg_fma(b6, k6, cfg_fma(b5, k5, cfg_fma(b4, k4,
                                            cfg_fma(b3, k3, b1 * k1)))), y[i]);
                        e_i = dx * cfg_fma(e6, k6, cfg_fma(e5, k5, cfg_fma(e4, k4,
                                       cfg_fma(e3, k3, e1 * k1))));
                    }
                    norm.take(fabs(e_i),
                              cfg_fma(s.rel_tol, larger_magnitude(y[i], yt[i]), s.abs_tol), i);
                }
            }
            double nerr = norm.value(), ndx = 0.0;
            int ew = norm.state;
            bool accept = false;
            if constexpr (W > 1) {
                sh.err[P][lane] = nerr;
                sh.worst[P][lane] = ew;
                tile_sync<W>();
            }
            if (W == 1 || P == 0) {
                if constexpr (W > 1) {
                    // the largest rounded ratio is the largest ratio, rounded
#pragma unroll
                    for (int q = 1; q < W; ++q)
                        if (sh.err[q][lane] > nerr) {
                            nerr = sh.err[q][lane];
                            ew = sh.worst[q][lane];
                        }
                }
                accept = !(nerr > 1);
                if (!accept) {
                    double scale = s.safe_scale * pow(nerr, -s.alpha_dec);
                    if (scale < s.min_scale) scale = s.min_scale;
                    ndx = scale;
                } else if (nerr > s.inc_threshold) {
                    double scale = s.safe_scale * pow(nerr, -s.alpha_inc);
                    if (scale > s.max_scale) scale = s.max_scale;
                    ndx = scale;
                } else {
                    ndx = exact_mul(s.safe_scale, s.max_scale);
                }
                ndx = exact_mul(ndx, dx);
            }
            if constexpr (W > 1) {
                if constexpr (P == 0) {
                    sh.step[lane] = ndx;
                    sh.norm[lane] = nerr;
                    sh.norm_state[lane] = ew;
                    sh.accept[lane] = accept;
                }
                tile_sync<W>();
                if constexpr (P != 0) {
                    ndx = sh.step[lane];
                    nerr = sh.norm[lane];
                    ew = sh.norm_state[lane];
                    accept = sh.accept[lane] != 0;
                }
            }
            if (at_end) {
                err = nerr;
                worst = ew;
                fail_steps = n;
                fail_x = x;
                fail_dx = accept ? dx : ndx;
                if (!accept) {
                    dx = ndx;
                    sg = 1;   // k1 is evaluated once per adaptive step
                    new_try = true;
                    if (dx < 1e-300) {
                        reason = 2;
                        done = true;
                    }
                } else {
                    x = exact_add(x, dx);
#pragma unroll
                    for (int i = 0; i < NS; ++i)
                        if (S::moves(i) && Q::own(i)) y[i] = yt[i];
                    step_dx = ndx;
                    // --- back in ODESolver::solve
                    if (exact_mul(exact_sub(x, xe), exact_sub(xe, xs)) >= 0) {
                        if (n > 0 && last) step_dx = dx_try0;
                        step = step_dx;
                        done = true;
                    }
                    ++n;
                    begin = true;
                }
            }
        }
        if (!done && !at_end) ++sg;
    }
    // the current at the end of the step: computeVariables at tEnd, whose
    // Iion the rates body computes too
    if constexpr (W > 1) {
#pragma unroll
        for (int i = 0; i < NS; ++i) {
            if (S::moves(i) && Q::own(i)) sh.y[buf][i][lane] = y[i];
            if (i == 0 && !SV && P == 0) sh.y[buf][0][lane] = y[0];
        }
        tile_sync<W>();
    }
    if constexpr (P == 0) {
        double d[NS], iion;
        if constexpr (W > 1) iion = rates(xe, SharedState{&sh.y[buf][0][lane]}, d);
        else iion = rates(xe, ArrayView<double>{y}, d);
        const double im = iion * M::IION_SCALE;
        if (live) {
            ++evals;
            if (!isfinite(im)) atomicOr(p.status, CFG_ERR_NONFINITE);
            if (p.im) p.im[cell] = im;
            p.step[c] = step;
        }
    }
    if (live) {
        if (reason != 0 && (worst < 0 ? P == 0 : Q::own(worst))) {
            // the thread that raised the flag first writes the record
            const int prev = atomicOr(p.status, CFG_ERR_ODE_STEPS);
            if (p.fail_record && !(prev & CFG_ERR_ODE_STEPS)) {
                double* r = p.fail_record;
                r[0] = double(cell); r[1] = reason; r[2] = fail_x; r[3] = fail_dx;
                r[4] = worst; r[5] = err; r[6] = worst >= 0 ? value_at(y, worst) : 0.0;
                r[7] = double(fail_steps);
            }
        }
#pragma unroll
        for (int i = 0; i < NS; ++i)
            if ((S::moves(i) && Q::own(i)) || (i == 0 && !SV && P == 0))
                p.yw[(long long)L::slot(i) * p.n + c] = y[i];
    }
    tile_sync<W>();   // the buffers are free for the next tile
}

// Tissue / single-cell ionic update of one PDE step for all cells (the plain
// FP64 form; the mixed form runs ionic_mixed_kernel).
// TISSUE > 0: every cell has that tissue flag and no per-cell scales, and the
// constants are compile-time values; TISSUE == 0: constants are evaluated per
// cell (per-cell tissue flags or conductance scales), W = 1.
// W = 1: each warp takes tiles in turn; W = 4: each block of 128 threads does.
template <class M, bool SV, int TISSUE, int W>
__global__ void __launch_bounds__(128, CFG_IONIC_MIN_BLOCKS) ionic_step_kernel(IonicLaunch p)
{
    __shared__ StepShared<M::NS, W> sh;
    unsigned evals = 0;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    // consecutive tiles go to different SMs
    const long long workers = W > 1 ? gridDim.x : (long long)gridDim.x * (blockDim.x >> 5);
    const long long first = W > 1 ? blockIdx.x : (long long)warp * gridDim.x + blockIdx.x;
    const long long tiles = (p.count + 31) / 32;
    for (long long t = first; t < tiles; t += workers) {
        const long long at = 32 * t + lane;
        const bool live = at < p.count;
        const long long c = p.first + (live ? at : p.count - 1);
        if constexpr (TISSUE > 0) {
            const ConstFold<double, M, TISSUE> K{};
            if constexpr (W == 1) {
                fp64_tile<M, SV, 1, 0>(p, K, TISSUE, c, live, sh, evals);
            } else {
                if (warp == 0) fp64_tile<M, SV, W, 0>(p, K, TISSUE, c, live, sh, evals);
                else if (warp == 1) fp64_tile<M, SV, W, 1>(p, K, TISSUE, c, live, sh, evals);
                else if (warp == 2) fp64_tile<M, SV, W, 2>(p, K, TISSUE, c, live, sh, evals);
                else fp64_tile<M, SV, W, 3>(p, K, TISSUE, c, live, sh, evals);
            }
        } else {
            const int tissue = p.tissue_cell ? int(p.tissue_cell[c]) : p.tissue;
            double C[M::NC] = {};   // the reference zero-fills CONSTANTS
            double yinit[M::NS] = {};
            double sc[6];
            const double* scp = nullptr;
            if (p.scales) {
#pragma unroll
                for (int j = 0; j < 6; ++j) sc[j] = p.scales[j * p.scale_stride + c];
                scp = sc;
            }
            M::init(C, yinit, tissue, scp);
            fp64_tile<M, SV, 1, 0>(p, ConstView<double>{C}, tissue, c, live, sh, evals);
        }
    }
    if (p.rhs_evals) {
        unsigned long long v = evals;
        for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
        if (lane == 0 && v) atomicAdd(p.rhs_evals, v);
    }
}

// Launch of the plain form's step.  Up to two tiles per SM, four warps share
// each tile: 32 to 4864 cells of ORd take 174 us (277 us with two tiles per SM)
// against 380 us with one warp per tile; from there on the shared tiles' larger
// sum of instructions loses (445 against 381 us at 305 tiles).  Beyond, two
// blocks of four warps per SM take the tiles in turn, consecutive tiles on
// different SMs, so that every SM ends within a tile of the others (1641 tiles,
// 52,500 cells of ORd: 1160 us; a block per tile, dealt by the hardware to
// whichever SM frees up first, 1840 us).  A shape set by the caller gives each
// block block * cells_per_thread cells' worth of tiles, one warp to a tile.
template <class M, bool SV, int T>
void launch_step(const IonicLaunch& p, cudaStream_t s, int block)
{
    const long long tiles = (p.count + 31) / 32;
    if (block > 0) {
        const long long cells = (long long)block * (p.cells_per_thread > 0 ? p.cells_per_thread : 1);
        const unsigned grid = unsigned((p.count + cells - 1) / cells);
        ionic_step_kernel<M, SV, T, 1><<<grid, block, 0, s>>>(p);
        return;
    }
    static const int sms = [] {   // of the device type
        int dev = 0, v = 0;
        if (cudaGetDevice(&dev) != cudaSuccess ||
            cudaDeviceGetAttribute(&v, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess)
            v = 152;
        return v;
    }();
    const unsigned grid = unsigned(tiles < 2 * sms ? tiles : 2 * sms);
    if constexpr (T > 0 && StepSplit<M, SV>::any_rest()) {
        if (tiles <= 2 * sms) {
            ionic_step_kernel<M, SV, T, 4><<<grid, 128, 0, s>>>(p);
            return;
        }
    }
    ionic_step_kernel<M, SV, T, 1><<<grid, 128, 0, s>>>(p);
}

// Initial states and constants for n cells (initConsts per cell).
template <class M, bool FP64>
__global__ void ionic_init_kernel(long long n, int tissue, const unsigned char* tissue_cell,
                                  const double* scales, long long scale_stride, double init_step,
                                  double* yw, float* yn, double* step)
{
    using L = Layout<M, FP64>;
    const long long c = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (c >= n) return;
    const int t = tissue_cell ? int(tissue_cell[c]) : tissue;
    double C[M::NC] = {};
    double y[M::NS] = {};   // states initConsts leaves unset are zero
    double sc[6];
    const double* scp = nullptr;
    if (scales) {
        for (int j = 0; j < 6; ++j) sc[j] = scales[j * scale_stride + c];
        scp = sc;
    }
    M::init(C, y, t, scp);
#pragma unroll
    for (int i = 0; i < M::NS; ++i) {
        if (FP64) {
            yw[(long long)L::slot(i) * n + c] = y[i];
        } else if (is_wide<M::WIDE_MASK>(i)) {
            // mixed form: the slot holds the FP32 pair (hi, lo) of the state
            const float hi = float(y[i]);
            reinterpret_cast<float2*>(yw)[(long long)L::slot(i) * n + c] =
                make_float2(hi, float(y[i] - double(hi)));
        } else {
            yn[(long long)L::slot(i) * n + c] = float(y[i]);
        }
    }
    step[c] = init_step;
}

}  // namespace cfg
