// RKF45 on a linear gate in closed form (tissue mode).
//
// While the PDE owns Vm, the rate of most gates is f(y) = a - b y with a and b
// fixed over the PDE step (LIN_MASK of a model, found by the emitter).  The
// six Fehlberg stages of a trial step h from y are then polynomials in
// z = -h b times k1 = f(y):
//
//   stage input   y + (h k1) q_s(z)      stage slope   k1 (1 + z q_s(z))
//   5th order     y + (h k1) u(z)        error         (h k1) e(z)
//
// so the gate needs neither stage slots nor a place in the stage loop's
// right-hand side.  e(z) has no terms below z^4 (the order conditions of the
// embedded pair): evaluated as a polynomial the error carries its own relative
// rounding only, where the sum of e_j k_j cancels to the rounding of its
// terms.  The coefficients are evaluated by the compiler in double.
#pragma once

#include "ionic_common.cuh"

namespace cfg {
namespace lingate {

struct Polys {
    double q[6][5] = {};   // [stage][power of z]
    double u[6] = {};      // 5th-order increment
    double e[6] = {};      // embedded error
};

constexpr Polys make_polys()
{
    using namespace rkf;
    const double a[6][5] = {{0, 0, 0, 0, 0},         {a21, 0, 0, 0, 0},
                            {a31, a32, 0, 0, 0},     {a41, a42, a43, 0, 0},
                            {a51, a52, a53, a54, 0}, {a61, a62, a63, a64, a65}};
    const double b[6] = {b1, 0, b3, b4, b5, b6}, e[6] = {e1, 0, e3, e4, e5, e6};
    double p[6][6] = {};   // stage slope over k1
    Polys r{};
    for (int s = 0; s < 6; ++s) {
        for (int j = 0; j < s; ++j)
            for (int k = 0; k < 5; ++k) r.q[s][k] += a[s][j] * p[j][k];
        p[s][0] = 1.0;
        for (int k = 0; k < 5; ++k) p[s][k + 1] += r.q[s][k];
    }
    for (int s = 0; s < 6; ++s)
        for (int k = 0; k < 6; ++k) {
            r.u[k] += b[s] * p[s][k];
            r.e[k] += e[s] * p[s][k];
        }
    return r;
}

constexpr Polys kPolys = make_polys();

constexpr bool small(double v) { return v < 1e-15 && v > -1e-15; }
static_assert(small(kPolys.e[0]) && small(kPolys.e[1]) && small(kPolys.e[2]) &&
                  small(kPolys.e[3]),
              "the embedded pair's error starts at z^4");

CFG_D __forceinline__ double fma_r(double a, double b, double c) { return __fma_rn(a, b, c); }

// single coefficients as scalar constants (device code cannot index kPolys)
template <int S, int K>
constexpr double q_coef = kPolys.q[S][K];
template <int K>
constexpr double u_coef = kPolys.u[K];
template <int K>
constexpr double e_coef = kPolys.e[K];

// q_S(z) of one stage, its degree S - 1, by Horner's rule from power K up
template <int S, class R, int K = 0>
CFG_D __forceinline__ R stage_poly(R z)
{
    if constexpr (K == S - 1) return R(q_coef<S, K>);
    else return fma_r(stage_poly<S, R, K + 1>(z), z, R(q_coef<S, K>));
}

template <class R, int K = 0>
CFG_D __forceinline__ R increment_poly(R z)
{
    if constexpr (K == 5) return R(u_coef<K>);
    else return fma_r(increment_poly<R, K + 1>(z), z, R(u_coef<K>));
}

template <class R>
CFG_D __forceinline__ R error_poly(R z)
{
    const R z2 = z * z;
    return (z2 * z2) * fma_r(R(e_coef<5>), z, R(e_coef<4>));
}

}  // namespace lingate

// The linear gates among a model's states in tissue mode: they follow the
// polynomials above.  State 0 (Vm) does not change, the others go through the
// stage slots.
template <class M>
struct TissueSplit {
    static CFG_HD constexpr bool lin(int i) { return i > 0 && ((M::LIN_MASK >> i) & 1ull); }
};

}  // namespace cfg
