// Implicit diffusion of one monodomain step as ONE persistent kernel: every
// PIMPLE corrector and every PCG iteration of the step runs inside a single
// cooperative launch whose blocks meet at grid barriers, instead of two to
// four kernel launches per iteration.
//
// The numerics are those of the per-kernel path (diffusion.cu): the same
// right-hand side, lduMatrix::Amul order, normFactor, L1 residual,
// convergence test and PIMPLE residual control.  Two things change:
//   * each thread owns a fixed set of rows for the whole step, so its own
//     entries of x, r, p, b, A.x and A.p are only ever touched by it; z and
//     x (read at the neighbours) and the reduction partials cross blocks,
//     and those are read through L2 (ld.global.cg), which is coherent;
//   * A.p is updated as A.z + beta A.p, so one halo exchange (of z) serves
//     both the new direction and its product, and an iteration needs two
//     grid sums, each of which is its own barrier (grid_sync.cuh).  GB300
//     executes FP64 at 1/64 of the FP32 rate, so the FP64 instruction count
//     per row (15 per PCG iteration here) and the sums set the speed of
//     the solve, not HBM: its vectors stay in L2.
//
// Two further savings leave the bits alone: sum(x) of the next corrector's
// normFactor is formed with the last update of x, and its residual, normFactor
// and z in one pass, where each had a pass and a barrier; and a corrector
// whose predecessor needed no iteration and had the same right-hand side is
// that predecessor again (same x, same b), so its recorded result is repeated.
// Measured per step, before and after all of this: 3,360 cells in FP64 95 to
// 46 us, 52,500 in FP64 114 to 72 us, 420,000 in float pairs 133 to 111 us
// (steady state, 3 + 0 + 0 iterations), a ventricle of 563,616 tetrahedra with its
// corrections 379 to 301 us in FP64, the default there, and 299 to 265 in float
// pairs.
//
// On a general mesh every corrector first forms the cell gradient of the
// iterate (one more barrier) for the explicit correction of the Laplacian
// in the source.
//
// k_implicit_pair is the same solve with the PCG in float pairs (the mixed
// form's default on meshes without explicit corrections).
//
// Grid barriers are cooperative-launch safe (all blocks co-resident) and
// bounded: a block that waits longer than the context's spin limit (~1 s by
// default) sets an abort flag, every block leaves at its next sum, and
// the step reports CFG_ERR_PCG.
#include <cuda_runtime.h>

#include "diffusion_kernels.cuh"
#include "grid_sync.cuh"

namespace cfg {

namespace {

// threads of the largest block: FP64 (tetrahedral rows and pairs: twice that)
constexpr int kCoopBlock = 512;
constexpr int kWideBlock = 1024;

// x / d for 0 <= x < 2^31 by multiply-high (round-up method): avoids the
// 64-bit integer division of a cell index in every stencil row.
struct FastDiv {
    unsigned m, s;
};

__device__ __forceinline__ unsigned fdiv(unsigned x, FastDiv f)
{
    return (__umulhi(x, f.m) + x) >> f.s;
}

}  // namespace

struct CoopArgs {
    FastDiv div_nx, div_ny;   // stencil form only
};

// A.q for row c (diag*q_c, then each -coef*q_nb in column order), q read
// through L2.  Stencil neighbours come from (i, j, k) = row decomposition.
template <int W>
__device__ __forceinline__ double amul_cg(const DiffusionArgs& a, const CoopArgs& ca,
                                          unsigned c, double d, const double* q)
{
    double acc = d * __ldcg(&q[c]);
    if (a.sx) {
        const unsigned nx = unsigned(a.sx), nxy = nx * unsigned(a.sy);
        const unsigned line = fdiv(c, ca.div_nx), i = c - line * nx;
        const unsigned k = fdiv(line, ca.div_ny), j = line - k * unsigned(a.sy);
        if (k > 0) acc += (-a.cz) * __ldcg(&q[c - nxy]);
        if (j > 0) acc += (-a.cy) * __ldcg(&q[c - nx]);
        if (i > 0) acc += (-a.cx) * __ldcg(&q[c - 1]);
        if (i + 1 < nx) acc += (-a.cx) * __ldcg(&q[c + 1]);
        if (j + 1 < unsigned(a.sy)) acc += (-a.cy) * __ldcg(&q[c + nx]);
        if (k + 1 < unsigned(a.sz)) acc += (-a.cz) * __ldcg(&q[c + nxy]);
    } else if constexpr (W > 0) {
        // padded slots: coefficient 0 and column 0, an exact zero term
#pragma unroll
        for (int e = 0; e < W; ++e)
            acc += (-ld_stream(&a.ell_coef[(long long)e * a.n + c])) *
                   __ldcg(&q[ld_stream(&a.ell_col[(long long)e * a.n + c])]);
    } else {
        const int cnt = a.ell_cnt[c];
        for (int e = 0; e < cnt; ++e)
            acc += (-a.ell_coef[(long long)e * a.n + c]) *
                   __ldcg(&q[a.ell_col[(long long)e * a.n + c]]);
    }
    return acc;
}

// The whole implicit diffusion of one step (all correctors, all PCG
// iterations) and the activation-time update.  Launched cooperatively with
// every block resident; rows are strided over the grid, two per loop trip so
// that two independent FP64 chains are in flight per thread.
//
// PCG iteration with two grid barriers (lduMatrix PCG in exact arithmetic):
//   halo pass:   w = A.z (z of the neighbours through L2), p = z + beta p,
//                A.p = w + beta A.p (linearity of A), sum p.A.p  | barrier
//   update pass: x += alpha p, r -= alpha A.p, z = D^-1 r (published for
//                the next halo pass), sums |r| and z.r           | barrier
template <class CR, int W>
__global__ void __launch_bounds__(W == 4 ? kWideBlock : kCoopBlock, 1)
    k_implicit_coop(DiffusionArgs a, CoopArgs ca)
{
    constexpr int kBlock = W == 4 ? kWideBlock : kCoopBlock;
    PcgState* st = a.st;
    const unsigned n = unsigned(a.n);
    const unsigned stride = gridDim.x * blockDim.x;
    const unsigned first = blockIdx.x * blockDim.x + threadIdx.x;
    const bool lead = blockIdx.x == 0 && threadIdx.x == 0;
    // values every block reads before block 0 may update them
    int n_old = st->n_old;
    const double t_step = st->t, t0 = st->t0;
    const double tol = st->tol, rel_tol = st->rel_tol, outer_tol = st->outer_tol;
    const int max_iter = st->max_iter, n_outer = st->n_outer;
    double* __restrict__ x = a.vm;
    double* __restrict__ b = a.b;
    double* __restrict__ ax = a.ax;
    double* __restrict__ r = a.r;
    double* __restrict__ z = a.z;     // published: read by neighbours
    double* __restrict__ p = a.pA;    // own rows only
    double* __restrict__ ap = a.ap;   // own rows only
    gsync::Exchange* const xch = a.xch;
    unsigned arrivals = 0;   // at the sums, each a grid barrier
    int set = 0;
    const auto sum = [&](auto& v) {
        constexpr int K = sizeof(v) / sizeof(v[0]);
        return gsync::sync_sums<kBlock, K, gsync::SumDouble>(xch, &st->bar_abort, arrivals, set,
                                                                 a.spin_limit, v);
    };
    const auto meet = [&] {
        fp::P none[1] = {fp::make(0.0f)};
        return gsync::sync_sums<kBlock, 1, gsync::SumPair>(xch, &st->bar_abort, arrivals, set,
                                                               a.spin_limit, none);
    };
    int n_solves = 0, status = 0;
    bool converged_outer = false, abort_step = false;
    long long step_iters = 0;
    double last_init = 0.0, last_res = 0.0;
    int last_iter = 0, last_v = 0;
    int bsrc_variant = -1;            // ddt coefficient set of the kept source
    double sum_x = 0.0;               // of the iterate, once an update pass has added it up
    bool have_sum = false;

    for (int corr = 1;; ++corr) {
        const int v = ddt_variant(a, n_old);
        double init_res = last_init, res = last_res;
        int iter = 0;
        bool aborted = false;
        // a corrector that took no iteration left the iterate, so the one
        // after it with the same coefficients repeats it number for number
        if (corr == 1 || v != last_v || last_iter > 0) {
            const double* __restrict__ diag = a.diag2 + size_t(v) * n;
            const double* __restrict__ rdiag = a.rdiag2 + size_t(v) * n;
            const double* __restrict__ sumA = a.sumA2 + size_t(v) * n;
            const double cft0 = a.cft0[v], cft00 = a.cft00[v];
            // --- general mesh: gradient of the current iterate for the
            // Laplacian's explicit correction, published for the neighbours
            CR* __restrict__ grad = static_cast<CR*>(a.grad);
            if (a.nc_gw) {
                for (unsigned c = first; c < n; c += stride) {
                    CR g[3];
                    nc_gradient<CR, W>(a, c, [x](long long q) { return __ldcg(&x[q]); }, g);
                    __stcg(&grad[c], g[0]);
                    __stcg(&grad[size_t(n) + c], g[1]);
                    __stcg(&grad[2 * size_t(n) + c], g[2]);
                }
                if (!meet()) { abort_step = true; break; }
            }
            // --- source, A.x, r = b - A.x; sums of x and |r|.  The ddt, ionic
            // and stimulus parts of the source change between correctors only
            // with the ddt coefficient set (the first step creates the old-time
            // levels in its first corrector): kept in bsrc for the others.
            double s1[3] = {0.0, 0.0, 0.0};
            const bool fresh = corr == 1 || v != bsrc_variant;
            bsrc_variant = v;
            auto rhs_row = [&](unsigned c) {
                double rhs;
                if (fresh) {
                    const double V = a.vol[c];
                    double ddt_src;
                    if (a.ddt_backward)
                        ddt_src = a.rdt * V * (cft0 * a.vm_old[c] - cft00 * a.vm_oldold[c]);
                    else
                        ddt_src = a.rdt * a.vm_old[c] * V;
                    double bb = a.chicm * ddt_src;
                    double su = -(a.chicm * a.iion[c]) * V;
                    su = su + box_source(a, c, t0) * V;
                    rhs = bb + su;
                    a.bsrc[c] = rhs;
                } else {
                    rhs = a.bsrc[c];
                }
                if (a.nc_gw)
                    rhs = rhs + nc_correction<CR, W>(a, c, [grad, n](long long q, int k) {
                              return __ldcg(&grad[size_t(k) * n + size_t(q)]);
                          });
                return rhs;
            };
            // normFactor's terms of row c and z = D^-1 r with its z.r, in the same
            // pass as the residual when the mean of the iterate is known
            double avg = have_sum ? sum_x / double(n) : 0.0;
            const auto norm_row = [&](unsigned c, double mean, double axc, double bc, double rc,
                                      double& nf, double& zr) {
                const double pa = sumA[c] * mean;
                nf += fabs(axc - pa) + fabs(bc - pa);
                const double zc = rdiag[c] * rc;
                __stcg(&z[c], zc);
                zr += zc * rc;
            };
            for (unsigned c = first; c < n; c += 2 * stride) {
                const unsigned c2 = c + stride;
                const bool two = c2 < n;
                const double b0 = rhs_row(c), b1 = two ? rhs_row(c2) : 0.0;
                const double a0 = amul_cg<W>(a, ca, c, diag[c], x);
                const double a1 = two ? amul_cg<W>(a, ca, c2, diag[c2], x) : 0.0;
                const double r0 = b0 - a0, r1 = b1 - a1;
                r[c] = r0;
                s1[1] += fabs(r0);
                if (two) {
                    r[c2] = r1;
                    s1[1] += fabs(r1);
                }
                if (have_sum) {
                    norm_row(c, avg, a0, b0, r0, s1[0], s1[2]);
                    if (two) norm_row(c2, avg, a1, b1, r1, s1[0], s1[2]);
                } else {
                    b[c] = b0; ax[c] = a0;
                    s1[0] += x[c];
                    if (two) {
                        b[c2] = b1; ax[c2] = a1;
                        s1[0] += x[c2];
                    }
                }
            }
            if (!sum(s1)) { abort_step = true; break; }
            // fvm::ddt created the old time levels
            if (n_old < 1) n_old = 1;
            if (a.ddt_backward && n_old < 2) n_old = 2;
            // --- normFactor, z = D^-1 r (published), z.r
            double s2[2] = {s1[0], s1[2]};
            if (!have_sum) {
                avg = s1[0] / double(n);
                s2[0] = s2[1] = 0.0;
                for (unsigned c = first; c < n; c += stride)
                    norm_row(c, avg, ax[c], b[c], r[c], s2[0], s2[1]);
                if (!sum(s2)) { abort_step = true; break; }
            }
            const double normf = s2[0] + 1e-20;
            init_res = s1[1] / normf;
            res = init_res;
            double wArA = s2[1], beta = 0.0;
            const auto conv = [&](double rr) {
                return rr < tol || (rel_tol > 1e-20 && rr < rel_tol * init_res);
            };
            if (!conv(res)) {
                for (;;) {
                    // --- halo pass: w = A.z, p = z + beta p, A.p = w + beta A.p
                    double s3[1] = {0.0};
                    const bool first_it = iter == 0;
                    for (unsigned c = first; c < n; c += 2 * stride) {
                        const unsigned c2 = c + stride;
                        const bool two = c2 < n;
                        const double w0 = amul_cg<W>(a, ca, c, diag[c], z);
                        const double w1 = two ? amul_cg<W>(a, ca, c2, diag[c2], z) : 0.0;
                        const double z0 = __ldcg(&z[c]);
                        const double z1 = two ? __ldcg(&z[c2]) : 0.0;
                        double p0, p1, q0, q1;
                        if (first_it) {
                            p0 = z0; p1 = z1; q0 = w0; q1 = w1;
                        } else {
                            p0 = z0 + beta * p[c];
                            q0 = w0 + beta * ap[c];
                            p1 = two ? z1 + beta * p[c2] : 0.0;
                            q1 = two ? w1 + beta * ap[c2] : 0.0;
                        }
                        p[c] = p0; ap[c] = q0;
                        s3[0] += q0 * p0;
                        if (two) {
                            p[c2] = p1; ap[c2] = q1;
                            s3[0] += q1 * p1;
                        }
                    }
                    if (!sum(s3)) { aborted = true; break; }
                    const double(&g3)[1] = s3;
                    // checkSingularity and alpha, once per block
                    double q3[2];
                    gsync::block_scalars<2>(0, q3, [&](int k) {
                        return k == 0 ? (fabs(g3[0]) / normf < 1e-300 ? 1.0 : 0.0) : wArA / g3[0];
                    });
                    if (q3[0] != 0.0) break;
                    const double alpha = q3[1];
                    // --- update pass: x, r, z; |r|, z.r and the sum of x
                    double s4[3] = {0.0, 0.0, 0.0};
                    for (unsigned c = first; c < n; c += 2 * stride) {
                        const unsigned c2 = c + stride;
                        const bool two = c2 < n;
                        const double x0 = x[c] + alpha * p[c];
                        const double r0 = r[c] - alpha * ap[c];
                        const double z0 = rdiag[c] * r0;
                        x[c] = x0; r[c] = r0;
                        __stcg(&z[c], z0);
                        s4[0] += fabs(r0);
                        s4[1] += z0 * r0;
                        s4[2] += x0;
                        if (two) {
                            const double x1 = x[c2] + alpha * p[c2];
                            const double r1 = r[c2] - alpha * ap[c2];
                            const double z1 = rdiag[c2] * r1;
                            x[c2] = x1; r[c2] = r1;
                            __stcg(&z[c2], z1);
                            s4[0] += fabs(r1);
                            s4[1] += z1 * r1;
                            s4[2] += x1;
                        }
                    }
                    if (!sum(s4)) { aborted = true; break; }
                    const double(&g4)[3] = s4;
                    sum_x = g4[2];
                    have_sum = true;
                    // the residual and beta, once per block
                    double q4[2];
                    gsync::block_scalars<2>(1, q4, [&](int k) {
                        return k == 0 ? g4[0] / normf : g4[1] / wArA;
                    });
                    res = q4[0];
                    ++iter;
                    ++step_iters;
                    if (conv(res) || iter >= max_iter) {
                        if (!conv(res)) status |= CFG_ERR_PCG;
                        break;
                    }
                    if (step_iters >= a.iter_cap) {
                        // guard of the in-kernel loops: give up the step
                        status |= CFG_ERR_PCG;
                        aborted = true;
                        break;
                    }
                    wArA = g4[1];
                    beta = q4[1];
                }
            }
        }
        if (lead && n_solves < kMaxSolves) {
            st->iters[n_solves] = iter;
            st->init_r[n_solves] = init_res;
            st->final_r[n_solves] = res;
        }
        ++n_solves;
        last_init = init_res; last_res = res; last_iter = iter; last_v = v;
        if (aborted) { abort_step = true; break; }
        // pimpleLoop: the corrector after a converged one is the last
        if (converged_outer || corr + 1 > n_outer) break;
        if (init_res < outer_tol) converged_outer = true;
        // the next corrector reads other blocks' rows of x only through
        // amul_cg (L2), after the last barrier of this one
    }
    // --- activation time (MyocardiumDomain::updateActivationTime)
    if (abort_step) status |= CFG_ERR_PCG;
    else
        for (unsigned c = first; c < n; c += stride)
            activation(a, c, x[c], a.vm_old[c], t_step - a.dt);
    if (lead) {
        st->n_old = n_old;
        st->n_solves = n_solves;
        st->iter = last_iter;
        st->init_res = last_init;
        st->res = last_res;
        st->variant = last_v;
        st->step_iters = step_iters;
        st->corr = n_solves + 1;
        st->solve_active = 0;
        st->outer_active = 0;
        st->converged_outer = converged_outer ? 1 : 0;
    }
    if (status && threadIdx.x == 0) atomicOr(&st->status, status);
}

// ---------------------------------------------------------------- float pairs
// The same solve with the PCG in float pairs (the mixed form): the operator,
// the source and every vector of the iteration as (hi, lo) pairs on the FP32
// pipe, the system scaled by 2^pair_shift so that its quantities sit well
// inside the float range.  The corrector's source is formed in FP64 as above
// (once per corrector) and split; the iterate x is published as a pair (px)
// for the neighbours and written back to Vm in FP64 after each solve.  The
// scalars (alpha, beta, the residuals) are formed by every thread from the
// same block-order sums, so every block takes the same decisions without a
// shared-memory broadcast.

template <int W, class F>
__device__ __forceinline__ fp::P amul_pair(const DiffusionArgs& a, const CoopArgs& ca, unsigned c,
                                           fp::P d, F q)
{
    fp::Acc acc;
    acc.add_prod(d, q(c));
    if (a.sx) {
        const unsigned nx = unsigned(a.sx), nxy = nx * unsigned(a.sy);
        const unsigned line = fdiv(c, ca.div_nx), i = c - line * nx;
        const unsigned k = fdiv(line, ca.div_ny), j = line - k * unsigned(a.sy);
        if (k > 0) acc.sub_prod(a.pcz, q(c - nxy));
        if (j > 0) acc.sub_prod(a.pcy, q(c - nx));
        if (i > 0) acc.sub_prod(a.pcx, q(c - 1));
        if (i + 1 < nx) acc.sub_prod(a.pcx, q(c + 1));
        if (j + 1 < unsigned(a.sy)) acc.sub_prod(a.pcy, q(c + nx));
        if (k + 1 < unsigned(a.sz)) acc.sub_prod(a.pcz, q(c + nxy));
    } else if constexpr (W > 0) {
#pragma unroll
        for (int e = 0; e < W; ++e)
            acc.sub_prod(ld_stream(&a.pcoef[(long long)e * a.n + c]),
                         q(unsigned(ld_stream(&a.ell_col[(long long)e * a.n + c]))));
    } else {
        const int cnt = a.ell_cnt[c];
        for (int e = 0; e < cnt; ++e)
            acc.sub_prod(a.pcoef[(long long)e * a.n + c],
                         q(unsigned(a.ell_col[(long long)e * a.n + c])));
    }
    return acc.value();
}

template <class CR, int W>
__global__ void __launch_bounds__(kWideBlock, 1) k_implicit_pair(DiffusionArgs a, CoopArgs ca)
{
    constexpr int kBlock = kWideBlock;
    using fp::P;
    PcgState* st = a.st;
    const unsigned n = unsigned(a.n);
    const unsigned stride = gridDim.x * blockDim.x;
    const unsigned first = blockIdx.x * blockDim.x + threadIdx.x;
    const bool lead = blockIdx.x == 0 && threadIdx.x == 0;
    int n_old = st->n_old;
    const double t_step = st->t, t0 = st->t0;
    const bool use_rel = st->rel_tol > 1e-20;
    const P tol = fp::split(st->tol), outer_tol = fp::split(st->outer_tol);
    const P rel = fp::split(st->rel_tol);
    const int max_iter = st->max_iter, n_outer = st->n_outer;
    const int sh = a.pair_shift;
    // the ratio sum|r| / normFactor is scale free when the small number
    // lduMatrix adds to normFactor is scaled with the system
    const P small = fp::split(1e-20, sh);
    const P count = fp::split(double(n));
    double* __restrict__ x = a.vm;
    P* __restrict__ px = a.px;                          // published
    P* __restrict__ b = reinterpret_cast<P*>(a.b);
    P* __restrict__ ax = reinterpret_cast<P*>(a.ax);
    P* __restrict__ r = reinterpret_cast<P*>(a.r);
    P* __restrict__ z = reinterpret_cast<P*>(a.z);      // published
    P* __restrict__ p = reinterpret_cast<P*>(a.pA);
    P* __restrict__ ap = reinterpret_cast<P*>(a.ap);
    gsync::Exchange* const xch = a.xch;
    unsigned arrivals = 0;   // at the sums, each a grid barrier
    int set = 0;
    const auto sum = [&](auto& v) {
        constexpr int K = sizeof(v) / sizeof(v[0]);
        return gsync::sync_sums<kBlock, K, gsync::SumPair>(xch, &st->bar_abort, arrivals, set,
                                                                 a.spin_limit, v);
    };
    const auto meet = [&] {
        P none[1] = {fp::make(0.0f)};
        return sum(none);
    };
    int n_solves = 0, status = 0;
    bool converged_outer = false, abort_step = false;
    long long step_iters = 0;
    P last_init = fp::make(0.0f), last_res = fp::make(0.0f);
    int last_iter = 0, last_v = 0;
    int bsrc_variant = -1;
    P sum_x = fp::make(0.0f);   // of the iterate, once an update pass has added it up
    bool have_sum = false;

    for (int corr = 1;; ++corr) {
        const int v = ddt_variant(a, n_old);
        P init_res = last_init, res = last_res;
        int iter = 0;
        bool aborted = false;
        // a corrector that took no iteration left the iterate, so the one
        // after it with the same coefficients repeats it number for number
        if (corr == 1 || v != last_v || last_iter > 0) {
            const P* __restrict__ diag = a.pdiag2 + size_t(v) * n;
            const P* __restrict__ rdiag = a.prdiag2 + size_t(v) * n;
            const P* __restrict__ sumA = a.psumA2 + size_t(v) * n;
            const double cft0 = a.cft0[v], cft00 = a.cft00[v];
            // the iterate of the neighbours: Vm itself in the first corrector,
            // the published pair afterwards
            const bool from_vm = corr == 1;
            const auto xq = [x, px, from_vm](unsigned q) {
                return from_vm ? fp::split(__ldcg(&x[q])) : __ldcg(&px[q]);
            };
            CR* __restrict__ grad = static_cast<CR*>(a.grad);
            if (a.nc_gw) {
                for (unsigned c = first; c < n; c += stride) {
                    CR g[3];
                    nc_gradient<CR, W>(a, c, [&xq](long long q) { return xq(unsigned(q)); }, g);
                    __stcg(&grad[c], g[0]);
                    __stcg(&grad[size_t(n) + c], g[1]);
                    __stcg(&grad[2 * size_t(n) + c], g[2]);
                }
                if (!meet()) { abort_step = true; break; }
            }
            // --- source (FP64, split), A.x, r = b - A.x; sums of x and |r|
            P s1[3] = {fp::make(0.0f), fp::make(0.0f), fp::make(0.0f)};
            const bool fresh = corr == 1 || v != bsrc_variant;
            bsrc_variant = v;
            const auto row_rhs = [&](unsigned c) {
                double rhs;
                if (fresh) {
                    const double V = a.vol[c];
                    double ddt_src;
                    if (a.ddt_backward)
                        ddt_src = a.rdt * V * (cft0 * a.vm_old[c] - cft00 * a.vm_oldold[c]);
                    else
                        ddt_src = a.rdt * a.vm_old[c] * V;
                    double bb = a.chicm * ddt_src;
                    double su = -(a.chicm * a.iion[c]) * V;
                    su = su + box_source(a, c, t0) * V;
                    rhs = bb + su;
                    a.bsrc[c] = rhs;
                } else {
                    rhs = a.bsrc[c];
                }
                if (a.nc_gw)
                    rhs = rhs + nc_correction<CR, W>(a, c, [grad, n](long long q, int k) {
                              return __ldcg(&grad[size_t(k) * n + size_t(q)]);
                          });
                return fp::split(rhs, sh);
            };
            // normFactor's terms of a row and z = D^-1 r (published) with its z.r,
            // in the same pass as the residual when the mean of the iterate is known
            P avg = have_sum ? fp::div(sum_x, count) : fp::make(0.0f);
            const auto norm_row = [&](unsigned c, P sa, P axc, P bc, P rc, P m, P& nf, P& zr) {
                const P pa = fp::mul(sa, avg);
                nf = fp::add(nf, fp::add(fp::abs(fp::sub(axc, pa)), fp::abs(fp::sub(bc, pa))));
                const P zc = fp::mul(m, rc);
                __stcg(&z[c], zc);
                zr = fp::madd(zc, rc, zr);
            };
            const auto row_res = [&](unsigned c, P bc, P axc) {
                const P rc = fp::sub(bc, axc);
                r[c] = rc;
                s1[1] = fp::add(s1[1], fp::abs(rc));
                if (have_sum) {
                    norm_row(c, sumA[c], axc, bc, rc, rdiag[c], s1[0], s1[2]);
                } else {
                    const P xc = xq(c);
                    b[c] = bc; ax[c] = axc;
                    if (from_vm) __stcg(&px[c], xc);
                    s1[0] = fp::add(s1[0], xc);
                }
            };
            for (unsigned c = first; c < n; c += 2 * stride) {
                const unsigned c2 = c + stride;
                const bool two = c2 < n;
                const P b0 = row_rhs(c);
                const P b1 = two ? row_rhs(c2) : fp::make(0.0f);
                const P a0 = amul_pair<W>(a, ca, c, diag[c], xq);
                const P a1 = two ? amul_pair<W>(a, ca, c2, diag[c2], xq) : fp::make(0.0f);
                row_res(c, b0, a0);
                if (two) row_res(c2, b1, a1);
            }
            if (!sum(s1)) { abort_step = true; break; }
            if (n_old < 1) n_old = 1;
            if (a.ddt_backward && n_old < 2) n_old = 2;
            // --- normFactor, z = D^-1 r (published), z.r
            P s2[2] = {s1[0], s1[2]};
            if (!have_sum) {
                avg = fp::div(s1[0], count);
                s2[0] = s2[1] = fp::make(0.0f);
                for (unsigned c = first; c < n; c += 2 * stride) {
                    const unsigned c2 = c + stride;
                    const bool two = c2 < n;
                    const unsigned d = two ? c2 : c;
                    const P sa0 = sumA[c], sa1 = sumA[d], a0 = ax[c], a1 = ax[d], b0 = b[c], b1 = b[d];
                    const P r0 = r[c], r1 = r[d], m0 = rdiag[c], m1 = rdiag[d];
                    norm_row(c, sa0, a0, b0, r0, m0, s2[0], s2[1]);
                    if (two) norm_row(c2, sa1, a1, b1, r1, m1, s2[0], s2[1]);
                }
                if (!sum(s2)) { abort_step = true; break; }
            }
            const P normf = fp::add(s2[0], small);
            init_res = fp::div(s1[1], normf);
            const P rel_init = fp::mul(rel, init_res);
            res = init_res;
            P wArA = s2[1], beta = fp::make(0.0f);
            const auto conv = [&](P rr) {
                return fp::less(rr, tol) || (use_rel && fp::less(rr, rel_init));
            };
            if (!conv(res)) {
                for (;;) {
                    // --- halo pass: w = A.z, p = z + beta p, A.p = w + beta A.p
                    P s3[1] = {fp::make(0.0f)};
                    const bool first_it = iter == 0;
                    const auto zq = [z](unsigned q) { return __ldcg(&z[q]); };
                    const auto dir = [&](unsigned c, P w) {
                        const P zc = __ldcg(&z[c]);
                        P pc = zc, qc = w;
                        if (!first_it) {
                            pc = fp::madd(beta, p[c], zc);
                            qc = fp::madd(beta, ap[c], w);
                        }
                        p[c] = pc; ap[c] = qc;
                        s3[0] = fp::madd(qc, pc, s3[0]);
                    };
                    // two rows per trip: both products' loads are in flight together
                    for (unsigned c = first; c < n; c += 2 * stride) {
                        const unsigned c2 = c + stride;
                        const bool two = c2 < n;
                        const P w0 = amul_pair<W>(a, ca, c, diag[c], zq);
                        const P w1 = two ? amul_pair<W>(a, ca, c2, diag[c2], zq) : fp::make(0.0f);
                        dir(c, w0);
                        if (two) dir(c2, w1);
                    }
                    if (!sum(s3)) { aborted = true; break; }
                    const P(&g3)[1] = s3;
                    if (g3[0].x == 0.0f) break;   // checkSingularity
                    const P alpha = fp::div(wArA, g3[0]);
                    const P nalpha = fp::neg(alpha);
                    // --- update pass: x, r, z; |r|, z.r and the sum of x
                    P s4[3] = {fp::make(0.0f), fp::make(0.0f), fp::make(0.0f)};
                    // two rows per trip, all of their loads issued first (the
                    // pass streams from HBM when the vectors exceed L2)
                    for (unsigned c = first; c < n; c += 2 * stride) {
                        const unsigned c2 = c + stride;
                        const bool two = c2 < n;
                        const unsigned d = two ? c2 : c;
                        const P p0 = p[c], p1 = p[d], q0 = ap[c], q1 = ap[d];
                        const P r0 = r[c], r1 = r[d], x0 = __ldcg(&px[c]), x1 = __ldcg(&px[d]);
                        const P m0 = rdiag[c], m1 = rdiag[d];
                        const P xc = fp::madd(alpha, p0, x0);
                        __stcg(&px[c], xc);
                        s4[2] = fp::add(s4[2], xc);
                        const P rc = fp::madd(nalpha, q0, r0);
                        r[c] = rc;
                        const P zc = fp::mul(m0, rc);
                        __stcg(&z[c], zc);
                        s4[0] = fp::add(s4[0], fp::abs(rc));
                        s4[1] = fp::madd(zc, rc, s4[1]);
                        if (two) {
                            const P xd = fp::madd(alpha, p1, x1);
                            __stcg(&px[c2], xd);
                            s4[2] = fp::add(s4[2], xd);
                            const P rd = fp::madd(nalpha, q1, r1);
                            r[c2] = rd;
                            const P zd = fp::mul(m1, rd);
                            __stcg(&z[c2], zd);
                            s4[0] = fp::add(s4[0], fp::abs(rd));
                            s4[1] = fp::madd(zd, rd, s4[1]);
                        }
                    }
                    if (!sum(s4)) { aborted = true; break; }
                    const P(&g4)[3] = s4;
                    sum_x = g4[2];
                    have_sum = true;
                    res = fp::div(g4[0], normf);
                    ++iter;
                    ++step_iters;
                    if (conv(res) || iter >= max_iter) {
                        if (!conv(res)) status |= CFG_ERR_PCG;
                        break;
                    }
                    if (step_iters >= a.iter_cap) {
                        status |= CFG_ERR_PCG;
                        aborted = true;
                        break;
                    }
                    beta = fp::div(g4[1], wArA);
                    wArA = g4[1];
                }
            }
        }
        if (lead && n_solves < kMaxSolves) {
            st->iters[n_solves] = iter;
            st->init_r[n_solves] = fp::join(init_res);
            st->final_r[n_solves] = fp::join(res);
        }
        ++n_solves;
        last_init = init_res; last_res = res; last_iter = iter; last_v = v;
        if (aborted) { abort_step = true; break; }
        if (converged_outer || corr + 1 > n_outer) break;
        if (fp::less(init_res, outer_tol)) converged_outer = true;
    }
    if (abort_step) status |= CFG_ERR_PCG;
    else
        // the step's iterate back into Vm (own rows: between correctors the
        // neighbours read px, so Vm is written once), and the activation time
        for (unsigned c = first; c < n; c += stride) {
            const double xc = fp::join(__ldcg(&px[c]));
            x[c] = xc;
            activation(a, c, xc, a.vm_old[c], t_step - a.dt);
        }
    if (lead) {
        st->n_old = n_old;
        st->n_solves = n_solves;
        st->iter = last_iter;
        st->init_res = fp::join(last_init);
        st->res = fp::join(last_res);
        st->variant = last_v;
        st->step_iters = step_iters;
        st->corr = n_solves + 1;
        st->solve_active = 0;
        st->outer_active = 0;
        st->converged_outer = converged_outer ? 1 : 0;
    }
    if (status && threadIdx.x == 0) atomicOr(&st->status, status);
}

// Host helpers: fast-division constants and the cooperative launch.
static FastDiv make_fastdiv(unsigned d)
{
    unsigned s = 0;
    while ((1ull << s) < d) ++s;
    const unsigned long long m = ((1ull << 32) * ((1ull << s) - d)) / d + 1;
    return FastDiv{unsigned(m), s};
}

// rows of a general mesh are visited over the full ELL width when it is 4
// (tetrahedra) or 6 (hexahedra); CR is the type the explicit correction's
// arrays are kept in, by the ionic form and not by the PCG's arithmetic
template <class CR>
static void* coop_kernel_of(bool pair, int w)
{
    if (pair)
        return w == 4   ? (void*)k_implicit_pair<CR, 4>
               : w == 6 ? (void*)k_implicit_pair<CR, 6>
                        : (void*)k_implicit_pair<CR, 0>;
    return w == 4   ? (void*)k_implicit_coop<CR, 4>
           : w == 6 ? (void*)k_implicit_coop<CR, 6>
                    : (void*)k_implicit_coop<CR, 0>;
}

static void* coop_kernel(bool pair, bool nc_fp32, int w)
{
    return nc_fp32 ? coop_kernel_of<float>(pair, w) : coop_kernel_of<double>(pair, w);
}

// Block size and grid of a kernel for n rows, one block per SM: the smallest
// block with which every row has a thread, so that a small system is spread
// over all SMs (3,360 rows in FP64: 64 us a step in blocks of 512, seven SMs'
// FP64 units), else the kernel's largest, whose threads take rows in turn.  A
// block per SM rather than two of half the size: half as many blocks to meet
// (420,000 rows of pairs: 111 against 117 us).  The two largest kernels are
// built for 64 registers a thread, which 1024 threads leave.
static cudaError_t coop_shape(const void* fn, long long n, int largest, int& block, int& grid)
{
    int dev = 0, sms = 0, per = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (!e) e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    if (e) return e;
    block = largest;
    for (int b : {128, 256, 384, 512})
        if (b < largest && (n + b - 1) / b <= sms) {
            block = b;
            break;
        }
    e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, fn, block, 0);
    if (e) return e;
    const long long want = (n + block - 1) / block;
    const long long cap = per > 0 ? sms < gsync::kMaxBlocks ? sms : gsync::kMaxBlocks : 0;
    grid = int(want < cap ? want : cap);
    return cudaSuccess;
}

int coop_grid_blocks(long long n)
{
    // the persistent solve is available when every kernel's grid is
    int least = 1 << 30;
    for (bool pair : {false, true})
        for (bool fp32 : {false, true})
            for (int w : {0, 4, 6}) {
                int block = 0, grid = 0;
                if (coop_shape(coop_kernel(pair, fp32, w), n,
                               pair || w == 4 ? kWideBlock : kCoopBlock, block, grid))
                    return 0;
                least = grid < least ? grid : least;
            }
    return least;
}

cudaError_t launch_implicit_coop(const DiffusionArgs& a, cudaStream_t s)
{
    CoopArgs ca{};
    if (a.sx) {
        ca.div_nx = make_fastdiv(unsigned(a.sx));
        ca.div_ny = make_fastdiv(unsigned(a.sy));
    }
    DiffusionArgs args = a;
    void* params[] = {&args, &ca};
    const int w = (!a.sx && (a.width == 4 || a.width == 6)) ? a.width : 0;
    // pairs without corrections: the form with float ones, which spills less at 64
    // registers (420,000 rows: 110 against 112 us a step)
    void* fn = coop_kernel(a.pair != 0, a.nc_fp32 != 0 || (a.pair && !a.nc_gw), w);
    int block = 0, grid = 0;
    if (cudaError_t e = coop_shape(fn, a.n, a.pair || w == 4 ? kWideBlock : kCoopBlock, block,
                                   grid))
        return e;
    return cudaLaunchCooperativeKernel(fn, dim3(grid), dim3(block), params, 0, s);
}

}  // namespace cfg
