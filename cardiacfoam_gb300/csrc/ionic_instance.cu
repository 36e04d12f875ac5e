// One ionic model in one precision form.  Compiled once per (model,
// precision) with -DCFG_MODEL=<namespace> -DCFG_FP64=<0|1>.
#include <cuda_runtime.h>

#include "ionic_kernels.cuh"
#include "ionic_mixed.cuh"
#include "ionic_batch.cuh"

#define CFG_STR2(x) #x
#define CFG_STR(x) CFG_STR2(x)
#define CFG_CAT3_(a, b, c) a##b##c
#define CFG_CAT3(a, b, c) CFG_CAT3_(a, b, c)
#include CFG_STR(models/CFG_MODEL.cuh)
#if CFG_FP64
#define CFG_PLAIN_HEADER(m) CFG_STR(models/m##_plain.cuh)
#define CFG_PLAIN_(m) CFG_PLAIN_HEADER(m)
#include CFG_PLAIN_(CFG_MODEL)
#endif

#if CFG_FP64
#define CFG_PREC_TAG _fp64
#else
#define CFG_PREC_TAG _mixed
#endif

#if CFG_FP64
using M = cfg::CFG_MODEL::plain::Model;
#else
using M = cfg::CFG_MODEL::Model;
#endif
static constexpr bool kFP64 = CFG_FP64 != 0;

using cfg::TissueList;
using Tissues = cfg::CFG_MODEL::TissueSet;

// The plain form runs ionic_step_kernel (one cell per lane, or per four lanes
// of as many warps); the mixed form runs ionic_mixed_kernel (stage data in
// shared memory, block size fixed by the model's slice length).
// `block` threads per block (the plain form: at most 128, 0 = by the rule
// below; the mixed form: at most the model's slice block, 0 = that block) and
// p.cells_per_thread slots per thread; every slot's arithmetic is independent
// of both, so the results are too.
#if CFG_FP64
// constants per cell: a warp to a tile of 32 cells
template <bool SV, int T>
static void launch_one(const cfg::IonicLaunch& p, cudaStream_t s, int block)
{
    static_assert(T == 0, "the kernels of one tissue are in ionic_tissue.cu");
    cfg::launch_step<M, SV, T>(p, s, block);
}
#else
template <bool SV, int T>
static void launch_one(const cfg::IonicLaunch& p, cudaStream_t s, int block)
{
    const long long cpt = p.cells_per_thread > 0 ? p.cells_per_thread : 1;
    using S = cfg::mixed::Slice<M>;
    const int b = (block > 0 && block <= S::block && block % 32 == 0) ? block : S::block;
    const unsigned grid = unsigned((p.count + b * cpt - 1) / (b * cpt));
    cfg::ionic_mixed_kernel<M, SV, T><<<grid, b, size_t(b) * S::len * 4, s>>>(p);
}
#endif

extern "C" int CFG_CAT3(cfg_ionic_max_block_, CFG_MODEL, CFG_PREC_TAG)()
{
    if constexpr (kFP64) return 128;
    else return cfg::mixed::Slice<M>::block;
}

// Opt the mixed kernels into their dynamic shared memory (above the 48 KB
// default) on the current device; runs when a model is created, before any
// launch can be captured into a graph.
template <bool SV, int T>
static cudaError_t prepare_one()
{
    if constexpr (kFP64) {
        return cudaSuccess;
    } else {
        return cudaFuncSetAttribute(&cfg::ionic_mixed_kernel<M, SV, T>,
                                    cudaFuncAttributeMaxDynamicSharedMemorySize,
                                    cfg::mixed::Slice<M>::smem_bytes);
    }
}

template <int... TS>
static cudaError_t prepare_all(TissueList<TS...>)
{
    cudaError_t e = prepare_one<true, 0>();
    if (e == cudaSuccess) e = prepare_one<false, 0>();
    cudaError_t r[] = {cudaSuccess, prepare_one<false, TS>()...};
    for (cudaError_t x : r)
        if (e == cudaSuccess) e = x;
    return e;
}

#if CFG_FP64
// ionic_tissue.cu, compiled once per tissue flag
#define CFG_CAT5_(a, b, c, d, e) a##b##c##d##e
#define CFG_CAT5(a, b, c, d, e) CFG_CAT5_(a, b, c, d, e)
#define CFG_TISSUE_STEP(T) CFG_CAT5(cfg_ionic_step_, CFG_MODEL, _tissue, T, )
#define CFG_TISSUE_DECL(T) \
    extern "C" void CFG_TISSUE_STEP(T)(const cfg::IonicLaunch& p, int solve_vm, cudaStream_t s, int block);
#define CFG_TISSUE_CASE(T) \
    case T: CFG_TISSUE_STEP(T)(p, solve_vm, s, block); return true;
CFG_FOR_TISSUES(CFG_TISSUE_DECL)
static bool launch_uniform(const cfg::IonicLaunch& p, int solve_vm, cudaStream_t s, int block)
{
    switch (p.tissue) {
        CFG_FOR_TISSUES(CFG_TISSUE_CASE)
    default: return false;
    }
}
#else
template <int T0, int... TR>
static bool launch_uniform(const cfg::IonicLaunch& p, cudaStream_t s, int block,
                           TissueList<T0, TR...>)
{
    if (p.tissue == T0) {
        launch_one<false, T0>(p, s, block);
        return true;
    }
    if constexpr (sizeof...(TR) > 0) return launch_uniform(p, s, block, TissueList<TR...>{});
    return false;
}
#endif

extern "C" cudaError_t CFG_CAT3(cfg_ionic_step_, CFG_MODEL, CFG_PREC_TAG)(
    const cfg::IonicLaunch& p, int solve_vm, cudaStream_t stream, int block)
{
    if (p.n <= 0 || p.count <= 0) return cudaSuccess;
    const bool uniform = !p.tissue_cell && !p.scales;
    // a uniform tissue without scales runs the kernel that folds its constants;
    // for the single-cell form only in FP64, whose time is the FP64
    // instruction count
#if CFG_FP64
    if (uniform && launch_uniform(p, solve_vm, stream, block)) return cudaGetLastError();
#else
    if (!solve_vm && uniform && launch_uniform(p, stream, block, Tissues{}))
        return cudaGetLastError();
#endif
    if (solve_vm) launch_one<true, 0>(p, stream, block);
    else launch_one<false, 0>(p, stream, block);
    return cudaGetLastError();
}

extern "C" cudaError_t CFG_CAT3(cfg_ionic_init_, CFG_MODEL, CFG_PREC_TAG)(
    long long n, int tissue, const unsigned char* tissue_cell, const double* scales,
    long long stride, double init_step, double* yw, float* yn, double* step,
    cudaStream_t stream)
{
    if (cudaError_t e = prepare_all(Tissues{})) return e;
    if (n <= 0) return cudaSuccess;
    const int block = 128;
    const unsigned grid = unsigned((n + block - 1) / block);
    cfg::ionic_init_kernel<M, kFP64><<<grid, block, 0, stream>>>(n, tissue, tissue_cell, scales,
                                                                stride, init_step, yw, yn, step);
    return cudaGetLastError();
}

#if CFG_FP64
// host-side initConsts of this model (compiled once, in the plain TU)
extern "C" void CFG_CAT3(cfg_ionic_host_init_, CFG_MODEL, )(double* C, double* y, int tissue,
                                                             const double* scale)
{
    M::init(C, y, tissue, scale);
}
#endif

// ---------------------------------------------------------------- batched single cells

// persistent grid: every block resident, cells handed out by the queue
static cudaError_t batch_launch_on(void (*fn)(cfg::BatchLaunch), int& per_sm, int sms, int block,
                                   int smem, const cfg::BatchLaunch& p, cudaStream_t s)
{
    if (!per_sm) {
        cudaError_t e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, fn, block, smem);
        if (e) return e;
        if (per_sm < 1) per_sm = 1;
    }
    const long long want = (p.n + block - 1) / block;
    const long long cap = (long long)sms * per_sm;
    const unsigned grid = unsigned(want < cap ? want : cap);
    fn<<<grid, block, smem, s>>>(p);
    return cudaGetLastError();
}

template <int T>
static cudaError_t batch_launch(const cfg::BatchLaunch& p, cudaStream_t s)
{
    static int sms = 0, per_sm = 0;
    if (!sms) {
        int dev = 0;
        cudaError_t e = cudaGetDevice(&dev);
        if (!e) e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
        if (e) return e;
    }
    if constexpr (kFP64) {
        return batch_launch_on(cfg::batch_fp64_kernel<M, T>, per_sm, sms, 128, 0, p, s);
    } else {
        // all states in shared memory while every cell is resident that way; see
        // ionic_batch.cuh for both sides
        using All = cfg::BatchShape<M, 0>;
        constexpr int R = cfg::batch_registers<M>();
        if constexpr (R > 0) {
            using Some = cfg::BatchShape<M, R>;
            static int per_sm_some = 0;
            if (p.n > (long long)sms * All::threads)
                return batch_launch_on(cfg::batch_mixed_kernel<M, T, R>, per_sm_some, sms,
                                       Some::block, Some::smem_bytes, p, s);
        }
        return batch_launch_on(cfg::batch_mixed_kernel<M, T, 0>, per_sm, sms, All::block,
                               All::smem_bytes, p, s);
    }
}

template <int T0, int... TR>
static cudaError_t batch_dispatch(const cfg::BatchLaunch& p, int tissue, cudaStream_t s,
                                  TissueList<T0, TR...>)
{
    if (tissue == T0) return batch_launch<T0>(p, s);
    if constexpr (sizeof...(TR) > 0) return batch_dispatch(p, tissue, s, TissueList<TR...>{});
    return cudaErrorInvalidValue;
}

template <int R, int... TS>
static cudaError_t batch_prepare(TissueList<TS...>)
{
    if constexpr (!kFP64) {
        cudaError_t r[] = {cudaSuccess,
                           cudaFuncSetAttribute(&cfg::batch_mixed_kernel<M, TS, R>,
                                                cudaFuncAttributeMaxDynamicSharedMemorySize,
                                                cfg::BatchShape<M, R>::smem_bytes)...};
        for (cudaError_t x : r)
            if (x) return x;
    }
    return cudaSuccess;
}

extern "C" cudaError_t CFG_CAT3(cfg_batch_init_, CFG_MODEL, CFG_PREC_TAG)(
    const cfg::BatchLaunch& p, const double* scales, int tissue, double init_step,
    cudaStream_t stream)
{
    if (cudaError_t e = batch_prepare<0>(Tissues{})) return e;
    if constexpr (cfg::batch_registers<M>() > 0)
        if (cudaError_t e = batch_prepare<cfg::batch_registers<M>()>(Tissues{})) return e;
    if (p.n <= 0) return cudaSuccess;
    const int block = 128;
    const unsigned grid = unsigned((p.n + block - 1) / block);
    cfg::batch_init_kernel<M, kFP64><<<grid, block, 0, stream>>>(p, scales, tissue, init_step);
    return cudaGetLastError();
}

extern "C" cudaError_t CFG_CAT3(cfg_batch_step_, CFG_MODEL, CFG_PREC_TAG)(
    const cfg::BatchLaunch& p, int tissue, cudaStream_t stream)
{
    if (p.n <= 0) return cudaSuccess;
    return batch_dispatch(p, tissue, stream, Tissues{});
}
