// The plain FP64 step of one model for one tissue flag (its constants are
// compile-time values).  Compiled once per (model, tissue) with
// -DCFG_MODEL=<namespace> -DCFG_TISSUE=<flag>: four warps' parts of a large
// right-hand side take long to compile.
#include <cuda_runtime.h>

#include "ionic_kernels.cuh"

#define CFG_STR2(x) #x
#define CFG_STR(x) CFG_STR2(x)
#define CFG_CAT4_(a, b, c, d) a##b##c##d
#define CFG_CAT4(a, b, c, d) CFG_CAT4_(a, b, c, d)
#define CFG_PLAIN_HEADER(m) CFG_STR(models/m##_plain.cuh)
#define CFG_PLAIN_(m) CFG_PLAIN_HEADER(m)
#include CFG_PLAIN_(CFG_MODEL)

using M = cfg::CFG_MODEL::plain::Model;

extern "C" void CFG_CAT4(cfg_ionic_step_, CFG_MODEL, _tissue, CFG_TISSUE)(
    const cfg::IonicLaunch& p, int solve_vm, cudaStream_t s, int block)
{
    if (solve_vm) cfg::launch_step<M, true, CFG_TISSUE>(p, s, block);
    else cfg::launch_step<M, false, CFG_TISSUE>(p, s, block);
}
