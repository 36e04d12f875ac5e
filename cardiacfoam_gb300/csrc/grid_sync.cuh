// Grid-wide synchronisation and deterministic reductions for persistent
// cooperative kernels (every block resident).  The waits are bounded: a block
// that waits longer than the spin limit (by default seconds) sets an abort flag
// and every block leaves at its next sum.
#pragma once

#include <cuda_runtime.h>

#include <type_traits>

#include "float_pair.cuh"

namespace cfg {
namespace gsync {

constexpr long long kSpinLimit = 1LL << 25;   // x >= 32 ns per spin: about a second

__device__ __forceinline__ int ld_relaxed_int(const int* p)
{
    int v;
    asm volatile("ld.relaxed.gpu.global.s32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
    return v;
}

// K scalars derived from reduction results (ratios of sums), scalar k
// computed by warp k's first lane as f(k) and read by every thread of the
// block.  Every thread holds the same sums, so every block gets the same
// values; doing the arithmetic once per block instead of once per thread
// matters because an FP64 division is about nine instructions of 64 clocks on
// an SM partition that the row work shares, and a warp per scalar because two
// divisions on one partition take twice as long.  `set` alternates between
// consecutive calls.
template <int K, class F>
__device__ __forceinline__ void block_scalars(int set, double (&out)[K], F f)
{
    __shared__ double v[2][K];
    if ((threadIdx.x & 31) == 0 && (threadIdx.x >> 5) < K)
        v[set & 1][threadIdx.x >> 5] = f(int(threadIdx.x >> 5));
    __syncthreads();
#pragma unroll
    for (int k = 0; k < K; ++k) out[k] = v[set & 1][k];
}

// ---------------------------------------------------------------- sums that are barriers
// The persistent kernels meet only to add numbers up, so a sum is a barrier: a
// block adds its threads' summands, writes its partial sums and counts itself
// in (release increments), waits for the others' increments, and adds
// everybody's partial sums in the same fixed order, so all blocks hold the
// same bits.  The increments release and the wait acquires, so the blocks'
// writes before the call are visible to their reads after it.  Partial sums of
// two calls alternate: a block writes a slot again only after every block has
// counted itself in for, and so has finished reading before, the call between.
// The counter starts at zero in every launch (the caller resets it).
//
// Warp k of a block sees sum k through from the block's partial sum to the
// total, so a call costs two block barriers (three in double) where separate
// block sums, grid barrier and grid sums cost five.
//
// Tried and slower: slots of (value, phase) that every block polls in place of
// the counter (one L2 round trip less, but 143 blocks polling the lines that
// they write: 3998 against 2970 us per bidomain step of 64,000 cells).
constexpr int kMaxBlocks = 512, kMaxSums = 3;

struct Exchange {
    unsigned count;
    unsigned pad[3];
    unsigned long long slot[2][kMaxSums][kMaxBlocks];
};

__device__ __forceinline__ unsigned ld_acquire(const unsigned* p)
{
    unsigned v;
    asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
    return v;
}

__device__ __forceinline__ void red_release_add(unsigned* p, unsigned v)
{
    asm volatile("red.release.gpu.global.add.u32 [%0], %1;" :: "l"(p), "r"(v) : "memory");
}

struct SumDouble {
    using T = double;
    static __device__ __forceinline__ T zero() { return 0.0; }
    static __device__ __forceinline__ T add(T a, T b) { return a + b; }
    static __device__ __forceinline__ unsigned long long bits(T a)
    {
        return (unsigned long long)__double_as_longlong(a);
    }
    static __device__ __forceinline__ T of(unsigned long long b)
    {
        return __longlong_as_double((long long)b);
    }
    static __device__ __forceinline__ T shift(T a, int o) { return __shfl_down_sync(~0u, a, o); }
};

struct SumPair {
    using T = fp::P;
    static __device__ __forceinline__ T zero() { return fp::make(0.0f); }
    static __device__ __forceinline__ T add(T a, T b) { return fp::add(a, b); }
    static __device__ __forceinline__ unsigned long long bits(T a)
    {
        return (unsigned long long)__float_as_uint(a.x) |
               ((unsigned long long)__float_as_uint(a.y) << 32);
    }
    static __device__ __forceinline__ T of(unsigned long long b)
    {
        return make_float2(__uint_as_float(unsigned(b)), __uint_as_float(unsigned(b >> 32)));
    }
    static __device__ __forceinline__ T shift(T a, int o)
    {
        return make_float2(__shfl_down_sync(~0u, a.x, o), __shfl_down_sync(~0u, a.y, o));
    }
};

template <class S>
__device__ __forceinline__ typename S::T warp_total(typename S::T v)
{
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v = S::add(v, S::shift(v, o));
    return v;   // lane 0
}

// v[k]: in, this thread's summands; out, the grid's sums.  All threads of all
// blocks call it the same number of times; `arrivals` counts the increments
// expected so far.  False when the launch was aborted (some block waited more
// than `spin_limit` spins).
//
// In double the summands of a block go through shared memory to four warps per
// sum, one on each SM partition, rather than through a shuffle tree in every
// warp: an FP64 addition holds a partition for 64 clocks whatever its active
// lanes, so 16 warps of trees cost 20 additions per partition and sum, this 8.
// kBlock: the most threads a block has; it has at least 32 K.
// `met`, if given, runs on every thread once all blocks have counted themselves
// in and before the total is formed: loads of what the others published, which
// need not wait for it.
struct Nothing {
    __device__ __forceinline__ void operator()() const {}
};

template <int kBlock, int K, class S, class F = Nothing>
__device__ __forceinline__ bool sync_sums(Exchange* x, int* abort, unsigned& arrivals, int& set,
                                          long long spin_limit, typename S::T (&v)[K],
                                          F met = F())
{
    using T = typename S::T;
    constexpr bool kDouble = std::is_same<S, SumDouble>::value;
    static_assert(K >= 1 && K <= kMaxSums && kBlock <= 1024, "a warp per sum, a lane per warp");
    __shared__ T sh[K][kDouble ? kBlock : kBlock / 32];
    __shared__ T part[K][4];
    __shared__ T total[2][K];
    __shared__ int good;
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, warps = blockDim.x >> 5;
    const int parts = warps >= 4 * K ? 4 : warps / K;   // warps that add one sum
    arrivals += (kDouble ? K : 1) * gridDim.x;
    set ^= 1;
    if (threadIdx.x == 0) good = 1;
    T s = S::zero();
    if constexpr (kDouble) {
#pragma unroll
        for (int k = 0; k < K; ++k) sh[k][threadIdx.x] = v[k];
        __syncthreads();
        if (w < K * parts) {
            const int k = w / parts, q = w - k * parts;
            s = sh[k][32 * q + lane];
            for (int j = q + parts; j < warps; j += parts) s = S::add(s, sh[k][32 * j + lane]);
            s = warp_total<S>(s);
            if (lane == 0) part[k][q] = s;
        }
        __syncthreads();
        if (w < K && lane == 0) {
            s = part[w][0];
            for (int q = 1; q < parts; ++q) s = S::add(s, part[w][q]);
        }
    } else {
#pragma unroll
        for (int k = 0; k < K; ++k) {
            const T t = warp_total<S>(v[k]);
            if (lane == 0) sh[k][w] = t;
        }
        __syncthreads();
        if (w < K) s = warp_total<S>(lane < warps ? sh[w][lane] : S::zero());
    }
    if (w < K) {
        unsigned long long* slots = x->slot[set][w];
        if (lane == 0) __stcg(&slots[blockIdx.x], S::bits(s));
        // Pairs: one increment and one waiting warp per block, once all of its
        // partial sums are written: increments of one address queue up, and every
        // poll is in the way of the loads of the blocks that are waited for (with
        // three waiting warps a bidomain step of 64,000 rows takes 2.64 to 3.08 ms,
        // 2.59 with one, of 125,000 rows 4.84 to 5.45, 4.80 with one; both vary with
        // the chip).  Double: a warp per sum, because the warps end their sums at
        // different times.
        if constexpr (!kDouble && K > 1)
            asm volatile("bar.sync 1, %0;" ::"n"(32 * K) : "memory");
        if (lane == 0 && (kDouble || w == 0)) {
            red_release_add(&x->count, 1u);
            long long spins = 0;
            while (ld_acquire(&x->count) < arrivals) {
                if (ld_relaxed_int(abort)) { good = 0; break; }
                if (++spins > spin_limit) {
                    atomicExch(abort, 1);
                    good = 0;
                    break;
                }
                // short waits spin; long ones back off (a waiting block then
                // polls L2 less often)
                if (spins > 4096) __nanosleep(64);
            }
        }
        __syncwarp();
        // the other warps' reads of the sums come after that wait
        if constexpr (!kDouble && K > 1 && std::is_same<F, Nothing>::value)
            asm volatile("bar.sync 1, %0;" ::"n"(32 * K) : "memory");
    }
    if constexpr (!std::is_same<F, Nothing>::value) {
        __syncthreads();
        met();
    }
    if (w < K) {
        const unsigned long long* slots = x->slot[set][w];
        s = S::zero();
        for (unsigned b = lane; b < gridDim.x; b += 32) s = S::add(s, S::of(__ldcg(&slots[b])));
        s = warp_total<S>(s);
        if (lane == 0) total[set][w] = s;
    }
    __syncthreads();
#pragma unroll
    for (int k = 0; k < K; ++k) v[k] = total[set][k];
    return good != 0;   // set again only by a caller that read 1 here
}

}  // namespace gsync
}  // namespace cfg
