// hc_scan.cuh -- block scans and the decoupled look-back shared by the sort and
// the tree build.
//
// Single-pass prefix sums over tiles with decoupled look-back (Merrill and
// Garland, "Single-pass parallel prefix scan with decoupled look-back", 2016):
// tiles take their index from a counter in launch order, publish their sum, and
// read the earlier tiles' published words back to the first one that already
// holds its inclusive prefix.  A tile waits only on tiles that hold their
// index, so every wait ends; each wait is bounded nonetheless and reports an
// error.  Words hold a flag (2 bits) and a value below 2^30 (bodies + cells
// are fewer).
#pragma once
#include <stdint.h>
#include "hc_internal.cuh"

constexpr uint32_t LB_AGG = 1u << 30, LB_PRE = 2u << 30, LB_VAL = (1u << 30) - 1u;
constexpr int LB_SPIN = 1 << 20;

__device__ __forceinline__ uint32_t ld_relaxed(const uint32_t *p)
{
    uint32_t v;
    asm volatile("ld.relaxed.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
    return v;
}
__device__ __forceinline__ void st_relaxed(uint32_t *p, uint32_t v)
{
    asm volatile("st.relaxed.gpu.global.u32 [%0], %1;" ::"l"(p), "r"(v) : "memory");
}

template <typename T>
__device__ __forceinline__ T warp_inclusive_scan(T x)
{
    const int lane = threadIdx.x & 31;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const T y = __shfl_up_sync(0xffffffffu, x, o);
        if (lane >= o) x += y;
    }
    return x;
}

// warp scan with shuffles, then scan of the warp sums; sh: 32 words
template <typename T>
__device__ T block_exclusive_scan(T v, T *sh, T *total)
{
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5, nw = blockDim.x >> 5;
    const T x = warp_inclusive_scan(v);
    if (lane == 31) sh[wid] = x;
    __syncthreads();
    if (wid == 0) {
        const T w = warp_inclusive_scan(lane < nw ? sh[lane] : T(0));
        if (lane < nw) sh[lane] = w;
    }
    __syncthreads();
    const T base = wid > 0 ? sh[wid - 1] : T(0);
    if (total) *total = sh[nw - 1];
    __syncthreads();
    return base + x - v;
}

// One warp: publishes the tile's sum and returns the sum of all earlier tiles
// (32 tiles' words per step).
__device__ __forceinline__ uint32_t tile_prefix(uint32_t *status, int64_t tile, uint32_t agg, int *err)
{
    const int lane = threadIdx.x & 31;
    if (tile == 0) {
        if (lane == 0) st_relaxed(status, LB_PRE | agg);
        return 0;
    }
    if (lane == 0) st_relaxed(status + tile, LB_AGG | agg);
    uint32_t prefix = 0;
    for (int64_t t0 = tile - 1;; t0 -= 32) {
        const int64_t t = t0 - lane;
        uint32_t w = LB_PRE;                      // before tile 0: an empty prefix
        if (t >= 0) {
            w = ld_relaxed(status + t);
            for (int spin = 0; (w & ~LB_VAL) == 0 && spin < LB_SPIN; spin++) w = ld_relaxed(status + t);
            if ((w & ~LB_VAL) == 0) {             // a tile that never published: report, stop
                atomicCAS(err, 0, HC_ERR_STATE);
                w = LB_PRE;
            }
        }
        const unsigned pre = __ballot_sync(0xffffffffu, (w & ~LB_VAL) == LB_PRE);
        const int stop = pre ? __ffs(pre) - 1 : 31;
        prefix += __reduce_add_sync(0xffffffffu, lane <= stop ? (w & LB_VAL) : 0u);
        if (pre) break;
    }
    if (lane == 0) st_relaxed(status + tile, LB_PRE | (prefix + agg));
    return prefix;
}

// One digit per thread: publishes the tile's count of the digit (word
// status[tile * ndigit + digit]) and returns the earlier tiles' sum, LB_WIN
// tiles' words loaded per step.
constexpr int LB_WIN = 8;
__device__ __forceinline__ uint32_t digit_prefix(uint32_t *status, int64_t tile, int ndigit, int digit, uint32_t cnt,
                                                 int *err)
{
    uint32_t *mine = status + tile * ndigit + digit;
    if (tile == 0) {
        st_relaxed(mine, LB_PRE | cnt);
        return 0;
    }
    st_relaxed(mine, LB_AGG | cnt);
    uint32_t prefix = 0;
    bool done = false;
    for (int64_t t0 = tile - 1; t0 >= 0 && !done; t0 -= LB_WIN) {
        uint32_t v[LB_WIN];
#pragma unroll
        for (int j = 0; j < LB_WIN; j++) v[j] = t0 - j >= 0 ? ld_relaxed(status + (t0 - j) * ndigit + digit) : LB_PRE;
#pragma unroll
        for (int j = 0; j < LB_WIN; j++) {
            if (done || t0 - j < 0) continue;
            const uint32_t *q = status + (t0 - j) * ndigit + digit;
            for (int spin = 0; (v[j] & ~LB_VAL) == 0 && spin < LB_SPIN; spin++) v[j] = ld_relaxed(q);
            if ((v[j] & ~LB_VAL) == 0) {          // a tile that never published: report, stop
                atomicCAS(err, 0, HC_ERR_STATE);
                done = true;
                continue;
            }
            prefix += v[j] & LB_VAL;
            if ((v[j] & ~LB_VAL) == LB_PRE) done = true;
        }
    }
    st_relaxed(mine, LB_PRE | (prefix + cnt));
    return prefix;
}
