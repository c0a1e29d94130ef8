// hc_tree.cu -- octree construction and moments on the GPU.
//
// Reference: maketree/expandbox/loadtree/intcoord/subindex/hackcofm,
// src/nbody/evolve/hackcode/hackcode1/load.c:32-248.
//
// The reference inserts massive bodies one at a time.  Its final tree is a
// pure function of the root box and the multiset of integer coordinates: a
// cell exists for every octree node (integer prefix) holding two or more
// massive bodies, bodies are leaves, there is no leaf bucket and no path
// compression.  The one exception is expandbox (load.c:68-95): when the second
// massive body forces the box to double K >= 2 times, the K-1 intermediate
// root cells hold only the first body.  The build here reproduces that set:
//
//   1. expandbox replay on the device (one block, FP64, body order),
//   2. 90-bit keys: floor(2^30 (x - rmin) / rsize) per axis, Morton order,
//   3. radix sort; compaction of the massive bodies where there are massless ones,
//   4. d[a] = common octal digits of adjacent keys; cells starting at sorted
//      body a have levels (d[a-1], d[a]]: the bodies in key order, each after
//      the cells that start at it, are the nodes in DFS pre-order.  One pass
//      counts the nodes of every depth; a second gives each node its
//      breadth-first place (nodes of its depth before it in pre-order) and its
//      first child's place (the nodes one deeper before it), so that the
//      children of each cell are contiguous and in subindex order 0..7 and no
//      node has to search for its parent or children,
//   5. node records, cells grouped by depth and child count,
//   6. level-synchronous upward pass (one cooperative kernel, a grid barrier
//      per level): mass and centre of mass in FP64, children summed in the
//      same order as hackcofm so they are bit-identical (they decide cell
//      openings); the quadrupole, which the walk consumes in FP32, is
//      accumulated in FP32 from FP64 offsets.
#include <cooperative_groups.h>
#include <memory>
#include "hc_scan.cuh"

namespace cg = cooperative_groups;

namespace {

__device__ __forceinline__ double dmul(double a, double b) { return __dmul_rn(a, b); }
__device__ __forceinline__ double dadd(double a, double b) { return __dadd_rn(a, b); }
__device__ __forceinline__ double dsub(double a, double b) { return __dsub_rn(a, b); }
__device__ __forceinline__ double ddiv(double a, double b) { return __ddiv_rn(a, b); }

// (x - rmin) / rsize.  A power-of-two rsize (hackcode1's box is 4 * 2^k)
// divides exactly as a multiplication by its reciprocal: the same correctly
// rounded result, without an FP64 division.
__device__ __forceinline__ double scaled(double x, double rmin, double rsize)
{
    int e;
    const double f = frexp(rsize, &e);
    return f == 0.5 ? dmul(dsub(x, rmin), ldexp(1.0, 1 - e)) : ddiv(dsub(x, rmin), rsize);
}

// intcoord (load.c:135-156): xsc = (x - rmin)/rsize; inside iff 0 <= xsc < 1.
__device__ __forceinline__ bool intcoord1(double x, double rmin, double rsize, int *xi)
{
    double xsc = scaled(x, rmin, rsize);
    if (0.0 <= xsc && xsc < 1.0) {
        *xi = (int)floor(dmul((double)HC_IMAX, xsc));
        return true;
    }
    return false;
}

__device__ __forceinline__ bool inbox(double x, double y, double z, const double *rmin, double rsize)
{
    int t;
    bool a = intcoord1(x, rmin[0], rsize, &t);
    bool b = intcoord1(y, rmin[1], rsize, &t);
    bool c = intcoord1(z, rmin[2], rsize, &t);
    return a && b && c;
}

// ---------------- expandbox replay ----------------

// the two smallest of two pairs of ascending body indices (INT_MAX: none)
__device__ __forceinline__ int2 min2(int2 a, int2 b)
{
    return make_int2(min(a.x, b.x), min(max(a.x, b.x), min(a.y, b.y)));
}

__device__ __forceinline__ int2 warp_min2(int2 v)
{
#pragma unroll
    for (int o = 16; o; o >>= 1) {
        const int2 w = make_int2(__shfl_xor_sync(0xffffffffu, v.x, o), __shfl_xor_sync(0xffffffffu, v.y, o));
        v = min2(v, w);
    }
    return v;
}

// The massive bodies outside the box (intcoord's test, load.c:135-156), in body
// order, and each tile's first two massive bodies (the expansion replay needs
// the first two of all).  A body clearly inside by an FP32 estimate with a
// margin far above its error skips the exact FP64 test (the FP64 pipe runs at a
// small fraction of the FP32 rate); the rest take it.  One pass: a tile's place
// in the list comes from decoupled look-back (as three kernels -- flags, scan,
// compaction -- this took 21 + 13 + 5 us at N = 2^20 and two more launches).
// Tiles of 1024 bodies up to 2^18, of 4096 above (4096 bodies: 15 -> 8 us; at
// 2^20 the larger tile is 4 us faster).
constexpr int BOX_SMALL = 1 << 18;
static inline int box_items(int64_t n) { return n <= BOX_SMALL ? 4 : 16; }
template <int BOX_ITEMS>
__global__ void __launch_bounds__(256) k_box_outside(const double *mass, const double *px, const double *py,
                                                     const double *pz, int64_t n, const hc_box *box, int32_t *cand,
                                                     int32_t *ncand, int2 *first2, uint32_t *status, uint32_t *ctr,
                                                     int *err)
{
    constexpr int BOX_TILE = 256 * BOX_ITEMS;
    __shared__ int2 wf[8];
    __shared__ uint32_t wsum[8], s_tile, s_prefix;
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    if (threadIdx.x == 0) s_tile = atomicAdd(ctr, 1u);
    __syncthreads();
    const int64_t tile = s_tile, base = tile * BOX_TILE + wid * (BOX_TILE / 8);
    double rmin[3] = {box->rmin[0], box->rmin[1], box->rmin[2]};
    double rsize = box->rsize;
    const float lo[3] = {hc_d2f_rn(rmin[0]), hc_d2f_rn(rmin[1]), hc_d2f_rn(rmin[2])}, sz = hc_d2f_rn(rsize);
    int2 f2 = make_int2(INT_MAX, INT_MAX);     // this thread's first two massive bodies (ascending i)
    uint32_t out = 0, cnt = 0;                 // rounds in which this lane's body is outside; the warp's number
#pragma unroll 4
    for (int r = 0; r < BOX_ITEMS; r++) {
        const int64_t i = base + r * 32 + lane;
        bool o = false;
        if (i < n) {
            const bool m = hc_nonzero(mass[i]);
            if (m && f2.y == INT_MAX) {
                if (f2.x == INT_MAX) f2.x = (int)i;
                else f2.y = (int)i;
            }
            const double x[3] = {px[i], py[i], pz[i]};
            bool clear = true;
#pragma unroll
            for (int k = 0; k < 3; k++) {
                float f;
                if (!hc_approx_f32(x[k], &f)) {
                    clear = false;
                    continue;
                }
                const float u = f - lo[k], margin = 0x1p-16f * sz + 0x1p-18f * fabsf(f);
                clear = clear && u >= margin && u <= sz - margin;
            }
            o = m && !(clear || inbox(x[0], x[1], x[2], rmin, rsize));
        }
        cnt += __popc(__ballot_sync(0xffffffffu, o));
        out |= (uint32_t)o << r;
    }
    f2 = warp_min2(f2);
    if (lane == 0) {
        wf[wid] = f2;
        wsum[wid] = cnt;
    }
    __syncthreads();
    if (wid == 0) {
        const uint32_t agg = __reduce_add_sync(0xffffffffu, lane < 8 ? wsum[lane] : 0u);
        const uint32_t prefix = tile_prefix(status, tile, agg, err);
        if (lane == 0) {
            s_prefix = prefix;
            if ((tile + 1) * BOX_TILE >= n) *ncand = (int32_t)(prefix + agg);     // the last tile
            for (int w = 1; w < 8; w++) f2 = min2(f2, wf[w]);
            first2[tile] = f2;
        }
    }
    __syncthreads();
    if (cnt == 0) return;                      // the whole warp
    uint32_t pos = s_prefix;
    for (int w = 0; w < wid; w++) pos += wsum[w];
    for (int r = 0; r < BOX_ITEMS; r++) {
        const unsigned b = __ballot_sync(0xffffffffu, (out >> r) & 1u);
        if ((out >> r) & 1u) cand[pos + __popc(b & ((1u << lane) - 1u))] = (int32_t)(base + r * 32 + lane);
        pos += __popc(b);
    }
}

// One block replays expandbox over the bodies that were outside the box at
// the start, in body order.  The box only grows, so a body inside stays
// inside; each round finds the first remaining body outside, expands for
// it, and continues after it.
// The first two massive bodies come from k_box_outside's per-tile pairs: the
// first one (original order) is where the expansion-chain cells hang, the
// second is the body whose insertion may graft them.
__global__ void __launch_bounds__(256) k_box_replay(const double *px, const double *py, const double *pz,
                                                    const int32_t *cand, const int32_t *ncand_p, const int2 *first2,
                                                    int nblk, hc_box *box, hc_status *st, int nmassive)
{
    __shared__ int first;
    __shared__ double rmin[3], rsize;
    __shared__ int doublings, chain_before, chain_k;
    __shared__ int2 wf[8];
    __shared__ int second_massive;
    const int ncand = *ncand_p;
    {
        int2 f2 = make_int2(INT_MAX, INT_MAX);
        for (int b = threadIdx.x; b < nblk; b += blockDim.x) f2 = min2(f2, first2[b]);
        f2 = warp_min2(f2);
        if ((threadIdx.x & 31) == 0) wf[threadIdx.x >> 5] = f2;
        __syncthreads();
        if (threadIdx.x == 0) {
            for (int w = 1; w < (int)(blockDim.x >> 5); w++) f2 = min2(f2, wf[w]);
            box->first_massive = f2.x == INT_MAX ? -1 : f2.x;
            if (nmassive >= 0) box->nmassive = nmassive;       // every body has mass
            second_massive = f2.y == INT_MAX ? -1 : f2.y;
        }
    }
    if (threadIdx.x == 0) {
        rmin[0] = box->rmin[0];
        rmin[1] = box->rmin[1];
        rmin[2] = box->rmin[2];
        rsize = box->rsize;
        doublings = 0;
        chain_before = -1;
        chain_k = 0;
    }
    __syncthreads();
    int pos = 0;
    while (pos < ncand) {
        if (threadIdx.x == 0) first = INT_MAX;
        __syncthreads();
        for (int base = pos; base < ncand; base += blockDim.x) {
            int i = base + threadIdx.x;
            if (i < ncand) {
                int b = cand[i];
                if (!inbox(px[b], py[b], pz[b], rmin, rsize)) atomicMin(&first, i);
            }
            __syncthreads();
            if (first != INT_MAX) break;
            __syncthreads();
        }
        int f = first;
        __syncthreads();
        if (f == INT_MAX) break;
        if (threadIdx.x == 0) {
            int b = cand[f];
            double x[3] = {px[b], py[b], pz[b]};
            int k = 0;
            while (!inbox(x[0], x[1], x[2], rmin, rsize)) {     // load.c:74-93
                if (k >= 1100) {          // non-finite position: the box can never hold it
                    doublings = -1000000;
                    break;
                }
                double rmid[3];
                for (int d = 0; d < 3; d++) rmid[d] = dadd(rmin[d], dmul(0.5, rsize));
                for (int d = 0; d < 3; d++)
                    if (x[d] < rmid[d]) rmin[d] = dsub(rmin[d], rsize);
                rsize = dmul(2.0, rsize);
                k++;
            }
            if (b == second_massive && k >= 2) {   // grafted over a lone first body
                chain_before = doublings;
                chain_k = k;
            }
            doublings += k;
        }
        __syncthreads();
        pos = f + 1;
    }
    // A non-finite position of a massive body, or a chain whose cells lie deeper
    // than the node arrays go: refused, the box stays as it was.
    const int chain = chain_before >= 0 ? doublings - chain_before - 1 : -1;
    if (threadIdx.x == 0 && (doublings < 0 || chain > HC_MAXLEVEL)) {
        if (atomicCAS(&st->error, 0, HC_ERR_ARG) == 0) st->info = doublings < 0 ? -1 : chain;
        box->chain_lmax = box->chain_lmin = -1;
        return;
    }
    if (threadIdx.x == 0) {
        box->rmin[0] = rmin[0];
        box->rmin[1] = rmin[1];
        box->rmin[2] = rmin[2];
        box->rsize = rsize;
        if (chain_before >= 0) {
            int e = doublings - chain_before;       // levels between that box and the final root
            box->chain_lmax = e - 1;
            box->chain_lmin = e - chain_k + 1;
        } else {
            box->chain_lmax = -1;
            box->chain_lmin = -1;
        }
        double d = dmul(rsize, rsize);
        for (int l = 0; l <= HC_MAXLEVEL; l++) {
            box->dsq[l] = d;
            d = ddiv(d, 4.0);
        }
    }
}

// ---------------- keys ----------------

__device__ __forceinline__ unsigned long long spread21(unsigned v)
{
    unsigned long long x = v & 0x1fffffull;
    x = (x | (x << 32)) & 0x1f00000000ffffull;
    x = (x | (x << 16)) & 0x1f0000ff0000ffull;
    x = (x | (x << 8)) & 0x100f00f00f00f00full;
    x = (x | (x << 4)) & 0x10c30c30c30c30c3ull;
    x = (x | (x << 2)) & 0x1249249249249249ull;
    return x;
}

__device__ __forceinline__ uint32_t spread9(unsigned v)
{
    uint32_t x = v & 0x1ffu;
    x = (x | (x << 16)) & 0x030000ffu;
    x = (x | (x << 8)) & 0x0300f00fu;
    x = (x | (x << 4)) & 0x030c30c3u;
    x = (x | (x << 2)) & 0x09249249u;
    return x;
}

__device__ __forceinline__ int intcoord_clamped(double x, double rmin, double rsize)
{
    int xi;
    if (intcoord1(x, rmin, rsize, &xi)) return xi;
    double xsc = scaled(x, rmin, rsize);
    return xsc < 0.0 ? 0 : HC_IMAX - 1;   // massless bodies / test points outside the box
}

// intcoord_clamped for a box of size 2^E, with one FP64 operation.  With a
// power-of-two size the reference's only rounding step is d = x - rmin (the
// scaling by 2^-E and by IMAX = 2^30 is exact), so
// floor(IMAX (x - rmin) / rsize) is d's significand shifted right by
// 22 + E - exponent(d), and 0 <= xsc < 1 reads off d's sign and exponent.
// Outside the box: 0 below it (negative d), IMAX - 1 above it and for NaN.
__device__ __forceinline__ int intcoord_pow2(double x, double rmin, int E)
{
    const long long b = __double_as_longlong(dsub(x, rmin));
    const int ef = (int)((b >> 52) & 0x7ff);
    const long long frac = b & 0xfffffffffffffll;
    if (ef == 0x7ff) return frac ? HC_IMAX - 1 : (b < 0 ? 0 : HC_IMAX - 1);   // NaN, -inf, +inf
    if (b < 0) return 0;                    // negative, or -0.0 (inside, cell 0)
    const int ex = ef ? ef - 1023 : -1022;  // d = sig * 2^(ex - 52)
    if (ex >= E) return HC_IMAX - 1;        // d >= 2^E: xsc >= 1
    const long long sig = ef ? (frac | (1ll << 52)) : frac;
    const int s = 22 + E - ex;              // > 22
    return s >= 64 ? 0 : (int)(sig >> s);
}

// Keys of the bodies (or test points), the digit counts of the sort's eight
// passes (counts: [8][256], null for the small sort), and with body the bodies'
// positions and masses as one 32-byte record each: the leaf records gather one
// sector per body from it instead of four.
__global__ void __launch_bounds__(256) k_keys(const double *x, const double *y, const double *z, const double *mass,
                                              int64_t n, const hc_box *box, unsigned long long *khi, uint32_t *klo,
                                              double4_32a *body, uint32_t *counts)
{
    __shared__ uint32_t h[8][256];
    if (counts) {
        for (int p = 0; p < 8; p++) h[p][threadIdx.x] = 0;
        __syncthreads();
    }
    double r0 = box->rmin[0], r1 = box->rmin[1], r2 = box->rmin[2], rs = box->rsize;
    // rs = 2^E exactly when its significand bits are zero (a normal double)
    const uint64_t rb = hc_dbits(rs);
    const int ref = (int)((rb >> 52) & 0x7ff), E = ref - 1023;
    const bool pow2 = (rb & 0xfffffffffffffull) == 0 && ref > 0 && ref < 0x7ff && !(rb >> 63);
#pragma unroll 2
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
        const double xi = x[i], yi = y[i], zi = z[i];
        unsigned ix, iy, iz;
        if (pow2) {
            ix = intcoord_pow2(xi, r0, E);
            iy = intcoord_pow2(yi, r1, E);
            iz = intcoord_pow2(zi, r2, E);
        } else {
            ix = intcoord_clamped(xi, r0, rs);
            iy = intcoord_clamped(yi, r1, rs);
            iz = intcoord_clamped(zi, r2, rs);
        }
        const unsigned long long k = (spread21(ix >> 9) << 2) | (spread21(iy >> 9) << 1) | spread21(iz >> 9);
        khi[i] = k;
        if (klo) klo[i] = (spread9(ix) << 2) | (spread9(iy) << 1) | spread9(iz);
        if (body) body[i] = make_double4_32a(xi, yi, zi, mass[i]);
        if (counts)
#pragma unroll
            for (int p = 0; p < 8; p++) atomicAdd(&h[p][(k >> (8 * p)) & 255u], 1u);
    }
    if (counts) {
        __syncthreads();
        for (int p = 0; p < 8; p++)
            if (h[p][threadIdx.x]) atomicAdd(&counts[p * 256 + threadIdx.x], h[p][threadIdx.x]);
    }
}

// ---------------- massive compaction and cell enumeration ----------------

// Massive bodies in key order (tree input) and the walk's target order: massive
// bodies in key order, then massless ones in key order (their number is known
// after the pass; k_target_tail appends them).  Only for systems that have
// massless bodies: otherwise the sorted arrays are the massive ones.
constexpr int MC_ITEMS = 8, MC_TILE = 256 * MC_ITEMS;
__global__ void __launch_bounds__(256) k_massive(const uint32_t *sidx, const unsigned long long *khi, const double *mass,
                                                 int64_t n, hc_box *box, unsigned long long *mhi, uint32_t *midx,
                                                 uint32_t *massless, uint32_t *status, uint32_t *ctr, int *err)
{
    __shared__ uint32_t wsum[8], s_tile, s_prefix;
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    if (threadIdx.x == 0) s_tile = atomicAdd(ctr, 1u);
    __syncthreads();
    const int64_t tile = s_tile, base = tile * MC_TILE + wid * (MC_TILE / 8);
    uint32_t idx[MC_ITEMS], bal[MC_ITEMS], cnt = 0;
#pragma unroll
    for (int r = 0; r < MC_ITEMS; r++) {
        const int64_t s = base + r * 32 + lane;
        idx[r] = s < n ? sidx[s] : 0u;
        bal[r] = __ballot_sync(0xffffffffu, s < n && hc_nonzero(mass[idx[r]]));
        cnt += __popc(bal[r]);
    }
    if (lane == 0) wsum[wid] = cnt;
    __syncthreads();
    if (wid == 0) {
        const uint32_t agg = __reduce_add_sync(0xffffffffu, lane < 8 ? wsum[lane] : 0u);
        const uint32_t prefix = tile_prefix(status, tile, agg, err);
        if (lane == 0) {
            s_prefix = prefix;
            if ((tile + 1) * MC_TILE >= n) box->nmassive = (int)(prefix + agg);   // the last tile
        }
    }
    __syncthreads();
    uint32_t rank = s_prefix;
    for (int w = 0; w < wid; w++) rank += wsum[w];
#pragma unroll
    for (int r = 0; r < MC_ITEMS; r++) {
        const int64_t s = base + r * 32 + lane;
        const uint32_t mine = rank + __popc(bal[r] & ((1u << lane) - 1u));
        if (s < n) {
            if ((bal[r] >> lane) & 1u) {
                mhi[mine] = khi[s];
                midx[mine] = idx[r];
            } else {
                massless[s - mine] = idx[r];
            }
        }
        rank += __popc(bal[r]);
    }
}

__global__ void k_target_tail(int64_t n, const hc_box *box, const uint32_t *massless, uint32_t *tord)
{
    const int64_t M = box->nmassive;
    for (int64_t i = M + blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
        tord[i] = massless[i - M];
}

// common leading octal digits of the keys of massive bodies a and b (30 =
// identical); the low keys are in body order and only read where the high tie
__device__ __forceinline__ int lcp_digits(unsigned long long ha, unsigned long long hb, const uint32_t *klo,
                                          const uint32_t *midx, int a, int b)
{
    const unsigned long long x = ha ^ hb;
    if (x) return (__clzll(x) - 1) / 3;
    const uint32_t y = klo[midx[a]] ^ klo[midx[b]];
    if (y) return 21 + (__clz(y) - 5) / 3;
    return 30;
}

// Levels of the cells that start at massive body a: (dp, dm], dp = lcp with the
// body before, dm = lcp with the body after, deepened to the expansion chain's
// lowest level at the first massive body.
struct Levels {
    int dp, dm;
};

__device__ __forceinline__ int chain_level(int dm, const uint32_t *midx, int a, int chain, int first_massive)
{
    return chain > dm && (int)midx[a] == first_massive ? chain : dm;
}

// Nodes of every depth: each body's cells and its leaf, counted in columns of
// shared memory, one per lane (no conflicts, no atomics).
__global__ void __launch_bounds__(256) k_depth_count(const unsigned long long *mhi, const uint32_t *klo,
                                                     const uint32_t *midx, const hc_box *box, uint32_t *count,
                                                     hc_status *st)
{
    __shared__ uint32_t h[8][32][32];
    const int M = box->nmassive, chain = box->chain_lmax, fm = box->first_massive;
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    if ((int64_t)blockIdx.x * blockDim.x >= M) return;
    for (int d = 0; d < 32; d++) h[wid][d][lane] = 0;
    for (int a = blockIdx.x * blockDim.x + threadIdx.x; a < M; a += gridDim.x * blockDim.x) {
        const unsigned long long k = mhi[a];
        const int dp = a > 0 ? min(lcp_digits(mhi[a - 1], k, klo, midx, a - 1, a), 29) : -1;
        int dm = -1;
        if (a + 1 < M) {
            dm = lcp_digits(k, mhi[a + 1], klo, midx, a, a + 1);
            if (dm >= 30) {                    // assert(l != 0), load.c:113
                if (atomicCAS(&st->error, 0, HC_ERR_COINCIDENT) == 0) st->info = (int)midx[a];
                dm = 29;
            }
        }
        dm = chain_level(dm, midx, a, chain, fm);
        for (int L = dp + 1; L <= dm; L++) h[wid][L][lane]++;
        const int leaf = max(dp, dm) + 1;
        if (leaf <= HC_MAXLEVEL) h[wid][leaf][lane]++;     // else the chain's: k_emit_nodes adds it
    }
    __syncthreads();
    // warp w sums depths w, w + 8, ... over all warps' columns
    for (int d = wid; d < 32; d += 8) {
        uint32_t v = 0;
#pragma unroll
        for (int w = 0; w < 8; w++) v += h[w][d][lane];
        v = __reduce_add_sync(0xffffffffu, v);
        if (lane == 0 && v) atomicAdd(&count[d], v);
    }
}

// The nodes in breadth-first order.  A tile holds TB consecutive massive
// bodies, TI per thread; a thread's nodes are counted per depth, the counts
// scanned over the threads and (look-back, one depth per lane) over the tiles.
// A node's place is its depth's start + the nodes of its depth before it in
// pre-order; link = the start of the next depth + the nodes of that depth
// before it: a cell's first child, and the next node's link is the end of its
// children.
constexpr int TI = 8, TB = 256 * TI;
__global__ void __launch_bounds__(256) k_emit_nodes(const unsigned long long *mhi, const uint32_t *klo,
                                                    const uint32_t *midx, hc_box *box, int64_t maxcell,
                                                    const uint32_t *count, uint32_t *bfs_a, int32_t *bfs_link,
                                                    uint8_t *bfs_d, uint32_t *status, uint32_t *ctr, hc_status *st)
{
    __shared__ unsigned long long sk[TB + 2];      // keys of bodies base - 1 .. base + TB
    __shared__ __align__(16) uint16_t cnt[32][256];    // scanned in 16-byte words
    __shared__ int start[33], place[33];
    __shared__ uint32_t s_tile;
    const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
    if (tid == 0) s_tile = atomicAdd(ctr, 1u);
    __syncthreads();
    const int64_t tile = s_tile, base = tile * TB;
    const int M = box->nmassive, chain = box->chain_lmax, fm = box->first_massive;
    if (base >= M && tile > 0) return;
    if (wid == 0) {
        const uint32_t c = count[lane], incl = warp_inclusive_scan(c);
        start[lane] = (int)(incl - c);
        if (lane == 31) start[32] = (int)incl;
    }
    __syncthreads();
    // a chain down to the last level has its body one deeper, the only node there
    const int total = start[32] + (chain == HC_MAXLEVEL ? 1 : 0), ncell = total - M;
    const bool fits = ncell <= maxcell;            // makecell, load.c:237-239
    if (tile == 0) {
        if (tid < 33) box->level_start[tid] = fits ? start[tid] : 0;
        if (tid == 33) box->level_start[33] = fits ? total : 0;
        if (tid == 0) {
            int md = 0;
            for (int l = 0; l < 32; l++)
                if (fits && start[l + 1] > start[l]) md = l;
            box->max_depth = md;
            box->ncell = fits ? ncell : 0;         // else later kernels see an empty tree
            box->nnode = fits ? total : 0;
            if (!fits) {
                if (atomicCAS(&st->error, 0, HC_ERR_CELLS) == 0) st->info = (int)maxcell;
            }
        }
    }
    if (!fits || base >= M) return;                // the whole tile, and every other
    const int tn = (int)(M - base < TB ? M - base : TB);
    for (int j = tid; j < tn + 2; j += 256) {
        const int64_t a = base + j - 1;
        sk[j] = a >= 0 && a < M ? mhi[a] : 0ull;
    }
    for (int d = 0; d < 32; d++) cnt[d][tid] = 0;
    __syncthreads();
    int8_t lev[TI + 1];                            // lcp of bodies a - 1, a for the thread's a and one more
#pragma unroll
    for (int j = 0; j <= TI; j++) {
        const int e = tid * TI + j;
        const int64_t a = base + e;
        lev[j] = e <= tn && a > 0 && a < M
                     ? (int8_t)min(lcp_digits(sk[e], sk[e + 1], klo, midx, (int)a - 1, (int)a), 29)
                     : (int8_t)-1;
    }
#pragma unroll
    for (int j = 0; j < TI; j++) {
        const int e = tid * TI + j;
        if (e >= tn) continue;
        const int dp = lev[j], dm = chain_level(lev[j + 1], midx, (int)base + e, chain, fm);
        for (int L = dp + 1; L <= dm; L++) cnt[L][tid]++;
        if (max(dp, dm) < HC_MAXLEVEL) cnt[max(dp, dm) + 1][tid]++;
    }
    __syncthreads();
    // warp w scans depths 4 w .. 4 w + 3 over the threads (eight per lane)
#pragma unroll
    for (int q = 0; q < 4; q++) {
        const int d = wid * 4 + q;
        uint4 v = *reinterpret_cast<const uint4 *>(&cnt[d][lane * 8]);
        uint32_t w[4] = {v.x, v.y, v.z, v.w}, sum = 0;
#pragma unroll
        for (int i = 0; i < 4; i++) {
            const uint32_t lo = w[i] & 0xffffu, hi = w[i] >> 16;
            w[i] = sum | (sum + lo) << 16;
            sum += lo + hi;
        }
        const uint32_t incl = warp_inclusive_scan(sum), ex = incl - sum;
        *reinterpret_cast<uint4 *>(&cnt[d][lane * 8]) =
            make_uint4(w[0] + ex * 0x10001u, w[1] + ex * 0x10001u, w[2] + ex * 0x10001u, w[3] + ex * 0x10001u);
        if (lane == 31) place[d] = (int)incl;      // the tile's count of depth d
    }
    __syncthreads();
    if (wid == 0) {
        const uint32_t before = digit_prefix(status, tile, 32, lane, (uint32_t)place[lane], &st->error);
        __syncwarp();
        place[lane] = start[lane] + (int)before;
        if (lane == 0) place[32] = 0;
    }
    __syncthreads();
#pragma unroll
    for (int j = 0; j < TI; j++) {
        const int e = tid * TI + j;
        if (e >= tn) continue;
        const int a = (int)base + e, dp = lev[j], dm = chain_level(lev[j + 1], midx, a, chain, fm);
        const int leaf = max(dp, dm) + 1;          // its parent is the deepest cell holding the body
        for (int L = dp + 1; L <= leaf; L++) {
            if (L > dm) L = leaf;
            const int k = L <= HC_MAXLEVEL ? place[L] + cnt[L][tid]++ : total - 1;
            bfs_a[k] = L == leaf ? (uint32_t)(-1 - a) : (uint32_t)a;
            bfs_link[k] = L < 31 ? place[L + 1] + cnt[L + 1][tid] : start[32];
            bfs_d[k] = (uint8_t)L;
        }
    }
}

// hi = RN_f32(v), lo = RN_f32(v - hi), on the double's bits (no FP64 pipe)
__device__ __forceinline__ void split_hilo(double v, float *hi, float *lo) { hc_split_hilo(v, hi, lo); }

// The upward pass takes each level's cells only, grouped by child count: the
// cells of a warp then run the same number of FP64 child steps and no lane
// idles on a body leaf (the levels interleave cells and leaves in key order).
// Group of a cell: depth * 8 + (children - 1); order inside a group is free.
__device__ __forceinline__ int cell_group(int2 C) { return min((C.y >> 8), 31) * 8 + (C.y & 255) - 1; }

// Node records that do not need the upward pass: body leaves (from the bodies'
// 32-byte records) and the child range of every cell; counts the cells of each
// group.  Bound by the gather of the leaves' records and the stores (36 us at
// N = 2^20): with the four FP64 arrays gathered apart (four 32-byte sectors a
// leaf instead of one) it took 56 us, 380 at 2^22 and 1960 at 2^24.
__global__ void __launch_bounds__(256) k_node_init(const uint8_t *bdep, const uint32_t *ba, const int32_t *blink,
                                                   const uint32_t *midx, const double4_32a *body, const hc_box *box,
                                                   int2 *nodeC, float4 *nodeAB, float4 *nodeQ, double4_32a *nodeD,
                                                   uint32_t *gcount, hc_status *st)
{
    __shared__ uint32_t h[256];
    const int nn = box->nnode;
    if ((int64_t)blockIdx.x * blockDim.x >= nn) return;
    h[threadIdx.x] = 0;
    __syncthreads();
    for (int k = blockIdx.x * blockDim.x + threadIdx.x; k < nn; k += gridDim.x * blockDim.x) {
        const int D = (int)bdep[k];
        int a = (int)ba[k];
        if (a < 0) {
            a = -1 - a;
            const double4_32a b = body[midx[a]];
            nodeD[k] = b;
            float4 A, B;
            split_hilo(b.x, &A.x, &B.x);
            split_hilo(b.y, &A.y, &B.y);
            split_hilo(b.z, &A.z, &B.z);
            A.w = hc_d2f_rn(b.w);
            B.w = -1.0f;
            nodeAB[2 * (int64_t)k] = A;
            nodeAB[2 * (int64_t)k + 1] = B;
            nodeQ[2 * (int64_t)k] = make_float4(0.f, 0.f, 0.f, 0.f);
            nodeQ[2 * (int64_t)k + 1] = make_float4(0.f, 0.f, 1.f, 0.f);   // no quadrupole, one body, bmax 0
            nodeC[k] = make_int2(-1 - a, D << 8);      // body leaf: -1 - massive rank
        } else {
            // the children end where those of the next node of the depth begin
            int fc = blink[k];
            const int end = k + 1 < box->level_start[D + 1] ? blink[k + 1] : box->level_start[D + 2];
            int nc = end - fc;
            if (fc <= k || nc < 1 || nc > 8 || fc + nc > nn) {   // children follow their parent
                if (atomicCAS(&st->error, 0, HC_ERR_STATE) == 0) st->info = k;
                fc = k + 1;
                nc = 0;
            }
            const int2 C = make_int2(fc, nc | (D << 8));
            nodeC[k] = C;
            if (nc >= 1) atomicAdd(&h[cell_group(C)], 1u);
        }
    }
    __syncthreads();
    if (h[threadIdx.x]) atomicAdd(&gcount[threadIdx.x], h[threadIdx.x]);
}

// Places each block's cells: the group offsets are the exclusive scan of the 256
// counts (every block makes its own; block 0 leaves them in off[0..256] for
// the upward pass), then one reservation per group per block and slots handed
// out inside the reservation.
__global__ void __launch_bounds__(256) k_cell_place(const int2 *nodeC, const hc_box *box, const uint32_t *count,
                                                    uint32_t *cur, uint32_t *off, int4 *perm)
{
    __shared__ uint32_t h[256], base[256], first[256], sh[32];
    const int nn = box->nnode;
    if (blockIdx.x > 0 && (int64_t)blockIdx.x * blockDim.x >= nn) return;
    {
        const uint32_t v = count[threadIdx.x];
        uint32_t total;
        first[threadIdx.x] = block_exclusive_scan<uint32_t>(v, sh, &total);
        if (blockIdx.x == 0) {
            off[threadIdx.x] = first[threadIdx.x];
            if (threadIdx.x == 0) off[256] = total;
        }
    }
    for (int k0 = blockIdx.x * blockDim.x; k0 < nn; k0 += gridDim.x * blockDim.x) {
        const int k = k0 + threadIdx.x;
        h[threadIdx.x] = 0;
        __syncthreads();
        int grp = -1, slot = 0;
        int2 C = make_int2(-1, 0);
        if (k < nn) {
            C = nodeC[k];
            if (C.x >= 0 && (C.y & 255) >= 1) {
                grp = cell_group(C);
                slot = (int)atomicAdd(&h[grp], 1u);
            }
        }
        __syncthreads();
        if (h[threadIdx.x]) base[threadIdx.x] = first[threadIdx.x] + atomicAdd(&cur[threadIdx.x], h[threadIdx.x]);
        __syncthreads();
        if (grp >= 0) perm[base[grp] + slot] = make_int4(k, C.x, C.y, 0);   // the cell and its child links
        __syncthreads();
    }
}

// hackcofm (load.c:183-226), deepest level first.  Children are summed in
// subindex order exactly as hackcofm does.
//
// Bound by the dependent chain of a cell (children's loads, FP64 sums,
// divisions, records) at every level, and by the FP64 pipe at levels of 10^5
// cells.  So the two halves of the work run beside each other on warps of their
// own: in one step the FP64 half (mass and centre of mass) of level D, and the
// FP32 half (quadrupole, extent, body count) of level D + 1, which reads what
// the step before wrote.  Levels with few cells give each cell four lanes (x,
// y, z, mass), so that its three divisions run at once; with many cells one
// lane a cell does a third less work on the FP64 pipe.  One warp doing both
// halves of a cell one after the other took 119 us at 50,021 bodies (now 78),
// 243 at 2^20 (206) and 543 at 2^22 (537, bound by the FP64 pipe).  Four lanes
// a cell in the FP32 half too, or fewer children in flight, were slower.

// mass and centre of mass, one lane per cell; load.c:193-224, bit-exact
__device__ __forceinline__ void cofm_mass(int4 P, float dsqf, double4_32a *nodeD, float4 *nodeAB)
{
    const int k = P.x, fc = P.y, nc = P.z & 255;
    double m = 0.0, cx = 0.0, cy = 0.0, cz = 0.0;
#pragma unroll
    for (int h = 0; h < 8; h += 4) {
        // the children's loads are issued together (predicated on the child
        // count), not one dependent round trip per child
        double4_32a c[4];
#pragma unroll
        for (int i = 0; i < 4; i++)
            if (h + i < nc) c[i] = nodeD[fc + h + i];
#pragma unroll
        for (int i = 0; i < 4; i++) {
            if (h + i < nc) {
                m = dadd(m, c[i].w);
                cx = dadd(cx, dmul(c[i].x, c[i].w));
                cy = dadd(cy, dmul(c[i].y, c[i].w));
                cz = dadd(cz, dmul(c[i].z, c[i].w));
            }
        }
    }
    cx = ddiv(cx, m);
    cy = ddiv(cy, m);
    cz = ddiv(cz, m);
    float4 A, B;
    split_hilo(cx, &A.x, &B.x);
    split_hilo(cy, &A.y, &B.y);
    split_hilo(cz, &A.z, &B.z);
    A.w = hc_d2f_rn(m);
    B.w = dsqf;
    nodeD[k] = make_double4_32a(cx, cy, cz, m);
    nodeAB[2 * (int64_t)k] = A;
    nodeAB[2 * (int64_t)k + 1] = B;
}

// the same with four lanes per cell: lane q = 0, 1, 2 the coordinates, 3 the mass
__device__ __forceinline__ void cofm_mass4(int4 P, int q, float dsqf, double *nodeD, float *nodeAB)
{
    const int64_t k = P.x;
    const int nc = P.z & 255;
    const double *c = nodeD + 4 * (int64_t)P.y;
    double cm[8], cq[8], m = 0.0, v = 0.0;
#pragma unroll
    for (int i = 0; i < 8; i++)
        if (i < nc) {
            cm[i] = c[4 * i + 3];
            cq[i] = c[4 * i + q];
        }
#pragma unroll
    for (int i = 0; i < 8; i++)
        if (i < nc) {
            m = dadd(m, cm[i]);
            v = dadd(v, dmul(cq[i], cm[i]));
        }
    float hi, lo;
    if (q < 3) {
        v = ddiv(v, m);
        split_hilo(v, &hi, &lo);
    } else {
        v = m;
        hi = hc_d2f_rn(m);
        lo = dsqf;
    }
    nodeD[4 * k + q] = v;
    nodeAB[8 * k + q] = hi;
    nodeAB[8 * k + 4 + q] = lo;
}

// Quadrupole, extent and body count of a cell.  Children's offsets from the
// centre of mass in FP32, from the hi + lo positions ((hi - hi) + (lo - lo)):
// no FP64 work per child.  bmax: children's extents shifted to the new centre;
// Q = sum_child [ m (3 dr dr^T - |dr|^2 I) + Q_child ], dr = x_child - x_cm.
__device__ __forceinline__ void cofm_quad(int4 P, int usequad, const float4 *nodeAB, float4 *nodeQ)
{
    const int k = P.x, fc = P.y, nc = P.z & 255;
    const float4 A = nodeAB[2 * (int64_t)k], B = nodeAB[2 * (int64_t)k + 1];
    float bmax = 0.f, nbody = 0.f;
    float Q[6] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
#pragma unroll
    for (int h = 0; h < 8; h += 4) {
        float4 ca[4], cb[4], q0[4], q1[4];
#pragma unroll
        for (int i = 0; i < 4; i++) {
            const int64_t ch = 2 * (int64_t)(fc + h + i);
            if (h + i < nc) {
                ca[i] = nodeAB[ch];
                cb[i] = nodeAB[ch + 1];
                q1[i] = nodeQ[ch + 1];
                if (usequad) q0[i] = nodeQ[ch];
            }
        }
#pragma unroll
        for (int i = 0; i < 4; i++) {
            if (h + i >= nc) continue;
            const float dx = (ca[i].x - A.x) + (cb[i].x - B.x), dy = (ca[i].y - A.y) + (cb[i].y - B.y),
                        dz = (ca[i].z - A.z) + (cb[i].z - B.z);
            const float r2 = dx * dx + dy * dy + dz * dz;
            bmax = fmaxf(bmax, sqrtf(r2) + q1[i].w);
            nbody += q1[i].z;                // bodies in the cell (exact below 2^24)
            if (usequad) {
                const float mr = ca[i].w;
                Q[0] += mr * (3.f * dx * dx - r2) + q0[i].x;
                Q[1] += mr * (3.f * dx * dy) + q0[i].y;
                Q[2] += mr * (3.f * dx * dz) + q0[i].z;
                Q[3] += mr * (3.f * dy * dy - r2) + q0[i].w;
                Q[4] += mr * (3.f * dy * dz) + q1[i].x;
                Q[5] += mr * (3.f * dz * dz - r2) + q1[i].y;
            }
        }
    }
    nodeQ[2 * (int64_t)k] = make_float4(Q[0], Q[1], Q[2], Q[3]);
    nodeQ[2 * (int64_t)k + 1] = make_float4(Q[4], Q[5], nbody, bmax);
}

// One step: w of nw warps works on its half's level (mass: level D, else D + 1).
// Consecutive 32-cell chunks go to consecutive warps, which the callers number
// so that they sit on different SMs.
__device__ __forceinline__ void cofm_step(bool mass, int D, int maxd, int w, int nw, int usequad, const hc_box *box,
                                          double4_32a *nodeD, float4 *nodeAB, float4 *nodeQ, const int4 *cperm,
                                          const uint32_t *coff)
{
    const int L = mass ? D : D + 1, lane = (int)(threadIdx.x & 31);
    if (L < 0 || L > maxd) return;
    // the level's cells only, grouped by child count (coff: group offsets)
    const int ls = (int)coff[L * 8], le = (int)coff[L * 8 + 8];
    const float dsqf = hc_d2f_rn(box->dsq[L]);
    if (!mass) {
        for (int j = ls + w * 32 + lane; j < le; j += nw * 32) cofm_quad(cperm[j], usequad, nodeAB, nodeQ);
    } else if (le - ls <= nw * 8) {
        const int j = ls + w * 8 + (lane >> 2);
        if (j < le) cofm_mass4(cperm[j], lane & 3, dsqf, reinterpret_cast<double *>(nodeD), reinterpret_cast<float *>(nodeAB));
    } else {
        for (int j = ls + w * 32 + lane; j < le; j += nw * 32) cofm_mass(cperm[j], dsqf, nodeD, nodeAB);
    }
}

__global__ void __launch_bounds__(256, 2) k_cofm_all(int usequad, const hc_box *box, double4_32a *nodeD, float4 *nodeAB,
                                                     float4 *nodeQ, const int4 *cperm, const uint32_t *coff)
{
    cg::grid_group grid = cg::this_grid();
    const int maxd = box->nnode > 0 ? box->max_depth : -1, wid = (int)(threadIdx.x >> 5);
    const int w = (wid >> 1) * (int)gridDim.x + (int)blockIdx.x, nw = (int)(blockDim.x >> 6) * (int)gridDim.x;
    for (int D = maxd; D >= -1; D--) {
        cofm_step(!(wid & 1), D, maxd, w, nw, usequad, box, nodeD, nodeAB, nodeQ, cperm, coff);
        if (D >= 0) grid.sync();
    }
}

// The same for small systems in one cluster of eight blocks: a cluster barrier
// per level instead of the grid's, and registers for all of a cell's loads
// (128 bodies: 68 -> 33 us, 4096: 103 -> 61).  Above COFM_SMALL eight SMs' FP64
// pipes would take longer than the grid's barriers cost.
constexpr int COFM_CLUSTER = 8, COFM_SMALL = 16384, COFM_THREADS = 256;
__global__ void __cluster_dims__(COFM_CLUSTER, 1, 1) __launch_bounds__(COFM_THREADS, 1)
    k_cofm_small(int usequad, const hc_box *box, double4_32a *nodeD, float4 *nodeAB, float4 *nodeQ, const int4 *cperm,
                 const uint32_t *coff)
{
    cg::cluster_group cluster = cg::this_cluster();
    const int maxd = box->nnode > 0 ? box->max_depth : -1, wid = (int)(threadIdx.x >> 5);
    const int w = (wid >> 1) * COFM_CLUSTER + (int)blockIdx.x;
    for (int D = maxd; D >= -1; D--) {
        cofm_step(!(wid & 1), D, maxd, w, COFM_THREADS / 64 * COFM_CLUSTER, usequad, box, nodeD, nodeAB, nodeQ, cperm,
                  coff);
        if (D >= 0) cluster.sync();
    }
}

// ---------------- walk groups aligned with the tree ----------------
// A group is a run of massive bodies (in key order) that lie in one cell of
// at most gmax (<= HC_GROUP) bodies: the cells (and lone bodies) with <= gmax bodies
// whose parent has more, consecutive siblings packed while they fit.

// A node's body count: the upward pass's, 1 for a leaf (FP32, exact below 2^24;
// above it only "more than gmax" matters here).
__device__ __forceinline__ int node_count(const float4 *nodeQ, int k) { return (int)fminf(nodeQ[2 * (int64_t)k + 1].z, 2.0e9f); }

// Packs of node k's children into groups (for the root also itself, when it is
// small): calls f(first body, bodies) for each and returns their number.  cnt:
// the node's bodies.  The children are read together: one after the other they
// were a chain of up to eight round trips, in a kernel that only waits (2^22
// bodies 155 -> 120 us).
template <typename F>
__device__ __forceinline__ int node_packs(const uint32_t *ba, const float4 *nodeQ, const int2 *nodeC, int k, int cnt,
                                          int gmax, F f)
{
    int packs = 0;
    if (cnt <= gmax) {                         // only the root can be a small group on its own here
        if (k == 0) {
            const int a = (int)ba[k];
            f(a < 0 ? -1 - a : a, cnt);
            packs = 1;
        }
        return packs;
    }
    const int2 C = nodeC[k];
    const int fc = C.x, nc = C.y & 255;
    int first[8], cc[8];
#pragma unroll
    for (int i = 0; i < 8; i++) {
        first[i] = i < nc ? (int)ba[fc + i] : 0;
        cc[i] = i < nc ? node_count(nodeQ, fc + i) : 0;
    }
    int cur = 0, cur_first = 0;
#pragma unroll
    for (int i = 0; i < 8; i++) {
        if (i >= nc) break;
        if (cc[i] > gmax || cur + cc[i] > gmax) {
            if (cur > 0) {
                f(cur_first, cur);
                packs++;
                cur = 0;
            }
            if (cc[i] > gmax) continue;
        }
        if (cur == 0) cur_first = first[i] < 0 ? -1 - first[i] : first[i];
        cur += cc[i];
    }
    if (cur > 0) {
        f(cur_first, cur);
        packs++;
    }
    return packs;
}

// The group table in node order, in one pass (decoupled look-back over tiles of
// GI rounds of 256 consecutive nodes).
constexpr int GI = 4, GTILE = 256 * GI;
__global__ void __launch_bounds__(256) k_groups(const uint32_t *ba, const float4 *nodeQ, const int2 *nodeC, hc_box *box,
                                                int gmax, int32_t *gstart, int32_t *gcount, uint32_t *status,
                                                uint32_t *ctr, int *err)
{
    __shared__ uint32_t s_tile, s_prefix, wsum[GI][8];
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    if (threadIdx.x == 0) s_tile = atomicAdd(ctr, 1u);
    __syncthreads();
    const int64_t tile = s_tile, base = tile * GTILE + threadIdx.x;
    const int nn = box->nnode;
    if (tile * GTILE >= nn) {
        if (tile == 0 && threadIdx.x == 0) box->ngroups = 0;
        return;
    }
    uint32_t n[GI], ex[GI];
    int cnt[GI];
#pragma unroll
    for (int r = 0; r < GI; r++) cnt[r] = base + r * 256 < nn ? node_count(nodeQ, (int)(base + r * 256)) : 0;
#pragma unroll
    for (int r = 0; r < GI; r++) {
        const int64_t k = base + r * 256;
        n[r] = k < nn ? (uint32_t)node_packs(ba, nodeQ, nodeC, (int)k, cnt[r], gmax, [](int, int) {}) : 0u;
    }
#pragma unroll
    for (int r = 0; r < GI; r++) {
        const uint32_t incl = warp_inclusive_scan(n[r]);
        ex[r] = incl - n[r];
        if (lane == 31) wsum[r][wid] = incl;
    }
    __syncthreads();
    if (wid == 0) {                            // GI * 8 sums, one per lane, in node order
        static_assert(GI * 8 == 32, "one warp scans the warps' sums");
        const uint32_t v = (&wsum[0][0])[lane], incl = warp_inclusive_scan(v);
        const uint32_t agg = __shfl_sync(0xffffffffu, incl, 31);
        (&wsum[0][0])[lane] = incl - v;
        const uint32_t prefix = tile_prefix(status, tile, agg, err);
        if (lane == 0) {
            s_prefix = prefix;
            if ((tile + 1) * GTILE >= nn) box->ngroups = (int)(prefix + agg);    // the last tile
        }
    }
    __syncthreads();
#pragma unroll
    for (int r = 0; r < GI; r++) {
        if (n[r] == 0) continue;
        uint32_t out = s_prefix + wsum[r][wid] + ex[r];
        node_packs(ba, nodeQ, nodeC, (int)(base + r * 256), cnt[r], gmax, [&](int first, int bodies) {
            gstart[out] = first;
            gcount[out] = bodies;
            out++;
        });
    }
}

// ---------------- treecode1 critical radii ----------------
// setrcrit (treecode1/treeload.c:232-252) for every cell: the cell's centre
// and size follow from the integer coordinate of its first body at the
// cell's depth; cm is the FP64 centre of mass.
//   bh86: (size/theta)^2;  sw94: (max distance from cm to a corner)^2/theta^2;
//   "new" (treecode1's default): (size/theta + |cm - centre|)^2;
//   theta = 0: (2 rsize)^2 (always open).
__global__ void k_rcrit(int kind, double theta, const hc_box *box, const uint32_t *ba,
                        const uint32_t *midx, const double *px, const double *py, const double *pz, const int2 *nodeC,
                        const double4_32a *nodeD, float *rcrit2)
{
    const int nn = box->nnode;
    const double rsize = box->rsize;
    for (int k = blockIdx.x * blockDim.x + threadIdx.x; k < nn; k += gridDim.x * blockDim.x) {
        const int2 C = nodeC[k];
        if (C.x < 0) continue;                           // body leaf
        const int D = C.y >> 8;
        const uint32_t o = midx[ba[k]];
        const double4_32a nd = nodeD[k];
        const double p[3] = {px[o], py[o], pz[o]}, cm[3] = {nd.x, nd.y, nd.z};
        const double size = ldexp(rsize, -D), unit = ldexp(rsize, -30);
        const int shift = 30 - D;
        double off2 = 0.0, bmax2 = 0.0;
        for (int d = 0; d < 3; d++) {
            int xi = 0;
            intcoord1(p[d], box->rmin[d], rsize, &xi);
            const double corner = box->rmin[d] + (double)((xi >> shift) << shift) * unit;
            const double dk = cm[d] - (corner + 0.5 * size);       // offset of cm from the centre
            off2 += dk * dk;
            const double dc = dk + 0.5 * size;                      // distance from the low corner
            const double m = dc > size - dc ? dc : size - dc;
            bmax2 += m * m;
        }
        double r2;
        if (theta == 0.0) r2 = 4.0 * rsize * rsize;
        else if (kind == 1) r2 = (size / theta) * (size / theta);
        else if (kind == 2) r2 = bmax2 / (theta * theta);
        else {
            const double r = size / theta + sqrt(off2);
            r2 = r * r;
        }
        rcrit2[k] = (float)r2;
    }
}

}  // namespace

void hc_rcrit_launch(hc_ctx *c, int kind, double theta)
{
    k_rcrit<<<hc_grid(c->maxnode, 256), 256, 0, c->stream>>>(kind, theta, c->box, c->bfs_a, c->xidx,
                                                              c->px, c->py, c->pz, c->nodeC, c->nodeD, c->rcrit2);
    c->launches++;
}

void hc_keys_for_points(hc_ctx *c, const double *x, const double *y, const double *z, int64_t n,
                        unsigned long long *khi, uint32_t *klo, double4_32a *body, uint32_t *scratch)
{
    const bool counts = !hc_sort_counts_digits(n);
    // enough blocks to hide the loads; each adds up to 2048 digit counts
    k_keys<<<hc_grid(n, 256, counts ? 152 * 4 : 152 * 16), 256, 0, c->stream>>>(x, y, z, c->mass, n, c->box, khi, klo, body,
                                                                               counts ? scratch : nullptr);
    c->launches++;
}

// The build's own scratch after the sort's: look-back words and counters, all
// zeroed together at the start of a build.
namespace {
struct BuildScratch {
    uint32_t *ctr;                       // tile counters of box, massive, emit, groups
    uint32_t *depth, *gcount, *gcur, *goff;
    uint32_t *box, *massive, *emit, *groups;
    int64_t words;                       // of all, sort included
};

BuildScratch build_scratch(uint32_t *p, int64_t n, int64_t maxnode)
{
    BuildScratch b;
    int64_t w = hc_sort_scratch_words(n);
    auto take = [&](int64_t count) {
        uint32_t *q = p ? p + w : nullptr;
        w += (count + 31) / 32 * 32;
        return q;
    };
    b.ctr = take(32);
    b.depth = take(32);
    b.gcount = take(256);
    b.gcur = take(256);
    b.goff = take(257);
    b.box = take((n + 1023) / 1024);
    b.massive = take((n + MC_TILE - 1) / MC_TILE);
    b.emit = take((n + TB - 1) / TB * 32);
    b.groups = take((maxnode + GTILE - 1) / GTILE);
    b.words = w;
    return b;
}
}  // namespace

int64_t hc_build_scratch_words(int64_t n, int64_t maxnode) { return build_scratch(nullptr, n, maxnode).words; }

// The current tree's table of walk groups of at most gmax bodies.  The build leaves
// the scratch zeroed; a table made before has used it.
int hc_groups_launch(hc_ctx *c, int gmax)
{
    const BuildScratch b = build_scratch(c->hist, c->n, c->maxnode);
    const int64_t tiles = (c->maxnode + GTILE - 1) / GTILE;
    if (c->groups_gmax > 0) {
        HC_CUDA(cudaMemsetAsync(b.groups, 0, sizeof(uint32_t) * tiles, c->stream));
        HC_CUDA(cudaMemsetAsync(b.ctr + 3, 0, sizeof(uint32_t), c->stream));
    }
    k_groups<<<(unsigned)tiles, 256, 0, c->stream>>>(c->bfs_a, c->nodeQ, c->nodeC, c->box, gmax, c->gstart, c->gcount,
                                                     b.groups, b.ctr + 3, &c->st->error);
    c->groups_gmax = gmax;
    c->launches++;
    return HC_OK;
}

// Whether a build of this configuration makes the group table: the per-body
// rule over consecutive bodies does not use it.  A walk that needs the table of
// a tree built without it makes it first (hc_walk_launch).
bool hc_build_makes_groups(const hc_ctx *c) { return c->criterion != HC_CRITERION_BODY || c->group_kind == 1; }

// Launch the whole build on the context stream without host synchronisation
// (graph-capturable); errors land in the device status word.
int hc_tree_build(hc_ctx *c)
{
    const int64_t n = c->n;
    cudaStream_t s = c->stream;
    const int B = 256;
    const BuildScratch b = build_scratch(c->hist, n, c->maxnode);
    HC_CUDA(cudaMemsetAsync(c->hist, 0, sizeof(uint32_t) * b.words, s));

    // 1. expandbox replay
    const int boxtile = 256 * box_items(n), boxtiles = (int)((n + boxtile - 1) / boxtile);
    auto *box_outside = box_items(n) == 4 ? k_box_outside<4> : k_box_outside<16>;
    box_outside<<<boxtiles, B, 0, s>>>(c->mass, c->px, c->py, c->pz, n, c->box, c->cand, c->ncand, c->first2, b.box,
                                         b.ctr, &c->st->error);
    k_box_replay<<<1, 256, 0, s>>>(c->px, c->py, c->pz, c->cand, c->ncand, c->first2, boxtiles, c->box, c->st,
                                   c->all_massive ? (int)n : -1);
    c->launches += 2;

    // 2-3. keys, sort, massive compaction
    hc_keys_for_points(c, c->px, c->py, c->pz, n, c->khi[0], c->klo, c->body, c->hist);
    const int sel = hc_radix_sort_keys(c, c->hist, c->khi, c->kval, n, c->klo);
    if (c->all_massive) {
        c->xhi = c->khi[sel];
        c->xidx = c->tord = c->kval[sel];
    } else {
        // the other buffers of the sort are free again
        c->xhi = c->khi[sel ^ 1];
        c->xidx = c->tord = c->kval[sel ^ 1];
        uint32_t *massless = reinterpret_cast<uint32_t *>(c->cand);
        k_massive<<<(unsigned)((n + MC_TILE - 1) / MC_TILE), B, 0, s>>>(c->kval[sel], c->khi[sel], c->mass, n, c->box,
                                                                        c->khi[sel ^ 1], c->kval[sel ^ 1], massless,
                                                                        b.massive, b.ctr + 1, &c->st->error);
        k_target_tail<<<hc_grid(n, B), B, 0, s>>>(n, c->box, massless, c->kval[sel ^ 1]);
        c->launches += 2;
    }

    // 4. the nodes in breadth-first order
    k_depth_count<<<hc_grid(n, B, 152 * 4), B, 0, s>>>(c->xhi, c->klo, c->xidx, c->box, b.depth, c->st);
    k_emit_nodes<<<(unsigned)((n + TB - 1) / TB), B, 0, s>>>(c->xhi, c->klo, c->xidx, c->box, c->maxcell, b.depth, c->bfs_a,
                                                           c->bfs_link, c->bfs_d, b.emit, b.ctr + 2, c->st);

    // 5. node records; cells grouped by depth and child count
    const int Gn = hc_grid(c->maxnode, B);
    k_node_init<<<Gn, B, 0, s>>>(c->bfs_d, c->bfs_a, c->bfs_link, c->xidx, c->body, c->box, c->nodeC, c->nodeAB, c->nodeQ,
                                 c->nodeD, b.gcount, c->st);
    k_cell_place<<<Gn, B, 0, s>>>(c->nodeC, c->box, b.gcount, b.gcur, b.goff, c->cperm);
    c->launches += 4;

    // 6. upward pass, deepest level first, one cooperative launch.  Work forked
    // onto the side stream joins here: nothing else runs beside the
    // cooperative launch.
    if (c->join_pending) {
        c->join_pending = false;
        HC_CUDA(cudaStreamWaitEvent(s, c->ev_join, 0));
    }
    if (n <= COFM_SMALL) {
        k_cofm_small<<<COFM_CLUSTER, COFM_THREADS, 0, s>>>(c->prm.usequad, c->box, c->nodeD, c->nodeAB, c->nodeQ, c->cperm, b.goff);
        c->launches++;
    } else {
        int usequad = c->prm.usequad;
        uint32_t *goff = b.goff;
        void *args[] = {&usequad, &c->box, &c->nodeD, &c->nodeAB, &c->nodeQ, &c->cperm, &goff};
        cudaLaunchConfig_t cfg = {};
        cfg.gridDim = dim3(c->cofm_grid);
        cfg.blockDim = dim3(256);
        cfg.stream = s;
        cudaLaunchAttribute attr;
        attr.id = cudaLaunchAttributeCooperative;
        attr.val.cooperative = 1;
        cfg.attrs = &attr;
        cfg.numAttrs = 1;
        HC_CUDA(cudaLaunchKernelExC(&cfg, (const void *)k_cofm_all, args));
        c->launches++;
    }

    // 7. walk groups aligned with the tree
    c->table_gmax = hc_table_gmax(c);
    c->groups_gmax = 0;
    c->radii_current = false;
    return hc_build_makes_groups(c) ? hc_groups_launch(c, c->table_gmax) : HC_OK;
}

int hc_tree_setup(hc_ctx *c)
{
    if (int r = hc_sort_setup(c)) return r;
    int dev = 0, nsm = 0, per = 0;
    HC_CUDA(cudaGetDevice(&dev));
    HC_CUDA(cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev));
    HC_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, k_cofm_all, 256, 0));
    if (per < 1) per = 1;
    c->cofm_grid = nsm * (per > 4 ? 4 : per);
    return HC_OK;
}

// ---------------- tree dump (host assembly from device arrays) ----------------

int hc_tree_dump_impl(hc_ctx *c, int32_t *level, int32_t *corner, int32_t *count, double *mass, double *cm,
                      double *quad, int32_t *bparent)
{
    HC_CUDA(cudaMemcpy(c->h_box, c->box, sizeof(hc_box), cudaMemcpyDeviceToHost));
    const int M = c->h_box->nmassive, nn = c->h_box->nnode;
    for (int64_t i = 0; i < c->n && bparent; i++) bparent[i] = -1;
    if (nn <= 0) return 0;
    auto H = [&](size_t bytes) { return std::unique_ptr<char[]>(new char[bytes > 0 ? bytes : 1]); };
    auto hl = H(sizeof(uint32_t) * c->n), ha = H(sizeof(int32_t) * nn), hbb = H(sizeof(int32_t) * nn),
         hmhi = H(sizeof(unsigned long long) * M), hmidx = H(sizeof(uint32_t) * M), hd = H(sizeof(double) * 4 * nn),
         hq = H(sizeof(float4) * 2 * nn);
    int32_t *pa = (int32_t *)ha.get(), *pb = (int32_t *)hbb.get();
    unsigned long long *mhi = (unsigned long long *)hmhi.get();
    uint32_t *klo = (uint32_t *)hl.get(), *midx = (uint32_t *)hmidx.get();
    double *nd = (double *)hd.get();
    float *nq = (float *)hq.get();
    std::unique_ptr<int2[]> C(new int2[nn]);
    HC_CUDA(cudaMemcpy(C.get(), c->nodeC, sizeof(int2) * nn, cudaMemcpyDeviceToHost));
    HC_CUDA(cudaMemcpy(pa, c->bfs_a, sizeof(int32_t) * nn, cudaMemcpyDeviceToHost));
    // bodies per node, summed up the children links (breadth-first: children
    // follow their parent, so one pass from the back)
    for (int k = nn - 1; k >= 0; k--) {
        int cnt = 1;
        if (C[k].x >= 0) {
            cnt = 0;
            for (int i = 0; i < (C[k].y & 255); i++) cnt += pb[C[k].x + i];
        }
        pb[k] = cnt;
    }
    HC_CUDA(cudaMemcpy(mhi, c->xhi, sizeof(unsigned long long) * M, cudaMemcpyDeviceToHost));
    HC_CUDA(cudaMemcpy(klo, c->klo, sizeof(uint32_t) * c->n, cudaMemcpyDeviceToHost));
    HC_CUDA(cudaMemcpy(midx, c->xidx, sizeof(uint32_t) * M, cudaMemcpyDeviceToHost));
    HC_CUDA(cudaMemcpy(nd, c->nodeD, sizeof(double) * 4 * nn, cudaMemcpyDeviceToHost));
    HC_CUDA(cudaMemcpy(nq, c->nodeQ, sizeof(float4) * 2 * nn, cudaMemcpyDeviceToHost));
    auto unspread = [](unsigned long long hi, uint32_t lo, int axis) {
        // axis 0 = x (bit 2 of each digit), 1 = y, 2 = z
        unsigned v = 0;
        int sh = 2 - axis;
        for (int b = 0; b < 21; b++) v |= (unsigned)((hi >> (3 * b + sh)) & 1ull) << (b + 9);
        for (int b = 0; b < 9; b++) v |= ((lo >> (3 * b + sh)) & 1u) << b;
        return v;
    };
    int ci = 0;
    for (int k = 0; k < nn; k++) {
        const int D = C[k].y >> 8, a = pa[k];
        if (a < 0) {
            if (bparent) bparent[midx[-1 - a]] = D - 1;
            continue;
        }
        if (level) level[ci] = D;
        if (corner) {
            for (int ax = 0; ax < 3; ax++) {
                unsigned v = unspread(mhi[a], klo[midx[a]], ax);
                unsigned mask = D >= 30 ? 0xffffffffu : ~((1u << (30 - D)) - 1u);
                corner[3 * ci + ax] = (int32_t)(v & mask);
            }
        }
        if (count) count[ci] = pb[k];
        if (mass) mass[ci] = nd[4 * (int64_t)k + 3];
        if (cm)
            for (int ax = 0; ax < 3; ax++) cm[3 * ci + ax] = nd[4 * (int64_t)k + ax];
        if (quad)
            for (int q = 0; q < 6; q++) quad[6 * ci + q] = nq[(int64_t)8 * k + q];
        ci++;
    }
    return ci;
}
