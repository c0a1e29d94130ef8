// hc_sort.cu -- device radix sort for the octree keys.
//
// The reference inserts bodies one by one (loadtree, load.c:101-128); the
// GB300 build instead sorts all bodies by their 90-bit integer-coordinate key
// (top 63 bits radix sorted, the low 27 bits resolved inside runs of equal
// high keys), so that every octree cell is a contiguous run of sorted bodies.
// The sort moves the high key and the body index, 12 bytes a body; the low key
// stays in body order and is looked up through the index where high keys tie.
//
// One-sweep LSD radix sort: the key kernel counts the digits of all passes, then
// one kernel per 8-bit pass.  A pass's tiles (1024 to 4096 keys) count their digits,
// find the counts of all earlier tiles by decoupled look-back (hc_scan.cuh) and
// scatter through shared memory, stable, so that each digit's run is written
// contiguously.  Bound by latency up to 10^6 bodies (about 17 us a pass), above
// it by the scatter's memory traffic.
// Up to SORT_SMALL bodies one block sorts in shared memory: one launch instead
// of eleven (a pass costs a launch and two global round trips, 10 us at 4096
// bodies; here about 1 us).
#include <algorithm>
#include "hc_scan.cuh"

namespace {

constexpr int SORT_THREADS = 256;
constexpr int SORT_WARPS = SORT_THREADS / 32;
constexpr int NPASS = 8;

// Keys a thread of a pass takes: few where tiles of 4096 leave most SMs idle and
// a pass is one tile's latency, many where the tiles' counts (1 KB a tile and
// pass) and the length of the digits' runs matter.  Build of 2^14, 2^16, 2^18,
// 2^19, 2^20 bodies with 4 keys: 160, 175, 259, 365, 536 us, with 8: 165, 176,
// 245, 343, 503, with 16: 179, 189, 253, 333, 485.
constexpr int64_t SORT_LINE4 = 1 << 15, SORT_LINE8 = 1 << 18;
int sort_items(int64_t n) { return n <= SORT_LINE4 ? 4 : n <= SORT_LINE8 ? 8 : 16; }

// dynamic shared memory of k_sort_pass: the tile's keys and values in digit
// order (staged so that each digit's run is written out contiguously)
constexpr size_t sort_pass_smem(int items)
{
    return (size_t)items * SORT_THREADS * (sizeof(unsigned long long) + sizeof(uint32_t));
}

// Rank of each of a warp's keys among the warp's earlier keys of the same digit,
// rounds of 32 keys in index order, with warp-private digit counters (no block
// barrier per round).  One round: digit dr (256 or more: no key).
template <typename C>
__device__ __forceinline__ uint32_t rank_round(C *cnt, int dr, int lane)
{
    // lanes of the same digit by one ballot per bit: __match_any_sync took longer
    // (one-block sort of 4096 bodies 43 -> 34 us, eight passes of 50,021 89 -> 77)
    unsigned peers = __ballot_sync(0xffffffffu, dr < 256);
#pragma unroll
    for (int b = 0; b < 8; b++) {
        const unsigned bit = __ballot_sync(0xffffffffu, (dr >> b) & 1);
        peers &= (dr >> b) & 1 ? bit : ~bit;
    }
    const int leader = peers ? __ffs(peers) - 1 : lane;
    uint32_t before = 0;
    if (dr < 256 && lane == leader) {
        before = cnt[dr];
        cnt[dr] = (C)(before + __popc(peers));
    }
    before = __shfl_sync(0xffffffffu, before, leader);
    __syncwarp();
    return before + __popc(peers & ((1u << lane) - 1u));
}

// counts: digit counts of this pass over all keys; look: look-back words.
// first: the values are the indices themselves (not read).
template <int ITEMS>
__global__ void __launch_bounds__(SORT_THREADS) k_sort_pass(
    const unsigned long long *__restrict__ ihi, const uint32_t *__restrict__ ival,
    unsigned long long *__restrict__ ohi, uint32_t *__restrict__ oval, int64_t n, int shift, bool first,
    const uint32_t *counts, uint32_t *look, uint32_t *tile_ctr, int *err)
{
    constexpr int TILE = ITEMS * SORT_THREADS, WARP_KEYS = ITEMS * 32;   // a warp ranks contiguous keys
    extern __shared__ unsigned long long stage_k[];                    // [TILE]
    uint32_t *stage_v = reinterpret_cast<uint32_t *>(stage_k + TILE);  // [TILE]
    __shared__ uint32_t s_tile;
    __shared__ uint32_t gbase[256];        // global position of the tile's first key of each digit
    __shared__ uint32_t lbase[256];        // start of each digit's run in the stage
    __shared__ uint32_t wcnt[SORT_WARPS][256];   // per warp: digit counts, then the warp's offsets in a run
    __shared__ uint32_t scan_sh[32];
    const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
    if (tid == 0) s_tile = atomicAdd(tile_ctr, 1u);
    const uint32_t total = counts[tid];
#pragma unroll
    for (int w = 0; w < SORT_WARPS; w++) wcnt[w][tid] = 0;
    __syncthreads();
    const int64_t tile = s_tile, base = tile * TILE;
    const int tn = (int)(n - base < TILE ? n - base : TILE);
    // each warp loads and ranks its contiguous slice [wid * WARP_KEYS, +WARP_KEYS)
    unsigned long long k[ITEMS];
    uint32_t va[ITEMS];
#pragma unroll
    for (int r = 0; r < ITEMS; r++) {
        const int e = wid * WARP_KEYS + r * 32 + lane;
        k[r] = e < tn ? ihi[base + e] : 0ull;
        va[r] = first ? (uint32_t)(base + e) : (e < tn ? ival[base + e] : 0u);
    }
    uint32_t rk[ITEMS / 2];           // ranks in the warp, two 16-bit values per word
#pragma unroll
    for (int r = 0; r < ITEMS; r++) {
        const int e = wid * WARP_KEYS + r * 32 + lane;
        const uint32_t rank = rank_round(wcnt[wid], e < tn ? (int)((k[r] >> shift) & 255u) : 256 + lane, lane);
        if (r & 1) rk[r >> 1] |= rank << 16;
        else rk[r >> 1] = rank;
    }
    __syncthreads();
    // thread = digit: the tile's count, each warp's offset inside the digit's run
    uint32_t cnt = 0;
#pragma unroll
    for (int w = 0; w < SORT_WARPS; w++) {
        const uint32_t c = wcnt[w][tid];
        wcnt[w][tid] = cnt;
        cnt += c;
    }
    const uint32_t prefix = digit_prefix(look, tile, 256, tid, cnt, err);
    gbase[tid] = block_exclusive_scan<uint32_t>(total, scan_sh, nullptr) + prefix;
    lbase[tid] = block_exclusive_scan<uint32_t>(cnt, scan_sh, nullptr);
    __syncthreads();
    // stage in digit order: run start + earlier warps' keys of the digit + rank in the warp
#pragma unroll
    for (int r = 0; r < ITEMS; r++) {
        const int e = wid * WARP_KEYS + r * 32 + lane;
        if (e >= tn) continue;
        const int dr = (int)((k[r] >> shift) & 255u);
        const uint32_t off = lbase[dr] + wcnt[wid][dr] + ((rk[r >> 1] >> ((r & 1) * 16)) & 0xffffu);
        stage_k[off] = k[r];
        stage_v[off] = va[r];
    }
    __syncthreads();
    // write out in stage order: consecutive keys of one digit go to consecutive places
    for (int e = tid; e < tn; e += SORT_THREADS) {
        const unsigned long long key = stage_k[e];
        const int dd = (int)((key >> shift) & 255u);
        const uint32_t pos = gbase[dd] + (uint32_t)e - lbase[dd];
        ohi[pos] = key;
        oval[pos] = stage_v[e];
    }
}

// Stable insertion sort of the run [i, e] of equal high keys by the low key, which
// is a gather through the index: not read again for keys in order (many massless
// bodies outside the box share one key), found by bisection for the others.
__device__ __forceinline__ void order_run(const uint32_t *lo, uint32_t *val, int64_t i, int64_t e)
{
    uint32_t top = lo[val[i]];                       // largest so far, at a - 1
    for (int64_t a = i + 1; a <= e; a++) {
        const uint32_t kv = val[a], kl = lo[kv];
        if (kl >= top) {
            top = kl;
            continue;
        }
        int64_t p = i, q = a - 1;                    // the first larger one
        while (p < q) {
            const int64_t mid = (p + q) >> 1;
            if (lo[val[mid]] > kl) q = mid;
            else p = mid + 1;
        }
        for (int64_t b = a; b > q; b--) val[b] = val[b - 1];
        val[q] = kv;
    }
}

// Runs of equal 63-bit high keys (two bodies closer than 2^-21 of the root
// box) are ordered by the low 27 key bits; runs are a few entries long.
__global__ void k_tie_fix(const unsigned long long *hi, const uint32_t *lo, uint32_t *val, int64_t n)
{
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
        if (i + 1 >= n || hi[i + 1] != hi[i]) continue;
        if (i > 0 && hi[i - 1] == hi[i]) continue;
        int64_t e = i + 1;
        while (e + 1 < n && hi[e + 1] == hi[i]) e++;
        order_run(lo, val, i, e);
    }
}

// All passes of a small sort in one block; with lo the runs of equal high keys
// are ordered too.  Thread t of quarter q = t / 256 sums digit t % 256 over
// eight warps; keys stay in registers between passes and change places through
// shared memory.
constexpr int SMALL_THREADS = 1024, SMALL_WARPS = 32;
constexpr int SORT_SMALL = 8 * SMALL_THREADS;

template <int ITEMS>
constexpr size_t small_smem()
{
    return (size_t)ITEMS * SMALL_THREADS * (sizeof(unsigned long long) + sizeof(uint32_t)) +
           SMALL_WARPS * 256 * sizeof(uint16_t) + (4 * 256 + 256 + 32) * sizeof(uint32_t);
}

template <int ITEMS>
__global__ void __launch_bounds__(SMALL_THREADS) k_sort_small(const unsigned long long *ihi, int n,
                                                              unsigned long long *ohi, uint32_t *oval,
                                                              const uint32_t *lo)
{
    extern __shared__ unsigned long long sk[];                      // [ITEMS * SMALL_THREADS]
    uint32_t *const sv = reinterpret_cast<uint32_t *>(sk + ITEMS * SMALL_THREADS);
    uint16_t(*const wcnt)[256] = reinterpret_cast<uint16_t(*)[256]>(sv + ITEMS * SMALL_THREADS);
    uint32_t(*const quarter)[256] = reinterpret_cast<uint32_t(*)[256]>(wcnt + SMALL_WARPS);
    uint32_t *const lbase = &quarter[4][0], *const scan_sh = lbase + 256;
    const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5, digit = tid & 255, q = tid >> 8;
    unsigned long long k[ITEMS];
    uint32_t v[ITEMS];
#pragma unroll
    for (int r = 0; r < ITEMS; r++) {
        const int e = (wid * ITEMS + r) * 32 + lane;
        k[r] = e < n ? ihi[e] : 0ull;
        v[r] = (uint32_t)e;
    }
    for (int pass = 0; pass < NPASS; pass++) {
        const int shift = 8 * pass;
        for (int i = tid; i < SMALL_WARPS * 256 / 2; i += SMALL_THREADS) reinterpret_cast<uint32_t *>(wcnt)[i] = 0u;
        __syncthreads();
        uint32_t rk[ITEMS];
#pragma unroll
        for (int r = 0; r < ITEMS; r++) {
            const bool valid = (wid * ITEMS + r) * 32 + lane < n;
            rk[r] = rank_round(wcnt[wid], valid ? (int)((k[r] >> shift) & 255u) : 256 + lane, lane);
        }
        __syncthreads();
        uint32_t c[8], sum = 0;
#pragma unroll
        for (int w = 0; w < 8; w++) {
            c[w] = sum;
            sum += wcnt[q * 8 + w][digit];
        }
        quarter[q][digit] = sum;
        __syncthreads();
        uint32_t before = 0, total = 0;
#pragma unroll
        for (int j = 0; j < 4; j++) {
            if (j < q) before += quarter[j][digit];
            total += quarter[j][digit];
        }
        // exclusive scan of the 256 digit counts (the first eight warps')
        const uint32_t incl = warp_inclusive_scan(total);
        if (q == 0 && lane == 31) scan_sh[wid] = incl;
        __syncthreads();
        if (q == 0) {
            uint32_t b = incl - total;
            for (int w = 0; w < wid; w++) b += scan_sh[w];
            lbase[digit] = b;
        }
        __syncthreads();
        before += lbase[digit];
#pragma unroll
        for (int w = 0; w < 8; w++) wcnt[q * 8 + w][digit] = (uint16_t)(before + c[w]);
        __syncthreads();
#pragma unroll
        for (int r = 0; r < ITEMS; r++) {
            if ((wid * ITEMS + r) * 32 + lane >= n) continue;
            const uint32_t pos = wcnt[wid][(k[r] >> shift) & 255u] + rk[r];
            sk[pos] = k[r];
            sv[pos] = v[r];
        }
        __syncthreads();
#pragma unroll
        for (int r = 0; r < ITEMS; r++) {
            const int e = (wid * ITEMS + r) * 32 + lane;
            if (e < n) {
                k[r] = sk[e];
                v[r] = sv[e];
            }
        }
    }
    if (lo) {
        __syncthreads();
        for (int i = tid; i < n; i += SMALL_THREADS) {
            if (i + 1 >= n || sk[i + 1] != sk[i] || (i > 0 && sk[i - 1] == sk[i])) continue;
            int e = i + 1;
            while (e + 1 < n && sk[e + 1] == sk[i]) e++;
            order_run(lo, sv, i, e);
        }
        __syncthreads();
    }
    for (int i = tid; i < n; i += SMALL_THREADS) {
        ohi[i] = sk[i];
        oval[i] = sv[i];
    }
}

template <int ITEMS>
int small_setup(hc_ctx *c)
{
    HC_CUDA(cudaFuncSetAttribute(k_sort_small<ITEMS>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 (int)small_smem<ITEMS>()));
    return HC_OK;
}

template <int ITEMS>
void small_launch(hc_ctx *c, const unsigned long long *ihi, int64_t n, unsigned long long *ohi, uint32_t *oval,
                  const uint32_t *lo)
{
    k_sort_small<ITEMS><<<1, SMALL_THREADS, small_smem<ITEMS>(), c->stream>>>(ihi, (int)n, ohi, oval, lo);
}

}  // namespace

// once per context, before any capture
int hc_sort_setup(hc_ctx *c)
{
    HC_CUDA(cudaFuncSetAttribute(k_sort_pass<16>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sort_pass_smem(16)));
    int r = small_setup<1>(c);
    if (r == HC_OK) r = small_setup<2>(c);
    if (r == HC_OK) r = small_setup<4>(c);
    if (r == HC_OK) r = small_setup<8>(c);
    return r;
}

// scratch: [0, 2048) digit counts per pass, [2048, 2056) tile counters,
// [4096, ...) look-back words, ntiles x 256 per pass
int64_t hc_sort_scratch_words(int64_t n)
{
    const int64_t tile = sort_items(n) * SORT_THREADS, ntiles = (n + tile - 1) / tile;
    return 4096 + (int64_t)NPASS * 256 * (ntiles < 1 ? 1 : ntiles);
}

// Not the words of n itself: just below a line the tiles are smaller and more
// (200,000 keys take 98 tiles, 300,000 take 74).
int64_t hc_sort_scratch_capacity(int64_t n)
{
    return std::max({hc_sort_scratch_words(n), hc_sort_scratch_words(std::min(n, SORT_LINE4)),
                     hc_sort_scratch_words(std::min(n, SORT_LINE8))});
}

// the small sort counts its digits itself and needs no scratch
bool hc_sort_counts_digits(int64_t n) { return n <= SORT_SMALL; }

// Sort n high keys khi[0] (63 bits) with their indices.  scratch: zeroed, with
// the digit counts of all passes in its first 2048 words (hc_keys_for_points).
// lo (body order): runs of equal high keys are ordered by it.  Returns the
// buffer that holds the result.
int hc_radix_sort_keys(hc_ctx *c, uint32_t *scratch, unsigned long long *khi[2], uint32_t *kval[2], int64_t n,
                       const uint32_t *lo)
{
    if (n <= 0) return 0;
    if (hc_sort_counts_digits(n)) {
        if (n <= SMALL_THREADS) small_launch<1>(c, khi[0], n, khi[1], kval[1], lo);
        else if (n <= 2 * SMALL_THREADS) small_launch<2>(c, khi[0], n, khi[1], kval[1], lo);
        else if (n <= 4 * SMALL_THREADS) small_launch<4>(c, khi[0], n, khi[1], kval[1], lo);
        else small_launch<8>(c, khi[0], n, khi[1], kval[1], lo);
        c->launches++;
        return 1;
    }
    const int items = sort_items(n);
    const int64_t tile = items * SORT_THREADS, ntiles = (n + tile - 1) / tile;
    auto *pass = items == 4 ? k_sort_pass<4> : items == 8 ? k_sort_pass<8> : k_sort_pass<16>;
    uint32_t *counts = scratch, *ctr = scratch + 2048, *look = scratch + 4096;
    int sel = 0;
    for (int p = 0; p < NPASS; p++) {
        pass<<<(unsigned)ntiles, SORT_THREADS, sort_pass_smem(items), c->stream>>>(
            khi[sel], kval[sel], khi[sel ^ 1], kval[sel ^ 1], n, 8 * p, p == 0, counts + 256 * p,
            look + (int64_t)p * 256 * ntiles, ctr + p, &c->st->error);
        c->launches++;
        sel ^= 1;
    }
    if (lo) {
        k_tie_fix<<<hc_grid(n, 256), 256, 0, c->stream>>>(khi[sel], lo, kval[sel], n);
        c->launches++;
    }
    return sel;
}
