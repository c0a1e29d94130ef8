// hc_ensemble.cu -- ensembles of independent systems of uneven size, stepped
// together (no counterpart in hackcode1, which evolves one system per run).
//
// Layout (internal order: tree systems first, then direct-sum systems; the
// host API converts from and to the caller's order):
//   FP64 SoA over all bodies: mass, x/y/z (each system in its own
//   coordinates), v, a, phi.  The tree systems' mass / v / a / phi arrays
//   are the first n_tree entries of these and are shared with one forest
//   context (hc_ctx) whose positions are forest coordinates.
//
// One step, all of it captured in one CUDA graph:
//   1. per tree system, hackcode1's expandbox replay (load.c:68-95) on its
//      own persistent root box, which starts at (-2,-2,-2), 4 (code.c:119-120)
//      and only grows -- one block per system, bodies in order;
//   2. slot layout: every system box is placed in its own slot of one forest
//      box (slots of the largest system's size on a G^3 grid, G a power of
//      two), so that the system box is exactly a forest cell; positions are
//      translated into the slot;
//   3. the single-system build (keys, sort, cells, upward pass, groups) on
//      the forest -- cells never straddle systems, and every walk group lies
//      in one system;
//   4. the walk of each group starts at its system's root cell (found among
//      the nodes), so no system sees another;
//   5. systems of at most direct_max bodies: FP32 direct sum, one block per
//      64 bodies, positions split hi + lo relative to the system's first body;
//   6. closing half-kick inside 3-5 (code.c:175-179), per-system energies,
//      then kick-drift of every body (code.c:182-188).
//
// Differences from running hackcode1 once per system: a system's keys keep
// 30 - depth(system root in the forest) bits per axis (bodies closer than
// that are reported as coincident), and the one-body cells that hackcode1
// grafts when its second body expands the box twice or more are not formed.
#include <algorithm>
#include <climits>
#include <cmath>
#include <cstring>
#include <vector>
#include "hc_internal.cuh"

#define HC_TRY(x)                   \
    do {                            \
        int r_ = (x);               \
        if (r_ != HC_OK) return r_; \
    } while (0)

namespace {

constexpr int DTHREADS = 256;       // energy kernel; the direct sum's block size is tuned (128..512)

struct SysBox {
    double rmin[3];
    double rsize;
};

__device__ __forceinline__ bool inbox_d(double x, double y, double z, const double *rmin, double rsize)
{
    // intcoord (load.c:135-156): 0 <= (x - rmin) / rsize < 1 on every axis
    const double p[3] = {x, y, z};
#pragma unroll
    for (int k = 0; k < 3; k++) {
        const double s = __ddiv_rn(__dsub_rn(p[k], rmin[k]), rsize);
        if (!(0.0 <= s && s < 1.0)) return false;
    }
    return true;
}

// 1. expandbox replay, one block per tree system.  The box only grows, so a
// body found inside stays inside: each round finds the first body of the
// remaining range outside the current box and expands for it.  A body clearly
// inside by an FP32 estimate skips the exact test (as in k_box_outside): with
// the exact test's three FP64 divisions for every body, one warp per system
// took 1.26 ms for systems of up to 16,384 bodies.
__global__ void __launch_bounds__(256) k_ens_replay(const int64_t *off, const double *mass, const double *px,
                                                    const double *py, const double *pz, SysBox *box, hc_status *st)
{
    constexpr int CHUNK = 256 * 8;              // bodies between two looks for an early end
    __shared__ double rmin[3], rsize;
    __shared__ int first, bad;
    const int s = blockIdx.x, tid = threadIdx.x;
    const int64_t b0 = off[s];
    const int n = (int)(off[s + 1] - b0);
    if (tid == 0) {
        for (int d = 0; d < 3; d++) rmin[d] = box[s].rmin[d];
        rsize = box[s].rsize;
        first = INT_MAX;
        bad = 0;
    }
    __syncthreads();
    int pos = 0;
    while (true) {
        const float lo[3] = {hc_d2f_rn(rmin[0]), hc_d2f_rn(rmin[1]), hc_d2f_rn(rmin[2])}, sz = hc_d2f_rn(rsize);
        for (int base = pos; base < n; base += CHUNK) {
            int mine = INT_MAX;
#pragma unroll
            for (int r = 0; r < CHUNK / 256; r++) {
                const int i = base + r * 256 + tid;
                if (i >= n) continue;
                const double x[3] = {px[b0 + i], py[b0 + i], pz[b0 + i]};
                bool clear = true;
#pragma unroll
                for (int d = 0; d < 3; d++) {
                    float f;
                    if (!hc_approx_f32(x[d], &f)) {
                        clear = false;
                        continue;
                    }
                    const float u = f - lo[d], margin = 0x1p-16f * sz + 0x1p-18f * fabsf(f);
                    clear = clear && u >= margin && u <= sz - margin;
                }
                if (!clear && hc_nonzero(mass[b0 + i]) && !inbox_d(x[0], x[1], x[2], rmin, rsize)) mine = min(mine, i);
            }
            if (__syncthreads_or(mine != INT_MAX)) {
                if (mine != INT_MAX) atomicMin(&first, mine);
                __syncthreads();
                break;
            }
        }
        const int f = first;
        __syncthreads();
        if (f == INT_MAX) break;
        if (tid == 0) {
            const double x[3] = {px[b0 + f], py[b0 + f], pz[b0 + f]};
            int k = 0;
            while (!inbox_d(x[0], x[1], x[2], rmin, rsize)) {         // load.c:74-93
                if (++k > 1100) {                                      // non-finite position
                    atomicCAS(&st->error, 0, HC_ERR_ARG);
                    st->info = (int)(b0 + f);
                    bad = 1;
                    break;
                }
                double rmid[3];
                for (int d = 0; d < 3; d++) rmid[d] = __dadd_rn(rmin[d], __dmul_rn(0.5, rsize));
                for (int d = 0; d < 3; d++)
                    if (x[d] < rmid[d]) rmin[d] = __dsub_rn(rmin[d], rsize);
                rsize = __dmul_rn(2.0, rsize);
            }
            first = INT_MAX;
        }
        __syncthreads();
        if (bad) return;
        pos = f + 1;
    }
    if (tid == 0) box[s] = SysBox{{rmin[0], rmin[1], rmin[2]}, rsize};
}

// 2a. slot layout (one block): slot size = largest system box, G^3 slots;
// forest box (0,0,0), G * slot; depth of each system root in the forest.
__global__ void k_ens_layout(int nsys_tree, int gbits, const SysBox *box, double *origin, int32_t *depth,
                             int32_t *root, hc_box *fbox, hc_status *st)
{
    __shared__ double smax;
    if (threadIdx.x == 0) smax = 0.0;
    __syncthreads();
    double lmax = 0.0;
    for (int s = threadIdx.x; s < nsys_tree; s += blockDim.x) lmax = fmax(lmax, box[s].rsize);
    // block max via shared atomics on the bit pattern (positive doubles order like integers)
    atomicMax(reinterpret_cast<unsigned long long *>(&smax), (unsigned long long)__double_as_longlong(lmax));
    __syncthreads();
    const double S = smax;
    const int G = 1 << gbits;
    for (int s = threadIdx.x; s < nsys_tree; s += blockDim.x) {
        const int gx = s & (G - 1), gy = (s >> gbits) & (G - 1), gz = s >> (2 * gbits);
        origin[3 * s + 0] = __dmul_rn((double)gx, S);
        origin[3 * s + 1] = __dmul_rn((double)gy, S);
        origin[3 * s + 2] = __dmul_rn((double)gz, S);
        // rsize values are 4 * 2^k: S / rsize is an exact power of two
        int e = 0;
        double r = box[s].rsize;
        while (r < S && e < 64) {
            r = __dmul_rn(2.0, r);
            e++;
        }
        depth[s] = gbits + e;
        root[s] = -1;
        if (gbits + e > 29) {                 // no key bits left inside the system
            atomicCAS(&st->error, 0, HC_ERR_ARG);
            st->info = s;
        }
    }
    if (threadIdx.x == 0) {
        fbox->rmin[0] = fbox->rmin[1] = fbox->rmin[2] = 0.0;
        fbox->rsize = __dmul_rn((double)G, S);
        fbox->first_massive = -1;
        fbox->chain_lmax = fbox->chain_lmin = -1;
    }
}

// 2b. forest coordinates: x_f = (x - rmin_s) + origin_s; a massive body stays
// inside its system's cell (massless ones are only targets and may lie outside)
__global__ void k_ens_translate(int64_t n_tree, const int32_t *body_sys, const SysBox *box, const double *origin,
                                const double *mass, const double *px, const double *py, const double *pz,
                                double *fx, double *fy, double *fz)
{
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n_tree;
         i += (int64_t)gridDim.x * blockDim.x) {
        const int s = body_sys[i];
        const SysBox b = box[s];
        const bool massive = mass[i] != 0.0;
        const double p[3] = {px[i], py[i], pz[i]};
        double q[3];
#pragma unroll
        for (int k = 0; k < 3; k++) {
            const double o = origin[3 * s + k];
            double v = __dadd_rn(__dsub_rn(p[k], b.rmin[k]), o);
            const double hi = __dadd_rn(o, b.rsize);
            if (massive && v >= hi) v = nextafter(hi, o);      // rounding must not leave the cell
            if (massive && v < o) v = o;
            q[k] = v;
        }
        fx[i] = q[0];
        fy[i] = q[1];
        fz[i] = q[2];
    }
}

// 4. root cell of each tree system: the cell at the system's depth that
// holds its first body in key order
__global__ void k_ens_roots(const hc_box *fbox, const int2 *nodeC, const uint32_t *bfs_a, const uint32_t *midx,
                            const int32_t *body_sys, const int32_t *depth, int32_t *root)
{
    const int nn = fbox->nnode;
    for (int k = blockIdx.x * blockDim.x + threadIdx.x; k < nn; k += gridDim.x * blockDim.x) {
        const int2 C = nodeC[k];
        if (C.x < 0) continue;                        // a body
        const int s = body_sys[midx[bfs_a[k]]];
        if (C.y >> 8 == depth[s]) root[s] = k;
    }
}

__device__ __forceinline__ void kahan(float &sum, float &comp, float x)
{
    const float y = __fsub_rn(x, comp);
    const float t = __fadd_rn(sum, y);
    comp = __fsub_rn(__fsub_rn(t, sum), y);
    sum = t;
}

// 5. direct sum of the small systems (FP32, hi + lo positions relative to the
// system's first body; Kahan over 64-body partials).  A block takes 64 bodies
// of one system (work: system, first body) and the whole system as sources,
// staged in pairs: both bodies' values of one quantity adjacent, the operands
// of one packed FP32x2 instruction.  Its T / 64 slices of warps take a slice of
// the sources each, added at the end in slice order.  (One block per whole
// system with scalar arithmetic: 253 us for 53 systems of up to 1024 bodies.)
constexpr int DROWS = 64;
static size_t ens_direct_smem(int n, int threads)
{
    return sizeof(float4) * (4 * (size_t)((n + 1) / 2) + 2 * (size_t)threads);
}
__global__ void __launch_bounds__(512) k_ens_direct(const int2 *work, const int64_t *off, const double *mass,
                                                    const double *px, const double *py, const double *pz,
                                                    float eps2, double kick_dthf, int64_t nstep, double *vx,
                                                    double *vy, double *vz, double *ax, double *ay, double *az,
                                                    double *phi)
{
    extern __shared__ float4 sm[];
    const int s = work[blockIdx.x].x, row = work[blockIdx.x].y + threadIdx.x % DROWS;
    const int slice = threadIdx.x / DROWS, nslice = blockDim.x / DROWS;
    const int64_t b0 = off[s];
    const int n = (int)(off[s + 1] - b0), np = (n + 1) / 2;
    float4(*const pair)[4] = reinterpret_cast<float4(*)[4]>(sm);   // (hx hy) (hz m) (lx ly) (lz -), for two bodies
    float4 *const part = sm + 4 * np;
    const double cx = px[b0], cy = py[b0], cz = pz[b0];
    for (int j = threadIdx.x; j < 2 * np; j += blockDim.x) {
        float *f = reinterpret_cast<float *>(pair[j >> 1]) + (j & 1);
        if (j < n) {
            hc_split_hilo(px[b0 + j] - cx, &f[0], &f[8]);          // on the doubles' bits (no FP64-pipe conversions)
            hc_split_hilo(py[b0 + j] - cy, &f[2], &f[10]);
            hc_split_hilo(pz[b0 + j] - cz, &f[4], &f[12]);
            f[6] = hc_d2f_rn(mass[b0 + j]);
        } else {                                                    // pad: massless, far away
            f[0] = f[2] = f[4] = 1.0e4f;
            f[6] = f[8] = f[10] = f[12] = 0.f;
        }
    }
    __syncthreads();
    float4 S = make_float4(0.f, 0.f, 0.f, 0.f), C = S;              // Kahan sums x, y, z, -phi
    if (row < n) {
        const float *f = reinterpret_cast<const float *>(pair[row >> 1]) + (row & 1);
        const float2 bx = splat2(-f[0]), by = splat2(-f[2]), bz = splat2(-f[4]), blx = splat2(-f[8]), bly = splat2(-f[10]),
                     blz = splat2(-f[12]), e2 = splat2(eps2);
        const int p1 = (int)((int64_t)np * (slice + 1) / nslice);
        for (int p0 = (int)((int64_t)np * slice / nslice); p0 < p1; p0 += 32) {
            float2 qx = splat2(0.f), qy = qx, qz = qx, qp = qx;
            const int pe = p0 + 32 < p1 ? p0 + 32 : p1;
#pragma unroll 4
            for (int p = p0; p < pe; p++) {
                const float4 H0 = pair[p][0], H1 = pair[p][1], L0 = pair[p][2], L1 = pair[p][3];
                const float2 dx = __fadd2_rn(__fadd2_rn(lo2(H0), bx), __fadd2_rn(lo2(L0), blx));
                const float2 dy = __fadd2_rn(__fadd2_rn(hi2(H0), by), __fadd2_rn(hi2(L0), bly));
                const float2 dz = __fadd2_rn(__fadd2_rn(lo2(H1), bz), __fadd2_rn(lo2(L1), blz));
                const float2 r2 = __ffma2_rn(dx, dx, __ffma2_rn(dy, dy, __ffma2_rn(dz, dz, e2)));
                const float2 w = make_float2(2 * p != row ? rsqrtf(r2.x) : 0.f, 2 * p + 1 != row ? rsqrtf(r2.y) : 0.f);
                const float2 mr = __fmul2_rn(hi2(H1), w);
                const float2 mr3 = __fmul2_rn(mr, __fmul2_rn(w, w));
                qp = __fadd2_rn(qp, mr);
                qx = __ffma2_rn(mr3, dx, qx);
                qy = __ffma2_rn(mr3, dy, qy);
                qz = __ffma2_rn(mr3, dz, qz);
            }
            kahan(S.x, C.x, qx.x + qx.y);
            kahan(S.y, C.y, qy.x + qy.y);
            kahan(S.z, C.z, qz.x + qz.y);
            kahan(S.w, C.w, qp.x + qp.y);
        }
    }
    part[2 * threadIdx.x] = S;
    part[2 * threadIdx.x + 1] = C;
    __syncthreads();
    if (slice > 0 || row >= n) return;
    double r[4] = {0.0, 0.0, 0.0, 0.0};
    for (int q = 0; q < nslice; q++) {
        const float4 a = part[2 * (threadIdx.x + q * DROWS)], c = part[2 * (threadIdx.x + q * DROWS) + 1];
        r[0] += (double)a.x - (double)c.x;
        r[1] += (double)a.y - (double)c.y;
        r[2] += (double)a.z - (double)c.z;
        r[3] += (double)a.w - (double)c.w;
    }
    const int64_t o = b0 + row;
    if (kick_dthf != 0.0 && nstep > 0) {          // closing half kick (code.c:175-179)
        vx[o] = __dadd_rn(vx[o], __dmul_rn(__dsub_rn(r[0], ax[o]), kick_dthf));
        vy[o] = __dadd_rn(vy[o], __dmul_rn(__dsub_rn(r[1], ay[o]), kick_dthf));
        vz[o] = __dadd_rn(vz[o], __dmul_rn(__dsub_rn(r[2], az[o]), kick_dthf));
    }
    ax[o] = r[0];
    ay[o] = r[1];
    az[o] = r[2];
    phi[o] = -r[3];
}

// 6a. kinetic and potential energy of each system (code_io.c:160-197): a block
// per chunk of ECHUNK bodies (work: system, first body), then each system's
// chunks in order.  (One block per system held one SM's FP64 pipe for 54 us at
// 16,384 bodies.)
constexpr int ECHUNK = 1024;
__global__ void __launch_bounds__(DTHREADS) k_ens_energy(const int2 *work, const int64_t *off, const double *mass,
                                                         const double *vx, const double *vy, const double *vz,
                                                         const double *phi, double2 *part)
{
    const int64_t i0 = off[work[blockIdx.x].x] + work[blockIdx.x].y, end = off[work[blockIdx.x].x + 1];
    const int64_t i1 = i0 + ECHUNK < end ? i0 + ECHUNK : end;
    double ke = 0.0, pe = 0.0;
    for (int64_t i = i0 + threadIdx.x; i < i1; i += DTHREADS) {
        const double hm = __dmul_rn(0.5, mass[i]);
        double v2 = __dmul_rn(vx[i], vx[i]);
        v2 = __dadd_rn(v2, __dmul_rn(vy[i], vy[i]));
        v2 = __dadd_rn(v2, __dmul_rn(vz[i], vz[i]));
        ke += __dmul_rn(hm, v2);
        pe += __dmul_rn(hm, phi[i]);
    }
    __shared__ double rk[DTHREADS], rp[DTHREADS];
    rk[threadIdx.x] = ke;
    rp[threadIdx.x] = pe;
    __syncthreads();
    for (int o = DTHREADS / 2; o; o >>= 1) {
        if (threadIdx.x < o) {
            rk[threadIdx.x] += rk[threadIdx.x + o];
            rp[threadIdx.x] += rp[threadIdx.x + o];
        }
        __syncthreads();
    }
    if (threadIdx.x == 0) part[blockIdx.x] = make_double2(rk[0], rp[0]);
}

__global__ void k_ens_energy_sum(int nsys, const int32_t *chunk0, const int32_t *user_of, const double2 *part, double *out)
{
    const int s = blockIdx.x * blockDim.x + threadIdx.x;
    if (s >= nsys) return;
    double ke = 0.0, pe = 0.0;
    for (int c = chunk0[s]; c < chunk0[s + 1]; c++) {
        ke += part[c].x;
        pe += part[c].y;
    }
    const int u = user_of[s];
    out[3 * u + 0] = ke;
    out[3 * u + 1] = pe;
    out[3 * u + 2] = ke + pe;
}

// 6b. v += a dt/2; x += v dt; v += a dt/2  (code.c:182-188)
__global__ void k_ens_kick_drift(int64_t n, double dt, double *px, double *py, double *pz, double *vx, double *vy,
                                 double *vz, const double *ax, const double *ay, const double *az)
{
    const double dthf = 0.5 * dt;
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
        double *p[3] = {px, py, pz}, *v[3] = {vx, vy, vz};
        const double *a[3] = {ax, ay, az};
#pragma unroll
        for (int k = 0; k < 3; k++) {
            const double dvel = __dmul_rn(a[k][i], dthf);
            const double vel1 = __dadd_rn(v[k][i], dvel);
            p[k][i] = __dadd_rn(p[k][i], __dmul_rn(vel1, dt));
            v[k][i] = __dadd_rn(vel1, dvel);
        }
    }
}

__global__ void k_unpack_sys(const double *phase, int64_t n, double *px, double *py, double *pz, double *vx,
                             double *vy, double *vz)
{
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
        const double *q = phase + 6 * i;
        px[i] = q[0];
        py[i] = q[1];
        pz[i] = q[2];
        vx[i] = q[3];
        vy[i] = q[4];
        vz[i] = q[5];
    }
}

// State of all bodies in the caller's order, packed: [n][2][3] positions and
// velocities, [n][3] accelerations, [n] potentials, whichever are asked for.
// user0: a system's first body in the caller's order.
__global__ void k_pack_user(int64_t n, const int32_t *body_sys, const int64_t *off, const int64_t *user0,
                            const double *px, const double *py, const double *pz, const double *vx, const double *vy,
                            const double *vz, const double *ax, const double *ay, const double *az, const double *phi,
                            double *ophase, double *oacc, double *ophi)
{
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
        const int s = body_sys[i];
        const int64_t u = user0[s] + (i - off[s]);
        if (ophase) {
            double *q = ophase + 6 * u;
            q[0] = px[i];
            q[1] = py[i];
            q[2] = pz[i];
            q[3] = vx[i];
            q[4] = vy[i];
            q[5] = vz[i];
        }
        if (oacc) {
            oacc[3 * u] = ax[i];
            oacc[3 * u + 1] = ay[i];
            oacc[3 * u + 2] = az[i];
        }
        if (ophi) ophi[u] = phi[i];
    }
}

__global__ void k_init_boxes(int n, SysBox *box)
{
    for (int s = blockIdx.x * blockDim.x + threadIdx.x; s < n; s += gridDim.x * blockDim.x)
        box[s] = SysBox{{-2.0, -2.0, -2.0}, 4.0};    // code.c:119-120
}

template <typename T>
int ens_alloc(std::string &err, T **p, int64_t count)
{
    const size_t bytes = sizeof(T) * (size_t)std::max<int64_t>(count, 1);
    if (cudaMalloc((void **)p, bytes) != cudaSuccess) {
        err = "cudaMalloc(" + std::to_string(bytes) + ") failed";
        *p = nullptr;
        return HC_ERR_NOMEM;
    }
    return HC_OK;
}

}  // namespace

struct hc_ens {
    std::string err;
    hc_ens_params prm{};
    int nsys = 0, nsys_tree = 0, nsys_direct = 0, gbits = 0;
    int64_t ntot = 0, n_tree = 0;
    std::vector<int64_t> user_count, user_off;   // caller's order
    std::vector<int> order;                      // internal slot -> caller's system
    std::vector<int64_t> int_off;                // internal offsets [nsys + 1]
    hc_ctx *forest = nullptr;                    // tree systems (n_tree bodies), or null
    cudaStream_t stream = nullptr;               // forest's stream or own
    bool own_stream = false;
    cudaEvent_t ev[4] = {};
    // device, internal order
    double *mass = nullptr, *px = nullptr, *py = nullptr, *pz = nullptr, *vx = nullptr, *vy = nullptr,
           *vz = nullptr, *ax = nullptr, *ay = nullptr, *az = nullptr, *phi = nullptr;
    int64_t *d_off = nullptr;
    int32_t *d_body_sys = nullptr, *d_user_of = nullptr;
    int2 *d_dwork = nullptr, *d_ework = nullptr; // (system, first body) of the direct sum's and the energies' blocks
    int32_t *d_echunk0 = nullptr;                // [nsys + 1] first energy chunk of each system
    double2 *d_epart = nullptr;
    int ndwork = 0, nework = 0;
    int32_t *d_root = nullptr, *d_depth = nullptr;
    SysBox *d_box = nullptr;
    int64_t *d_user0 = nullptr;                  // [internal slot] first body in the caller's order
    double *d_origin = nullptr, *d_energy = nullptr, *h_energy = nullptr, *d_stage = nullptr;
    bool uploaded = false;
    int max_direct_n = 0;
    int direct_threads = 256;                    // block size of the direct sum (tuned)
    cudaGraphExec_t graph[2] = {nullptr, nullptr};
    double graph_dt[2] = {0.0, 0.0};
    int64_t launches = 0, graph_launches[2] = {0, 0};
    float tree_ms = 0.f, direct_ms = 0.f;
};

#define EC(call)                                                                 \
    do {                                                                         \
        cudaError_t e_ = (call);                                                 \
        if (e_ != cudaSuccess) {                                                 \
            e->err = std::string(#call) + ": " + cudaGetErrorString(e_);         \
            return HC_ERR_CUDA;                                                  \
        }                                                                        \
    } while (0)

namespace {

// Everything of one step after the positions are final, on e->stream,
// without host synchronisation (graph-capturable).
int ens_enqueue(hc_ens *e, double kick_dthf, int64_t nstep, double dt, bool capturing, bool advance = true)
{
    cudaStream_t s = e->stream;
    const unsigned rflags = capturing ? cudaEventRecordExternal : cudaEventRecordDefault;
    e->launches = 0;
    EC(cudaEventRecordWithFlags(e->ev[0], s, rflags));
    if (e->forest) {
        hc_ctx *c = e->forest;
        EC(cudaMemsetAsync(c->st, 0, sizeof(hc_status), s));
        k_ens_replay<<<e->nsys_tree, 256, 0, s>>>(e->d_off, e->mass, e->px, e->py, e->pz, e->d_box, c->st);
        k_ens_layout<<<1, 256, 0, s>>>(e->nsys_tree, e->gbits, e->d_box, e->d_origin, e->d_depth, e->d_root, c->box,
                                       c->st);
        k_ens_translate<<<hc_grid(e->n_tree, 256), 256, 0, s>>>(e->n_tree, e->d_body_sys, e->d_box, e->d_origin,
                                                                e->mass, e->px, e->py, e->pz, c->px, c->py, c->pz);
        e->launches += 3;
        c->launches = 0;
        int r = hc_tree_build(c);
        if (r != HC_OK) {
            e->err = c->err;
            return r;
        }
        k_ens_roots<<<hc_grid(c->maxnode, 256), 256, 0, s>>>(c->box, c->nodeC, c->bfs_a, c->xidx,
                                                             e->d_body_sys, e->d_depth, e->d_root);
        r = hc_walk_launch(c, true, c->n, c->tord, c->px, c->py, c->pz, c->ax, c->ay, c->az, c->phi, kick_dthf,
                           nstep);
        if (r != HC_OK) {
            e->err = c->err;
            return r;
        }
        e->launches += c->launches + 1;
    }
    EC(cudaEventRecordWithFlags(e->ev[1], s, rflags));
    if (e->nsys_direct > 0) {
        k_ens_direct<<<e->ndwork, e->direct_threads, ens_direct_smem(e->max_direct_n, e->direct_threads), s>>>(
            e->d_dwork, e->d_off, e->mass, e->px, e->py, e->pz, (float)(e->prm.eps * e->prm.eps), kick_dthf, nstep,
            e->vx, e->vy, e->vz, e->ax, e->ay, e->az, e->phi);
        e->launches++;
    }
    EC(cudaEventRecordWithFlags(e->ev[2], s, rflags));
    if (!advance) return HC_OK;          // forces only (the autotuner's evaluations)
    k_ens_energy<<<e->nework, DTHREADS, 0, s>>>(e->d_ework, e->d_off, e->mass, e->vx, e->vy, e->vz, e->phi, e->d_epart);
    k_ens_energy_sum<<<(e->nsys + 127) / 128, 128, 0, s>>>(e->nsys, e->d_echunk0, e->d_user_of, e->d_epart, e->d_energy);
    k_ens_kick_drift<<<hc_grid(e->ntot, 256), 256, 0, s>>>(e->ntot, dt, e->px, e->py, e->pz, e->vx, e->vy, e->vz,
                                                           e->ax, e->ay, e->az);
    e->launches += 3;
    EC(cudaMemcpyAsync(e->h_energy, e->d_energy, sizeof(double) * 3 * e->nsys, cudaMemcpyDeviceToHost, s));
    if (e->forest) EC(cudaMemcpyAsync(e->forest->h_st, e->forest->st, sizeof(hc_status), cudaMemcpyDeviceToHost, s));
    return HC_OK;
}

const char *status_text(int code)
{
    switch (code) {
    case HC_ERR_COINCIDENT: return "two bodies of one system share a key at the forest's resolution";
    case HC_ERR_CELLS: return "cell pool exhausted";
    case HC_ERR_STACK: return "walk stack overflow";
    case HC_ERR_ARG: return "non-finite position, or a system box too large for the forest";
    case HC_ERR_STATE: return "a tree system has no root cell";
    default: return "device error";
    }
}

}  // namespace

extern "C" {

int hc_ens_create(hc_ens **out, int nsys, const int64_t *counts, const hc_ens_params *params)
{
    if (!out || nsys < 1 || !counts || !params) return HC_ERR_ARG;
    if (params->direct_max < 0 || params->direct_max > HC_ENS_DIRECT_LIMIT || !(params->eps >= 0.0) ||
        !(params->tol >= 0.0) || !std::isfinite(params->eps) || !std::isfinite(params->tol))
        return HC_ERR_ARG;
    hc_ens *e = new hc_ens();
    *out = e;
    e->prm = *params;
    e->nsys = nsys;
    e->user_count.assign(counts, counts + nsys);
    e->user_off.assign(nsys + 1, 0);
    for (int s = 0; s < nsys; s++) {
        if (counts[s] < 1) {
            e->err = "every system needs at least one body";
            return HC_ERR_ARG;
        }
        if (counts[s] > (1LL << 28) || e->user_off[s] + counts[s] > (1LL << 28)) {
            e->err = "at most 2^28 bodies in all";
            return HC_ERR_ARG;
        }
        e->user_off[s + 1] = e->user_off[s] + counts[s];
    }
    e->ntot = e->user_off[nsys];
    if (e->ntot > (1LL << 28)) {
        e->err = "at most 2^28 bodies in all";
        return HC_ERR_ARG;
    }
    // internal order: tree systems (more than direct_max bodies) first
    for (int s = 0; s < nsys; s++)
        if (counts[s] > params->direct_max) e->order.push_back(s);
    e->nsys_tree = (int)e->order.size();
    for (int s = 0; s < nsys; s++)
        if (counts[s] <= params->direct_max) {
            e->order.push_back(s);
            e->max_direct_n = std::max<int>(e->max_direct_n, (int)counts[s]);
        }
    e->nsys_direct = nsys - e->nsys_tree;
    e->int_off.assign(nsys + 1, 0);
    for (int k = 0; k < nsys; k++) e->int_off[k + 1] = e->int_off[k] + counts[e->order[k]];
    e->n_tree = e->int_off[e->nsys_tree];
    while ((1LL << (3 * e->gbits)) < e->nsys_tree) e->gbits++;

    const int64_t n = e->ntot;
    double **arrs[] = {&e->mass, &e->px, &e->py, &e->pz, &e->vx, &e->vy, &e->vz, &e->ax, &e->ay, &e->az, &e->phi};
    for (double **p : arrs) HC_TRY(ens_alloc(e->err, p, n));
    HC_TRY(ens_alloc(e->err, &e->d_off, nsys + 1));
    HC_TRY(ens_alloc(e->err, &e->d_body_sys, n));
    HC_TRY(ens_alloc(e->err, &e->d_user_of, nsys));
    HC_TRY(ens_alloc(e->err, &e->d_user0, nsys));
    std::vector<int2> dwork, ework;
    std::vector<int32_t> echunk0(nsys + 1, 0);
    for (int k = 0; k < nsys; k++) {
        const int cnt = (int)(e->int_off[k + 1] - e->int_off[k]);
        if (k >= e->nsys_tree)
            for (int r = 0; r < cnt; r += DROWS) dwork.push_back(make_int2(k, r));
        for (int r = 0; r < cnt; r += ECHUNK) ework.push_back(make_int2(k, r));
        echunk0[k + 1] = (int32_t)ework.size();
    }
    e->ndwork = (int)dwork.size();
    e->nework = (int)ework.size();
    HC_TRY(ens_alloc(e->err, &e->d_dwork, std::max(1, e->ndwork)));
    HC_TRY(ens_alloc(e->err, &e->d_ework, e->nework));
    HC_TRY(ens_alloc(e->err, &e->d_epart, e->nework));
    HC_TRY(ens_alloc(e->err, &e->d_echunk0, nsys + 1));
    HC_TRY(ens_alloc(e->err, &e->d_root, std::max(1, e->nsys_tree)));
    HC_TRY(ens_alloc(e->err, &e->d_depth, std::max(1, e->nsys_tree)));
    HC_TRY(ens_alloc(e->err, &e->d_box, std::max(1, e->nsys_tree)));
    HC_TRY(ens_alloc(e->err, &e->d_origin, 3 * std::max(1, e->nsys_tree)));
    HC_TRY(ens_alloc(e->err, &e->d_energy, 3 * nsys));
    EC(cudaMallocHost((void **)&e->h_energy, sizeof(double) * 3 * nsys));
    {
        std::vector<int32_t> body_sys(n), user_of(nsys);
        for (int k = 0; k < nsys; k++) {
            user_of[k] = e->order[k];
            for (int64_t i = e->int_off[k]; i < e->int_off[k + 1]; i++) body_sys[i] = k;
        }
        std::vector<int64_t> user0(nsys);
        for (int k = 0; k < nsys; k++) user0[k] = e->user_off[e->order[k]];
        EC(cudaMemcpy(e->d_user0, user0.data(), sizeof(int64_t) * nsys, cudaMemcpyHostToDevice));
        EC(cudaMemcpy(e->d_off, e->int_off.data(), sizeof(int64_t) * (nsys + 1), cudaMemcpyHostToDevice));
        EC(cudaMemcpy(e->d_body_sys, body_sys.data(), sizeof(int32_t) * n, cudaMemcpyHostToDevice));
        EC(cudaMemcpy(e->d_user_of, user_of.data(), sizeof(int32_t) * nsys, cudaMemcpyHostToDevice));
        if (e->ndwork) EC(cudaMemcpy(e->d_dwork, dwork.data(), sizeof(int2) * dwork.size(), cudaMemcpyHostToDevice));
        EC(cudaMemcpy(e->d_ework, ework.data(), sizeof(int2) * ework.size(), cudaMemcpyHostToDevice));
        EC(cudaMemcpy(e->d_echunk0, echunk0.data(), sizeof(int32_t) * (nsys + 1), cudaMemcpyHostToDevice));
    }
    if (e->nsys_tree > 0) {
        hc_params p = {params->tol, params->eps, params->fcells > 0 ? params->fcells : 1.0, params->usequad, 0};
        int r = hc_create(&e->forest, e->n_tree, &p);
        if (r != HC_OK) {
            e->err = e->forest ? std::string("forest: ") + e->forest->err : "forest context";
            return r;
        }
        hc_ctx *c = e->forest;
        // the forest shares the tree systems' mass, velocity, acceleration, potential
        double **mine[] = {&c->mass, &c->vx, &c->vy, &c->vz, &c->ax, &c->ay, &c->az, &c->phi};
        double *ens[] = {e->mass, e->vx, e->vy, e->vz, e->ax, e->ay, e->az, e->phi};
        for (int k = 0; k < 8; k++) {
            cudaFree(*mine[k]);
            *mine[k] = ens[k];
        }
        c->group_kind = HC_GROUPS_TREE;      // groups must not straddle systems
        c->all_massive = true;               // hc_ens_upload takes no others
        c->walk_sys_root = e->d_root;
        c->walk_body_sys = e->d_body_sys;
        e->stream = c->stream;
        k_init_boxes<<<hc_grid(e->nsys_tree, 256), 256, 0, e->stream>>>(e->nsys_tree, e->d_box);
    } else {
        EC(cudaStreamCreateWithFlags(&e->stream, cudaStreamNonBlocking));
        e->own_stream = true;
    }
    for (auto &ev : e->ev) EC(cudaEventCreate(&ev));
    if (e->max_direct_n > 0) {
        // the kernel's attribute is the process's, not this ensemble's: always the largest
        EC(cudaFuncSetAttribute(k_ens_direct, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                (int)ens_direct_smem(HC_ENS_DIRECT_LIMIT, 512)));
    }
    EC(cudaStreamSynchronize(e->stream));
    return HC_OK;
}

void hc_ens_destroy(hc_ens *e)
{
    if (!e) return;
    if (e->stream) cudaStreamSynchronize(e->stream);
    for (auto &g : e->graph)
        if (g) cudaGraphExecDestroy(g);
    if (e->forest) {
        hc_ctx *c = e->forest;
        c->mass = c->vx = c->vy = c->vz = c->ax = c->ay = c->az = c->phi = nullptr;   // owned here
        hc_destroy(c);
    } else if (e->own_stream && e->stream) {
        cudaStreamDestroy(e->stream);
    }
    void *ptrs[] = {e->mass, e->px, e->py, e->pz, e->vx, e->vy, e->vz, e->ax, e->ay, e->az, e->phi, e->d_off,
                    e->d_body_sys, e->d_user_of, e->d_dwork, e->d_ework, e->d_epart, e->d_echunk0, e->d_root, e->d_depth, e->d_box, e->d_origin,
                    e->d_energy, e->d_stage, e->d_user0};
    for (void *p : ptrs)
        if (p) cudaFree(p);
    if (e->h_energy) cudaFreeHost(e->h_energy);
    for (auto &ev : e->ev)
        if (ev) cudaEventDestroy(ev);
    delete e;
}

const char *hc_ens_last_error(const hc_ens *e) { return e ? e->err.c_str() : "null ensemble"; }

int hc_ens_upload(hc_ens *e, const double *mass, const double *phase)
{
    if (!e || !mass || !phase) return HC_ERR_ARG;
    const int64_t n = e->ntot;
    std::vector<double> m(n), ph(6 * n);
    for (int k = 0; k < e->nsys; k++) {
        const int u = e->order[k];
        const int64_t cnt = e->user_count[u];
        std::memcpy(&m[e->int_off[k]], mass + e->user_off[u], sizeof(double) * cnt);
        std::memcpy(&ph[6 * e->int_off[k]], phase + 6 * e->user_off[u], sizeof(double) * 6 * cnt);
    }
    for (int64_t i = 0; i < n; i++)
        if (!std::isfinite(m[i]) || !(m[i] > 0.0)) {
            // a massless body is walked in a run of 32 with its neighbours in
            // key order, which may belong to another system
            e->err = "ensemble bodies need positive, finite masses";
            return HC_ERR_ARG;
        }
    if (!e->d_stage) {
        HC_TRY(ens_alloc(e->err, &e->d_stage, 10 * n));      // the largest download too
    }
    EC(cudaMemcpyAsync(e->mass, m.data(), sizeof(double) * n, cudaMemcpyHostToDevice, e->stream));
    EC(cudaMemcpyAsync(e->d_stage, ph.data(), sizeof(double) * 6 * n, cudaMemcpyHostToDevice, e->stream));
    k_unpack_sys<<<hc_grid(n, 256), 256, 0, e->stream>>>(e->d_stage, n, e->px, e->py, e->pz, e->vx, e->vy, e->vz);
    double *z[] = {e->ax, e->ay, e->az, e->phi};
    for (double *p : z) EC(cudaMemsetAsync(p, 0, sizeof(double) * n, e->stream));
    if (e->nsys_tree > 0)
        k_init_boxes<<<hc_grid(e->nsys_tree, 256), 256, 0, e->stream>>>(e->nsys_tree, e->d_box);
    EC(cudaStreamSynchronize(e->stream));
    EC(cudaGetLastError());
    e->uploaded = true;
    return HC_OK;
}

int hc_ens_step(hc_ens *e, double dt, int64_t nstep, double *energy)
{
    if (!e || !(dt > 0) || nstep < 0) return HC_ERR_ARG;
    const double kick = nstep > 0 ? 0.5 * dt : 0.0;
    const int slot = nstep > 0 ? 1 : 0;
    if (!e->graph[slot] || e->graph_dt[slot] != dt) {
        if (e->graph[slot]) cudaGraphExecDestroy(e->graph[slot]);
        e->graph[slot] = nullptr;
        cudaGraph_t g = nullptr;
        EC(cudaStreamBeginCapture(e->stream, cudaStreamCaptureModeThreadLocal));
        int r = ens_enqueue(e, kick, nstep > 0 ? 1 : 0, dt, true);
        cudaError_t ce = cudaStreamEndCapture(e->stream, &g);
        if (r != HC_OK) {
            if (g) cudaGraphDestroy(g);
            return r;
        }
        if (ce != cudaSuccess) {
            e->err = std::string("stream capture: ") + cudaGetErrorString(ce);
            return HC_ERR_CUDA;
        }
        ce = cudaGraphInstantiate(&e->graph[slot], g, 0);
        cudaGraphDestroy(g);
        if (ce != cudaSuccess) {
            e->graph[slot] = nullptr;
            e->err = std::string("graph instantiate: ") + cudaGetErrorString(ce);
            return HC_ERR_CUDA;
        }
        e->graph_dt[slot] = dt;
        e->graph_launches[slot] = e->launches;
    }
    EC(cudaGraphLaunch(e->graph[slot], e->stream));
    e->launches = e->graph_launches[slot];
    EC(cudaStreamSynchronize(e->stream));
    EC(cudaGetLastError());
    if (e->forest) {
        const hc_status &st = *e->forest->h_st;
        if (st.error) {
            e->err = std::string("ensemble step: ") + status_text(st.error) + " (info " + std::to_string(st.info) + ")";
            return st.error;
        }
    }
    EC(cudaEventElapsedTime(&e->tree_ms, e->ev[0], e->ev[1]));
    EC(cudaEventElapsedTime(&e->direct_ms, e->ev[1], e->ev[2]));
    if (energy) std::memcpy(energy, e->h_energy, sizeof(double) * 3 * e->nsys);
    return HC_OK;
}

int hc_ens_set_tuning(hc_ens *e, const hc_ens_tuning *t)
{
    if (!e || !t) return HC_ERR_ARG;
    if (t->direct_threads != 128 && t->direct_threads != 256 && t->direct_threads != 512) {
        e->err = "hc_ens_set_tuning: direct_threads 128, 256 or 512";
        return HC_ERR_ARG;
    }
    if (e->forest) {
        hc_tuning w{t->group_max, t->list_depth, HC_GROUPS_TREE, 0.0};   // forest groups never straddle systems
        int r = hc_set_tuning(e->forest, &w);
        if (r != HC_OK) {
            e->err = std::string("forest: ") + e->forest->err;
            return r;
        }
    }
    e->direct_threads = t->direct_threads;
    for (int k = 0; k < 2; k++)
        if (e->graph[k]) {
            cudaGraphExecDestroy(e->graph[k]);
            e->graph[k] = nullptr;
        }
    return HC_OK;
}

int hc_ens_get_tuning(hc_ens *e, hc_ens_tuning *t)
{
    if (!e || !t) return HC_ERR_ARG;
    hc_tuning w{HC_GROUP2, 64, HC_GROUPS_TREE, 0.0};
    if (e->forest) hc_get_tuning(e->forest, &w);
    t->group_max = w.group_max;
    t->list_depth = w.list_depth;
    t->direct_threads = e->direct_threads;
    t->tree_ms = t->direct_ms = 0.0;
    return HC_OK;
}

// Times the force phases (tree systems, direct systems) of the current bodies
// for each candidate and keeps the fastest.  Positions and velocities do not
// move; the accelerations and potentials the step in progress needs are
// restored afterwards.
int hc_ens_autotune(hc_ens *e, hc_ens_tuning *best)
{
    if (!e) return HC_ERR_ARG;
    if (!e->uploaded) {
        e->err = "hc_ens_autotune: upload the bodies first";
        return HC_ERR_STATE;
    }
    const int64_t n = e->ntot;
    const size_t b = sizeof(double) * (size_t)n;
    double *const keep[4] = {e->ax, e->ay, e->az, e->phi};
    for (int k = 0; k < 4; k++) EC(cudaMemcpyAsync(e->d_stage + k * n, keep[k], b, cudaMemcpyDeviceToDevice, e->stream));
    hc_ens_tuning cur;
    hc_ens_get_tuning(e, &cur);
    auto timed = [&](const hc_ens_tuning &t, double *tree, double *direct) -> int {
        HC_TRY(hc_ens_set_tuning(e, &t));
        *tree = *direct = 1e300;
        for (int rep = 0; rep < 3; rep++) {
            HC_TRY(ens_enqueue(e, 0.0, 0, 0.0, false, false));
            EC(cudaStreamSynchronize(e->stream));
            if (e->forest) {
                EC(cudaMemcpy(e->forest->h_st, e->forest->st, sizeof(hc_status), cudaMemcpyDeviceToHost));
                if (e->forest->h_st->error) {
                    e->err = std::string("ensemble autotune: ") + status_text(e->forest->h_st->error);
                    return e->forest->h_st->error;
                }
            }
            float t0 = 0.f, t1 = 0.f;
            EC(cudaEventElapsedTime(&t0, e->ev[0], e->ev[1]));
            EC(cudaEventElapsedTime(&t1, e->ev[1], e->ev[2]));
            *tree = std::min(*tree, (double)t0);
            *direct = std::min(*direct, (double)t1);
        }
        return HC_OK;
    };
    hc_ens_tuning win = cur;
    win.tree_ms = win.direct_ms = 1e300;
    int r = HC_OK;
    // the two phases are independent: tree tuning first, then the direct block size
    const int gms[] = {HC_GROUP2 / 2, 3 * HC_GROUP2 / 4, HC_GROUP2}, lds[] = {32, 48, 64}, dts[] = {128, 256, 512};
    for (int gm : gms) {
        if (!e->forest && gm != cur.group_max) continue;
        for (int ld : lds) {
            if (!e->forest && ld != cur.list_depth) continue;
            hc_ens_tuning t{gm, ld, cur.direct_threads, 0.0, 0.0};
            double tr, di;
            if ((r = timed(t, &tr, &di)) != HC_OK) break;
            if (tr < win.tree_ms) {
                win.group_max = gm;
                win.list_depth = ld;
                win.tree_ms = tr;
            }
        }
        if (r != HC_OK) break;
    }
    for (int dt : dts) {
        if (r != HC_OK || e->nsys_direct == 0) break;
        hc_ens_tuning t{win.group_max, win.list_depth, dt, 0.0, 0.0};
        double tr, di;
        if ((r = timed(t, &tr, &di)) != HC_OK) break;
        if (di < win.direct_ms) {
            win.direct_threads = dt;
            win.direct_ms = di;
        }
    }
    for (int k = 0; k < 4; k++) EC(cudaMemcpyAsync(keep[k], e->d_stage + k * n, b, cudaMemcpyDeviceToDevice, e->stream));
    EC(cudaStreamSynchronize(e->stream));
    if (r != HC_OK) {                        // keep the caller's tuning and the error message
        const std::string err = e->err;
        hc_ens_set_tuning(e, &cur);
        e->err = err;
        return r;
    }
    HC_TRY(hc_ens_set_tuning(e, &win));
    if (e->nsys_direct == 0) win.direct_ms = 0.0;
    if (!e->forest) win.tree_ms = 0.0;
    if (best) *best = win;
    return HC_OK;
}

int hc_ens_download(hc_ens *e, double *phase, double *acc, double *phi)
{
    if (!e) return HC_ERR_ARG;
    const int64_t n = e->ntot;
    const int64_t np = phase ? 6 * n : 0, na = acc ? 3 * n : 0, nf = phi ? n : 0;
    if (np + na + nf == 0) {
        EC(cudaStreamSynchronize(e->stream));
        return HC_OK;
    }
    // Packed in the caller's order on the device, then one copy per array.  (Each
    // of the ten components fetched apart and spread over the caller's arrays by
    // the host took 4.4 ms of a 6.7 ms step and download of 320,000 bodies.)
    if (!e->d_stage) {
        HC_TRY(ens_alloc(e->err, &e->d_stage, 10 * n));
    }
    double *d = e->d_stage;
    k_pack_user<<<hc_grid(n, 256), 256, 0, e->stream>>>(n, e->d_body_sys, e->d_off, e->d_user0, e->px, e->py, e->pz, e->vx,
                                                        e->vy, e->vz, e->ax, e->ay, e->az, e->phi, phase ? d : nullptr,
                                                        acc ? d + np : nullptr, phi ? d + np + na : nullptr);
    if (phase) EC(cudaMemcpyAsync(phase, d, sizeof(double) * np, cudaMemcpyDeviceToHost, e->stream));
    if (acc) EC(cudaMemcpyAsync(acc, d + np, sizeof(double) * na, cudaMemcpyDeviceToHost, e->stream));
    if (phi) EC(cudaMemcpyAsync(phi, d + np + na, sizeof(double) * nf, cudaMemcpyDeviceToHost, e->stream));
    EC(cudaStreamSynchronize(e->stream));
    EC(cudaGetLastError());
    return HC_OK;
}

int hc_ens_info(hc_ens *e, hc_ens_stats *out)
{
    if (!e || !out) return HC_ERR_ARG;
    std::memset(out, 0, sizeof *out);
    out->nsys_tree = e->nsys_tree;
    out->nsys_direct = e->nsys_direct;
    out->bodies_tree = e->n_tree;
    out->bodies_direct = e->ntot - e->n_tree;
    int64_t pairs = 0;
    for (int k = e->nsys_tree; k < e->nsys; k++) {
        const int64_t c = e->int_off[k + 1] - e->int_off[k];
        pairs += c * (c - 1);
    }
    out->interactions_direct = pairs;
    if (e->forest) {
        out->interactions_tree = (int64_t)(e->forest->h_st->n2b + e->forest->h_st->nbc);
    }
    out->tree_ms = e->tree_ms;
    out->direct_ms = e->direct_ms;
    out->launches = e->launches;
    return HC_OK;
}

}  // extern "C"
