// hc_learn.cu -- training and test-inference kernels of the learned opening
// criterion's network (hc_mlp.cuh).
//
// Parameters are kept as FP32 master weights in a flat vector
//   W1[64][12], b1[64], W2[64][64], b2[64], W3[64], b3     (5057 floats)
// and packed into the BF16 shared-memory image used by the walk.  Training is
// mini-batch Adam on a binary cross-entropy loss; the forward pass rounds
// weights and activations to BF16 exactly where inference does (straight-
// through gradients), so the trained network is the one the walk evaluates.
#include <cmath>
#include <cuda_pipeline_primitives.h>
#include "hc_internal.cuh"
#include "hc_mlp.cuh"

namespace {

constexpr int NP = MLP_H * MLP_IN + MLP_H + MLP_H * MLP_H + MLP_H + MLP_H + 1;   // 5057
constexpr int OFF_W1 = 0, OFF_B1 = OFF_W1 + MLP_H * MLP_IN, OFF_W2 = OFF_B1 + MLP_H,
              OFF_B2 = OFF_W2 + MLP_H * MLP_H, OFF_W3 = OFF_B2 + MLP_H, OFF_B3 = OFF_W3 + MLP_H;

__device__ __forceinline__ float bf(float x) { return __bfloat162float(__float2bfloat16_rn(x)); }
__device__ __forceinline__ float sigm(float x) { return sigm_fast(x); }          // hidden units (as inference)
__device__ __forceinline__ float sig_out(float x) { return __frcp_rn(1.0f + __expf(-x)); }   // output probability

__global__ void k_mlp_pack(const float *p, MlpSmem *out)
{
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < MLP_H * MLP_S2; i += gridDim.x * blockDim.x) {
        const int n = i / MLP_S2, k = i % MLP_S2;
        out->w2t[i] = __float2bfloat16_rn(k < MLP_H ? p[OFF_W2 + n * MLP_H + k] : 0.f);
        if (n < 8) out->w3t[i] = __float2bfloat16_rn((n == 0 && k < MLP_H) ? p[OFF_W3 + k] : 0.f);
        if (k < MLP_S1) out->w1t[n * MLP_S1 + k] = __float2bfloat16_rn(k < MLP_IN ? p[OFF_W1 + n * MLP_IN + k] : 0.f);
    }
    if (blockIdx.x == 0) {
        for (int j = threadIdx.x; j < MLP_H; j += blockDim.x) {
            out->b1[j] = p[OFF_B1 + j];
            out->b2[j] = p[OFF_B2 + j];
        }
        if (threadIdx.x == 0) out->b3 = p[OFF_B3];
    }
}

// Test inference: 32 rows per warp through the walk's mma.sync network.
__global__ void k_mlp_infer(const MlpSmem *params, const float *x, int64_t n, float *logits)
{
    __shared__ MlpSmem P;
    __shared__ __nv_bfloat16 tile[4][32 * MLP_XS];
    __shared__ float zbuf[4][32];
    mlp_load(P, params);
    __syncthreads();
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const int64_t row = ((int64_t)blockIdx.x * 4 + w) * 32 + lane;
    for (int k = 0; k < MLP_XS; k++)
        tile[w][lane * MLP_XS + k] = __float2bfloat16_rn((row < n && k < MLP_IN) ? x[row * MLP_IN + k] : 0.f);
    __syncwarp();
    const float z = mlp_warp_lean(P, tile[w], zbuf[w], 32);     // the walk's network round
    if (row < n) logits[row] = z;
}

// Gradient of the mean (weighted) binary cross-entropy over rows [0, n) of
// one mini-batch: each block takes TB rows and writes its partial gradient
// (NP floats, NPS apart) and loss.
//
// A batch of 4096 rows is 64 blocks and a chain of 64 x 64 x 64 products (the
// second layer, its transpose, its weights' gradient): bound by the latency of
// one block.  Four warps make the products, a tile of 8 x 4 per thread (3600
// cycles a product; the arithmetic alone would take 2048), and the other four the
// sums beside them: the last layer, the biases and the first layer's weights.  Operands needed along
// both dimensions are stored twice, laid out so that neither store meets a bank
// twice; the weights come rounded and in that layout from the step before
// (MlpImage: 900 cycles to load, 4700 from the parameters).  Pre-activations
// stay in registers from the forward to the backward pass.  Every sum keeps one
// order (inputs, rows, blocks ascending).  A step of 4096 rows, gradient and
// update: 46 us with one output at a time and operands strided over the banks,
// 12.8 us so (14.4 with all eight warps on every part).
constexpr int TB = 64;
constexpr int GT = 256;
constexpr int LD = MLP_H + 4;
constexpr int NPS = (NP + 3) / 4 * 4;

struct alignas(16) MlpImage {                  // weights bf16-rounded
    float W2[MLP_H * LD], W2T[MLP_H * LD];     // W2[j][k], W2T[k][j]
    float W1T[MLP_IN * LD];                    // W1[k][j]
    float W3[MLP_H], b1[MLP_H], b2[MLP_H], b3[4];
};

struct GradSmem {
    MlpImage P;                                // W2T later dz1[s][k] (turned rows)
    float H1[TB * MLP_H], H1T[MLP_H * LD];     // H1[s][k] (turned rows), H1T[k][s]
    float D2[TB * MLP_H], D2T[MLP_H * LD];     // dz2[s][j] (turned rows), dz2[j][s]
    float H2T[MLP_H * LD];                     // H2[j][s]
    float XT[MLP_IN * LD], X[TB * 16];         // inputs [k][s]; [s][k], then 1 and zeros
    float D[TB], red[32];                      // D: dL/dz3
};
static_assert(sizeof(GradSmem) <= 227 * 1024, "shared memory of a block");

__device__ __forceinline__ void image_put(MlpImage *m, int i, float v)
{
    if (i < OFF_B1) {
        m->W1T[i % MLP_IN * LD + i / MLP_IN] = bf(v);
    } else if (i < OFF_W2) {
        m->b1[i - OFF_B1] = v;
    } else if (i < OFF_B2) {
        const int j = (i - OFF_W2) / MLP_H, k = (i - OFF_W2) % MLP_H;
        m->W2[j * LD + k] = m->W2T[k * LD + j] = bf(v);
    } else if (i < OFF_W3) {
        m->b2[i - OFF_B2] = v;
    } else if (i < OFF_B3) {
        m->W3[i - OFF_W3] = bf(v);
    } else {
        m->b3[0] = v;
    }
}

__global__ void k_mlp_image(const float *p, MlpImage *m)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < NP) image_put(m, i, p[i]);
}

// Programmatic dependent launch: a kernel of the training loop starts while its
// predecessor drains, and waits here for all of it.
__device__ __forceinline__ void wait_predecessor()
{
    asm volatile("griddepcontrol.wait;" ::: "memory");
    asm volatile("griddepcontrol.launch_dependents;");
}

__device__ __forceinline__ float4 ld4(const float *p) { return *reinterpret_cast<const float4 *>(p); }

// Row r of a transposed array (64 floats) is stored turned by r / 4 chunks of four, so
// that lanes that write one chunk each of every fourth row meet no bank twice.
__device__ __forceinline__ int turned(int r, int chunk) { return r * MLP_H + 4 * ((chunk + (r >> 2)) & (MLP_H / 4 - 1)); }

// out[i][q] += sum over r < ROWS of a[r][R + i] b[r][C + q], r ascending (arrays of
// turned rows or of rows LD apart): tile rows in packed pairs, half the instructions
// to issue
template <int ROWS, bool TURNED>
__device__ __forceinline__ void tile_product(const float *a, const float *b, int R, int C, float (&out)[8][4])
{
    float2 o[4][4];
#pragma unroll
    for (int i = 0; i < 4; i++)
#pragma unroll
        for (int q = 0; q < 4; q++) o[i][q] = make_float2(out[2 * i][q], out[2 * i + 1][q]);
#pragma unroll 2
    for (int r0 = 0; r0 < ROWS; r0 += 4) {
        const float *a0 = a + (TURNED ? turned(r0, R / 4) : r0 * LD + R), *a1 = a + (TURNED ? turned(r0, R / 4 + 1) : r0 * LD + R + 4),
                    *b0 = b + (TURNED ? turned(r0, C / 4) : r0 * LD + C);
#pragma unroll
        for (int d = 0; d < 4; d++) {
            const int step = d * (TURNED ? MLP_H : LD);
            const float4 u0 = ld4(a0 + step), u1 = ld4(a1 + step), v = ld4(b0 + step);
            const float2 u[4] = {lo2(u0), hi2(u0), lo2(u1), hi2(u1)};
            const float vq[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
            for (int i = 0; i < 4; i++)
#pragma unroll
                for (int q = 0; q < 4; q++) o[i][q] = __ffma2_rn(u[i], splat2(vq[q]), o[i][q]);
        }
    }
#pragma unroll
    for (int i = 0; i < 4; i++)
#pragma unroll
        for (int q = 0; q < 4; q++) {
            out[2 * i][q] = o[i][q].x;
            out[2 * i + 1][q] = o[i][q].y;
        }
}

// a tile as rows LD apart, and its transpose as turned rows
__device__ __forceinline__ void tile_rows(const float (&t)[8][4], int R, int C, float *rows)
{
#pragma unroll
    for (int i = 0; i < 8; i++)
        *reinterpret_cast<float4 *>(rows + (R + i) * LD + C) = make_float4(t[i][0], t[i][1], t[i][2], t[i][3]);
}
__device__ __forceinline__ void tile_cols(const float (&t)[8][4], int R, int C, float *cols)
{
#pragma unroll
    for (int q = 0; q < 4; q++)
#pragma unroll
        for (int i = 0; i < 8; i += 4)
            *reinterpret_cast<float4 *>(cols + turned(C + q, (R + i) / 4)) =
                make_float4(t[i][q], t[i + 1][q], t[i + 2][q], t[i + 3][q]);
}

#define TILE_EACH                                                                                                      \
    _Pragma("unroll") for (int i = 0; i < 8; i++) _Pragma("unroll") for (int q = 0; q < 4; q++)

__global__ void __launch_bounds__(GT) k_mlp_grad(const MlpImage *img, const float *x, const float *y, const float *wt,
                                                 int64_t n, float inv_norm, float *gpart, float *lpart)
{
    extern __shared__ float4 grad_sm[];
    GradSmem &S = *reinterpret_cast<GradSmem *>(grad_sm);
    const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
    // the first four warps make the products, a tile of 8 x 4 per thread: rows R..,
    // columns C..; the others the sums beside them
    const bool tiles = w < 4;
    const int R = 16 * (w & 3) + 8 * (lane >> 4), C = 4 * (lane & 15);
    const int64_t r0 = (int64_t)blockIdx.x * TB;
    // the rows do not depend on the step before
    for (int i = tid; i < TB * 16; i += GT) {
        const int k = i & 15;
        const int64_t r = r0 + (i >> 4);
        const float v = k < MLP_IN ? (r < n ? bf(x[r * MLP_IN + k]) : 0.f) : k == MLP_IN ? 1.f : 0.f;
        S.X[i] = v;
        if (k < MLP_IN) S.XT[k * LD + (i >> 4)] = v;
    }
    const int row = tid - 128;                          // the row of a thread of the fifth and sixth warp
    float yy = 0.f, ww = 0.f;
    if (row >= 0 && row < TB && r0 + row < n) {
        yy = y[r0 + row];
        ww = wt ? wt[r0 + row] : 1.f;
    }
    wait_predecessor();
    for (int i = tid; i < (int)(sizeof(MlpImage) / 16); i += GT)
        __pipeline_memcpy_async(reinterpret_cast<float4 *>(&S.P) + i, reinterpret_cast<const float4 *>(img) + i, 16);
    __pipeline_commit();
    __pipeline_wait_prior(0);
    __syncthreads();
    // forward: hidden units R.., rows C..
    float z1[8][4], z2[8][4], t[8][4];
    if (tiles) {
        TILE_EACH
        {
            z1[i][q] = S.P.b1[R + i];
            z2[i][q] = S.P.b2[R + i];
        }
        tile_product<MLP_IN, false>(S.P.W1T, S.XT, R, C, z1);
        TILE_EACH t[i][q] = bf(silu(z1[i][q]));
        tile_rows(t, R, C, S.H1T);
        tile_cols(t, R, C, S.H1);
    }
    __syncthreads();
    if (tiles) {
        tile_product<MLP_H, false>(S.P.W2T, S.H1T, R, C, z2);
        TILE_EACH t[i][q] = bf(silu(z2[i][q]));
        tile_rows(t, R, C, S.H2T);
    }
    __syncthreads();
    float lsum = 0.f;
    if (row >= 0 && row < TB) {
        float z = S.P.b3[0];
#pragma unroll 16
        for (int k = 0; k < MLP_H; k++) z = fmaf(S.P.W3[k], S.H2T[k * LD + row], z);
        float d = 0.f;
        if (r0 + row < n) {
            // BCE with logits: max(z,0) - z y + log(1 + exp(-|z|))
            lsum += ww * (fmaxf(z, 0.f) - z * yy + log1pf(__expf(-fabsf(z))));
            d = ww * (sig_out(z) - yy) * inv_norm;
        }
        S.D[row] = d;
        if (row >= 32) S.red[lane] = lsum;
    }
    __syncthreads();
    if (tiles) {
        // backward: dz2 = d * w3 * silu'(z2)
        TILE_EACH
        {
            const float z = z2[i][q], sg = sigm(z);
            t[i][q] = S.D[C + q] * S.P.W3[R + i] * sg * (1.f + z * (1.f - sg));
        }
        tile_rows(t, R, C, S.D2T);
        tile_cols(t, R, C, S.D2);
    } else if (w == 4) {
        float l = lsum + S.red[lane];
        for (int o = 16; o; o >>= 1) l += __shfl_down_sync(0xffffffffu, l, o);
        if (lane == 0) lpart[blockIdx.x] = l;
    }
    __syncthreads();
    float *dz1 = S.P.W2T, *gp = gpart + (int64_t)blockIdx.x * NPS;
    if (tiles) {
        // dh1 = W2^T dz2 ; dz1 = dh1 * silu'(z1), over W2T
        TILE_EACH t[i][q] = 0.f;
        tile_product<MLP_H, false>(S.P.W2, S.D2T, R, C, t);
        TILE_EACH
        {
            const float z = z1[i][q], sg = sigm(z);
            t[i][q] = t[i][q] * sg * (1.f + z * (1.f - sg));
        }
        tile_cols(t, R, C, dz1);
    } else if (w < 6) {
        // b2, and b3 by one lane
        const int j = tid - 128;
        float g = 0.f, g3 = 0.f;
#pragma unroll 16
        for (int s = 0; s < TB; s++) {
            g += S.D2[turned(s, j / 4) + (j & 3)];
            g3 += S.D[s];
        }
        gp[OFF_B2 + j] = g;
        if (j == 0) gp[OFF_B3] = g3;
    } else {
        const int k = tid - 192;
        float g = 0.f;
#pragma unroll 4
        for (int s = 0; s < TB; s += 4) {
            const float4 h = ld4(S.H2T + k * LD + s), d = ld4(S.D + s);
            g = fmaf(d.x, h.x, g);
            g = fmaf(d.y, h.y, g);
            g = fmaf(d.z, h.z, g);
            g = fmaf(d.w, h.w, g);
        }
        gp[OFF_W3 + k] = g;
    }
    __syncthreads();
    if (tiles) {
        TILE_EACH t[i][q] = 0.f;
        tile_product<TB, true>(S.D2, S.H1, R, C, t);
#pragma unroll
        for (int i = 0; i < 8; i++)
            *reinterpret_cast<float4 *>(gp + OFF_W2 + (R + i) * MLP_H + C) = make_float4(t[i][0], t[i][1], t[i][2], t[i][3]);
    } else {
        // first layer: units R.., input `in`; the column of ones gives the biases
        const int in = lane & 15;
        float2 g[4];
#pragma unroll
        for (int i = 0; i < 4; i++) g[i] = splat2(0.f);
#pragma unroll 8
        for (int s = 0; s < TB; s++) {
            const float4 u0 = ld4(dz1 + turned(s, R / 4)), u1 = ld4(dz1 + turned(s, R / 4 + 1));
            const float2 v = splat2(S.X[s * 16 + in]);
            g[0] = __ffma2_rn(lo2(u0), v, g[0]);
            g[1] = __ffma2_rn(hi2(u0), v, g[1]);
            g[2] = __ffma2_rn(lo2(u1), v, g[2]);
            g[3] = __ffma2_rn(hi2(u1), v, g[3]);
        }
        if (in <= MLP_IN) {
            const bool wt1 = in < MLP_IN;
            float *o = gp + (wt1 ? OFF_W1 + R * MLP_IN + in : OFF_B1 + R);
            const int step = wt1 ? MLP_IN : 1;
#pragma unroll
            for (int i = 0; i < 4; i++) {
                o[2 * i * step] = g[i].x;
                o[(2 * i + 1) * step] = g[i].y;
            }
        }
    }
}

__device__ __forceinline__ float sum_blocks(const float *part, int nblk, int64_t stride)
{
    float g = 0.f;
#pragma unroll 32
    for (int b = 0; b < nblk; b++) g += part[b * stride];
    return g;
}

constexpr int RT = 32;                                   // one warp per block: a parameter per thread over all SMs
constexpr int RB = (NP + RT - 1) / RT + 1;               // the last block adds the losses

__global__ void __launch_bounds__(RT) k_mlp_reduce(const float *gpart, int nblk, float *grad, const float *lpart, float *loss)
{
    const int i = blockIdx.x * RT + threadIdx.x;
    if (i < NP) grad[i] = sum_blocks(gpart + i, nblk, NPS);
    if (blockIdx.x == RB - 1 && threadIdx.x == 0 && loss) *loss = sum_blocks(lpart, nblk, 1);
}

// the gradient's sum over the blocks and Adam's step
__global__ void __launch_bounds__(RT) k_mlp_adam(const float *gpart, int nblk, const float *lpart, float *loss, float *p, float *m,
                                                 float *v, MlpImage *img, float lr, float b1, float b2, float eps, int t)
{
    const int i = blockIdx.x * RT + threadIdx.x;
    const float c1 = 1.f - powf(b1, (float)t), c2 = 1.f - powf(b2, (float)t);
    wait_predecessor();
    if (blockIdx.x == RB - 1) {
        if (threadIdx.x == 0) *loss = sum_blocks(lpart, nblk, 1);
        return;
    }
    if (i >= NP) return;
    const float mi = m[i], vi = v[i], pi = p[i];
    const float g = sum_blocks(gpart + i, nblk, NPS);
    // contracted explicitly: which product is rounded first is amplified over
    // hundreds of steps (weights rounded to BF16 change their neighbour)
    const float mn = fmaf(1.f - b1, g, b1 * mi);
    const float vn = fmaf((1.f - b2) * g, g, b2 * vi);
    m[i] = mn;
    v[i] = vn;
    const float pn = pi - lr * (mn / c1) / (sqrtf(vn / c2) + eps);
    p[i] = pn;
    image_put(img, i, pn);
}

}  // namespace

int hc_mlp_nparams() { return NP; }

int hc_mlp_pack(hc_ctx *c)
{
    k_mlp_pack<<<32, 256, 0, c->stream>>>(c->mlp_p, c->mlp_packed);
    c->launches++;
    return HC_OK;
}

int hc_mlp_infer_impl(hc_ctx *c, const float *x_dev, int64_t n, float *logits_dev)
{
    const int64_t blocks = (n + 127) / 128;
    k_mlp_infer<<<(unsigned)blocks, 128, 0, c->stream>>>(c->mlp_packed, x_dev, n, logits_dev);
    c->launches++;
    return HC_OK;
}

int64_t hc_mlp_partials(int blocks) { return (int64_t)blocks * NPS; }

int64_t hc_mlp_image_floats() { return sizeof(MlpImage) / sizeof(float); }

// Before a gradient or a training: the image of the current parameters.  The
// attribute is set here, per call of the library: it belongs to the current device,
// and a process may drive contexts on several
int hc_mlp_train_setup(hc_ctx *c)
{
    HC_CUDA(cudaFuncSetAttribute(k_mlp_grad, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(GradSmem)));
    k_mlp_image<<<(NP + 255) / 256, 256, 0, c->stream>>>(c->mlp_p, reinterpret_cast<MlpImage *>(c->mlp_image));
    c->launches++;
    return HC_OK;
}

// mean-loss gradient over rows [0, n) (norm = 1/sum of weights), into grad_dev
int hc_mlp_grad_impl(hc_ctx *c, const float *x, const float *y, const float *w, int64_t n, float inv_norm,
                     float *grad_dev, float *loss_dev)
{
    const int nblk = (int)((n + TB - 1) / TB);
    if (nblk > c->mlp_gcap) return HC_ERR_ARG;
    k_mlp_grad<<<nblk, GT, sizeof(GradSmem), c->stream>>>(reinterpret_cast<const MlpImage *>(c->mlp_image), x, y, w, n, inv_norm, c->mlp_gpart, c->mlp_lpart);
    k_mlp_reduce<<<RB, RT, 0, c->stream>>>(c->mlp_gpart, nblk, grad_dev, c->mlp_lpart, loss_dev);
    c->launches += 2;
    return HC_OK;
}

// One step of the training: the gradient of rows [0, n) and Adam's update t,
// each launched while the kernel before it drains.
int hc_mlp_step_impl(hc_ctx *c, const float *x, const float *y, const float *w, int64_t n, float inv_norm, float *loss_dev,
                     float lr, int t)
{
    const int nblk = (int)((n + TB - 1) / TB);
    if (nblk > c->mlp_gcap) return HC_ERR_ARG;
    cudaLaunchAttribute attr;
    attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr.val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(nblk);
    cfg.blockDim = dim3(GT);
    cfg.dynamicSmemBytes = sizeof(GradSmem);
    cfg.stream = c->stream;
    cfg.attrs = &attr;
    cfg.numAttrs = 1;
    HC_CUDA(cudaLaunchKernelEx(&cfg, k_mlp_grad, reinterpret_cast<const MlpImage *>(c->mlp_image), x, y, w, n, inv_norm, c->mlp_gpart, c->mlp_lpart));
    cfg.gridDim = dim3(RB);
    cfg.blockDim = dim3(RT);
    cfg.dynamicSmemBytes = 0;
    HC_CUDA(cudaLaunchKernelEx(&cfg, k_mlp_adam, (const float *)c->mlp_gpart, nblk, (const float *)c->mlp_lpart, loss_dev,
                               c->mlp_p, c->mlp_m, c->mlp_v, reinterpret_cast<MlpImage *>(c->mlp_image), lr, 0.9f, 0.999f, 1e-8f, t));
    c->launches += 2;
    return HC_OK;
}

namespace {

// ---- the training set's shuffle ----
// perm is that of Fisher and Yates's loop
//     for i = n - 1 ... 1: j(i) = draw(n - 1 - i) mod (i + 1); swap(perm[i], perm[j(i)])
// with draws of a 64-bit linear congruential generator, found without the loop.
// Step i fixes perm[i] as what stands at j(i), and moves what stood at i there.
// What stands at p before step i was moved there by the latest step before it,
// the smallest i' > i with j(i') = p, from i'; if there is none it is p.  So with
// first(p) the smallest i' > p with j(i') = p, what stands at p before step p is
// found by following first from p to its end, about ln(n / p) links.
// (262,144 samples: an epoch of 64 steps 1.85 -> 0.99 ms against the loop on the
// host; the steps themselves take 0.92.)
constexpr unsigned NONE = 0xffffffffu;
constexpr int DRAWS = 16;                                // consecutive draws per thread

__global__ void __launch_bounds__(256) k_shuffle_draw(uint64_t seed, int n, unsigned *j_of, unsigned *head, unsigned *next,
                                                      unsigned *first)
{
    const uint64_t A = 6364136223846793005ULL, C = 1442695040888963407ULL;
    const int k0 = (blockIdx.x * blockDim.x + threadIdx.x) * DRAWS;
    if (k0 >= n - 1) return;
    // the state after k0 draws: k0-fold composition of s -> A s + C by squaring
    uint64_t s = seed * 2862933555777941757ULL + 3037000493ULL, a = A, c = C;
    for (int k = k0; k; k >>= 1) {
        if (k & 1) s = a * s + c;
        c = a * c + c;
        a = a * a;
    }
    for (int k = k0; k < k0 + DRAWS && k < n - 1; k++) {
        s = A * s + C;
        const unsigned i = (unsigned)(n - 1 - k), j = (unsigned)(s >> 33) % (i + 1);
        j_of[i] = j;
        next[i] = atomicExch(&head[j], i);               // the steps that draw j
        if (j < i) atomicMin(&first[j], i);
    }
}

__global__ void __launch_bounds__(256) k_shuffle_resolve(int n, const unsigned *j_of, const unsigned *head, const unsigned *next,
                                                         const unsigned *first, int *perm)
{
    const unsigned i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= (unsigned)n) return;
    unsigned p = 0, from = 0;                            // what ends up at 0 stood there before "step 0"
    if (i > 0) {
        p = j_of[i];
        from = NONE;
        for (unsigned q = head[p]; q != NONE; q = next[q])
            if (q > i && q < from) from = q;
    }
    if (from != NONE)
        for (p = from; first[p] != NONE; p = first[p]) {}
    perm[i] = (int)p;
}

// x: 48-byte rows
__global__ void __launch_bounds__(256) k_gather_samples(const int *perm, int n, const float4 *x, const float *y, const float *w,
                                                        float4 *ox, float *oy, float *ow)
{
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        const int64_t j = perm[i];
#pragma unroll
        for (int k = 0; k < 3; k++) ox[3 * (int64_t)i + k] = x[3 * j + k];
        oy[i] = y[j];
        ow[i] = w[j];
    }
}

// Sum of each mini-batch's weights (FP64), a block per batch.
__global__ void __launch_bounds__(256) k_batch_weights(const float *w, int n, int batch, double *sum)
{
    __shared__ double red[256];
    const int b0 = blockIdx.x * batch, nb = n - b0 < batch ? n - b0 : batch;
    double s = 0.0;
    for (int i = threadIdx.x; i < nb; i += 256) s += w[b0 + i];
    red[threadIdx.x] = s;
    __syncthreads();
    for (int o = 128; o; o >>= 1) {
        if (threadIdx.x < o) red[threadIdx.x] += red[threadIdx.x + o];
        __syncthreads();
    }
    if (threadIdx.x == 0) sum[blockIdx.x] = red[0];
}

__global__ void k_relabel(const float *rel, int n, float thr, float *y)
{
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) y[i] = rel[i] <= thr ? 1.f : 0.f;
}
}  // namespace

int hc_relabel_impl(hc_ctx *c, float thr)
{
    if (c->nsample <= 0) return HC_OK;
    k_relabel<<<hc_grid(c->nsample, 256), 256, 0, c->stream>>>(c->sample_rel, c->nsample, thr, c->sample_y);
    c->launches++;
    return HC_OK;
}

int hc_mlp_shuffle(hc_ctx *c, uint64_t seed, int n, unsigned *scratch, int *perm)
{
    unsigned *j_of = scratch, *next = j_of + n, *head = next + n, *first = head + n;
    HC_CUDA(cudaMemsetAsync(head, 0xff, sizeof(unsigned) * 2 * (size_t)n, c->stream));
    k_shuffle_draw<<<(unsigned)((n + 256 * DRAWS - 1) / (256 * DRAWS)), 256, 0, c->stream>>>(seed, n, j_of, head, next, first);
    k_shuffle_resolve<<<(unsigned)((n + 255) / 256), 256, 0, c->stream>>>(n, j_of, head, next, first, perm);
    c->launches += 2;
    return HC_OK;
}

int hc_mlp_gather(hc_ctx *c, const int *perm, int n, float *x, float *y, float *w, int batch, int batches, double *sum)
{
    k_gather_samples<<<hc_grid(n, 256), 256, 0, c->stream>>>(perm, n, reinterpret_cast<const float4 *>(c->sample_x),
                                                             c->sample_y, c->sample_w, reinterpret_cast<float4 *>(x), y, w);
    k_batch_weights<<<batches, 256, 0, c->stream>>>(w, n, batch, sum);
    c->launches += 2;
    return HC_OK;
}
