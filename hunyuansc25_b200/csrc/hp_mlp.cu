// hp_mlp.cu — training and stand-alone inference of the move-scoring MLP, and
// the move log the plain refiner records for training.
//
// No counterpart in the reference (its refinement has no learned component).
// Training is plain FP32 on CUDA cores (mini-batch Adam; the network has 1,377
// parameters; gradients summed in a fixed order, so training is reproducible), inference inside refinement is BF16 tensor-core MMA with FP32
// accumulation (hp_mlp.cuh).  The network only proposes: an LP candidate it
// scores below the threshold is dropped before the exact integer afterburner,
// and every accepted move is still checked and applied in integers.
#include "hp_internal.cuh"
#include "hp_mlp.cuh"

namespace {

// FP32 forward of one sample.
__device__ __forceinline__ float mlp_fwd(const float *__restrict__ P, const float x[HP_MLP_IN])
{
    float a1[HP_MLP_H];
    for (int j = 0; j < HP_MLP_H; j++) {
        float s = P[HP_MLP_OFF_B1 + j];
        for (int i = 0; i < HP_MLP_IN; i++) s += P[HP_MLP_OFF_W1 + j * HP_MLP_IN + i] * x[i];
        a1[j] = fmaxf(s, 0.f);
    }
    float y = P[HP_MLP_OFF_B3];
    for (int j = 0; j < HP_MLP_H; j++) {
        float s = P[HP_MLP_OFF_B2 + j];
        for (int i = 0; i < HP_MLP_H; i++) s += P[HP_MLP_OFF_W2 + j * HP_MLP_H + i] * a1[i];
        y += P[HP_MLP_OFF_W3 + j] * fmaxf(s, 0.f);
    }
    return y;
}

// Gradient of the mean binary cross-entropy (with logits), deterministic: no
// float atomics, so the same samples and parameters give the same gradient bit
// for bit on every run.
//   mlp_grad_kernel    a warp takes 32 samples at a time, one per lane.  The lane
//                      runs its sample forward and backward; the activations and
//                      their gradients go through the warp's shared-memory tile
//                      (one row per sample), from which the lanes add the 32
//                      samples' outer products to the parameter gradients they
//                      hold in registers (a 4 x 8 block of W2 each).  At the end
//                      each CTA sums its warps in order and writes one row of
//                      partial gradients;
//   mlp_finish_kernel  adds the CTAs' rows in a fixed order (in double: the rows
//                      are few) and, in training, takes the Adam step.
// The work is about 3,600 multiply-adds per sample against 36 bytes; the bound is the
// shared-memory pipe that feeds them (4 M samples: the pipe 93 % busy, issue 59 %).  The
// W2 block of 32 registers per lane takes three shared-memory reads per sample for its 32
// multiply-adds; four weights come with every broadcast read of the forward and backward
// layers.  Writing every sample's 1,377
// gradient terms to memory and summing them afterwards, as before, moved 11 KB
// per sample: 2,107 us against 125 us (17.5 TFLOP/s) for 300,000 samples, with
// an error against 64-bit sums of 8.9e-8 against 2.7e-8.
constexpr int MG_WARPS = 4;
constexpr int MG_THREADS = 32 * MG_WARPS;
constexpr int MG_CTAS_PER_SM = 4;              // 128 registers per thread, 47 KB of shared memory per CTA
constexpr int MG_ROW = HP_MLP_H + 4;           // row stride of a tile: 16-byte accesses of 8 lanes hit 32 banks
constexpr int MG_TILE = 32 * MG_ROW;
constexpr int MLP_ROWS = HP_MLP_NPARAM + 1;    // the parameters, then the loss
static_assert(HP_MLP_H == 32 && HP_MLP_IN == 8, "one lane per hidden unit, two float4 per sample");
static_assert(HP_MLP_OFF_W2 % 4 == 0 && HP_MLP_OFF_B2 % 4 == 0 && HP_MLP_OFF_W3 % 4 == 0 && HP_MLP_OFF_B1 % 4 == 0,
              "the layers are read as float4");

struct MlpGradSmem {
    float P[(HP_MLP_NPARAM + 3) / 4 * 4];
    float dy[MG_WARPS][32];
    float x[MG_WARPS][32 * HP_MLP_IN];
    float a1[MG_WARPS][MG_TILE];   // layer 1 activations, then their pre-activation gradients
    float a2[MG_WARPS][MG_TILE];   // layer 2 likewise
};
static_assert(sizeof(float) * MG_WARPS * MLP_ROWS <= sizeof(float) * 2 * MG_WARPS * MG_TILE,
              "the CTA's sum over its warps reuses the tiles");

__device__ __forceinline__ float4 ld4(const float *p) { return *reinterpret_cast<const float4 *>(p); }

__global__ void __launch_bounds__(MG_THREADS, MG_CTAS_PER_SM)
mlp_grad_kernel(const float *__restrict__ P, const float *__restrict__ X, const float *__restrict__ Y,
                const int32_t *__restrict__ idx, int64_t b0, int64_t nb, float scale, float *__restrict__ part)
{
    __shared__ __align__(16) MlpGradSmem sm;
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    for (int i = threadIdx.x; i < HP_MLP_NPARAM; i += MG_THREADS) sm.P[i] = P[i];
    __syncthreads();
    float *A1 = sm.a1[wid], *A2 = sm.a2[wid], *sx = sm.x[wid], *sdy = sm.dy[wid];
    float *row1 = A1 + lane * MG_ROW, *row2 = A2 + lane * MG_ROW;   // the lane's own sample
    const float *W1 = sm.P + HP_MLP_OFF_W1, *B1 = sm.P + HP_MLP_OFF_B1, *W2 = sm.P + HP_MLP_OFF_W2;
    const float *B2 = sm.P + HP_MLP_OFF_B2, *W3 = sm.P + HP_MLP_OFF_W3;
    const int j0 = (lane >> 2) * 4, i0 = (lane & 3) * 8;   // the lane's block of W2: rows j0..+4, columns i0..+8
    float g2[4][8], g1[HP_MLP_IN], gb1 = 0.f, gb2 = 0.f, gw3 = 0.f, gb3 = 0.f;
    double loss = 0.0;   // (one addition per sample: its rounding would show in the mean)
#pragma unroll
    for (int a = 0; a < 4; a++)
#pragma unroll
        for (int b = 0; b < 8; b++) g2[a][b] = 0.f;
#pragma unroll
    for (int c = 0; c < HP_MLP_IN; c++) g1[c] = 0.f;

    const int64_t nwarps = (int64_t)gridDim.x * MG_WARPS;
    for (int64_t t0 = ((int64_t)blockIdx.x * MG_WARPS + wid) * 32; t0 < nb; t0 += nwarps * 32) {
        const int64_t s = t0 + lane;
        const bool ok = s < nb;
        const int64_t r = !ok ? 0 : idx ? idx[b0 + s] : b0 + s;
        float x[HP_MLP_IN], a1[HP_MLP_H];
#pragma unroll
        for (int c = 0; c < HP_MLP_IN; c++) x[c] = ok ? X[r * HP_MLP_IN + c] : 0.f;
        const float t = ok ? Y[r] : 0.f;
        // forward
#pragma unroll
        for (int i = 0; i < HP_MLP_H; i++) {
            const float4 wa = ld4(W1 + i * HP_MLP_IN), wb = ld4(W1 + i * HP_MLP_IN + 4);
            float z = B1[i];
            z += wa.x * x[0];
            z += wa.y * x[1];
            z += wa.z * x[2];
            z += wa.w * x[3];
            z += wb.x * x[4];
            z += wb.y * x[5];
            z += wb.z * x[6];
            z += wb.w * x[7];
            a1[i] = fmaxf(z, 0.f);
        }
        __syncwarp();   // every lane is done with the previous samples' rows
#pragma unroll
        for (int i = 0; i < HP_MLP_H; i += 4)
            *reinterpret_cast<float4 *>(row1 + i) = make_float4(a1[i], a1[i + 1], a1[i + 2], a1[i + 3]);
        *reinterpret_cast<float4 *>(sx + lane * HP_MLP_IN) = make_float4(x[0], x[1], x[2], x[3]);
        *reinterpret_cast<float4 *>(sx + lane * HP_MLP_IN + 4) = make_float4(x[4], x[5], x[6], x[7]);
        float y = sm.P[HP_MLP_OFF_B3];
#pragma unroll 1
        for (int j = 0; j < HP_MLP_H; j += 4) {
            const float4 bj = ld4(B2 + j), wj = ld4(W3 + j);
            float z[4] = {bj.x, bj.y, bj.z, bj.w};
#pragma unroll
            for (int i = 0; i < HP_MLP_H; i += 4) {
#pragma unroll
                for (int q = 0; q < 4; q++) {
                    const float4 w = ld4(W2 + (j + q) * HP_MLP_H + i);
                    z[q] += w.x * a1[i];
                    z[q] += w.y * a1[i + 1];
                    z[q] += w.z * a1[i + 2];
                    z[q] += w.w * a1[i + 3];
                }
            }
#pragma unroll
            for (int q = 0; q < 4; q++) z[q] = fmaxf(z[q], 0.f);
            y += wj.x * z[0];
            y += wj.y * z[1];
            y += wj.z * z[2];
            y += wj.w * z[3];
            *reinterpret_cast<float4 *>(row2 + j) = make_float4(z[0], z[1], z[2], z[3]);
        }
        if (!ok)   // no sample: no activations (they may overflow where no sample's do, and 0 x inf counts)
            for (int j = 0; j < HP_MLP_H; j++) row1[j] = row2[j] = 0.f;
        // loss = softplus(y) - t*y ; dL/dy = sigmoid(y) - t
        const float sp = y > 0 ? y + log1pf(__expf(-y)) : log1pf(__expf(y));
        const float dy = ok ? (1.f / (1.f + __expf(-y)) - t) * scale : 0.f;
        loss += ok ? (double)((sp - t * y) * scale) : 0.0;
        gb3 += dy;
        sdy[lane] = dy;
        __syncwarp();
#pragma unroll 8
        for (int q = 0; q < 32; q++) gw3 += sdy[q] * A2[q * MG_ROW + lane];
        __syncwarp();   // the activations of layer 2 are read: their gradients take their place
        // backward: dz2 into row2, da1 in registers
        float da1[HP_MLP_H];
#pragma unroll
        for (int i = 0; i < HP_MLP_H; i++) da1[i] = 0.f;
#pragma unroll 1
        for (int j = 0; j < HP_MLP_H; j += 4) {
            const float4 a = ld4(row2 + j), wj = ld4(W3 + j);
            const float d[4] = {a.x > 0.f ? dy * wj.x : 0.f, a.y > 0.f ? dy * wj.y : 0.f,
                                a.z > 0.f ? dy * wj.z : 0.f, a.w > 0.f ? dy * wj.w : 0.f};
#pragma unroll
            for (int q = 0; q < 4; q++)
#pragma unroll
                for (int i = 0; i < HP_MLP_H; i += 4) {
                    const float4 w = ld4(W2 + (j + q) * HP_MLP_H + i);
                    da1[i] += d[q] * w.x;
                    da1[i + 1] += d[q] * w.y;
                    da1[i + 2] += d[q] * w.z;
                    da1[i + 3] += d[q] * w.w;
                }
            *reinterpret_cast<float4 *>(row2 + j) = make_float4(d[0], d[1], d[2], d[3]);
        }
        __syncwarp();
        // W2 and b2: the 32 samples' outer products dz2 x a1
#pragma unroll 4
        for (int q = 0; q < 32; q++) {
            const float4 d = ld4(A2 + q * MG_ROW + j0);
            const float4 u = ld4(A1 + q * MG_ROW + i0), w = ld4(A1 + q * MG_ROW + i0 + 4);
            const float dq[4] = {d.x, d.y, d.z, d.w};
#pragma unroll
            for (int a = 0; a < 4; a++) {
                g2[a][0] += dq[a] * u.x;
                g2[a][1] += dq[a] * u.y;
                g2[a][2] += dq[a] * u.z;
                g2[a][3] += dq[a] * u.w;
                g2[a][4] += dq[a] * w.x;
                g2[a][5] += dq[a] * w.y;
                g2[a][6] += dq[a] * w.z;
                g2[a][7] += dq[a] * w.w;
            }
            gb2 += A2[q * MG_ROW + lane];
        }
        // dz1 in the place of the layer 1 activations (the lane's own are in its row)
        __syncwarp();
#pragma unroll
        for (int i = 0; i < HP_MLP_H; i += 4) {
            const float4 a = ld4(row1 + i);
            *reinterpret_cast<float4 *>(row1 + i) =
                make_float4(a.x > 0.f ? da1[i] : 0.f, a.y > 0.f ? da1[i + 1] : 0.f, a.z > 0.f ? da1[i + 2] : 0.f,
                            a.w > 0.f ? da1[i + 3] : 0.f);
        }
        __syncwarp();
        // W1 (lane: one hidden unit's row) and b1
#pragma unroll 4
        for (int q = 0; q < 32; q++) {
            const float d = A1[q * MG_ROW + lane];
            const float4 u = ld4(sx + q * HP_MLP_IN), w = ld4(sx + q * HP_MLP_IN + 4);
            gb1 += d;
            g1[0] += d * u.x;
            g1[1] += d * u.y;
            g1[2] += d * u.z;
            g1[3] += d * u.w;
            g1[4] += d * w.x;
            g1[5] += d * w.y;
            g1[6] += d * w.z;
            g1[7] += d * w.w;
        }
    }
    // the CTA's sums over its warps, in warp order
    __syncthreads();
    float *sums = &sm.a1[0][0];   // MG_WARPS rows of MLP_ROWS (the tiles are read)
    float *my = sums + wid * MLP_ROWS;
#pragma unroll
    for (int c = 0; c < HP_MLP_IN; c++) my[HP_MLP_OFF_W1 + lane * HP_MLP_IN + c] = g1[c];
    my[HP_MLP_OFF_B1 + lane] = gb1;
#pragma unroll
    for (int a = 0; a < 4; a++)
#pragma unroll
        for (int b = 0; b < 8; b++) my[HP_MLP_OFF_W2 + (j0 + a) * HP_MLP_H + i0 + b] = g2[a][b];
    my[HP_MLP_OFF_B2 + lane] = gb2;
    my[HP_MLP_OFF_W3 + lane] = gw3;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        gb3 += __shfl_xor_sync(HP_FULL_MASK, gb3, o);
        loss += __shfl_xor_sync(HP_FULL_MASK, loss, o);
    }
    if (lane == 0) {
        my[HP_MLP_OFF_B3] = gb3;
        my[HP_MLP_NPARAM] = (float)loss;
    }
    __syncthreads();
    for (int p = threadIdx.x; p < MLP_ROWS; p += MG_THREADS) {
        float t = sums[p];
#pragma unroll
        for (int w = 1; w < MG_WARPS; w++) t += sums[w * MLP_ROWS + p];
        part[(int64_t)blockIdx.x * MLP_ROWS + p] = t;
    }
}

// The Adam step of a training batch (m == nullptr: none).
struct AdamStep {
    float *P, *m, *v;
    float lr, b1, b2, eps, c1, c2;
};

// Gradient row p = the CTAs' partial sums added in a fixed order: 32 rows per
// block, warp w the CTAs w, w + 8, ...; then the warps in order.  Written to
// out[p] (p < HP_MLP_NPARAM) and, when loss is set, added to *loss.
constexpr int MF_WARPS = 8;

__global__ void __launch_bounds__(32 * MF_WARPS)
mlp_finish_kernel(const float *__restrict__ part, int ncta, float *__restrict__ out, float *__restrict__ loss,
                  AdamStep A)
{
    __shared__ double s[MF_WARPS][32];
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    const int p = blockIdx.x * 32 + lane;
    double acc = 0.0;
    if (p < MLP_ROWS) {
#pragma unroll 8
        for (int c = wid; c < ncta; c += MF_WARPS) acc += (double)part[(int64_t)c * MLP_ROWS + p];
    }
    s[wid][lane] = acc;
    __syncthreads();
    if (wid != 0 || p >= MLP_ROWS) return;
    for (int w = 1; w < MF_WARPS; w++) acc += s[w][lane];
    const float g = (float)acc;
    if (p == HP_MLP_NPARAM) {
        if (loss) *loss += g;
        return;
    }
    out[p] = g;
    if (!A.m) return;
    const float mi = A.b1 * A.m[p] + (1.f - A.b1) * g;
    const float vi = A.b2 * A.v[p] + (1.f - A.b2) * g * g;
    A.m[p] = mi;
    A.v[p] = vi;
    A.P[p] -= A.lr * (mi / A.c1) / (sqrtf(vi / A.c2) + A.eps);
}

inline int64_t mlp_grad_ctas(const hp_context *c) { return (int64_t)c->sm_count * MG_CTAS_PER_SM; }

// Gradient (and loss) of samples [b0, b0 + nb) of the index list, scaled by
// `scale`, into g (added to *loss), summed in a fixed order; then A's step.
int mlp_grad_det(hp_context *c, cudaStream_t st, const float *X, const float *Y, const int32_t *idx, int64_t b0,
                 int64_t nb, float scale, float *loss, const AdamStep &A)
{
    const int64_t tiles = (nb + 31) / 32;
    const unsigned ncta = (unsigned)std::min<int64_t>((tiles + MG_WARPS - 1) / MG_WARPS, mlp_grad_ctas(c));
    mlp_grad_kernel<<<ncta, MG_THREADS, 0, st>>>(c->mlp_params, X, Y, idx, b0, nb, scale, c->mlp_scratch);
    mlp_finish_kernel<<<(MLP_ROWS + 31) / 32, 32 * MF_WARPS, 0, st>>>(c->mlp_scratch, (int)ncta, c->mlp_grad, loss, A);
    HP_CUDA(cudaGetLastError());
    return HP_OK;
}

// Stand-alone inference: tensor-core BF16 path (one warp per 32 samples) or
// the FP32 reference path.
__global__ void __launch_bounds__(128)
mlp_infer_kernel(const float *__restrict__ P, const float *__restrict__ X, int64_t n, float *__restrict__ out,
                 int tensor)
{
    hp::pdl_wait();
    __shared__ hp::MlpSmem sm;
    hp::mlp_load_smem(sm, P);
    __syncthreads();
    const int64_t base = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) & ~31ll;
    for (int64_t w0 = base; w0 < n; w0 += (int64_t)gridDim.x * blockDim.x) {
        const int64_t r = w0 + (threadIdx.x & 31);
        float x[HP_MLP_IN];
        for (int i = 0; i < HP_MLP_IN; i++) x[i] = r < n ? X[r * HP_MLP_IN + i] : 0.f;
        float y;
        if (tensor) {
            y = hp::mlp_warp_logit(sm, x);
        } else {
            y = mlp_fwd(P, x);
        }
        if (r < n) out[r] = y;
    }
}

}  // namespace

// ---- context-side state ------------------------------------------------------------
int hp_mlp_ensure(hp_context *c)
{
    if (c->mlp_params) return HP_OK;
    void *p = nullptr;
    HP_CUDA(cudaMalloc(&p, sizeof(float) * 4 * HP_MLP_NPARAM));
    c->mlp_params = (float *)p;
    c->mlp_grad = c->mlp_params + HP_MLP_NPARAM;
    c->mlp_m = c->mlp_grad + HP_MLP_NPARAM;
    c->mlp_v = c->mlp_m + HP_MLP_NPARAM;
    HP_CUDA(cudaMemset(p, 0, sizeof(float) * 4 * HP_MLP_NPARAM));
    HP_CUDA(cudaStreamSynchronize(cudaStreamLegacy));   // (the library's streams do not wait for it)
    return HP_OK;
}

// The CTAs' partial gradients (MLP_ROWS floats each, 3 MB), allocated on the
// first training or gradient call of a context.
int hp_mlp_ensure_scratch(hp_context *c)
{
    if (c->mlp_scratch) return HP_OK;
    void *p = nullptr;
    if (cudaMalloc(&p, sizeof(float) * (size_t)MLP_ROWS * (size_t)mlp_grad_ctas(c)) != cudaSuccess) {
        cudaGetLastError();
        return HP_ERR_NOMEM;
    }
    c->mlp_scratch = (float *)p;
    return HP_OK;
}

#define HP_API extern "C" __attribute__((visibility("default")))

HP_API int hp_mlp_set_params(hp_context *c, const float *params, int32_t count, float threshold)
{
    if (!c || !params || count != HP_MLP_NPARAM) return HP_ERR_INVALID_ARG;
    HP_CUDA(cudaSetDevice(c->device));
    HP_TRY(hp_mlp_ensure(c));
    HP_CUDA(cudaMemcpy(c->mlp_params, params, sizeof(float) * HP_MLP_NPARAM, cudaMemcpyHostToDevice));
    HP_CUDA(cudaMemset(c->mlp_m, 0, sizeof(float) * 2 * HP_MLP_NPARAM));
    HP_CUDA(cudaStreamSynchronize(cudaStreamLegacy));   // (the library's streams do not wait for it)
    c->mlp_threshold = threshold;
    c->mlp_ready = true;
    return HP_OK;
}

HP_API int hp_mlp_get_params(hp_context *c, float *params, int32_t count)
{
    if (!c || !params || count != HP_MLP_NPARAM || !c->mlp_params) return HP_ERR_INVALID_ARG;
    HP_CUDA(cudaSetDevice(c->device));
    HP_CUDA(cudaMemcpy(params, c->mlp_params, sizeof(float) * HP_MLP_NPARAM, cudaMemcpyDeviceToHost));
    return HP_OK;
}

HP_API int hp_mlp_loss_grad(hp_context *c, const float *d_x, const float *d_y, int64_t n, float *grad,
                            float *loss)
{
    if (!c || !d_x || !d_y || n <= 0 || !grad || !c->mlp_params) return HP_ERR_INVALID_ARG;
    HP_CUDA(cudaSetDevice(c->device));
    cudaStream_t s = c->own_stream;
    HP_TRY(hp_mlp_ensure_scratch(c));
    HP_CUDA(cudaMemsetAsync(c->d_scal, 0, sizeof(float), s));
    HP_TRY(mlp_grad_det(c, s, d_x, d_y, nullptr, 0, n, 1.0f / (float)n, (float *)c->d_scal, AdamStep{}));
    HP_CUDA(cudaMemcpyAsync(grad, c->mlp_grad, sizeof(float) * HP_MLP_NPARAM, cudaMemcpyDeviceToHost, s));
    float l = 0;
    HP_CUDA(cudaMemcpyAsync(&l, c->d_scal, sizeof(float), cudaMemcpyDeviceToHost, s));
    HP_CUDA(cudaStreamSynchronize(s));
    if (loss) *loss = l;
    return HP_OK;
}

HP_API int hp_mlp_train(hp_context *c, const float *d_x, const float *d_y, const int32_t *d_perm, int64_t n,
                        int32_t epochs, int32_t batch, float lr, float *final_loss)
{
    if (!c || !d_x || !d_y || n <= 0 || epochs <= 0 || batch <= 0 || !c->mlp_params) return HP_ERR_INVALID_ARG;
    HP_CUDA(cudaSetDevice(c->device));
    cudaStream_t s = c->own_stream;
    HP_TRY(hp_mlp_ensure_scratch(c));
    const float b1 = 0.9f, b2 = 0.999f, eps = 1e-8f;
    float p1 = 1.f, p2 = 1.f;
    for (int e = 0; e < epochs; e++) {
        const bool last_epoch = e == epochs - 1;
        if (last_epoch) HP_CUDA(cudaMemsetAsync(c->d_scal, 0, sizeof(float), s));
        for (int64_t b0 = 0; b0 < n; b0 += batch) {
            const int64_t nb = std::min<int64_t>(batch, n - b0);
            p1 *= b1;
            p2 *= b2;
            HP_TRY(mlp_grad_det(c, s, d_x, d_y, d_perm, b0, nb, 1.0f / (float)nb,
                                last_epoch ? (float *)c->d_scal : (float *)nullptr,
                                AdamStep{c->mlp_params, c->mlp_m, c->mlp_v, lr, b1, b2, eps, 1.f - p1, 1.f - p2}));
        }
    }
    float l = 0;
    HP_CUDA(cudaMemcpyAsync(&l, c->d_scal, sizeof(float), cudaMemcpyDeviceToHost, s));
    HP_CUDA(cudaStreamSynchronize(s));
    if (final_loss) *final_loss = l * (float)batch / (float)n;   // mean over the batches of the last epoch
    c->mlp_ready = true;
    return HP_OK;
}

HP_API int hp_mlp_infer(hp_context *c, const float *d_x, int64_t n, float *d_out, int32_t tensor_cores)
{
    if (!c || !d_x || !d_out || n < 0 || !c->mlp_params) return HP_ERR_INVALID_ARG;
    HP_CUDA(cudaSetDevice(c->device));
    if (n == 0) return HP_OK;
    const unsigned grid = (unsigned)std::min<int64_t>((n + 127) / 128, c->sm_count * 8);
    mlp_infer_kernel<<<grid, 128, 0, c->own_stream>>>(c->mlp_params, d_x, n, d_out, tensor_cores);
    HP_CUDA(cudaGetLastError());
    HP_CUDA(cudaStreamSynchronize(c->own_stream));
    return HP_OK;
}

// ---- move log ------------------------------------------------------------------------
HP_API int hp_movelog_enable(hp_context *c, int64_t capacity)
{
    if (!c || capacity < 0) return HP_ERR_INVALID_ARG;
    HP_CUDA(cudaSetDevice(c->device));
    if (c->log_x) { cudaFree(c->log_x); c->log_x = nullptr; }
    c->log_cap = capacity;
    if (capacity == 0) return HP_OK;
    void *p = nullptr;
    // features, label, and per record: vertex, destination, accepted flag
    const size_t bytes = (size_t)capacity * (sizeof(float) * (HP_MLP_IN + 1) + sizeof(int32_t) * 3) + 256;
    if (cudaMalloc(&p, bytes) != cudaSuccess) { cudaGetLastError(); c->log_cap = 0; return HP_ERR_NOMEM; }
    c->log_x = (float *)p;
    c->log_y = c->log_x + (size_t)capacity * HP_MLP_IN;
    c->log_v = (int32_t *)(c->log_y + capacity);
    c->log_d = c->log_v + capacity;
    c->log_acc = c->log_d + capacity;
    c->log_count = (unsigned long long *)(c->log_acc + capacity);
    HP_CUDA(cudaMemset(c->log_count, 0, sizeof(unsigned long long)));
    HP_CUDA(cudaStreamSynchronize(cudaStreamLegacy));   // (the library's streams do not wait for it)
    return HP_OK;
}

HP_API int64_t hp_movelog_count(hp_context *c)
{
    if (!c || !c->log_x) return 0;
    unsigned long long n = 0;
    if (cudaMemcpy(&n, c->log_count, sizeof(n), cudaMemcpyDeviceToHost) != cudaSuccess) return HP_ERR_CUDA;
    return (int64_t)std::min<unsigned long long>(n, (unsigned long long)c->log_cap);
}

HP_API int hp_movelog_copy(hp_context *c, float *features, float *labels, int64_t count)
{
    if (!c || !c->log_x || count < 0) return HP_ERR_INVALID_ARG;
    int64_t have = hp_movelog_count(c);
    if (count > have) return HP_ERR_INVALID_ARG;
    HP_CUDA(cudaSetDevice(c->device));
    if (features)
        HP_CUDA(cudaMemcpy(features, c->log_x, sizeof(float) * HP_MLP_IN * (size_t)count, cudaMemcpyDeviceToHost));
    if (labels) HP_CUDA(cudaMemcpy(labels, c->log_y, sizeof(float) * (size_t)count, cudaMemcpyDeviceToHost));
    return HP_OK;
}

HP_API int hp_movelog_reset(hp_context *c)
{
    if (!c || !c->log_x) return HP_ERR_INVALID_ARG;
    HP_CUDA(cudaSetDevice(c->device));
    HP_CUDA(cudaMemset(c->log_count, 0, sizeof(unsigned long long)));
    HP_CUDA(cudaStreamSynchronize(cudaStreamLegacy));   // (the library's streams do not wait for it)
    return HP_OK;
}
