// Training and inference kernels of the learned separating-axis MLP.
//
// Training is plain fp32 CUDA-core arithmetic on bf16-rounded weights
// (fp32 master copy, Adam state in fp32):
//   mlp_fused_grads:      forward pass, softmax cross-entropy, backward pass
//       and weight gradients of tiles of samples, one partial row per CTA
//   mlp_reduce_partials:  the rows summed in a fixed order (deterministic)
//   mlp_adam:             bias-corrected Adam on the fp32 masters
//   mlp_pack:             bf16 mma.m16n8k16 B fragments for inference
// Inference (mlp_predict and the fused SAT kernels) runs the packed weights
// on the bf16 tensor cores (axis_mlp.cuh).
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include <mutex>

#include "axis_mlp.cuh"
#include "mlp_launch.h"

namespace rp3dg {

__device__ __forceinline__ float bf16r(float v) { return __bfloat162float(__float2bfloat16_rn(v)); }

// Loss and gradients of a batch, fused: a CTA takes tiles of MLP_TILE samples,
// runs the forward and backward pass of a tile as small register-blocked
// products over shared memory, and keeps its share of every weight gradient
// in registers; at the end it writes one partial per parameter (and the
// summed loss) to its row of `partial`.  Sums run over 32 samples, then over
// a CTA's tiles, then over the CTAs (mlp_reduce_partials), always in the same
// order: the result is the same on every run and, being a tree, closer to the
// exact sum than one running sum over the batch.  Products use explicit
// fused multiply-adds.
//
// Bound: shared-memory loads and FP32 issue; activations and their gradients
// never leave the SM (one thread per sample and one thread per weight, with
// 1088 bytes of scratch per sample between them, took 681 us a call for 8192
// samples; this takes 54 us, the read-back of the loss included).  The tile of 32
// gives 128 CTAs at 4096 samples and 256 at 8192; 296 CTAs (two per SM) take any larger
// batch, so that the partials stay at 8 MB and the reduction at one pass.
// Row strides of 68 and 20 floats keep the float4 reads of 8 consecutive
// rows (the backward products) on distinct banks.
constexpr int MLP_S64 = MLP_H + 4, MLP_S16 = MLP_OUT + 4, MLP_SX = MLP_IN + 4;
constexpr int MLP_SM_W1 = 0;
constexpr int MLP_SM_W2 = MLP_SM_W1 + MLP_IN * MLP_H;
constexpr int MLP_SM_W3 = MLP_SM_W2 + MLP_H * MLP_S64;
constexpr int MLP_SM_X = MLP_SM_W3 + MLP_H * MLP_S16;
constexpr int MLP_SM_H1 = MLP_SM_X + MLP_TILE * MLP_SX;
constexpr int MLP_SM_H2 = MLP_SM_H1 + MLP_TILE * MLP_S64;
constexpr int MLP_SM_D1 = MLP_SM_H2 + MLP_TILE * MLP_S64;
constexpr int MLP_SM_D2 = MLP_SM_D1 + MLP_TILE * MLP_S64;
constexpr int MLP_SM_DZ = MLP_SM_D2 + MLP_TILE * MLP_S64;
constexpr int MLP_SM_FLOATS = MLP_SM_DZ + MLP_TILE * MLP_S16;
constexpr int MLP_GRAD_THREADS = 256;

__device__ __forceinline__ float4 lds4(const float* p) { return *reinterpret_cast<const float4*>(p); }
__device__ __forceinline__ float part4(const float4& v, int i) { return i == 0 ? v.x : (i == 1 ? v.y : (i == 2 ? v.z : v.w)); }

// acc[s][c] += sum_k in[s0 + 16 s][k] * w[k][4 g + c], k in steps of 4
template <int K, int IN_STRIDE, int W_STRIDE>
__device__ __forceinline__ void mlp_rows_times_w(const float* in, const float* w, int s0, int g, float (&acc)[2][4]) {
#pragma unroll 4
    for (int k = 0; k < K; k += 4) {
        const float4 a0 = lds4(in + s0 * IN_STRIDE + k), a1 = lds4(in + (s0 + 16) * IN_STRIDE + k);
#pragma unroll
        for (int kk = 0; kk < 4; kk++) {
            const float4 b = lds4(w + (k + kk) * W_STRIDE + 4 * g);
            const float x0 = part4(a0, kk), x1 = part4(a1, kk);
            acc[0][0] = fmaf(x0, b.x, acc[0][0]); acc[0][1] = fmaf(x0, b.y, acc[0][1]);
            acc[0][2] = fmaf(x0, b.z, acc[0][2]); acc[0][3] = fmaf(x0, b.w, acc[0][3]);
            acc[1][0] = fmaf(x1, b.x, acc[1][0]); acc[1][1] = fmaf(x1, b.y, acc[1][1]);
            acc[1][2] = fmaf(x1, b.z, acc[1][2]); acc[1][3] = fmaf(x1, b.w, acc[1][3]);
        }
    }
}

// acc[s][r] += sum_j in[s0 + 16 s][j] * w[g + 16 r][j] (the transposed product)
template <int J, int IN_STRIDE, int W_STRIDE>
__device__ __forceinline__ void mlp_rows_times_wt(const float* in, const float* w, int s0, int g, float (&acc)[2][4]) {
#pragma unroll 4
    for (int j = 0; j < J; j += 4) {
        const float4 a0 = lds4(in + s0 * IN_STRIDE + j), a1 = lds4(in + (s0 + 16) * IN_STRIDE + j);
#pragma unroll
        for (int r = 0; r < 4; r++) {
            const float4 b = lds4(w + (g + 16 * r) * W_STRIDE + j);
            acc[0][r] = fmaf(a0.w, b.w, fmaf(a0.z, b.z, fmaf(a0.y, b.y, fmaf(a0.x, b.x, acc[0][r]))));
            acc[1][r] = fmaf(a1.w, b.w, fmaf(a1.z, b.z, fmaf(a1.y, b.y, fmaf(a1.x, b.x, acc[1][r]))));
        }
    }
}

__device__ __forceinline__ void mlp_outer(float (&acc)[4], float a, const float4& b) {
    acc[0] = fmaf(a, b.x, acc[0]); acc[1] = fmaf(a, b.y, acc[1]);
    acc[2] = fmaf(a, b.z, acc[2]); acc[3] = fmaf(a, b.w, acc[3]);
}

__global__ void __launch_bounds__(MLP_GRAD_THREADS, 2)
mlp_fused_grads(const float* __restrict__ params, const float* __restrict__ x, const uint8_t* __restrict__ y, uint32_t n,
                float* __restrict__ partial) {
    extern __shared__ __align__(16) float sm[];
    __shared__ float s_b1[MLP_H], s_b2[MLP_H], s_b3[MLP_OUT], s_loss[MLP_TILE];
    const int tid = threadIdx.x, g = tid & 15, s0 = tid >> 4;
    for (int k = tid; k < MLP_IN * MLP_H; k += MLP_GRAD_THREADS) sm[MLP_SM_W1 + k] = bf16r(params[MLP_OFF_W1 + k]);
    for (int k = tid; k < MLP_H * MLP_H; k += MLP_GRAD_THREADS)
        sm[MLP_SM_W2 + (k / MLP_H) * MLP_S64 + k % MLP_H] = bf16r(params[MLP_OFF_W2 + k]);
    for (int k = tid; k < MLP_H * MLP_OUT; k += MLP_GRAD_THREADS)
        sm[MLP_SM_W3 + (k / MLP_OUT) * MLP_S16 + k % MLP_OUT] = bf16r(params[MLP_OFF_W3 + k]);
    if (tid < MLP_H) { s_b1[tid] = params[MLP_OFF_B1 + tid]; s_b2[tid] = params[MLP_OFF_B2 + tid]; }
    if (tid < MLP_OUT) s_b3[tid] = params[MLP_OFF_B3 + tid];
    // this thread's share of the gradients: w2 rows 4 s0 .. + 3, columns 4 g
    // .. + 3; w1 rows 2 s0, 2 s0 + 1 (s0 < 12); w3 row tid / 4, columns
    // 4 (tid % 4) .. + 3; one bias (tid < 144)
    float g2[4][4] = {}, g1[2][4] = {}, g3[4] = {}, gb = 0.0f, loss = 0.0f;
    const float inv_n = 1.0f / float(n);
    for (uint32_t t0 = blockIdx.x * MLP_TILE; t0 < n; t0 += gridDim.x * MLP_TILE) {
        __syncthreads();   // the previous tile's reads are done
        // samples past the end are zero rows with zero output gradients
        for (int k = tid; k < MLP_TILE * MLP_IN; k += MLP_GRAD_THREADS) {
            const uint32_t r = uint32_t(k) / MLP_IN, i = t0 + r;
            sm[MLP_SM_X + r * MLP_SX + uint32_t(k) % MLP_IN] = i < n ? x[size_t(t0) * MLP_IN + k] : 0.0f;
        }
        __syncthreads();
        {
            float a[2][4];
#pragma unroll
            for (int c = 0; c < 4; c++) a[0][c] = a[1][c] = s_b1[4 * g + c];
            mlp_rows_times_w<MLP_IN, MLP_SX, MLP_H>(sm + MLP_SM_X, sm + MLP_SM_W1, s0, g, a);
#pragma unroll
            for (int s = 0; s < 2; s++)
                *reinterpret_cast<float4*>(sm + MLP_SM_H1 + (s0 + 16 * s) * MLP_S64 + 4 * g) =
                    make_float4(fmaxf(a[s][0], 0.0f), fmaxf(a[s][1], 0.0f), fmaxf(a[s][2], 0.0f), fmaxf(a[s][3], 0.0f));
        }
        __syncthreads();
        {
            float a[2][4];
#pragma unroll
            for (int c = 0; c < 4; c++) a[0][c] = a[1][c] = s_b2[4 * g + c];
            mlp_rows_times_w<MLP_H, MLP_S64, MLP_S64>(sm + MLP_SM_H1, sm + MLP_SM_W2, s0, g, a);
#pragma unroll
            for (int s = 0; s < 2; s++)
                *reinterpret_cast<float4*>(sm + MLP_SM_H2 + (s0 + 16 * s) * MLP_S64 + 4 * g) =
                    make_float4(fmaxf(a[s][0], 0.0f), fmaxf(a[s][1], 0.0f), fmaxf(a[s][2], 0.0f), fmaxf(a[s][3], 0.0f));
        }
        __syncthreads();
        {   // logits, softmax cross-entropy: 8 threads a sample, two logits each
            const int s = tid >> 3, j = 2 * (tid & 7);
            float z0 = s_b3[j], z1 = s_b3[j + 1];
            const float* h = sm + MLP_SM_H2 + s * MLP_S64;
#pragma unroll 4
            for (int k = 0; k < MLP_H; k++) {
                const float2 w = *reinterpret_cast<const float2*>(sm + MLP_SM_W3 + k * MLP_S16 + j);
                z0 = fmaf(h[k], w.x, z0);
                z1 = fmaf(h[k], w.y, z1);
            }
            float zmax = fmaxf(z0, z1);
#pragma unroll
            for (int o = 1; o < 8; o <<= 1) zmax = fmaxf(zmax, __shfl_xor_sync(0xffffffffu, zmax, o));
            const float e0 = expf(z0 - zmax), e1 = expf(z1 - zmax);
            float se = e0 + e1;
#pragma unroll
            for (int o = 1; o < 8; o <<= 1) se += __shfl_xor_sync(0xffffffffu, se, o);
            const uint32_t i = t0 + s;
            const bool in = i < n;
            const uint32_t yi = in ? (y[i] < MLP_OUT ? uint32_t(y[i]) : uint32_t(MLP_NO_PROPOSAL)) : 0xffffffffu;
            const float p0 = e0 / se, p1 = e1 / se;
            if (uint32_t(j) == yi) s_loss[s] = -logf(fmaxf(p0, 1e-30f));
            if (uint32_t(j + 1) == yi) s_loss[s] = -logf(fmaxf(p1, 1e-30f));
            if (!in && j == 0) s_loss[s] = 0.0f;
            *reinterpret_cast<float2*>(sm + MLP_SM_DZ + s * MLP_S16 + j) =
                in ? make_float2((p0 - (uint32_t(j) == yi ? 1.0f : 0.0f)) * inv_n,
                                 (p1 - (uint32_t(j + 1) == yi ? 1.0f : 0.0f)) * inv_n)
                   : make_float2(0.0f, 0.0f);
        }
        __syncthreads();
        {
            float a[2][4] = {};
            mlp_rows_times_wt<MLP_OUT, MLP_S16, MLP_S16>(sm + MLP_SM_DZ, sm + MLP_SM_W3, s0, g, a);
#pragma unroll
            for (int s = 0; s < 2; s++)
#pragma unroll
                for (int r = 0; r < 4; r++) {
                    const int o = (s0 + 16 * s) * MLP_S64 + g + 16 * r;
                    sm[MLP_SM_D2 + o] = sm[MLP_SM_H2 + o] > 0.0f ? a[s][r] : 0.0f;
                }
        }
        __syncthreads();
        {
            float a[2][4] = {};
            mlp_rows_times_wt<MLP_H, MLP_S64, MLP_S64>(sm + MLP_SM_D2, sm + MLP_SM_W2, s0, g, a);
#pragma unroll
            for (int s = 0; s < 2; s++)
#pragma unroll
                for (int r = 0; r < 4; r++) {
                    const int o = (s0 + 16 * s) * MLP_S64 + g + 16 * r;
                    sm[MLP_SM_D1 + o] = sm[MLP_SM_H1 + o] > 0.0f ? a[s][r] : 0.0f;
                }
        }
        __syncthreads();
        // the tile's own sums first, then onto the CTA's
        float t2[4][4] = {}, t1[2][4] = {}, t3[4] = {}, tb = 0.0f;
#pragma unroll 4
        for (int s = 0; s < MLP_TILE; s++) {
            const float4 d2 = lds4(sm + MLP_SM_D2 + s * MLP_S64 + 4 * g), h = lds4(sm + MLP_SM_H1 + s * MLP_S64 + 4 * s0);
#pragma unroll
            for (int r = 0; r < 4; r++) mlp_outer(t2[r], part4(h, r), d2);
            mlp_outer(t3, sm[MLP_SM_H2 + s * MLP_S64 + (tid >> 2)], lds4(sm + MLP_SM_DZ + s * MLP_S16 + 4 * (tid & 3)));
        }
        if (s0 < MLP_IN / 2) {
#pragma unroll 4
            for (int s = 0; s < MLP_TILE; s++) {
                const float4 d1 = lds4(sm + MLP_SM_D1 + s * MLP_S64 + 4 * g);
                const float2 xv = *reinterpret_cast<const float2*>(sm + MLP_SM_X + s * MLP_SX + 2 * s0);
                mlp_outer(t1[0], xv.x, d1);
                mlp_outer(t1[1], xv.y, d1);
            }
        }
        if (tid < 2 * MLP_H + MLP_OUT) {
            const float* col = tid < MLP_H ? sm + MLP_SM_D1 + tid : (tid < 2 * MLP_H ? sm + MLP_SM_D2 + tid - MLP_H : sm + MLP_SM_DZ + tid - 2 * MLP_H);
            const int stride = tid < 2 * MLP_H ? MLP_S64 : MLP_S16;
#pragma unroll 4
            for (int s = 0; s < MLP_TILE; s++) tb += col[s * stride];
        } else if (tid == 2 * MLP_H + MLP_OUT) {
            float l = 0.0f;
            for (int s = 0; s < MLP_TILE; s++) l += s_loss[s];
            loss += l;
        }
#pragma unroll
        for (int r = 0; r < 4; r++)
#pragma unroll
            for (int c = 0; c < 4; c++) g2[r][c] += t2[r][c];
#pragma unroll
        for (int c = 0; c < 4; c++) { g1[0][c] += t1[0][c]; g1[1][c] += t1[1][c]; g3[c] += t3[c]; }
        gb += tb;
    }
    float* out = partial + size_t(blockIdx.x) * MLP_PARTIAL_ROW;
    auto put = [&](int at, const float* v) { *reinterpret_cast<float4*>(out + at) = make_float4(v[0], v[1], v[2], v[3]); };
#pragma unroll
    for (int r = 0; r < 4; r++) put(MLP_OFF_W2 + (4 * s0 + r) * MLP_H + 4 * g, g2[r]);
    if (s0 < MLP_IN / 2) {
        put(MLP_OFF_W1 + (2 * s0) * MLP_H + 4 * g, g1[0]);
        put(MLP_OFF_W1 + (2 * s0 + 1) * MLP_H + 4 * g, g1[1]);
    }
    put(MLP_OFF_W3 + (tid >> 2) * MLP_OUT + 4 * (tid & 3), g3);
    if (tid < MLP_H) out[MLP_OFF_B1 + tid] = gb;
    else if (tid < 2 * MLP_H) out[MLP_OFF_B2 + tid - MLP_H] = gb;
    else if (tid < 2 * MLP_H + MLP_OUT) out[MLP_OFF_B3 + tid - 2 * MLP_H] = gb;
    else if (tid == 2 * MLP_H + MLP_OUT) out[MLP_NPARAMS] = loss;
}

// Gradients (and the summed loss, when wanted) from the CTAs' partials: 32
// parameters a block, 8 threads a parameter over every eighth row.
__global__ void __launch_bounds__(256) mlp_reduce_partials(const float* __restrict__ partial, uint32_t rows,
                                                           float* __restrict__ grads, float* __restrict__ loss_sum) {
    __shared__ float red[8][32];
    const uint32_t lane = threadIdx.x & 31u, q = threadIdx.x >> 5, p = blockIdx.x * 32u + lane;
    float s = 0.0f;
    if (p <= uint32_t(MLP_NPARAMS)) {
#pragma unroll 8
        for (uint32_t r = q; r < rows; r += 8) s += partial[size_t(r) * MLP_PARTIAL_ROW + p];
    }
    red[q][lane] = s;
    __syncthreads();
    if (q == 0 && p <= uint32_t(MLP_NPARAMS)) {
        for (int k = 1; k < 8; k++) s += red[k][lane];
        if (p < uint32_t(MLP_NPARAMS)) grads[p] = s;
        else if (loss_sum) *loss_sum = s;
    }
}

__global__ void mlp_adam(float* __restrict__ params, const float* __restrict__ grads, float* __restrict__ m,
                         float* __restrict__ v, float lr, float beta1, float beta2, float eps, float bc1, float bc2) {
    const uint32_t p = blockIdx.x * blockDim.x + threadIdx.x;
    if (p >= uint32_t(MLP_NPARAMS)) return;
    const float g = grads[p];
    const float mi = beta1 * m[p] + (1.0f - beta1) * g;
    const float vi = beta2 * v[p] + (1.0f - beta2) * g * g;
    m[p] = mi;
    v[p] = vi;
    params[p] -= lr * (mi / bc1) / (sqrtf(vi / bc2) + eps);
}

// bf16 B fragments of the three layers (layout in axis_mlp.cuh).
__global__ void mlp_pack(const float* __restrict__ params, MlpPacked* __restrict__ out) {
    const uint32_t e = blockIdx.x * blockDim.x + threadIdx.x;
    auto frag = [&](int off, int K, int N, int ks, int nt, int lane) {
        const int g = lane >> 2, t = lane & 3, col = 8 * nt + g;
        auto w = [&](int k) { return k < K ? params[off + k * N + col] : 0.0f; };
        const int k0 = 16 * ks + 2 * t;
        uint2 r;
        r.x = pack_bf16x2(w(k0), w(k0 + 1));
        r.y = pack_bf16x2(w(k0 + 8), w(k0 + 9));
        return r;
    };
    if (e < uint32_t(MLP_FRAG_L1)) {
        const int lane = e & 31, blk = e >> 5, nt = blk % (MLP_H / 8), ks = blk / (MLP_H / 8);
        out->l1[e] = frag(MLP_OFF_W1, MLP_IN, MLP_H, ks, nt, lane);
    } else if (e < uint32_t(MLP_FRAG_L1 + MLP_FRAG_L2)) {
        const uint32_t q = e - MLP_FRAG_L1;
        const int lane = q & 31, blk = q >> 5, nt = blk % (MLP_H / 8), ks = blk / (MLP_H / 8);
        out->l2[q] = frag(MLP_OFF_W2, MLP_H, MLP_H, ks, nt, lane);
    } else if (e < uint32_t(MLP_FRAG_L1 + MLP_FRAG_L2 + MLP_FRAG_L3)) {
        const uint32_t q = e - MLP_FRAG_L1 - MLP_FRAG_L2;
        const int lane = q & 31, blk = q >> 5, nt = blk % (MLP_OUT / 8), ks = blk / (MLP_OUT / 8);
        out->l3[q] = frag(MLP_OFF_W3, MLP_H, MLP_OUT, ks, nt, lane);
    }
    if (e < uint32_t(MLP_H)) { out->b1[e] = params[MLP_OFF_B1 + e]; out->b2[e] = params[MLP_OFF_B2 + e]; }
    if (e < uint32_t(MLP_OUT)) out->b3[e] = params[MLP_OFF_B3 + e];
}

// Tensor-core inference over feature rows: one warp per 32 rows.
__global__ void __launch_bounds__(128) mlp_predict(const MlpPacked* __restrict__ w, const float* __restrict__ x,
                                                   uint32_t n, uint8_t* __restrict__ cls) {
    __shared__ float tile[4][32][MLP_KPAD];
    __shared__ uint32_t out[4][32];
    __shared__ MlpPacked s_w;
    {
        const uint32_t* src = reinterpret_cast<const uint32_t*>(w);
        uint32_t* dst = reinterpret_cast<uint32_t*>(&s_w);
        for (uint32_t k = threadIdx.x; k < sizeof(MlpPacked) / 4; k += blockDim.x) dst[k] = src[k];
    }
    __syncthreads();
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const uint32_t nwarps = gridDim.x * 4;
    for (uint32_t t0 = (blockIdx.x * 4 + warp) * 32u; t0 < n; t0 += nwarps * 32u) {
        const uint32_t i = t0 + lane;
#pragma unroll
        for (int k = 0; k < MLP_KPAD; k++) tile[warp][lane][k] = (i < n && k < MLP_IN) ? x[size_t(i) * MLP_IN + k] : 0.0f;
        __syncwarp();
        const uint32_t c = mlp_infer_tile(tile[warp], s_w, lane, out[warp]);
        if (i < n) cls[i] = uint8_t(c);
        __syncwarp();
    }
}

// ---------------------------------------------------------------------------
// features and labels of pair batches
// ---------------------------------------------------------------------------
RD bool shape_poly(const rp3dg_shape* shapes, int32_t idx, const BoxTables* bt, const uint32_t* mesh_words,
                   BoxPoly& b, MeshPoly& m) {
    const float4 prm = reinterpret_cast<const float4*>(shapes + idx)[0];
    const int4 kk = reinterpret_cast<const int4*>(shapes + idx)[1];
    if (kk.x == RP3DG_SHAPE_BOX) {
        b.he = V(prm.x, prm.y, prm.z);
        b.t = bt;
        return true;
    }
    m.h = reinterpret_cast<const MeshHdr*>(mesh_words) + kk.y;
    m.w = mesh_words;
    return false;
}

__global__ void axis_features_kernel(const MlpPairArgs a, float* __restrict__ feat) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= a.n) return;
    float f[MLP_IN];
    const int32_t i1 = a.shape1[i], i2 = a.shape2[i];
    if (uint32_t(i1) >= a.nb_shapes || uint32_t(i2) >= a.nb_shapes) {
        for (int k = 0; k < MLP_IN; k++) feat[size_t(i) * MLP_IN + k] = 0.0f;
        return;
    }
    const float4 p1 = a.pos1[i], q1 = a.rot1[i], p2 = a.pos2[i], q2 = a.rot2[i];
    const xform t1 = X(V(p1.x, p1.y, p1.z), Q(q1.x, q1.y, q1.z, q1.w));
    const xform t2 = X(V(p2.x, p2.y, p2.z), Q(q2.x, q2.y, q2.z, q2.w));
    BoxPoly b1, b2;
    MeshPoly m1, m2;
    const bool isb1 = shape_poly(a.shapes, i1, a.box, a.mesh_words, b1, m1);
    const bool isb2 = shape_poly(a.shapes, i2, a.box, a.mesh_words, b2, m2);
    if (isb1 && isb2) axis_features(t1, t2, b1, b2, false, f);
    else if (!isb1 && isb2) axis_features(t1, t2, m1, b2, true, f);
    else if (isb1 && !isb2) axis_features(t1, t2, b1, m2, false, f);
    else axis_features(t1, t2, m1, m2, true, f);
    for (int k = 0; k < MLP_IN; k++) feat[size_t(i) * MLP_IN + k] = f[k];
}

__global__ void axis_labels_kernel(const MlpPairArgs a, const uint8_t* __restrict__ colliding,
                                   const rp3dg_lastframe* __restrict__ cache, uint8_t* __restrict__ labels) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= a.n) return;
    const int32_t i1 = a.shape1[i], i2 = a.shape2[i];
    if (uint32_t(i1) >= a.nb_shapes || uint32_t(i2) >= a.nb_shapes) { labels[i] = MLP_NO_PROPOSAL; return; }
    const int k1 = reinterpret_cast<const int4*>(a.shapes + i1)[1].x;
    const int k2 = reinterpret_cast<const int4*>(a.shapes + i2)[1].x;
    const uint4 c = reinterpret_cast<const uint4*>(cache)[i];
    LastFrame lf;
    lf.flags = c.w & 0xffu;
    lf.sat_face = (c.w >> 8) & 0xffu;
    lf.sat_e1 = (c.w >> 16) & 0xffu;
    lf.sat_e2 = (c.w >> 24) & 0xffu;
    labels[i] = uint8_t(axis_label(colliding[i] != 0, lf, k1 == RP3DG_SHAPE_BOX, k2 == RP3DG_SHAPE_BOX, a.box));
}

// Box topology for this translation unit (uploaded with the narrow-phase copy).
__constant__ BoxTables c_mlp_box_tables;

void upload_mlp_box_tables(const BoxTables& t, cudaStream_t s) {
    cudaMemcpyToSymbolAsync(c_mlp_box_tables, &t, sizeof(BoxTables), 0, cudaMemcpyHostToDevice, s);
}

cudaError_t launch_axis_features(const MlpPairArgs& a, float* feat, cudaStream_t s) {
    if (a.n == 0) return cudaSuccess;
    MlpPairArgs b = a;
    void* box = nullptr;
    cudaError_t e = cudaGetSymbolAddress(&box, c_mlp_box_tables);
    if (e != cudaSuccess) return e;
    b.box = static_cast<const BoxTables*>(box);
    axis_features_kernel<<<(a.n + 127) / 128, 128, 0, s>>>(b, feat);
    return cudaGetLastError();
}

cudaError_t launch_axis_labels(const MlpPairArgs& a, const uint8_t* colliding, const rp3dg_lastframe* cache,
                               uint8_t* labels, cudaStream_t s) {
    if (a.n == 0) return cudaSuccess;
    MlpPairArgs b = a;
    void* box = nullptr;
    cudaError_t e = cudaGetSymbolAddress(&box, c_mlp_box_tables);
    if (e != cudaSuccess) return e;
    b.box = static_cast<const BoxTables*>(box);
    axis_labels_kernel<<<(a.n + 127) / 128, 128, 0, s>>>(b, colliding, cache, labels);
    return cudaGetLastError();
}

cudaError_t launch_mlp_grads(const float* params, const float* x, const uint8_t* y, uint32_t n, float* scratch,
                             float* grads, float* loss_sum, cudaStream_t s) {
    if (n == 0) return cudaErrorInvalidValue;
    constexpr int smem = MLP_SM_FLOATS * int(sizeof(float));
    const cudaError_t e = cudaFuncSetAttribute(mlp_fused_grads, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
    if (e != cudaSuccess) return e;
    const uint32_t rows = mlp_partial_rows(n);
    mlp_fused_grads<<<rows, MLP_GRAD_THREADS, smem, s>>>(params, x, y, n, scratch);
    mlp_reduce_partials<<<(MLP_NPARAMS + 1 + 31) / 32, 256, 0, s>>>(scratch, rows, grads, loss_sum);
    return cudaGetLastError();
}

cudaError_t launch_mlp_adam(float* params, const float* grads, float* m, float* v, float lr, int step, cudaStream_t s) {
    const float beta1 = 0.9f, beta2 = 0.999f, eps = 1e-8f;
    const float bc1 = 1.0f - powf(beta1, float(step)), bc2 = 1.0f - powf(beta2, float(step));
    mlp_adam<<<(MLP_NPARAMS + 127) / 128, 128, 0, s>>>(params, grads, m, v, lr, beta1, beta2, eps, bc1, bc2);
    return cudaGetLastError();
}

cudaError_t launch_mlp_pack(const float* params, MlpPacked* out, cudaStream_t s) {
    const int total = MLP_FRAG_L1 + MLP_FRAG_L2 + MLP_FRAG_L3;
    mlp_pack<<<(total + 127) / 128, 128, 0, s>>>(params, out);
    return cudaGetLastError();
}

// ---------------------------------------------------------------------------
// Allocation-free gradients (rp3dg_axis_mlp_grads_noalloc).
//
// Some callers cannot allocate device memory while they run: an engine whose
// host application hands out a fixed GPU memory budget at start-up and
// forbids later cudaMalloc calls (allocations can stall every stream of the
// device and can fail once the budget is in use).  rp3dg_axis_mlp_grads grows
// its training scratch with cudaMalloc whenever a larger batch comes in; this
// variant uses a fixed array in the library's device image instead.  Every
// GPU that loads the library holds the array (3.5 MB) until the process exits.
// All calls share it and it keeps the previous call's contents: the loss word
// and the rows in use are fully rewritten on every call, and calls that
// overlap on the GPU (two streams, two threads) race.
// ---------------------------------------------------------------------------
constexpr uint32_t NOALLOC_ROWS = mlp_partial_rows(MLP_NOALLOC_MAX_SAMPLES);
static __device__ __align__(256) float g_mlp_noalloc_scratch[NOALLOC_ROWS * MLP_PARTIAL_ROW + 64];

namespace {
constexpr int NOALLOC_MAX_DEVICES = 64;
float* g_noalloc_ptr[NOALLOC_MAX_DEVICES] = {};
std::mutex g_noalloc_mutex;
}  // namespace

// Device address of the scratch array on the current device, looked up once
// per device (the host-side name of the array is not a device address).  The
// address belongs to the device's current context: a process that resets the
// device (cudaDeviceReset) while the library is loaded gets a new module
// image, so the cached address is dropped whenever a call fails and the next
// call looks it up again; callers that reset a device must not have a call of
// this entry point in flight on it.
static void noalloc_forget() {
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= NOALLOC_MAX_DEVICES) return;
    std::lock_guard<std::mutex> lock(g_noalloc_mutex);
    g_noalloc_ptr[dev] = nullptr;
}

static cudaError_t noalloc_scratch(float** out) {
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return e;
    if (dev < 0 || dev >= NOALLOC_MAX_DEVICES) return cudaErrorInvalidDevice;
    std::lock_guard<std::mutex> lock(g_noalloc_mutex);
    if (!g_noalloc_ptr[dev]) {
        void* p = nullptr;
        e = cudaGetSymbolAddress(&p, g_mlp_noalloc_scratch);
        if (e != cudaSuccess) return e;
        g_noalloc_ptr[dev] = static_cast<float*>(p);
    }
    *out = g_noalloc_ptr[dev];
    return cudaSuccess;
}

cudaError_t launch_mlp_grads_noalloc(const float* params, const float* x, const uint8_t* y, uint32_t n, float* grads,
                                     float* loss_host, cudaStream_t s) {
    if (n == 0 || n > MLP_NOALLOC_MAX_SAMPLES) return cudaErrorInvalidValue;
    float* scratch = nullptr;
    cudaError_t e = noalloc_scratch(&scratch);
    if (e != cudaSuccess) return e;
    float* loss_word = scratch + size_t(NOALLOC_ROWS) * MLP_PARTIAL_ROW;
    e = launch_mlp_grads(params, x, y, n, scratch, grads, loss_word, s);
    if (e != cudaSuccess) { noalloc_forget(); return e; }
    if (!loss_host) return e;
    float sum = 0.0f;
    e = cudaMemcpyAsync(&sum, loss_word, sizeof(float), cudaMemcpyDeviceToHost, s);
    if (e == cudaSuccess) e = cudaStreamSynchronize(s);
    if (e == cudaSuccess) *loss_host = sum / float(n);
    else noalloc_forget();
    return e;
}

cudaError_t launch_mlp_predict(const MlpPacked* w, const float* x, uint32_t n, uint8_t* cls, int num_sms, cudaStream_t s) {
    if (n == 0) return cudaSuccess;
    const uint32_t blocks_needed = (n + 127) / 128;
    const uint32_t cap = uint32_t(num_sms) * 8u;
    mlp_predict<<<blocks_needed < cap ? blocks_needed : cap, 128, 0, s>>>(w, x, n, cls);
    return cudaGetLastError();
}

}  // namespace rp3dg
