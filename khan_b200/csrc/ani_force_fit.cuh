// Force training: the loss, and the second-order pass through the atomic networks.
//
// Force training minimises a function of the coordinate gradients x = J^T (dE/dF).  With v = dLoss/dx and
// u = J v (the directional derivative of the features along v), the derivative of the loss with respect to
// the weights is that of the scalar sum over atoms of <u, dE/dF>, i.e. of the forward-mode derivative of E
// along u -- the mixed product that the reference leaves to tf.gradients of tf.gradients
// (khan/training/trainer_multi_tower.py:377-399).  With T_l the tangents of the pre-activations, D_l and
// S_l the first and second derivatives of the activation, P_l = dE/dZ_l and R_l = dE/dA_l from the backward
// kernel, mlp_chain_kernel in its tangent mode computes for a tile of 128 atoms of one element
//   T1 = U W1,  A1' = D1 T1,  T2 = A1' W2,  A2' = D2 T2,  T3 = A2' W3,  A3' = D3 T3        (tangent, forward)
//   Q3 = S3 T3 w4,  Q2 = S2 T2 R2 + D2 (Q3 W3^T),  Q1 = S1 T1 R1 + D1 (Q2 W2^T)            (reverse)
// and the weight gradients are U^T P1 + F^T Q1, A1'^T P2 + A1^T Q2, A2'^T P3 + A2^T Q3, sum A3' and the
// column sums of the Q_l (two passes of the weight-gradient kernel).
// This replaced 750 launches of dense torch ops per batch (9.5 ms for 256 molecules, almost all of it host time).
#pragma once

#include "ani_mlp_chain.cuh"

namespace ani {

// celu's second derivative jumps from 10 to 0 where the pre-activation changes its sign, so the sign of a value
// within rounding of 0 decides about a whole term.  The signs therefore come from pre-activations in plain
// float32 products, not from the three tf32 products of the forward kernel.
//
// One CTA takes 32 atoms of an element through the three hidden layers: their features stay in shared memory, the weights
// come in chunks of 32 rows through two stages, a thread has 4 x 4 outputs (2 x 4 in layer 3), the rows of a warp are the
// same for all its lanes.  A pre-activation is one chain of fused multiply-adds in float32 over k = 0, 1, 2 ..., from 0, and
// the bias added to its result: the same bits whatever the batch.  (Sums of 32 products added up would be closer to
// float64, but every sign that another order changes moves single gradients by a thousandth of their rms.)  It runs beside the first-order pass, whose network kernels fill a fifth of the device for 256
// molecules.  Before, these were twelve library GEMMs and twelve launches of bias and activation, issued by four threads:
// 90 us of host time and 60 us at the end of the chain in a batch of 256 molecules, now one launch of 33 us beside the
// networks: four such batches 990 -> 783 us.
constexpr int kCeluRows = 32, kCeluThreads = 256;
struct CeluPreParams {
    const float* feat;              // [atoms][384], element-sorted
    const float* w[3][kTypes];
    const float* bias[3][kTypes];
    float* z[3];                    // [atoms][128], [128], [64]
    int count[kTypes], row_start[kTypes];
    int tile_start[kTypes + 1];     // prefix of ceil(count / 32)
    bool aligned;                   // weights and features take 16-byte copies
};
struct CeluPreShared {
    static constexpr int kLdF = kMlpIn + 4, kLdH = kMlpH1 + 4;
    alignas(16) float x[kCeluRows * kLdF];           // the features, later A2
    alignas(16) float h[kCeluRows * kLdH];           // A1
    alignas(16) float w[2][32 * kMlpH1];
};

// `floats` (a multiple of 4 * kCeluThreads) consecutive floats.
__device__ __forceinline__ void celu_copy(float* dst, const float* src, int floats, bool aligned)
{
    if (aligned) {
        for (int i = threadIdx.x * 4; i < floats; i += kCeluThreads * 4)
            asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(smem_u32(dst + i)), "l"(src + i) : "memory");
    } else {
        for (int i = threadIdx.x; i < floats; i += kCeluThreads)
            asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(smem_u32(dst + i)), "l"(src + i) : "memory");
    }
}

// One layer: out[row][col] of rows R ty .., columns 4 tx .. from a [32][lda] and w [K][N].  The first chunk of w has been
// requested; `next` (or null): the next layer's first chunk, `next_floats` long, requested before the last product.
template <int K, int N, int R>
__device__ __forceinline__ void celu_layer(CeluPreShared& sh, const float* a, int lda, const float* w, const float* next,
                                           int next_floats, bool aligned, int* stage, float (&sum)[R][4])
{
    constexpr int kChunks = K / 32;
    const int tx = threadIdx.x % (N / 4), ty = threadIdx.x / (N / 4);
#pragma unroll
    for (int r = 0; r < R; r++)
#pragma unroll
        for (int q = 0; q < 4; q++) sum[r][q] = 0.0f;
    const float* rows = a + R * ty * lda;
#pragma unroll 1
    for (int c = 0; c < kChunks; c++) {
        const float* b = sh.w[*stage] + 4 * tx;
        *stage ^= 1;
        if (c + 1 < kChunks) celu_copy(sh.w[*stage], w + (size_t)(c + 1) * 32 * N, 32 * N, aligned);
        else if (next) celu_copy(sh.w[*stage], next, next_floats, aligned);
        asm volatile("cp.async.commit_group;" ::: "memory");
        asm volatile("cp.async.wait_group 1;" ::: "memory");
        __syncthreads();
#pragma unroll
        for (int k = 0; k < 32; k += 4) {
            float v[R][4];
#pragma unroll
            for (int r = 0; r < R; r++) load4(rows + r * lda + c * 32 + k, v[r]);
#pragma unroll
            for (int i = 0; i < 4; i++) {
                const float4 q = *reinterpret_cast<const float4*>(b + (k + i) * N);
#pragma unroll
                for (int r = 0; r < R; r++) {
                    sum[r][0] = fmaf(v[r][i], q.x, sum[r][0]);
                    sum[r][1] = fmaf(v[r][i], q.y, sum[r][1]);
                    sum[r][2] = fmaf(v[r][i], q.z, sum[r][2]);
                    sum[r][3] = fmaf(v[r][i], q.w, sum[r][3]);
                }
            }
        }
        __syncthreads();      // the stage is free again
    }
}

__global__ void __launch_bounds__(kCeluThreads, 2) celu_preactivations_kernel(const CeluPreParams p)
{
    extern __shared__ __align__(16) unsigned char celu_smem_raw[];
    CeluPreShared& sh = *reinterpret_cast<CeluPreShared*>(celu_smem_raw);
    int e = 0;
#pragma unroll
    for (int t = 1; t < kTypes; t++) e += (int)blockIdx.x >= p.tile_start[t] ? 1 : 0;
    const int row_in = ((int)blockIdx.x - p.tile_start[e]) * kCeluRows;
    const int n_rows = min(kCeluRows, p.count[e] - row_in);
    const size_t row0 = (size_t)p.row_start[e] + row_in;
    int stage = 0;
    pdl_wait();
    celu_copy(sh.w[0], p.w[0][e], 32 * kMlpH1, p.aligned);
    for (int i = threadIdx.x; i < kCeluRows * (kMlpIn / 4); i += kCeluThreads) {
        const int r = i / (kMlpIn / 4), k = 4 * (i - r * (kMlpIn / 4));
        float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
        if (r < n_rows) {
            const float* s = p.feat + (row0 + r) * kMlpIn + k;
            v = p.aligned ? *reinterpret_cast<const float4*>(s) : make_float4(s[0], s[1], s[2], s[3]);
        }
        *reinterpret_cast<float4*>(sh.x + r * CeluPreShared::kLdF + k) = v;
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
    // z = sum + bias to global memory (rows past the end are not written), celu(z) to the next layer's operand
    auto finish = [&](auto& sum, int layer, int width, float* out) {
        constexpr int R = sizeof(sum) / sizeof(sum[0]);
        const int tx = threadIdx.x % (width / 4), ty = threadIdx.x / (width / 4);
        const float* b = p.bias[layer][e] + 4 * tx;
        const float b0 = b[0], b1 = b[1], b2 = b[2], b3 = b[3];
#pragma unroll
        for (int r = 0; r < R; r++) {
            const int row = R * ty + r;
            const float4 z = make_float4(sum[r][0] + b0, sum[r][1] + b1, sum[r][2] + b2, sum[r][3] + b3);
            if (row < n_rows) *reinterpret_cast<float4*>(p.z[layer] + (row0 + row) * width + 4 * tx) = z;
            if (out)
                *reinterpret_cast<float4*>(out + row * CeluPreShared::kLdH + 4 * tx) =
                    make_float4(mlp_activation<kActCelu>(z.x), mlp_activation<kActCelu>(z.y), mlp_activation<kActCelu>(z.z),
                                mlp_activation<kActCelu>(z.w));
        }
    };
    float s4[4][4], s2[2][4];
    celu_layer<kMlpIn, kMlpH1, 4>(sh, sh.x, CeluPreShared::kLdF, p.w[0][e], p.w[1][e], 32 * kMlpH2, p.aligned, &stage, s4);
    finish(s4, 0, kMlpH1, sh.h);
    celu_layer<kMlpH1, kMlpH2, 4>(sh, sh.h, CeluPreShared::kLdH, p.w[1][e], p.w[2][e], 32 * kMlpH3, p.aligned, &stage, s4);
    finish(s4, 1, kMlpH2, sh.x);
    celu_layer<kMlpH2, kMlpH3, 2>(sh, sh.x, CeluPreShared::kLdH, p.w[2][e], nullptr, 0, p.aligned, &stage, s2);
    finish(s2, 2, kMlpH3, nullptr);
}

// Between two dense layers that somebody else computes: z += bias of the row's element, a = celu(z).  rows x width values,
// 4 per thread.
struct BiasCeluParams {
    float* z;
    float* a;                       // or null: last layer
    const float* bias[kTypes];
    int row_end[kTypes];            // rows of elements 0 .. t end here
    int rows, width;                // width: a multiple of 4
};
__global__ void __launch_bounds__(256) bias_celu_kernel(const BiasCeluParams p)
{
    pdl_wait();
    pdl_trigger();
    const int i = blockIdx.x * 256 + threadIdx.x;
    const int per_row = p.width >> 2;
    const int row = i / per_row, c = (i - row * per_row) * 4;
    if (row >= p.rows) return;
    const int e = (row >= p.row_end[0]) + (row >= p.row_end[1]) + (row >= p.row_end[2]);
    const float4 b = *reinterpret_cast<const float4*>(p.bias[e] + c);
    float4* zp = reinterpret_cast<float4*>(p.z + (size_t)row * p.width + c);
    float4 z = *zp;
    z.x += b.x; z.y += b.y; z.z += b.z; z.w += b.w;
    *zp = z;
    if (p.a)
        *reinterpret_cast<float4*>(p.a + (size_t)row * p.width + c) =
            make_float4(mlp_activation<kActCelu>(z.x), mlp_activation<kActCelu>(z.y), mlp_activation<kActCelu>(z.z),
                        mlp_activation<kActCelu>(z.w));
}

// ---- the loss: exp(sum over the axes of the rmse between the forces and their targets), as the reference's
// train_op_forces (khan/training/trainer_multi_tower.py:377-399) ----
constexpr int kForceLossThreads = 256;
constexpr int kForceLossBlocks = 64;

// Squared differences per axis, one partial sum per block; grid = kForceLossBlocks.
__global__ void __launch_bounds__(kForceLossThreads)
    force_residual_kernel(const float* __restrict__ gx, const float* __restrict__ gy, const float* __restrict__ gz,
                          const float* __restrict__ fx, const float* __restrict__ fy, const float* __restrict__ fz, int n,
                          double* __restrict__ partial)
{
    __shared__ double red[kForceLossThreads / kWarp][3];
    pdl_wait();
    pdl_trigger();
    double s[3] = {0.0, 0.0, 0.0};
    for (int i = blockIdx.x * kForceLossThreads + threadIdx.x; i < n; i += gridDim.x * kForceLossThreads) {
        const float a = gx[i] + fx[i], b = gy[i] + fy[i], c = gz[i] + fz[i];      // -(force - target)
        s[0] += (double)(a * a); s[1] += (double)(b * b); s[2] += (double)(c * c);
    }
#pragma unroll
    for (int k = 0; k < 3; k++) {
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) s[k] += __shfl_xor_sync(kFull, s[k], o);
        if (lane_id() == 0) red[warp_id()][k] = s[k];
    }
    __syncthreads();
    if (threadIdx.x < 3) {
        double t = 0.0;
        for (int w = 0; w < kForceLossThreads / kWarp; w++) t += red[w][threadIdx.x];
        partial[blockIdx.x * 3 + threadIdx.x] = t;       // summed in block order below: reproducible
    }
}

// v = dLoss/d(coordinate gradient); *rmse = sum of the three rmses.  Every block sums the partial sums itself.
__global__ void __launch_bounds__(kForceLossThreads)
    force_loss_kernel(const float* __restrict__ gx, const float* __restrict__ gy, const float* __restrict__ gz,
                      const float* __restrict__ fx, const float* __restrict__ fy, const float* __restrict__ fz, int n,
                      const double* __restrict__ partial, float* __restrict__ vx, float* __restrict__ vy,
                      float* __restrict__ vz, float* __restrict__ rmse)
{
    __shared__ double per_axis[3];
    pdl_wait();
    pdl_trigger();
    if (threadIdx.x < 3) {
        double t = 0.0;
        for (int b = 0; b < kForceLossBlocks; b++) t += partial[b * 3 + threadIdx.x];
        per_axis[threadIdx.x] = sqrt(t / (double)n);
    }
    __syncthreads();
    const double total = per_axis[0] + per_axis[1] + per_axis[2];
    if (blockIdx.x == 0 && threadIdx.x == 0) *rmse = (float)total;
    float f[3];
#pragma unroll
    for (int k = 0; k < 3; k++) f[k] = (float)(exp(total) / ((double)n * fmax(per_axis[k], 1e-300)));
    for (int i = blockIdx.x * kForceLossThreads + threadIdx.x; i < n; i += gridDim.x * kForceLossThreads) {
        vx[i] = f[0] * (gx[i] + fx[i]);
        vy[i] = f[1] * (gy[i] + fy[i]);
        vz[i] = f[2] * (gz[i] + fz[i]);
    }
}

}  // namespace ani
