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
// float32 products (ForceFitStep forms them with library GEMMs, as the differentiable path does), not from the
// three tf32 products of the forward kernel.  This kernel is what lies between two of those GEMMs: z += bias
// of the row's element, a = celu(z).  rows x width values, 4 per thread.
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
