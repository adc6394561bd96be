// Second-order pass of force training through the atomic networks, one kernel on the tensor cores.
//
// Force training minimises a function of the coordinate gradients x = J^T (dE/dF).  With v = dLoss/dx and
// u = J v (the directional derivative of the features along v), the derivative of the loss with respect to
// the weights is that of the scalar sum over atoms of <u, dE/dF>, i.e. of the forward-mode derivative of E
// along u -- the mixed product that the reference leaves to tf.gradients of tf.gradients
// (khan/training/trainer_multi_tower.py:377-399).  With T_l the tangents of the pre-activations, D_l and
// S_l the first and second derivatives of the activation, P_l = dE/dZ_l and R_l = dE/dA_l from the backward
// kernel, a CTA computes for its tile of 128 atoms of one element
//   T1 = U W1,  A1' = D1 T1,  T2 = A1' W2,  A2' = D2 T2,  T3 = A2' W3,  A3' = D3 T3        (tangent, forward)
//   Q3 = S3 T3 w4,  Q2 = S2 T2 R2 + D2 (Q3 W3^T),  Q1 = S1 T1 R1 + D1 (Q2 W2^T)            (reverse)
// and the weight gradients are U^T P1 + F^T Q1, A1'^T P2 + A1^T Q2, A2'^T P3 + A2^T Q3, sum A3' and the
// column sums of the Q_l (two passes of the weight-gradient kernel).
// Five products of the machinery of ani_mlp_pipe.cuh; what it replaced was 750 launches of dense torch ops per
// batch (9.5 ms for 256 molecules, almost all of it host time; 0.34 ms now).
#pragma once

#include "ani_mlp_pipe.cuh"

namespace ani {

struct MlpTangentParams {
    int count[kTypes];
    int tile_start[kTypes + 1];
    const float* u[kTypes];          // [count][384]
    const float* w4[kTypes];         // [64]
    const float *act1[kTypes], *act2[kTypes], *act3[kTypes];       // activations, [count][128], [128], [64] (celu: or
                                                                   // pre-activations, only the sign is used)
    const float *dact1[kTypes], *dact2[kTypes], *dact3[kTypes];    // their derivatives
    const float *r1[kTypes], *r2[kTypes];                          // dE/dA_l of the backward kernel
    float *adot1[kTypes], *adot2[kTypes], *adot3[kTypes];
    float *q1[kTypes], *q2[kTypes], *q3[kTypes];
    const unsigned char* packed[kTypes];
};

// Second derivative of the activation from the activation a and its first derivative d.
template <int ACT> __device__ __forceinline__ float mlp_activation_second(float a, float d)
{
    if (ACT == kActCelu) return a < 0.0f ? 10.0f * d : 0.0f;                       // exp(x / 0.1) / 0.1
    if (ACT == kActGaussian) return a > 0.0f ? d * d / a - 2.0f * a : 0.0f;        // (4 x^2 - 2) a, d = -2 x a
    if (ACT == kActNormal) return a > 0.0f ? d * d / a - a : 0.0f;                 // (x^2 - 1) a, d = -x a
    return d * (1.0f - d);
}

template <int ACT, bool SPLIT>
__global__ void __launch_bounds__(kMlpAllThreads, 1) mlp_tangent_kernel(const MlpTangentParams p)
{
    extern __shared__ unsigned char mlp_smem_raw[];
    MlpShared& sh = *reinterpret_cast<MlpShared*>(
        (reinterpret_cast<uintptr_t>(mlp_smem_raw) + 1023) & ~(uintptr_t)1023);
    const int tid = threadIdx.x, warp = tid >> 5;
    const int erow = (warp & 3) * 32 + (tid & 31), c0 = (warp >> 2) * 32;

    int e = 0;
#pragma unroll
    for (int t = 1; t < kTypes; t++) e += (int)blockIdx.x >= p.tile_start[t] ? 1 : 0;
    const int row0 = ((int)blockIdx.x - p.tile_start[e]) * kMlpTile;
    const int n_rows = min(kMlpTile, p.count[e] - row0);

    if (warp == 0) tmem_alloc(&sh.tmem_base, kMlpTmemCols);
    if (tid == 0) {
        mbar_init(&sh.stage_bar[0], 1);
        mbar_init(&sh.stage_bar[1], 1);
        mbar_init(&sh.full_bar[0], kMlpThreads);
        mbar_init(&sh.full_bar[1], kMlpThreads);
        sh.failed = 0;
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    pdl_wait();
    pdl_trigger();
    const unsigned tmem = sh.tmem_base;

    if (warp == kMlpThreads / 32) {
        IssueState is;
        pipe_issue<SPLIT>(sh, tmem, kMlpH1, kMlpIn / kPipeK, true, is);
        pipe_issue<SPLIT>(sh, tmem, kMlpH2, kMlpH1 / kPipeK, true, is);
        pipe_issue<SPLIT>(sh, tmem, kMlpH3, kMlpH2 / kPipeK, true, is);
        pipe_issue<SPLIT>(sh, tmem, kMlpH2, kMlpH3 / kPipeK, true, is);
        pipe_issue<SPLIT>(sh, tmem, kMlpH1, kMlpH2 / kPipeK, true, is);
    } else {
        PipeState ps;
        const DirectShared<SPLIT> a_sh{sh.act};
        DirectGlobal<SPLIT> a_u{p.u[e] + (size_t)row0 * kMlpIn, (size_t)kMlpIn, kMlpTile, n_rows, 0};
        const int tile_row0 = (warp & 3) * 32, tile_rows = n_rows - tile_row0;
        const unsigned lane_addr = tmem + ((unsigned)tile_row0 << 16);
        const size_t atom0 = (size_t)(row0 + tile_row0);
        float* scratch = warp_scratch(sh);
        const float* step_a[3] = {p.act1[e], p.act2[e], p.act3[e]};
        const float* step_d[3] = {p.dact1[e], p.dact2[e], p.dact3[e]};
        const float* step_r[2] = {p.r1[e], p.r2[e]};
        float* step_adot[3] = {p.adot1[e], p.adot2[e], p.adot3[e]};
        float* step_q[3] = {p.q1[e], p.q2[e], p.q3[e]};
        if (tid < kMlpH3) sh.vec[tid] = p.w4[e][tid];      // read after the first drain barrier
        bool ok = true;

        // ---- tangent, forward ----
#pragma unroll 1
        for (int l = 0; l < 3 && ok; l++) {
            const int N = l == 2 ? kMlpH3 : 128;
            const int first = l == 0 ? kPackFwdL1 : (l == 1 ? kPackFwdL2 : kPackFwdL3);
            PackedB b{p.packed[e] + (size_t)first * kPackedChunkBytes};
            if (l == 0) pipe_produce<SPLIT, false>(sh, kMlpIn / kPipeK, ps, a_u, a_sh, b);
            else pipe_produce<SPLIT, true>(sh, kMlpH1 / kPipeK, ps, a_u, a_sh, b);
            ok = pipe_drain(sh, ps);
            if (!ok) break;
            if (c0 < N) {
                const size_t g0 = atom0 * N + c0;
                float t[32], d[32], s[32];
                warp_tile_from_global(scratch, s, step_a[l] + g0, N, tile_rows);
                warp_tile_from_global(scratch, d, step_d[l] + g0, N, tile_rows);
#pragma unroll
                for (int i = 0; i < 32; i++) s[i] = mlp_activation_second<ACT>(s[i], d[i]);
                if (l < 2) {
                    warp_tile_from_global(scratch, t, step_r[l] + g0, N, tile_rows);
#pragma unroll
                    for (int i = 0; i < 32; i++) s[i] *= t[i];
                } else {
#pragma unroll
                    for (int i = 0; i < 32; i++) s[i] *= sh.vec[c0 + i];
                }
                tmem_load32(lane_addr + c0, t);
#pragma unroll
                for (int i = 0; i < 32; i++) {
                    s[i] *= t[i];                  // S T R: what Q gets from this layer itself
                    d[i] *= t[i];                  // A'
                    sh.act[erow * kMlpActStride + c0 + i] = l < 2 ? d[i] : s[i];     // the next product's A operand
                }
                warp_tile_to_global<false>(scratch, d, step_adot[l] + g0, N, tile_rows);
                warp_tile_to_global<false>(scratch, s, step_q[l] + g0, N, tile_rows);
            }
            tc_fence_before();
            producer_sync();
        }
        // ---- reverse ----
#pragma unroll 1
        for (int l = 1; l >= 0 && ok; l--) {
            PackedB b{p.packed[e] + (size_t)(l == 1 ? kPackBwdS0 : kPackBwdS1) * kPackedChunkBytes};
            pipe_produce<SPLIT, true>(sh, (l == 1 ? kMlpH3 : kMlpH2) / kPipeK, ps, a_u, a_sh, b);
            ok = pipe_drain(sh, ps);
            if (!ok) break;
            const size_t g0 = atom0 * 128 + c0;
            float t[32], d[32], s[32];
            warp_tile_from_global(scratch, d, step_d[l] + g0, 128, tile_rows);
            warp_tile_from_global(scratch, s, step_q[l] + g0, 128, tile_rows);     // written by this warp above
            tmem_load32(lane_addr + c0, t);
#pragma unroll
            for (int i = 0; i < 32; i++) {
                s[i] += d[i] * t[i];
                sh.act[erow * kMlpActStride + c0 + i] = s[i];
            }
            warp_tile_to_global<false>(scratch, s, step_q[l] + g0, 128, tile_rows);
            tc_fence_before();
            producer_sync();
        }
        if (!ok && tid == 0) report(ANI_ERR_TIMEOUT);
    }
    __syncthreads();
    if (warp == 0) tmem_dealloc(tmem, kMlpTmemCols);
}

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
