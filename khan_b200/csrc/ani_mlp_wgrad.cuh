// Weight and bias gradients of the per-element atomic networks on the Blackwell tensor cores:
//   dW1 = F^T dZ1 [384 x 128],  dW2 = A1^T dZ2 [128 x 128],  dW3 = A2^T dZ3 [128 x 64],
//   db_l = column sums of dZ_l,
// products whose long dimension is the ATOM index.  A CTA takes one range of atoms (sized on the
// host so that the whole grid is one wave) of one element and one 128-row block of one weight matrix
// (three blocks for W1, one each for W2 and W3), accumulates its [128 x N] block in tensor memory
// over the range, and adds it to the output with 16-byte global reductions (the call ADDS to its
// outputs).  The CTA of the W3 block also does the output layer (dw4 = A3^T g, db4 = sum g).
//
// K is the atom, so both operands are transposes of what is in memory, and getting them transposed is what the
// kernel spends its time on: 32 atoms are 0.43 us of the tensor core.  A thread takes one COLUMN (a feature or
// activation for A, an output for B) of 32 atoms, one coalesced 128-byte load per warp and atom.  For A that is a
// row of the operand already: it goes to tensor memory (lane = column of the matrix, 32 TMEM columns = 32 atoms)
// without touching shared memory.  For B four consecutive atoms are one 16-byte piece of the K-major layout.  Four
// groups of four warps take the chunks in turn, so that four chunks' loads are in flight.  (Loading 16 bytes along
// the row and scattering them to four operand rows with 4-byte stores, one chunk ahead: 3.2 us a chunk, 52 us for
// 14 k atoms.)
//
// Same mathematics as the weight part of tf.gradients through AtomNN (khan/model/nn.py:39-67
// under khan/training/trainer_multi_tower.py:396-397).
#pragma once

#include "ani_mlp_chain.cuh"

namespace ani {

constexpr int kWgradBlocks = 5;    // W1 rows 0-127, 128-255, 256-383; W2; W3 (+ the output layer w4, b4)
constexpr int kWgradMaxSets = 2;

struct MlpWgradParams {
    const float* feat[kTypes];     // [count][384]
    const float* act1[kTypes];     // [count][128]
    const float* act2[kTypes];     // [count][128]
    const float* dz1[kTypes];      // [count][128]
    const float* dz2[kTypes];      // [count][128]
    const float* dz3[kTypes];      // [count][64]
    float* dw1[kTypes];            // [384][128]
    float* dw2[kTypes];            // [128][128]
    float* dw3[kTypes];            // [128][64]
    float* db1[kTypes];            // [128] or null, as db2, db3
    float* db2[kTypes];            // [128]
    float* db3[kTypes];            // [64]
    const float* act3[kTypes];     // [count][64]
    const float* grad_energy[kTypes];   // [count], or null: ones
    float* dw4[kTypes];            // [64], or null: no output layer
    float* db4[kTypes];            // [1] or null
};
// One launch for up to two sets of operands over the same atoms (force training has two).
struct MlpWgradSets {
    int count[kTypes];
    int range;                     // atoms per CTA, a multiple of 32
    int range_start[kTypes + 1];   // prefix of ceil(count / range)
    MlpWgradParams set[kWgradMaxSets];
};

struct WgradShared {
    alignas(1024) unsigned char b[kChainGroups][2 * kPipeOperandBytes];
    alignas(8) unsigned long long full[kChainGroups], empty[kChainGroups], done;
    unsigned tmem_base;
    int failed;
};

// Columns col (A, row stride LDA) and `me` (B, row stride N; threads >= N have none) of 32 atoms; atoms >= valid are
// zero.
template <int LDA, int N>
__device__ __forceinline__ void wgrad_load(const float* a, const float* b, int me, int valid, float* va, float* vb)
{
    if (valid >= kPipeK) {
#pragma unroll
        for (int k = 0; k < kPipeK; k++) va[k] = a[(size_t)k * LDA];
#pragma unroll
        for (int k = 0; k < kPipeK; k++) vb[k] = me < N ? b[(size_t)k * N] : 0.0f;
    } else {
#pragma unroll
        for (int k = 0; k < kPipeK; k++) va[k] = k < valid ? a[(size_t)k * LDA] : 0.0f;
#pragma unroll
        for (int k = 0; k < kPipeK; k++) vb[k] = k < valid && me < N ? b[(size_t)k * N] : 0.0f;
    }
}

template <bool SPLIT>
__global__ void __launch_bounds__(kMlpAllThreads, 1) mlp_wgrad_kernel(const MlpWgradSets sets)
{
    extern __shared__ __align__(1024) unsigned char wgrad_smem_raw[];
    WgradShared& sh = *reinterpret_cast<WgradShared*>(wgrad_smem_raw);
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const MlpWgradParams& p = sets.set[blockIdx.z];

    int e = 0;
#pragma unroll
    for (int t = 1; t < kTypes; t++) e += (int)blockIdx.x >= sets.range_start[t] ? 1 : 0;
    const long long first = (long long)((int)blockIdx.x - sets.range_start[e]) * sets.range;
    const int n_here = (int)min((long long)sets.range, (long long)sets.count[e] - first);
    const int blk = blockIdx.y;
    const int N = blk == 4 ? kMlpH3 : 128;
    const int nchunks = (n_here + kPipeK - 1) / kPipeK;

    if (warp == kMlpThreads / 32) tmem_alloc(&sh.tmem_base, 512);
    if (tid == 0) {
        for (int g = 0; g < kChainGroups; g++) {
            mbar_init(&sh.full[g], kMlpThreads / kChainGroups);
            mbar_init(&sh.empty[g], 1);
        }
        mbar_init(&sh.done, 1);
        sh.failed = 0;
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    pdl_wait();
    pdl_trigger();
    const unsigned tmem = sh.tmem_base;

    if (warp == kMlpThreads / 32) {
        // ---- the products: one thread; barriers of the next chunk looked at between two instructions ----
        if (lane == 0) {
            bool ok = true;
            unsigned seen = 0;
            for (int c = 0; c < nchunks && ok; c++) {
                const int g = c % kChainGroups;
                if (!seen) ok = mbar_wait(&sh.full[g], (unsigned)(c / kChainGroups) & 1u);
                if (!ok) break;
                tc_fence_after();
                const unsigned idesc = instr_desc(kMlpTile, N);
                const unsigned b_hi = smem_u32(sh.b[g]), b_lo = b_hi + kPipeOperandBytes;
                const unsigned a_hi = tmem + kTmemHi + g * 2 * kPipeK, a_lo = a_hi + kPipeK;
                seen = 0;
#pragma unroll
                for (int ks = 0; ks < kPipeK / 8; ks++) {
                    const unsigned step = ks * 2 * kMlpLbo, col = ks * 8;
                    // (hi hi and hi lo as one instruction of 256 columns, as in mlp_chain_kernel, was slower here: 19.6 us)
                    mma_tf32_ts(tmem + kTmemAcc, a_hi + col, pipe_desc(b_hi + step), idesc, !(c == 0 && ks == 0));
                    if (SPLIT) {
                        mma_tf32_ts(tmem + kTmemSmall, a_hi + col, pipe_desc(b_lo + step), idesc, !(c == 0 && ks == 0));
                        mma_tf32_ts(tmem + kTmemSmall, a_lo + col, pipe_desc(b_hi + step), idesc, true);
                    }
                    if (ks == 1 && c + 1 < nchunks)
                        seen = mbar_test(&sh.full[(c + 1) % kChainGroups], (unsigned)((c + 1) / kChainGroups) & 1u);
                }
                mma_commit(&sh.empty[g]);
            }
            if (ok) mma_commit(&sh.done);
            else sh.failed = 1;
        }
    } else {
        // ---- staging: group g of 128 threads takes chunks g, g + 4, ... ----
        ChainWait wait;
        const int g = warp >> 2, me = tid & 127;
        const unsigned lanes = tmem + ((unsigned)((warp & 3) * 32) << 16);
        const float* a_src = blk < 3 ? p.feat[e] + blk * 128 : (blk == 3 ? p.act1[e] : p.act2[e]);
        const float* b_src = blk < 3 ? p.dz1[e] : (blk == 3 ? p.dz2[e] : p.dz3[e]);
        a_src += first * (blk < 3 ? kMlpIn : 128) + me;
        b_src += first * N + (me < N ? me : 0);
        float colsum = 0.0f;
        bool timed_out = false;
        for (int c = g, turn = 0; c < nchunks; c += kChainGroups, turn++) {
            float va[kPipeK], vb[kPipeK];
            const size_t k0 = (size_t)c * kPipeK;
            const int valid = n_here - c * kPipeK;
            if (blk < 3) wgrad_load<kMlpIn, 128>(a_src + k0 * kMlpIn, b_src + k0 * 128, me, valid, va, vb);
            else if (blk == 3) wgrad_load<128, 128>(a_src + k0 * 128, b_src + k0 * 128, me, valid, va, vb);
            else wgrad_load<128, kMlpH3>(a_src + k0 * 128, b_src + k0 * kMlpH3, me, valid, va, vb);
            if (turn > 0 && !timed_out) {
                timed_out = !mbar_wait(&sh.empty[g], (unsigned)(turn - 1) & 1u);
                if (timed_out) sh.failed = 1;
                tc_fence_after();
            }
            if (me < N) {
#pragma unroll
                for (int k = 0; k < kPipeK; k += 4) {
                    colsum += (vb[k] + vb[k + 1]) + (vb[k + 2] + vb[k + 3]);
                    pipe_store4<SPLIT>(sh.b[g], sh.b[g] + kPipeOperandBytes, pipe_offset(me, k),
                                       make_float4(vb[k], vb[k + 1], vb[k + 2], vb[k + 3]));
                }
            }
            fence_async_smem();
            float part[kPipeK];
#pragma unroll
            for (int k = 0; k < kPipeK; k++) part[k] = tf32_round(va[k]);
            tmem_store32(lanes + kTmemHi + g * 2 * kPipeK, part);
            if (SPLIT) {
#pragma unroll
                for (int k = 0; k < kPipeK; k++) part[k] = va[k] - part[k];
                tmem_store32(lanes + kTmemHi + g * 2 * kPipeK + kPipeK, part);
            }
            tmem_store_wait();
            tc_fence_before();
            mbar_arrive(&sh.full[g]);
        }
        if (blk == 4 && p.dw4[e]) {
            // output layer, done by the CTA with the lightest product while that comes to its end: dw4 = A3^T g and
            // db4 = sum g over this range; no tensor cores involved.  Eight atoms' loads at once: one behind the other,
            // and behind the product, they made the kernel 21.8 us long for 1024 molecules instead of 18.9.
            const int q = tid & 15, a_in = tid >> 4;      // 16 column quads x 32 atoms per pass
            const float* act = p.act3[e] + (size_t)first * kMlpH3 + 4 * q;
            const float* up = p.grad_energy[e] ? p.grad_energy[e] + first : nullptr;
            float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
            float gsum = 0.0f;
            constexpr int kStep = kMlpThreads / 16;
            for (int k0 = a_in; k0 < n_here; k0 += 8 * kStep) {
                float4 v[8];
                float ge[8];
#pragma unroll
                for (int i = 0; i < 8; i++) {
                    const int k = k0 + i * kStep;
                    ge[i] = k < n_here ? (up ? up[k] : 1.0f) : 0.0f;
                    v[i] = k < n_here ? *reinterpret_cast<const float4*>(act + (size_t)k * kMlpH3) : make_float4(0.f, 0.f, 0.f, 0.f);
                }
#pragma unroll
                for (int i = 0; i < 8; i++) {
                    acc.x += v[i].x * ge[i]; acc.y += v[i].y * ge[i]; acc.z += v[i].z * ge[i]; acc.w += v[i].w * ge[i];
                    gsum += q == 0 ? ge[i] : 0.0f;
                }
            }
            // the two halves of a warp hold the same columns
            acc.x += __shfl_xor_sync(kFull, acc.x, 16);
            acc.y += __shfl_xor_sync(kFull, acc.y, 16);
            acc.z += __shfl_xor_sync(kFull, acc.z, 16);
            acc.w += __shfl_xor_sync(kFull, acc.w, 16);
            gsum += __shfl_xor_sync(kFull, gsum, 16);
            if (lane < 16) {
                atomicAdd(p.dw4[e] + 4 * q + 0, acc.x);
                atomicAdd(p.dw4[e] + 4 * q + 1, acc.y);
                atomicAdd(p.dw4[e] + 4 * q + 2, acc.z);
                atomicAdd(p.dw4[e] + 4 * q + 3, acc.w);
                if (q == 0 && p.db4[e]) atomicAdd(p.db4[e], gsum);
            }
        }
        bool ok = n_here > 0 && !timed_out;
        if (ok && !mbar_wait(&sh.done, 0u)) {
            ok = false;
            sh.failed = 1;
        }
        tc_fence_after();
        producer_sync();      // the operand stages become transposition scratch
        if (ok && !sh.failed) {
            // warp w: rows 32 (w % 4) .. of the weight block (TMEM lanes), columns 32 (w / 4) ..
            const int tile_row0 = (warp & 3) * 32, c0 = (warp >> 2) * 32;
            float* out = blk < 3 ? p.dw1[e] + (size_t)blk * 128 * 128 : (blk == 3 ? p.dw2[e] : p.dw3[e]);
            float* bias_out = blk == 0 ? p.db1[e] : (blk == 3 ? p.db2[e] : (blk == 4 ? p.db3[e] : nullptr));
            if (c0 < N) {
                float v[32];
                tmem_load32(lanes + kTmemAcc + c0, v);
                if (SPLIT) {
                    float small[32];
                    tmem_load32(lanes + kTmemSmall + c0, small);
#pragma unroll
                    for (int i = 0; i < 32; i++) v[i] += small[i];
                }
                float* scratch = reinterpret_cast<float*>(sh.b[0]) + warp * (32 * kMlpScratchStride);
                warp_tile_to_global<true>(scratch, v, out + (size_t)tile_row0 * N + c0, N, 32);
            }
            if (bias_out && me < N && g < nchunks) atomicAdd(bias_out + me, colsum);
        }
    }
    tc_fence_before();
    __syncthreads();
    if (tid == 0 && sh.failed) report(ANI_ERR_TIMEOUT);
    tc_fence_after();
    if (warp == kMlpThreads / 32) tmem_dealloc(tmem, 512);
}

}  // namespace ani
