// Atomic networks 384-128-128-64-1 as ONE chain of products per tile of 128 atoms, on the tensor cores, with
// packed weights: forward, forward + backward to the features, backward alone, or the second-order pass of
// force training.
//
// Computes what ani_mlp_forward.cuh / ani_mlp_backward.cuh compute (AtomNN of the reference,
// khan/model/nn.py:39-67,165-172, and its gradient, khan/training/trainer_multi_tower.py:350-419); those remain
// for weights that are not packed.  The second-order pass is described in ani_force_fit.cuh.
//
// A tile is three products forward (K = 384, 128, 128) and five backward (K = 64, 128, 3 x 128), 38 chunks of 32
// values of K, each 0.4 us of the tensor core (three tf32 products).  The previous kernels took 1-2 us a chunk and
// 2-3 us between two products: two stages for both operands, weights requested by a thread that also stages
// activations and runs epilogues, and every activation through shared memory and back as the next A operand.  Here
//   * one thread streams the weights through a ring of four stages, ahead over the whole chain, also across
//     epilogues;
//   * every A operand is in tensor memory: an epilogue reads the accumulator, splits the new activations into
//     their tf32 parts and stores those to TMEM, where the next product takes them (columns: accumulator 0-127,
//     spare 128-255, A high 256-383, A low 384-511).  The shared memory's 128 bytes a clock are what a chunk is
//     short of: with both operands there, the products read 96 KB of it and staging wrote 64 KB, 1250 clocks
//     against the tensor core's 830; now the weights are 80 KB of it;
//   * the features of a chunk are copied to shared memory as they are (16 KB), four warps read them row by row and
//     store their parts to TMEM; four groups of four warps take the chunks in turn (four stages of 64 columns in
//     the place of the later A operands).
//   * forward + backward in one kernel needs nothing of the activations in global memory: the derivatives of
//     layer 1 wait in the spare columns, those of layer 2 where the feature stages were.
// TODO_CHAIN
// Split precision: x = hi + lo with hi rounded to nearest, hi hi + hi lo + lo hi accumulated.  Every wait is
// bounded; after a timeout the kernel reports, waits for its own copies, frees its tensor memory and returns.
#pragma once

#include "ani_mlp_pipe.cuh"

namespace ani {

constexpr int kChainA = 8, kChainB = 3;                 // feature chunks of 16 KB, weight stages of 32 KB (high, low)
constexpr int kChainEpi = 512;                          // epilogue / staging threads (16 warps)
constexpr int kChainThreads = kChainEpi + 64;           // + the MMA warp + the weight warp
constexpr int kChainGroups = 4;                         // groups of 128 threads that take the feature chunks in turn
constexpr unsigned kTmemAcc = 0, kTmemSpare = 128, kTmemHi = 256, kTmemLo = 384;

enum ChainMode { kChainForward = 0, kChainForces = 1, kChainBackward = 2, kChainTangent = 3 };

struct MlpChainParams {
    int count[kTypes];
    int tile_start[kTypes + 1];
    const unsigned char* packed[kTypes];
    const float* feat[kTypes];       // [count][384]          (forward; tangent: rates of the features)
    const float *b1[kTypes], *b2[kTypes], *b3[kTypes], *b4[kTypes];
    const float* w4[kTypes];         // [64]
    float* energy[kTypes];           // [count]
    float *act1[kTypes], *act2[kTypes], *act3[kTypes];      // optional (forward); read by the tangent mode (celu:
                                                            // or pre-activations there, only the sign is used)
    float *dact1[kTypes], *dact2[kTypes], *dact3[kTypes];   // optional; read by the backward and tangent modes
    const float* grad_energy[kTypes];   // [count], null: ones                          (forces, backward)
    float *dz1[kTypes], *dz2[kTypes], *dz3[kTypes];         //                          (backward)
    float *r1[kTypes], *r2[kTypes];  // optional: dL/dA of the inner layers (backward); read by the tangent mode
    float *adot1[kTypes], *adot2[kTypes], *adot3[kTypes];   // rates of the activations (tangent)
    float *q1[kTypes], *q2[kTypes], *q3[kTypes];            //                          (tangent)
    float* grad_feat[kTypes];        // [count][384]; optional in the backward mode
};

struct ChainShared {
    alignas(1024) unsigned char a[kChainA][kPipeOperandBytes];
    alignas(1024) unsigned char b[kChainB][2 * kPipeOperandBytes];
    float bias[kMlpH1 + kMlpH2 + kMlpH3], w4[kMlpH3];
    float epart[kMlpTile];
    alignas(8) unsigned long long a_full[kChainGroups], a_empty[kChainGroups], b_full[kChainB], b_empty[kChainB];
    unsigned long long acc_full[2];      // accumulator (0) / spare (1) holds a finished product
    unsigned long long operand_ready;    // the epilogue has stored the next A operand
    unsigned long long acc_free;         // the epilogue has read the accumulator
    unsigned tmem_base;
    int failed;
};
static_assert(sizeof(ChainShared) <= 227 * 1024, "one CTA per SM");

// A operand in tensor memory, B in shared memory.
__device__ __forceinline__ void mma_tf32_ts(unsigned d_tmem, unsigned a_tmem, unsigned long long b_desc, unsigned idesc,
                                            bool accumulate)
{
    asm volatile(
        "{\n"
        ".reg .pred p;\n"
        "setp.ne.u32 p, %4, 0;\n"
        "tcgen05.mma.cta_group::1.kind::tf32 [%0], [%1], %2, %3, {%5, %6, %7, %8}, p;\n"
        "}\n" ::"r"(d_tmem),
        "r"(a_tmem), "l"(b_desc), "r"(idesc), "r"((unsigned)accumulate), "r"(0u), "r"(0u), "r"(0u), "r"(0u)
        : "memory");
}
// 32 consecutive columns of this thread's row (TMEM lane); completion: tmem_store_wait().
__device__ __forceinline__ void tmem_store32(unsigned taddr, const float* v)
{
    asm volatile(
        "tcgen05.st.sync.aligned.32x32b.x32.b32 [%0], "
        "{%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16, "
        "%17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31, %32};" ::"r"(taddr),
        "f"(v[0]), "f"(v[1]), "f"(v[2]), "f"(v[3]), "f"(v[4]), "f"(v[5]), "f"(v[6]), "f"(v[7]), "f"(v[8]), "f"(v[9]),
        "f"(v[10]), "f"(v[11]), "f"(v[12]), "f"(v[13]), "f"(v[14]), "f"(v[15]), "f"(v[16]), "f"(v[17]), "f"(v[18]),
        "f"(v[19]), "f"(v[20]), "f"(v[21]), "f"(v[22]), "f"(v[23]), "f"(v[24]), "f"(v[25]), "f"(v[26]), "f"(v[27]),
        "f"(v[28]), "f"(v[29]), "f"(v[30]), "f"(v[31])
        : "memory");
}
__device__ __forceinline__ void tmem_store_wait() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }

// Barrier wait of one role: no wait after the first that ran out.
struct ChainWait {
    bool ok = true;
    __device__ __forceinline__ bool operator()(ChainShared& sh, unsigned long long* bar, unsigned parity)
    {
        if (ok && !mbar_wait(bar, parity)) {
            ok = false;
            sh.failed = 1;
        }
        return ok;
    }
};

// Second derivative of the activation from the activation a and its first derivative d.
template <int ACT> __device__ __forceinline__ float mlp_activation_second(float a, float d)
{
    if (ACT == kActCelu) return a < 0.0f ? 10.0f * d : 0.0f;                       // exp(x / 0.1) / 0.1
    if (ACT == kActGaussian) return a > 0.0f ? d * d / a - 2.0f * a : 0.0f;        // (4 x^2 - 2) a, d = -2 x a
    if (ACT == kActNormal) return a > 0.0f ? d * d / a - a : 0.0f;                 // (x^2 - 1) a, d = -x a
    return d * (1.0f - d);
}

template <int ACT, bool SPLIT, int MODE>
__global__ void __launch_bounds__(kChainThreads, 1) mlp_chain_kernel(const MlpChainParams p)
{
    extern __shared__ __align__(1024) unsigned char chain_smem_raw[];
    ChainShared& sh = *reinterpret_cast<ChainShared*>(chain_smem_raw);
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    constexpr bool kHasForward = MODE != kChainBackward, kHasBackward = MODE != kChainForward;

    int e = 0;
#pragma unroll
    for (int t = 1; t < kTypes; t++) e += (int)blockIdx.x >= p.tile_start[t] ? 1 : 0;
    const int row0 = ((int)blockIdx.x - p.tile_start[e]) * kMlpTile;
    const int n_rows = min(kMlpTile, p.count[e] - row0);
    const bool want_feat = kHasBackward && MODE != kChainTangent && p.grad_feat[e] != nullptr;

    if (warp == kChainEpi / 32) tmem_alloc(&sh.tmem_base, 512);
    if (tid == 0) {
        for (int s = 0; s < kChainGroups; s++) {
            mbar_init(&sh.a_full[s], kChainEpi / kChainGroups);
            mbar_init(&sh.a_empty[s], 1);
        }
        for (int s = 0; s < kChainB; s++) {
            mbar_init(&sh.b_full[s], 1);
            mbar_init(&sh.b_empty[s], 1);
        }
        mbar_init(&sh.acc_full[0], 1);
        mbar_init(&sh.acc_full[1], 1);
        mbar_init(&sh.operand_ready, kChainEpi);
        mbar_init(&sh.acc_free, kChainEpi);
        sh.failed = 0;
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    pdl_wait();
    pdl_trigger();
    const unsigned tmem = sh.tmem_base;
    // chunks of packed weights in the order of the chain
    const int n_chunks = (kHasForward ? 20 : 0) + (kHasBackward ? 6 + (want_feat ? 12 : 0) : 0);
    constexpr int kFirstChunk = kHasForward ? kPackFwdL1 : kPackBwdS0;   // the packed order is the chain's order

    if (warp == kChainEpi / 32 + 1) {
        // ---- the weights: one thread, a ring of kChainB stages ----
        if (lane == 0) {
            ChainWait wait;
            int filled = 0;
            for (int c = 0; c < n_chunks; c++, filled++) {
                const int s = c % kChainB;
                if (c >= kChainB && !wait(sh, &sh.b_empty[s], (unsigned)(c / kChainB - 1) & 1u)) break;
                const int chunk = kFirstChunk + c;
                const unsigned char* src = p.packed[e] + (size_t)chunk * kPackedChunkBytes;
                // layer 3 has 64 output columns: half of each part
                const unsigned bytes = chunk >= kPackFwdL3 && chunk < kPackBwdS0 ? kPipeOperandBytes / 2 : kPipeOperandBytes;
                // the one arrival that a phase takes comes with the byte count, before the copies
                asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(&sh.b_full[s])),
                             "r"(SPLIT ? 2 * bytes : bytes)
                             : "memory");
                bulk_copy_to_shared(sh.b[s], src, bytes, &sh.b_full[s]);
                if (SPLIT) bulk_copy_to_shared(sh.b[s] + kPipeOperandBytes, src + kPipeOperandBytes, bytes, &sh.b_full[s]);
            }
            // copies in flight land before the CTA may end (after a timeout nobody else waits for them)
            for (int c = filled > kChainB ? filled - kChainB : 0; c < filled; c++)
                mbar_wait(&sh.b_full[c % kChainB], (unsigned)(c / kChainB) & 1u);
        }
    } else if (warp == kChainEpi / 32) {
        // ---- the products ----
        ChainWait wait;
        int bc = 0, ready = 0;
        auto issue = [&](unsigned d, unsigned a_hi, unsigned a_lo, int s, int N, bool first) {
            const unsigned idesc = instr_desc(kMlpTile, N);
            const unsigned b_hi = smem_u32(sh.b[s]), b_lo = b_hi + kPipeOperandBytes;
#pragma unroll
            for (int ks = 0; ks < kPipeK / 8; ks++) {
                const unsigned step = ks * 2 * kMlpLbo, col = ks * 8;
                mma_tf32_ts(d, tmem + a_hi + col, pipe_desc(b_hi + step), idesc, !(first && ks == 0));
                if (SPLIT) {
                    mma_tf32_ts(d, tmem + a_hi + col, pipe_desc(b_lo + step), idesc, true);
                    mma_tf32_ts(d, tmem + a_lo + col, pipe_desc(b_hi + step), idesc, true);
                }
            }
        };
        // one product behind layer 1
        auto product = [&](unsigned d, int chunks, int N, unsigned long long* done) {
            for (int c = 0; c < chunks; c++, bc++) {
                const int s = bc % kChainB;
                if (wait(sh, &sh.b_full[s], (unsigned)(bc / kChainB) & 1u) && lane == 0) {
                    tc_fence_after();
                    issue(tmem + d, kTmemHi + c * kPipeK, kTmemLo + c * kPipeK, s, N, c == 0);
                    mma_commit(&sh.b_empty[s]);
                    if (c == chunks - 1) mma_commit(done);
                }
                __syncwarp();
            }
        };
        auto operand = [&]() {
            wait(sh, &sh.operand_ready, (unsigned)ready & 1u);
            ready++;
            tc_fence_after();
        };
        if (kHasForward) {
            for (int c = 0; c < kMlpIn / kPipeK; c++, bc++) {
                const int s = bc % kChainB, sa = c % kChainGroups;
                wait(sh, &sh.a_full[sa], (unsigned)(c / kChainGroups) & 1u);
                if (wait(sh, &sh.b_full[s], (unsigned)(bc / kChainB) & 1u) && lane == 0) {
                    tc_fence_after();
                    issue(tmem + kTmemAcc, kTmemHi + sa * 2 * kPipeK, kTmemHi + sa * 2 * kPipeK + kPipeK, s, kMlpH1, c == 0);
                    mma_commit(&sh.b_empty[s]);
                    mma_commit(&sh.a_empty[sa]);
                    if (c == kMlpIn / kPipeK - 1) mma_commit(&sh.acc_full[0]);
                }
                __syncwarp();
            }
            operand();
            product(kTmemAcc, kMlpH1 / kPipeK, kMlpH2, &sh.acc_full[0]);
            operand();
            product(kTmemAcc, kMlpH2 / kPipeK, kMlpH3, &sh.acc_full[0]);
        }
        if (kHasBackward) {
            operand();
            product(kTmemAcc, kMlpH3 / kPipeK, kMlpH2, &sh.acc_full[0]);
            operand();
            product(kTmemAcc, kMlpH2 / kPipeK, kMlpH1, &sh.acc_full[0]);
            if (want_feat) {
                operand();
                product(kTmemAcc, kMlpH1 / kPipeK, 128, &sh.acc_full[0]);
                product(kTmemSpare, kMlpH1 / kPipeK, 128, &sh.acc_full[1]);
                wait(sh, &sh.acc_free, 0u);
                tc_fence_after();
                product(kTmemAcc, kMlpH1 / kPipeK, 128, &sh.acc_full[0]);
            }
        }
    } else {
        // ---- feature staging and epilogues: warp w has rows 32 (w % 4) .. and columns 32 (w / 4) .. ----
        ChainWait wait;
        const int c0 = (warp >> 2) * 32, tile_row0 = (warp & 3) * 32, row = tile_row0 + lane;
        const int tile_rows = n_rows - tile_row0;
        const size_t atom0 = (size_t)(row0 + tile_row0);
        const unsigned lanes = tmem + ((unsigned)tile_row0 << 16);
        // per-warp 32 x 33 transposition scratch over the feature stages (idle outside layer 1)
        float* scratch = reinterpret_cast<float*>(sh.a[0]) + warp * (32 * kMlpScratchStride);
        float* hold2 = reinterpret_cast<float*>(sh.a[0]);      // forces mode: derivatives of layer 2, [128][128 rows]
        int acc_phase = 0;
        auto to_operand = [&](const float* v) {      // the next A operand: 32 columns of this thread's row
            float part[32];
#pragma unroll
            for (int i = 0; i < 32; i++) part[i] = tf32_round(v[i]);
            tmem_store32(lanes + kTmemHi + c0, part);
            if (SPLIT) {
#pragma unroll
                for (int i = 0; i < 32; i++) part[i] = v[i] - part[i];
                tmem_store32(lanes + kTmemLo + c0, part);
            }
        };
        auto operand_done = [&]() {
            tmem_store_wait();
            tc_fence_before();
            mbar_arrive(&sh.operand_ready);
        };
        auto accumulator = [&]() {
            wait(sh, &sh.acc_full[0], (unsigned)acc_phase & 1u);
            acc_phase++;
            tc_fence_after();
        };

        if (kHasForward && MODE != kChainTangent) {
            if (tid < kMlpH1) sh.bias[tid] = p.b1[e][tid];
            else if (tid < kMlpH1 + kMlpH2) sh.bias[tid] = p.b2[e][tid - kMlpH1];
            else if (tid < kMlpH1 + kMlpH2 + kMlpH3) sh.bias[tid] = p.b3[e][tid - kMlpH1 - kMlpH2];
        }
        if (tid >= kChainEpi - kMlpH3) sh.w4[tid - (kChainEpi - kMlpH3)] = p.w4[e][tid - (kChainEpi - kMlpH3)];
        producer_sync();

        if (kHasForward) {
            // ---- layer 1: group g of 128 threads takes chunks g, g + 4, g + 8; thread = row (TMEM lane) ----
            const int g = warp >> 2, me = tid & 127;
            const float* feat = p.feat[e] + (size_t)row0 * kMlpIn;
            auto request = [&](int j) {      // 16-byte pieces, piece q of row r at place q ^ (r mod 8): no bank conflicts
                unsigned char* dst = sh.a[g * 2 + (j & 1)];
                const float* src = feat + (g + 4 * j) * kPipeK;
#pragma unroll
                for (int i = 0; i < 8; i++) {
                    const int rr = i * 16 + (me >> 3), q = me & 7;
                    const unsigned bytes = rr < n_rows ? 16u : 0u;      // rows past the end become zeros
                    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(
                                     smem_u32(dst + rr * 128 + ((q ^ (rr & 7)) << 4))),
                                 "l"(src + (size_t)(rr < n_rows ? rr : 0) * kMlpIn + q * 4), "r"(bytes)
                                 : "memory");
                }
                asm volatile("cp.async.commit_group;" ::: "memory");
            };
            request(0);
            request(1);
#pragma unroll
            for (int j = 0; j < 3; j++) {
                if (j < 2) asm volatile("cp.async.wait_group 1;" ::: "memory");
                else asm volatile("cp.async.wait_group 0;" ::: "memory");
                asm volatile("bar.sync %0, 128;" ::"r"(3 + g) : "memory");
                float v[32];
                const unsigned char* src = sh.a[g * 2 + (j & 1)] + me * 128;
#pragma unroll
                for (int q = 0; q < 8; q++) {
                    const float4 x = *reinterpret_cast<const float4*>(src + ((q ^ (me & 7)) << 4));
                    v[4 * q] = x.x; v[4 * q + 1] = x.y; v[4 * q + 2] = x.z; v[4 * q + 3] = x.w;
                }
                if (j == 0) {      // the buffer has been read: the group's last chunk
                    asm volatile("bar.sync %0, 128;" ::"r"(3 + g) : "memory");
                    request(2);
                }
                if (j > 0) {
                    wait(sh, &sh.a_empty[g], (unsigned)(j - 1) & 1u);
                    tc_fence_after();
                }
                float part[32];
#pragma unroll
                for (int i = 0; i < 32; i++) part[i] = tf32_round(v[i]);
                tmem_store32(lanes + kTmemHi + g * 2 * kPipeK, part);
                if (SPLIT) {
#pragma unroll
                    for (int i = 0; i < 32; i++) part[i] = v[i] - part[i];
                    tmem_store32(lanes + kTmemHi + g * 2 * kPipeK + kPipeK, part);
                }
                tmem_store_wait();
                tc_fence_before();
                mbar_arrive(&sh.a_full[g]);
            }
            if (MODE == kChainTangent) {
                // ---- A' = D T goes on, S T R stays (q); layer 3: its q is the first operand of the way back ----
#pragma unroll 1
                for (int l = 0; l < 3; l++) {
                    const int N = l == 2 ? kMlpH3 : 128;
                    if (c0 >= N) {
                        accumulator();
                        operand_done();
                        continue;
                    }
                    const size_t g0 = atom0 * N + c0;
                    float t[32], d[32], s[32];
                    accumulator();
                    warp_tile_from_global(scratch, s, (l == 0 ? p.act1[e] : (l == 1 ? p.act2[e] : p.act3[e])) + g0, N, tile_rows);
                    warp_tile_from_global(scratch, d, (l == 0 ? p.dact1[e] : (l == 1 ? p.dact2[e] : p.dact3[e])) + g0, N,
                                          tile_rows);
#pragma unroll
                    for (int i = 0; i < 32; i++) s[i] = mlp_activation_second<ACT>(s[i], d[i]);
                    if (l < 2) {
                        warp_tile_from_global(scratch, t, (l == 0 ? p.r1[e] : p.r2[e]) + g0, N, tile_rows);
#pragma unroll
                        for (int i = 0; i < 32; i++) s[i] *= t[i];
                    } else {
#pragma unroll
                        for (int i = 0; i < 32; i++) s[i] *= sh.w4[c0 + i];
                    }
                    tmem_load32(lanes + kTmemAcc + c0, t);
#pragma unroll
                    for (int i = 0; i < 32; i++) {
                        s[i] *= t[i];
                        d[i] *= t[i];
                    }
                    if (l < 2) to_operand(d);
                    else to_operand(s);
                    operand_done();
                    warp_tile_to_global<false>(scratch, d, (l == 0 ? p.adot1[e] : (l == 1 ? p.adot2[e] : p.adot3[e])) + g0, N,
                                               tile_rows);
                    warp_tile_to_global<false>(scratch, s, (l == 0 ? p.q1[e] : (l == 1 ? p.q2[e] : p.q3[e])) + g0, N, tile_rows);
                }
            } else {
            // ---- epilogues of layers 1 and 2 ----
#pragma unroll 1
            for (int l = 0; l < 2; l++) {
                accumulator();
                float v[32], d[32];
                tmem_load32(lanes + kTmemAcc + c0, v);
                const float* bias = sh.bias + l * kMlpH1 + c0;
#pragma unroll
                for (int i = 0; i < 32; i++) {
                    const float x = v[i] + bias[i];
                    v[i] = mlp_activation<ACT>(x);
                    d[i] = mlp_activation_grad<ACT>(x, v[i]);
                }
                to_operand(v);
                if (MODE == kChainForces) {
                    if (l == 0) {
                        tmem_store32(lanes + kTmemSpare + c0, d);
                    } else {
#pragma unroll
                        for (int i = 0; i < 32; i++) hold2[(c0 + i) * kMlpTile + row] = d[i];
                    }
                }
                operand_done();
                if (MODE == kChainForward) {
                    float* act = l == 0 ? p.act1[e] : p.act2[e];
                    float* dact = l == 0 ? p.dact1[e] : p.dact2[e];
                    if (act) warp_tile_to_global<false>(scratch, v, act + atom0 * 128 + c0, 128, tile_rows);
                    if (dact) warp_tile_to_global<false>(scratch, d, dact + atom0 * 128 + c0, 128, tile_rows);
                }
            }
            // ---- layer 3 and the output layer (the warps of columns 0-63) ----
            accumulator();
            if (c0 < kMlpH3) {
                float v[32], d[32];
                tmem_load32(lanes + kTmemAcc + c0, v);
                const float* bias = sh.bias + kMlpH1 + kMlpH2 + c0;
                float sum = c0 == 0 ? p.b4[e][0] : 0.0f;
#pragma unroll
                for (int i = 0; i < 32; i++) {
                    const float x = v[i] + bias[i];
                    v[i] = mlp_activation<ACT>(x);
                    d[i] = mlp_activation_grad<ACT>(x, v[i]);
                }
                // the energy, in the order of the columns: columns 0-31 here, 32-63 by the other warp of these rows
                if (c0 == 0) {
#pragma unroll
                    for (int i = 0; i < 32; i++) sum += v[i] * sh.w4[i];
                    sh.epart[row] = sum;
                }
                asm volatile("bar.sync 2, 256;" ::: "memory");
                if (c0 != 0) {
                    sum = sh.epart[row];
#pragma unroll
                    for (int i = 0; i < 32; i++) sum += v[i] * sh.w4[32 + i];
                    if (row < n_rows && wait.ok) p.energy[e][row0 + row] = sum;
                }
                if (MODE == kChainForward) {
                    if (p.act3[e]) warp_tile_to_global<false>(scratch, v, p.act3[e] + atom0 * kMlpH3 + c0, kMlpH3, tile_rows);
                    if (p.dact3[e]) warp_tile_to_global<false>(scratch, d, p.dact3[e] + atom0 * kMlpH3 + c0, kMlpH3, tile_rows);
                } else {
                    const float g = p.grad_energy[e] && row < n_rows ? p.grad_energy[e][row0 + row] : 1.0f;
#pragma unroll
                    for (int i = 0; i < 32; i++) v[i] = g * sh.w4[c0 + i] * d[i];      // dZ3
                    to_operand(v);
                }
            }
            if (MODE == kChainForces) operand_done();
            }
        } else {
            // ---- dZ3 = g w4 D3 ----
            if (c0 < kMlpH3) {
                const float g = p.grad_energy[e] ? (row < n_rows ? p.grad_energy[e][row0 + row] : 0.0f) : 1.0f;
                float v[32];
                warp_tile_from_global(scratch, v, p.dact3[e] + atom0 * kMlpH3 + c0, kMlpH3, tile_rows);
#pragma unroll
                for (int i = 0; i < 32; i++) v[i] *= g * sh.w4[c0 + i];
                to_operand(v);
                operand_done();
                warp_tile_to_global<false>(scratch, v, p.dz3[e] + atom0 * kMlpH3 + c0, kMlpH3, tile_rows);
            } else {
                operand_done();
            }
        }
        if (kHasBackward) {
            // ---- dZ2 = (dZ3 W3^T) D2, dZ1 = (dZ2 W2^T) D1 ----
#pragma unroll 1
            for (int l = 1; l >= 0; l--) {
                float v[32], d[32];
                const float* dact = l == 1 ? p.dact2[e] : p.dact1[e];
                if (MODE == kChainBackward || MODE == kChainTangent)      // before the wait: the loads run under the product
                    warp_tile_from_global(scratch, d, dact + atom0 * 128 + c0, 128, tile_rows);
                accumulator();
                tmem_load32(lanes + kTmemAcc + c0, v);
                if (MODE == kChainForces) {
                    if (l == 1) {
#pragma unroll
                        for (int i = 0; i < 32; i++) d[i] = hold2[(c0 + i) * kMlpTile + row];
                    } else {
                        tmem_load32(lanes + kTmemSpare + c0, d);
                    }
                }
                float* raw = MODE == kChainBackward ? (l == 1 ? p.r2[e] : p.r1[e]) : nullptr;
                if (raw) warp_tile_to_global<false>(scratch, v, raw + atom0 * 128 + c0, 128, tile_rows);
#pragma unroll
                for (int i = 0; i < 32; i++) v[i] *= d[i];
                if (MODE == kChainTangent) {      // + what this warp stored on the way forward
                    float* q = (l == 1 ? p.q2[e] : p.q1[e]) + atom0 * 128 + c0;
                    warp_tile_from_global(scratch, d, q, 128, tile_rows);
#pragma unroll
                    for (int i = 0; i < 32; i++) v[i] += d[i];
                    if (l == 1) {
                        to_operand(v);
                        operand_done();
                    }
                    warp_tile_to_global<false>(scratch, v, q, 128, tile_rows);
                    continue;
                }
                if (l == 1 || want_feat) {
                    to_operand(v);
                    operand_done();
                }
                if (MODE == kChainBackward) {
                    float* dz = l == 1 ? p.dz2[e] : p.dz1[e];
                    warp_tile_to_global<false>(scratch, v, dz + atom0 * 128 + c0, 128, tile_rows);
                }
            }
            // ---- dF = dZ1 W1^T, 128 feature columns at a time ----
            if (want_feat) {
                if (MODE == kChainForces) producer_sync();      // every warp has read its derivatives: scratch again
#pragma unroll 1
                for (int blk = 0; blk < 3; blk++) {
                    float v[32];
                    if (blk == 1) {
                        wait(sh, &sh.acc_full[1], 0u);
                        tc_fence_after();
                    } else {
                        accumulator();
                    }
                    tmem_load32(lanes + (blk == 1 ? kTmemSpare : kTmemAcc) + c0, v);
                    if (blk == 0) {
                        tc_fence_before();
                        mbar_arrive(&sh.acc_free);
                    }
                    warp_tile_to_global<false>(scratch, v, p.grad_feat[e] + atom0 * kMlpIn + blk * 128 + c0, kMlpIn, tile_rows);
                }
            }
        }
        if (!wait.ok && tid == 0) report(ANI_ERR_TIMEOUT);
    }
    tc_fence_before();
    __syncthreads();
    if (tid == 0 && sh.failed) report(ANI_ERR_TIMEOUT);
    tc_fence_after();
    if (warp == kChainEpi / 32) tmem_dealloc(tmem, 512);
}

}  // namespace ani
