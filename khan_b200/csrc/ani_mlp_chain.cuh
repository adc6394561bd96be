// Atomic networks 384-128-128-64-1 as ONE chain of products per tile of 128 atoms, on the tensor cores, with
// packed weights: forward, forward + backward to the features, backward alone, or the second-order pass of
// force training.
//
// Computes what ani_mlp_forward.cuh / ani_mlp_backward.cuh compute (AtomNN of the reference,
// khan/model/nn.py:39-67,165-172, and its gradient, khan/training/trainer_multi_tower.py:350-419); those remain
// for weights that are not packed.  The second-order pass is described in ani_force_fit.cuh.
//
// A tile is three products forward (K = 384, 128, 128) and five backward (K = 64, 128, 3 x 128), 38 chunks of 32
// values of K, three tf32 products each: 8 instructions, two of the products being one of 256 columns (12 in layer 3, which
// has 64 columns), at the tensor core's nominal rate 0.43 us (a chunk of layer 1 was measured at 0.52); the rest has to
// hide behind that.  The previous kernels took 1-2 us a chunk and 2-3 us between two products.  Here
//   * one thread streams the weights through a ring of stages, ahead over the whole chain, also across epilogues;
//   * every A operand is in tensor memory: an epilogue reads the accumulator, splits the new activations into
//     their tf32 parts and stores those to TMEM, where the next product takes them (columns: accumulators 0-127 for
//     hi hi and 128-255 for hi lo + lo hi, A high 256-383, A low 384-511).  With both operands in shared memory a chunk needs 160 KB of
//     its bandwidth, 1250 clocks against the tensor core's 830; now the weights are 80 KB of it;
//   * an epilogue of all 16 warps reads the accumulators and then hands over 32 columns at a time, and the next
//     product starts with the first of them: its 3300 clocks run beside the epilogue's 3000 to 5000;
//   * the features of a chunk are copied to shared memory as they are (16 KB), four warps read them row by row and
//     store their parts to TMEM; four groups of four warps take the chunks in turn (four stages of 64 columns in
//     the place of the later A operands);
//   * the thread that issues the products looks at the next chunk's barriers between two of its instructions: an
//     instruction is issued only when the tensor core is about to take it, so every clock that this thread waits
//     elsewhere (300 a barrier) is lost there;
//   * forward + backward in one kernel needs nothing of the activations in global memory: their derivatives wait
//     where the feature chunks were.
// Split precision: x = hi + lo with hi rounded to nearest, hi hi + hi lo + lo hi accumulated; the two small products
// apart, because the tensor core cuts its sums off at the accumulator's last place and three times the additions
// there were most of the error (energies against float64: 5e-6 -> 1.2e-6, plain float32 products give 0.7e-6).  Every wait is
// bounded; after a timeout the kernel reports, waits for its own copies, frees its tensor memory and returns.
#pragma once

#include "ani_mlp_pipe.cuh"

namespace ani {

constexpr int kChainA = 8, kChainB = 3;                 // feature chunks of 16 KB, weight stages of 32 KB (high, low)
constexpr int kChainEpi = 512;                          // epilogue / staging threads (16 warps)
constexpr int kChainThreads = kChainEpi + 64;           // + the MMA warp + the weight warp
constexpr int kChainGroups = 4;                         // groups of 128 threads that take the feature chunks in turn
constexpr unsigned kTmemAcc = 0, kTmemSmall = 128, kTmemHi = 256, kTmemLo = 384;

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
    int early_weights;               // nothing less than two kernels back writes weights: they may be read ahead of the
                                     // kernel before this one
};

struct ChainShared {
    alignas(1024) unsigned char a[kChainA][kPipeOperandBytes];
    alignas(1024) unsigned char b[kChainB][2 * kPipeOperandBytes];
    float bias[kMlpH1 + kMlpH2 + kMlpH3], w4[kMlpH3];
    float more_shares[2 * kMlpTile];
    alignas(8) unsigned long long a_full[kChainGroups], a_empty[kChainGroups], b_full[kChainB], b_empty[kChainB];
    unsigned long long acc_full;         // the accumulators hold a finished product
    unsigned long long operand_ready[4]; // the epilogue has stored columns 32 c .. of the next A operand
    unsigned long long acc_free;         // the epilogue has read a block of the feature gradient
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
// 32 / 8 consecutive columns of this thread's row (TMEM lane); completion: tmem_store_wait().
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
__device__ __forceinline__ void tmem_store8(unsigned taddr, const float* v)
{
    asm volatile("tcgen05.st.sync.aligned.32x32b.x8.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};" ::"r"(taddr), "f"(v[0]),
                 "f"(v[1]), "f"(v[2]), "f"(v[3]), "f"(v[4]), "f"(v[5]), "f"(v[6]), "f"(v[7])
                 : "memory");
}
__device__ __forceinline__ void tmem_store_wait() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }
// 8 consecutive columns of this thread's row; the registers are valid after tmem_load_wait().
__device__ __forceinline__ void tmem_load8(unsigned taddr, unsigned* r)
{
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7])
                 : "r"(taddr)
                 : "memory");
}
__device__ __forceinline__ void tmem_load_wait() { asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory"); }
__device__ __forceinline__ unsigned mbar_test(unsigned long long* bar, unsigned parity)
{
    unsigned done;
    asm volatile(
        "{\n"
        ".reg .pred p;\n"
        "mbarrier.test_wait.parity.shared::cta.b64 p, [%1], %2;\n"
        "selp.u32 %0, 1, 0, p;\n"
        "}\n"
        : "=r"(done)
        : "r"(smem_u32(bar)), "r"(parity)
        : "memory");
    return done;
}

// The columns of an epilogue: value i of a thread of the column group `sub` (warp / 4) is column
// 32 (i / 8) + 8 sub + i mod 8, so that 8 values of every thread are 32 whole columns of the tile.  Tiles of SEGS
// such blocks go to and from a row-major global matrix through shared memory: the four warps of 32 rows exchange
// their columns, and each moves 8 whole rows (512 or 256 bytes) with 16-byte accesses.  (Each warp on its own
// touched sixteen 128-byte lines an access: 4 us more in the backward pass.)  The 16-byte pieces of a row are
// permuted by the row number, which keeps both sides free of bank conflicts; two buffers in turn, so that one
// barrier of the four warps a tile is enough.
struct ChainTile {
    float* buffer;      // two of [128][128]
    int which;
    __device__ __forceinline__ float* next()
    {
        which ^= 1;
        return buffer + which * (kMlpTile * 128);
    }
    __device__ __forceinline__ static void meet(int quarter)
    {
        asm volatile("bar.sync %0, 128;" ::"r"(7 + quarter) : "memory");
    }
    // the same rows in every tile, however wide: only the four warps of a quarter wait for one another
    __device__ __forceinline__ static float4* at(float* t, int row, int piece)
    {
        return reinterpret_cast<float4*>(t) + row * 32 + (piece ^ (row & 7));
    }
    // gbase: row 0, column 0 of the tile; rows past n_rows are not written
    template <int SEGS> __device__ __forceinline__ void store(const float* v, float* gbase, size_t ld, int n_rows)
    {
        const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, quarter = warp & 3, sub = warp >> 2;
        float* t = next();
#pragma unroll
        for (int i = 0; i < 2 * SEGS; i++)
            *at(t, quarter * 32 + lane, 8 * (i >> 1) + 2 * sub + (i & 1)) =
                make_float4(v[4 * i], v[4 * i + 1], v[4 * i + 2], v[4 * i + 3]);
        meet(quarter);
        constexpr int kLanes = 8 * SEGS;      // lanes of a row
#pragma unroll
        for (int k = 0; k < 8 * kLanes / 32; k++) {
            const int r = quarter * 32 + sub * 8 + k * (32 / kLanes) + lane / kLanes, piece = lane % kLanes;
            const float4 q = *at(t, r, piece);
            if (r < n_rows) *reinterpret_cast<float4*>(gbase + (size_t)r * ld + 4 * piece) = q;
        }
    }
    // rows past n_rows read as zero
    template <int SEGS> __device__ __forceinline__ void load(float* v, const float* gbase, size_t ld, int n_rows)
    {
        const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, quarter = warp & 3, sub = warp >> 2;
        float* t = next();
        constexpr int kLanes = 8 * SEGS, kSteps = 8 * kLanes / 32;
        float4 q[kSteps];
#pragma unroll
        for (int k = 0; k < kSteps; k++) {
            const int r = quarter * 32 + sub * 8 + k * (32 / kLanes) + lane / kLanes, piece = lane % kLanes;
            q[k] = make_float4(0.f, 0.f, 0.f, 0.f);
            if (r < n_rows) q[k] = *reinterpret_cast<const float4*>(gbase + (size_t)r * ld + 4 * piece);
        }
#pragma unroll
        for (int k = 0; k < kSteps; k++) {
            const int r = quarter * 32 + sub * 8 + k * (32 / kLanes) + lane / kLanes, piece = lane % kLanes;
            *at(t, r, piece) = q[k];
        }
        meet(quarter);
#pragma unroll
        for (int i = 0; i < 2 * SEGS; i++) {
            const float4 x = *at(t, quarter * 32 + lane, 8 * (i >> 1) + 2 * sub + (i & 1));
            v[4 * i] = x.x; v[4 * i + 1] = x.y; v[4 * i + 2] = x.z; v[4 * i + 3] = x.w;
        }
    }
};

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
        mbar_init(&sh.acc_full, 1);
        for (int c = 0; c < 4; c++) mbar_init(&sh.operand_ready[c], kChainEpi);
        mbar_init(&sh.acc_free, kChainEpi);
        sh.failed = 0;
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    if (!(p.early_weights && warp == kChainEpi / 32 + 1)) {      // the weight warp may run ahead
        pdl_wait();
        // Energies + forces: the CTAs of the gradient kernel behind would gather on the SMs that have no tile, the largest
        // molecules first (1024 molecules, a third of the SMs without one: 116 us a pass, 107.5 without the trigger).
        if (MODE != kChainForces) pdl_trigger();
    }
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
        // ---- the products: one thread ----
        if (lane == 0) {
            ChainWait wait;
            int b_stage = 0;
            unsigned b_parity = 0, ready_parity = 0;      // bit c: parity of operand_ready[c]
            unsigned b_seen = 0, a_seen = 0;              // the next chunk's barriers, looked at while issuing this one
            // The products of a chunk; `next_a` / `next_parity`: barrier of the next chunk's A operand (or null).
            auto issue = [&](unsigned a_hi, unsigned a_lo, int N, bool first, unsigned long long* next_a,
                             unsigned next_parity) {
                const unsigned idesc = instr_desc(kMlpTile, N);
                const unsigned b_hi = smem_u32(sh.b[b_stage]), b_lo = b_hi + kPipeOperandBytes;
                unsigned long long* used = &sh.b_empty[b_stage];
                if (++b_stage == kChainB) {
                    b_stage = 0;
                    b_parity ^= 1u;
                }
#pragma unroll
                for (int ks = 0; ks < kPipeK / 8; ks++) {
                    const unsigned step = ks * 2 * kMlpLbo, col = ks * 8;
                    const bool add = !(first && ks == 0);
                    static_assert(kPipeOperandBytes == (kMlpTile / 8) * kPipeSbo && kTmemSmall == kTmemAcc + kMlpTile,
                                  "the low part of B is rows 128 to 255 of the high part, and so are the accumulators' columns");
                    if (SPLIT && N == 128) {
                        // hi hi and hi lo as one instruction of 256 columns (the two parts of B lie behind one another, and so
                        // do the two accumulators): a chunk of layer 1 takes 0.52 us instead of 0.64, forward + backward of
                        // 1024 molecules' atoms 36 us instead of 40
                        mma_tf32_ts(tmem + kTmemAcc, tmem + a_hi + col, pipe_desc(b_hi + step), instr_desc(kMlpTile, 256), add);
                        mma_tf32_ts(tmem + kTmemSmall, tmem + a_lo + col, pipe_desc(b_hi + step), idesc, true);
                    } else {
                        mma_tf32_ts(tmem + kTmemAcc, tmem + a_hi + col, pipe_desc(b_hi + step), idesc, add);
                        if (SPLIT) {
                            mma_tf32_ts(tmem + kTmemSmall, tmem + a_hi + col, pipe_desc(b_lo + step), idesc, add);
                            mma_tf32_ts(tmem + kTmemSmall, tmem + a_lo + col, pipe_desc(b_hi + step), idesc, true);
                        }
                    }
                    if (ks == 1) {
                        b_seen = mbar_test(&sh.b_full[b_stage], b_parity);
                        a_seen = next_a ? mbar_test(next_a, next_parity) : 0u;
                    }
                }
                mma_commit(used);
            };
            auto weights = [&]() {
                if (!b_seen) wait(sh, &sh.b_full[b_stage], b_parity);
            };
            // one product behind layer 1; fresh: its A operand comes from the epilogue, else it is the last one's
            auto product = [&](int chunks, int N, bool fresh) {
                for (int c = 0; c < chunks; c++) {
                    if (fresh) {
                        if (!a_seen) wait(sh, &sh.operand_ready[c], (ready_parity >> c) & 1u);
                        ready_parity ^= 1u << c;
                    }
                    weights();
                    if (!wait.ok) return;
                    tc_fence_after();
                    const bool more = fresh && c + 1 < chunks;
                    issue(kTmemHi + c * kPipeK, kTmemLo + c * kPipeK, N, c == 0,
                          more ? &sh.operand_ready[c + 1] : nullptr, more ? (ready_parity >> (c + 1)) & 1u : 0u);
                }
                mma_commit(&sh.acc_full);
                a_seen = 0;
            };
            if (kHasForward) {
                for (int c = 0; c < kMlpIn / kPipeK; c++) {
                    const int g = c % kChainGroups;
                    if (!a_seen) wait(sh, &sh.a_full[g], (unsigned)(c / kChainGroups) & 1u);
                    weights();
                    if (!wait.ok) break;
                    tc_fence_after();
                    const bool more = c + 1 < kMlpIn / kPipeK;
                    issue(kTmemHi + g * 2 * kPipeK, kTmemHi + g * 2 * kPipeK + kPipeK, kMlpH1, c == 0,
                          more ? &sh.a_full[(c + 1) % kChainGroups] : nullptr, (unsigned)((c + 1) / kChainGroups) & 1u);
                    mma_commit(&sh.a_empty[g]);
                }
                if (wait.ok) mma_commit(&sh.acc_full);
                a_seen = 0;
                product(kMlpH1 / kPipeK, kMlpH2, true);
                product(kMlpH2 / kPipeK, kMlpH3, true);
            }
            if (kHasBackward) {
                product(kMlpH3 / kPipeK, kMlpH2, true);
                product(kMlpH2 / kPipeK, kMlpH1, true);
                if (want_feat) {
                    product(kMlpH1 / kPipeK, 128, true);
                    wait(sh, &sh.acc_free, 0u);
                    product(kMlpH1 / kPipeK, 128, false);
                    wait(sh, &sh.acc_free, 1u);
                    product(kMlpH1 / kPipeK, 128, false);
                }
            }
        }
    } else {
        // ---- feature staging and epilogues: warp w has rows 32 (w % 4) .. and the columns of group w / 4 ----
        ChainWait wait;
        const int sub = warp >> 2, tile_row0 = (warp & 3) * 32, row = tile_row0 + lane;
        const size_t atom0 = (size_t)row0;
        const unsigned lanes = tmem + ((unsigned)tile_row0 << 16);
        // over the feature chunks, idle outside layer 1: tiles on their way to and from global memory, or (forces mode)
        // the derivatives of layers 1 and 2, [128 columns][128 rows]
        ChainTile tile{reinterpret_cast<float*>(sh.a[0]), 0};
        float* hold1 = reinterpret_cast<float*>(sh.a[0]);
        float* hold2 = hold1 + kMlpH1 * kMlpTile;
        int done_products = 0;

        // the result of the next product, 8 values of each of the first `segs` blocks of 32 columns
        auto accumulator = [&](float* v, int segs) {
            wait(sh, &sh.acc_full, (unsigned)done_products & 1u);
            done_products++;
            tc_fence_after();
            unsigned r[32], q[32];
#pragma unroll
            for (int s = 0; s < 4; s++)
                if (s < segs) {
                    tmem_load8(lanes + kTmemAcc + s * 32 + sub * 8, r + 8 * s);
                    if (SPLIT) tmem_load8(lanes + kTmemSmall + s * 32 + sub * 8, q + 8 * s);
                }
            tmem_load_wait();
#pragma unroll
            for (int i = 0; i < 32; i++)
                if (i < 8 * segs) v[i] = SPLIT ? __uint_as_float(r[i]) + __uint_as_float(q[i]) : __uint_as_float(r[i]);
        };
        // 8 values of block s of the next A operand
        auto operand = [&](const float* v, int s) {
            float part[8];
#pragma unroll
            for (int i = 0; i < 8; i++) part[i] = tf32_round(v[i]);
            tmem_store8(lanes + kTmemHi + s * 32 + sub * 8, part);
            if (SPLIT) {
#pragma unroll
                for (int i = 0; i < 8; i++) part[i] = v[i] - part[i];
                tmem_store8(lanes + kTmemLo + s * 32 + sub * 8, part);
            }
        };
        // blocks are handed over one behind the stores, so that these run under the next block's arithmetic
        auto hand_over = [&](int s) {
            tmem_store_wait();
            tc_fence_before();
            mbar_arrive(&sh.operand_ready[s]);
        };

        const int g = warp >> 2, me = tid & 127;
        const float* feat = kHasForward ? p.feat[e] + (size_t)row0 * kMlpIn : nullptr;
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
        if (kHasForward) {
            request(0);
            request(1);
        }
        // biases and output weights, one value per thread: requested here, stored behind layer 1
        float vec = 0.0f;
        constexpr int kBiases = kMlpH1 + kMlpH2 + kMlpH3;
        if (kHasForward && MODE != kChainTangent && tid < kBiases)
            vec = tid < kMlpH1 ? p.b1[e][tid] : (tid < kMlpH1 + kMlpH2 ? p.b2[e][tid - kMlpH1] : p.b3[e][tid - kMlpH1 - kMlpH2]);
        if (tid >= kBiases && tid < kBiases + kMlpH3) vec = p.w4[e][tid - kBiases];
        auto store_vec = [&]() {
            if (tid < kBiases) sh.bias[tid] = vec;
            else if (tid < kBiases + kMlpH3) sh.w4[tid - kBiases] = vec;
            producer_sync();
        };
        if (!kHasForward) store_vec();

        if (kHasForward) {
            // ---- layer 1: group g of 128 threads takes chunks g, g + 4, g + 8; thread = row (TMEM lane) ----
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
            store_vec();      // (behind it the feature chunks have been read, too)
            if (MODE == kChainTangent) {
                // ---- A' = D T goes on, S T R stays (q); layer 3: its q is the first operand of the way back ----
#pragma unroll 1
                for (int l = 0; l < 3; l++) {
                    float t[32], d[32], s[32];
                    const size_t g0 = atom0 * (l == 2 ? kMlpH3 : 128);
                    const float* act = (l == 0 ? p.act1[e] : (l == 1 ? p.act2[e] : p.act3[e])) + g0;
                    const float* dact = (l == 0 ? p.dact1[e] : (l == 1 ? p.dact2[e] : p.dact3[e])) + g0;
                    float* adot = (l == 0 ? p.adot1[e] : (l == 1 ? p.adot2[e] : p.adot3[e])) + g0;
                    float* q = (l == 0 ? p.q1[e] : (l == 1 ? p.q2[e] : p.q3[e])) + g0;
                    if (l < 2) {
                        tile.load<4>(s, act, 128, n_rows);
                        tile.load<4>(d, dact, 128, n_rows);
                        tile.load<4>(t, (l == 0 ? p.r1[e] : p.r2[e]) + g0, 128, n_rows);
#pragma unroll
                        for (int i = 0; i < 32; i++) s[i] = mlp_activation_second<ACT>(s[i], d[i]) * t[i];
                        accumulator(t, 4);
#pragma unroll
                        for (int b = 0; b < 4; b++) {
#pragma unroll
                            for (int i = 8 * b; i < 8 * b + 8; i++) {
                                s[i] *= t[i];
                                d[i] *= t[i];
                            }
                            if (b > 0) hand_over(b - 1);
                            operand(d + 8 * b, b);
                        }
                        hand_over(3);
                        tile.store<4>(d, adot, 128, n_rows);
                        tile.store<4>(s, q, 128, n_rows);
                    } else {
                        tile.load<2>(s, act, kMlpH3, n_rows);
                        tile.load<2>(d, dact, kMlpH3, n_rows);
                        accumulator(t, 2);
#pragma unroll
                        for (int b = 0; b < 2; b++) {
#pragma unroll
                            for (int i = 8 * b; i < 8 * b + 8; i++) {
                                s[i] = mlp_activation_second<ACT>(s[i], d[i]) * sh.w4[32 * b + 8 * sub + (i & 7)] * t[i];
                                d[i] *= t[i];
                            }
                            if (b > 0) hand_over(b - 1);
                            operand(s + 8 * b, b);
                        }
                        hand_over(1);
                        tile.store<2>(d, adot, kMlpH3, n_rows);
                        tile.store<2>(s, q, kMlpH3, n_rows);
                    }
                }
            } else {
                // ---- epilogues of layers 1 and 2 ----
#pragma unroll 1
                for (int l = 0; l < 2; l++) {
                    float v[32], d[32];
                    accumulator(v, 4);
                    const float* bias = sh.bias + l * kMlpH1 + sub * 8;
                    float* hold = l == 0 ? hold1 : hold2;
#pragma unroll
                    for (int b = 0; b < 4; b++) {
#pragma unroll
                        for (int i = 8 * b; i < 8 * b + 8; i++) {
                            const float x = v[i] + bias[32 * b + (i & 7)];
                            v[i] = mlp_activation<ACT>(x);
                            d[i] = mlp_activation_grad<ACT>(x, v[i]);
                        }
                        if (b > 0) hand_over(b - 1);
                        operand(v + 8 * b, b);
                        if (MODE == kChainForces) {
#pragma unroll
                            for (int i = 8 * b; i < 8 * b + 8; i++)
                                hold[(32 * b + 8 * sub + (i & 7)) * kMlpTile + row] = d[i];
                        }
                    }
                    hand_over(3);
                    if (MODE == kChainForward) {
                        float* act = l == 0 ? p.act1[e] : p.act2[e];
                        float* dact = l == 0 ? p.dact1[e] : p.dact2[e];
                        if (act) tile.store<4>(v, act + atom0 * 128, 128, n_rows);
                        if (dact) tile.store<4>(d, dact + atom0 * 128, 128, n_rows);
                    }
                }
                // ---- layer 3 and the output layer ----
                float v[32], d[32];
                accumulator(v, 2);
                const float* bias = sh.bias + kMlpH1 + kMlpH2 + sub * 8;
                float share = 0.0f;      // of the energy: this thread's 16 columns
                const float ge = MODE == kChainForces && p.grad_energy[e] && row < n_rows ? p.grad_energy[e][row0 + row] : 1.0f;
#pragma unroll
                for (int b = 0; b < 2; b++) {
#pragma unroll
                    for (int i = 8 * b; i < 8 * b + 8; i++) {
                        const float x = v[i] + bias[32 * b + (i & 7)];
                        const float w = sh.w4[32 * b + 8 * sub + (i & 7)];
                        v[i] = mlp_activation<ACT>(x);
                        d[i] = mlp_activation_grad<ACT>(x, v[i]);
                        share += v[i] * w;
                        if (MODE == kChainForces) v[i] = ge * w * d[i];      // dZ3
                    }
                    if (MODE == kChainForces) {
                        if (b > 0) hand_over(b - 1);
                        operand(v + 8 * b, b);
                    }
                }
                if (MODE == kChainForces) hand_over(1);
                // the biases of layers 1 and 2 have been used by every warp: their place takes two of the four shares
                float* shares = sub < 2 ? sh.bias + sub * kMlpTile : sh.more_shares + (sub - 2) * kMlpTile;
                shares[row] = share;
                if (MODE == kChainForward) {
                    if (p.act3[e]) tile.store<2>(v, p.act3[e] + atom0 * kMlpH3, kMlpH3, n_rows);
                    if (p.dact3[e]) tile.store<2>(d, p.dact3[e] + atom0 * kMlpH3, kMlpH3, n_rows);
                }
                producer_sync();
                if (tid < n_rows && wait.ok)
                    p.energy[e][row0 + tid] = p.b4[e][0] + sh.bias[tid] + sh.bias[kMlpTile + tid] + sh.more_shares[tid] +
                                              sh.more_shares[kMlpTile + tid];
            }
        } else {
            // ---- dZ3 = g w4 D3 ----
            const float ge = p.grad_energy[e] ? (row < n_rows ? p.grad_energy[e][row0 + row] : 0.0f) : 1.0f;
            float v[32];
            tile.load<2>(v, p.dact3[e] + atom0 * kMlpH3, kMlpH3, n_rows);
#pragma unroll
            for (int b = 0; b < 2; b++) {
#pragma unroll
                for (int i = 8 * b; i < 8 * b + 8; i++) v[i] *= ge * sh.w4[32 * b + 8 * sub + (i & 7)];
                if (b > 0) hand_over(b - 1);
                operand(v + 8 * b, b);
            }
            hand_over(1);
            tile.store<2>(v, p.dz3[e] + atom0 * kMlpH3, kMlpH3, n_rows);
        }
        if (kHasBackward) {
            // ---- dZ2 = (dZ3 W3^T) D2, dZ1 = (dZ2 W2^T) D1 ----
#pragma unroll 1
            for (int l = 1; l >= 0; l--) {
                float v[32], d[32];
                const size_t g0 = atom0 * 128;
                if (MODE != kChainForces)      // before the wait: the loads run under the product
                    tile.load<4>(d, (l == 1 ? p.dact2[e] : p.dact1[e]) + g0, 128, n_rows);
                accumulator(v, 4);
                if (MODE == kChainTangent) {      // + what this warp stored on the way forward
                    float* q = (l == 1 ? p.q2[e] : p.q1[e]) + g0;
#pragma unroll
                    for (int i = 0; i < 32; i++) v[i] *= d[i];
                    tile.load<4>(d, q, 128, n_rows);
#pragma unroll
                    for (int b = 0; b < 4; b++) {
#pragma unroll
                        for (int i = 8 * b; i < 8 * b + 8; i++) v[i] += d[i];
                        if (l == 1) {
                            if (b > 0) hand_over(b - 1);
                            operand(v + 8 * b, b);
                        }
                    }
                    if (l == 1) hand_over(3);
                    tile.store<4>(v, q, 128, n_rows);
                    continue;
                }
                float* raw = MODE == kChainBackward ? (l == 1 ? p.r2[e] : p.r1[e]) : nullptr;
                if (raw) tile.store<4>(v, raw + g0, 128, n_rows);
                const float* hold = l == 1 ? hold2 : hold1;
#pragma unroll
                for (int b = 0; b < 4; b++) {
#pragma unroll
                    for (int i = 8 * b; i < 8 * b + 8; i++)
                        v[i] *= MODE == kChainForces ? hold[(32 * b + 8 * sub + (i & 7)) * kMlpTile + row] : d[i];
                    if (l == 1 || want_feat) {
                        if (b > 0) hand_over(b - 1);
                        operand(v + 8 * b, b);
                    }
                }
                if (l == 1 || want_feat) hand_over(3);
                if (MODE == kChainBackward)
                    tile.store<4>(v, (l == 1 ? p.dz2[e] : p.dz1[e]) + g0, 128, n_rows);
            }
            // ---- dF = dZ1 W1^T, 128 feature columns at a time ----
            if (want_feat) {
                if (MODE == kChainForces) producer_sync();      // every warp has read its derivatives: tiles again
#pragma unroll 1
                for (int blk = 0; blk < 3; blk++) {
                    float v[32];
                    accumulator(v, 4);
                    if (blk < 2) {
                        tc_fence_before();
                        mbar_arrive(&sh.acc_free);
                    }
                    tile.store<4>(v, p.grad_feat[e] + atom0 * kMlpIn + blk * 128, kMlpIn, n_rows);
                }
            }
        }
    }
    tc_fence_before();
    __syncthreads();
    if (tid == 0 && sh.failed) report(ANI_ERR_TIMEOUT);
    tc_fence_after();
    if (warp == kChainEpi / 32) tmem_dealloc(tmem, 512);
}

}  // namespace ani
