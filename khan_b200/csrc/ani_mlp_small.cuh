// Atomic networks of FEW atoms, and of double precision: forward pass and the backward pass to the
// features in one kernel, on the FMA pipes.
//
// Computes what ani_mlp_forward.cuh and ani_mlp_backward.cuh compute together for energies and forces
// (khan/model/nn.py:39-67,165-172 and its gradient, khan/training/trainer_multi_tower.py:350-399).
//
// A chain of six products on a handful of atoms is bound by latency: the tensor-core kernels walk 38
// operand chunks one behind the other on ONE SM per element, whatever the number of atoms.  Here a tile of
// 16 atoms of one element is the work of a CLUSTER of 8 CTAs: each owns an eighth of the output columns of
// every layer (so the weights of the tile are loaded once, spread over 8 SMs, all of them requested at the
// start and, in a chain, before the features exist), and the activations go to all 8 CTAs through
// distributed shared memory, one cluster barrier per layer.  Inside a CTA a product is 2 x 2 register tiles
// over four or eight slices of K, summed through shared memory.
//
// Double precision has no other kernel: there the tiles simply queue up, each fetching the weights of its element from
// L2 again.  Measured, forward / with backward: 891 atoms 40 / 68 us, 3.6 k 137 / 244, 14 k 516 / 939, 28 k 1034 / 1879:
// 37 / 67 ns an atom, 4.4 TFLOP/s, an eighth of the FP64 rate.  (Before it, dense products: coordinate gradients of a data
// set of 8,192 molecules 33.6 ms, 8.6 with it; energies 5.5 and 4.8.)
#pragma once

#include "ani_common.cuh"
#include "ani_launch.cuh"
#include "ani_mlp_pipe.cuh"

namespace ani {

constexpr int kSmallTile = 16;       // atoms of a cluster
constexpr int kSmallCtas = 8;        // CTAs of a cluster
constexpr int kSmallThreads = 256;
constexpr int kSmallC = kMlpH1 / kSmallCtas;      // 16 columns of layers 1 and 2 per CTA
constexpr int kSmallC3 = kMlpH3 / kSmallCtas;     // 8 columns of layer 3
constexpr int kSmallF = kMlpIn / kSmallCtas;      // 48 feature columns of the gradient

template <typename T> struct MlpSmallParams {
    const T* feat;               // [atoms][384], element-sorted
    int count[kTypes];
    int row_start[kTypes];       // first row of each element
    int tile_start[kTypes + 1];  // prefix of ceil(count / 16)
    const T* w1[kTypes];
    const T* b1[kTypes];
    const T* w2[kTypes];
    const T* b2[kTypes];
    const T* w3[kTypes];
    const T* b3[kTypes];
    const T* w4[kTypes];
    const T* b4[kTypes];
    const T* grad_energy;        // [atoms] dL/dE, or null: ones
    T* energy;                   // [atoms]
    T* grad_feat;                // [atoms][384], or null: forward only
    int activation;
    int early_weights;           // a featurizer kernel of the same call precedes: the weights may be read ahead of it
};

template <typename T> struct MlpSmallShared {
    static constexpr int kPad = 16 / (int)sizeof(T);
    static constexpr int kLdF = kMlpIn + kPad, kLdH = kMlpH1 + kPad, kLd3 = kMlpH3 + kPad;
    static constexpr int kX = kSmallTile * kLdF > kSmallF * kLdH ? kSmallTile * kLdF : kSmallF * kLdH;
    alignas(16) T x[kX];                         // the features; later rows 48 r .. of W1
    alignas(16) T w1c[kMlpIn * kSmallC];         // columns 16 r .. of W1; later partial sums
    alignas(16) T w2c[kMlpH1 * kSmallC];
    alignas(16) T w3c[kMlpH2 * kSmallC3];
    alignas(16) T w2r[kSmallC * kLdH];           // rows 16 r .. of W2
    alignas(16) T w3r[kSmallC * kLd3];
    alignas(16) T h1[kSmallTile * kLdH];         // A1, later dZ2
    alignas(16) T h2[kSmallTile * kLdH];         // partial sums of layer 1, then A2, later dZ1
    alignas(16) T h3[kSmallTile * kLd3];         // dZ3
    T epart[kSmallCtas * kSmallTile];            // CTA 0: the other CTAs' shares of the energies
};

__device__ __forceinline__ void cluster_arrive() { asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory"); }
__device__ __forceinline__ void cluster_wait() { asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory"); }
__device__ __forceinline__ unsigned cluster_rank()
{
    unsigned r;
    asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
    return r;
}
// Stores v at the place of `local` in the shared memory of CTA `rank` of the cluster.
__device__ __forceinline__ void store_remote(const void* local, unsigned rank, float v)
{
    unsigned a;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(a) : "r"(smem_u32(local)), "r"(rank));
    asm volatile("st.shared::cluster.f32 [%0], %1;" ::"r"(a), "f"(v) : "memory");
}
__device__ __forceinline__ void store_remote(const void* local, unsigned rank, double v)
{
    unsigned a;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(a) : "r"(smem_u32(local)), "r"(rank));
    asm volatile("st.shared::cluster.f64 [%0], %1;" ::"r"(a), "d"(v) : "memory");
}

__device__ __forceinline__ double exp_full(double x) { return exp(x); }
__device__ __forceinline__ float exp_full(float x) { return expf(x); }
__device__ __forceinline__ double log1p_full(double x) { return log1p(x); }
__device__ __forceinline__ float log1p_full(float x) { return log1pf(x); }

// Activation and its derivative (khan/model/activations.py:62-74).
template <typename T> __device__ __forceinline__ void small_activation(int act, T x, T* a, T* d)
{
    if (act == kActCelu) {
        const T e = exp_full((x < (T)0 ? x : (T)0) * (T)10);
        *a = x >= (T)0 ? x : (T)0.1 * (e - (T)1);
        *d = x >= (T)0 ? (T)1 : e;
    } else if (act == kActGaussian) {
        *a = exp_full(-x * x);
        *d = (T)-2 * x * *a;
    } else if (act == kActNormal) {
        *a = exp_full((T)-0.5 * x * x);
        *d = -x * *a;
    } else {
        *a = (x > (T)20 ? x : log1p_full(exp_full(x))) - (T)0.69314718056;
        *d = (T)1 / ((T)1 + exp_full(-x));
    }
}

__device__ __forceinline__ void small_copy16(void* dst, const void* src)
{
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(smem_u32(dst)), "l"(src) : "memory");
}
// rows x cols of a row-major matrix (row stride ld) into shared memory (row stride lds).
template <typename T>
__device__ __forceinline__ void small_load(T* dst, int lds, const T* src, int ld, int rows, int cols)
{
    constexpr int V = 16 / (int)sizeof(T);
    const int per_row = cols / V;
    for (int i = threadIdx.x; i < rows * per_row; i += kSmallThreads) {
        const int r = i / per_row, c = (i - r * per_row) * V;
        small_copy16(dst + r * lds + c, src + (size_t)r * ld + c);
    }
}

// 16 bytes of consecutive values.
template <typename T> struct SmallVec;
template <> struct SmallVec<float> {
    static constexpr int N = 4;
    float v[4];
    __device__ __forceinline__ explicit SmallVec(const float* p)
    {
        const float4 q = *reinterpret_cast<const float4*>(p);
        v[0] = q.x; v[1] = q.y; v[2] = q.z; v[3] = q.w;
    }
};
template <> struct SmallVec<double> {
    static constexpr int N = 2;
    double v[2];
    __device__ __forceinline__ explicit SmallVec(const double* p)
    {
        const double2 q = *reinterpret_cast<const double2*>(p);
        v[0] = q.x; v[1] = q.y;
    }
};

// out[atom][col] += sum over k in [k0, k1) of a[atom][k] w[k][col]: w row-major along the columns; atoms
// 2 ap, 2 ap + 1 and columns 2 cp, 2 cp + 1 of this thread.  Partial sums to red[group][atom * cols + col].
template <typename T>
__device__ __forceinline__ void small_product(const T* a, int lda, const T* w, int cols, int ap, int cp, int k0, int k1,
                                              T* red)
{
    constexpr int V = SmallVec<T>::N;
    T s00 = (T)0, s01 = (T)0, s10 = (T)0, s11 = (T)0;
    const T* a0 = a + 2 * ap * lda;
    const T* a1 = a0 + lda;
#pragma unroll 4
    for (int k = k0; k < k1; k += V) {
        const SmallVec<T> x0(a0 + k), x1(a1 + k);
#pragma unroll
        for (int i = 0; i < V; i++) {
            const Vec2<T> q = *reinterpret_cast<const Vec2<T>*>(w + (k + i) * cols + 2 * cp);
            s00 += x0.v[i] * q.x; s01 += x0.v[i] * q.y;
            s10 += x1.v[i] * q.x; s11 += x1.v[i] * q.y;
        }
    }
    T* out = red + 2 * ap * cols + 2 * cp;
    out[0] = s00; out[1] = s01; out[cols] = s10; out[cols + 1] = s11;
}

// The same with w given by its rows, w[col][k] (row stride ldw): NC columns cp, cp + 8, ... of this thread,
// `cols` = 8 NC of them in all.
template <typename T, int NC>
__device__ __forceinline__ void small_product_t(const T* a, int lda, const T* w, int ldw, int ap, int cp, int k0, int k1,
                                                T* red)
{
    constexpr int V = SmallVec<T>::N;
    constexpr int kCols = 8 * NC;
    T s[2][NC];
#pragma unroll
    for (int c = 0; c < NC; c++) s[0][c] = s[1][c] = (T)0;
    const T* a0 = a + 2 * ap * lda;
    const T* a1 = a0 + lda;
#pragma unroll 2
    for (int k = k0; k < k1; k += V) {
        const SmallVec<T> x0(a0 + k), x1(a1 + k);
#pragma unroll
        for (int c = 0; c < NC; c++) {
            const SmallVec<T> q(w + (cp + 8 * c) * ldw + k);
#pragma unroll
            for (int i = 0; i < V; i++) {
                s[0][c] += x0.v[i] * q.v[i];
                s[1][c] += x1.v[i] * q.v[i];
            }
        }
    }
#pragma unroll
    for (int c = 0; c < NC; c++) {
        red[2 * ap * kCols + cp + 8 * c] = s[0][c];
        red[(2 * ap + 1) * kCols + cp + 8 * c] = s[1][c];
    }
}

template <typename T>
__global__ void __launch_bounds__(kSmallThreads, 1) mlp_small_kernel(const MlpSmallParams<T> p, const MlpPackParams pack)
{
    // The clusters behind the tiles pack the weights for later passes.  (In front of the sort, where larger batches have
    // them, the packing made a pass over one molecule 31.0 us long instead of 29.3.)
    if ((int)blockIdx.x >= p.tile_start[kTypes] * kSmallCtas) {
        const int c = (int)blockIdx.x - p.tile_start[kTypes] * kSmallCtas;
        pdl_wait();      // no trigger: weights are written
        pack_chunk(pack, c % kPackChunks, c / kPackChunks);
        return;
    }
    extern __shared__ __align__(16) unsigned char small_smem_raw[];
    using S = MlpSmallShared<T>;
    S& sh = *reinterpret_cast<S*>(small_smem_raw);
    const int tid = threadIdx.x;
    const unsigned rank = cluster_rank();
    const int tile = (int)blockIdx.x / kSmallCtas;
    int e = 0;
#pragma unroll
    for (int t = 1; t < kTypes; t++) e += tile >= p.tile_start[t] ? 1 : 0;
    const int row_in = (tile - p.tile_start[e]) * kSmallTile;
    const int n_rows = min(kSmallTile, p.count[e] - row_in);
    const size_t row0 = (size_t)p.row_start[e] + row_in;
    const bool backward = p.grad_feat != nullptr;

    if (!p.early_weights) pdl_wait();
    cluster_arrive();      // (0) every CTA of the cluster runs before the first store into its memory
    // ---- weights first (they do not depend on the features), then the features ----
    small_load(sh.w1c, kSmallC, p.w1[e] + kSmallC * rank, kMlpH1, kMlpIn, kSmallC);
    asm volatile("cp.async.commit_group;" ::: "memory");
    const int atom = tid >> 4, col = tid & 15;            // this thread's value of layers 1 and 2
    const int atom3 = (tid >> 3) & 15, col3 = tid & 7;    // and of layer 3 (threads 0 .. 127)
    const T bias1 = p.b1[e][kSmallC * rank + col], bias2 = p.b2[e][kSmallC * rank + col];
    const T bias3 = p.b3[e][kSmallC3 * rank + col3], out3 = p.w4[e][kSmallC3 * rank + col3];
    const T bias4 = p.b4[e][0];
    pdl_wait();
    pdl_trigger();
    small_load(sh.x, S::kLdF, p.feat + row0 * kMlpIn, kMlpIn, n_rows, kMlpIn);
    asm volatile("cp.async.commit_group;" ::: "memory");
    for (int i = tid; i < (kSmallTile - n_rows) * kMlpIn; i += kSmallThreads)      // atoms that do not exist
        sh.x[(n_rows + i / kMlpIn) * S::kLdF + i % kMlpIn] = (T)0;
    small_load(sh.w2c, kSmallC, p.w2[e] + kSmallC * rank, kMlpH2, kMlpH1, kSmallC);
    small_load(sh.w3c, kSmallC3, p.w3[e] + kSmallC3 * rank, kMlpH3, kMlpH2, kSmallC3);
    if (backward) {
        small_load(sh.w3r, S::kLd3, p.w3[e] + (size_t)kSmallC * rank * kMlpH3, kMlpH3, kSmallC, kMlpH3);
        small_load(sh.w2r, S::kLdH, p.w2[e] + (size_t)kSmallC * rank * kMlpH2, kMlpH2, kSmallC, kMlpH2);
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
    asm volatile("cp.async.wait_group 1;" ::: "memory");
    __syncthreads();

    const int kg = tid >> 6, ap = (tid >> 3) & 7, cp = tid & 7;   // slice of K, atom pair, column pair
    // ---- layer 1: 384 -> own 16 columns ----
    small_product<T>(sh.x, S::kLdF, sh.w1c, kSmallC, ap, cp, kg * 96, kg * 96 + 96, sh.h2 + kg * 256);
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    __syncthreads();
    if (backward) {      // the features are used up: their place takes the rows of W1 for the last product
        small_load(sh.x, S::kLdH, p.w1[e] + (size_t)kSmallF * rank * kMlpH1, kMlpH1, kSmallF, kMlpH1);
        asm volatile("cp.async.commit_group;" ::: "memory");
    }
    T d1, d2, d3 = (T)0, v;
    small_activation<T>(p.activation, sh.h2[tid] + sh.h2[256 + tid] + sh.h2[512 + tid] + sh.h2[768 + tid] + bias1, &v, &d1);
    cluster_wait();      // (0)
#pragma unroll
    for (int q = 0; q < kSmallCtas; q++) store_remote(&sh.h1[atom * S::kLdH + kSmallC * rank + col], q, v);
    cluster_arrive();    // (1) A1 is everywhere, nobody reads its partial sums any more
    cluster_wait();
    // ---- layer 2 ----
    T* red = sh.w1c;
    small_product<T>(sh.h1, S::kLdH, sh.w2c, kSmallC, ap, cp, kg * 32, kg * 32 + 32, red + kg * 256);
    __syncthreads();
    small_activation<T>(p.activation, red[tid] + red[256 + tid] + red[512 + tid] + red[768 + tid] + bias2, &v, &d2);
#pragma unroll
    for (int q = 0; q < kSmallCtas; q++) store_remote(&sh.h2[atom * S::kLdH + kSmallC * rank + col], q, v);
    cluster_arrive();    // (2) A2
    cluster_wait();
    // ---- layer 3: own 8 columns, eight slices of K; its share of the energy, and dZ3 = w4 * D3 ----
    small_product<T>(sh.h2, S::kLdH, sh.w3c, kSmallC3, (tid >> 2) & 7, tid & 3, (tid >> 5) * 16, (tid >> 5) * 16 + 16,
                     red + (tid >> 5) * 128);
    __syncthreads();
    if (tid < kSmallTile * kSmallC3) {
        T s = bias3;
#pragma unroll
        for (int q = 0; q < 8; q++) s += red[q * 128 + tid];
        small_activation<T>(p.activation, s, &v, &d3);
        T share = v * out3;
#pragma unroll
        for (int o = 4; o > 0; o >>= 1) share += __shfl_xor_sync(kFull, share, o);
        if (col3 == 0) store_remote(&sh.epart[rank * kSmallTile + atom3], 0, share);
        if (backward) {
            const T g = p.grad_energy && atom3 < n_rows ? p.grad_energy[row0 + atom3] : (T)1;
            const T dz = g * out3 * d3;
#pragma unroll
            for (int q = 0; q < kSmallCtas; q++) store_remote(&sh.h3[atom3 * S::kLd3 + kSmallC3 * rank + col3], q, dz);
        }
    }
    cluster_arrive();    // (3) dZ3 and the energies
    cluster_wait();
    if (rank == 0 && tid < n_rows) {
        T s = bias4;
#pragma unroll
        for (int q = 0; q < kSmallCtas; q++) s += sh.epart[q * kSmallTile + tid];
        p.energy[row0 + tid] = s;
    }
    if (!backward) return;
    // ---- dZ2 = (dZ3 W3^T) * D2, own 16 columns ----
    small_product_t<T, 2>(sh.h3, S::kLd3, sh.w3r, S::kLd3, ap, cp, kg * 16, kg * 16 + 16, red + kg * 256);
    __syncthreads();
    v = (red[tid] + red[256 + tid] + red[512 + tid] + red[768 + tid]) * d2;
#pragma unroll
    for (int q = 0; q < kSmallCtas; q++) store_remote(&sh.h1[atom * S::kLdH + kSmallC * rank + col], q, v);
    cluster_arrive();    // (4) dZ2
    cluster_wait();
    // ---- dZ1 = (dZ2 W2^T) * D1 ----
    small_product_t<T, 2>(sh.h1, S::kLdH, sh.w2r, S::kLdH, ap, cp, kg * 32, kg * 32 + 32, red + kg * 256);
    __syncthreads();
    v = (red[tid] + red[256 + tid] + red[512 + tid] + red[768 + tid]) * d1;
#pragma unroll
    for (int q = 0; q < kSmallCtas; q++) store_remote(&sh.h2[atom * S::kLdH + kSmallC * rank + col], q, v);
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    cluster_arrive();    // (5) dZ1, and this CTA's rows of W1
    cluster_wait();
    // ---- own 48 columns of the feature gradient ----
    small_product_t<T, 6>(sh.h2, S::kLdH, sh.x, S::kLdH, ap, cp, kg * 32, kg * 32 + 32, red + kg * (kSmallTile * kSmallF));
    __syncthreads();
    for (int i = tid; i < n_rows * kSmallF; i += kSmallThreads) {
        constexpr int kAll = kSmallTile * kSmallF;
        p.grad_feat[(row0 + i / kSmallF) * kMlpIn + kSmallF * rank + i % kSmallF] =
            red[i] + red[kAll + i] + red[2 * kAll + i] + red[3 * kAll + i];
    }
}

}  // namespace ani
