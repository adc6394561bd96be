// AniSort on the device: stable sort of a batch's atoms by element id (a 2-bit key), returned
// as the three index arrays of the reference op (gpu_featurizer/ani_sort.cpp:71-115):
//   scatter[i] = rank of atom i among atoms of its element, gather[i] = element start + rank,
//   counts[4].
//
// The batch is cut into tiles of kSortTile consecutive atoms, one CTA per tile, one thread per
// atom.  Inside a tile the rank is a warp-level split: each warp ranks its 32-atom segment
// with one ballot per element and a popc of the lanes below, and a warp's base is the sum of the
// counts of the warps in front of it.  What differs between the two variants is
// where a tile learns how many atoms of each element precede it:
//   * single launch (batches up to kSortSingleLaunchMax atoms): every CTA recounts the whole
//     batch straight from the (L2-resident) input with wide, unrolled loads, so no scratch
//     memory and no second launch are needed;
//   * three launches (any size): a histogram kernel writes per-tile counts to a scratch
//     array of (tiles + 1) x 4 ints, one CTA scans it in place, and the ranking kernel reads
//     the scanned entry of its tile.
#pragma once

#include "ani_common.cuh"
#include "ani_launch.cuh"
#include "ani_mlp_pipe.cuh"

namespace ani {

constexpr int kSortThreads = 1024;
constexpr int kSortWarps = kSortThreads / kWarp;
constexpr int kSortTile = kSortThreads;                 // 1024 atoms per CTA
constexpr int kSortSingleLaunchMax = 64 * kSortTile;    // 65536 atoms

struct Count4 {
    int c[kTypes];
};

// Counts travel as four fields of one or two words: bytes within a thread (at most 65 atoms each), 16-bit pairs of the
// elements 0, 2 and 1, 3 within a warp, so that an atom costs a shift and an add and a sum over a warp one instruction a
// word.  Element by element (a compare and an add each, five shuffles a sum, and a scan over the warps by the first one)
// the kernel was a chain of shuffles and barriers: microseconds alone before -> now, 20 atoms 3.8 -> 1.9, 900 atoms 4.3 ->
// 2.2, 14 thousand 5.9 -> 2.8, 28 thousand 8.7 -> 3.8, 55 thousand 13.3 -> 5.1.  What is left is a launch, two reads of
// the L2 cache one behind the other and one barrier.
struct Pair16 {
    unsigned even, odd;      // elements 0 | 2 << 16 and 1 | 3 << 16
};
// 1 in the byte of the element (the funnel shift takes its distance modulo 32: elements modulo 4, as checked_type has them)
__device__ __forceinline__ unsigned one_byte(int t) { return __funnelshift_l(0u, 1u, 8 * t); }
__device__ __forceinline__ Pair16 widen(unsigned bytes) { return Pair16{bytes & 0x00ff00ffu, (bytes >> 8) & 0x00ff00ffu}; }
__device__ __forceinline__ Pair16 warp_sum(Pair16 v)
{
    return Pair16{__reduce_add_sync(kFull, v.even), __reduce_add_sync(kFull, v.odd)};
}
__device__ __forceinline__ Count4 unpack(Pair16 v)
{
    return Count4{{(int)(v.even & 0xffffu), (int)(v.odd & 0xffffu), (int)(v.even >> 16), (int)(v.odd >> 16)}};
}

struct SortShared {
    uint4 counted[kSortWarps];     // per warp: what it counted in front of the tile and in all
    Pair16 own[kSortWarps];        // per warp: its atoms of the tile
};

// Byte counts of types[0, n), n <= kSortSingleLaunchMax: everything (`total`) and the part in front of
// `split` (`before`), a multiple of 4.  Loads are 16 bytes wide and issued four
// at a time so that their L2 latencies overlap.
__device__ __forceinline__ void count_two_ranges(const int* __restrict__ types, int n, int split,
                                                 unsigned* before, unsigned* total)
{
    unsigned vb = 0u, vt = 0u, seen = 0u;
    const bool aligned = (reinterpret_cast<uintptr_t>(types) & 15u) == 0;
    const int nvec = aligned ? n / 4 : 0;
    const int4* p4 = reinterpret_cast<const int4*>(types);
    constexpr int kUnroll = 4;
    for (int k0 = threadIdx.x; k0 < nvec; k0 += kSortThreads * kUnroll) {
        int4 q[kUnroll];
#pragma unroll
        for (int u = 0; u < kUnroll; u++) {
            const int k = k0 + u * kSortThreads;
            q[u] = k < nvec ? p4[k] : make_int4(0, 0, 0, 0);
        }
#pragma unroll
        for (int u = 0; u < kUnroll; u++) {
            const int k = k0 + u * kSortThreads;
            const unsigned v = one_byte(q[u].x) + one_byte(q[u].y) + one_byte(q[u].z) + one_byte(q[u].w);
            seen |= (unsigned)(q[u].x | q[u].y | q[u].z | q[u].w);
            if (k < nvec) vt += v;
            if (k < nvec && 4 * k < split) vb += v;
        }
    }
    for (int k = nvec * 4 + threadIdx.x; k < n; k += kSortThreads) {
        const int t = types[k];
        seen |= (unsigned)t;
        vt += one_byte(t);
        if (k < split) vb += one_byte(t);
    }
    if (seen >= (unsigned)kTypes) report(ANI_ERR_BAD_ELEMENT);
    *before = vb;
    *total = vt;
}

// An atom's rank among the atoms of its element in its warp, and the warp's counts.  t = -1: no atom.
__device__ __forceinline__ int rank_in_warp(int t, Pair16* counts)
{
    unsigned m[kTypes], mine = 0u;
#pragma unroll
    for (int g = 0; g < kTypes; g++) {
        m[g] = __ballot_sync(kFull, t == g);
        if (t == g) mine = m[g];
    }
    *counts = Pair16{(unsigned)(__popc(m[0]) | __popc(m[2]) << 16), (unsigned)(__popc(m[1]) | __popc(m[3]) << 16)};
    return __popc(mine & lanemask_lt());
}

// Atoms of each element in the warps of the tile in front of this one; `own` holds every warp's counts.
__device__ __forceinline__ Count4 warps_in_front(const Pair16* own)
{
    const Pair16 v = own[lane_id()];
    const bool front = lane_id() < warp_id();
    return unpack(warp_sum(Pair16{front ? v.even : 0u, front ? v.odd : 0u}));
}

__device__ __forceinline__ void place_atom(int i, int t, int rank, const Count4& before, const Count4& in_tile,
                                           const Count4& total, int* __restrict__ scatter, int* __restrict__ gather)
{
    int start = 0;
#pragma unroll
    for (int g = 0; g < kTypes; g++) {
        if (t == g) {
            const int r = before.c[g] + in_tile.c[g] + rank;
            scatter[i] = r;
            gather[i] = start + r;
        }
        start += total.c[g];
    }
}

// Tile `tile` of a single-launch sort.
__device__ __forceinline__ void sort_tile(const int* __restrict__ types, int n_atoms, int tile, int* __restrict__ scatter,
                                          int* __restrict__ gather, int* __restrict__ counts, SortShared& sh)
{
    static_assert(kSortSingleLaunchMax / kSortThreads + 1 <= 255, "a byte per element and thread");
    static_assert(kSortSingleLaunchMax - kSortTile < 1 << 16, "16 bits for what lies in front of a tile");
    const int lane = lane_id(), warp = warp_id();
    const int i = tile * kSortTile + threadIdx.x;
    const int t = i < n_atoms ? types[i] & 3 : -1;      // (bad elements are reported where everything is counted)
    unsigned vb, vt;
    count_two_ranges(types, n_atoms, tile * kSortTile, &vb, &vt);
    Pair16 own;
    const int rank = rank_in_warp(t, &own);
    const Pair16 warp_before = warp_sum(widen(vb)), warp_total = warp_sum(widen(vt));
    if (lane == 0) {
        sh.counted[warp] = make_uint4(warp_before.even, warp_before.odd, warp_total.even, warp_total.odd);
        sh.own[warp] = own;
    }
    __syncthreads();
    const uint4 v = sh.counted[lane];
    const Count4 before = unpack(warp_sum(Pair16{v.x, v.y})), in_tile = warps_in_front(sh.own);
    Count4 total = unpack(Pair16{v.z, v.w});      // a whole batch of one element may be 2^16 atoms
#pragma unroll
    for (int g = 0; g < kTypes; g++) total.c[g] = __reduce_add_sync(kFull, total.c[g]);
    if (tile == 0 && threadIdx.x == 0) {
#pragma unroll
        for (int g = 0; g < kTypes; g++) counts[g] = total.c[g];
    }
    if (t >= 0) place_atom(i, t, rank, before, in_tile, total, scatter, gather);
}

// Single launch: grid = number of tiles.
__global__ void __launch_bounds__(kSortThreads)
    sort_single_kernel(const int* __restrict__ types, int n_atoms, int* __restrict__ scatter,
                       int* __restrict__ gather, int* __restrict__ counts)
{
    __shared__ SortShared sh;
    pdl_wait();
    sort_tile(types, n_atoms, blockIdx.x, scatter, gather, counts, sh);
    pdl_trigger();
}

// The same with the weight packing of a pass in the CTAs behind the tiles: the two have nothing to do with
// one another, either is bound by latency (5 us and 3 us) and together they fill a wave of the device.
__global__ void __launch_bounds__(kSortThreads)
    sort_and_pack_kernel(const int* __restrict__ types, int n_atoms, int n_tiles, int* __restrict__ scatter,
                         int* __restrict__ gather, int* __restrict__ counts, const MlpPackParams pack)
{
    __shared__ SortShared sh;
    pdl_wait();     // no early trigger: the kernel writes weights
    if ((int)blockIdx.x >= n_tiles) {
        const int c = (int)blockIdx.x - n_tiles;
        pack_chunk(pack, c % kPackChunks, c / kPackChunks);
        return;
    }
    sort_tile(types, n_atoms, blockIdx.x, scatter, gather, counts, sh);
}

// Large batches, first: per-tile element counts into scratch[tile][4].
__global__ void __launch_bounds__(kSortThreads)
    sort_histogram_kernel(const int* __restrict__ types, int n_atoms, int* __restrict__ tile_counts)
{
    __shared__ Pair16 red[kSortWarps];
    const int tile = blockIdx.x, i = tile * kSortTile + threadIdx.x;
    Pair16 own;
    rank_in_warp(i < n_atoms ? checked_type(types[i]) : -1, &own);
    if (lane_id() == 0) red[warp_id()] = own;
    __syncthreads();
    if (warp_id() == 0) {
        const Count4 c = unpack(warp_sum(red[lane_id()]));
        if (threadIdx.x == 0) {
#pragma unroll
            for (int g = 0; g < kTypes; g++) tile_counts[tile * kTypes + g] = c.c[g];
        }
    }
}

// Large batches, second: exclusive scan over tiles, in place, by one CTA.  On return
// tile_counts[tile] holds the counts in front of the tile and tile_counts[n_tiles] the totals.
__global__ void __launch_bounds__(kSortThreads)
    sort_scan_kernel(int* __restrict__ tile_counts, int n_tiles)
{
    __shared__ int warp_tot[kSortWarps][kTypes];
    __shared__ int carry[kTypes];
    const int lane = lane_id(), warp = warp_id();
    if (threadIdx.x < kTypes) carry[threadIdx.x] = 0;
    __syncthreads();
    for (int k0 = 0; k0 < n_tiles; k0 += kSortThreads) {
        const int k = k0 + threadIdx.x;
        int v[kTypes], incl[kTypes];
#pragma unroll
        for (int g = 0; g < kTypes; g++) {
            v[g] = k < n_tiles ? tile_counts[k * kTypes + g] : 0;
            int x = v[g];
#pragma unroll
            for (int o = 1; o < kWarp; o <<= 1) {
                const int y = __shfl_up_sync(kFull, x, o);
                if (lane >= o) x += y;
            }
            incl[g] = x;
            if (lane == kWarp - 1) warp_tot[warp][g] = x;
        }
        __syncthreads();
#pragma unroll
        for (int g = 0; g < kTypes; g++) {
            int base = carry[g];
            for (int w = 0; w < warp; w++) base += warp_tot[w][g];
            if (k < n_tiles) tile_counts[k * kTypes + g] = base + incl[g] - v[g];
        }
        __syncthreads();
        if (threadIdx.x < kTypes) {
            int s = carry[threadIdx.x];
            for (int w = 0; w < kSortWarps; w++) s += warp_tot[w][threadIdx.x];
            carry[threadIdx.x] = s;
        }
        __syncthreads();
    }
    if (threadIdx.x < kTypes) tile_counts[n_tiles * kTypes + threadIdx.x] = carry[threadIdx.x];
}

// Large batches, third: rank each tile from the scanned counts.
__global__ void __launch_bounds__(kSortThreads)
    sort_rank_kernel(const int* __restrict__ types, int n_atoms,
                     const int* __restrict__ tile_counts, int n_tiles, int* __restrict__ scatter,
                     int* __restrict__ gather, int* __restrict__ counts)
{
    __shared__ Pair16 red[kSortWarps];
    const int tile = blockIdx.x, i = tile * kSortTile + threadIdx.x;
    const int t = i < n_atoms ? types[i] & 3 : -1;      // (bad elements were reported by the histogram)
    Count4 before, total;
#pragma unroll
    for (int g = 0; g < kTypes; g++) {
        before.c[g] = tile_counts[tile * kTypes + g];
        total.c[g] = tile_counts[n_tiles * kTypes + g];
    }
    if (tile == 0 && threadIdx.x == 0) {
#pragma unroll
        for (int g = 0; g < kTypes; g++) counts[g] = total.c[g];
    }
    Pair16 own;
    const int rank = rank_in_warp(t, &own);
    if (lane_id() == 0) red[warp_id()] = own;
    __syncthreads();
    const Count4 in_tile = warps_in_front(red);
    if (t >= 0) place_atom(i, t, rank, before, in_tile, total, scatter, gather);
}

// n_atoms == 0: the reference still returns atom_counts = {0, 0, 0, 0}.
__global__ void sort_empty_kernel(int* counts)
{
    if (threadIdx.x < kTypes) counts[threadIdx.x] = 0;
}

}  // namespace ani
