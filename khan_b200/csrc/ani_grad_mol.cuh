// Coordinate-gradient kernel for batches of small molecules (at most 32 atoms each).
//
// One CTA per molecule, NW warps that share every step evenly, whatever the molecule's neighbourhoods look like:
//   - the upstream values come with 16-byte asynchronous copies (cp.async), requested as soon as elements and rows are known:
//     the radial ones of every atom, the angular ones of as many central atoms as a batch may have;
//   - pairs of atoms: lane = unordered pair.  The radial derivatives of both directions are one contraction with the SUM of
//     the two atoms' upstream values, and the pairs within A_Rc set a bit in both atoms' neighbour masks;
//   - the central atoms go in BATCHES (limits in MolGradCfg; most molecules are one batch).  Per batch:
//       entries  lane = (central atom, neighbour): unit vector, distance and cutoff into the list;
//       pairs    lane = (central atom, neighbours a and b), all pairs of the batch in one numbering, so that all lanes of
//                all warps work but for the last 32 pairs: the 32 upstream values contract to (dL/dcos, dL/dr_a, dL/dr_b);
//       forces   lane = entry: sums over the k - 1 pairs it is in, in a fixed order;
//       sums     lane = atom: what the central atoms hand to it less what it hands out.
// Every output value is written once, nothing is accumulated with atomics, the outputs need no zero fill and the result is
// bit-reproducible.
//
// Before, a warp took central atoms of its own, three at a time, with a lane per neighbour: 73 % of the lanes busy in the
// pairs, and the warps of a large molecule (a cost that grows with the cube of its size) went on alone.  Microseconds alone,
// before -> now: float, 1 molecule 8.5 -> 7.0, 64: 14.6 -> 10.6, 592: 20.5 -> 18.9, 1024: 34.3 -> 27.1, 2048: 49.1 -> 41.4;
// double, 1: 18.8 -> 13.7, 64: 34.9 -> 23.5, 500: 50.8 -> 39.6, 1024: 78.3 -> 62.2.  Beside other launches (eight streams)
// 1024 molecules 18.5 -> 18.5, 2048: 37.0 -> 36.8, 148: 4.0 -> 3.6; double, 1024: 59.7 -> 56.4.  There it was slower at
// first (1024 molecules 19.9, 2048: 39.7): every warp sought the molecule of its CTA, which the first warp now does for all
// (0.2 us), and the central atom of every list entry, which is now written with the entry (0.75 us); and the sums at the
// end tested every place of their tables, which are now without gaps and read four values at a time, the radial part beside
// the forces of the first batch (0.5 us).  What bounds it: instruction issue (1002 an atom, in a cold capture 0.55 a cycle
// and scheduler, the busiest 1.36 times the average), held up by shared memory (half of its wavefronts, the upstream values
// of 32 lanes with different element pairs) and barriers, and, for one molecule, the chain of eight steps.
//
// A molecule with more than 32 atoms met by this kernel goes through the streaming routines
// (zero fill by its own CTA, then global atomics, all inside the CTA).
//
// Computes what featurize_grad_cpu of the reference computes
// (gpu_featurizer/kernel_cpu.cpp:217-366).
#pragma once

#include "ani_common.cuh"
#include "ani_featurize_mol.cuh"
#include "ani_grad.cuh"

namespace ani {

__device__ __forceinline__ void cp_async16(void* smem_dst, const void* gmem_src)
{
    const unsigned s = (unsigned)__cvta_generic_to_shared(smem_dst);
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(s), "l"(gmem_src) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N> __device__ __forceinline__ void cp_async_wait()
{
    asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory");
}

constexpr int kMolGradPitch = kMolMaxAtoms + 4;      // rows in 16-byte reads, rows and columns conflict-free
constexpr int kMolGradRow = kPairBuckets * kGradBucketStride;

// CTAS of them fit an SM.  What the tables of one hold of a batch: upstream rows, list entries, neighbour pairs.  A batch
// takes at least one atom with 31 neighbours, so kEntries >= 31 and kSlots >= 465.  With twelve warps the tables are for the
// whole molecule, but for the largest; with eight, for most.  More batches cost
// barriers and pairs short of 32: 1024 molecules in float take 27 us with these tables, and 43 (when it was 29.5 with them)
// with 8 rows, 160 entries and 512 pairs and four warps.  (One CTA in double: with 512 entries its 197 KB leave less of the
// first-level cache, 500 molecules 41.7 us instead of 39.6.)
template <typename T, int NW, int CTAS> struct MolGradCfg {
    static constexpr bool kFloat = sizeof(T) == 4;
    static constexpr int kRows = NW == 12 ? (kFloat ? (CTAS == 1 ? 32 : 28) : 24) : (kFloat ? 14 : 12);
    static constexpr int kEntries = NW == 12 ? (kFloat ? (CTAS == 1 ? 512 : 384) : 448) : (kFloat ? 224 : 256);
    static constexpr int kSlots = NW == 12 ? (kFloat ? (CTAS == 1 ? 3072 : 2560) : 2048) : 1024;
    static constexpr int kRadPitch = kRadial + 16 / (int)sizeof(T);   // rows of 64 values, conflict-free in 16-byte reads
    static_assert(kRows >= 1 && kEntries >= kMolMaxAtoms - 1 && kEntries < 1 << 12 && kSlots < 1 << 13 &&
                  kSlots >= (kMolMaxAtoms - 1) * (kMolMaxAtoms - 2) / 2, "any atom fits a batch");
};

template <typename T, int NW, int CTAS> struct MolGradShared {
    using Cfg = MolGradCfg<T, NW, CTAS>;
    alignas(16) T g[Cfg::kRows][kMolGradRow];     // angular upstream values, blocks of 32 at stride 36
    // row d of a central atom with k neighbours, place a: dL/dcos(theta) and the part along bond a of the pairs
    // (a, a + d) and (a - d, a)
    alignas(32) Vec2<T> pair[2 * Cfg::kSlots];
    Vec4<T> u[Cfg::kEntries], w[Cfg::kEntries];   // unit vector and r; 1 / r, f_C, f_C', element
    alignas(16) T force[Cfg::kRows][3][kMolGradPitch];        // of a central atom of the batch on an atom (0: not within A_Rc)
    alignas(16) T radial[kMolMaxAtoms][kMolGradPitch];        // dL/dr / r of two atoms
    alignas(16) T xyz[3][kMolMaxAtoms];
    int4 molecule;                                // number (< 0: none), atoms, first atom, usable
    int type[kMolMaxAtoms];
    unsigned near[kMolMaxAtoms];                  // atoms within A_Rc
    unsigned short list[kMolMaxAtoms * (kMolMaxAtoms - 1)];   // the same as a list of all of them: atom | neighbour << 8
    // the radial upstream values lie over the pairs: they have been used before the first pair
    __device__ __forceinline__ T* rad(int c) { return &pair[0].x + c * Cfg::kRadPitch; }
    static_assert(sizeof(T) * kMolMaxAtoms * Cfg::kRadPitch <= sizeof(pair), "radial rows");
};

// Bucket of the element pair (ta, tb), four bits per entry of the 4 x 4 table.
constexpr unsigned long long kBucketLut =
    0x0ull | (0x1ull << 4) | (0x2ull << 8) | (0x3ull << 12) | (0x1ull << 16) | (0x4ull << 20) | (0x5ull << 24) |
    (0x6ull << 28) | (0x2ull << 32) | (0x5ull << 36) | (0x7ull << 40) | (0x8ull << 44) | (0x3ull << 48) |
    (0x6ull << 52) | (0x8ull << 56) | (0x9ull << 60);
__device__ __forceinline__ int bucket_of(int ta, int tb) { return (int)(kBucketLut >> (4 * (ta * kTypes + tb))) & 15; }

// Radial part of the gradient of one central atom of a LARGE molecule, with global atomics
// (the angular part is grad_atom_streaming of ani_grad.cuh).  g = upstream row in shared memory.
template <typename T>
__device__ __noinline__ void grad_atom_streaming_radial(const T* __restrict__ xs, const T* __restrict__ ys,
                                                        const T* __restrict__ zs, const int* __restrict__ types,
                                                        int base, int n, int i, const T* g, T* gx, T* gy, T* gz)
{
    const int lane = lane_id();
    const T xi = xs[base + i], yi = ys[base + i], zi = zs[base + i];
    T fix = (T)0, fiy = (T)0, fiz = (T)0;
    for (int j0 = 0; j0 < n; j0 += kWarp) {
        const int j = j0 + lane;
        if (j < n && j != i) {
            const T dx = xi - xs[base + j], dy = yi - ys[base + j], dz = zi - zs[base + j];
            T r, inv;
            length_and_inverse(dx * dx + dy * dy + dz * dz, &r, &inv);
            if (r < (T)kR_Rc) {
                T fc, dfc;
                cutoff<T>(r, (T)kR_Rc, &fc, &dfc);
                const T d = radial_vjp_dev<T>(r, fc, dfc, g + (types[base + j] & 3) * kNumRs);
                const T fx = d * dx * inv, fy = d * dy * inv, fz = d * dz * inv;
                fix += fx; fiy += fy; fiz += fz;
                atomicAdd(&gx[base + j], -fx);
                atomicAdd(&gy[base + j], -fy);
                atomicAdd(&gz[base + j], -fz);
            }
        }
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        fix += __shfl_xor_sync(kFull, fix, o);
        fiy += __shfl_xor_sync(kFull, fiy, o);
        fiz += __shfl_xor_sync(kFull, fiz, o);
    }
    if (lane == 0) {
        atomicAdd(&gx[base + i], fix);
        atomicAdd(&gy[base + i], fiy);
        atomicAdd(&gz[base + i], fiz);
    }
}

// Molecule energies on the side: a pass that wants energies and forces has one launch less (2 to 3 us), and the warp
// that takes none of the three output planes at the end has nothing else to do.  mol_energy == nullptr: none.
template <typename T> struct MolEnergySums {
    const T* atom_energy_sorted;
    const int* gather;
    T* mol_energy;
};

// Molecules whose CTAs are put into order of size, when not all molecules are resident at once.  Without the order 1024
// molecules in float take 32.5 us alone instead of 27.1, in double 78.6 instead of 62.2; with eight streams in flight, where
// other batches fill the gaps, 18.0 instead of 18.5 and 55.6 instead of 56.4.
constexpr int kMolGradOrder = 16;

// length_and_inverse with one Newton step on the SFU's reciprocal root in float: the distances are computed once per pair
// of atoms here, and their error is what the Gaussians enlarge most.
__device__ __forceinline__ void refined_length_and_inverse(float d2, float* r, float* inv)
{
    const float rs = d2 > 0.0f ? sfu_rsqrt(d2) : 0.0f;
    const float h = d2 * rs;
    const float e = fmaf(-h, rs, 1.0f);             // 1 - d2 rs^2
    *inv = fmaf(0.5f * rs, e, rs);
    *r = fmaf(0.5f * h, e, h);
}
__device__ __forceinline__ void refined_length_and_inverse(double d2, double* r, double* inv) { length_and_inverse(d2, r, inv); }

// The lane (central atom) among `members` whose range of a prefix sum holds `first + lane`; off = where the range of this
// lane's atom starts.  All lanes call it; `first + lane` must lie inside the total.
__device__ __forceinline__ int owner_of(unsigned members, int off, int first, int index)
{
    const bool member = (members >> lane_id()) & 1u;
    const int lo = 31 - __clz(__ballot_sync(kFull, member && off <= first));
    const int hi = 31 - __clz(__ballot_sync(kFull, member && off <= first + kWarp - 1));
    int c = lo;
    for (int q = lo + 1; q <= hi; q++) c += index >= __shfl_sync(kFull, off, q) ? 1 : 0;
    return c;
}

// early_inputs: nothing less than two kernels back writes coordinates, elements, rows or the molecule table: they are read,
// and the distances formed, ahead of the kernel before this one, whose upstream values come last.  Energies + forces of one
// molecule 32.3 -> 31.0 us.
template <typename T, int NW, int CTAS>
__global__ void __launch_bounds__(NW* kWarp, CTAS)
    featurize_grad_mol_kernel(const T* __restrict__ xs, const T* __restrict__ ys, const T* __restrict__ zs,
                              const int* __restrict__ types, const int* __restrict__ mol_offsets,
                              const int* __restrict__ mol_counts, int n_mols, int n_atoms,
                              const int* __restrict__ scatter, const T* gh, const T* gc, const T* gn, const T* go,
                              T* gx, T* gy, T* gz, int acs0, int acs1, int acs2, int acs3,
                              const MolEnergySums<T> sums, bool early_inputs)
{
    using Cfg = MolGradCfg<T, NW, CTAS>;
    constexpr int kThreads = NW * kWarp;
    extern __shared__ __align__(128) unsigned char smem_raw[];
    MolGradShared<T, NW, CTAS>& sh = *reinterpret_cast<MolGradShared<T, NW, CTAS>*>(smem_raw);
    const int lane = lane_id(), warp = warp_id();
    if (!early_inputs) pdl_wait();

    // In a grid of (X, Y) CTAs the molecules i, i + X, i + 2 X ... share the CTAs (i, 0), (i, 1), (i, 2) ... in order of
    // their sizes: CTAs start in index order, so the expensive molecules start first and the cheap ones fill the SMs
    // behind them.  The first warp of a CTA finds its molecule from the Y sizes; only the CTAs behind the end of the
    // batch have none.
    int m = blockIdx.x;
    MolRange mol;
    bool usable;
    if (gridDim.y == 1) {
        usable = load_molecule(mol_offsets, mol_counts, m, n_atoms, &mol);
    } else {
        if (warp == 0) {
            const int mine = blockIdx.x + lane * gridDim.x;
            const bool there = lane < kMolGradOrder && mine < n_mols;
            const int size = there ? mol_counts[mine] : 0, first = there ? mol_offsets[mine] : 0;
            // the blockIdx.y-th largest, bit by bit (all above 32 atoms alike)
            const int key = min(max(size, 0), 63);
            unsigned left = __ballot_sync(kFull, there);
            int y = blockIdx.y;
            const bool exists = y < __popc(left);
#pragma unroll
            for (int bit = 5; bit >= 0; bit--) {
                const unsigned with = __ballot_sync(kFull, (key >> bit) & 1) & left;
                const int c = __popc(with);
                if (y < c) left = with;
                else {
                    y -= c;
                    left &= ~with;
                }
            }
            if (exists && ((left >> lane) & 1u) && __popc(left & lanemask_lt()) == y) {
                usable = check_molecule(size, first, n_atoms, &mol);
                sh.molecule = make_int4(mine, mol.n, mol.base, usable ? 1 : 0);
            }
            if (!exists && lane == 0) sh.molecule = make_int4(-1, 0, 0, 0);
        }
        __syncthreads();
        const int4 found = sh.molecule;
        m = found.x;
        mol.n = found.y;
        mol.base = found.z;
        usable = found.w != 0;
        if (m < 0) return;
    }
    if (!usable) {
        pdl_wait();
        if (sums.mol_energy && threadIdx.x == 0) sums.mol_energy[m] = (T)0;
        return;
    }
    const int n = mol.n, base = mol.base;

    T energy = (T)0;      // of the molecule, summed by the last warp and written at the end
    auto load_energy = [&] {
        if (!sums.mol_energy || warp != NW - 1) return;
        for (int i = lane; i < n; i += kWarp) {
            const int g = sums.gather[base + i];
            if (g >= 0 && g < n_atoms) energy += load_fresh(sums.atom_energy_sorted + g);
            else report(ANI_ERR_BAD_INDEX);
        }
    };
    auto write_energy = [&] {
        if (!sums.mol_energy || warp != NW - 1) return;
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) energy += __shfl_xor_sync(kFull, energy, o);
        if (lane == 0) sums.mol_energy[m] = energy;
    };

    if (n > kMolMaxAtoms) {   // a large molecule in a batch of small ones
        pdl_wait();
        load_energy();
        write_energy();
        for (int j = threadIdx.x; j < n; j += kThreads) {
            gx[base + j] = (T)0;
            gy[base + j] = (T)0;
            gz[base + j] = (T)0;
        }
        __syncthreads();
        T* g = reinterpret_cast<T*>(smem_raw) + warp * kGradRowWords;
        static_assert(NW * kGradRowWords * sizeof(T) <= sizeof(MolGradShared<T, NW, CTAS>), "a row per warp");
        for (int i = warp; i < n; i += NW) {
            const int gi = base + i;
            const int ti = checked_type(types[gi]);
            const int srow = scatter[gi];
            const int cap = ti == 0 ? acs0 : (ti == 1 ? acs1 : (ti == 2 ? acs2 : acs3));
            if (srow < 0 || srow >= cap) {
                if (lane == 0) report(ANI_ERR_BAD_INDEX);
                continue;
            }
            const T* grow = (ti == 0 ? gh : (ti == 1 ? gc : (ti == 2 ? gn : go))) + (size_t)srow * kTotal;
            g[lane] = load_fresh(grow + lane);
            g[32 + lane] = load_fresh(grow + 32 + lane);
            for (int bk = 0; bk < kPairBuckets; bk++)
                g[kRadial + bk * kGradBucketStride + lane] = load_fresh(grow + kRadial + bk * kTS + lane);
            __syncwarp();
            grad_atom_streaming_radial<T>(xs, ys, zs, types, base, n, i, g, gx, gy, gz);
            grad_atom_streaming<T>(xs, ys, zs, types, base, n, i, g, gx, gy, gz);
            __syncwarp();
        }
        return;
    }

    // ---- the molecule: lane = atom in every warp (element and row), coordinates in shared memory ----
    int my_type = 0, my_row = -1;
    if (lane < n) {
        my_type = types[base + lane];
        my_row = scatter[base + lane];
    }
    if (threadIdx.x < n) {      // warp 0
        sh.xyz[0][lane] = xs[base + lane];
        sh.xyz[1][lane] = ys[base + lane];
        sh.xyz[2][lane] = zs[base + lane];
        sh.near[lane] = 0u;
        sh.radial[lane][lane] = (T)0;
        for (int j = n; j & 3; j++) sh.radial[lane][j] = (T)0;      // rows are read four values at a time
    }
    if (my_type < 0 || my_type >= kTypes) my_type = warp == 0 ? checked_type(my_type) : my_type & 3;
    {
        const int cap = my_type == 0 ? acs0 : (my_type == 1 ? acs1 : (my_type == 2 ? acs2 : acs3));
        if (lane < n && (my_row < 0 || my_row >= cap)) {
            if (warp == 0) report(ANI_ERR_BAD_INDEX);
            my_row = -1;
        }
    }
    if (threadIdx.x < n) sh.type[lane] = my_type;
    const unsigned ok_mask = __ballot_sync(kFull, my_row >= 0);   // atoms that have an upstream row
    const unsigned long long my_src = reinterpret_cast<unsigned long long>(
        (my_type == 0 ? gh : (my_type == 1 ? gc : (my_type == 2 ? gn : go))) + (my_row >= 0 ? (size_t)my_row * kTotal : 0));

    // upstream values, 16 bytes per copy: the radial ones of every atom, the angular ones of the rows [r0, r1)
    constexpr int kPiece = 16 / (int)sizeof(T), kRadPieces = kRadial / kPiece, kPieces = kTotal / kPiece;
    auto row_of = [&](int c) -> const T* {
        return reinterpret_cast<const T*>(__shfl_sync(kFull, my_src, c));
    };
    auto request_angular = [&](const T* src, T* dst) {
#pragma unroll
        for (int s = 0; s < (kPieces - kRadPieces + kWarp - 1) / kWarp; s++) {
            const int v = (lane + s * kWarp) * kPiece;
            if (v < kAngular) cp_async16(dst + (v >> 5) * kGradBucketStride + (v & 31), src + kRadial + v);
        }
    };
    int r0 = 0, r1 = min(n, Cfg::kRows);
    auto request_first = [&] {
        for (int c = warp; c < n; c += NW) {
            const T* src = row_of(c);
            if (lane < kRadPieces) {
                if ((ok_mask >> c) & 1u) cp_async16(sh.rad(c) + lane * kPiece, src + lane * kPiece);
                else
#pragma unroll
                    for (int q = 0; q < kPiece; q++) sh.rad(c)[lane * kPiece + q] = (T)0;
            }
            if (c < r1 && ((ok_mask >> c) & 1u)) request_angular(src, sh.g[c]);
        }
        cp_async_commit();
    };
    if (!early_inputs) request_first();
    auto clear_forces = [&] {
        for (int i = threadIdx.x; i < min(n, Cfg::kRows) * (int)(sizeof(sh.force[0]) / 16); i += kThreads)
            reinterpret_cast<Vec4<float>*>(sh.force)[i] = Vec4<float>{0.f, 0.f, 0.f, 0.f};
    };
    clear_forces();
    __syncthreads();

    // ---- every two atoms once: pair p of n (n - 1) / 2 is (i, i + d mod n), d = 1, 2 ... ----
    constexpr int kMaxPairs = (kMolMaxAtoms * (kMolMaxAtoms - 1) / 2 + kThreads - 1) / kThreads;
    const int n_pairs = n * (n - 1) / 2;
    const unsigned recip = (unsigned)(65536.0f * __frcp_rn((float)n)) + 1u;
    T pr[kMaxPairs], pinv[kMaxPairs];
    int pij[kMaxPairs];
#pragma unroll
    for (int s = 0; s < kMaxPairs; s++) {
        const int p = s * kThreads + threadIdx.x;
        if (p < n_pairs) {
            const int d0 = (int)(((unsigned)p * recip) >> 16), i = p - d0 * n;
            int j = i + d0 + 1;
            if (j >= n) j -= n;
            const T dx = sh.xyz[0][i] - sh.xyz[0][j], dy = sh.xyz[1][i] - sh.xyz[1][j], dz = sh.xyz[2][i] - sh.xyz[2][j];
            refined_length_and_inverse(dx * dx + dy * dy + dz * dz, &pr[s], &pinv[s]);
            pij[s] = i | (j << 8);
            if (pr[s] < (T)kA_Rc) {
                atomicOr(&sh.near[i], 1u << j);
                atomicOr(&sh.near[j], 1u << i);
            }
        }
    }
    if (early_inputs) {
        pdl_wait();
        request_first();
    }
    load_energy();      // (the last warp has no pair of atoms in most molecules)
    cp_async_wait<0>();
    __syncthreads();
    // lane = central atom: its neighbours and pairs, and where they start in the molecule's numbering
    const unsigned my_near = lane < n ? sh.near[lane] : 0u;
    const int my_k = (ok_mask >> lane) & 1u ? __popc(my_near) : 0, my_pairs = my_k * (my_k - 1) / 2;
    int incl = my_k | (my_pairs << 12);      // at most 992 neighbours
#pragma unroll
    for (int o = 1; o < kWarp; o <<= 1) {
        const int y = __shfl_up_sync(kFull, incl, o);
        if (lane >= o) incl += y;
    }
    const int excl = incl - (my_k | (my_pairs << 12));
    const int k_first = excl & 0xfff, p_first = excl >> 12, k_end = incl & 0xfff, p_end = incl >> 12;
#pragma unroll
    for (int s = 0; s < kMaxPairs; s++) {
        const int p = s * kThreads + threadIdx.x;
        if (s * kThreads + warp * kWarp >= n_pairs) break;
        const int i = p < n_pairs ? pij[s] & 0xff : 0, j = p < n_pairs ? pij[s] >> 8 : 0;
        const int at_i = __shfl_sync(kFull, k_first, i), at_j = __shfl_sync(kFull, k_first, j);
        if (p < n_pairs) {
            T force = (T)0;
            if (pr[s] < (T)kR_Rc) {
                T fc, dfc;
                cutoff<T>(pr[s], (T)kR_Rc, &fc, &dfc);
                const T *wi = sh.rad(i) + sh.type[j] * kNumRs, *wj = sh.rad(j) + sh.type[i] * kNumRs;
                T w[kNumRs], v[4];
#pragma unroll
                for (int q = 0; q < kNumRs; q += 4) {
                    load4(wi + q, w + q);
                    load4(wj + q, v);
#pragma unroll
                    for (int k = 0; k < 4; k++) w[q + k] += v[k];
                }
                force = radial_vjp_dev<T>(pr[s], fc, dfc, w) * pinv[s];
            }
            sh.radial[i][j] = force;
            sh.radial[j][i] = force;
            if (pr[s] < (T)kA_Rc) {
                if ((ok_mask >> i) & 1u) sh.list[at_i + __popc(sh.near[i] & ((1u << j) - 1u))] = (unsigned short)(i | j << 8);
                if ((ok_mask >> j) & 1u) sh.list[at_j + __popc(sh.near[j] & ((1u << i) - 1u))] = (unsigned short)(j | i << 8);
            }
        }
    }
    const unsigned k_recip = (unsigned)(65536.0f * __frcp_rn((float)max(my_k, 1))) + 1u;
    __syncthreads();

    // the last three warps, lane = atom: one component of its gradient.  The radial part first, beside the first batch's forces
    const int plane = warp - (NW - 3);
    T sum = (T)0;
    int c0 = 0;
    auto batch_end = [&](int from) {
        const int k0 = __shfl_sync(kFull, k_first, from), p0 = __shfl_sync(kFull, p_first, from);
        const bool fits = lane >= from && lane < n && lane - from < Cfg::kRows && k_end - k0 <= Cfg::kEntries &&
                          p_end - p0 <= Cfg::kSlots;
        return from + __popc(__ballot_sync(kFull, fits));
    };
    int c1 = batch_end(0);
    while (true) {
        const unsigned members = low_lanes(c1) & ~low_lanes(c0);
        const int k0 = __shfl_sync(kFull, k_first, c0), p0 = __shfl_sync(kFull, p_first, c0);
        const int n_entries = __shfl_sync(kFull, k_end, c1 - 1) - k0, n_slots = __shfl_sync(kFull, p_end, c1 - 1) - p0;
        const int my_entry = k_first - k0, my_slot = p_first - p0, my_at = my_slot | (my_k << 13) | (my_entry << 19);
        // ---- list entries of the batch, lane = entry ----
        for (int first = warp * kWarp; first < n_entries; first += kThreads) {
            const int e = min(first + lane, n_entries - 1);
            const int at = sh.list[k0 + e], c = at & 0xff, j = at >> 8;
            const T dx = sh.xyz[0][c] - sh.xyz[0][j], dy = sh.xyz[1][c] - sh.xyz[1][j], dz = sh.xyz[2][c] - sh.xyz[2][j];
            T r, inv, fc, dfc;
            refined_length_and_inverse(dx * dx + dy * dy + dz * dz, &r, &inv);
            cutoff<T>(r, (T)kA_Rc, &fc, &dfc);
            sh.u[e] = Vec4<T>{dx * inv, dy * inv, dz * inv, r};
            sh.w[e] = Vec4<T>{inv, fc, dfc, bits_as((T)0, sh.type[j])};
        }
        cp_async_wait<0>();
        __syncthreads();
        if (c0 > 0) clear_forces();
        // ---- neighbour pairs of the batch, lane = pair; the pairs of a central atom with k neighbours in circulant order:
        // pair q is (a, a + d mod k) with d = 1 + q / k, a = q mod k ----
        for (int first = ((warp + NW - 3) % NW) * kWarp; first < n_slots; first += kThreads) {
            const int p = min(first + lane, n_slots - 1);
            const int c = owner_of(members, my_slot, first, p);
            const int at = __shfl_sync(kFull, my_at, c);
            const unsigned rk = __shfl_sync(kFull, k_recip, c);
            const int q = p - (at & 0x1fff), k = (at >> 13) & 0x3f, list = at >> 19;
            const int d0 = (int)(((unsigned)q * rk) >> 16), a = q - d0 * k;
            int b = a + d0 + 1;
            if (b >= k) b -= k;
            const Vec4<T> ua = sh.u[list + a], ub = sh.u[list + b], wa = sh.w[list + a], wb = sh.w[list + b];
            T cosv = ua.x * ub.x + ua.y * ub.y + ua.z * ub.z;
            cosv = Num<T>::max_((T)-1, Num<T>::min_((T)1, cosv));
            const T s2 = sin2_from_cross<T>(ua.x, ua.y, ua.z, ub.x, ub.y, ub.z);
            T gl[kTS];
            const T* gsrc = sh.g[c - r0] + bucket_of(as_bits(wa.w), as_bits(wb.w)) * kGradBucketStride;
#pragma unroll
            for (int i = 0; i < kTS; i += 4) load4(gsrc + i, gl + i);
            T dc, dra, drb;
            angular_vjp_dev<T>(cosv, s2, ua.w, ub.w, wa.y, wa.z, wb.y, wb.z, gl, &dc, &dra, &drb);
            Vec2<T>* out = sh.pair + 2 * (p - a);
            out[2 * a] = Vec2<T>{dc, cosv * dc * wa.x - dra};
            out[2 * (2 * (d0 + 1) == k ? a : b) + 1] = Vec2<T>{dc, cosv * dc * wb.x - drb};
        }
        __syncthreads();
        // ---- the next batch's rows, if they are not here ----
        const int c2 = c1 < n ? batch_end(c1) : c1;
        if (c2 > r1) {
            r0 = c1;
            r1 = min(r0 + Cfg::kRows, n);
            for (int c = r0 + warp; c < r1; c += NW) {
                const T* src = row_of(c);
                if ((ok_mask >> c) & 1u) request_angular(src, sh.g[c - r0]);
            }
            cp_async_commit();
        }
        if (plane >= 0 && c0 == 0 && lane < n) {
            const T* x = sh.xyz[plane];
            const T xi = x[lane];
            for (int j = 0; j < n; j += 4) {
                T f[4], xj[4];
                load4(&sh.radial[lane][j], f);
                load4(x + j, xj);
#pragma unroll
                for (int q = 0; q < 4; q++)
                    if (f[q] != (T)0) sum += f[q] * (xi - xj[q]);
            }
        }
        // ---- lane = entry: the force on it from the pairs that it is in ----
        for (int first = warp * kWarp; first < n_entries; first += kThreads) {
            const int e = min(first + lane, n_entries - 1);
            const int whose = sh.list[k0 + e], c = whose & 0xff;
            const int at = __shfl_sync(kFull, my_at, c);
            const int k = (at >> 13) & 0x3f, list = at >> 19, a = e - list;
            const Vec4<T>*u = sh.u + list, *row = reinterpret_cast<const Vec4<T>*>(sh.pair) + (at & 0x1fff) + a;
            T fx = (T)0, fy = (T)0, fz = (T)0, along = (T)0;
            int b = a, z = a;
            for (int left = k; left > 2; left -= 2, row += k) {
                b = b + 1 >= k ? 0 : b + 1;
                z = z == 0 ? k - 1 : z - 1;
                const Vec4<T> ub = u[b], uz = u[z], q = *row;
                along += q.y + q.w;
                fx += q.x * ub.x + q.z * uz.x;
                fy += q.x * ub.y + q.z * uz.y;
                fz += q.x * ub.z + q.z * uz.z;
            }
            if (!(k & 1)) {      // the last row of an even k has k / 2 pairs; a + k / 2 = a - k / 2 (mod k)
                b = b + 1 >= k ? 0 : b + 1;
                const Vec4<T> ub = u[b];
                const Vec2<T> q = reinterpret_cast<const Vec2<T>*>(row)[a < (k >> 1) ? 0 : 1 - k];
                along += q.y;
                fx += q.x * ub.x;
                fy += q.x * ub.y;
                fz += q.x * ub.z;
            }
            const Vec4<T> ua = u[a];
            const T inv = sh.w[e].x;
            const int j = whose >> 8;
            sh.force[c - c0][0][j] = along * ua.x - inv * fx;
            sh.force[c - c0][1][j] = along * ua.y - inv * fy;
            sh.force[c - c0][2][j] = along * ua.z - inv * fz;
        }
        __syncthreads();
        // ---- what the batch's central atoms hand to an atom, less what it hands out ----
        if (plane >= 0) {
#pragma unroll 4
            for (int q = 0; q < c1 - c0; q++) sum += sh.force[q][plane][lane];
            if ((members >> lane) & 1u)
                for (int q = 0; q < n; q += 4) {
                    T v[4];
                    load4(&sh.force[lane - c0][plane][q], v);
                    sum -= v[0]; sum -= v[1]; sum -= v[2]; sum -= v[3];
                }
        }
        if (c1 >= n) break;
        c0 = c1;
        c1 = c2;
    }
    pdl_trigger();
    write_energy();
    if (plane >= 0 && lane < n) (plane == 0 ? gx : (plane == 1 ? gy : gz))[base + lane] = sum;
}

}  // namespace ani
