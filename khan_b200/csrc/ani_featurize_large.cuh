// Forward kernel for batches of larger molecules (mean size above what the molecule-per-warp kernel
// takes; BASELINE's 64-256-atom molecules).
//
// Same decomposition as featurize_mol_kernel -- a CTA is one warp, a unit of work is a ROUND of up to
// four central atoms of one molecule, and passes T, B and C (group table, triplet factors with
// lane = slot over the groups of ALL central atoms of the round, contraction with lane = (theta,
// shift)) are the very same code, ani_featurize_round_passes.inl -- but the molecule does not fit the lanes,
// so the scan differs:
//   A. the molecule is read from global memory 32 candidates at a time, once per round; every lane tests its candidate
//      against the (up to) four central atoms, whose coordinates all lanes hold, by squared distance, and keeps no more
//      than the ballots: lane = (central atom, one of eight groups of 32 candidates).  Then every lane writes the indices of
//      its set bits to the central atom's radial list;
//   L. lane = list entry: length and cutoff from the neighbour's coordinates (in the scan 3 of 32 lanes had work for them);
//      angular neighbours go to the angular list (32 at most) in arrival order;
//   R. radial features of the whole round, lane = (central atom, pair of shifts): every lane walks
//      the radial list of its central atom and adds to the sum of the neighbour's element;
//   S. each angular list is put into element order by one ballot sort (lane = entry), which is what
//      pass T needs; the per-element counts fall out of the same ballots.
// When a radial list is full (64 entries), pass R works it off and the scan goes on behind the last whole group of 32; a
// central atom with more
// than 32 angular neighbours goes through the streaming routine of ani_featurize.cuh.  A CTA takes the rounds r, r + R0, r + 2 R0, ... of its molecule
// (R0 rounds per molecule in the grid, chosen by the host from the mean molecule size), so molecules
// of any size are covered.  Nothing is accumulated with atomics; rows need no zero fill by the caller.
//
// Bound by instruction issue.  With neighbours written to both lists inside the scan (ballots, counts and stores for every
// 32 candidates of every central atom) and sums over all four elements added to for every neighbour, microseconds alone
// before -> now: 256 molecules of 64 to 256 atoms 97 -> 82 (79.5 -> 72.8 a batch with eight streams in flight), 64: 43 -> 36,
// 8: 21.3 -> 18.5; double, 256: 257 -> 247.
//
// Computes what featurize_cpu of the reference computes (gpu_featurizer/kernel_cpu.cpp:406-537).
#pragma once

#include "ani_common.cuh"
#include "ani_device_math.cuh"
#include "ani_featurize.cuh"
#include "ani_featurize_mol.cuh"

namespace ani {

constexpr int kLargeCapR = 64;   // radial neighbours kept per central atom
constexpr int kLargeCapA = 32;   // angular neighbours kept per central atom (one ballot sort covers 32 entries)
constexpr int kLargeBlock = 8 * kWarp;   // candidates of a scan: eight masks of 32 for each of four central atoms

__device__ __forceinline__ void add_where(bool on, Pair<float> v, Pair<float>* sum)      // one packed add, predicated
{
    unsigned long long s = pack2(sum->x, sum->y);
    asm("{\n.reg .pred p;\nsetp.ne.s32 p, %2, 0;\n@p add.rn.f32x2 %0, %0, %1;\n}" : "+l"(s) : "l"(pack2(v.x, v.y)), "r"((int)on));
    *sum = unpack2(s);
}
__device__ __forceinline__ void add_where(bool on, Pair<double> v, Pair<double>* sum)
{
    sum->x += on ? v.x : 0.0;
    sum->y += on ? v.y : 0.0;
}

template <typename T> struct LargeFwdWarpShared {
    MolAngularShared<T, kMolCentrals * kLargeCapA, kLargeCapA> ang;
    Vec2<T> rad[kMolCentrals][kLargeCapR];           // index of the neighbour; from step L on (r, f_C(r, R_Rc))
    unsigned char rad_t[kMolCentrals][kLargeCapR];   // element of that neighbour
    unsigned char ang_t[kMolCentrals * kLargeCapA];    // element of each angular neighbour before the sort
    int cnt_r[kMolCentrals];
};

template <typename T>
__global__ void __launch_bounds__(kWarp, sizeof(T) == 4 ? 22 : 1)
    featurize_large_kernel(const T* __restrict__ xs, const T* __restrict__ ys, const T* __restrict__ zs,
                           const int* __restrict__ types, const int* __restrict__ mol_offsets,
                           const int* __restrict__ mol_counts, int n_mols, int n_atoms, int per_round,
                           const int* __restrict__ scatter, T* out_h, T* out_c, T* out_n, T* out_o,
                           int acs0, int acs1, int acs2, int acs3)
{
    __shared__ LargeFwdWarpShared<T> ws;
    using Granule = Vec4<float>;
    constexpr int kPerGranule = 16 / (int)sizeof(T);
    const int lane = lane_id();
    pdl_wait();
    pdl_trigger();

    // round-major grid, as in featurize_mol_kernel: the first rounds of all molecules start first
    const int round0 = blockIdx.x / n_mols, m = blockIdx.x - round0 * n_mols;
    MolRange mol;
    if (!load_molecule(mol_offsets, mol_counts, m, n_atoms, &mol)) return;
    const int n = mol.n, base = mol.base;
    const int n_rounds = (n + per_round - 1) / per_round, rounds_in_grid = gridDim.x / n_mols;

    for (int round = round0; round < n_rounds; round += rounds_in_grid) {
        // round r takes the central atoms r, r + R, r + 2 R, r + 3 R (R = rounds of the molecule)
        const int G = (n - round + n_rounds - 1) / n_rounds;
        __syncwarp();   // the previous round's readers are done
        if (lane == 0) {
            ws.ang.ang_u[0] = Vec4<T>{(T)1, (T)0, (T)0, (T)1};
            ws.ang.ang_fc[0] = (T)0;
        }
        if (lane < kMolCentrals * kTypes) ws.ang.cnt_a[lane] = 0;

        // ---- the central atoms: coordinates to all lanes, rows, zero fill of the angular blocks ----
        T xi[kMolCentrals], yi[kMolCentrals], zi[kMolCentrals];
        int ci[kMolCentrals];
        unsigned skip = 0;   // central atoms that are refused or finished by the streaming routine
#pragma unroll
        for (int g = 0; g < kMolCentrals; g++) {
            ci[g] = g < G ? round + g * n_rounds : -1;
            const int gi = base + (g < G ? ci[g] : 0);
            xi[g] = xs[gi]; yi[g] = ys[gi]; zi[g] = zs[gi];
            if (g < G) {
                const int ti = checked_type(types[gi]);
                const int srow = scatter[gi];
                const int cap = ti == 0 ? acs0 : (ti == 1 ? acs1 : (ti == 2 ? acs2 : acs3));
                if (srow < 0 || srow >= cap) {
                    if (lane == 0) report(ANI_ERR_BAD_INDEX);
                    skip |= 1u << g;
                } else {
                    T* row = element_buffer<T>(ti, out_h, out_c, out_n, out_o) + (size_t)srow * kTotal;
                    if (lane == 0) ws.ang.row[g] = row;
                    Granule* zero = reinterpret_cast<Granule*>(row + kRadial);
                    constexpr int kGranules = kAngular / kPerGranule;
#pragma unroll
                    for (int i = 0; i < (kGranules + kWarp - 1) / kWarp; i++)
                        if (i * kWarp + lane < kGranules) zero[i * kWarp + lane] = Granule{0.f, 0.f, 0.f, 0.f};
                }
            } else {
                skip |= 1u << g;
            }
        }

        // ---- A: scan, up to kLargeBlock candidates against all central atoms of the round ----
        int cA[kMolCentrals] = {0, 0, 0, 0}, cR[kMolCentrals];
        int j0 = 0;
        bool again = false;   // pass R has written the rows once: it adds from now on
        do {
#pragma unroll
        for (int g = 0; g < kMolCentrals; g++) cR[g] = 0;
        bool full = false;
        while (j0 < n && !full) {
            // lane 8 g + k: which of the candidates j0 + 32 k + (0 .. 31) are within R_Rc of central atom g
            unsigned mask = 0u;
#pragma unroll
            for (int k = 0; k < kLargeBlock / kWarp; k++) {
                const int j = j0 + k * kWarp + lane;
                if (j0 + k * kWarp >= n) break;
                const int gj = base + (j < n ? j : 0);
                const T px = xs[gj], py = ys[gj], pz = zs[gj];
#pragma unroll
                for (int g = 0; g < kMolCentrals; g++) {
                    if ((skip >> g) & 1u) continue;   // warp-uniform
                    const T dx = xi[g] - px, dy = yi[g] - py, dz = zi[g] - pz;
                    const unsigned m = __ballot_sync(kFull, j < n && j != ci[g] && dx * dx + dy * dy + dz * dz < (T)(kR_Rc * kR_Rc));
                    if (lane == 8 * g + k) mask = m;
                }
            }
            // as many groups of 32 candidates as the lists have room for; the rest comes again after pass R
            int incl = __popc(mask);
#pragma unroll
            for (int o = 1; o < 8; o <<= 1) {
                const int y = __shfl_up_sync(kFull, incl, o, 8);
                if ((lane & 7) >= o) incl += y;
            }
            int at = pick4(cR, lane >> 3) + incl - __popc(mask);
            unsigned over = __ballot_sync(kFull, pick4(cR, lane >> 3) + incl > kLargeCapR);
            over |= over >> 16;
            over = (over | over >> 8) & 0xffu;
            const int taken = over ? __ffs(over) - 1 : 8;
            full = over != 0u;
            if ((lane & 7) < taken)
                for (; mask; mask &= mask - 1)
                    ws.rad[lane >> 3][at++].x = bits_as((T)0, j0 + 32 * (lane & 7) + __ffs(mask) - 1);
            if (taken > 0)
#pragma unroll
                for (int g = 0; g < kMolCentrals; g++) cR[g] += __shfl_sync(kFull, incl, 8 * g + taken - 1);
            j0 += kWarp * taken;
        }
        __syncwarp();
        if (lane < kMolCentrals) ws.cnt_r[lane] = pick4(cR, lane);

        // ---- L: lane = list entry: length and cutoff; angular neighbours to their own list ----
#pragma unroll
        for (int g = 0; g < kMolCentrals; g++)
            for (int p0 = 0; p0 < cR[g]; p0 += kWarp) {
                const int p = p0 + lane;
                const bool have = p < cR[g];
                const int gj = base + (have ? as_bits(ws.rad[g][p].x) : 0);
                const T dx = xi[g] - xs[gj], dy = yi[g] - ys[gj], dz = zi[g] - zs[gj];
                const int tj = checked_type(types[gj]);
                const T d2 = dx * dx + dy * dy + dz * dz;
                T r, inv;
                length_and_inverse(d2, &r, &inv);
                const bool in_ang = have && d2 < (T)(kA_Rc * kA_Rc);
                const unsigned mA = __ballot_sync(kFull, in_ang);
                if (have) {
                    ws.rad[g][p] = Vec2<T>{r, cutoff_value<T>(r, (T)kR_Rc)};
                    ws.rad_t[g][p] = (unsigned char)tj;
                }
                const int pos = cA[g] + __popc(mA & lanemask_lt());
                if (in_ang && pos < kLargeCapA) {
                    const int q = g * kLargeCapA + pos;
                    ws.ang.ang_u[q] = Vec4<T>{dx * inv, dy * inv, dz * inv, r};
                    ws.ang_t[q] = (unsigned char)tj;
                }
                cA[g] += __popc(mA);
            }
        __syncwarp();

        // ---- R: radial features of the round, lane = (central atom, pair of shifts) ----
        {
            const int g = lane >> 3, sp = lane & 7;
            const T sh0 = (T)c_tab.R_Rs[2 * sp], sh1 = (T)c_tab.R_Rs[2 * sp + 1];
            const int cnt = ws.cnt_r[g];
            Pair<T> acc[kTypes];
#pragma unroll
            for (int t = 0; t < kTypes; t++) acc[t] = Pair<T>{(T)0, (T)0};
            for (int p = 0; p < cnt; p++) {
                const Vec2<T> e = ws.rad[g][p];
                const int t = ws.rad_t[g][p];
                const Pair<T> d{e.x - sh0, e.x - sh1};
                const Pair<T> d2 = pmul(d, d);
                const Pair<T> v{Num<T>::exp_neg((T)kR_eta, d2.x) * e.y, Num<T>::exp_neg((T)kR_eta, d2.y) * e.y};
#pragma unroll
                for (int k = 0; k < kTypes; k++) add_where(t == k, v, &acc[k]);
            }
            if (!((skip >> g) & 1u)) {
                T* row = ws.ang.row[g];
#pragma unroll
                for (int t = 0; t < kTypes; t++) {
                    Vec2<T>* at = reinterpret_cast<Vec2<T>*>(row + t * kNumRs + 2 * sp);
                    const Vec2<T> had = again ? *at : Vec2<T>{(T)0, (T)0};
                    *at = Vec2<T>{had.x + acc[t].x, had.y + acc[t].y};
                }
            }
        }
        again = true;
        __syncwarp();
        } while (j0 < n);

        // ---- S: each angular list into element order; denser neighbourhoods stream ----
#pragma unroll
        for (int g = 0; g < kMolCentrals; g++) {
            if ((skip >> g) & 1u) continue;
            if (cA[g] > kLargeCapA) {
                featurize_atom_streaming<T>(xs, ys, zs, types, base, n, ci[g], ws.ang.row[g]);
                skip |= 1u << g;
                __syncwarp();
                continue;
            }
            const bool have = lane < cA[g];
            const int p = g * kLargeCapA + (have ? lane : 0);
            const Vec4<T> v = ws.ang.ang_u[p];
            const int t = have ? ws.ang_t[p] : kTypes;
            const unsigned m0 = __ballot_sync(kFull, t == 0), m1 = __ballot_sync(kFull, t == 1),
                           m2 = __ballot_sync(kFull, t == 2), m3 = __ballot_sync(kFull, t == 3);
            const int c0 = __popc(m0), c1 = __popc(m1), c2 = __popc(m2);
            const unsigned mine = t == 0 ? m0 : (t == 1 ? m1 : (t == 2 ? m2 : m3));
            const int start = t == 0 ? 0 : (t == 1 ? c0 : (t == 2 ? c0 + c1 : c0 + c1 + c2));
            __syncwarp();   // every entry has been read
            if (have) {
                const int q = g * kLargeCapA + start + __popc(mine & lanemask_lt());
                ws.ang.ang_u[q] = v;
                ws.ang.ang_fc[q] = cutoff_value<T>(v.w, (T)kA_Rc);
            }
            if (lane == 0)
                *reinterpret_cast<int4*>(&ws.ang.cnt_a[g * kTypes]) = make_int4(c0, c1, c2, __popc(m3));
        }
        __syncwarp();

#include "ani_featurize_round_passes.inl"
    }
}

}  // namespace ani
