// Directional derivative of the features (Jacobian-vector product) for batches of small molecules: the
// forward-mode form of featurize_mol_kernel.  Same rounds of four central atoms per warp, same passes T, B
// and C (ani_featurize_round_passes.inl with ANI_ROUND_TANGENT); a list entry also carries the rate of its
// unit vector, distance and cutoff along v, a slot evaluates the factors and their rates together, and a
// block accumulates dA BF + A dBF.
//
// Why: the warp-per-atom kernel of ani_grad_inverse.cuh evaluates every (theta, shift) of every neighbour
// pair from scratch in every lane.  What a pass of force training spends here (3.4 k atoms): 100 us with it,
// 25 us with this kernel.  A molecule of more than 32 atoms in such a batch goes through its routine.
//
// Computes the product that featurize_grad_inverse of the reference stands for
// (gpu_featurizer/kernel_cpu.cpp:37-179; see ani_grad_inverse.cuh).
#pragma once

#include "ani_featurize_mol.cuh"
#include "ani_grad_inverse.cuh"

namespace ani {

// The lists of a round share 96 entries: an atom whose list does not fit any more waits until T, B and C have worked off
// the ones before it (31 neighbours of one atom always fit).
constexpr int kTangentPool = 96;

template <typename T> struct TangentRound : MolAngularShared<T, kTangentPool, kMolMaxAtoms - 1> {
    int list_base[kMolCentrals];                   // first entry of each central atom's list
    Vec4<T> du[kTangentPool];                      // d (unit vector) and d r along v
    T fc_dot[kTangentPool];                        // d f_C(r, A_Rc)
    alignas(16) T dA[kNumThetas][kMolChunkStride];
    alignas(16) T dBF[kNumARs][kMolChunkStride];
    Vec4<T> slope[kMolCentrals][kMolMaxAtoms];     // r, -2 eta f_C dr, df_C dr of every atom of the molecule (R_Rc)
    __device__ __forceinline__ int first(int g) const { return list_base[g]; }
};

template <typename T> struct TangentWarpShared {
    union {
        TangentRound<T> ang;
        JvpNeighbor<T> list[kJvpMaxNeighbors];     // molecules of more than 32 atoms
    };
    MolSortShared sort;
    __device__ TangentWarpShared() {}
};

template <typename T>
__global__ void __launch_bounds__(kWarp, sizeof(T) == 4 ? 16 : 10)
    featurize_tangent_mol_kernel(const T* __restrict__ xs, const T* __restrict__ ys, const T* __restrict__ zs,
                                 const int* __restrict__ types, const int* __restrict__ mol_offsets,
                                 const int* __restrict__ mol_counts, int n_mols, int n_atoms,
                                 const int* __restrict__ scatter, const T* __restrict__ vx, const T* __restrict__ vy,
                                 const T* __restrict__ vz, T* out_h, T* out_c, T* out_n, T* out_o, int acs0, int acs1,
                                 int acs2, int acs3, int per_round, int per_round_recip)
{
    __shared__ TangentWarpShared<T> ws;
    using Granule = Vec4<float>;
    constexpr int kPerGranule = 16 / (int)sizeof(T);
    const int lane = lane_id();
    pdl_wait();
    pdl_trigger();

    const int round = blockIdx.x / n_mols, m = blockIdx.x - round * n_mols;   // round-major, as in featurize_mol_kernel
    MolRange mol;
    if (!load_molecule(mol_offsets, mol_counts, m, n_atoms, &mol)) return;
    const int n = mol.n, base = mol.base;

    if (n > kMolMaxAtoms) {
        for (int i = round; i < n; i += gridDim.x / n_mols) {
            const int gi = base + i;
            const int ti = checked_type(types[gi]);
            const int srow = scatter[gi];
            const int cap = ti == 0 ? acs0 : (ti == 1 ? acs1 : (ti == 2 ? acs2 : acs3));
            if (srow < 0 || srow >= cap) {
                if (lane == 0) report(ANI_ERR_BAD_INDEX);
                continue;
            }
            jvp_atom_streaming<T>(xs, ys, zs, types, vx, vy, vz, base, n, i, ws.list,
                                  element_buffer<T>(ti, out_h, out_c, out_n, out_o) + (size_t)srow * kTotal);
        }
        return;
    }
    const int n_rounds = ((n + per_round - 1) * per_round_recip) >> 16;   // / per_round; n is at most 32 here
    if (round >= n_rounds) return;
    const int G = (n - round + n_rounds - 1) / n_rounds;

    MolLanes<T> ml;
    load_sorted_molecule<T>(xs, ys, zs, types, scatter, base, n, &ws.sort, &ml);
    const int gj = base + (lane < n ? ws.sort.src[lane] : 0);
    const T mvx = vx[gj], mvy = vy[gj], mvz = vz[gj];

    if (lane == 0) {   // padding slots read entry 0
        ws.ang.ang_u[0] = Vec4<T>{(T)1, (T)0, (T)0, (T)1};
        ws.ang.du[0] = Vec4<T>{(T)0, (T)0, (T)0, (T)0};
        ws.ang.ang_fc[0] = (T)0;
        ws.ang.fc_dot[0] = (T)0;
    }
    unsigned skip = 0;
    int g = 0;
    do {
        if (lane < kMolCentrals * kTypes) ws.ang.cnt_a[lane] = 0;
        __syncwarp();

        // ---- A: scan, one central atom after another, as many as the lists have room for ----
        int used = 0;
        for (; g < G; g++) {
            const int c = round + g * n_rounds;
            const T xi = __shfl_sync(kFull, ml.x, c), yi = __shfl_sync(kFull, ml.y, c), zi = __shfl_sync(kFull, ml.z, c);
            const int ti = __shfl_sync(kFull, ml.type, c);
            const int srow = ws.sort.srow[c];
            const int cap = ti == 0 ? acs0 : (ti == 1 ? acs1 : (ti == 2 ? acs2 : acs3));
            const T wx = __shfl_sync(kFull, mvx, c) - mvx, wy = __shfl_sync(kFull, mvy, c) - mvy,
                    wz = __shfl_sync(kFull, mvz, c) - mvz;
            if (srow < 0 || srow >= cap) {
                if (lane == 0) report(ANI_ERR_BAD_INDEX);
                skip |= 1u << g;
                continue;
            }
            T* row = element_buffer<T>(ti, out_h, out_c, out_n, out_o) + (size_t)srow * kTotal;
            if (lane == 0) ws.ang.row[g] = row;

            const T dx = xi - ml.x, dy = yi - ml.y, dz = zi - ml.z;
            T r, inv;
            length_and_inverse(dx * dx + dy * dy + dz * dz, &r, &inv);
            const bool in_rad = lane < n && lane != c && r < (T)kR_Rc;
            const bool in_ang = in_rad && r < (T)kA_Rc;
            const unsigned mA = __ballot_sync(kFull, in_ang);
            if (used + __popc(mA) > kTangentPool) break;
            {
                Granule* zero = reinterpret_cast<Granule*>(row + kRadial);
                constexpr int kGranules = kAngular / kPerGranule;
#pragma unroll
                for (int i = 0; i < (kGranules + kWarp - 1) / kWarp; i++)
                    if (i * kWarp + lane < kGranules) zero[i * kWarp + lane] = Granule{0.f, 0.f, 0.f, 0.f};
            }
            const T ux = dx * inv, uy = dy * inv, uz = dz * inv;
            const T rate = ux * wx + uy * wy + uz * wz;      // d r along v
            Vec4<T> slope{r, (T)0, (T)0, (T)0};
            if (in_rad) {
                T fc, dfc;
                cutoff<T>(r, (T)kR_Rc, &fc, &dfc);
                slope.y = (T)-2 * (T)kR_eta * fc * rate;
                slope.z = dfc * rate;
            }
            ws.ang.slope[g][lane] = slope;
            if (in_ang) {
                const int p = used + __popc(mA & lanemask_lt());
                T fc, dfc;
                cutoff<T>(r, (T)kA_Rc, &fc, &dfc);
                ws.ang.ang_u[p] = Vec4<T>{ux, uy, uz, r};
                ws.ang.du[p] = Vec4<T>{(wx - rate * ux) * inv, (wy - rate * uy) * inv, (wz - rate * uz) * inv, rate};
                ws.ang.ang_fc[p] = fc;
                ws.ang.fc_dot[p] = dfc * rate;
            }
            if (lane < kTypes) ws.ang.cnt_a[g * kTypes + lane] = __popc(mA & ws.sort.tmask[lane]);
            if (lane == 0) ws.ang.list_base[g] = used;
            used += __popc(mA);
        }
        __syncwarp();

#define ANI_ROUND_TANGENT
#include "ani_featurize_round_passes.inl"
#undef ANI_ROUND_TANGENT
    } while (g < G);

    // ---- R: radial blocks of the round, lane = (central atom, pair of shifts) ----
    {
        const int c = lane >> 3, sp = lane & 7;
        const Vec4<T>* list = ws.ang.slope[c];
        const T sh0 = (T)c_tab.R_Rs[2 * sp], sh1 = (T)c_tab.R_Rs[2 * sp + 1];
        const uint4 tmq = *reinterpret_cast<const uint4*>(ws.sort.tmask);
        const int run_end[kTypes] = {__popc(tmq.x), __popc(tmq.x | tmq.y), __popc(tmq.x | tmq.y | tmq.z), n};
        Pair<T> acc[kTypes];
        int p = 0;
#pragma unroll
        for (int t = 0; t < kTypes; t++) {
            acc[t] = Pair<T>{(T)0, (T)0};
            for (; p < run_end[t]; p++) {
                const Vec4<T> e = list[p];
                const Pair<T> d{e.x - sh0, e.x - sh1};
                const Pair<T> d2 = pmul(d, d);
                const Pair<T> v{Num<T>::exp_neg((T)kR_eta, d2.x), Num<T>::exp_neg((T)kR_eta, d2.y)};
                acc[t] = pfma(v, pfma(d, Pair<T>{e.y, e.y}, Pair<T>{e.z, e.z}), acc[t]);
            }
        }
        if (c < G && !((skip >> c) & 1u)) {
            T* row = ws.ang.row[c];
#pragma unroll
            for (int t = 0; t < kTypes; t++)
                *reinterpret_cast<Vec2<T>*>(row + t * kNumRs + 2 * sp) = Vec2<T>{acc[t].x, acc[t].y};
        }
    }
}

}  // namespace ani
