// Coordinate-gradient kernel for batches of larger molecules (and for upstream rows that are not 16-byte aligned).
//
// A CTA is one warp, a unit of work a ROUND of up to three central atoms of one molecule (round r of R takes the atoms
// r, r + R, r + 2 R).  Per round:
//   - the upstream rows are copied to shared memory with asynchronous 16-byte copies under the scan;
//   - A. one central atom after another scans the molecule, 32 candidates at a time.  The scan does no more than compare
//     squared distances; neighbours within R_Rc are compacted into the warp's pool (distance vector, element, index, and
//     their place in the angular list when within A_Rc), the central atoms one behind the other;
//   - R. lane = pool entry: the lengths, cutoffs and the radial force on every neighbour in the pool, angular list
//     entries written by the same lane;
//   - B. the neighbour pairs of all central atoms in the list (ani_grad_pair_pass.inl), forces added to the pool;
//   - C. lane = pool entry: one atomic add per component for each neighbour; lane = (central atom, component): minus the
//     sum of what it handed out.
// A central atom that does not fit what is left of the pool (96) or of the list (32) opens the next pass; one that fits
// neither alone goes through the streaming routines.
//
// Bound by instructions: with the radial terms evaluated during the scan (lane = candidate) 3 of 32 lanes had work, and
// one central atom alone left two thirds of the lanes idle in B -- 1950 warp instructions per central atom.  256
// molecules of 64 to 256 atoms 136 -> 101 us, in double (where a length is a library square root) 689 -> 258; 8
// molecules 37 -> 14 us, as a warp then takes one central atom only.
//
// Contributions of different central atoms meet in the outputs through atomic adds: these must be zero before, and the
// order of summation may differ between runs.
//
// Computes what featurize_grad_cpu of the reference computes (gpu_featurizer/kernel_cpu.cpp:217-366).
#pragma once

#include "ani_common.cuh"
#include "ani_grad.cuh"
#include "ani_grad_mol.cuh"
#include "ani_launch.cuh"

namespace ani {

constexpr int kLargeGradCentrals = 3;
constexpr int kLargeGradPool = 96;
constexpr int kLargeGradNoPlace = 63;              // not in the angular list
constexpr int kLargeGradMaxAtoms = 1 << 22;        // index bits of a pool entry

template <typename T> struct alignas(16) LargeGradNeighbor {
    Vec4<T> u;         // (x_c - x_j) / r, r
    T inv_r, fc, dfc;  // 1 / r, f_C(r, A_Rc) and its derivative
    int info;          // element | lane of j << 2 | first list entry of its central atom << 7 |
                       // neighbours of that central atom << 12 | row buffer << 18 | lane of the central atom << 20
};

template <typename T> struct LargeGradWarpShared {
    alignas(16) T g[kLargeGradCentrals][kGradRowWords];   // upstream rows, blocks of 32 at stride 36
    LargeGradNeighbor<T> nb[kWarp];
    Vec4<T> pool[kLargeGradPool];        // distance vector and its square; from step R on the force on the neighbour
    unsigned info[kLargeGradPool];       // element | central atom << 2 | place in the angular list << 4 | atom << 10
    int list[kLargeGradCentrals];        // of a central atom: first angular entry << 7 | angular neighbours << 12 | row << 18
    int first[kLargeGradCentrals + 1];   // first pool entry of each central atom
    int atom[kLargeGradCentrals];
    unsigned char pool_of[kWarp];        // pool entry of each angular list entry
};

template <typename T>
__global__ void __launch_bounds__(kWarp, sizeof(T) == 4 ? 20 : 12)
    featurize_grad_large_kernel(const T* __restrict__ xs, const T* __restrict__ ys, const T* __restrict__ zs,
                                const int* __restrict__ types, const int* __restrict__ mol_offsets,
                                const int* __restrict__ mol_counts, int n_mols, int n_atoms, int per_round, bool aligned,
                                const int* __restrict__ scatter, const T* __restrict__ gh, const T* __restrict__ gc,
                                const T* __restrict__ gn, const T* __restrict__ go, T* gx, T* gy, T* gz, int acs0,
                                int acs1, int acs2, int acs3)
{
    extern __shared__ __align__(128) unsigned char smem_raw[];
    LargeGradWarpShared<T>& ws = *reinterpret_cast<LargeGradWarpShared<T>*>(smem_raw);
    const int lane = lane_id();
    pdl_wait();
    pdl_trigger();

    const int rounds_in_grid = gridDim.x / n_mols;
    const int round0 = blockIdx.x / n_mols, m = blockIdx.x - round0 * n_mols;
    MolRange mol;
    if (!load_molecule(mol_offsets, mol_counts, m, n_atoms, &mol)) return;
    const int n = mol.n, base = mol.base;
    const int n_rounds = (n + per_round - 1) / per_round;

    for (int round = round0; round < n_rounds; round += rounds_in_grid) {
        const int G = (n - round + n_rounds - 1) / n_rounds;
        // ---- upstream rows ----
        unsigned refused = 0;
        for (int g = 0; g < G; g++) {
            const int gi = base + round + g * n_rounds;
            const int ti = checked_type(types[gi]);
            const int srow = scatter[gi];
            const int cap = ti == 0 ? acs0 : (ti == 1 ? acs1 : (ti == 2 ? acs2 : acs3));
            if (srow < 0 || srow >= cap) {
                if (lane == 0) report(ANI_ERR_BAD_INDEX);
                refused |= 1u << g;
                continue;
            }
            const T* grow = (ti == 0 ? gh : (ti == 1 ? gc : (ti == 2 ? gn : go))) + (size_t)srow * kTotal;
            auto place = [](int v) {
                return v < kRadial ? v : kRadial + ((v - kRadial) >> 5) * kGradBucketStride + ((v - kRadial) & 31);
            };
            if (aligned) {
                constexpr int V = 16 / (int)sizeof(T);
#pragma unroll
                for (int s = 0; s < kTotal / V / kWarp; s++) {
                    const int v = (lane + s * kWarp) * V;
                    cp_async16(&ws.g[g][place(v)], grow + v);
                }
            } else {
                for (int v = lane; v < kTotal; v += kWarp) ws.g[g][place(v)] = grow[v];
            }
        }
        cp_async_commit();

        int g = 0;
        while (g < G) {
            // ---- A: scan central atoms into the pool until it, or the angular list, is full ----
            int entries = 0, used = 0, max_half = 0;
            const int g_first = g;
            for (; g < G; g++) {
                const int c = round + g * n_rounds;
                int n_rad = 0, n_ang = 0;
                if (!((refused >> g) & 1u)) {
                    const T xi = xs[base + c], yi = ys[base + c], zi = zs[base + c];
                    int gj = base + (lane < n ? lane : 0);
                    T qx = xs[gj], qy = ys[gj], qz = zs[gj];
                    int qt = types[gj];
                    for (int j0 = 0; j0 < n; j0 += kWarp) {
                        const int j = j0 + lane;
                        const T dx = xi - qx, dy = yi - qy, dz = zi - qz;
                        const int tj = qt;
                        if (j0 + kWarp < n) {   // the next candidates are requested before this chunk's arithmetic
                            gj = base + (j + kWarp < n ? j + kWarp : 0);
                            qx = xs[gj]; qy = ys[gj]; qz = zs[gj];
                            qt = types[gj];
                        }
                        const T d2 = dx * dx + dy * dy + dz * dz;
                        const bool in_rad = j < n && j != c && d2 < (T)(kR_Rc * kR_Rc);
                        const bool in_ang = in_rad && d2 < (T)(kA_Rc * kA_Rc);
                        const unsigned mR = __ballot_sync(kFull, in_rad);
                        if (mR == 0) continue;
                        const unsigned mA = __ballot_sync(kFull, in_ang);
                        if (in_rad) {
                            const int p = entries + n_rad + __popc(mR & lanemask_lt());
                            const int q = used + n_ang + __popc(mA & lanemask_lt());
                            if (p < kLargeGradPool) {
                                ws.pool[p] = Vec4<T>{dx, dy, dz, d2};
                                ws.info[p] = (unsigned)checked_type(tj) | (unsigned)g << 2 |
                                             (unsigned)(in_ang && q < kWarp ? q : kLargeGradNoPlace) << 4 | (unsigned)j << 10;
                                if (in_ang && q < kWarp) ws.pool_of[q] = (unsigned char)p;
                            }
                        }
                        n_rad += __popc(mR);
                        n_ang += __popc(mA);
                    }
                }
                if (entries + n_rad > kLargeGradPool || used + n_ang > kWarp || n > kLargeGradMaxAtoms) {
                    if (entries > 0) break;   // this central atom opens the next pass
                    cp_async_wait<0>();
                    __syncwarp();
                    grad_atom_streaming_radial<T>(xs, ys, zs, types, base, n, c, ws.g[g], gx, gy, gz);
                    grad_atom_streaming<T>(xs, ys, zs, types, base, n, c, ws.g[g], gx, gy, gz);
                    n_rad = n_ang = 0;
                }
                if (lane == 0) {
                    ws.first[g] = entries;
                    ws.first[g + 1] = entries + n_rad;
                    ws.list[g] = used << 7 | n_ang << 12 | g << 18;
                    ws.atom[g] = base + c;
                }
                entries += n_rad;
                used += n_ang;
                max_half = max(max_half, n_ang >> 1);
            }
            cp_async_wait<0>();
            __syncwarp();

            // ---- R: lane = pool entry ----
            for (int p = lane; p < entries; p += kWarp) {
                const Vec4<T> v = ws.pool[p];
                const unsigned info = ws.info[p];
                const int t = info & 3, gg = (info >> 2) & 3, q = (info >> 4) & 63;
                T r, inv, fc, dfc;
                length_and_inverse(v.w, &r, &inv);
                cutoff<T>(r, (T)kR_Rc, &fc, &dfc);
                T w[kNumRs];
#pragma unroll
                for (int s = 0; s < kNumRs; s += 4) load4(&ws.g[gg][t * kNumRs + s], w + s);
                const T ux = v.x * inv, uy = v.y * inv, uz = v.z * inv;
                const T d = -radial_vjp_dev<T>(r, fc, dfc, w);
                ws.pool[p] = Vec4<T>{d * ux, d * uy, d * uz, (T)0};
                if (q != kLargeGradNoPlace) {
                    LargeGradNeighbor<T> e;
                    e.u = Vec4<T>{ux, uy, uz, r};
                    e.inv_r = inv;
                    cutoff<T>(r, (T)kA_Rc, &e.fc, &e.dfc);
                    e.info = t | ws.list[gg];
                    ws.nb[q] = e;
                }
            }
            __syncwarp();

            // ---- B: neighbour pairs of every central atom in the list, circulant order ----
            if (max_half > 0) {
#include "ani_grad_pair_pass.inl"
                if (lane < used) {
                    Vec4<T>& f = ws.pool[ws.pool_of[lane]];
                    f.x += fax;
                    f.y += fay;
                    f.z += faz;
                }
                __syncwarp();
            }

            // ---- C: forces out ----
            for (int p = lane; p < entries; p += kWarp) {
                const Vec4<T> f = ws.pool[p];
                const int gj = base + (int)(ws.info[p] >> 10);
                atomicAdd(&gx[gj], f.x);
                atomicAdd(&gy[gj], f.y);
                atomicAdd(&gz[gj], f.z);
            }
            if (lane < 3 * (g - g_first)) {
                const int gg = g_first + lane / 3, axis = lane % 3, end = ws.first[gg + 1];
                T sum = (T)0;
                for (int p = ws.first[gg]; p < end; p++) sum += reinterpret_cast<const T*>(&ws.pool[p])[axis];
                atomicAdd((axis == 0 ? gx : (axis == 1 ? gy : gz)) + ws.atom[gg], -sum);
            }
            __syncwarp();
        }
    }
}

}  // namespace ani
