// What the coordinate-gradient kernels (ani_grad_mol.cuh, ani_grad_large.cuh) share: dL/dx, dL/dy, dL/dz from dL/dAEV,
// the vector-Jacobian product.
//
// Computes what featurize_grad_cpu of the reference computes
// (gpu_featurizer/kernel_cpu.cpp:217-366); the reference has no GPU kernel for this op.
#pragma once

#include "ani_common.cuh"
#include "ani_launch.cuh"
#include "ani_device_math.cuh"

namespace ani {

constexpr int kGradBucketStride = 36;  // upstream values of one type pair, padded against bank conflicts
constexpr int kGradRowWords = kRadial + kPairBuckets * kGradBucketStride;

// Slow path for an atom whose angular neighbourhood does not fit the sub-lists: angular part
// only (the radial part never needs a list).  lane = k, j is a warp-uniform loop.
template <typename T>
__device__ __noinline__ void grad_atom_streaming(const T* __restrict__ xs, const T* __restrict__ ys,
                                                 const T* __restrict__ zs,
                                                 const int* __restrict__ types, int base, int n,
                                                 int i, const T* g, T* gx, T* gy, T* gz)
{
    const int lane = lane_id();
    const T xi = xs[base + i], yi = ys[base + i], zi = zs[base + i];
    T fix = (T)0, fiy = (T)0, fiz = (T)0;
    for (int j = 0; j < n; j++) {
        if (j == i) continue;
        const T dxj = xi - xs[base + j], dyj = yi - ys[base + j], dzj = zi - zs[base + j];
        const T rj = Num<T>::sqrt_(dxj * dxj + dyj * dyj + dzj * dzj);
        if (!(rj < (T)kA_Rc)) continue;
        T fj, dfj;
        cutoff<T>(rj, (T)kA_Rc, &fj, &dfj);
        const int tj = types[base + j] & 3;
        const T ujx = dxj / rj, ujy = dyj / rj, ujz = dzj / rj;
        T fjx = (T)0, fjy = (T)0, fjz = (T)0;
        for (int k0 = j + 1; k0 < n; k0 += kWarp) {
            const int k = k0 + lane;
            if (k < n && k != i) {
                const T dxk = xi - xs[base + k], dyk = yi - ys[base + k], dzk = zi - zs[base + k];
                const T rk = Num<T>::sqrt_(dxk * dxk + dyk * dyk + dzk * dzk);
                if (rk < (T)kA_Rc) {
                    T fk, dfk;
                    cutoff<T>(rk, (T)kA_Rc, &fk, &dfk);
                    const T ukx = dxk / rk, uky = dyk / rk, ukz = dzk / rk;
                    T c = ujx * ukx + ujy * uky + ujz * ukz;
                    c = Num<T>::max_((T)-1, Num<T>::min_((T)1, c));
                    const int bk = pair_bucket(tj, types[base + k] & 3);
                    T dc, drj, drk;
                    const T s2 = sin2_from_cross<T>(ujx, ujy, ujz, ukx, uky, ukz);
                    angular_vjp_dev<T>(c, s2, rj, rk, fj, dfj, fk, dfk,
                                      g + kRadial + bk * kGradBucketStride, &dc, &drj, &drk);
                    const T aj = -dc / rj, bj = c * dc / rj - drj;
                    const T ak = -dc / rk, bkk = c * dc / rk - drk;
                    const T gjx = aj * ukx + bj * ujx, gjy = aj * uky + bj * ujy, gjz = aj * ukz + bj * ujz;
                    const T gkx = ak * ujx + bkk * ukx, gky = ak * ujy + bkk * uky, gkz = ak * ujz + bkk * ukz;
                    fjx += gjx; fjy += gjy; fjz += gjz;
                    fix -= gjx + gkx; fiy -= gjy + gky; fiz -= gjz + gkz;
                    atomicAdd(&gx[base + k], gkx);
                    atomicAdd(&gy[base + k], gky);
                    atomicAdd(&gz[base + k], gkz);
                }
            }
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            fjx += __shfl_xor_sync(kFull, fjx, o);
            fjy += __shfl_xor_sync(kFull, fjy, o);
            fjz += __shfl_xor_sync(kFull, fjz, o);
        }
        if (lane == 0) {
            atomicAdd(&gx[base + j], fjx);
            atomicAdd(&gy[base + j], fjy);
            atomicAdd(&gz[base + j], fjz);
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

// Zero fill of the three gradient arrays in one launch (the gradient kernel accumulates into
// them; the reference zero-fills in its functor, gpu_featurizer/functor_op_cpu.cpp:70-72).
template <typename T> __global__ void zero3_kernel(T* a, T* b, T* c, int n)
{
    pdl_wait();
    pdl_trigger();
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        a[i] = (T)0;
        b[i] = (T)0;
        c[i] = (T)0;
    }
}

}  // namespace ani
