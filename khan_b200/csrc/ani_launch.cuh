// Launches with programmatic dependent launch, and the device side of it.
//
// A pass over one batch is a chain of five to eight kernels of 3 to 40 us, so the gap between two of them
// (drain of the last CTAs, launch, ramp-up: about 3 us) counts.  A kernel launched by launch_chain() may be
// set up while its predecessor drains; pdl_wait() holds it until everything before it in the stream has
// finished and is visible.  Rules that every kernel of this library launched this way keeps:
//   * pdl_wait() comes before the first access to memory that an earlier kernel of the stream may write,
//     and before the first store, and in some CTA of every launch, whatever the batch looks like (a kernel that ends
//     without a wait may end before its predecessor, and the kernel behind would take both for finished); weights and the geometry may be read ahead of it where the kernel before is one of
//     the same call and known not to write any (early_weights of the network kernels, after_sort of the features,
//     early_inputs of the gradient);
//   * a kernel that reads anything ahead of pdl_wait() takes what the kernel before it writes through load_fresh() or
//     asynchronous copies, never through a read-only (const __restrict__) pointer: such a load may be moved above the
//     wait, and a line fetched for a neighbouring array ahead of the wait may still be in the first-level cache;
//   * pdl_trigger() comes after pdl_wait(), so whatever lies two kernels back has finished when a kernel
//     starts; a kernel that writes weights never triggers;
//   * the kernels that fill the device with small molecules, and the sort in front of them, do not trigger at once.
//     Thousands of CTAs of the next kernel then sat in pdl_wait() in slots that other streams' CTAs could have used:
//     ani_sort, featurize and featurize_grad on 1024 molecules took 35.9 us a batch with eight streams in flight, 34.7
//     now (in double with four streams 108 -> 106). The sort and the gradient trigger when a CTA is nearly done; the
//     features half way, because the network kernel behind them sets up and fetches its first weights meanwhile
//     (energies + forces of 1024 molecules: 113 us at the start or half way, 116 at the end). The kernels for larger
//     molecules lose by a late trigger (173.3 -> 174.7 us a batch, four streams) and trigger at the start.
#pragma once

#include <cuda_runtime.h>

namespace ani {

__device__ __forceinline__ void pdl_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void pdl_trigger() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }

// What the kernel before may just have written: read in this place, from the second-level cache.
__device__ __forceinline__ int load_fresh(const int* p)
{
    int v;
    asm volatile("ld.global.cg.s32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
    return v;
}
__device__ __forceinline__ float load_fresh(const float* p)
{
    float v;
    asm volatile("ld.global.cg.f32 %0, [%1];" : "=f"(v) : "l"(p) : "memory");
    return v;
}
__device__ __forceinline__ double load_fresh(const double* p)
{
    double v;
    asm volatile("ld.global.cg.f64 %0, [%1];" : "=d"(v) : "l"(p) : "memory");
    return v;
}

// cluster = 1: no cluster.
template <typename... P, typename... A>
cudaError_t launch_chain(void (*kernel)(P...), dim3 grid, dim3 block, size_t smem, cudaStream_t stream, int cluster,
                         A... args)
{
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = grid;
    cfg.blockDim = block;
    cfg.dynamicSmemBytes = smem;
    cfg.stream = stream;
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    attr[1].id = cudaLaunchAttributeClusterDimension;
    attr[1].val.clusterDim.x = (unsigned)cluster;
    attr[1].val.clusterDim.y = attr[1].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = cluster > 1 ? 2 : 1;
    return cudaLaunchKernelEx(&cfg, kernel, static_cast<P>(args)...);
}

}  // namespace ani
