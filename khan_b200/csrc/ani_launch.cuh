// Launches with programmatic dependent launch, and the device side of it.
//
// A pass over one batch is a chain of five to eight kernels of 3 to 40 us, so the gap between two of them
// (drain of the last CTAs, launch, ramp-up: about 3 us) counts.  A kernel launched by launch_chain() may be
// set up while its predecessor drains; pdl_wait() holds it until everything before it in the stream has
// finished and is visible.  Rules that every kernel of this library launched this way keeps:
//   * pdl_wait() comes before the first access to memory that an earlier kernel of the stream may write,
//     and before the first store; weights and the geometry may be read ahead of it where the kernel before is one of
//     the same call and known not to write any (early_weights of the network kernels, after_sort of the features,
//     early_inputs of the gradient);
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
