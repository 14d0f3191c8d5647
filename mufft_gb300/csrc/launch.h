// Kernel launches that overlap the previous launch's end.
#pragma once

#include <cuda_runtime.h>

namespace mgb {

// Launches a kernel that starts with dependent_start() (fft_device.cuh) so
// that its CTAs are set up while the stream's previous kernel drains and go on
// the moment that kernel's writes are visible (programmatic dependent launch).
// After anything but a kernel, an ordinary launch.
//
// Ordinary back-to-back launches of one stream start on a grid of about 2 us
// here, 2-3 us after the previous kernel's end (kernels of 1 / 3 / 5 us on 608
// CTAs repeat every 4.1 / 6.2 / 8.2 us); dependent ones repeat every 2.1 / 4.2
// / 6.2 us.  Same runs, ordinary -> dependent, executes queued back to back: c2c
// 1024 x 4096 15.4 -> 13.0 us, 2^24 130.0 -> 116.3, 2^22 40.1 -> 31.3, 2^19 12.3 ->
// 8.2, r2c 2^18 x 61 72.0 -> 63.6, 4096^2 r2c + c2r 143.3 -> 120.7, 1024 x 512 c2c
// 12.3 -> 8.0 (8.0 .. 10 from run to run; all with the tiles' forms of
// fft_device.cuh).  An execute that the host waits for keeps only what its own
// launches overlap: with all of the tiles' changes c2c 1024 x 4096, one launch,
// takes 20.7 us instead of 21.2, 512 x 512 16.2 instead of 18.7, 2^19 18.3 instead
// of 22.8.
inline cudaError_t launch_dependent(const void *fn, dim3 grid, dim3 block, void **args, size_t smem, cudaStream_t st,
                                    unsigned cluster = 1)
{
    cudaLaunchConfig_t cfg = {};
    cudaLaunchAttribute attr[2];
    cfg.gridDim = grid;
    cfg.blockDim = block;
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    if (cluster > 1) {
        attr[1].id = cudaLaunchAttributeClusterDimension;
        attr[1].val.clusterDim.x = cluster;
        attr[1].val.clusterDim.y = 1;
        attr[1].val.clusterDim.z = 1;
        cfg.numAttrs = 2;
    }
    return cudaLaunchKernelExC(&cfg, fn, args);
}

}  // namespace mgb
