// frames.cu -- per-epoch ITRS->GCRS matrix table on the device (replaces TimePointParamsKernel and
// the seven batched 3x3 GEMMs of lib/force_model/src/time_points.cu:26-71,146-201). One block per epoch
// (frames_block.cuh).
#include "frames_block.cuh"

namespace gpop {

__global__ void __launch_bounds__(kFrameThreads) frames_kernel(FrameData fd, int y, int mo, int d, int hh, int mi,
    FrameRange a, FrameRange b)
{
    const bool second = (int)blockIdx.x >= a.count;
    const FrameRange r = second ? b : a;
    const int e = (int)blockIdx.x - (second ? a.count : 0);
    frames_epoch(fd, y, mo, d, hh, mi, r.sec_args[e], r.m_out + (size_t)e * 9, r.mjd_out ? r.mjd_out + e : nullptr);
}

cudaError_t launch_frames(const FrameData& fd, int y, int mo, int d, int hh, int mi, const FrameRange& a,
    const FrameRange& b, cudaStream_t s)
{
    if (a.count + b.count <= 0)
        return cudaSuccess;
    frames_kernel<<<a.count + b.count, kFrameThreads, 0, s>>>(fd, y, mo, d, hh, mi, a, b);
    return cudaGetLastError();
}

} // namespace gpop
