// gbmp_rrtc_k_lo.cu -- single-problem planning kernels for 1 to 4 spheres per lane (one of the
// four translation units that instantiate the planner's kernels, so that they compile in
// parallel).
#include "gbmp_rrtc_device.cuh"

namespace gbmp {
GBMP_RRTC_DEFINE_LAUNCHER(rrtc_launch_lo, 1)

// One problem with the edge checks by chunks, for every robot whose spheres a lane are then no
// matter.  At most 168 registers: three blocks an SM measured 646 us at 1,024 lanes (the
// shelf, range 0.1; as few as one block 654), four 736, five 842; k_rrtc 866.
__global__ void __launch_bounds__(kRrtcThreads, 3) k_rrtc_chunk(DevRobot R, DevEnv E, RrtcDev P, RrtcParams prm) {
    rrtc_lane<1, true, kRrtcSoloChunk>(R, E, P, prm, blockIdx.x);
}

cudaError_t rrtc_launch_chunk(int grid, size_t smem, cudaStream_t st, const DevRobot &R, const DevEnv &E,
                            const RrtcDev &P, const RrtcParams &prm) {
    cudaError_t ce = cudaFuncSetAttribute(k_rrtc_chunk, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (ce != cudaSuccess) return ce;
    k_rrtc_chunk<<<grid, kRrtcThreads, smem, st>>>(R, E, P, prm);
    return cudaGetLastError();
}
}  // namespace gbmp
