// gbmp_rrtc_k_lo.cu -- single-problem planning kernels for 1 to 4 spheres per lane (one of the
// four translation units that instantiate the planner's kernels, so that they compile in
// parallel).
#include "gbmp_rrtc_device.cuh"

namespace gbmp {
GBMP_RRTC_DEFINE_LAUNCHER(rrtc_launch_lo, 1)

// One problem with the edge checks by chunks, for every robot whose spheres a lane are then no
// matter.  Bounded to 168 registers it takes 120, so that four blocks fit on an SM.  At 1,024
// lanes, p50 on the shelf (range 0.1) and ten problems without a path, all lanes at once: 0.45
// ms and 53 ms; bounded to four blocks (111 registers) 0.46 and 54, to five with chunks of 4
// (90 registers) 0.51 and 43; k_rrtc 0.68 and 67.
__global__ void __launch_bounds__(kRrtcThreads, 3) k_rrtc_chunk(DevRobot R, DevEnv E, RrtcDev P, RrtcParams prm) {
    if ((int)blockIdx.x >= prm.early) {   // (bounded; a problem that has ended lets everyone go)
        if (threadIdx.x == 0)
            for (int poll = 0; poll < kRrtcEarlyPolls; ++poll) {
                if (*(volatile int *)P.state != kStRunning || *(volatile int *)(P.state + 5) >= kRrtcEarlyIters) break;
                __nanosleep(1000);
            }
        __syncthreads();
    }
    rrtc_lane<1, true, kRrtcSoloChunk>(R, E, P, prm, blockIdx.x);
}

cudaError_t rrtc_launch_chunk(int grid, size_t smem, cudaStream_t st, const DevRobot &R, const DevEnv &E,
                            const RrtcDev &P, const RrtcParams &prm) {
    const cudaError_t ce = rrtc_raise_smem(k_rrtc_chunk, smem);
    if (ce != cudaSuccess) return ce;
    k_rrtc_chunk<<<grid, kRrtcThreads, smem, st>>>(R, E, P, prm);
    return cudaGetLastError();
}
}  // namespace gbmp
