// megakernel_found.cu - the path-per-thread kernel for frames whose camera rays
// were traced as packets (wavefront_camera_hits).
#include "megakernel.cuh"

namespace pgpu {

// megakernel_found_small.cu
cudaError_t launch_mk_found_small(const SceneView& S, const PathParams& P, int G,
                                  const float4* found, long long threads, float* out, float* m2,
                                  cudaStream_t st);

cudaError_t launch_mk_found(const SceneView& S, const PathParams& P, int G, const float4* found,
                            long long threads, float* out, float* m2, cudaStream_t st) {
    if (threads <= kMkSmallThreads)
        return launch_mk_found_small(S, P, G, found, threads, out, m2, st);
    mk_render<false, false, false, true, false, kMkMinBlocks, true>
        <<<mk_grid(threads), kMkBlock, kMkSmem, st>>>(S, P, G, 32, out, m2, nullptr, found);
    return cudaGetLastError();
}

}  // namespace pgpu
