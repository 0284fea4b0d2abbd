// megakernel_found_small.cu - megakernel_found.cu's kernel for launches that do
// not fill the GPU.
#include "megakernel.cuh"

namespace pgpu {

cudaError_t launch_mk_found_small(const SceneView& S, const PathParams& P, int G,
                                  const float4* found, long long threads, float* out, float* m2,
                                  cudaStream_t st) {
    mk_render<false, false, false, true, false, kMkSmallBlocks, true>
        <<<mk_grid(threads), kMkBlock, kMkSmem, st>>>(S, P, G, 32, out, m2, nullptr, found);
    return cudaGetLastError();
}

}  // namespace pgpu
