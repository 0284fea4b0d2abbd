// megakernel_small.cu - the path-per-thread kernel for launches that do not
// fill the GPU.
#include "megakernel.cuh"

namespace pgpu {

// A launch that does not fill the GPU twice at four blocks per SM waits for its
// longest paths rather than for issue slots, and gets the registers instead
// (128, next to no spills). 8 / 4 blocks: 19,200 paths of three spheres 0.068 /
// 0.062 ms, 12,288 among 20,000 spheres 0.334 / 0.271, 20,000 on a mesh 0.591 /
// 0.512, 120,000 in a room 1.16 / 1.10; 230,400 among 20,000 spheres 0.69 / 0.79,
// 262,144 on a mesh 1.70 / 1.93. The reference-exact tiles, which are always
// that small, 1.81 / 1.47 and 0.42 / 0.31.
constexpr int kMkSmallBlocks = 4;
constexpr long long kMkSmallThreads = 2LL * 148 * kMkSmallBlocks * 128;

// Pixels per warp of the reference-exact mode (Pencil's per-pixel stream, both
// glass branches). A launch too small to fill the GPU (a worker's 64x64 tile
// has 4096 pixels) ends with its longest path, a serial chain of node loads
// through glass. Such a launch gives each pixel a team of lanes that trace
// the shadow rays of its vertices side by side, as long as its warps fit the
// GPU at once (32 on each of 148 SMs, what 64 registers allow). Teams of 8: a
// 64x64 tile of six rooms of 63 primitives took 4.12 / 0.67 / 1.13 / 12.2 /
// 1.36 / 6.5 ms with one lane per pixel, 1.93 / 0.45 / 0.67 / 5.4 / 0.73 / 3.3
// with 8 (6 shadow rays a vertex), 2.82 / 0.90 / 0.98 / 6.1 / 1.02 / 2.9 with
// 32: more warps than a team can use only take issue slots from each other.
constexpr long long kTeamWarps = 148 * 32;
constexpr int kMaxTeam = 8;
static int pixels_per_warp(long long pixels) {
    int per = 32 / kMaxTeam;
    while (per < 32 && (pixels + per - 1) / per > kTeamWarps) per *= 2;
    return per;
}

cudaError_t launch_mk_small(const SceneView& S, const PathParams& P, int G, long long threads,
                            float* out, float* m2, cudaStream_t st, bool* done) {
    *done = threads <= kMkSmallThreads;
    if (!*done) return cudaSuccess;
    mk_render<false, false, false, true, false, kMkSmallBlocks>
        <<<mk_grid(threads), kMkBlock, kMkSmem, st>>>(S, P, G, 32, out, m2, nullptr);
    return cudaGetLastError();
}

cudaError_t launch_mk_team(const SceneView& S, const PathParams& P, bool wide, long long pixels,
                           float* out, float* m2, cudaStream_t st, bool* done) {
    const int per_warp = pixels_per_warp(pixels);
    *done = per_warp < 32;
    if (!*done) return cudaSuccess;
    const unsigned grid = mk_grid(pixels * (32 / per_warp));
    if (wide)
        mk_render<false, true, true, true, true, kMkSmallBlocks>
            <<<grid, kMkBlock, kMkSmem, st>>>(S, P, 1, per_warp, out, m2, nullptr);
    else
        mk_render<false, true, true, false, true, kMkSmallBlocks>
            <<<grid, kMkBlock, kMkSmem, st>>>(S, P, 1, per_warp, out, m2, nullptr);
    return cudaGetLastError();
}

}  // namespace pgpu
