// megakernel_small.cu - the path-per-thread kernel for launches that do not
// fill the GPU.
#include "megakernel.cuh"

namespace pgpu {

// Lanes of a pixel's team in the reference-exact mode (Pencil's per-pixel
// stream, both glass branches). A launch too small to fill the GPU (a worker's
// 64x64 tile has 4096 pixels) ends with its longest path, a serial chain of node
// loads through glass; such a launch gives each pixel a team of lanes that trace
// the shadow rays of its vertices side by side, `records` of them a vertex. The
// closest hits and the rest are done by every lane of a team alike, so a team
// pays as long as the GPU has issue slots to spare, which path tracing, whose
// vertices are mostly closest hits, uses up sooner (pixels per SM below).
// Teams of 8 / 4 / 2 lanes by one lane's time, rooms of 14 to 252 primitives of
// every kind, 1 to 9 samples:
//   Whitted, 6 records: 4,096 pixels 0.43-0.71 / 0.63-0.80 / 0.70-0.90; 16,384
//     0.47-0.99 / 0.56-0.95 / 0.60-0.78; 25,600 0.49-1.07 / 0.62-1.15 /
//     0.59-0.88; 73,984 0.76-1.21 / 0.90-1.35 / 0.70-0.92
//   Whitted, 4: 16,384 0.50-1.08 / 0.53-0.84 / 0.62-0.79; 37,632 0.61-1.16 /
//     0.59-0.87 / 0.59-0.86; 73,984 - / 0.66-0.94 / 0.68-0.89
//   Whitted, 1: 9,216 0.86-1.06 / 0.79-1.00 / 0.84-1.00; 37,632 - / 0.82-1.24 /
//     0.70-1.00; 73,984 - / - / 0.78-1.03; 2: 73,984 - / - / 0.73-0.94
//   path tracing, 3: 4,096 0.54-0.86 / 0.59-0.80 / 0.67-0.84; 6,144 0.68-1.31 /
//     0.77-1.08 / 0.78-0.96; 9,216 0.87-1.46 / 0.89-1.24 / 0.87-1.13
//   path tracing, 1: 1,024 0.53-0.69 / 0.56-0.78 / 0.73-0.88; 4,096 0.86-1.14 /
//     0.81-1.03 / 0.88-0.96; 6,144 - / - / 0.83-1.12; 2: 6,144 - / - / 0.74-0.96
static int team_lanes(int mode, long long records, long long pixels) {
    const double per_sm = (double)pixels / 148;
    if (records < 1) return 1;
    if (mode != kModeWhitted) {
        if (per_sm <= 32) return records >= 3 ? 8 : 4;
        return records >= 2 && per_sm <= 48 ? 2 : 1;
    }
    if (records >= 5 && per_sm <= 128) return 8;
    if (records <= 4 && per_sm <= (records >= 3 ? 256 : 64)) return 4;
    return per_sm <= (records >= 2 ? 512 : 256) ? 2 : 1;
}

cudaError_t launch_mk_small(const SceneView& S, const PathParams& P, int G, long long threads,
                            float* out, float* m2, cudaStream_t st, bool* done) {
    *done = threads <= kMkSmallThreads;
    if (!*done) return cudaSuccess;
    mk_render<false, false, false, true, false, kMkSmallBlocks>
        <<<mk_grid(threads), kMkBlock, kMkSmem, st>>>(S, P, G, 32, out, m2, nullptr);
    return cudaGetLastError();
}

cudaError_t launch_mk_team(const SceneView& S, const PathParams& P, bool wide, long long records,
                           long long pixels, float* out, float* m2, cudaStream_t st, bool* done) {
    const int team = team_lanes(P.mode, records, pixels), per_warp = 32 / team;
    *done = team > 1;
    if (!*done) return cudaSuccess;
    const unsigned grid = mk_grid(pixels * team);
    if (wide)
        mk_render<false, true, true, true, true, kMkSmallBlocks>
            <<<grid, kMkBlock, kMkSmem, st>>>(S, P, 1, per_warp, out, m2, nullptr);
    else
        mk_render<false, true, true, false, true, kMkSmallBlocks>
            <<<grid, kMkBlock, kMkSmem, st>>>(S, P, 1, per_warp, out, m2, nullptr);
    return cudaGetLastError();
}

}  // namespace pgpu
