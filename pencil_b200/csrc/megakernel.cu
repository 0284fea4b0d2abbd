// megakernel.cu - the plain GPU path tracer: one thread per (pixel, sample
// lane), every bounce, shadow ray and the Whitted continuation in one kernel.
// It traverses the same 4-wide tree as the wavefront by default (the
// baseline the wavefront is measured against), or Pencil's binary tree with
// PGPU_FLAG_BINARY_TREE.
//
// Thread mapping. Counter RNG: G = largest power of two <= min(spp, 32)
// lanes share a pixel; lane g traces samples g, g + G, ... and the G partial
// sums are combined by a butterfly of warp shuffles, so the pixel sum is
// deterministic. Per-pixel RNG: one thread per pixel consumes Pencil's
// per-pixel xorshift32 stream over its samples in Pencil's order.
#include "megakernel.cuh"

namespace pgpu {

// megakernel_small.cu: launches that do not fill the GPU (*done), with a team of
// lanes per pixel in the reference-exact mode.
cudaError_t launch_mk_small(const SceneView& S, const PathParams& P, int G, long long threads,
                            float* out, float* m2, cudaStream_t st, bool* done);
cudaError_t launch_mk_team(const SceneView& S, const PathParams& P, bool wide, long long records,
                           long long pixels, float* out, float* m2, cudaStream_t st, bool* done);

template <bool COUNT, bool TREE, bool PIXEL_SEQ, bool WIDE>
static cudaError_t launch_mk(const SceneView& S, const PathParams& P, int G, long long records,
                             float* out, float* m2, unsigned long long* counters,
                             cudaStream_t st) {
    const long long threads =
        (P.tile_w > 0 ? (long long)P.tile_w * P.tile_h : (long long)P.W * P.H) * G;
    if constexpr (!COUNT && ((TREE && PIXEL_SEQ) || (!TREE && !PIXEL_SEQ && WIDE))) {
        bool done = false;
        const cudaError_t e = TREE ? launch_mk_team(S, P, WIDE, records, threads, out, m2, st,
                                                    &done)
                                   : launch_mk_small(S, P, G, threads, out, m2, st, &done);
        if (done || e != cudaSuccess) return e;
    }
    mk_render<COUNT, TREE, PIXEL_SEQ, WIDE, false, kMkMinBlocks>
        <<<mk_grid(threads), kMkBlock, kMkSmem, st>>>(S, P, G, 32, out, m2, counters);
    return cudaGetLastError();
}

// megakernel_found.cu
cudaError_t launch_mk_found(const SceneView& S, const PathParams& P, int G, const float4* found,
                            long long threads, float* out, float* m2, cudaStream_t st);

// found: the closest hits of the camera rays, path by path (or null).
cudaError_t launch_megakernel(const SceneView& S, const RenderCfg& c, const float4* found,
                              float* out, float* m2, unsigned long long* counters,
                              cudaStream_t st) {
    PathParams P{c.W, c.H, c.n, c.spp, c.depth, c.mode, c.rng, c.glass, c.soft, c.bias, c.salt,
                 c.sample_offset, c.mis ? 1 : 0, c.win[0], c.win[1], c.win[2], c.win[3],
                 c.worker ? 1 : 0};
    const bool seq = c.rng == PGPU_RNG_PIXEL_SEQUENTIAL;
    const bool tree = c.glass == PGPU_GLASS_BOTH_BRANCHES;
    int G = 1;
    if (!seq) {
        int lim = c.spp < 32 ? c.spp : 32;
        while (G * 2 <= lim) G *= 2;
    }
    if (found) return launch_mk_found(S, P, G, found, c.pixels() * G, out, m2, st);
    const bool wide = !c.binary_tree;
#define PGPU_MK_CASE(CNT, TR, SQ)                                                \
    if (c.count == CNT && tree == TR && seq == SQ)                               \
        return wide ? launch_mk<CNT, TR, SQ, true>(S, P, G, c.records, out, m2, counters, st) \
                    : launch_mk<CNT, TR, SQ, false>(S, P, G, c.records, out, m2, counters, st);
    PGPU_MK_CASE(false, false, false)
    PGPU_MK_CASE(false, false, true)
    PGPU_MK_CASE(false, true, false)
    PGPU_MK_CASE(false, true, true)
    PGPU_MK_CASE(true, false, false)
    PGPU_MK_CASE(true, false, true)
    PGPU_MK_CASE(true, true, false)
    PGPU_MK_CASE(true, true, true)
#undef PGPU_MK_CASE
    return cudaErrorInvalidValue;
}

}  // namespace pgpu
