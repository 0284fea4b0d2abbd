// megakernel.cuh - the path-per-thread kernel, shared by megakernel.cu (launches
// that fill the GPU), megakernel_small.cu (those that do not) and the two
// megakernel_found files (the same for frames whose camera hits are given). Each
// has its own instantiations: with both register budgets in one translation unit
// the compiler no longer inlines the path loop into the larger launches' kernel
// (100,000-sphere cloud, 3.7M paths: 21.2 -> 31.3 ms).
#pragma once

#include <cuda_runtime.h>

#include "host_internal.h"
#include "path.cuh"

namespace pgpu {

constexpr int kMkBlock = 128;
constexpr int kMkShared = 16;   // stack entries per thread kept in shared memory
constexpr size_t kMkSmem = (size_t)kMkShared * kMkBlock * 8;

// A launch that does not fill the GPU twice at four blocks per SM waits for its
// longest paths rather than for issue slots, and gets the registers instead
// (128, next to no spills). 8 / 4 blocks: 19,200 paths of three spheres 0.068 /
// 0.062 ms, 12,288 among 20,000 spheres 0.334 / 0.271, 20,000 on a mesh 0.591 /
// 0.512, 120,000 in a room 1.16 / 1.10; 230,400 among 20,000 spheres 0.69 / 0.79,
// 262,144 on a mesh 1.70 / 1.93. The reference-exact tiles, which are always
// that small, 1.81 / 1.47 and 0.42 / 0.31.
constexpr int kMkSmallBlocks = 4;
constexpr long long kMkSmallThreads = 2LL * 148 * kMkSmallBlocks * 128;

// Held to 64 registers (eight blocks of 128 threads per SM) otherwise: more
// resident warps hide more of the divergent paths' load latency than the spilled
// words cost. Sphere-cloud frame 85.8 ms at the compiler's choice (96-128
// registers) -> 73.4 at 72 -> 71.8 at 64; mesh frame 443.5 -> 378.0 ->
// 382.3 ms.
constexpr int kMkMinBlocks = 8;

// FOUND: entry k of `found` is the closest hit of path k's camera ray.
template <bool COUNT, bool TREE, bool PIXEL_SEQ, bool WIDE, bool COOP, int MINB, bool FOUND = false>
__global__ void __launch_bounds__(kMkBlock, MINB)
mk_render(SceneView S, PathParams P, int G, int per_warp, float* __restrict__ out,
          float* __restrict__ m2, unsigned long long* __restrict__ counters,
          const float4* __restrict__ found = nullptr) {
    extern __shared__ int smem[];
    TravStack<kMkShared> stk;
    stk.sref = smem + threadIdx.x;
    stk.st = reinterpret_cast<float*>(smem + kMkShared * blockDim.x) + threadIdx.x;
    stk.stride = blockDim.x;
    RayCount rc = {};
    // COOP: a team of 32 / per_warp lanes for each of the warp's pixels
    const int team = COOP ? 32 / per_warp : 1;
    Tracer<kMkShared, COUNT, WIDE, COOP> tr{S, P, stk, rc, team};
    const long long gid = ((long long)blockIdx.x * blockDim.x + threadIdx.x) / team;
    const bool tile = P.tile_w > 0;
    const int outW = tile ? P.tile_w : P.W, outH = tile ? P.tile_h : P.H;
    const long long npix = (long long)outW * outH;
    const long long pix = gid / G;
    const int lane_g = (int)(gid % G);
    const bool active = pix < npix;
    V3 acc = v3(0, 0, 0), acc2 = v3(0, 0, 0);
    if (active) {
        // pixel of the full image
        const int i = (int)(pix % outW) + (tile ? P.tile_x : 0);
        const int j = (int)(pix / outW) + (tile ? P.tile_y : 0);
        if (PIXEL_SEQ) {
            Rng rng{pixel_seed(i, j)};
            for (int sy = 0; sy < P.n; ++sy) {
                for (int sx = 0; sx < P.n; ++sx) {
                    float u, v;
                    sample_uv(i, j, sx, sy, P.W, P.H, P.n, rng, u, v, P.worker != 0);
                    V3 c = tr.template sample<TREE>(camera_ray(S.cam, u, v), rng);
                    acc = acc + c;
                    acc2 = acc2 + c * c;
                }
            }
        } else {
            for (int s = lane_g; s < P.spp; s += G) {
                Rng rng{path_seed(i, j, s + P.sample_offset, P.salt)};
                float u, v;
                sample_uv(i, j, s % P.n, s / P.n, P.W, P.H, P.n, rng, u, v, P.worker != 0);
                V3 c;
                if constexpr (FOUND)
                    c = tr.template sample<TREE, true>(camera_ray(S.cam, u, v), rng,
                                                       found + pix * P.spp + s);
                else
                    c = tr.template sample<TREE>(camera_ray(S.cam, u, v), rng);
                acc = acc + c;
                acc2 = acc2 + c * c;
            }
        }
    }
    for (int off = G >> 1; off > 0; off >>= 1) {
        acc.x += __shfl_xor_sync(0xffffffffu, acc.x, off);
        acc.y += __shfl_xor_sync(0xffffffffu, acc.y, off);
        acc.z += __shfl_xor_sync(0xffffffffu, acc.z, off);
        acc2.x += __shfl_xor_sync(0xffffffffu, acc2.x, off);
        acc2.y += __shfl_xor_sync(0xffffffffu, acc2.y, off);
        acc2.z += __shfl_xor_sync(0xffffffffu, acc2.z, off);
    }
    if (active && lane_g == 0 && (!COOP || threadIdx.x % team == 0)) {
        const float denom = (float)P.spp;
        out[3 * pix + 0] = acc.x / denom;
        out[3 * pix + 1] = acc.y / denom;
        out[3 * pix + 2] = acc.z / denom;
        if (m2) {
            m2[3 * pix + 0] = acc2.x / denom;
            m2[3 * pix + 1] = acc2.y / denom;
            m2[3 * pix + 2] = acc2.z / denom;
        }
    }
    if (COUNT) {
        unsigned long long v[6] = {rc.ext, rc.shadow, rc.ref, rc.tc.nodes, rc.tc.leaf_bytes,
                                   rc.tc.prims};
#pragma unroll
        for (int k = 0; k < 6; ++k) {
            unsigned long long x = v[k];
            for (int off = 16; off > 0; off >>= 1) x += __shfl_xor_sync(0xffffffffu, x, off);
            if ((threadIdx.x & 31) == 0) atomicAdd(counters + k, x);
        }
    }
}

inline unsigned mk_grid(long long threads) {
    return (unsigned)((threads + kMkBlock - 1) / kMkBlock);
}

}  // namespace pgpu
