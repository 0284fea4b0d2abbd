// tonemap.cu - Pencil's HDR -> 8-bit output path on the device
// (write_image / color_to_rgb8, src/image_io.hpp:40-113; tone curves,
// src/tonemap.hpp:27-61): exposure, tone curve, clamp, gamma 2.2, 8 bits.
//
// Exposure, ACES and Reinhard are plain float arithmetic and round on the
// device as on the host (--fmad=false, IEEE division). The gamma step calls
// the host's powf, whose last bits the device's powf need not match. The
// 8-bit result of that step is a non-decreasing function of the clamped
// value, so it is fully described by 255 thresholds: t[k] is the smallest
// float whose byte is >= k under the host's own powf. They are computed on
// the host by bisection over float bit patterns, once per process, and the
// kernel counts the thresholds at or below each value: the bytes equal the
// host's for every input (tests check the monotonicity over all floats in
// [0, 1] and the bytes against the oracle).
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstdint>
#include <cstring>
#include <mutex>

namespace pgpu {

struct GammaThresholds {
    float t[256];   // t[0] unused; t[k], k = 1..255
};

namespace {

uint8_t host_gamma_byte(float x) {
    x = x < 0.0f ? 0.0f : (x > 1.0f ? 1.0f : x);
    x = std::pow(x, 1.0f / 2.2f);
    return (uint8_t)(x * 255.0f + 0.5f);
}

float bits_float(uint32_t b) {
    float f;
    std::memcpy(&f, &b, 4);
    return f;
}

const GammaThresholds& thresholds() {
    static GammaThresholds g;
    static std::once_flag once;
    std::call_once(once, [] {
        g.t[0] = 0.0f;
        const uint32_t one = 0x3f800000u;   // 1.0f; non-negative floats order as their bits
        for (int k = 1; k < 256; ++k) {
            uint32_t lo = 0, hi = one;       // host_gamma_byte(1) = 255 >= k
            while (lo < hi) {
                const uint32_t mid = lo + (hi - lo) / 2;
                if (host_gamma_byte(bits_float(mid)) >= k) hi = mid;
                else lo = mid + 1;
            }
            g.t[k] = bits_float(lo);
        }
    });
    return g;
}

}  // namespace

// Exactly, the byte of a clamped value is found in two steps: the value's
// exponent and top 7 mantissa bits pick a cell whose lower end has `base`
// thresholds at or below it, and no cell holds a second threshold (a cell is
// 1/128 of its octave; the closest thresholds of the top octave lie 1.5 cells
// apart, those of lower octaves further; tone_table_host checks it), so one
// comparison with t[base + 1] finishes the count. Values below 2^-20 lie below
// t[1] = (0.5 / 255)^2.2 (checked too). Counting on while thresholds are at or
// below the value, which needs neither, makes a 4K frame 0.6 us slower.
constexpr int kCellShift = 23 - 7;
constexpr uint32_t kCellFirst = 0x35800000u;             // 2^-20
constexpr int kCells = (int)((0x3f800000u - kCellFirst) >> kCellShift) + 1;   // up to 1.0

struct ToneTable {
    float t[257];             // thresholds; t[256] = infinity (never reached)
    uint8_t base[kCells + 3];
};

__device__ __forceinline__ float rcp_approx(float x) {
    float y;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}
__device__ __forceinline__ float log2_approx(float x) {
    float y;
    asm("lg2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}
__device__ __forceinline__ float exp2_approx(float x) {
    float y;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}

template <int MODE>
__device__ __noinline__ uint32_t tone_byte(float x, const ToneTable* __restrict__ table) {
    if (MODE == 1) {
        const float a = 2.51f, b = 0.03f, c = 2.43f, d = 0.59f, f = 0.14f;
        const float y = (x * (a * x + b)) / (x * (c * x + d) + f);
        x = 0.0f < y ? y : 0.0f;                       // std::max(0.0f, y)
    } else if (MODE == 2) {
        x = x / (1.0f + x);
    }
    x = (x < 0.0f) ? 0.0f : (x > 1.0f) ? 1.0f : x;     // clampf
    // below the first cell (and NaN): no threshold is at or below the value
    if (!(x >= __uint_as_float(kCellFirst))) return 0;
    const uint32_t k = __ldg(&table->base[(__float_as_uint(x) - kCellFirst) >> kCellShift]);
    return k + (__ldg(&table->t[k + 1]) <= x ? 1u : 0u);
}

// The byte as 255 y^(1/2.2) rounded, from the hardware's approximate
// reciprocal, log2 and exp2. Their errors move that value by less than 5e-4
// (log2: 2^-22 of at most 20, divided by 2.2; the others and the roundings a
// few 2^-23), and the host's powf by 255 x 2^-23, so the byte is certain where
// the value is more than 1e-3 from the midpoint of two bytes. `sure` is false
// elsewhere, for the 0.2% that tone_byte decides, and for magnitudes whose
// products could overflow.
template <int MODE>
__device__ __forceinline__ uint32_t tone_byte_fast(float x, bool& sure) {
    float y = x;
    if (MODE == 1)
        y = __fmul_rn(x * __fmaf_rn(2.51f, x, 0.03f),
                      rcp_approx(__fmaf_rn(x, __fmaf_rn(2.43f, x, 0.59f), 0.14f)));
    else if (MODE == 2)
        y = x * rcp_approx(1.0f + x);
    y = __saturatef(y);                                // NaN: 0, as the clamp's byte
    const float v = 255.0f * exp2_approx(log2_approx(y) * (1.0f / 2.2f));
    const float m = v + 12582912.0f;                   // 1.5 * 2^23: v rounded, in the low bits
    sure = fabsf(v - (m - 12582912.0f)) < 0.499f && fabsf(x) < 1e15f;
    return __float_as_uint(m) & 0xffu;
}

// MODE: 0 none, 1 ACES, 2 Reinhard (pencil::ToneMap order). What has to move
// is 4 bytes read and 1 written per channel: a thread takes 16 channels as
// four 16-byte loads and one 16-byte store; the table stays in global memory,
// for the few channels that need it. `head` channels before the first 16-byte
// boundary and the last n3 % 16 go one by one. A call for a 3840x2160 frame
// (ACES, device buffers) takes 38 us, of which 19 are its 124 MB at the
// measured copy rate; with 4-byte loads, 1-byte stores, an IEEE division and
// a search of 8 dependent shared loads per channel it took 127, with that
// division and the table in shared memory 57.
template <int MODE>
__global__ void __launch_bounds__(256)
tm_rgb8(const float* __restrict__ hdr, long long n3, long long head, float e,
        const ToneTable* __restrict__ table, uint8_t* __restrict__ out) {
    const long long n16 = n3 > head ? (n3 - head) >> 4 : 0;
    const long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x;
    if (i < n16) {
        const float4* p = reinterpret_cast<const float4*>(hdr + head) + 4 * i;
        float4 v[4] = {__ldcs(p), __ldcs(p + 1), __ldcs(p + 2), __ldcs(p + 3)};
        uint32_t w[4];
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            v[k] = make_float4(v[k].x * e, v[k].y * e, v[k].z * e, v[k].w * e);
            bool s0, s1, s2, s3;
            uint32_t b0 = tone_byte_fast<MODE>(v[k].x, s0), b1 = tone_byte_fast<MODE>(v[k].y, s1);
            uint32_t b2 = tone_byte_fast<MODE>(v[k].z, s2), b3 = tone_byte_fast<MODE>(v[k].w, s3);
            if (!(s0 && s1 && s2 && s3)) {
                if (!s0) b0 = tone_byte<MODE>(v[k].x, table);
                if (!s1) b1 = tone_byte<MODE>(v[k].y, table);
                if (!s2) b2 = tone_byte<MODE>(v[k].z, table);
                if (!s3) b3 = tone_byte<MODE>(v[k].w, table);
            }
            w[k] = b0 | b1 << 8 | b2 << 16 | b3 << 24;
        }
        reinterpret_cast<uint4*>(out + head)[i] = make_uint4(w[0], w[1], w[2], w[3]);
    }
    // the ragged ends: [0, head) and [head + 16 n16, n3)
    const long long rest = n3 - 16 * n16;
    if (i < rest) {
        const long long at = i < head ? i : i + 16 * n16;
        out[at] = (uint8_t)tone_byte<MODE>(hdr[at] * e, table);
    }
}

// The table for upload to the device; null where the host's powf gives
// thresholds that tone_byte does not count exactly.
const void* tone_table_host(size_t* bytes) {
    static ToneTable g;
    static std::once_flag once;
    static bool exact = true;
    std::call_once(once, [] {
        const GammaThresholds& th = thresholds();
        std::memcpy(g.t, th.t, sizeof(th.t));
        g.t[256] = INFINITY;
        exact = g.t[1] >= bits_float(kCellFirst);
        for (int c = 0, k = 0; c < kCells; ++c) {
            const float lo = bits_float(kCellFirst + ((uint32_t)c << kCellShift));
            while (k < 255 && g.t[k + 1] <= lo) ++k;
            g.base[c] = (uint8_t)k;
            // (the second threshold beyond this cell's lower end, if in the cell)
            exact = exact && !(k < 254 && g.t[k + 2] < bits_float(
                                   kCellFirst + ((uint32_t)(c + 1) << kCellShift)));
        }
    });
    *bytes = sizeof(ToneTable);
    return exact ? &g : nullptr;
}

cudaError_t launch_tonemap(const float* d_hdr, long long n_pixels, int mode, float exposure,
                           uint8_t* d_out, const void* d_table, cudaStream_t st) {
    const float e = std::pow(2.0f, exposure);             // tonemap_color's exposure
    const long long n3 = 3 * n_pixels;
    // channels up to the first 16-byte boundary of the bytes; where the floats
    // are not on one there too, every channel goes one by one
    long long head = (long long)((16 - reinterpret_cast<uintptr_t>(d_out) % 16) % 16);
    if (head > n3 || (reinterpret_cast<uintptr_t>(d_hdr) + 4 * (uintptr_t)head) % 16 != 0)
        head = n3;
    const long long items = std::max((n3 - head) / 16, n3 - (n3 - head) / 16 * 16);
    const unsigned grid = (unsigned)((items + 255) / 256);
    const ToneTable* t = static_cast<const ToneTable*>(d_table);
    if (mode == 1) tm_rgb8<1><<<grid, 256, 0, st>>>(d_hdr, n3, head, e, t, d_out);
    else if (mode == 2) tm_rgb8<2><<<grid, 256, 0, st>>>(d_hdr, n3, head, e, t, d_out);
    else tm_rgb8<0><<<grid, 256, 0, st>>>(d_hdr, n3, head, e, t, d_out);
    return cudaGetLastError();
}

}  // namespace pgpu
