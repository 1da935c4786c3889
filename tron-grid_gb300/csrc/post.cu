// Bloom + post-process chain (include/tg_post.h) on sm_103a.
//
// The reference's bloomExtractMain / bloomDownsampleMain / bloomUpsampleMain
// (src/bloom_downsample.slang) and postprocessMain (src/postprocess.slang),
// in the reference host's order (src/main.cpp:306-430): extract into mip 0 and
// downsample into mips 1..N-1 (one launch builds mips 0..5: each CTA owns an
// aligned tile of every level), upsample mip N-2 .. 0 in place (each texel
// reads the next mip and its own value, so no texel is read after another
// thread writes it), then the post pass.  The bloom chain is one allocation of
// rgba16f mips (8 B per texel, as the reference's bloom image).
//
// All arithmetic is explicitly rounded IEEE single precision in the shaders'
// order (sums left to right, no contraction into FMA); only the sRGB curve's
// power (exp2f / log2f) is CUDA's.  Quotients by a divisor that several of them
// share are formed from its correctly rounded reciprocal and FMA residuals, which
// rounds correctly while nothing overflows (Markstein 1990; Brisebarre, Muller
// and Raina 2004).
//
// What bounds it: FP32 issue in the extraction and the post pass (the 4K chain's
// compulsory 100 MB take 15 us of the 6.8 TB/s a copy reaches), launch latency in
// the small upsamples.  So work that neighbours share is done once: an upsample
// thread owns the 2x2 texels that share a tent, a post thread two pixels that
// share a bloom texel (and, away from the corners, all three samples of a pixel
// are one), and the launches overlap by programmatic dependent launch.  Measured:
// the 3840x2160 chain (rgba16f to BGRA8) 166 -> 105 us, 1281x721 (rgba32f to
// rgba32f) 49.8 -> 24.3 us.
#include <cuda_fp16.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstdint>
#include <new>

#include "svgf_device.cuh"
#include "svgf_internal.h"
#include "tg_post.h"

namespace tg {
namespace {

constexpr int kPostTX = 32, kPostTY = 8;
constexpr int kMaxMips = 16;

__device__ __forceinline__ float add(float a, float b) { return __fadd_rn(a, b); }
__device__ __forceinline__ float sub(float a, float b) { return __fsub_rn(a, b); }
__device__ __forceinline__ float mul(float a, float b) { return __fmul_rn(a, b); }
__device__ __forceinline__ float dv(float a, float b) { return __fdiv_rn(a, b); }

// x / y by the correctly rounded reciprocal r of y, |x| < 2^100 and x / y far
// from the subnormals (or too small to matter to the caller), or x = 0.
__device__ __forceinline__ float div_by(float x, float y, float r)
{
    float q = mul(x, r);
    q = __fmaf_rn(__fmaf_rn(-q, y, x), r, q);
    return __fmaf_rn(__fmaf_rn(-q, y, x), r, q);
}
constexpr float kDivMax = 1.2676506e30f;  // 2^100

struct C3 {
    float r, g, b;
};

__device__ __forceinline__ float lum(C3 c) { return add(add(mul(c.r, 0.2126f), mul(c.g, 0.7152f)), mul(c.b, 0.0722f)); }

__device__ __forceinline__ C3 ld_h4(const uint2* p, long long i)
{
    const uint2 u = p[i];
    const float2 a = __half22float2(*reinterpret_cast<const __half2*>(&u.x));
    const float2 b = __half22float2(*reinterpret_cast<const __half2*>(&u.y));
    return {a.x, a.y, b.x};
}

__device__ __forceinline__ void st_h4(uint2* p, long long i, C3 c)
{
    const __half2 a = __floats2half2_rn(c.r, c.g), b = __floats2half2_rn(c.b, 1.0f);
    p[i] = make_uint2(*reinterpret_cast<const uint32_t*>(&a), *reinterpret_cast<const uint32_t*>(&b));
}

template <bool F16> __device__ __forceinline__ C3 ld_hdr(const char* base, long long pitch, int x, int y)
{
    const char* row = base + y * pitch;
    if constexpr (F16) {
        return ld_h4(reinterpret_cast<const uint2*>(row), x);
    } else {
        const float4 v = reinterpret_cast<const float4*>(row)[x];
        return {v.x, v.y, v.z};
    }
}

struct Mip {
    uint2* p;
    int w, h;
};

__device__ __forceinline__ C3 round16(C3 c)
{
    return {__half2float(__float2half_rn(c.r)), __half2float(__float2half_rn(c.g)), __half2float(__float2half_rn(c.b))};
}

// Two horizontally adjacent HDR pixels (x even) of row y: one 16-byte load of
// binary16 texels where the image is aligned for it (`vec`).
template <bool F16> __device__ __forceinline__ void ld_hdr2(const char* base, long long pitch, int x, int x1, int y, bool vec, C3 (&c)[2])
{
    if (F16 && vec) {
        const uint4 u = *reinterpret_cast<const uint4*>(base + y * pitch + x * 8LL);
        const float2 a0 = __half22float2(*reinterpret_cast<const __half2*>(&u.x)), a1 = __half22float2(*reinterpret_cast<const __half2*>(&u.z));
        c[0] = {a0.x, a0.y, __half2float(__ushort_as_half((unsigned short)(u.y & 0xffffu)))};
        c[1] = {a1.x, a1.y, __half2float(__ushort_as_half((unsigned short)(u.w & 0xffffu)))};
    } else {
        c[0] = ld_hdr<F16>(base, pitch, x, y);
        c[1] = ld_hdr<F16>(base, pitch, x1, y);
    }
}

// Mip-0 texel of the extraction (bloomExtractMain) from its 2x2 HDR block, before the fp16 store.  A sample below
// the threshold is zero: its luminance is 0 and its weight 1.  (No sample is infinite and below the threshold, so
// selecting equals the shader's multiplication by 0 or 1.)
__device__ __forceinline__ C3 extract_texel(const C3 (&in)[4], float thr)
{
    C3 s[4];
    float w[4];
#pragma unroll
    for (int k = 0; k < 4; ++k) {
        C3 c = in[k];
        c = {c.r > 0.f ? c.r : 0.f, c.g > 0.f ? c.g : 0.f, c.b > 0.f ? c.b : 0.f};
        const float l = lum(c);
        const bool keep = l >= thr;
        s[k] = keep ? c : C3{0.f, 0.f, 0.f};
        w[k] = keep ? __frcp_rn(add(1.f, l)) : 1.f;
    }
    const float ws = add(add(add(w[0], w[1]), w[2]), w[3]);
    const float den = ws > 1e-7f ? ws : 1e-7f;
    auto num = [&](float C3::*m) {
        return add(add(add(mul(s[0].*m, w[0]), mul(s[1].*m, w[1])), mul(s[2].*m, w[2])), mul(s[3].*m, w[3]));
    };
    const C3 n = {num(&C3::r), num(&C3::g), num(&C3::b)};
    if (fmaxf(fmaxf(n.r, n.g), n.b) < kDivMax) {  // (a quotient too small for div_by rounds to a binary16 zero)
        const float rd = __frcp_rn(den);
        return {div_by(n.r, den, rd), div_by(n.g, den, rd), div_by(n.b, den, rd)};
    }
    return {dv(n.r, den), dv(n.g, den), dv(n.b, den)};
}

// Mip i of the box-downsample chain from the 2x2 block of mip i-1 (bloomDownsampleMain).
__device__ __forceinline__ C3 box4(const C3 (&c)[4])
{
    return {mul(add(add(add(c[0].r, c[1].r), c[2].r), c[3].r), 0.25f), mul(add(add(add(c[0].g, c[1].g), c[2].g), c[3].g), 0.25f),
            mul(add(add(add(c[0].b, c[1].b), c[2].b), c[3].b), 0.25f)};
}

// Extraction and the downsample pyramid in one launch.  Mip i texel (x, y) reads exactly the 2x2 block
// (2x, 2y) .. (2x+1, 2y+1) of mip i-1 (clamped, and the clamp never leaves the block's aligned tile because
// mip i is floor(mip i-1 / 2) wide, or 1 wide when mip i-1 is), so a CTA that owns an aligned 32x32 tile of
// mip 0 owns the (32 >> i)-square tile of every mip i <= 5, with the values as the fp16 image stores them.
//
// A thread extracts the 2x2 block of mip 0 under its mip 1 texel (all 16 HDR pixels loaded up front); the next
// two mips are exchanged between lanes (a warp's mip 1 texels are 8 x 4, lane bits x0 y0 x1 y1 x2), and only
// the last two go through shared memory: one barrier instead of one per mip.  33.1 -> 23.8 us at 3840x2160 (under ncu).
constexpr int kPyrT = 32;
constexpr int kPyrLevels = 6;
struct MipSet {
    Mip m[kPyrLevels];
    int n;  // levels built here, 1 .. kPyrLevels
};

__device__ __forceinline__ C3 shfl_xor(C3 c, int bit)
{
    return {__shfl_xor_sync(0xffffffffu, c.r, bit), __shfl_xor_sync(0xffffffffu, c.g, bit), __shfl_xor_sync(0xffffffffu, c.b, bit)};
}

// The 2x2 block {(0,0), (1,0), (0,1), (1,1)} of the level below as the downsample reads it: a level one texel
// wide or high repeats it (`w1`, `h1`).
__device__ __forceinline__ C3 box_of(C3 c00, C3 c10, C3 c01, C3 c11, bool w1, bool h1)
{
    if (w1) {
        c10 = c00;
        c11 = c01;
    }
    if (h1) {
        c01 = c00;
        c11 = c10;
    }
    const C3 c[4] = {c00, c10, c01, c11};
    return round16(box4(c));
}

template <bool HDR16>
__global__ void __launch_bounds__(256) k_bloom_pyramid(const char* hdr, long long pitch, int W, int H, MipSet ms, float thr, int vec)
{
    __shared__ C3 s3[16];  // the CTA's 4x4 texels of mip 3
    pdl_begin();
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    // mip 1 texel of this thread: warps 2 across, 4 down
    const int tx = (warp & 1) * 8 + (lane & 1) + ((lane >> 1) & 2) + ((lane >> 2) & 4);
    const int ty = (warp >> 1) * 4 + ((lane >> 1) & 1) + ((lane >> 2) & 2);
    const int x1 = blockIdx.x * (kPyrT / 2) + tx, y1 = blockIdx.y * (kPyrT / 2) + ty;
    const Mip m0 = ms.m[0];
    // every HDR load of the thread's four texels is issued before the first is used
    C3 in[4][4];
#pragma unroll
    for (int q = 0; q < 4; ++q) {
        const int x = min(2 * x1 + (q & 1), m0.w - 1), y = min(2 * y1 + (q >> 1), m0.h - 1);
#pragma unroll
        for (int j = 0; j < 2; ++j) {
            C3 row[2];
            ld_hdr2<HDR16>(hdr, pitch, min(2 * x, W - 1), min(2 * x + 1, W - 1), min(2 * y + j, H - 1), vec, row);
            in[q][2 * j] = row[0];
            in[q][2 * j + 1] = row[1];
        }
    }
    C3 t0[4];
#pragma unroll
    for (int q = 0; q < 4; ++q) {
        t0[q] = round16(extract_texel(in[q], thr));
        const int x = 2 * x1 + (q & 1), y = 2 * y1 + (q >> 1);
        if (x < m0.w && y < m0.h) st_h4(m0.p, (long long)y * m0.w + x, t0[q]);
    }
    if (ms.n < 2) return;
    // (texels outside a mip hold values that no texel inside the next one reads)
    const C3 c1 = box_of(t0[0], t0[1], t0[2], t0[3], m0.w == 1, m0.h == 1);
    if (x1 < ms.m[1].w && y1 < ms.m[1].h) st_h4(ms.m[1].p, (long long)y1 * ms.m[1].w + x1, c1);
    if (ms.n < 3) return;
    // mips 2 and 3: the lane whose two bits of the pair are 0 holds the block's first texel
    C3 c = c1;
#pragma unroll
    for (int i = 2; i < 4; ++i) {
        if (ms.n <= i) return;
        const int bx = i == 2 ? 1 : 4, by = i == 2 ? 2 : 8;
        const C3 r = shfl_xor(c, bx), d = shfl_xor(c, by), rd = shfl_xor(r, by);
        c = box_of(c, r, d, rd, ms.m[i - 1].w == 1, ms.m[i - 1].h == 1);
        const int x = x1 >> (i - 1), y = y1 >> (i - 1);
        const bool first = (lane & (i == 2 ? 3 : 15)) == 0;
        if (first && x < ms.m[i].w && y < ms.m[i].h) st_h4(ms.m[i].p, (long long)y * ms.m[i].w + x, c);
    }
    if (ms.n < 5) return;
    if ((lane & 15) == 0) s3[(ty >> 2) * 4 + (tx >> 2)] = c;
    __syncthreads();
    if (warp != 0) return;
    // mips 4 (lanes 0 .. 3) and 5 (lane 0)
    const int i4 = (lane & 1) * 2 + ((lane >> 1) & 1) * 8;
    const C3 c4 = box_of(s3[i4], s3[i4 + 1], s3[i4 + 4], s3[i4 + 5], ms.m[3].w == 1, ms.m[3].h == 1);
    const int x4 = blockIdx.x * 2 + (lane & 1), y4 = blockIdx.y * 2 + ((lane >> 1) & 1);
    if (lane < 4 && x4 < ms.m[4].w && y4 < ms.m[4].h) st_h4(ms.m[4].p, (long long)y4 * ms.m[4].w + x4, c4);
    if (ms.n < 6) return;
    const C3 r = shfl_xor(c4, 1), d = shfl_xor(c4, 2), rd = shfl_xor(r, 2);
    const C3 c5 = box_of(c4, r, d, rd, ms.m[4].w == 1, ms.m[4].h == 1);
    if (lane == 0 && int(blockIdx.x) < ms.m[5].w && int(blockIdx.y) < ms.m[5].h)
        st_h4(ms.m[5].p, (long long)blockIdx.y * ms.m[5].w + blockIdx.x, c5);
}

__global__ void __launch_bounds__(kPostTX* kPostTY) k_bloom_down(Mip s, Mip d)
{
    pdl_begin();
    const int x = blockIdx.x * kPostTX + threadIdx.x, y = blockIdx.y * kPostTY + threadIdx.y;
    if (x >= d.w || y >= d.h) return;
    C3 c[4];
#pragma unroll
    for (int k = 0; k < 4; ++k)
        c[k] = ld_h4(s.p, (long long)min(2 * y + (k >> 1), s.h - 1) * s.w + min(2 * x + (k & 1), s.w - 1));
    st_h4(d.p, (long long)y * d.w + x, box4(c));
}

// One thread per 2x2 block of texels: the four add the same tent of the next mip
// (around x / 2, y / 2).
__global__ void __launch_bounds__(kPostTX* kPostTY) k_bloom_up(Mip s, Mip d)
{
    pdl_begin();
    const int bx = blockIdx.x * kPostTX + threadIdx.x, by = blockIdx.y * kPostTY + threadIdx.y;
    if (2 * bx >= d.w || 2 * by >= d.h) return;
    uint2* o[4];
    C3 e[4];
    bool in[4];
#pragma unroll
    for (int k = 0; k < 4; ++k) {
        const int x = 2 * bx + (k & 1), y = 2 * by + (k >> 1);
        in[k] = x < d.w && y < d.h;
        o[k] = d.p + (long long)y * d.w + x;
        e[k] = in[k] ? ld_h4(o[k], 0) : C3{0.f, 0.f, 0.f};
    }
    C3 sum = {0.f, 0.f, 0.f};
#pragma unroll
    for (int dy = -1; dy <= 1; ++dy)
#pragma unroll
        for (int dx = -1; dx <= 1; ++dx) {
            const float wk = float((dx == 0 ? 2 : 1) * (dy == 0 ? 2 : 1)) * 0.0625f;
            const C3 c = ld_h4(s.p, (long long)min(max(by + dy, 0), s.h - 1) * s.w + min(max(bx + dx, 0), s.w - 1));
            sum = {add(sum.r, mul(wk, c.r)), add(sum.g, mul(wk, c.g)), add(sum.b, mul(wk, c.b))};
        }
#pragma unroll
    for (int k = 0; k < 4; ++k)
        if (in[k]) st_h4(o[k], 0, {add(e[k].r, sum.r), add(e[k].g, sum.g), add(e[k].b, sum.b)});
}

// Clamp to [0, 1].  (The shader's clamp keeps a NaN, which the sRGB curve then maps to 0; here it is 0 at once.)
__device__ __forceinline__ float sat(float v) { return __saturatef(v); }

// c^(1/2.4) for c in (0.0031308, 1] as exp2f(log2f(c) / 2.4): full-precision library calls (a few ulp),
// far cheaper than the general powf; the 8-bit output absorbs the difference almost everywhere.
__device__ __forceinline__ float srgb(float c)
{
    constexpr float kExp = 1.0f / 2.4f;
    c = c > 0.f ? c : 0.f;
    if (c <= 0.0031308f) return mul(c, 12.92f);
    return sub(mul(1.055f, exp2f(mul(log2f(c), kExp))), 0.055f);
}

__device__ __forceinline__ float fit(float v)
{
    const float a = sub(mul(v, add(v, 0.0245786f)), 0.000090537f);
    const float b = add(mul(v, add(mul(0.983729f, v), 0.4329510f)), 0.238081f);
    return dv(a, b);
}

__device__ __forceinline__ C3 mat3(const float (&m)[9], C3 v)
{
    return {add(add(mul(m[0], v.r), mul(m[1], v.g)), mul(m[2], v.b)), add(add(mul(m[3], v.r), mul(m[4], v.g)), mul(m[5], v.b)),
            add(add(mul(m[6], v.r), mul(m[7], v.g)), mul(m[8], v.b))};
}

__constant__ float kAcesIn[9] = {0.59719f, 0.35458f, 0.04823f, 0.07600f, 0.90834f, 0.01566f, 0.02840f, 0.13383f, 0.83777f};
__constant__ float kAcesOut[9] = {1.60475f, -0.53108f, -0.07367f, -0.10208f, 1.10813f, -0.00605f, -0.00327f, -0.07276f, 1.07602f};

enum OutFmt { OUT_BGRA8 = 0, OUT_RGBA8 = 1, OUT_RGBA32F = 2 };

// ACES, sRGB, grade and vignette of one lit pixel.
__device__ __forceinline__ C3 display(C3 c, float d2)
{
    c = mat3(kAcesIn, c);
    c = {fit(c.r), fit(c.g), fit(c.b)};
    c = mat3(kAcesOut, c);
    c = {srgb(sat(c.r)), srgb(sat(c.g)), srgb(sat(c.b))};
    const float l = lum(c);
    const C3 cool = {mul(l, 0.9f), mul(l, 0.95f), mul(l, 1.1f)};
    c = {add(c.r, mul(sub(cool.r, c.r), 0.15f)), add(c.g, mul(sub(cool.g, c.g), 0.15f)), add(c.b, mul(sub(cool.b, c.b), 0.15f))};
    const float vig = sat(sub(1.f, mul(d2, 1.5f)));
    return {mul(c.r, vig), mul(c.g, vig), mul(c.b, vig)};
}

// Two pixels (2t, 2t + 1) of a row per thread; they share a bloom texel.  vec:
// the images are aligned for 16-byte HDR loads (binary16) and for paired stores.
// rw, rh: the reciprocals of W and H.
template <bool HDR16, int OUT>
__global__ void __launch_bounds__(kPostTX* kPostTY)
    k_post(const char* hdr, long long hpitch, char* out, long long opitch, int W, int H, Mip bl, float strength, float rw,
           float rh, int vec)
{
    pdl_begin();
    const int x = 2 * (blockIdx.x * kPostTX + threadIdx.x), y = blockIdx.y * kPostTY + threadIdx.y;
    if (x >= W || y >= H) return;
    const bool two = x + 1 < W;
    C3 h[2];
    ld_hdr2<HDR16>(hdr, hpitch, x, two ? x + 1 : x, y, (vec & 1) && two, h);
    const C3 b = ld_h4(bl.p, (long long)min(y / 2, bl.h - 1) * bl.w + min(x / 2, bl.w - 1));
    const C3 sb = {mul(strength, b.r), mul(strength, b.g), mul(strength, b.b)};
    const float v = div_by(add(float(y), 0.5f), float(H), rh), oy = sub(v, 0.5f), oy2 = mul(oy, oy);
    C3 res[2];
#pragma unroll
    for (int k = 0; k < 2; ++k) {
        const float u = div_by(add(float(x + k), 0.5f), float(W), rw), ox = sub(u, 0.5f);
        const float d2 = add(mul(ox, ox), oy2);
        const int px = int(mul(mul(mul(ox, d2), 0.0015f), float(W))), py = int(mul(mul(mul(oy, d2), 0.0015f), float(H)));
        C3 c = {add(h[k].r, sb.r), add(h[k].g, sb.g), add(h[k].b, sb.b)};
        if (px != 0 || py != 0) {  // chromatic aberration of a pixel or more: only towards the corners
            auto sample = [&](int cx, int cy) {
                cx = min(max(cx, 0), W - 1);
                cy = min(max(cy, 0), H - 1);
                const C3 hs = ld_hdr<HDR16>(hdr, hpitch, cx, cy);
                const C3 bs = ld_h4(bl.p, (long long)min(cy / 2, bl.h - 1) * bl.w + min(cx / 2, bl.w - 1));
                return C3{add(hs.r, mul(strength, bs.r)), add(hs.g, mul(strength, bs.g)), add(hs.b, mul(strength, bs.b))};
            };
            c.r = sample(x + k + px, y + py).r;
            c.b = sample(x + k - px, y - py).b;
        }
        res[k] = display(c, d2);
    }
    char* row = out + y * opitch;
    if constexpr (OUT == OUT_RGBA32F) {
        float4* o = reinterpret_cast<float4*>(row) + x;
        o[0] = make_float4(res[0].r, res[0].g, res[0].b, 1.f);
        if (two) o[1] = make_float4(res[1].r, res[1].g, res[1].b, 1.f);
    } else {
        uint32_t px8[2];
#pragma unroll
        for (int k = 0; k < 2; ++k) {
            auto q = [](float f) { return __float2uint_rn(__fmul_rn(sat(f), 255.0f)); };
            const uint32_t r = q(res[k].r), g = q(res[k].g), bb = q(res[k].b);
            px8[k] = OUT == OUT_BGRA8 ? (bb | (g << 8) | (r << 16) | (255u << 24)) : (r | (g << 8) | (bb << 16) | (255u << 24));
        }
        uint32_t* o = reinterpret_cast<uint32_t*>(row) + x;
        if (two && (vec & 2)) {
            *reinterpret_cast<uint2*>(o) = make_uint2(px8[0], px8[1]);
        } else {
            o[0] = px8[0];
            if (two) o[1] = px8[1];
        }
    }
}

} // namespace
} // namespace tg

using namespace tg;

struct tg_post {
    int device = 0;
    uint32_t w = 0, h = 0;
    tg_post_params p{};
    char* buf = nullptr;
    size_t bytes = 0;
    int n = 0;
    Mip mip[kMaxMips];
};

namespace {

struct DeviceGuard {
    int prev = -1;
    explicit DeviceGuard(int dev)
    {
        cudaGetDevice(&prev);
        if (prev != dev) cudaSetDevice(dev);
    }
    ~DeviceGuard()
    {
        int cur = -1;
        cudaGetDevice(&cur);
        if (prev >= 0 && cur != prev) cudaSetDevice(prev);
    }
};

int alloc_chain(tg_post* s)
{
    const uint32_t bw = std::max(s->w / 2, 1u), bh = std::max(s->h / 2, 1u);
    const uint32_t levels = uint32_t(std::floor(std::log2(float(std::max(bw, bh))))) + 1;
    s->n = int(std::min(std::min(levels, s->p.max_mips), uint32_t(kMaxMips)));
    size_t off[kMaxMips], total = 0;
    for (int i = 0; i < s->n; ++i) {
        s->mip[i].w = int(std::max(bw >> i, 1u));
        s->mip[i].h = int(std::max(bh >> i, 1u));
        off[i] = total;
        total += (size_t(s->mip[i].w) * s->mip[i].h * 8 + 255) / 256 * 256;
    }
    if (cudaMalloc(&s->buf, total) != cudaSuccess) {
        cudaGetLastError();
        s->buf = nullptr;
        return fail(TG_ERR_OOM, "cudaMalloc of %zu bloom bytes failed", total);
    }
    s->bytes = total;
    for (int i = 0; i < s->n; ++i) s->mip[i].p = reinterpret_cast<uint2*>(s->buf + off[i]);
    return TG_OK;
}

int check_img(const char* what, const tg_image* im, uint32_t w, const int* fmts, int nf, long long& pitch)
{
    if (!im || !im->ptr) return fail(TG_ERR_INVALID, "%s: null image", what);
    bool ok = false;
    for (int k = 0; k < nf; ++k) ok |= im->format == fmts[k];
    if (!ok) return fail(TG_ERR_INVALID, "%s: unsupported format %d", what, im ? im->format : -1);
    const long long tb = fmt_bytes(im->format);
    pitch = im->pitch_bytes ? im->pitch_bytes : tb * w;
    if (pitch < tb * (long long)w || pitch % tb || reinterpret_cast<uintptr_t>(im->ptr) % tb)
        return fail(TG_ERR_INVALID, "%s: address and pitch must be multiples of %lld bytes and cover a row", what, tb);
    return TG_OK;
}

} // namespace

int tg_post_params_default(tg_post_params* p)
{
    if (!p) return fail(TG_ERR_INVALID, "null params");
    *p = tg_post_params{1.0f, 0.095f, 6u, 0u};
    return TG_OK;
}

int tg_post_create(uint32_t width, uint32_t height, const tg_post_params* params, int device, tg_post** out)
{
    if (!out) return fail(TG_ERR_INVALID, "null output handle");
    *out = nullptr;
    if (width == 0 || height == 0 || width > 32768 || height > 32768)
        return fail(TG_ERR_INVALID, "size %ux%u outside 1..32768", width, height);
    tg_post_params p;
    tg_post_params_default(&p);
    if (params) p = *params;
    if (p.max_mips < 1 || !std::isfinite(p.bloom_threshold) || !std::isfinite(p.bloom_strength))
        return fail(TG_ERR_INVALID, "max_mips must be >= 1 and threshold / strength finite");
    if (device < 0 && cudaGetDevice(&device) != cudaSuccess) return fail(TG_ERR_CUDA, "no current CUDA device");
    DeviceGuard g(device);
    tg_post* s = new (std::nothrow) tg_post();
    if (!s) return fail(TG_ERR_OOM, "host allocation failed");
    s->device = device;
    s->w = width;
    s->h = height;
    s->p = p;
    const int st = alloc_chain(s);
    if (st) {
        delete s;
        return st;
    }
    *out = s;
    return TG_OK;
}

int tg_post_process(tg_post* s, const tg_image* hdr, const tg_image* out, void* stream)
{
    if (!s) return fail(TG_ERR_INVALID, "null handle");
    static const int kHdr[] = {TG_FMT_RGBA16F, TG_FMT_RGBA32F};
    static const int kOut[] = {TG_FMT_BGRA8, TG_FMT_RGBA8, TG_FMT_RGBA32F};
    long long hp = 0, op = 0;
    int st;
    if ((st = check_img("hdr", hdr, s->w, kHdr, 2, hp))) return st;
    if ((st = check_img("out", out, s->w, kOut, 3, op))) return st;
    DeviceGuard g(s->device);
    cudaStream_t cs = static_cast<cudaStream_t>(stream);
    const dim3 blk(kPostTX, kPostTY);
    auto grid = [](int w, int h) { return dim3((w + kPostTX - 1) / kPostTX, (h + kPostTY - 1) / kPostTY); };
    const char* hb = static_cast<const char*>(hdr->ptr);
    const bool h16 = hdr->format == TG_FMT_RGBA16F;
    const int W = int(s->w), H = int(s->h);
    // bit 0: pairs of binary16 HDR texels start on 16 bytes; bit 1: pairs of 4-byte display texels on 8
    const int vec = (reinterpret_cast<uintptr_t>(hb) % 16 == 0 && hp % 16 == 0 && W > 1 ? 1 : 0) |
                    (reinterpret_cast<uintptr_t>(out->ptr) % 8 == 0 && op % 8 == 0 ? 2 : 0);
    // extraction + mips 1..5 in one launch; mips beyond the sixth (max_mips > 6) one launch each
    MipSet ms;
    ms.n = std::min(s->n, kPyrLevels);
    for (int i = 0; i < ms.n; ++i) ms.m[i] = s->mip[i];
    const dim3 pgrid((s->mip[0].w + kPyrT - 1) / kPyrT, (s->mip[0].h + kPyrT - 1) / kPyrT);
    cudaError_t e = launch_chain(h16 ? k_bloom_pyramid<true> : k_bloom_pyramid<false>, pgrid, dim3(256), cs, hb, hp, W, H, ms,
                                 s->p.bloom_threshold, vec & 1);
    for (int i = kPyrLevels; i < s->n && e == cudaSuccess; ++i)
        e = launch_chain(k_bloom_down, grid(s->mip[i].w, s->mip[i].h), blk, cs, s->mip[i - 1], s->mip[i]);
    for (int i = s->n - 2; i >= 0 && e == cudaSuccess; --i)
        e = launch_chain(k_bloom_up, grid((s->mip[i].w + 1) / 2, (s->mip[i].h + 1) / 2), blk, cs, s->mip[i + 1], s->mip[i]);
    if (e != cudaSuccess) {
        cudaGetLastError();  // (reported here, not by the thread's next call)
        return fail(TG_ERR_CUDA, "bloom launch failed: %s", cudaGetErrorString(e));
    }
    typedef void (*PostFn)(const char*, long long, char*, long long, int, int, Mip, float, float, float, int);
    static const PostFn fns[2][3] = {{k_post<false, OUT_BGRA8>, k_post<false, OUT_RGBA8>, k_post<false, OUT_RGBA32F>},
                                     {k_post<true, OUT_BGRA8>, k_post<true, OUT_RGBA8>, k_post<true, OUT_RGBA32F>}};
    const int of = out->format == TG_FMT_BGRA8 ? OUT_BGRA8 : out->format == TG_FMT_RGBA8 ? OUT_RGBA8 : OUT_RGBA32F;
    e = launch_chain(fns[h16][of], grid((W + 1) / 2, H), blk, cs, hb, hp, static_cast<char*>(out->ptr), op, W, H, s->mip[0],
                     s->p.bloom_strength, 1.0f / float(W), 1.0f / float(H), vec);
    if (e != cudaSuccess) {
        cudaGetLastError();
        return fail(TG_ERR_CUDA, "post-process launch failed: %s", cudaGetErrorString(e));
    }
    return TG_OK;
}

int tg_post_resize(tg_post* s, uint32_t width, uint32_t height)
{
    if (!s) return fail(TG_ERR_INVALID, "null handle");
    if (width == 0 || height == 0 || width > 32768 || height > 32768)
        return fail(TG_ERR_INVALID, "size %ux%u outside 1..32768", width, height);
    DeviceGuard g(s->device);
    if (cudaDeviceSynchronize() != cudaSuccess) return fail(TG_ERR_CUDA, "synchronize failed");
    cudaFree(s->buf);
    s->buf = nullptr;
    s->w = width;
    s->h = height;
    return alloc_chain(s);
}

int tg_post_get_info(const tg_post* s, tg_post_info* info)
{
    if (!s || !info) return fail(TG_ERR_INVALID, "null handle or info");
    *info = tg_post_info{};
    info->width = s->w;
    info->height = s->h;
    info->mip_count = uint32_t(s->n);
    info->bloom_bytes = s->bytes;
    for (int i = 0; i < s->n; ++i) {
        info->mip_width[i] = uint32_t(s->mip[i].w);
        info->mip_height[i] = uint32_t(s->mip[i].h);
        info->mip_ptr[i] = s->mip[i].p;
    }
    return TG_OK;
}

void tg_post_destroy(tg_post* s)
{
    if (!s) return;
    {
        DeviceGuard g(s->device);
        cudaFree(s->buf);
    }
    delete s;
}
