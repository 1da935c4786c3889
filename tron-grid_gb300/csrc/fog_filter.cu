// Volumetric-fog froxel filter (include/tg_fog.h) on sm_103a.
//
// The reference's filterMain (src/volumetric_filter.slang:142-226).  A CTA covers
// 32 x 4 columns of up to 8 consecutive slices, one thread per column: the
// column's camera ray and the slices' view depths are computed once (they are the
// same for every froxel of a column / slice), then for each slice the 34 x 6 halo
// of injected texels is staged in shared memory, double-buffered (the next
// slice's texels are loaded while this slice is computed, one barrier per slice),
// and each thread places its froxel centre on its ray, projects it into the
// previous frame and fetches the history trilinearly.
//
// What bounds it: FP32 issue (510 instructions per froxel, the unfused
// interpolation of eight texels the largest part).  The compulsory traffic of a
// 320x180x64 rgba16f pass (88 MB, L2-resident) is 13 us of the 6.8 TB/s a copy
// reaches.  Measured there, with history: 79.9 us with two barriers per slice and a
// division per quotient, 58.3 us as here (56 registers, 9 CTAs per SM; 48
// registers and 16 slices per CTA 64, 64 registers 58.9); two columns per thread
// (6 shared loads per froxel instead of 9, half the CTAs) 61.8.
//
// Every add, multiply, divide and square root on the projection path is rounded
// as IEEE asks (no contraction into FMA), in the order the reference writes them,
// so the froxel coordinates that decide the rejection tests and the trilinear
// weights are the reference's own float arithmetic; only powf / logf (slice
// depth, its inverse) are CUDA's.  Divisors are the same for a whole box, column,
// froxel or launch, so quotients are formed by multiplying with the divisor's
// correctly rounded reciprocal and correcting with FMA residuals, which rounds
// correctly (Markstein 1990; Brisebarre, Muller and Raina 2004) while nothing
// overflows or underflows; operands outside that range take the division itself.
#include <cuda_fp16.h>
#include <cuda_runtime.h>

#include <cstdint>

#include "svgf_device.cuh"
#include "svgf_internal.h"
#include "tg_fog.h"

namespace tg {
namespace {

constexpr int kFogTX = 32, kFogTY = 4;  // columns of a CTA (256 threads: 74 us against 60)
constexpr int kFogSW = kFogTX + 2, kFogSH = kFogTY + 2;
constexpr int kFogZC = 8;  // most slices per CTA (FogArgs::zc)

struct FogArgs {
    float ivp[16], pvp[16], cam[3];
    float alpha, znear, zfar;
    int W, H, D, valid;
    int zc;         // slices per CTA
    int plain_div;  // the depth range is too extreme for quotients by reciprocal
    const char* raw;
    const char* hist;
    char* out;
    long long raw_row, raw_slice, hist_row, hist_slice, out_row, out_slice;
};

// A texel as stored: 4 x binary16 or 4 x float.
template <bool F16> struct Texel;
template <> struct Texel<true> {
    typedef uint2 raw;
    static constexpr int kBytes = 8;
    __device__ __forceinline__ static raw zero() { return make_uint2(0u, 0u); }
    __device__ __forceinline__ static float4 value(raw u)
    {
        const float2 a = __half22float2(*reinterpret_cast<const __half2*>(&u.x));
        const float2 b = __half22float2(*reinterpret_cast<const __half2*>(&u.y));
        return make_float4(a.x, a.y, b.x, b.y);
    }
};
template <> struct Texel<false> {
    typedef float4 raw;
    static constexpr int kBytes = 16;
    __device__ __forceinline__ static raw zero() { return make_float4(0.f, 0.f, 0.f, 0.f); }
    __device__ __forceinline__ static float4 value(raw v) { return v; }
};

template <bool F16, class Off> __device__ __forceinline__ typename Texel<F16>::raw ld_raw(const char* base, Off off)
{
    return __ldg(reinterpret_cast<const typename Texel<F16>::raw*>(base + off));
}

template <bool F16> __device__ __forceinline__ void st_texel(char* base, long long off, float4 v)
{
    if constexpr (F16) {
        const __half2 a = __floats2half2_rn(v.x, v.y), b = __floats2half2_rn(v.z, v.w);
        uint2 u;
        u.x = *reinterpret_cast<const uint32_t*>(&a);
        u.y = *reinterpret_cast<const uint32_t*>(&b);
        *reinterpret_cast<uint2*>(base + off) = u;
    } else {
        *reinterpret_cast<float4*>(base + off) = v;
    }
}

__device__ __forceinline__ float add(float a, float b) { return __fadd_rn(a, b); }
__device__ __forceinline__ float sub(float a, float b) { return __fsub_rn(a, b); }
__device__ __forceinline__ float mul(float a, float b) { return __fmul_rn(a, b); }
__device__ __forceinline__ float dv(float a, float b) { return __fdiv_rn(a, b); }

// clip = M (x, y, z, w), M column-major, the four column terms summed left to right
__device__ __forceinline__ void mat_vec(const float* m, float x, float y, float z, float w, float o[4])
{
#pragma unroll
    for (int r = 0; r < 4; ++r) o[r] = add(add(add(mul(m[r], x), mul(m[4 + r], y)), mul(m[8 + r], z)), mul(m[12 + r], w));
}

// x / y by the correctly rounded reciprocal r of y, |x| < 2^100.  One residual
// step is exact for the box counts (every binary32 significand over 3, 6 and 9 was
// checked; 1, 2 and 4 are exact), for subnormal quotients too but over 6, where a
// quotient can lie half-way between two subnormals and the step does not keep the
// tie: every x below 2^-99 was checked, the last wrong one lies below 2^-125.
// Two steps are exact for any divisor while x / y is far from the subnormals, or
// x = 0.
__device__ __forceinline__ float div_count(float x, float y, float r)
{
    const float q = mul(x, r);
    return __fmaf_rn(__fmaf_rn(-q, y, x), r, q);
}
__device__ __forceinline__ float div_by(float x, float y, float r)
{
    const float q = div_count(x, y, r);
    return __fmaf_rn(__fmaf_rn(-q, y, x), r, q);
}
constexpr float kDivMax = 1.2676506e30f;  // 2^100

__device__ __forceinline__ float lerp1(float a, float b, float t) { return add(a, mul(sub(b, a), t)); }

__device__ __forceinline__ float4 lerp4(float4 a, float4 b, float t)
{
    return make_float4(lerp1(a.x, b.x, t), lerp1(a.y, b.y, t), lerp1(a.z, b.z, t), lerp1(a.w, b.w, t));
}

// Off: byte offsets within a volume (32 bits unless one is 4 GB or more).
template <bool RAW16, bool OUT16, class Off>
__global__ void __launch_bounds__(kFogTX* kFogTY, 9) k_fog_filter(const FogArgs a)
{
    typedef Texel<RAW16> TR;
    typedef Texel<OUT16> TO;
    constexpr int kThreads = kFogTX * kFogTY;
    constexpr int kCells = (kFogSH * kFogSW + kThreads - 1) / kThreads;
    __shared__ float4 tile[2][kFogSH * kFogSW];
    __shared__ float view_z[kFogZC];
    pdl_begin();
    const int x0 = blockIdx.x * kFogTX, y0 = blockIdx.y * kFogTY, z0 = blockIdx.z * a.zc;
    const int tid = threadIdx.y * kFogTX + threadIdx.x;
    const int x = x0 + threadIdx.x, y = y0 + threadIdx.y;
    const bool inside = x < a.W && y < a.H;
    const int nz = min(a.zc, a.D - z0);
    const float ratio = dv(a.zfar, a.znear);

    // This thread's cells of a slice's halo tile (the same in every slice), and the first slice's texels.  Cells
    // outside the grid are staged as +0 and summed without a test: the running sum starts at +0 and so is never -0,
    // which makes adding +0 an exact no-op, the same sums as the reference's skipped taps.
    Off cell[kCells];
    bool cin[kCells];
    typename TR::raw next[kCells];
    const char* rs = a.raw + z0 * a.raw_slice;
#pragma unroll
    for (int e = 0; e < kCells; ++e) {
        const int k = tid + e * kThreads;
        const int qy = y0 - 1 + k / kFogSW, qx = x0 - 1 + k % kFogSW;
        cin[e] = k < kFogSH * kFogSW && qx >= 0 && qy >= 0 && qx < a.W && qy < a.H;
        cell[e] = cin[e] ? Off(qy) * Off(a.raw_row) + Off(qx * TR::kBytes) : Off(0);
        next[e] = cin[e] ? ld_raw<RAW16>(rs, cell[e]) : TR::zero();
    }

    // Per slice of the chunk: its view depth (:74-78).
    if (tid < nz) {
        const float tz = dv(add(float(z0 + tid), 0.5f), float(a.D));
        view_z[tid] = mul(a.znear, powf(ratio, tz));
    }
    // Per column: the normalised camera ray through the column's NDC and its cosine to the camera axis (:83-106).
    float ray[3] = {0.f, 0.f, 0.f}, rdf = 1.f, rrdf = 1.f, lnr = 1.f;
    if (a.valid && inside) {
        const float u = dv(add(float(x), 0.5f), float(a.W)), v = dv(add(float(y), 0.5f), float(a.H));
        const float nx = sub(mul(u, 2.f), 1.f), ny = sub(1.f, mul(v, 2.f));
        float nh[4], fh[4], fwd[3];
        mat_vec(a.ivp, nx, ny, 0.f, 1.f, nh);
        mat_vec(a.ivp, 0.f, 0.f, 0.f, 1.f, fh);
#pragma unroll
        for (int k = 0; k < 3; ++k) {
            ray[k] = sub(dv(nh[k], nh[3]), a.cam[k]);
            fwd[k] = sub(dv(fh[k], fh[3]), a.cam[k]);
        }
        const float rl = __fsqrt_rn(add(add(mul(ray[0], ray[0]), mul(ray[1], ray[1])), mul(ray[2], ray[2])));
        const float fl = __fsqrt_rn(add(add(mul(fwd[0], fwd[0]), mul(fwd[1], fwd[1])), mul(fwd[2], fwd[2])));
#pragma unroll
        for (int k = 0; k < 3; ++k) {
            ray[k] = dv(ray[k], rl);
            fwd[k] = dv(fwd[k], fl);
        }
        rdf = add(add(mul(ray[0], fwd[0]), mul(ray[1], fwd[1])), mul(ray[2], fwd[2]));
        rdf = rdf > 1e-4f ? rdf : 1e-4f;
        rrdf = __frcp_rn(rdf);
        lnr = logf(ratio);
    }
    const float rnear = __frcp_rn(a.znear), rlnr = __frcp_rn(lnr);
    // In-grid members of the column's 3x3 box.
    float n = 0.f;
#pragma unroll
    for (int dy = -1; dy <= 1; ++dy)
#pragma unroll
        for (int dx = -1; dx <= 1; ++dx)
            if (x + dx >= 0 && x + dx <= a.W - 1 && y + dy >= 0 && y + dy <= a.H - 1) n = add(n, 1.f);
    const float cnt = fmaxf(n, 1.f), rcnt = __frcp_rn(cnt);
    // Sums over six below which the division is taken (zeros too).  Binary16 texels cannot sum to less than 2^-24.  A warp
    // without such a column, at the grid's edge, skips the test: 59.8 us with float volumes at 320x180x64 against 59.4
    // with no test and 60.1 with one in every warp.
    const float least = cnt == 6.f ? 4.7019774e-38f : 0.f;  // 2^-124
    const bool sixes = __any_sync(0xffffffffu, cnt == 6.f);

    for (int zi = 0; zi < nz; ++zi) {
        const int z = z0 + zi;
        float4* t = tile[zi & 1];
#pragma unroll
        for (int e = 0; e < kCells; ++e)
            if (tid + e * kThreads < kFogSH * kFogSW) t[tid + e * kThreads] = TR::value(next[e]);
        // One barrier per slice: a thread reaches the next slice's stores into this half of the tile only after the
        // next barrier, which every thread passes after it has read this slice.
        __syncthreads();
        if (zi + 1 < nz) {
            rs += a.raw_slice;
#pragma unroll
            for (int e = 0; e < kCells; ++e) next[e] = cin[e] ? ld_raw<RAW16>(rs, cell[e]) : TR::zero();
        }
        if (!inside) continue;

        // 1. 3x3 mean over the in-grid neighbours of the slice (:152-166), summed in the reference's order
        float4 s = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
        for (int dy = 0; dy < 3; ++dy)
#pragma unroll
            for (int dx = 0; dx < 3; ++dx) {
                const float4 q = t[(threadIdx.y + dy) * kFogSW + threadIdx.x + dx];
                s = make_float4(add(s.x, q.x), add(s.y, q.y), add(s.z, q.z), add(s.w, q.w));
            }
        float4 res;
        bool plain = !(fmaxf(fmaxf(fabsf(s.x), fabsf(s.y)), fmaxf(fabsf(s.z), fabsf(s.w))) < kDivMax);
        if (!RAW16 && sixes) plain |= !(fminf(fminf(fabsf(s.x), fabsf(s.y)), fminf(fabsf(s.z), fabsf(s.w))) >= least);
        if (!plain)
            res = make_float4(div_count(s.x, cnt, rcnt), div_count(s.y, cnt, rcnt), div_count(s.z, cnt, rcnt),
                              div_count(s.w, cnt, rcnt));
        else
            res = make_float4(dv(s.x, cnt), dv(s.y, cnt), dv(s.z, cnt), dv(s.w, cnt));
        if (a.valid) {
            // 2. froxel centre on the column's ray at the slice's view depth (:100-106)
            const float tt = a.plain_div ? dv(view_z[zi], rdf) : div_by(view_z[zi], rdf, rrdf);
            const float wx = add(a.cam[0], mul(ray[0], tt)), wy = add(a.cam[1], mul(ray[1], tt)),
                        wz = add(a.cam[2], mul(ray[2], tt));

            // 3. previous-frame froxel coordinates and rejections (:177-213)
            float pc[4];
            mat_vec(a.pvp, wx, wy, wz, 1.f, pc);
            const float pz = pc[3];
            float ndx, ndy, lt;
            if (!a.plain_div && fmaxf(fmaxf(fabsf(pc[0]), fabsf(pc[1])), fabsf(pz)) < kDivMax) {
                const float rw = __frcp_rn(pz);
                ndx = div_by(pc[0], pz, rw);
                ndy = div_by(pc[1], pz, rw);
                lt = div_by(logf(div_by(pz, a.znear, rnear)), lnr, rlnr);
            } else {
                ndx = dv(pc[0], pz);
                ndy = dv(pc[1], pz);
                lt = dv(logf(dv(pz, a.znear)), lnr);
            }
            const float fx = mul(add(mul(ndx, 0.5f), 0.5f), float(a.W));
            const float fy = mul(add(mul(-ndy, 0.5f), 0.5f), float(a.H));
            const float fz = sub(mul(lt, float(a.D)), 0.5f);
            const bool rej = pz <= 1e-4f || pz < a.znear || pz > a.zfar || fx < 0.f || fx >= float(a.W) || fy < 0.f ||
                             fy >= float(a.H) || fz < 0.f || fz >= float(a.D);
            if (!rej) {
                // 4. trilinear history, clamp-to-edge (:111-140), then the EMA (:216-225)
                const int ix = int(floorf(fx)), iy = int(floorf(fy)), iz = int(floorf(fz));
                const float ax = sub(fx, float(ix)), ay = sub(fy, float(iy)), az = sub(fz, float(iz));
                const int xa = min(max(ix, 0), a.W - 1), xb = min(max(ix + 1, 0), a.W - 1);
                const int ya = min(max(iy, 0), a.H - 1), yb = min(max(iy + 1, 0), a.H - 1);
                const int za = min(max(iz, 0), a.D - 1), zb = min(max(iz + 1, 0), a.D - 1);
                const Off oxa = Off(xa * TO::kBytes), oxb = Off(xb * TO::kBytes);
                const Off at = Off(za) * Off(a.hist_slice) + Off(ya) * Off(a.hist_row);
                const Off dy = Off(yb - ya) * Off(a.hist_row), dz = Off(zb - za) * Off(a.hist_slice);
                typename TO::raw h[8];
#pragma unroll
                for (int k = 0; k < 8; ++k)
                    h[k] = ld_raw<OUT16>(a.hist, at + (k & 4 ? dz : Off(0)) + (k & 2 ? dy : Off(0)) + (k & 1 ? oxb : oxa));
                const float4 c0 = lerp4(lerp4(TO::value(h[0]), TO::value(h[1]), ax), lerp4(TO::value(h[2]), TO::value(h[3]), ax), ay);
                const float4 c1 = lerp4(lerp4(TO::value(h[4]), TO::value(h[5]), ax), lerp4(TO::value(h[6]), TO::value(h[7]), ax), ay);
                res = lerp4(lerp4(c0, c1, az), res, a.alpha);
            }
        }
        st_texel<OUT16>(a.out, z * a.out_slice + y * a.out_row + x * (long long)TO::kBytes, res);
    }
}

struct VolGeom {
    long long row, slice, bytes;
    int texel;
};

int check_volume(const char* what, const tg_volume* v, int W, int H, int D, VolGeom& g)
{
    if (!v || !v->ptr) return fail(TG_ERR_INVALID, "%s: null volume", what);
    if (v->format != TG_FMT_RGBA16F && v->format != TG_FMT_RGBA32F)
        return fail(TG_ERR_INVALID, "%s: format %d is not RGBA16F or RGBA32F", what, v->format);
    g.texel = v->format == TG_FMT_RGBA16F ? 8 : 16;
    g.row = v->row_pitch_bytes ? v->row_pitch_bytes : (long long)W * g.texel;
    g.slice = v->slice_pitch_bytes ? v->slice_pitch_bytes : (long long)H * g.row;
    if (g.row < (long long)W * g.texel || g.row % g.texel) return fail(TG_ERR_INVALID, "%s: bad row pitch %lld", what, g.row);
    if (g.slice < (long long)H * g.row || g.slice % g.texel)
        return fail(TG_ERR_INVALID, "%s: bad slice pitch %lld", what, g.slice);
    if (reinterpret_cast<uintptr_t>(v->ptr) % g.texel)
        return fail(TG_ERR_INVALID, "%s: address must be a multiple of %d bytes", what, g.texel);
    g.bytes = (long long)(D - 1) * g.slice + (long long)(H - 1) * g.row + (long long)W * g.texel;
    return TG_OK;
}

bool overlap(const void* a, long long na, const void* b, long long nb)
{
    const uintptr_t pa = reinterpret_cast<uintptr_t>(a), pb = reinterpret_cast<uintptr_t>(b);
    return pa < pb + uintptr_t(nb) && pb < pa + uintptr_t(na);
}

} // namespace
} // namespace tg

using namespace tg;

int tg_fog_filter(const tg_fog_filter_params* p, const tg_volume* raw, const tg_volume* hist, const tg_volume* out,
                  void* stream)
{
    if (!p) return fail(TG_ERR_INVALID, "null parameters");
    const uint32_t W = p->froxel_width, H = p->froxel_height, D = p->froxel_depth;
    if (W == 0 || H == 0 || D == 0 || W > 65535u * kFogTX || H > 65535u * kFogTY || D > 65535u)
        return fail(TG_ERR_INVALID, "froxel grid %ux%ux%u outside 1..(2097120, 262140, 65535)", W, H, D);
    if (!(p->near_plane > 0.f) || !(p->far_plane > p->near_plane))
        return fail(TG_ERR_INVALID, "depth range needs 0 < near_plane < far_plane");
    VolGeom gr, gh, go;
    int st;
    if ((st = check_volume("inject_raw", raw, W, H, D, gr))) return st;
    if ((st = check_volume("history", hist, W, H, D, gh))) return st;
    if ((st = check_volume("output", out, W, H, D, go))) return st;
    if (hist->format != out->format) return fail(TG_ERR_INVALID, "history and output formats differ");
    if (overlap(out->ptr, go.bytes, raw->ptr, gr.bytes) || overlap(out->ptr, go.bytes, hist->ptr, gh.bytes))
        return fail(TG_ERR_INVALID, "output overlaps inject_raw or history");
    FogArgs a;
    for (int k = 0; k < 16; ++k) {
        a.ivp[k] = p->inv_view_projection[k];
        a.pvp[k] = p->prev_view_projection[k];
    }
    for (int k = 0; k < 3; ++k) a.cam[k] = p->camera_pos[k];
    a.alpha = p->alpha;
    a.znear = p->near_plane;
    a.zfar = p->far_plane;
    a.W = int(W);
    a.H = int(H);
    a.D = int(D);
    a.valid = p->history_valid != 0;
    // quotients by reciprocal stay far from overflow and the subnormals while the depth range is within these bounds
    a.plain_div = !(p->near_plane >= 1e-15f && p->far_plane <= 1e15f && p->far_plane / p->near_plane >= 1.0001f);
    a.raw = static_cast<const char*>(raw->ptr);
    a.hist = static_cast<const char*>(hist->ptr);
    a.out = static_cast<char*>(out->ptr);
    a.raw_row = gr.row;
    a.raw_slice = gr.slice;
    a.hist_row = gh.row;
    a.hist_slice = gh.slice;
    a.out_row = go.row;
    a.out_slice = go.slice;
    // Slices per CTA: up to 8 share the column's set-up; a small grid takes fewer until it has 6 CTAs per SM, since its
    // pass is then one CTA's chain of slices.
    int dev = 0, sms = 1;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    const uint32_t tiles = ((W + kFogTX - 1) / kFogTX) * ((H + kFogTY - 1) / kFogTY);
    a.zc = kFogZC;
    while (a.zc > 1 && uint64_t(tiles) * ((D + a.zc - 1) / a.zc) < 6ull * sms) a.zc /= 2;
    const dim3 grid((W + kFogTX - 1) / kFogTX, (H + kFogTY - 1) / kFogTY, (D + a.zc - 1) / a.zc),
        block(kFogTX, kFogTY);
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    const bool r16 = raw->format == TG_FMT_RGBA16F, o16 = out->format == TG_FMT_RGBA16F;
    const bool wide = gr.bytes > 0xffffffffLL || gh.bytes > 0xffffffffLL;
    typedef void (*Fn)(const FogArgs);
    static const Fn fns[2][4] = {
        {k_fog_filter<false, false, uint32_t>, k_fog_filter<false, true, uint32_t>, k_fog_filter<true, false, uint32_t>,
         k_fog_filter<true, true, uint32_t>},
        {k_fog_filter<false, false, uint64_t>, k_fog_filter<false, true, uint64_t>, k_fog_filter<true, false, uint64_t>,
         k_fog_filter<true, true, uint64_t>}};
    const cudaError_t e = launch_chain(fns[wide][2 * r16 + o16], grid, block, s, a);
    if (e != cudaSuccess) {
        cudaGetLastError();  // (reported here, not by the thread's next call)
        return fail(TG_ERR_CUDA, "fog filter launch failed: %s", cudaGetErrorString(e));
    }
    return TG_OK;
}
