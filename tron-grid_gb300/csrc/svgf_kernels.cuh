// SVGF kernels for sm_103a: the reference-exact chain and the FULL chain.
//
// One thread per pixel over 2-D blocks of 32 x 4: a warp covers 32 adjacent
// pixels of one row, so every image access of a warp is one contiguous,
// coalesced segment (16 B/px float4 or 8 B/px half4 per lane).  The a-trous
// taps re-read neighbours through the read-only (L1) path.
#pragma once

#include "svgf_device.cuh"

namespace tg {

constexpr int kBlockX = 32;
constexpr int kBlockY = 4;

// Residue-major layout of the a-trous scratch for stride s = 2^lg: pixel
// (x, y) lives in plane (y mod s) * s + (x mod s) at position (x / s, y / s),
// each plane pw x ph.  For s = 1 this is the ordinary row-major image.  Level
// L reads its input in the layout of its own stride and writes its output in
// the layout of the next level's stride, so every tile a level stages and
// every 3x3 neighbourhood it reads is a contiguous run of memory.
struct ResLayout {
    int lg, pw, ph;
};

__device__ __forceinline__ size_t res_idx(const ResLayout& L, int x, int y)
{
    // (fewer than 2^31 cells: images are at most 32768 x 32768)
    const unsigned m = (1u << L.lg) - 1u;
    return ((((unsigned(y) & m) << L.lg) + (unsigned(x) & m)) * unsigned(L.ph) + (unsigned(y) >> L.lg)) * unsigned(L.pw) +
           (unsigned(x) >> L.lg);
}

__host__ __device__ inline ResLayout res_layout(int w, int h, int lg)
{
    ResLayout L;
    L.lg = lg;
    L.pw = (w + (1 << lg) - 1) >> lg;
    L.ph = (h + (1 << lg) - 1) >> lg;
    return L;
}

// ------------------------------------------------------------- REF-EXACT ----
// src/svgf_denoise.slang:152-275: the arguments of the REF_EXACT kernels
// (svgf_level.cuh; the init pass runs inside the first wavelet pass).

struct RefArgs {
    int w, h;
    Img raw;  // lighting_raw (b0)
    Img out;  // denoised_indirect (b3)
    const void* mom_prev; // moments_prev (b4)
    void* mom_curr;       // moments_curr (b5)
    const void* src;      // wavelet source (b1 or b2)
    void* dst;            // wavelet destination (b2 or b1)
    ResLayout lin, lout;  // scratch layouts of src and dst
    float phi;            // SIGMA_COLOR_BASE
    float alpha_m;        // ALPHA_MOMENTS
    float var_eps;        // VARIANCE_EPSILON
    int stride;
    int final_pass;
    int* err;             // device error word of bounded waits (may be null)
};

// ------------------------------------------------------------------ FULL ----

struct FullArgs {
    int w, h;
    Img radiance, depth, normal, motion, out;
    const void* guide_prev;
    const void* hist_prev;
    const void* mom_prev;
    void* guide_cur;
    void* hist_cur;
    void* mom_cur;
    void* tc;
    const void* col_src;
    void* col_dst;
    size_t var_off;         // byte offset of the variance plane in col_src / col_dst
    size_t ghalf;           // FP32 records: index of the guide half-plane (16-byte units)
    float2* grad;           // per-pixel depth gradient (written by the temporal kernel), at grad_col
    // Blocks of 32x4 pixels with a pixel that needs the spatial variance fallback: with a counter, fb_flags lists
    // their numbers (in any order) and *fb_count is how many; without one (variance_list, streams of a batch),
    // fb_flags[block] is 1.
    int* fb_flags;
    int* fb_count;
    int* err;               // device error word (bounded waits that gave up); may be null
    ResLayout lin, lout;    // scratch layouts of col_src and col_dst
    float alpha, alpha_m, sigma_l, sigma_n, sigma_z;
    int sq_n; // squarings for sigma_n = 2^sq_n, -1 otherwise
    int max_history, fallback_frames;
    int level, stride, last;
};

// Where the depth gradient of column x lies in its row: the four residues of x
// mod 4 one after the other.  A warp of a level reads every s-th column, which
// touches 2, 4, 8, 16, 32 cache lines of row-major gradients at strides 1 to 16,
// and 4, 2, 2, 4, 8 of these.
__device__ __forceinline__ int grad_col(int w, int x)
{
    const int r = x & 3;
    return r * (w >> 2) + min(r, w & 3) + (x >> 2);
}

// K1: guide write, reprojection (bilinear 2x2 with depth/normal test), history
// length, colour EMA and mean-centred moment EMA.  A pixel whose history is at
// least `fallback_frames` long also gets its level-0 variance-plane entry (the
// temporal variance as stored) here; the function returns true for the
// others, whose variance needs the neighbours' moments (K2).  Level 0 stages
// its input from tc, guide_cur and that plane, so no level-0 record is written.
template <int ST> __device__ __forceinline__ bool full_temporal_px(const FullArgs& a, int x, int y)
{
    typedef Stor<ST> S;
    typedef typename S::guide_t G;
    typedef typename S::c4_t C4;
    typedef typename S::mom_t M;
    const size_t i = size_t(y) * a.w + x;
    // The reprojection taps land next to (x, y) under small motion: start their lines towards L2 now, so the
    // gathers that depend on the motion load find them there instead of paying a second DRAM round trip.
    prefetch_l2(static_cast<const C4*>(a.hist_prev) + i);
    prefetch_l2(static_cast<const G*>(a.guide_prev) + i);
    prefetch_l2(static_cast<const M*>(a.mom_prev) + i);

    // Every load of this pixel is issued before its first store (the motion first: the reprojection gathers
    // depend on it), and the gathers before the guide and gradient work, which runs while they are in flight.
    const float2 mv = ld_motion(a.motion, x, y);
    const float4 c4 = ld_rgba(a.radiance, x, y);
    uint32_t enc = 0;
    const float3 n = ld_normal(a.normal, x, y, ST == ST_FP16, enc);
    const float z = ld_depth(a.depth, x, y);
    const bool hl = x > 0, hr = x < a.w - 1, hu = y > 0, hd = y < a.h - 1;
    const float zl = hl ? ld_depth(a.depth, x - 1, y) : 0.0f, zr = hr ? ld_depth(a.depth, x + 1, y) : 0.0f;
    const float zu = hu ? ld_depth(a.depth, x, y - 1) : 0.0f, zd = hd ? ld_depth(a.depth, x, y + 1) : 0.0f;

    const float px = __fadd_rn(float(x), mv.x);
    const float py = __fadd_rn(float(y), mv.y);
    const float fx0 = floorf(px), fy0 = floorf(py);
    const float fx = __fsub_rn(px, fx0), fy = __fsub_rn(py, fy0);
    const float lim = 1073741824.0f;
    const int x0 = int(fmaxf(-lim, fminf(lim, fx0)));
    const int y0 = int(fmaxf(-lim, fminf(lim, fy0)));
    const float ofx = __fsub_rn(1.0f, fx), ofy = __fsub_rn(1.0f, fy);
    const float bw[4] = {__fmul_rn(ofx, ofy), __fmul_rn(fx, ofy), __fmul_rn(ofx, fy), __fmul_rn(fx, fy)};

    const G* gp = static_cast<const G*>(a.guide_prev);
    const C4* hp = static_cast<const C4*>(a.hist_prev);
    const M* mp = static_cast<const M*>(a.mom_prev);
    // All four taps' history, guide and moments are loaded before any of them
    // is tested, so the gathers overlap instead of forming a dependent chain.
    size_t tj[4];
    bool tin[4];
#pragma unroll
    for (int k = 0; k < 4; ++k) {
        const int tx = x0 + (k & 1), ty = y0 + (k >> 1);
        tin[k] = tx >= 0 && ty >= 0 && tx < a.w && ty < a.h;
        tj[k] = tin[k] ? size_t(ty) * a.w + tx : 0;
    }
    float4 thv[4];
    typename S::graw_t tg[4];
    float2 tm[4];
#pragma unroll
    for (int k = 0; k < 4; ++k) {
        if (tin[k]) {
            thv[k] = S::ld4(hp, tj[k]);
            tg[k] = S::ld_graw(gp, tj[k]);
            tm[k] = S::ldm(mp, tj[k]);
        } else {
            thv[k] = make_float4(0.f, 0.f, 0.f, 0.f);
            tg[k] = typename S::graw_t{};
            tm[k] = make_float2(0.f, 0.f);
        }
    }

    const G gv = S::mk_guide(n, enc, z);
    static_cast<G*>(a.guide_cur)[i] = gv;
    const float gx = grad1(z, zl, zr, hl, hr);
    const float gy = grad1(z, zu, zd, hu, hd);
    a.grad[size_t(y) * a.w + grad_col(a.w, x)] = make_float2(gx, gy);
    const float cr = S::qin(c4.x), cg = S::qin(c4.y), cb = S::qin(c4.z);
    const float gsum = __fadd_rn(fabsf(gx), fabsf(gy));
    bool other = false;
#pragma unroll
    for (int k = 0; k < 4; ++k) other |= tin[k] && !S::same_normal(tg[k], gv);
    const float3 nt = S::test_normal(gv, other);
    const float ztol = __fadd_rn(__fadd_rn(__fmul_rn(kDepthRel, z), __fmul_rn(kDepthGrad, gsum)), kDepthAbs);
    float sw = 0.0f, hr_ = 0.0f, hg = 0.0f, hb = 0.0f, hmu = 0.0f;
    float tw[4];
    int lmax = 0;
#pragma unroll
    for (int k = 0; k < 4; ++k) {
        tw[k] = 0.0f;
        if (!tin[k] || !(thv[k].w > 0.0f)) continue;
        if (!(fabsf(__fsub_rn(S::graw_z(tg[k]), z)) <= ztol)) continue;
        if (!S::normal_close_to(tg[k], gv, nt)) continue;
        tw[k] = bw[k];
        sw = __fadd_rn(sw, bw[k]);
        hr_ += bw[k] * thv[k].x;
        hg += bw[k] * thv[k].y;
        hb += bw[k] * thv[k].z;
        hmu += bw[k] * tm[k].x;
        lmax = max(lmax, int(thv[k].w));
    }
    const float l = lum(cr, cg, cb);
    float orr, og, ob, mu, var;
    int len;
    if (sw > 0.0f) {
        const float inv = 1.0f / sw;
        hr_ *= inv;
        hg *= inv;
        hb *= inv;
        hmu *= inv;
        float hvv = 0.0f;
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            if (!(tw[k] > 0.0f)) continue;  // rejected taps never enter the sums
            const float dm = tm[k].x - hmu;
            hvv += tw[k] * (tm[k].y + dm * dm);
        }
        hvv *= inv;
        len = min(lmax + 1, a.max_history);
        const float ac = fmaxf(a.alpha, 1.0f / float(len));
        const float am = fmaxf(a.alpha_m, 1.0f / float(len));
        orr = hr_ + ac * (cr - hr_);
        og = hg + ac * (cg - hg);
        ob = hb + ac * (cb - hb);
        const float dl = l - hmu;
        mu = hmu + am * dl;
        var = (1.0f - am) * (hvv + am * dl * dl);
    } else {
        len = 1;
        orr = cr;
        og = cg;
        ob = cb;
        mu = l;
        var = 0.0f;
    }
    const float4 tcv = make_float4(orr, og, ob, float(len));
    const float2 mom = make_float2(mu, var);
    S::st4(static_cast<C4*>(a.tc), i, tcv);
    S::stm(static_cast<M*>(a.mom_cur), i, mom);
    const float4 t = S::rt4(tcv);
    if (int(t.w) < a.fallback_frames) return true;
    Rec::st_var(a.col_dst, a.var_off, i, S::rtm(mom).y);
    return false;
}

// K2: for histories shorter than `fallback_frames`, the variance is a 7x7
// depth/normal-weighted spatial estimate from the neighbours' moments; writes
// the level-0 variance-plane entry of such a pixel.  The other pixels' entries
// come from K1.
//
// A CTA stages the guides (decoded) and moments of its pixel block plus a
// 3-pixel halo in shared memory.  Cells outside the image hold a zero normal,
// whose weight max(0, n.n')^sigma_n = 2^(sigma_n lg2 0) is exactly 0, so the
// sums equal those over the inside neighbours only.
constexpr int kVarHalo = 3;
constexpr int kVarTW = kBlockX + 2 * kVarHalo;
constexpr int kVarTH = kBlockY + 2 * kVarHalo;
struct VarTile {
    float4 g[kVarTH * kVarTW];  // unit normal, depth
    float2 m[kVarTH * kVarTW];  // luminance mean, variance
};

// One thread estimates R vertically adjacent pixels (x, y) .. (x, y + R - 1), so a
// staged cell is read once for up to R of them.  With every block of a 1920x1080
// frame listed (89 us under ncu) issue is 67% busy and the L1/shared pipe 59%: the
// 1039 instructions per pixel bound it, at 80 registers and 24 warps per SM, too few
// to fill either.  `cell` is the first pixel's cell, need[k] whether pixel k takes
// the estimate, gr[k] its depth gradient.
template <int ST, int R>
__device__ __forceinline__ void full_variance_px(const FullArgs& a, int x, int y, int cell, const VarTile& vt,
                                                 const bool (&need)[R], const float2 (&gr)[R])
{
    // w = max(0, n.n')^sigma_n exp(-|dz| / (sigma_z |grad z . off| + eps_z)), as one ex2;
    // offsets (dx, dy) and (-dx, -dy) share the depth scale kz
    const float ez = kEpsZ * (1.0f / kLog2eF);
    float kz[R][25], s0[R], s1[R], s2[R];
    float4 g[R];
    float2 mom[R];
#pragma unroll
    for (int k = 0; k < R; ++k) {
        const float A_ = a.sigma_z * gr[k].x * (1.0f / kLog2eF), B_ = a.sigma_z * gr[k].y * (1.0f / kLog2eF);
#pragma unroll
        for (int q = 0; q < 25; ++q) {
            // q enumerates the offsets with dy < 0, or dy == 0 and dx <= 0 (the centre is q = 24)
            const int dy = q < 21 ? q / 7 - 3 : 0;
            const int dx = q < 21 ? q % 7 - 3 : q - 24;
            kz[k][q] = rcp_approx(fabsf(fmaf(float(dx), A_, float(dy) * B_)) + ez);
        }
        mom[k] = vt.m[cell + k * kVarTW];
        g[k] = vt.g[cell + k * kVarTW];
        s0[k] = s1[k] = s2[k] = 0.0f;
    }
#pragma unroll
    for (int r = -kVarHalo; r <= kVarHalo + R - 1; ++r) {
#pragma unroll
        for (int dx = -kVarHalo; dx <= kVarHalo; ++dx) {
            const float4 n = vt.g[cell + r * kVarTW + dx];
            const float2 m = vt.m[cell + r * kVarTW + dx];
#pragma unroll
            for (int k = 0; k < R; ++k) {
                const int dy = r - k;
                if (dy < -kVarHalo || dy > kVarHalo) continue;
                const bool neg = dy < 0 || (dy == 0 && dx <= 0);
                const int ex = neg ? dx : -dx, ey = neg ? dy : -dy;
                const int q = ey < 0 ? (ey + 3) * 7 + (ex + 3) : 24 + ex;
                const float d = fmaf(n.z, g[k].z, fmaf(n.y, g[k].y, n.x * g[k].x));
                float e = -fabsf(n.w - g[k].w) * kz[k][q];
                e = fmaf(a.sigma_n, lg2_approx(fmaxf(d, 0.0f)), e);
                const float wgt = ex2_approx(e);
                const float dm = m.x - mom[k].x;
                s0[k] += wgt;
                s1[k] = fmaf(wgt, dm, s1[k]);
                s2[k] = fmaf(wgt, fmaf(dm, dm, m.y), s2[k]);
            }
        }
    }
#pragma unroll
    for (int k = 0; k < R; ++k) {
        if (!need[k]) continue;
        float var = mom[k].y;
        if (s0[k] > 0.0f) {
            const float m1 = s1[k] / s0[k];
            var = fmaxf(0.0f, s2[k] / s0[k] - m1 * m1);
        }
        Rec::st_var(a.col_dst, a.var_off, size_t(y + k) * a.w + x, var);
    }
}

__device__ __forceinline__ int pixel_blocks(const FullArgs& a)
{
    return ((a.w + kBlockX - 1) / kBlockX) * ((a.h + kBlockY - 1) / kBlockY);
}

// One kBlockX x kBlockY pixel block `blk` (row-major over the image's blocks)
// of K1 and K2.  K1 records whether any pixel of the block needs the spatial
// fallback; K2 runs only those blocks.  Every thread of the CTA calls these (K1
// synchronises the CTA).
template <int ST> __device__ __forceinline__ void full_temporal_block(const FullArgs& a, int blk, int x, int y)
{
    const bool fb = (x < a.w && y < a.h) ? full_temporal_px<ST>(a, x, y) : false;
    const int any = __syncthreads_or(fb);
    if (threadIdx.x == 0 && threadIdx.y == 0) {
        if (!a.fb_count)
            a.fb_flags[blk] = any;
        else if (any) {
            const int at = atomicAdd(a.fb_count, 1);
            if (at < pixel_blocks(a)) a.fb_flags[at] = blk;  // (always: the counter is 0 before a frame)
        }
    }
}

// Pixels of a column per K2 thread: a CTA of 32 x (4 / R) threads takes a pixel
// block.  Two need 168 instead of 294 shared-memory wavefronts per 32 pixels; the
// persistent batch kernel, whose CTAs have 128 threads, takes one.  Measured at
// 1920x1080 after a cut (every block): frame 451 -> 423 us; a 3840x2160 frame
// with some of its blocks listed 1184 -> 1176 us (with two pixels per thread but
// flags instead of the list, 1184-1195: a CTA's share of the flagged blocks was
// uneven).  10, 11 and 16 CTAs per SM: 425, 431 and 430 us.
constexpr int kVarR = 2;
constexpr int kVarCtas = 12;

// K2 on one flagged pixel block at (bx, by); threadIdx is the thread's place in it.
template <int ST, int R> __device__ __forceinline__ void full_variance_tile(const FullArgs& a, int bx, int by, VarTile& vt)
{
    typedef Stor<ST> S;
    const int x = bx + int(threadIdx.x), y = by + int(threadIdx.y) * R;
    const int x0 = bx - kVarHalo, y0 = by - kVarHalo;
    const typename S::guide_t* gc = static_cast<const typename S::guide_t*>(a.guide_cur);
    const typename S::mom_t* mc = static_cast<const typename S::mom_t*>(a.mom_cur);
    // this thread's own pixels' inputs, loaded before the staging so that their latency overlaps it
    bool need[R];
    float2 gr[R];
    bool any = false;
#pragma unroll
    for (int k = 0; k < R; ++k) {
        const bool own = x < a.w && y + k < a.h;
        const size_t i = own ? size_t(y + k) * a.w + x : 0;
        need[k] = own && int(S::ld4_w(static_cast<const typename S::c4_t*>(a.tc), i)) < a.fallback_frames;
        gr[k] = own ? a.grad[size_t(y + k) * a.w + grad_col(a.w, x)] : make_float2(0.f, 0.f);
        any |= need[k];
    }
    for (int k = threadIdx.y * kBlockX + threadIdx.x; k < kVarTH * kVarTW; k += kBlockX * kBlockY / R) {
        const int qy = y0 + k / kVarTW, qx = x0 + k % kVarTW;
        float4 g = make_float4(0.f, 0.f, 0.f, 0.f);
        float2 m = make_float2(0.f, 0.f);
        if (qx >= 0 && qy >= 0 && qx < a.w && qy < a.h) {
            const size_t j = size_t(qy) * a.w + qx;
            g = S::ld_guide_w(gc, j);
            m = S::ldm(mc, j);
        }
        vt.g[k] = g;
        vt.m[k] = m;
    }
    __syncthreads();
    if (any)
        full_variance_px<ST, R>(a, x, y, (int(threadIdx.y) * R + kVarHalo) * kVarTW + int(threadIdx.x) + kVarHalo, vt, need, gr);
    __syncthreads();  // the tile's storage is reused by the caller's next block
}

// K2 grids over flags (batches): a CTA takes the pixel blocks base + t * stride (t < kVarPerCta) of
// its chunk, compacts the flagged ones into a shared list and runs only those,
// so that the mostly unflagged blocks of a frame cost one parallel flag read
// per chunk instead of one CTA each.
constexpr int kVarPerCta = 32;

__host__ __device__ inline int variance_grid(int items, int sms)
{
    const int lo = (items + kVarPerCta - 1) / kVarPerCta, hi = items < 12 * sms ? items : 12 * sms;
    return lo > hi ? lo : hi;
}

struct VarList {
    int item[kVarPerCta];
    int n;
};

// Fills `l` with the flagged items of the chunk at `base`; `flag(item)` reads an item's flag.
template <class Flag>
__device__ __forceinline__ void variance_compact(int base, int stride, int items, Flag flag, VarList& l)
{
    const int tid = threadIdx.y * kBlockX + threadIdx.x;
    if (tid == 0) l.n = 0;
    __syncthreads();
    if (tid < kVarPerCta) {
        const int item = base + tid * stride;
        if (item < items && flag(item)) l.item[atomicAdd(&l.n, 1)] = item;
    }
    __syncthreads();
}

// 8 CTAs of 128 threads per SM (64 registers a thread): 3% faster than 4 of 256.
template <int ST> __global__ void __launch_bounds__(kBlockX* kBlockY, 8) k_full_temporal(FullArgs a)
{
    pdl_begin();
    full_temporal_block<ST>(a, blockIdx.y * gridDim.x + blockIdx.x, blockIdx.x * kBlockX + threadIdx.x,
                            blockIdx.y * kBlockY + threadIdx.y);
}

// The listed blocks, one at a time per CTA of one resident wave (taken by ticket
// instead: 3840x2160 after a cut 1495 against 1520 us, but steady 1920x1080 328.1
// against 325.9).  Level 0 clears the counter for the next frame.
template <int ST> __global__ void __launch_bounds__(kBlockX* kBlockY / kVarR, kVarCtas) k_full_variance(FullArgs a)
{
    __shared__ VarTile vt;
    pdl_begin();
    const int tx = (a.w + kBlockX - 1) / kBlockX, n = min(__ldcg(a.fb_count), pixel_blocks(a));
    for (int e = blockIdx.x; e < n; e += gridDim.x) {
        const int b = __ldcg(a.fb_flags + e);
        full_variance_tile<ST, kVarR>(a, (b % tx) * kBlockX, (b / tx) * kBlockY, vt);
    }
}

// One CTA per pixel block, which looks at its own flag: no counter and no entry to
// wait for before the first block.  One pixel per thread:
// the frame waits for one block's time here, which two per thread would double.
template <int ST> __global__ void __launch_bounds__(kBlockX* kBlockY, 8) k_full_variance_flags(FullArgs a)
{
    __shared__ VarTile vt;
    pdl_begin();
    const int tx = (a.w + kBlockX - 1) / kBlockX, b = blockIdx.x;
    if (__ldcg(a.fb_flags + b)) full_variance_tile<ST, 1>(a, (b % tx) * kBlockX, (b / tx) * kBlockY, vt);
}

// Whether the estimate over a frame of `blocks` pixel blocks takes a list of them or
// flags.  Flags cost a CTA for every block that needs nothing: steady frames
// of 1280x720 (7200 blocks) take 163 us either way, 1920x1080 331.7 with flags against
// 326.0 and 3840x2160 1195 against 1154; 960x540 102.7 against 103.9, 564x307 58.8
// against 61.2, and right after a cut 122.5 against 130.1 and 67.9 against 71.2.
inline bool variance_list(int blocks, int sms) { return blocks > 48 * sms; }

// The list's counter between frames: level 0 leaves it 0, but a frame of which a
// launch was rejected may not have got there (`stale`), and the next frame would
// append to that frame's entries.  Called before such a frame's launches.  A
// captured frame keeps the clearing in its graph, so the next frame that runs at
// once still needs its own.
inline cudaError_t clear_stale_count(int* count, bool& stale, cudaStream_t st)
{
    if (!stale) return cudaSuccess;
    cudaStreamCaptureStatus cs = cudaStreamCaptureStatusNone;
    cudaError_t e = cudaStreamIsCapturing(st, &cs);
    if (e == cudaSuccess) e = cudaMemsetAsync(count, 0, sizeof *count, st);
    if (e == cudaSuccess && cs == cudaStreamCaptureStatusNone) stale = false;
    return e;
}

inline cudaError_t launch_variance(const FullArgs& a, bool f16, int blocks, int sms, cudaStream_t st)
{
    if (!variance_list(blocks, sms))
        return launch_chain(f16 ? k_full_variance_flags<ST_FP16> : k_full_variance_flags<ST_FP32>, dim3(blocks),
                            dim3(kBlockX, kBlockY), st, a);
    const int wave = kVarCtas * sms;
    return launch_chain(f16 ? k_full_variance<ST_FP16> : k_full_variance<ST_FP32>, dim3(blocks < wave ? blocks : wave),
                        dim3(kBlockX, kBlockY / kVarR), st, a);
}

} // namespace tg
