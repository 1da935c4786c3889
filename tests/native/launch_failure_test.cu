// The library's host code against a CUDA runtime that rejects launches, on the
// host alone: fake_cuda_runtime.cpp defines the runtime calls that the library
// makes, and its definitions take the place of libcudart's.
//
//   counter   A frame of which any launch is rejected leaves no entry in the
//             fallback list of the next one.  The fake launches do to the list
//             what the kernels do: the temporal pass appends every block, the
//             estimate needs exactly those, level 0 clears the counter.  The
//             handle, and the server's plain path, whose sessions share one
//             counter.
//   last      A call that reports a rejected launch takes the error with it:
//             the thread's last error is clear afterwards.
//
// Prints "ok" and exits 0 on success.
#include <cuda_runtime.h>

#include <cstdio>
#include <cstring>
#include <vector>

#include "fake_cuda_runtime.h"
#include "svgf_kernels.cuh"
#include "tg_fog.h"
#include "tg_post.h"
#include "tg_svgf.h"

namespace {

int g_per_frame = 0;  // launches of a filter frame; 0: launches are only counted
int g_bad_lists = 0;  // estimates that found other entries than their own frame's
int g_lists = 0;      // estimates over a list

void run(int stage, const tg::FullArgs& a)
{
    if (!a.fb_count || fake::capturing) return;
    const int blocks = ((a.w + 31) / 32) * ((a.h + 3) / 4);
    if (stage == 0)
        *a.fb_count += blocks;
    else if (stage == 1) {
        ++g_lists;
        if (*a.fb_count != blocks) ++g_bad_lists;
    } else if (stage == 2)
        *a.fb_count = 0;
}

int fails = 0;
void check(bool ok, const char* what, int k = 0)
{
    if (ok) return;
    std::printf("FAIL: %s (%d)\n", what, k);
    ++fails;
}

} // namespace

void fake::launched(int k, void** args)
{
    if (g_per_frame) run(k % g_per_frame, *static_cast<const tg::FullArgs*>(args[0]));
}

namespace {

struct Images {
    std::vector<char> rad, dep, nrm, mot, out;
    tg_svgf_inputs in{};
    tg_svgf_outputs o{};
    Images(size_t n) : rad(n * 16), dep(n * 4), nrm(n * 12), mot(n * 8), out(n * 16)
    {
        in.radiance = {rad.data(), 0, TG_FMT_RGBA32F, 0};
        in.depth = {dep.data(), 0, TG_FMT_R32F, 0};
        in.normal = {nrm.data(), 0, TG_FMT_RGB32F, 0};
        in.motion = {mot.data(), 0, TG_FMT_RG32F, 0};
        o.denoised = {out.data(), 0, TG_FMT_RGBA32F, 0};
    }
};

constexpr uint32_t kW = 1280, kH = 732;  // 40 x 183 blocks: more than 48 per multiprocessor, so by list

void reset(int per_frame, int reject)
{
    fake::launches = 0;
    g_per_frame = per_frame;
    fake::reject = reject;
}

void counter_handle()
{
    tg_svgf_desc d{};
    d.width = kW;
    d.height = kH;
    tg_svgf_params_default(TG_SVGF_MODE_FULL, TG_SVGF_STORAGE_FP32, &d.params);
    Images im(size_t(kW) * kH);
    const int n = d.params.levels + 2;
    for (int k = 0; k < n; ++k) {
        tg_svgf* s = nullptr;
        reset(n, -1);
        check(tg_svgf_create(&d, &s) == TG_OK, "create");
        cudaGetLastError();
        check(tg_svgf_denoise(s, &im.in, &im.o, nullptr) == TG_OK, "good frame", k);
        reset(n, k);
        g_bad_lists = g_lists = 0;
        check(tg_svgf_denoise(s, &im.in, &im.o, nullptr) == TG_ERR_CUDA, "a rejected launch is reported", k);
        g_bad_lists = 0;  // (the failed frame's own estimate may have run without its temporal pass)
        // a frame captured meanwhile runs nothing now, and leaves the clearing to the next one that does
        reset(n, -1);
        fake::capturing = true;
        check(tg_svgf_denoise(s, &im.in, &im.o, nullptr) == TG_OK, "captured frame", k);
        fake::capturing = false;
        for (int f = 0; f < 2; ++f) {
            reset(n, -1);
            check(tg_svgf_denoise(s, &im.in, &im.o, nullptr) == TG_OK, "frame after a failed one", k);
        }
        check(g_bad_lists == 0, "stale entries in the handle's list after launch", k);
        check(g_lists >= 2, "frames of this size take a list", k);
        tg_svgf_destroy(s);
    }
}

int serve(tg_svgf_server* sv, uint64_t session, uint32_t w, uint32_t h, Images& im)
{
    uint64_t t = 0;
    if (tg_svgf_server_submit(sv, session, w, h, &im.in, &im.o, &t) != TG_OK) return -1;
    tg_svgf_request_info r{};
    const int st = tg_svgf_server_wait(sv, t, 60000000, &r);
    return st == TG_OK ? r.status : st;
}

void counter_server()
{
    tg_svgf_server_desc d{};
    tg_svgf_params_default(TG_SVGF_MODE_FULL, TG_SVGF_STORAGE_FP32, &d.params);
    d.max_sessions = 4;
    d.max_batch = 1;
    d.hbm_budget_bytes = 1ull << 30;
    d.device = -1;
    d.batching = 0;
    const int n = d.params.levels + 2;
    Images big(size_t(kW) * kH), other(size_t(1288) * 1000);
    for (int k = 0; k < n; ++k) {
        tg_svgf_server* sv = nullptr;
        reset(n, -1);
        check(tg_svgf_server_create(&d, &sv) == TG_OK, "server create");
        check(serve(sv, 1, kW, kH, big) == TG_OK, "good request", k);
        reset(n, k);
        check(serve(sv, 1, kW, kH, big) == TG_ERR_CUDA, "a request with a rejected launch fails", k);
        g_bad_lists = g_lists = 0;
        reset(n, -1);
        // another session: its memory holds no list yet
        check(serve(sv, 2, 1288, 1000, other) == TG_OK, "another session's request", k);
        reset(n, -1);
        check(serve(sv, 1, kW, kH, big) == TG_OK, "next request", k);
        check(g_bad_lists == 0, "stale entries in the server's list after launch", k);
        check(g_lists == 2, "requests of this size take a list", k);
        tg_svgf_server_destroy(sv);
    }
}

void last_error()
{
    std::vector<char> hdr(64 * 48 * 16), disp(64 * 48 * 4);
    tg_post* p = nullptr;
    reset(0, -1);
    check(tg_post_create(64, 48, nullptr, -1, &p) == TG_OK, "post create");
    const tg_image in = {hdr.data(), 0, TG_FMT_RGBA32F, 0}, out = {disp.data(), 0, TG_FMT_BGRA8, 0};
    cudaGetLastError();
    check(tg_post_process(p, &in, &out, nullptr) == TG_OK, "post frame");
    const int launches = fake::launches;
    for (int k = 0; k < launches; ++k) {
        reset(0, k);
        check(tg_post_process(p, &in, &out, nullptr) == TG_ERR_CUDA, "post: a rejected launch is reported", k);
        check(cudaGetLastError() == cudaSuccess, "post leaves its error to the next call", k);
    }
    tg_post_destroy(p);

    std::vector<char> vol(3 * 8 * 8 * 8 * 16);
    tg_volume v[3];
    for (int k = 0; k < 3; ++k) v[k] = {vol.data() + k * 8 * 8 * 8 * 16, 0, 0, TG_FMT_RGBA32F, 0};
    tg_fog_filter_params fp{};
    fp.froxel_width = fp.froxel_height = fp.froxel_depth = 8;
    fp.near_plane = 0.1f;
    fp.far_plane = 100.f;
    reset(0, 0);
    check(tg_fog_filter(&fp, &v[0], &v[1], &v[2], nullptr) == TG_ERR_CUDA, "fog: a rejected launch is reported");
    check(cudaGetLastError() == cudaSuccess, "fog leaves its error to the next call");

    const uint32_t w = 64, h = 48;
    tg_svgf_batch_desc d{};
    d.n_streams = 1;
    d.widths = &w;
    d.heights = &h;
    d.device = -1;
    tg_svgf_params_default(TG_SVGF_MODE_FULL, TG_SVGF_STORAGE_FP32, &d.params);
    tg_svgf_batch* b = nullptr;
    check(tg_svgf_batch_create(&d, &b) == TG_OK, "batch create");
    if (!b) return;
    Images im(w * h);
    const uint32_t id = 0;
    cudaGetLastError();
    for (int k = 0; k < d.params.levels + 2; ++k) {
        reset(0, k);
        check(tg_svgf_batch_denoise(b, 1, &id, &im.in, &im.o, nullptr) == TG_ERR_CUDA, "batch: a rejected launch is reported", k);
        check(cudaGetLastError() == cudaSuccess, "batch leaves its error to the next call", k);
    }
    tg_svgf_batch_destroy(b);
}

} // namespace

int main(int argc, char** argv)
{
    const char* which = argc > 1 ? argv[1] : "";
    if (!std::strcmp(which, "counter")) {
        counter_handle();
        counter_server();
    } else if (!std::strcmp(which, "last")) {
        last_error();
    } else {
        return 2;
    }
    if (fails) return 1;
    std::printf("ok\n");
    return 0;
}
