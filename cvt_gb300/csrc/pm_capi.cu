/*
 * pm_capi.cu — the C ABI of include/cvtpm.h: context, scratch memory and the
 * host schedule of PMHuberStereo::depthMap (cvt/vision/PMHuberStereo.cpp:64-291)
 * over the kernels of pm_kernels.cu.
 *
 * Differences from the reference host code, none of which changes a result:
 *  - scratch lives in the context and is reused across calls (the reference
 *    allocates 14 images and 2 buffers per call, PMHuberStereo.cpp:78-122);
 *  - launches are stream-ordered with no host synchronisation (the reference
 *    blocks after every launch with runWait);
 *  - the debug block that writes PNGs and waits on getchar()
 *    (PMHuberStereo.cpp:153-185) is not reproduced;
 *  - the view-candidate buffers hold source positions instead of copies of
 *    the candidate planes (k_view_list).
 */
#include <algorithm>
#include <chrono>
#include <cstdio>
#include <cstring>
#include <memory>
#include <mutex>
#include <string>
#include <new>
#include <vector>

#include <nvtx3/nvToolsExt.h>

#include "cvtpm.h"
#include "cvtpm_tools.h"
#include "pm_kernels.cuh"

#define CVTPM_VERSION "cvt-gb300 0.1.0 (sm_103a)"
#define PM_MAX_WIDTH 12288

struct cvtpm_ctx {
    int device = 0;
    cvtpm_params prm;
    std::string err;
    /* scratch, carved from one allocation */
    void* pool = nullptr;
    size_t pool_bytes = 0;
    int capW = 0, capH = 0;
    float4 *col[2], *grad[2], *recA[2], *recB[2], *recC[2];
    float2* recD[2];
    float* wgt[2];
    float4* S[2][2];
    float4* smooth[2];
    float4 *tmp, *tmp2, *pdT;
    float* pdP[2];                    /* smoother duals (pm_pd_dual_bytes) */
    /* the right view's smoother runs on `side`, beside the next left pass,
     * with scratch of its own */
    float4 *tmpR, *tmp2R, *pdTR;
    float* pdPR[2];
    cudaStream_t side = nullptr;
    cudaEvent_t side_fork = nullptr, side_join = nullptr;
    short4* list[2];
    uint8_t* win[2];
    uint8_t* valid;
    float* occ;                       /* occlusion mask of depthMapInpaint */
    /* what a propagation pass needs to share work between its candidates (plan_pass),
     * when the budget allows */
    void* pass = nullptr;
    size_t pass_bytes = 0;
    size_t pass_pixels = 0;           /* the largest image it was allocated for */
    size_t pass_budget = SIZE_MAX;
    /* set while a launch sequence is being captured into a graph: scratch
     * must already be sized, nothing may be allocated */
    bool no_alloc = false;
    /* cvtpm_depthmap_batched: lanes (own scratch and stream each), the
     * captured graph of the last batch and the tuning record */
    struct Lane { cvtpm_ctx* c = nullptr; cudaStream_t s = nullptr; cudaEvent_t done = nullptr; };
    std::vector<Lane> lanes;
    /* phase-batched mode: one scratch context per pair of the batch, the
     * tuned launch knobs per batch shape and the knobs of the current graph */
    std::vector<cvtpm_ctx*> bpairs;
    struct TunedBatch { std::vector<unsigned char> key; PmBatchKnobs kn; bool phased; float mode_ms[2]; };
    std::vector<TunedBatch> tuned_knobs;
    PmBatchKnobs knobs{1, 16, 4};     /* pinned by cvtpm_set_batch_knobs */
    bool pinned_knobs = false;
    cudaStream_t bstream = nullptr;
    cudaEvent_t bfork = nullptr, bjoin = nullptr;
    cudaGraphExec_t bexec = nullptr;
    std::vector<unsigned char> bkey;
    std::vector<unsigned char> tkey;   /* shapes of the last tuned batch (no pointers) */
    int tuned_lanes = 0;
    int batch_lanes = 0;              /* 0: autotune */
    cvtpm_batch_info binfo{};
    /* staging for the *_host entry points */
    void* stage = nullptr;
    size_t stage_bytes = 0;
    /* cvtpm_depthmap_image: left and right converted to RGBA float32 */
    void* istage = nullptr;
    size_t istage_bytes = 0;
    /* observability (cvtpm_get_stats) */
    cvtpm_stats stats{};
    bool timing = false;
    unsigned long long* dcount = nullptr;            /* device counters: evaluations, taps */
    std::vector<std::pair<cudaEvent_t, cudaEvent_t>> ev_prop, ev_pd;
    std::vector<cudaEvent_t> ev_free;
};

namespace {

std::mutex g_table_mu;
struct TableKey { int device; float cw; int prof; bool ok; };
std::vector<TableKey> g_tables;

cvtpm_status fail(cvtpm_ctx* c, cvtpm_status s, const std::string& m) {
    if (c) c->err = m;
    return s;
}
cvtpm_status cuda_fail(cvtpm_ctx* c, cudaError_t e, const char* where) {
    return fail(c, CVTPM_ERR_CUDA, std::string(where) + ": " + cudaGetErrorString(e));
}
#define CK(call, where) do { cudaError_t e_ = (call); if (e_ != cudaSuccess) return cuda_fail(ctx, e_, where); } while (0)
/* a kernel launch: checked and counted */
#define LK(call, where) do { CK(call, where); ++ctx->stats.launches; } while (0)

cudaEvent_t take_event(cvtpm_ctx* ctx) {
    if (!ctx->ev_free.empty()) { cudaEvent_t e = ctx->ev_free.back(); ctx->ev_free.pop_back(); return e; }
    cudaEvent_t e = nullptr;
    if (cudaEventCreate(&e) != cudaSuccess) return nullptr;
    return e;
}

/* Records an event pair around a phase when timing is on. */
struct PhaseTimer {
    cvtpm_ctx* ctx; cudaStream_t st; std::vector<std::pair<cudaEvent_t, cudaEvent_t>>* list;
    cudaEvent_t a = nullptr, b = nullptr;
    PhaseTimer(cvtpm_ctx* c, cudaStream_t s, std::vector<std::pair<cudaEvent_t, cudaEvent_t>>& l) : ctx(c), st(s), list(&l) {
        if (ctx->timing) { a = take_event(ctx); b = take_event(ctx); if (a) cudaEventRecord(a, st); }
    }
    void stop() {
        if (a && b) { cudaEventRecord(b, st); list->push_back({a, b}); a = b = nullptr; }
    }
};

/* An NVTX range around the host-side enqueue of a phase (a profiler shows
 * the phase's kernels under it); no cost without a profiler attached. */
struct NvtxRange {
    explicit NvtxRange(const char* name) { nvtxRangePushA(name); }
    ~NvtxRange() { nvtxRangePop(); }
    NvtxRange(const NvtxRange&) = delete;
    NvtxRange& operator=(const NvtxRange&) = delete;
};

/* Ends a stream capture that an exception interrupted (a failed host
 * allocation inside the captured host code): the partial graph is discarded
 * and the contexts' capture flags are cleared, so the stream and the
 * contexts stay usable.  release() after the normal end of the capture. */
struct CaptureGuard {
    cudaStream_t st;
    std::vector<cvtpm_ctx*> ctxs;
    bool active = true;
    CaptureGuard(cudaStream_t s, std::vector<cvtpm_ctx*> c) : st(s), ctxs(std::move(c)) {}
    void release() { active = false; }
    ~CaptureGuard() {
        if (!active) return;
        cudaGraph_t g = nullptr;
        if (cudaStreamEndCapture(st, &g) == cudaSuccess && g) cudaGraphDestroy(g);
        cudaGetLastError();
        for (cvtpm_ctx* c : ctxs) c->no_alloc = false;
    }
};

/* Two timing events, destroyed on every exit. */
struct EventPair {
    cudaEvent_t a = nullptr, b = nullptr;
    ~EventPair() {
        if (a) cudaEventDestroy(a);
        if (b) cudaEventDestroy(b);
    }
};

size_t align_up(size_t v, size_t a) { return (v + a - 1) / a * a; }

/* Row pitch (elements) of the record planes: even and two columns past the
 * row, so 16-byte chunks of the float2 plane never leave a row. */
int rec_pitch(int W) { return (int)align_up((size_t)W + 2, 4); }

void mwc_pow2_table(unsigned long long* t) {
    const unsigned __int128 M = 18446383549859758079ull;
    unsigned long long v = 4294883355ull;                 /* A */
    for (int k = 0; k < 64; ++k) {
        t[k] = v;
        v = (unsigned long long)(((unsigned __int128)v * v) % M);
    }
}

cvtpm_status ensure_tables(cvtpm_ctx* ctx, const cvtpm_params& p, cudaStream_t st) {
    std::lock_guard<std::mutex> lk(g_table_mu);
    for (auto& t : g_tables)
        if (t.device == ctx->device && t.ok && t.cw == p.color_weight && t.prof == p.weight_profile) return CVTPM_OK;
    static unsigned long long pow2[64];
    static float prof[PM_PROF_N * PM_PROF_N];
    mwc_pow2_table(pow2);
    for (int dy = -PM_PMAX; dy <= PM_PMAX; ++dy)
        for (int dx = -PM_PMAX; dx <= PM_PMAX; ++dx)
            prof[(dy + PM_PMAX) * PM_PROF_N + (dx + PM_PMAX)] = pm_profile(dx, dy, p.color_weight, p.weight_profile);
    CK(pm_upload_tables(pow2, prof, st), "upload tables");
    CK(cudaStreamSynchronize(st), "upload tables");
    bool found = false;
    for (auto& t : g_tables)
        if (t.device == ctx->device) { t.cw = p.color_weight; t.prof = p.weight_profile; t.ok = true; found = true; }
    if (!found) g_tables.push_back({ctx->device, p.color_weight, p.weight_profile, true});
    return CVTPM_OK;
}

cvtpm_status ensure_buffers(cvtpm_ctx* ctx, int W, int H) {
    if (ctx->pool && W * (size_t)H <= (size_t)ctx->capW * ctx->capH && W <= ctx->capW) {
        /* reuse: the carve below depends only on n = W*H, recompute it */
    }
    const size_t n = (size_t)W * H;
    const size_t nr = (size_t)rec_pitch(W) * H;
    /* duals: the one-step kernel keeps two float4 per pixel, the blocked one six planes */
    const size_t pd = std::max(n * 32, pm_pd_dual_bytes(W, H));
    size_t off = 0;
    std::vector<std::pair<void**, size_t>> parts;
    auto add = [&](void** p, size_t bytes) { parts.push_back({p, bytes}); off = align_up(off, 256) + bytes; };
    for (int v = 0; v < 2; ++v) {
        add((void**)&ctx->col[v], n * 16);
        add((void**)&ctx->grad[v], n * 16);
        add((void**)&ctx->recA[v], nr * 16);
        add((void**)&ctx->recB[v], nr * 16);
        add((void**)&ctx->recC[v], nr * 16);
        add((void**)&ctx->recD[v], nr * 8);
        add((void**)&ctx->wgt[v], n * 4);
        add((void**)&ctx->S[v][0], n * 16);
        add((void**)&ctx->S[v][1], n * 16);
        add((void**)&ctx->smooth[v], n * 16);
        add((void**)&ctx->list[v], view_list_bytes(W, H));
        add((void**)&ctx->win[v], n);
        add((void**)&ctx->pdP[v], pd);
    }
    add((void**)&ctx->tmp, n * 16);
    add((void**)&ctx->tmp2, n * 16);
    add((void**)&ctx->pdT, n * 16);
    add((void**)&ctx->tmpR, n * 16);
    add((void**)&ctx->tmp2R, n * 16);
    add((void**)&ctx->pdTR, n * 16);
    add((void**)&ctx->pdPR[0], pd);
    add((void**)&ctx->pdPR[1], pd);
    add((void**)&ctx->valid, n);
    add((void**)&ctx->occ, n * 4);
    const size_t need = align_up(off, 256);
    if (!ctx->side) {
        if (ctx->no_alloc) return fail(ctx, CVTPM_ERR_ALLOC, "side stream not created before capture");
        cudaError_t e = cudaStreamCreateWithFlags(&ctx->side, cudaStreamNonBlocking);
        if (e == cudaSuccess) e = cudaEventCreateWithFlags(&ctx->side_fork, cudaEventDisableTiming);
        if (e == cudaSuccess) e = cudaEventCreateWithFlags(&ctx->side_join, cudaEventDisableTiming);
        if (e != cudaSuccess) return cuda_fail(ctx, e, "side stream");
    }
    if (need > ctx->pool_bytes) {
        if (ctx->no_alloc) return fail(ctx, CVTPM_ERR_ALLOC, "scratch not sized before capture");
        if (ctx->pool) { cudaFree(ctx->pool); ctx->pool = nullptr; ctx->pool_bytes = 0; }
        cudaError_t e = cudaMalloc(&ctx->pool, need);
        if (e != cudaSuccess) { ctx->pool = nullptr; return fail(ctx, CVTPM_ERR_ALLOC, std::string("scratch allocation: ") + cudaGetErrorString(e)); }
        ctx->pool_bytes = need;
    }
    size_t o = 0;
    for (auto& pr : parts) { o = align_up(o, 256); *pr.first = (char*)ctx->pool + o; o += pr.second; }
    ctx->capW = W; ctx->capH = H;
    return CVTPM_OK;
}

cvtpm_status check_params(cvtpm_ctx* ctx, const cvtpm_params& p) {
    if (p.patchsize < 1 || p.patchsize > PM_PMAX) return fail(ctx, CVTPM_ERR_SIZE, "patchsize must be in 1..31");
    if (!(p.depthmax > 0.0f)) return fail(ctx, CVTPM_ERR_INVALID_ARGUMENT, "depthmax must be > 0");
    if (p.iterations < 1) return fail(ctx, CVTPM_ERR_INVALID_ARGUMENT, "iterations must be >= 1");
    if (p.pd_iterations < 0) return fail(ctx, CVTPM_ERR_INVALID_ARGUMENT, "pd_iterations must be >= 0");
    if (p.rng != CVTPM_RNG_MWC64X && p.rng != CVTPM_RNG_PHILOX) return fail(ctx, CVTPM_ERR_INVALID_ARGUMENT, "bad rng");
    if (p.arith != CVTPM_ARITH_EXACT && p.arith != CVTPM_ARITH_FAST) return fail(ctx, CVTPM_ERR_INVALID_ARGUMENT, "bad arith");
    if (p.schedule != CVTPM_SCHEDULE_JACOBI && p.schedule != CVTPM_SCHEDULE_REDBLACK)
        return fail(ctx, CVTPM_ERR_INVALID_ARGUMENT, "schedule must be CVTPM_SCHEDULE_JACOBI or _REDBLACK");
    if (p.weight_profile != CVTPM_PROFILE_SMOOTHSTEP && p.weight_profile != CVTPM_PROFILE_CONSTANT)
        return fail(ctx, CVTPM_ERR_INVALID_ARGUMENT, "bad weight_profile");
    return CVTPM_OK;
}

cvtpm_status check_image(cvtpm_ctx* ctx, const void* p, int W, int H, size_t pitch, const char* what) {
    if (!p) return fail(ctx, CVTPM_ERR_INVALID_ARGUMENT, std::string(what) + " is NULL");
    if (W < 1 || H < 1 || W > PM_MAX_WIDTH || H > 65535) return fail(ctx, CVTPM_ERR_SIZE, "image size out of range");
    if (pitch % 16 != 0 || pitch < (size_t)W * 16) return fail(ctx, CVTPM_ERR_INVALID_ARGUMENT, std::string(what) + " pitch must be a multiple of 16 and >= 16*width");
    if (((uintptr_t)p & 15) != 0) return fail(ctx, CVTPM_ERR_INVALID_ARGUMENT, std::string(what) + " must be 16-byte aligned");
    return CVTPM_OK;
}

/* An empty view list: no sources, no entries. */
cudaError_t clear_view_list(short4* list, int W, int H, cudaStream_t st) {
    cudaError_t e = cudaMemsetAsync(list, 0xFF, (size_t)W * H * 8, st);
    return e != cudaSuccess ? e : cudaMemsetAsync(view_counts(list, W, H), 0, (size_t)H * 4, st);
}

PmPassArgs base_args(cvtpm_ctx* ctx, const cvtpm_params& p, int W, int H, int v1) {
    PmPassArgs a;
    memset(&a, 0, sizeof(a));
    a.k.W = W; a.k.H = H; a.k.P = p.patchsize;
    a.k.Wf = (float)W; a.k.Hf = (float)H;
    a.k.alpha = p.color_alpha; a.k.oma = 1.0f - p.color_alpha;
    a.k.cmax = p.color_maxdiff; a.k.gmax = p.grad_maxdiff;
    a.k.rp = rec_pitch(W);
    const int v2 = 1 - v1;
    a.v1 = {ctx->col[v1], ctx->grad[v1], ctx->recA[v1], ctx->recB[v1], ctx->recC[v1], ctx->recD[v1]};
    a.v2 = {ctx->col[v2], ctx->grad[v2], ctx->recA[v2], ctx->recB[v2], ctx->recC[v2], ctx->recD[v2]};
    a.lr = v1 == 0 ? 1 : 0;
    a.rng = p.rng;
    a.key0 = (uint32_t)p.seed; a.key1 = (uint32_t)(p.seed >> 32);
    a.depthmax = p.depthmax;
    a.color = -1;
    return a;
}

/* One propagation pass of a view: old states a.old -> a.out.  Jacobi (the
 * reference, pmhstereo.cl:286-404): every pixel from the old field.
 * Red/black (optional): the pixels with (x + y) even from the old field,
 * then the odd ones from the field with the even ones updated; the old
 * buffer is overwritten with that intermediate field. */
cvtpm_status propagate_view(cvtpm_ctx* ctx, PmPassArgs a, bool exact, bool redblack, size_t n, cudaStream_t st) {
    if (!redblack) {
        LK(pm_launch_pass_own(a, exact, st), "propagate");
        LK(pm_launch_pass_rest(a, exact, st), "propagate");
        return CVTPM_OK;
    }
    float4* A = const_cast<float4*>(a.old);
    for (int c = 0; c < 2; ++c) {
        if (c == 0) CK(cudaMemcpyAsync(a.out, A, n * 16, cudaMemcpyDeviceToDevice, st), "red/black copy");
        else CK(cudaMemcpyAsync(A, a.out, n * 16, cudaMemcpyDeviceToDevice, st), "red/black copy");
        a.color = c;
        LK(pm_launch_pass_own(a, exact, st), c ? "propagate black" : "propagate red");
        LK(pm_launch_pass_rest(a, exact, st), c ? "propagate black" : "propagate red");
    }
    return CVTPM_OK;
}

/* Gives the two views' passes the scratch that lets candidates share work:
 * per pixel of a small image 16 bytes for each of 16 candidates and 4 view
 * candidates (tap-parallel passes), else 4 bytes for each of 2 and 4 (shared
 * plane windows).  With the own candidates' part twice, the right view's first
 * part can run beside the left view's pass (*overlap); the view candidates'
 * part is used by one view at a time.  The most that fits the context's budget
 * and 60 % of the free memory is taken; with none of it every candidate is
 * evaluated per pixel.  Results are the same in every case.
 *
 * A caller's captured graphs hold the scratch's address, so it is replaced, as
 * the pool of ensure_buffers is, only for an image of more pixels than any
 * before: an allocation is large enough for every smaller image too (their
 * tap-parallel passes take more than the shared windows of larger ones), and
 * where memory was short then, what there is stays.  While `st` is captured
 * nothing is allocated. */
cvtpm_status plan_pass(cvtpm_ctx* ctx, const cvtpm_params& p, int W, int H, bool taps, cudaStream_t st, PmPassArgs* aL,
                       PmPassArgs* aR, bool* overlap) {
    const PmCostConsts k = base_args(ctx, p, W, H, 0).k;
    *overlap = p.schedule == CVTPM_SCHEDULE_JACOBI;
    if (!*overlap) return CVTPM_OK;
    const size_t n = (size_t)W * H;
    cudaStreamCaptureStatus cap = cudaStreamCaptureStatusNone;
    CK(cudaStreamIsCapturing(st, &cap), "capture status");
    const bool grow = !ctx->no_alloc && cap == cudaStreamCaptureStatusNone && (!ctx->pass || n > ctx->pass_pixels);
    const size_t small = taps ? std::min(n, (size_t)pm_tap_parallel_pixels()) * sizeof(float4) * 36 : 0;
    taps = taps && pm_tap_parallel(k);
    for (int plan = taps ? 0 : 2; plan < (pm_shared_windows(k) ? 4 : 2); ++plan) {
        const bool both = (plan & 1) == 0, t = plan < 2;
        const size_t need = t ? n * sizeof(float4) * (both ? 36 : 20) : n * sizeof(float) * (both ? 8 : 6);
        if (need > ctx->pass_budget) continue;
        if (need > ctx->pass_bytes) {
            if (!grow) continue;                     /* what is there */
            if (ctx->pass) { CK(cudaFree(ctx->pass), "free pass scratch"); ctx->pass = nullptr; ctx->pass_bytes = 0; }
            size_t fr = 0, tot = 0;
            CK(cudaMemGetInfo(&fr, &tot), "memory info");
            if ((double)need > 0.6 * (double)fr) continue;
            const size_t most = std::min(std::max(need, small), std::min(ctx->pass_budget, (size_t)(0.6 * (double)fr)));
            if (cudaMalloc(&ctx->pass, most) != cudaSuccess) {
                cudaGetLastError();                  /* clear the failed allocation */
                ctx->pass = nullptr;
                continue;
            }
            ctx->pass_bytes = most;
            ctx->pass_pixels = n;
        }
        if (t) {
            aL->cand = (float4*)ctx->pass;
            aR->cand = both ? aL->cand + 16 * n : aL->cand;
            aL->vcand = aR->vcand = aR->cand + 16 * n;
        } else {
            aL->costs = (float*)ctx->pass;
            aR->costs = both ? aL->costs + 2 * n : aL->costs;
            aL->vcosts = aR->vcosts = aR->costs + 2 * n;
        }
        *overlap = both;
        return CVTPM_OK;
    }
    return CVTPM_OK;
}

cvtpm_status prep_views(cvtpm_ctx* ctx, const cvtpm_params& p, const float* img0, const float* img1, int W, int H,
                        size_t pitch, cudaStream_t st, bool records = false) {
    const float* im[2] = {img0, img1};
    for (int v = 0; v < 2; ++v) {
        LK(pm_launch_prep((const float4*)im[v], pitch / 16, W, H, ctx->col[v], ctx->grad[v], ctx->wgt[v], st), "prep");
        if (p.arith == CVTPM_ARITH_FAST || records)
            LK(pm_launch_records(ctx->col[v], ctx->grad[v], W, H, rec_pitch(W), ctx->recA[v], ctx->recB[v], ctx->recC[v], ctx->recD[v], st), "records");
    }
    return CVTPM_OK;
}

/* PDROF::apply, cvt/gfx/PDROF.h:50-96 (mask == NULL), or
 * PDROFInpaint::apply, cvt/gfx/PDROFInpaint.h:50-98 (mask: the occlusion
 * map): u warm-starts from `output`, p from 0;
 * `iters` steps, plus one when `iters` is odd so the result lands in
 * `output` (:83-95).  The steps run pm_pd_block_steps() at a time in the
 * temporally blocked kernel (identical arithmetic); iters == 0 keeps the reference's single
 * extra step from a copy of the input. */
cvtpm_status pd_apply(cvtpm_ctx* ctx, float4* output, const float4* input, const float* wgt, float lambda, int iters,
                      int W, int H, cudaStream_t st, const float* mask = nullptr, int scratch = 0) {
    const size_t n = (size_t)W * H;
    float4* const pdT = scratch ? ctx->pdTR : ctx->pdT;
    float* const pdP0 = scratch ? ctx->pdPR[0] : ctx->pdP[0];
    float* const pdP1 = scratch ? ctx->pdPR[1] : ctx->pdP[1];
    PhaseTimer tm(ctx, st, ctx->ev_pd);
    if (iters == 0) {
        CK(cudaMemcpyAsync(pdT, input, n * 16, cudaMemcpyDeviceToDevice, st), "pd copy");
        CK(cudaMemsetAsync(pdP0, 0, n * 32, st), "pd clear");
        LK(pm_launch_pd_step(output, (float4*)pdP1, pdT, (const float4*)pdP0, input, wgt, mask, lambda, W, H, st), "pd step");
        ++ctx->stats.pd_launches;
        ++ctx->stats.pd_steps;
        tm.stop();
        return CVTPM_OK;
    }
    const int total = iters + (iters & 1);
    const int K = pm_pd_block_steps();
    float4* U[2] = {output, pdT};
    float* Pp[2] = {pdP0, pdP1};
    int l = 0;
    for (int done = 0; done < total; done += K, ++l) {
        const int steps = total - done < K ? total - done : K;
        LK(pm_launch_pd_block(U[(l + 1) & 1], Pp[(l + 1) & 1], U[l & 1], Pp[l & 1], l == 0 ? 1 : 0, input, wgt, mask,
                              lambda, steps, W, H, st), "pd block");
        ++ctx->stats.pd_launches;
        ctx->stats.pd_steps += (uint64_t)steps;
    }
    if (U[l & 1] != output) CK(cudaMemcpyAsync(output, U[l & 1], n * 16, cudaMemcpyDeviceToDevice, st), "pd copy");
    tm.stop();
    return CVTPM_OK;
}

float smoothstep01(float x) {                                      /* cvt/math/Math.h:88-92 */
    float t = (x < 0.0f) ? 0.0f : (x > 1.0f) ? 1.0f : x;
    return t * t * (3.0f - 2.0f * t);
}

/* The theta of iteration k of an N-iteration run (PMHuberStereo.cpp:264-265). */
float theta_at(int k, int N) {
    float theta = 0.0f;
    for (int iter = 0; iter < k; ++iter)
        if (iter >= 5) theta = smoothstep01(((float)iter - 5.0f) / ((float)N - 5.0f)) * 1.0f;
    return theta;
}

cvtpm_status check_checkpoint(cvtpm_ctx* ctx, const cvtpm_checkpoint* c, int N, const char* what) {
    if (!c) return CVTPM_OK;
    if (c->iteration < 0 || c->iteration > N)
        return fail(ctx, CVTPM_ERR_INVALID_ARGUMENT, std::string(what) + ": iteration out of 0..iterations");
    if (!c->states || !c->smooth || ((uintptr_t)c->states & 15) || ((uintptr_t)c->smooth & 15))
        return fail(ctx, CVTPM_ERR_INVALID_ARGUMENT, std::string(what) + ": states/smooth NULL or not 16-byte aligned");
    return CVTPM_OK;
}

/* The depthMap schedule.  resume (optional) starts at iteration
 * resume->iteration from its state instead of the random init; the run stops
 * before iteration `stop` (stop < 0: all iterations), saves the state there
 * into `save` (optional) and produces dmap only when it ran to the end. */
cvtpm_status run_depthmap(cvtpm_ctx* ctx, const cvtpm_params& p, float* dmap, size_t dpitch, const float* left,
                          const float* right, int W, int H, size_t pitch, float* nmap, size_t npitch,
                          const cvtpm_trace* trace, cudaStream_t st, const cvtpm_checkpoint* resume = nullptr,
                          int stop = -1, cvtpm_checkpoint* save = nullptr) {
    cvtpm_status s;
    if ((s = check_params(ctx, p)) != CVTPM_OK) return s;
    if ((s = check_image(ctx, left, W, H, pitch, "left")) != CVTPM_OK) return s;
    if ((s = check_image(ctx, right, W, H, pitch, "right")) != CVTPM_OK) return s;
    const int first = resume ? resume->iteration : 0;
    const int last = (stop < 0 || stop > p.iterations) ? p.iterations : stop;
    if ((s = check_checkpoint(ctx, resume, p.iterations, "resume")) != CVTPM_OK) return s;
    if (save && !save->states && !save->smooth) save = nullptr;
    if (save) {
        cvtpm_checkpoint chk = *save;
        chk.iteration = last;
        if ((s = check_checkpoint(ctx, &chk, p.iterations, "save")) != CVTPM_OK) return s;
    }
    if (last < first) return fail(ctx, CVTPM_ERR_INVALID_ARGUMENT, "stop comes before the resumed iteration");
    const bool finish = last == p.iterations;
    if (finish && !dmap) return fail(ctx, CVTPM_ERR_INVALID_ARGUMENT, "dmap is NULL");
    if (finish && (dpitch % 4 != 0 || dpitch < (size_t)W * 4)) return fail(ctx, CVTPM_ERR_INVALID_ARGUMENT, "dmap pitch");
    if (nmap && (npitch % 16 != 0 || npitch < (size_t)W * 16)) return fail(ctx, CVTPM_ERR_INVALID_ARGUMENT, "normalmap pitch");
    CK(cudaSetDevice(ctx->device), "cudaSetDevice");
    if ((s = ensure_buffers(ctx, W, H)) != CVTPM_OK) return s;
    if ((s = ensure_tables(ctx, p, st)) != CVTPM_OK) return s;
    if ((s = prep_views(ctx, p, left, right, W, H, pitch, st)) != CVTPM_OK) return s;

    const size_t n = (size_t)W * H;
    const bool exact = p.arith == CVTPM_ARITH_EXACT;
    const float dmax = p.depthmax;
    const float dscale = p.dscale <= 0.0f ? 1.0f / dmax : p.dscale;
    const int N = p.iterations;
    PmPassArgs aL = base_args(ctx, p, W, H, 0), aR = base_args(ctx, p, W, H, 1);
    bool overlap = false;
    if ((s = plan_pass(ctx, p, W, H, true, st, &aL, &aR, &overlap)) != CVTPM_OK) return s;
    if (!ctx->dcount) {
        if (ctx->no_alloc) return fail(ctx, CVTPM_ERR_ALLOC, "counters not allocated before capture");
        CK(cudaMalloc(&ctx->dcount, 2 * sizeof(unsigned long long)), "counters");
        CK(cudaMemset(ctx->dcount, 0, 2 * sizeof(unsigned long long)), "counters");
    }
    ++ctx->stats.calls;
    NvtxRange whole("cvtpm depthMap");

    if (!resume) {
        NvtxRange r("init");
        aL.out = ctx->S[0][0];                                     /* :124-143 */
        LK(pm_launch_init(aL, exact, st), "init");
        aR.out = ctx->S[1][0];
        LK(pm_launch_init(aR, exact, st), "init");
        CK(cudaMemsetAsync(ctx->smooth[0], 0, n * 16, st), "clear");   /* :108-113 */
        CK(cudaMemsetAsync(ctx->smooth[1], 0, n * 16, st), "clear");
        CK(clear_view_list(ctx->list[1], W, H, st), "clear");   /* :145-149 */
    } else {
        /* the state before iteration `first`: both views' planes and smoothed
         * fields; the left pass's view list is the one the right view's
         * planes give (or empty before iteration 0) */
        NvtxRange r("resume");
        const int sw0 = first & 1;
        for (int v = 0; v < 2; ++v) {
            CK(cudaMemcpyAsync(ctx->S[v][sw0], resume->states + (size_t)v * 4 * n, n * 16, cudaMemcpyDeviceToDevice, st),
               "resume");
            CK(cudaMemcpyAsync(ctx->smooth[v], resume->smooth + (size_t)v * 4 * n, n * 16, cudaMemcpyDeviceToDevice, st),
               "resume");
        }
        if (first == 0) CK(clear_view_list(ctx->list[1], W, H, st), "clear");
        else LK(pm_launch_view_list(ctx->S[1][sw0], W, H, ctx->list[1], st), "view list");
    }

    float theta = theta_at(first, N);
    aL.counters = aR.counters = ctx->dcount;
    aL.winners = ctx->win[0];
    aR.winners = ctx->win[1];
    /* The right view's candidates 1-16 need its own planes and smoothed field
     * only, so they run on the side stream behind its smoother, beside the left
     * view's smoother and pass: the launches of the two chains fill the SMs
     * that the other's last waves leave idle (321x243 51.0 -> 44.5 ms, 1242x375
     * 339.3 -> 335.5).  The right view's pass then takes the left view's planes
     * and refines on `st`.  Not while the phases are timed, on `st`. */
    overlap = overlap && !ctx->timing;
    auto right_own = [&](int iter, float th) -> cvtpm_status {
        const int sw = iter & 1;
        aR.iter = iter;
        aR.theta = th;
        aR.old = ctx->S[1][sw]; aR.out = ctx->S[1][1 - sw]; aR.smooth = ctx->smooth[1];
        LK(pm_launch_pass_own(aR, exact, ctx->side), "propagate");
        return CVTPM_OK;
    };
    if (overlap && first < last) {
        CK(cudaEventRecord(ctx->side_fork, st), "fork");
        CK(cudaStreamWaitEvent(ctx->side, ctx->side_fork, 0), "fork");
        if ((s = right_own(first, theta)) != CVTPM_OK) return s;
        CK(cudaEventRecord(ctx->side_join, ctx->side), "join");
    }
    for (int iter = first; iter < last; ++iter) {                  /* :151-266 */
        const int sw = iter & 1;
        const bool redblack = p.schedule == CVTPM_SCHEDULE_REDBLACK;
        const float next = iter >= 5 ? smoothstep01(((float)iter - 5.0f) / ((float)N - 5.0f)) * 1.0f : theta;
        aL.iter = iter;
        aL.theta = theta;
        aL.old = ctx->S[0][sw]; aL.out = ctx->S[0][1 - sw]; aL.smooth = ctx->smooth[0];
        aL.viewin = ctx->list[1]; aL.viewsrc = ctx->S[1][sw];
        {
            NvtxRange r("propagate left");
            PhaseTimer tm(ctx, st, ctx->ev_prop);
            if ((s = propagate_view(ctx, aL, exact, redblack, n, st)) != CVTPM_OK) return s;
            tm.stop();
        }
        LK(pm_launch_view_list(ctx->S[0][1 - sw], W, H, ctx->list[0], st), "view list");
        if (overlap || iter > first) CK(cudaStreamWaitEvent(st, ctx->side_join, 0), "join");   /* smooth[1] */
        aR.viewin = ctx->list[0]; aR.viewsrc = ctx->S[0][1 - sw];
        {
            NvtxRange r("propagate right");
            PhaseTimer tm(ctx, st, ctx->ev_prop);
            if (overlap) {
                LK(pm_launch_pass_rest(aR, exact, st), "propagate");
            } else {
                aR.iter = iter;
                aR.theta = theta;
                aR.old = ctx->S[1][sw]; aR.out = ctx->S[1][1 - sw]; aR.smooth = ctx->smooth[1];
                if ((s = propagate_view(ctx, aR, exact, redblack, n, st)) != CVTPM_OK) return s;
            }
            tm.stop();
        }
        ctx->stats.propagate_launches += 2;
        LK(pm_launch_view_list(ctx->S[1][1 - sw], W, H, ctx->list[1], st), "view list");
        const float lambda = theta * p.thetascale + 5.0f;
        /* :228-261.  The right view's consistency, fill and smoother need only
         * this iteration's planes and write only smooth[1] and scratch of
         * their own, so they run on the side stream beside the left view's and
         * the next left pass.  The next right pass waits for them (side_join). */
        CK(cudaEventRecord(ctx->side_fork, st), "fork");
        CK(cudaStreamWaitEvent(ctx->side, ctx->side_fork, 0), "fork");
        for (int v = 1; v >= 0; --v) {
            NvtxRange r(v == 0 ? "consistency, fill, PD left" : "consistency, fill, PD right");
            cudaStream_t sv = v == 0 ? st : ctx->side;
            float4* const t1 = v == 0 ? ctx->tmp : ctx->tmpR;
            float4* const t2 = v == 0 ? ctx->tmp2 : ctx->tmp2R;
            LK(pm_launch_consistency(ctx->S[v][1 - sw], ctx->S[1 - v][1 - sw], W, H, p.maxdispdiff, p.maxanglediff,
                                     v == 0 ? 1 : 0, t1, nullptr, sv), "consistency");
            LK(pm_launch_fill_state(t1, W, H, dmax, v == 0 ? 1 : 0, t2, sv), "fill");
            if ((s = pd_apply(ctx, ctx->smooth[v], t2, ctx->wgt[v], lambda, p.pd_iterations, W, H, sv, nullptr, v)) != CVTPM_OK)
                return s;
            if (v == 1) {
                if (overlap && iter + 1 < last && (s = right_own(iter + 1, next)) != CVTPM_OK) return s;
                CK(cudaEventRecord(ctx->side_join, ctx->side), "join");
            }
        }
        theta = next;
    }
    if (last > first) CK(cudaStreamWaitEvent(st, ctx->side_join, 0), "join");
    if (save) {
        const int sw = last & 1;
        for (int v = 0; v < 2; ++v) {
            CK(cudaMemcpyAsync(save->states + (size_t)v * 4 * n, ctx->S[v][sw], n * 16, cudaMemcpyDeviceToDevice, st), "save");
            CK(cudaMemcpyAsync(save->smooth + (size_t)v * 4 * n, ctx->smooth[v], n * 16, cudaMemcpyDeviceToDevice, st), "save");
        }
        save->iteration = last;
    }
    if (!finish) return CVTPM_OK;
    const int fin = 1 - ((N - 1) & 1);                              /* :268-290 */
    NvtxRange fr("final consistency and fill");
    LK(pm_launch_consistency(ctx->S[0][fin], ctx->S[1][fin], W, H, p.maxdispdiff, p.maxanglediff, 1, ctx->tmp,
                             ctx->valid, st), "consistency");
    LK(pm_launch_fill_output(ctx->tmp, W, H, dscale, dmap, dpitch / 4, (float4*)nmap, npitch / 16, st), "fill output");
    if (trace) {
        if (trace->winners) {
            CK(cudaMemcpyAsync(trace->winners, ctx->win[0], n, cudaMemcpyDeviceToDevice, st), "trace");
            CK(cudaMemcpyAsync(trace->winners + n, ctx->win[1], n, cudaMemcpyDeviceToDevice, st), "trace");
        }
        if (trace->valid) CK(cudaMemcpyAsync(trace->valid, ctx->valid, n, cudaMemcpyDeviceToDevice, st), "trace");
        if (trace->states) {
            CK(cudaMemcpyAsync(trace->states, ctx->S[0][fin], n * 16, cudaMemcpyDeviceToDevice, st), "trace");
            CK(cudaMemcpyAsync(trace->states + 4 * n, ctx->S[1][fin], n * 16, cudaMemcpyDeviceToDevice, st), "trace");
        }
    }
    return CVTPM_OK;
}

/* PMHuberStereo::depthMapInpaint, PMHuberStereo.cpp:293-506: the depthMap
 * schedule with the occlusion-masked smoother (PDROFInpaint, 100 steps,
 * lambda = 20*theta + 5, :442-480), theta ramped from iteration 4 (:481-482),
 * the final check on state buffer 1 whatever the iteration count
 * (clmatches[1], :491-496) with 1 px / 5 degrees, and the disparity in
 * pixels (scale 1, :503).  trace->states: the last propagation outputs. */
cvtpm_status run_depthmap_inpaint(cvtpm_ctx* ctx, const cvtpm_params& p, float* dmap, size_t dpitch,
                                  const float* left, const float* right, int W, int H, size_t pitch,
                                  const cvtpm_trace* trace, cudaStream_t st) {
    cvtpm_status s;
    if ((s = check_params(ctx, p)) != CVTPM_OK) return s;
    if ((s = check_image(ctx, left, W, H, pitch, "left")) != CVTPM_OK) return s;
    if ((s = check_image(ctx, right, W, H, pitch, "right")) != CVTPM_OK) return s;
    if (!dmap) return fail(ctx, CVTPM_ERR_INVALID_ARGUMENT, "dmap is NULL");
    if (dpitch % 4 != 0 || dpitch < (size_t)W * 4) return fail(ctx, CVTPM_ERR_INVALID_ARGUMENT, "dmap pitch");
    CK(cudaSetDevice(ctx->device), "cudaSetDevice");
    if ((s = ensure_buffers(ctx, W, H)) != CVTPM_OK) return s;
    if ((s = ensure_tables(ctx, p, st)) != CVTPM_OK) return s;
    if ((s = prep_views(ctx, p, left, right, W, H, pitch, st)) != CVTPM_OK) return s;
    const size_t n = (size_t)W * H;
    const bool exact = p.arith == CVTPM_ARITH_EXACT;
    const float dmax = p.depthmax;
    const int N = p.iterations;
    PmPassArgs aL = base_args(ctx, p, W, H, 0), aR = base_args(ctx, p, W, H, 1);
    bool overlap = false;                                          /* not used: one stream here */
    if ((s = plan_pass(ctx, p, W, H, true, st, &aL, &aR, &overlap)) != CVTPM_OK) return s;
    if (!ctx->dcount) {
        if (ctx->no_alloc) return fail(ctx, CVTPM_ERR_ALLOC, "counters not allocated before capture");
        CK(cudaMalloc(&ctx->dcount, 2 * sizeof(unsigned long long)), "counters");
        CK(cudaMemset(ctx->dcount, 0, 2 * sizeof(unsigned long long)), "counters");
    }
    ++ctx->stats.calls;
    aL.out = ctx->S[0][0];                                         /* :345-363 */
    LK(pm_launch_init(aL, exact, st), "init");
    aR.out = ctx->S[1][0];
    LK(pm_launch_init(aR, exact, st), "init");
    CK(cudaMemsetAsync(ctx->smooth[0], 0, n * 16, st), "clear");   /* :330-336 */
    CK(cudaMemsetAsync(ctx->smooth[1], 0, n * 16, st), "clear");
    CK(clear_view_list(ctx->list[1], W, H, st), "clear");   /* :365-369 */
    float theta = 0.0f;
    for (int iter = 0; iter < N; ++iter) {                         /* :371-483 */
        const int sw = iter & 1;
        aL.iter = aR.iter = iter;
        aL.theta = aR.theta = theta;
        aL.old = ctx->S[0][sw]; aL.out = ctx->S[0][1 - sw]; aL.smooth = ctx->smooth[0];
        aL.viewin = ctx->list[1]; aL.viewsrc = ctx->S[1][sw]; aL.winners = ctx->win[0];
        aL.counters = aR.counters = ctx->dcount;
        {
            NvtxRange r("propagate left");
            PhaseTimer tm(ctx, st, ctx->ev_prop);
            if ((s = propagate_view(ctx, aL, exact, p.schedule == CVTPM_SCHEDULE_REDBLACK, n, st)) != CVTPM_OK) return s;
            tm.stop();
        }
        LK(pm_launch_view_list(ctx->S[0][1 - sw], W, H, ctx->list[0], st), "view list");
        aR.old = ctx->S[1][sw]; aR.out = ctx->S[1][1 - sw]; aR.smooth = ctx->smooth[1];
        aR.viewin = ctx->list[0]; aR.viewsrc = ctx->S[0][1 - sw]; aR.winners = ctx->win[1];
        {
            NvtxRange r("propagate right");
            PhaseTimer tm(ctx, st, ctx->ev_prop);
            if ((s = propagate_view(ctx, aR, exact, p.schedule == CVTPM_SCHEDULE_REDBLACK, n, st)) != CVTPM_OK) return s;
            tm.stop();
        }
        ctx->stats.propagate_launches += 2;
        LK(pm_launch_view_list(ctx->S[1][1 - sw], W, H, ctx->list[1], st), "view list");
        const float lambda = theta * 20.0f + 5.0f;
        for (int v = 0; v < 2; ++v) {                              /* :442-480 */
            const int lr = v == 0 ? 1 : 0;
            LK(pm_launch_occmap(ctx->S[v][1 - sw], ctx->S[1 - v][1 - sw], W, H, 0.5f, lr, ctx->occ, st), "occmap");
            LK(pm_launch_normal_depth(ctx->S[v][1 - sw], W, H, dmax, lr, ctx->tmp2, st), "normal depth");
            if ((s = pd_apply(ctx, ctx->smooth[v], ctx->tmp2, ctx->wgt[v], lambda, 100, W, H, st, ctx->occ)) != CVTPM_OK)
                return s;
        }
        if (iter >= 4) theta = smoothstep01(((float)iter - 4.0f) / ((float)N - 4.0f)) * 1.0f;
    }
    LK(pm_launch_consistency(ctx->S[0][1], ctx->S[1][1], W, H, 1.0f, 5.0f, 1, ctx->tmp, ctx->valid, st),
       "consistency");
    LK(pm_launch_fill_output(ctx->tmp, W, H, 1.0f, dmap, dpitch / 4, nullptr, 0, st), "fill output");
    if (trace) {
        const int fin = 1 - ((N - 1) & 1);
        if (trace->winners) {
            CK(cudaMemcpyAsync(trace->winners, ctx->win[0], n, cudaMemcpyDeviceToDevice, st), "trace");
            CK(cudaMemcpyAsync(trace->winners + n, ctx->win[1], n, cudaMemcpyDeviceToDevice, st), "trace");
        }
        if (trace->valid) CK(cudaMemcpyAsync(trace->valid, ctx->valid, n, cudaMemcpyDeviceToDevice, st), "trace");
        if (trace->states) {
            CK(cudaMemcpyAsync(trace->states, ctx->S[0][fin], n * 16, cudaMemcpyDeviceToDevice, st), "trace");
            CK(cudaMemcpyAsync(trace->states + 4 * n, ctx->S[1][fin], n * 16, cudaMemcpyDeviceToDevice, st), "trace");
        }
    }
    return CVTPM_OK;
}

}  // namespace


/* ====================================================== public API === */
extern "C" {

const char* cvtpm_version(void) { return CVTPM_VERSION; }

const char* cvtpm_status_string(cvtpm_status s) {
    switch (s) {
        case CVTPM_OK: return "ok";
        case CVTPM_ERR_INVALID_ARGUMENT: return "invalid argument";
        case CVTPM_ERR_SIZE: return "size out of range";
        case CVTPM_ERR_INCONSISTENT: return "left/right images inconsistent";
        case CVTPM_ERR_CUDA: return "CUDA error";
        case CVTPM_ERR_ALLOC: return "device allocation failed";
        case CVTPM_ERR_TIMEOUT: return "device wait timed out";
        case CVTPM_ERR_NOT_SUPPORTED: return "not supported";
        case CVTPM_ERR_IO: return "file error";
    }
    return "unknown status";
}

cvtpm_status cvtpm_params_default(cvtpm_params* p, int preset) {
    if (!p) return CVTPM_ERR_INVALID_ARGUMENT;
    memset(p, 0, sizeof(*p));
    p->patchsize = 17;
    p->depthmax = 64.0f;
    p->iterations = 3;
    p->viewsamples = 4;
    p->dscale = -1.0f;
    p->maxdispdiff = 0.5f;
    p->maxanglediff = 10.0f;
    p->thetascale = 50.0f;
    p->pd_iterations = 250;
    p->color_weight = 26.0f;
    p->color_alpha = 0.05f;
    p->color_maxdiff = 0.04f;
    p->grad_maxdiff = 0.01f;
    p->weight_profile = CVTPM_PROFILE_SMOOTHSTEP;
    p->rng = CVTPM_RNG_MWC64X;
    p->seed = 0;
    p->arith = CVTPM_ARITH_EXACT;
    p->schedule = CVTPM_SCHEDULE_JACOBI;
    if (preset == CVTPM_PRESET_BASELINE) {
        p->color_weight = 25.5f;
        p->weight_profile = CVTPM_PROFILE_CONSTANT;
        p->color_alpha = 0.1f;
        p->color_maxdiff = 10.0f / 255.0f;
        p->grad_maxdiff = 2.0f / 255.0f;
        p->rng = CVTPM_RNG_PHILOX;
        p->seed = 0x5EED0000CAFEull;
        p->arith = CVTPM_ARITH_FAST;
    } else if (preset != CVTPM_PRESET_REFERENCE) {
        return CVTPM_ERR_INVALID_ARGUMENT;
    }
    return CVTPM_OK;
}

cvtpm_status cvtpm_create(cvtpm_ctx** out, int device) {
    if (!out) return CVTPM_ERR_INVALID_ARGUMENT;
    *out = nullptr;
    int n = 0;
    cudaError_t e = cudaGetDeviceCount(&n);
    if (e != cudaSuccess) return CVTPM_ERR_CUDA;
    if (device < 0 || device >= n) return CVTPM_ERR_INVALID_ARGUMENT;
    cvtpm_ctx* c = new (std::nothrow) cvtpm_ctx();
    if (!c) return CVTPM_ERR_ALLOC;
    c->device = device;
    cvtpm_params_default(&c->prm, CVTPM_PRESET_REFERENCE);
    {
        static std::mutex mu;
        static std::vector<int> prepared;
        std::lock_guard<std::mutex> lk(mu);
        bool done = false;
        for (int d : prepared) done |= d == device;
        if (!done) {
            if (cudaSetDevice(device) != cudaSuccess || pm_prepare_kernels() != cudaSuccess) {
                delete c;
                return CVTPM_ERR_CUDA;
            }
            prepared.push_back(device);
        }
    }
    *out = c;
    return CVTPM_OK;
}

cvtpm_status cvtpm_destroy(cvtpm_ctx* ctx) {
    if (!ctx) return CVTPM_ERR_INVALID_ARGUMENT;
    cudaSetDevice(ctx->device);
    if (ctx->pool) cudaFree(ctx->pool);
    if (ctx->bexec) cudaGraphExecDestroy(ctx->bexec);
    for (cvtpm_ctx* c : ctx->bpairs) cvtpm_destroy(c);
    for (auto& l : ctx->lanes) {
        if (l.c) cvtpm_destroy(l.c);
        if (l.s) cudaStreamDestroy(l.s);
        if (l.done) cudaEventDestroy(l.done);
    }
    if (ctx->side) cudaStreamDestroy(ctx->side);
    if (ctx->side_fork) cudaEventDestroy(ctx->side_fork);
    if (ctx->side_join) cudaEventDestroy(ctx->side_join);
    if (ctx->bstream) cudaStreamDestroy(ctx->bstream);
    if (ctx->bfork) cudaEventDestroy(ctx->bfork);
    if (ctx->bjoin) cudaEventDestroy(ctx->bjoin);
    if (ctx->stage) cudaFree(ctx->stage);
    if (ctx->pass) cudaFree(ctx->pass);
    if (ctx->istage) cudaFree(ctx->istage);
    if (ctx->dcount) cudaFree(ctx->dcount);
    for (auto& pr : ctx->ev_prop) { cudaEventDestroy(pr.first); cudaEventDestroy(pr.second); }
    for (auto& pr : ctx->ev_pd) { cudaEventDestroy(pr.first); cudaEventDestroy(pr.second); }
    for (auto e : ctx->ev_free) cudaEventDestroy(e);
    delete ctx;
    return CVTPM_OK;
}

cvtpm_status cvtpm_set_params(cvtpm_ctx* ctx, const cvtpm_params* p) {
    if (!ctx || !p) return CVTPM_ERR_INVALID_ARGUMENT;
    cvtpm_status s = check_params(ctx, *p);
    if (s != CVTPM_OK) return s;
    ctx->prm = *p;
    return CVTPM_OK;
}

cvtpm_status cvtpm_get_params(const cvtpm_ctx* ctx, cvtpm_params* p) {
    if (!ctx || !p) return CVTPM_ERR_INVALID_ARGUMENT;
    *p = ctx->prm;
    return CVTPM_OK;
}

const char* cvtpm_last_error(const cvtpm_ctx* ctx) { return ctx ? ctx->err.c_str() : pm_free_error(); }

cvtpm_status cvtpm_synchronize(cvtpm_ctx* ctx, void* stream) {
    if (!ctx) return CVTPM_ERR_INVALID_ARGUMENT;
    CK(cudaStreamSynchronize((cudaStream_t)stream), "synchronize");
    return CVTPM_OK;
}

cvtpm_status cvtpm_depthmap(cvtpm_ctx* ctx, float* dmap, size_t dmap_pitch, const float* left, const float* right,
                            int width, int height, size_t pitch, int patchsize, float depthmax, int iterations,
                            int viewsamples, float dscale, float* normalmap, size_t normalmap_pitch,
                            const cvtpm_trace* trace, void* stream) {
    if (!ctx) return CVTPM_ERR_INVALID_ARGUMENT;
    (void)viewsamples;   /* ignored, as in the reference (4 slots, pmhstereo.cl:40) */
    cvtpm_params p = ctx->prm;
    p.patchsize = patchsize;
    p.depthmax = depthmax;
    p.iterations = iterations;
    p.dscale = dscale;
    return run_depthmap(ctx, p, dmap, dmap_pitch, left, right, width, height, pitch, normalmap, normalmap_pitch,
                        trace, (cudaStream_t)stream);
}

cvtpm_status cvtpm_depthmap_resumable(cvtpm_ctx* ctx, float* dmap, size_t dmap_pitch, const float* left,
                                      const float* right, int width, int height, size_t pitch, int patchsize,
                                      float depthmax, int iterations, int viewsamples, float dscale, float* normalmap,
                                      size_t normalmap_pitch, const cvtpm_trace* trace,
                                      const cvtpm_checkpoint* resume, int stop, cvtpm_checkpoint* save,
                                      void* stream) {
    if (!ctx) return CVTPM_ERR_INVALID_ARGUMENT;
    (void)viewsamples;
    cvtpm_params p = ctx->prm;
    p.patchsize = patchsize;
    p.depthmax = depthmax;
    p.iterations = iterations;
    p.dscale = dscale;
    return run_depthmap(ctx, p, dmap, dmap_pitch, left, right, width, height, pitch, normalmap, normalmap_pitch, trace,
                        (cudaStream_t)stream, resume, stop, save);
}

cvtpm_status cvtpm_depthmap_image(cvtpm_ctx* ctx, float* dmap, size_t dmap_pitch, const cvtpm_image* left,
                                  const cvtpm_image* right, int patchsize, float depthmax, int iterations,
                                  int viewsamples, float dscale, float* normalmap, size_t normalmap_pitch,
                                  const cvtpm_trace* trace, void* stream) {
    if (!ctx) return CVTPM_ERR_INVALID_ARGUMENT;
    if (!left || !right) return fail(ctx, CVTPM_ERR_INVALID_ARGUMENT, "left or right descriptor is NULL");
    /* PMHuberStereo.cpp:66-68: sizes must agree; formats may differ */
    if (left->width != right->width || left->height != right->height)
        return fail(ctx, CVTPM_ERR_INCONSISTENT, "Left/Right stereo images inconsistent");
    if (left->width < 1 || left->height < 1) return fail(ctx, CVTPM_ERR_SIZE, "empty image");
    CK(cudaSetDevice(ctx->device), "cudaSetDevice");
    const int W = left->width, H = left->height;
    const size_t pitch = (size_t)W * 16, need = 2 * pitch * (size_t)H;
    cudaStream_t st = (cudaStream_t)stream;
    if (ctx->istage_bytes < need) {
        if (ctx->istage) {
            CK(cudaStreamSynchronize(st), "image staging");
            CK(cudaFree(ctx->istage), "free image staging");
            ctx->istage = nullptr;
            ctx->istage_bytes = 0;
        }
        if (cudaMalloc(&ctx->istage, need) != cudaSuccess) {
            cudaGetLastError();
            ctx->istage = nullptr;
            return fail(ctx, CVTPM_ERR_ALLOC, "image staging allocation failed");
        }
        ctx->istage_bytes = need;
    }
    float4* l = (float4*)ctx->istage;
    float4* r = (float4*)((char*)ctx->istage + pitch * (size_t)H);
    std::string msg;
    cvtpm_status s;
    if ((s = pm_image_to_rgbaf_checked(left, "left", l, pitch, st, &msg)) != CVTPM_OK) return fail(ctx, s, msg);
    if ((s = pm_image_to_rgbaf_checked(right, "right", r, pitch, st, &msg)) != CVTPM_OK) return fail(ctx, s, msg);
    ctx->stats.launches += 2;
    return cvtpm_depthmap(ctx, dmap, dmap_pitch, (const float*)l, (const float*)r, W, H, pitch, patchsize, depthmax,
                          iterations, viewsamples, dscale, normalmap, normalmap_pitch, trace, stream);
}

cvtpm_status cvtpm_depthmap_inpaint(cvtpm_ctx* ctx, float* dmap, size_t dmap_pitch, const float* left,
                                    const float* right, int width, int height, size_t pitch, int patchsize,
                                    float depthmax, int iterations, int viewsamples, const cvtpm_trace* trace,
                                    void* stream) {
    if (!ctx) return CVTPM_ERR_INVALID_ARGUMENT;
    (void)viewsamples;
    cvtpm_params p = ctx->prm;
    p.patchsize = patchsize;
    p.depthmax = depthmax;
    p.iterations = iterations;
    return run_depthmap_inpaint(ctx, p, dmap, dmap_pitch, left, right, width, height, pitch, trace,
                                (cudaStream_t)stream);
}

cvtpm_status cvtpm_depthmap_host(cvtpm_ctx* ctx, float* dmap, size_t dmap_pitch, const float* left,
                                 const float* right, int width, int height, size_t pitch, int patchsize,
                                 float depthmax, int iterations, int viewsamples, float dscale, float* normalmap,
                                 size_t normalmap_pitch, void* stream) {
    if (!ctx) return CVTPM_ERR_INVALID_ARGUMENT;
    if (!left || !right || !dmap) return fail(ctx, CVTPM_ERR_INVALID_ARGUMENT, "null host pointer");
    if (width < 1 || height < 1 || width > PM_MAX_WIDTH || height > 65535) return fail(ctx, CVTPM_ERR_SIZE, "image size out of range");
    if (pitch < (size_t)width * 16 || dmap_pitch < (size_t)width * 4) return fail(ctx, CVTPM_ERR_INVALID_ARGUMENT, "pitch");
    if (normalmap && normalmap_pitch < (size_t)width * 16) return fail(ctx, CVTPM_ERR_INVALID_ARGUMENT, "normalmap pitch");
    cudaStream_t st = (cudaStream_t)stream;
    CK(cudaSetDevice(ctx->device), "cudaSetDevice");
    const size_t n = (size_t)width * height;
    const size_t need = n * 16 * 2 + n * 4 + (normalmap ? n * 16 : 0) + 1024;
    if (need > ctx->stage_bytes) {
        if (ctx->stage) { cudaFree(ctx->stage); ctx->stage = nullptr; ctx->stage_bytes = 0; }
        cudaError_t e = cudaMalloc(&ctx->stage, need);
        if (e != cudaSuccess) { ctx->stage = nullptr; return fail(ctx, CVTPM_ERR_ALLOC, "staging allocation"); }
        ctx->stage_bytes = need;
    }
    float* dL = (float*)ctx->stage;
    float* dR = dL + n * 4;
    float* dD = dR + n * 4;
    float* dN = normalmap ? (float*)((char*)ctx->stage + align_up((n * 16 * 2 + n * 4), 256)) : nullptr;
    const size_t row = (size_t)width * 16;
    CK(cudaMemcpy2DAsync(dL, row, left, pitch, row, height, cudaMemcpyHostToDevice, st), "H2D left");
    CK(cudaMemcpy2DAsync(dR, row, right, pitch, row, height, cudaMemcpyHostToDevice, st), "H2D right");
    cvtpm_status s = cvtpm_depthmap(ctx, dD, (size_t)width * 4, dL, dR, width, height, row, patchsize, depthmax,
                                    iterations, viewsamples, dscale, dN, row, nullptr, stream);
    if (s != CVTPM_OK) return s;
    CK(cudaMemcpy2DAsync(dmap, dmap_pitch, dD, (size_t)width * 4, (size_t)width * 4, height, cudaMemcpyDeviceToHost, st), "D2H dmap");
    if (normalmap)
        CK(cudaMemcpy2DAsync(normalmap, normalmap_pitch, dN, row, row, height, cudaMemcpyDeviceToHost, st), "D2H normalmap");
    CK(cudaStreamSynchronize(st), "synchronize");
    return CVTPM_OK;
}

cvtpm_status cvtpm_cost_eval(cvtpm_ctx* ctx, const float* img1, const float* img2, int width, int height,
                             size_t pitch, const float* states, int lr, float* cost, void* stream) {
    if (!ctx) return CVTPM_ERR_INVALID_ARGUMENT;
    cvtpm_status s;
    const cvtpm_params& p = ctx->prm;
    if ((s = check_params(ctx, p)) != CVTPM_OK) return s;
    if ((s = check_image(ctx, img1, width, height, pitch, "img1")) != CVTPM_OK) return s;
    if ((s = check_image(ctx, img2, width, height, pitch, "img2")) != CVTPM_OK) return s;
    if (!states || ((uintptr_t)states & 15))
        return fail(ctx, CVTPM_ERR_INVALID_ARGUMENT, "states NULL or not 16-byte aligned");
    if (!cost || ((uintptr_t)cost & 3)) return fail(ctx, CVTPM_ERR_INVALID_ARGUMENT, "cost NULL or not 4-byte aligned");
    (void)lr;   /* the cost does not depend on the view flag (pmhstereo.cl:170-228) */
    cudaStream_t st = (cudaStream_t)stream;
    CK(cudaSetDevice(ctx->device), "cudaSetDevice");
    if ((s = ensure_buffers(ctx, width, height)) != CVTPM_OK) return s;
    if ((s = ensure_tables(ctx, p, st)) != CVTPM_OK) return s;
    if ((s = prep_views(ctx, p, img1, img2, width, height, pitch, st)) != CVTPM_OK) return s;
    PmPassArgs a = base_args(ctx, p, width, height, 0);
    LK(pm_launch_cost_field(a, p.arith == CVTPM_ARITH_EXACT, (const float4*)states, cost, st), "cost field");
    return CVTPM_OK;
}

cvtpm_status cvtpm_set_memory_budget(cvtpm_ctx* ctx, size_t bytes) {
    if (!ctx) return CVTPM_ERR_INVALID_ARGUMENT;
    if (bytes != ctx->pass_budget) ctx->pass_pixels = 0;   /* the next call may size the scratch anew */
    ctx->pass_budget = bytes;
    if (ctx->pass && ctx->pass_bytes > bytes) {
        CK(cudaSetDevice(ctx->device), "cudaSetDevice");
        CK(cudaFree(ctx->pass), "free pass scratch");
        ctx->pass = nullptr;
        ctx->pass_bytes = 0;
    }
    return CVTPM_OK;
}

cvtpm_status cvtpm_polish_planes(cvtpm_ctx* ctx, const float* img1, const float* img2, int width, int height,
                                 size_t pitch, float* planes, int lr, int steps, float* cost, void* stream) {
    if (!ctx) return CVTPM_ERR_INVALID_ARGUMENT;
    cvtpm_status s;
    const cvtpm_params& p = ctx->prm;
    if ((s = check_params(ctx, p)) != CVTPM_OK) return s;
    if ((s = check_image(ctx, img1, width, height, pitch, "img1")) != CVTPM_OK) return s;
    if ((s = check_image(ctx, img2, width, height, pitch, "img2")) != CVTPM_OK) return s;
    if (!planes || ((uintptr_t)planes & 15)) return fail(ctx, CVTPM_ERR_INVALID_ARGUMENT, "planes NULL or not 16-byte aligned");
    if (steps < 0) return fail(ctx, CVTPM_ERR_INVALID_ARGUMENT, "steps must be >= 0");
    cudaStream_t st = (cudaStream_t)stream;
    CK(cudaSetDevice(ctx->device), "cudaSetDevice");
    if ((s = ensure_buffers(ctx, width, height)) != CVTPM_OK) return s;
    if ((s = ensure_tables(ctx, p, st)) != CVTPM_OK) return s;
    if ((s = prep_views(ctx, p, img1, img2, width, height, pitch, st, true)) != CVTPM_OK) return s;
    const PmPassArgs a = base_args(ctx, p, width, height, 0);
    LK(pm_launch_gn_polish(a.k, a.v1, a.v2, (float4*)planes, lr, steps, cost, st), "plane polishing");
    return CVTPM_OK;
}

cvtpm_status cvtpm_set_timing(cvtpm_ctx* ctx, int enable) {
    if (!ctx) return CVTPM_ERR_INVALID_ARGUMENT;
    ctx->timing = enable != 0;
    return CVTPM_OK;
}

static cvtpm_status drain_events(cvtpm_ctx* ctx, std::vector<std::pair<cudaEvent_t, cudaEvent_t>>& list, float* acc) {
    for (auto& pr : list) {
        CK(cudaEventSynchronize(pr.second), "event");
        float ms = 0.0f;
        CK(cudaEventElapsedTime(&ms, pr.first, pr.second), "event");
        *acc += ms;
        ctx->ev_free.push_back(pr.first);
        ctx->ev_free.push_back(pr.second);
    }
    list.clear();
    return CVTPM_OK;
}

cvtpm_status cvtpm_reset_stats(cvtpm_ctx* ctx) {
    if (!ctx) return CVTPM_ERR_INVALID_ARGUMENT;
    CK(cudaSetDevice(ctx->device), "cudaSetDevice");
    CK(cudaDeviceSynchronize(), "synchronize");
    float dummy = 0.0f;
    cvtpm_status s;
    if ((s = drain_events(ctx, ctx->ev_prop, &dummy)) != CVTPM_OK) return s;
    if ((s = drain_events(ctx, ctx->ev_pd, &dummy)) != CVTPM_OK) return s;
    if (ctx->dcount) CK(cudaMemset(ctx->dcount, 0, 2 * sizeof(unsigned long long)), "counters");
    memset(&ctx->stats, 0, sizeof(ctx->stats));
    return CVTPM_OK;
}

cvtpm_status cvtpm_get_stats(cvtpm_ctx* ctx, cvtpm_stats* out) {
    if (!ctx || !out) return CVTPM_ERR_INVALID_ARGUMENT;
    CK(cudaSetDevice(ctx->device), "cudaSetDevice");
    CK(cudaDeviceSynchronize(), "synchronize");
    cvtpm_status s;
    if ((s = drain_events(ctx, ctx->ev_prop, &ctx->stats.propagate_ms)) != CVTPM_OK) return s;
    if ((s = drain_events(ctx, ctx->ev_pd, &ctx->stats.pd_ms)) != CVTPM_OK) return s;
    if (ctx->dcount) {
        unsigned long long c[2];
        CK(cudaMemcpy(c, ctx->dcount, sizeof(c), cudaMemcpyDeviceToHost), "counters");
        ctx->stats.cost_evals = c[0];
        ctx->stats.cost_taps = c[1];
    }
    *out = ctx->stats;
    return CVTPM_OK;
}

cvtpm_status cvtpm_cost_adjoint(cvtpm_ctx* ctx, const float* img1, const float* img2, int width, int height,
                                size_t pitch, const float* planes, int lr, const float* dcost, float* cost,
                                float* dplanes, float* dimg1, float* dimg2, void* stream) {
    if (!ctx) return CVTPM_ERR_INVALID_ARGUMENT;
    cvtpm_status s;
    const cvtpm_params& p = ctx->prm;
    if ((s = check_params(ctx, p)) != CVTPM_OK) return s;
    if ((s = check_image(ctx, img1, width, height, pitch, "img1")) != CVTPM_OK) return s;
    if ((s = check_image(ctx, img2, width, height, pitch, "img2")) != CVTPM_OK) return s;
    if (!planes) return fail(ctx, CVTPM_ERR_INVALID_ARGUMENT, "null planes");
    if (((uintptr_t)planes & 15) || ((uintptr_t)dplanes & 15))
        return fail(ctx, CVTPM_ERR_INVALID_ARGUMENT, "planes/dplanes must be 16-byte aligned");
    if (!dcost && (dplanes || dimg1 || dimg2))
        return fail(ctx, CVTPM_ERR_INVALID_ARGUMENT, "gradients requested without dcost");
    cudaStream_t st = (cudaStream_t)stream;
    CK(cudaSetDevice(ctx->device), "cudaSetDevice");
    if ((s = ensure_buffers(ctx, width, height)) != CVTPM_OK) return s;
    if ((s = ensure_tables(ctx, p, st)) != CVTPM_OK) return s;
    if ((s = prep_views(ctx, p, img1, img2, width, height, pitch, st, true)) != CVTPM_OK) return s;
    const PmPassArgs a = base_args(ctx, p, width, height, 0);
    /* the four image-adjoint accumulators reuse the propagation state buffers */
    const bool img = dimg1 || dimg2;
    const size_t n = (size_t)width * height;
    float4 *dI1 = ctx->S[0][0], *dG1 = ctx->S[0][1], *dI2 = ctx->S[1][0], *dG2 = ctx->S[1][1];
    if (img) {
        for (float4* b : {dI1, dG1, dI2, dG2}) CK(cudaMemsetAsync(b, 0, n * 16, st), "adjoint clear");
    }
    float* sums = nullptr;
    if (pm_tap_adjoint(a.k, dcost != nullptr, img)) {    /* small images: costs and weight sums first, into free scratch */
        sums = (float*)ctx->smooth[0];
        if (!cost) cost = (float*)ctx->smooth[1];
        LK(pm_launch_plane_sums(a, (const float4*)planes, lr, cost, sums, st), "plane sums");
    }
    if (!sums || dcost)
        LK(pm_launch_cost_adjoint(a.k, a.v1, a.v2, (const float4*)planes, lr, dcost, cost, (float4*)dplanes,
                                  img ? dI1 : nullptr, dG1, dI2, dG2, sums, st), "cost adjoint");
    if (dimg1) LK(pm_launch_adjoint_finish(dI1, dG1, width, height, dimg1, st), "adjoint image 1");
    if (dimg2) LK(pm_launch_adjoint_finish(dI2, dG2, width, height, dimg2, st), "adjoint image 2");
    return CVTPM_OK;
}

/* ---------------------------------------------------------- batched -- */
namespace {

cvtpm_status check_pair(cvtpm_ctx* ctx, const cvtpm_pair& q, int i) {
    const std::string w = "pair " + std::to_string(i);
    cvtpm_status s;
    if ((s = check_image(ctx, q.left, q.width, q.height, q.pitch, (w + " left").c_str())) != CVTPM_OK) return s;
    if ((s = check_image(ctx, q.right, q.width, q.height, q.pitch, (w + " right").c_str())) != CVTPM_OK) return s;
    if (!(q.depthmax > 0.0f)) return fail(ctx, CVTPM_ERR_INVALID_ARGUMENT, w + ": depthmax must be > 0");
    if (!q.dmap || q.dmap_pitch % 4 != 0 || q.dmap_pitch < (size_t)q.width * 4)
        return fail(ctx, CVTPM_ERR_INVALID_ARGUMENT, w + ": dmap is NULL or its pitch is too small");
    return CVTPM_OK;
}

/* Lanes: each has its own context (scratch, neighbour costs, counters) and
 * stream, so the pairs of different lanes run concurrently. */
cvtpm_status ensure_lanes(cvtpm_ctx* ctx, int k) {
    while ((int)ctx->lanes.size() < k) {
        cvtpm_ctx::Lane l;
        cvtpm_status s = cvtpm_create(&l.c, ctx->device);
        if (s != CVTPM_OK) return fail(ctx, s, "lane context");
        CK(cudaStreamCreateWithFlags(&l.s, cudaStreamNonBlocking), "lane stream");
        CK(cudaEventCreateWithFlags(&l.done, cudaEventDisableTiming), "lane event");
        CK(cudaMalloc(&l.c->dcount, 2 * sizeof(unsigned long long)), "lane counters");
        CK(cudaMemset(l.c->dcount, 0, 2 * sizeof(unsigned long long)), "lane counters");
        ctx->lanes.push_back(l);
    }
    if (!ctx->bstream) {
        CK(cudaStreamCreateWithFlags(&ctx->bstream, cudaStreamNonBlocking), "batch stream");
        CK(cudaEventCreateWithFlags(&ctx->bfork, cudaEventDisableTiming), "batch event");
        CK(cudaEventCreateWithFlags(&ctx->bjoin, cudaEventDisableTiming), "batch event");
    }
    return CVTPM_OK;
}

/* Longest-processing-time assignment of pairs to k lanes (work ~ W*H). */
std::vector<std::vector<int>> assign_lanes(const cvtpm_pair* pairs, int npairs, int k) {
    std::vector<int> order(npairs);
    for (int i = 0; i < npairs; ++i) order[i] = i;
    std::stable_sort(order.begin(), order.end(), [&](int a, int b) {
        return (size_t)pairs[a].width * pairs[a].height > (size_t)pairs[b].width * pairs[b].height;
    });
    std::vector<std::vector<int>> out(k);
    std::vector<size_t> load(k, 0);
    for (int i : order) {
        int best = 0;
        for (int j = 1; j < k; ++j)
            if (load[j] < load[best]) best = j;
        out[best].push_back(i);
        load[best] += (size_t)pairs[i].width * pairs[i].height;
    }
    return out;
}

/* Captures the whole batch (every pair's depthMap schedule, lanes as
 * parallel branches) into one graph and instantiates it. */
cvtpm_status capture_batch(cvtpm_ctx* ctx, const cvtpm_pair* pairs, int npairs, int k, int iterations,
                           cudaGraphExec_t* exec, size_t* nodes) {
    cvtpm_status s;
    if ((s = ensure_lanes(ctx, k)) != CVTPM_OK) return s;
    const auto plan = assign_lanes(pairs, npairs, k);
    cvtpm_params p = ctx->prm;
    p.iterations = iterations;
    /* size every lane for its pairs and load the tables, outside the capture */
    for (int j = 0; j < k; ++j) {
        cvtpm_ctx* c = ctx->lanes[j].c;
        c->prm = p;
        if ((s = cvtpm_set_memory_budget(c, ctx->pass_budget)) != CVTPM_OK) return fail(ctx, s, c->err);
        c->timing = false;
        for (int i : plan[j]) {
            if ((s = ensure_buffers(c, pairs[i].width, pairs[i].height)) != CVTPM_OK) return fail(ctx, s, c->err);
            PmPassArgs aL, aR;
            bool overlap;
            if ((s = plan_pass(c, p, pairs[i].width, pairs[i].height, true, ctx->bstream, &aL, &aR, &overlap)) != CVTPM_OK)
                return fail(ctx, s, c->err);
        }
    }
    if (k > 0 && (s = ensure_tables(ctx->lanes[0].c, p, ctx->bstream)) != CVTPM_OK) return fail(ctx, s, ctx->lanes[0].c->err);
    CK(cudaStreamSynchronize(ctx->bstream), "batch prepare");
    std::vector<cvtpm_ctx*> lane_ctx;
    for (int j = 0; j < k; ++j) lane_ctx.push_back(ctx->lanes[j].c);
    CK(cudaStreamBeginCapture(ctx->bstream, cudaStreamCaptureModeThreadLocal), "begin capture");
    CaptureGuard guard(ctx->bstream, std::move(lane_ctx));
    cvtpm_status err = CVTPM_OK;
    std::string msg;
    auto note = [&](cvtpm_status st, const std::string& m) { if (err == CVTPM_OK && st != CVTPM_OK) { err = st; msg = m; } };
    note(cudaEventRecord(ctx->bfork, ctx->bstream) == cudaSuccess ? CVTPM_OK : CVTPM_ERR_CUDA, "fork");
    for (int j = 0; j < k && err == CVTPM_OK; ++j) {
        cvtpm_ctx::Lane& l = ctx->lanes[j];
        note(cudaStreamWaitEvent(l.s, ctx->bfork, 0) == cudaSuccess ? CVTPM_OK : CVTPM_ERR_CUDA, "fork wait");
        l.c->no_alloc = true;
        for (int i : plan[j]) {
            if (err != CVTPM_OK) break;
            const cvtpm_pair& q = pairs[i];
            cvtpm_params pq = p;
            pq.depthmax = q.depthmax;
            cvtpm_status st = run_depthmap(l.c, pq, q.dmap, q.dmap_pitch, q.left, q.right, q.width, q.height, q.pitch,
                                           nullptr, 0, nullptr, l.s);
            note(st, "pair " + std::to_string(i) + ": " + l.c->err);
        }
        l.c->no_alloc = false;
        note(cudaEventRecord(l.done, l.s) == cudaSuccess ? CVTPM_OK : CVTPM_ERR_CUDA, "join record");
        note(cudaStreamWaitEvent(ctx->bstream, l.done, 0) == cudaSuccess ? CVTPM_OK : CVTPM_ERR_CUDA, "join wait");
    }
    cudaGraph_t graph = nullptr;
    cudaError_t e = cudaStreamEndCapture(ctx->bstream, &graph);
    guard.release();
    if (err != CVTPM_OK) { if (graph) cudaGraphDestroy(graph); return fail(ctx, err, msg); }
    if (e != cudaSuccess) { if (graph) cudaGraphDestroy(graph); return cuda_fail(ctx, e, "end capture"); }
    *nodes = 0;
    cudaGraphGetNodes(graph, nullptr, nodes);
    e = cudaGraphInstantiate(exec, graph, 0);
    cudaGraphDestroy(graph);
    if (e != cudaSuccess) return cuda_fail(ctx, e, "graph instantiate");
    return CVTPM_OK;
}

/* Runs a graph on the caller's stream order (the graph lives on the batch
 * stream, which waits for `st` before and is waited on after). */
cvtpm_status launch_batch(cvtpm_ctx* ctx, cudaGraphExec_t exec, cudaStream_t st) {
    CK(cudaEventRecord(ctx->bjoin, st), "batch order");
    CK(cudaStreamWaitEvent(ctx->bstream, ctx->bjoin, 0), "batch order");
    CK(cudaGraphLaunch(exec, ctx->bstream), "graph launch");
    CK(cudaEventRecord(ctx->bjoin, ctx->bstream), "batch order");
    CK(cudaStreamWaitEvent(st, ctx->bjoin, 0), "batch order");
    return CVTPM_OK;
}

/* The autotuner: times a one-iteration proxy of the batch (one graph launch
 * each) for 1, 2, 4 and 8 lanes and keeps the fastest. */
cvtpm_status tune_batch(cvtpm_ctx* ctx, const cvtpm_pair* pairs, int npairs, int* lanes_out) {
    std::vector<int> cand;
    for (int k : {1, 2, 4, 8})
        if (k == 1 || k <= npairs) cand.push_back(k);
    cvtpm_batch_info& bi = ctx->binfo;
    bi.ncand = 0;
    float best = 0.0f;
    EventPair ev;
    CK(cudaEventCreate(&ev.a), "tune event");
    CK(cudaEventCreate(&ev.b), "tune event");
    cudaEvent_t t0 = ev.a, t1 = ev.b;
    for (size_t ci = 0; ci < cand.size(); ++ci) {
        {
            const int k = cand[ci];
            cudaGraphExec_t ex = nullptr;
            size_t nodes = 0;
            cvtpm_status s = capture_batch(ctx, pairs, npairs, k, 1, &ex, &nodes);
            if (s != CVTPM_OK) return s;
            float ms = 0.0f;
            bool ok = cudaEventRecord(t0, ctx->bstream) == cudaSuccess &&
                      cudaGraphLaunch(ex, ctx->bstream) == cudaSuccess &&
                      cudaEventRecord(t1, ctx->bstream) == cudaSuccess &&
                      cudaEventSynchronize(t1) == cudaSuccess &&
                      cudaEventElapsedTime(&ms, t0, t1) == cudaSuccess;
            cudaGraphExecDestroy(ex);
            if (!ok) return cuda_fail(ctx, cudaGetLastError(), "tuning run");
            if (bi.ncand < CVTPM_BATCH_MAX_CAND) {
                bi.cand_lanes[bi.ncand] = k;
                bi.cand_grid_mult[bi.ncand] = bi.cand_pd_rows[bi.ncand] = bi.cand_pd_halo[bi.ncand] = 0;
                bi.cand_ms[bi.ncand] = ms;
                ++bi.ncand;
            }
            if (best == 0.0f || ms < best) { best = ms; *lanes_out = k; }
        }
    }
    return CVTPM_OK;
}

}  // namespace

}  // extern "C"

/* ------------------------------------------------ phase-batched mode -- */
/* PMHuberStereo::depthMap for a batch of pairs with one launch per phase of
 * the schedule (run_depthmap's order: prep, records, init, then per
 * iteration the neighbour costs, propagation and view lists of the left
 * view, the same for the right view, and per view the consistency check, the
 * fill and the PD smoother; finally the consistency check and the output
 * fill) covering every pair.  The kernels are the plain path's tile bodies
 * behind a persistent item loop (pm_kernels.cu, "batched phases"), so every
 * pair gets the bits of its plain call.  Each pair keeps its own scratch (a
 * context of its own), sized before the graph capture. */
namespace {

cvtpm_status ensure_batch_pairs(cvtpm_ctx* ctx, int n) {
    while ((int)ctx->bpairs.size() < n) {
        cvtpm_ctx* c = nullptr;
        cvtpm_status s = cvtpm_create(&c, ctx->device);
        if (s != CVTPM_OK) return fail(ctx, s, "pair context");
        ctx->bpairs.push_back(c);
        CK(cudaMalloc(&c->dcount, 2 * sizeof(unsigned long long)), "pair counters");
        CK(cudaMemset(c->dcount, 0, 2 * sizeof(unsigned long long)), "pair counters");
    }
    return CVTPM_OK;
}

/* Builds the PmBatch of `nent` entries (make(e, args, W, H) fills entry e),
 * in launches of at most PM_BATCH_MAX entries, and launches each. */
template <typename A, typename Make, typename Launch>
cvtpm_status run_phase(cvtpm_ctx* ctx, int nent, PmBatchKernel kind, const PmBatchKnobs& kn, Make make, Launch launch,
                       const char* what, long long* launches) {
    std::unique_ptr<PmBatch<A>> b(new PmBatch<A>());
    for (int e0 = 0; e0 < nent; e0 += PM_BATCH_MAX) {
        b->n = std::min(PM_BATCH_MAX, nent - e0);
        int items = 0;
        for (int i = 0; i < b->n; ++i) {
            int W = 0, H = 0, tx = 1, tiles = 0;
            make(e0 + i, b->a[i], W, H);
            pm_batch_tiles(kind, W, H, kn, &tx, &tiles);
            b->first[i] = items;
            b->tx[i] = tx;
            items += tiles;
        }
        b->first[b->n] = items;
        CK(launch(*b), what);
        ++ctx->stats.launches;
        if (launches) ++*launches;
    }
    return CVTPM_OK;
}

struct PhaseState {
    cvtpm_ctx* ctx;
    const cvtpm_pair* pairs;
    int n;
    cvtpm_params p;
    PmBatchKnobs kn;
    cudaStream_t st;
    int maxW;
    long long launches;
    std::vector<PmPassArgs> aL, aR;
};

/* Sizes every pair's scratch and neighbour-cost buffer (outside any capture). */
cvtpm_status phase_prepare(PhaseState& S) {
    cvtpm_status s;
    if ((s = ensure_batch_pairs(S.ctx, S.n)) != CVTPM_OK) return s;
    S.maxW = 1;
    for (int i = 0; i < S.n; ++i) {
        cvtpm_ctx* c = S.ctx->bpairs[i];
        c->prm = S.p;
        c->prm.depthmax = S.pairs[i].depthmax;
        c->pass_budget = S.ctx->pass_budget;
        c->timing = false;
        if ((s = ensure_buffers(c, S.pairs[i].width, S.pairs[i].height)) != CVTPM_OK) return fail(S.ctx, s, c->err);
        PmPassArgs aL, aR;
        bool overlap;
        if ((s = plan_pass(c, c->prm, S.pairs[i].width, S.pairs[i].height, false, S.st, &aL, &aR, &overlap)) != CVTPM_OK)
            return fail(S.ctx, s, c->err);
        S.maxW = std::max(S.maxW, S.pairs[i].width);
    }
    return ensure_tables(S.ctx->bpairs[0], S.p, S.st) == CVTPM_OK ? CVTPM_OK
                                                                   : fail(S.ctx, CVTPM_ERR_CUDA, S.ctx->bpairs[0]->err);
}

/* prep, records, init and the clears: every pair ready for iteration 0 */
cvtpm_status phase_start(PhaseState& S) {
    cvtpm_ctx* ctx = S.ctx;
    const bool exact = S.p.arith == CVTPM_ARITH_EXACT;
    cvtpm_status s;
    auto pc = [&](int i) { return ctx->bpairs[i]; };
    if ((s = run_phase<PmPrepArgs>(ctx, 2 * S.n, PMB_PREP, S.kn, [&](int e, PmPrepArgs& a, int& W, int& H) {
            const int i = e >> 1, v = e & 1;
            const cvtpm_pair& q = S.pairs[i];
            W = q.width; H = q.height;
            a = {(const float4*)(v ? q.right : q.left), q.pitch / 16, W, H, pc(i)->col[v], pc(i)->grad[v], pc(i)->wgt[v]};
        }, [&](const PmBatch<PmPrepArgs>& b) { return pm_batch_prep(b, S.kn, S.st); }, "batched prep", &S.launches)) != CVTPM_OK)
        return s;
    if (!exact &&
        (s = run_phase<PmRecArgs>(ctx, 2 * S.n, PMB_RECORDS, S.kn, [&](int e, PmRecArgs& a, int& W, int& H) {
            const int i = e >> 1, v = e & 1;
            W = S.pairs[i].width; H = S.pairs[i].height;
            cvtpm_ctx* c = pc(i);
            a = {c->col[v], c->grad[v], W, H, rec_pitch(W), c->recA[v], c->recB[v], c->recC[v], c->recD[v]};
        }, [&](const PmBatch<PmRecArgs>& b) { return pm_batch_records(b, S.kn, S.st); }, "batched records", &S.launches)) != CVTPM_OK)
        return s;
    S.aL.resize(S.n);
    S.aR.resize(S.n);
    for (int i = 0; i < S.n; ++i) {
        cvtpm_ctx* c = pc(i);
        const int W = S.pairs[i].width, H = S.pairs[i].height;
        S.aL[i] = base_args(c, c->prm, W, H, 0);
        S.aR[i] = base_args(c, c->prm, W, H, 1);
        bool overlap;
        if ((s = plan_pass(c, c->prm, W, H, false, S.st, &S.aL[i], &S.aR[i], &overlap)) != CVTPM_OK) return fail(ctx, s, c->err);
        S.aL[i].counters = S.aR[i].counters = c->dcount;
        S.aL[i].out = c->S[0][0];
        S.aR[i].out = c->S[1][0];
    }
    if ((s = run_phase<PmPassArgs>(ctx, 2 * S.n, PMB_PIXEL, S.kn, [&](int e, PmPassArgs& a, int& W, int& H) {
            const int i = e >> 1;
            a = (e & 1) ? S.aR[i] : S.aL[i];
            W = a.k.W; H = a.k.H;
        }, [&](const PmBatch<PmPassArgs>& b) { return pm_batch_init(b, exact, S.kn, S.st); }, "batched init", &S.launches)) != CVTPM_OK)
        return s;
    for (int i = 0; i < S.n; ++i) {                                 /* :108-113, :145-149 */
        cvtpm_ctx* c = pc(i);
        const size_t npx = (size_t)S.pairs[i].width * S.pairs[i].height;
        CK(cudaMemsetAsync(c->smooth[0], 0, npx * 16, S.st), "clear");
        CK(cudaMemsetAsync(c->smooth[1], 0, npx * 16, S.st), "clear");
        CK(clear_view_list(c->list[1], S.pairs[i].width, S.pairs[i].height, S.st), "clear");
    }
    return CVTPM_OK;
}

/* One view's propagation pass for every pair (shared windows where the pair
 * has its cost buffer), then the view lists. */
cvtpm_status phase_propagate(PhaseState& S, std::vector<PmPassArgs>& args, short4* (*list_of)(cvtpm_ctx*),
                             const float4* (*src_of)(cvtpm_ctx*, int), int sw) {
    cvtpm_ctx* ctx = S.ctx;
    const bool exact = S.p.arith == CVTPM_ARITH_EXACT;
    cvtpm_status s;
    std::vector<int> shared, plain;
    for (int i = 0; i < S.n; ++i) (args[i].costs ? shared : plain).push_back(i);
    auto phase = [&](const std::vector<int>& of, PmBatchKernel kind, auto launch, const char* what) -> cvtpm_status {
        if (of.empty()) return CVTPM_OK;
        return run_phase<PmPassArgs>(ctx, (int)of.size(), kind, S.kn, [&](int e, PmPassArgs& a, int& W, int& H) {
                a = args[of[e]];
                W = a.k.W; H = a.k.H;
            }, [&](const PmBatch<PmPassArgs>& b) { return launch(b, exact, S.kn, S.st); }, what, &S.launches);
    };
    if ((s = phase(shared, PMB_PIXEL, pm_batch_sweep, "batched sweep")) != CVTPM_OK ||
        (s = phase(shared, PMB_PIXEL, pm_batch_views, "batched view candidates")) != CVTPM_OK ||
        (s = phase(shared, PMB_SHARE, pm_batch_share, "batched shared windows")) != CVTPM_OK ||
        (s = phase(shared, PMB_PIXEL, pm_batch_refine, "batched refinement")) != CVTPM_OK ||
        (s = phase(plain, PMB_PIXEL, pm_batch_propagate, "batched propagate")) != CVTPM_OK)
        return s;
    return run_phase<PmViewListArgs>(ctx, S.n, PMB_ROW, S.kn, [&](int e, PmViewListArgs& a, int& W, int& H) {
            cvtpm_ctx* c = ctx->bpairs[e];
            W = S.pairs[e].width; H = S.pairs[e].height;
            a = {src_of(c, sw), W, H, list_of(c)};
        }, [&](const PmBatch<PmViewListArgs>& b) { return pm_batch_view_list(b, S.maxW, S.kn, S.st); },
        "batched view list", &S.launches);
}

/* PDROF::apply (PDROF.h:50-96) of view v for every pair, kn.pd_halo steps per
 * launch; pd_apply's schedule of buffers (iters == 0 runs pd_apply per pair). */
cvtpm_status phase_pd(PhaseState& S, int v, float lambda) {
    cvtpm_ctx* ctx = S.ctx;
    cvtpm_status s;
    const int iters = S.p.pd_iterations;
    if (iters == 0) {
        for (int i = 0; i < S.n; ++i) {
            cvtpm_ctx* c = ctx->bpairs[i];
            if ((s = pd_apply(c, c->smooth[v], c->tmp2, c->wgt[v], lambda, 0, S.pairs[i].width, S.pairs[i].height, S.st)) !=
                CVTPM_OK)
                return fail(ctx, s, c->err);
            ++S.launches;
        }
        return CVTPM_OK;
    }
    const int total = iters + (iters & 1);
    const int K = S.kn.pd_halo;
    int l = 0;
    for (int done = 0; done < total; done += K, ++l) {
        const int steps = total - done < K ? total - done : K;
        if ((s = run_phase<PmPdArgs>(ctx, S.n, PMB_PD, S.kn, [&](int e, PmPdArgs& a, int& W, int& H) {
                cvtpm_ctx* c = ctx->bpairs[e];
                W = S.pairs[e].width; H = S.pairs[e].height;
                float4* U[2] = {c->smooth[v], c->pdT};
                float* Pp[2] = {c->pdP[0], c->pdP[1]};
                a.uout = U[(l + 1) & 1]; a.pout = Pp[(l + 1) & 1];
                a.uin = U[l & 1]; a.pin = Pp[l & 1];
                a.f = c->tmp2; a.wgt = c->wgt[v];
                a.pzero = l == 0 ? 1 : 0; a.nsteps = steps; a.W = W; a.H = H; a.lambda = lambda;
            }, [&](const PmBatch<PmPdArgs>& b) { return pm_batch_pd(b, S.kn, S.st); }, "batched PD", &S.launches)) != CVTPM_OK)
            return s;
    }
    if (l & 1)                                          /* the result sits in pdT */
        for (int i = 0; i < S.n; ++i) {
            cvtpm_ctx* c = ctx->bpairs[i];
            CK(cudaMemcpyAsync(c->smooth[v], c->pdT, (size_t)S.pairs[i].width * S.pairs[i].height * 16,
                               cudaMemcpyDeviceToDevice, S.st), "pd copy");
        }
    return CVTPM_OK;
}

short4* list0(cvtpm_ctx* c) { return c->list[0]; }
short4* list1(cvtpm_ctx* c) { return c->list[1]; }

/* The whole schedule for `iterations` iterations, stream-ordered on S.st. */
cvtpm_status phase_schedule(PhaseState& S, int iterations) {
    cvtpm_ctx* ctx = S.ctx;
    cvtpm_status s;
    NvtxRange whole("cvtpm depthMap batch (phase-batched)");
    if ((s = phase_start(S)) != CVTPM_OK) return s;
    float theta = 0.0f;
    const int N = iterations;
    for (int iter = 0; iter < N; ++iter) {                         /* PMHuberStereo.cpp:151-266 */
        const int sw = iter & 1;
        for (int i = 0; i < S.n; ++i) {
            cvtpm_ctx* c = ctx->bpairs[i];
            PmPassArgs& L = S.aL[i];
            L.iter = iter; L.theta = theta;
            L.old = c->S[0][sw]; L.out = c->S[0][1 - sw]; L.smooth = c->smooth[0];
            L.viewin = c->list[1]; L.viewsrc = c->S[1][sw]; L.winners = c->win[0];
        }
        if ((s = phase_propagate(S, S.aL, list0, [](cvtpm_ctx* c, int sw_) { return (const float4*)c->S[0][1 - sw_]; }, sw)) !=
            CVTPM_OK)
            return s;
        for (int i = 0; i < S.n; ++i) {
            cvtpm_ctx* c = ctx->bpairs[i];
            PmPassArgs& R = S.aR[i];
            R.iter = iter; R.theta = theta;
            R.old = c->S[1][sw]; R.out = c->S[1][1 - sw]; R.smooth = c->smooth[1];
            R.viewin = c->list[0]; R.viewsrc = c->S[0][1 - sw]; R.winners = c->win[1];
        }
        if ((s = phase_propagate(S, S.aR, list1, [](cvtpm_ctx* c, int sw_) { return (const float4*)c->S[1][1 - sw_]; }, sw)) !=
            CVTPM_OK)
            return s;
        const float lambda = theta * S.p.thetascale + 5.0f;
        for (int v = 0; v < 2; ++v) {                              /* :228-261 */
            if ((s = run_phase<PmConsArgs>(ctx, S.n, PMB_PIXEL, S.kn, [&](int e, PmConsArgs& a, int& W, int& H) {
                    cvtpm_ctx* c = ctx->bpairs[e];
                    W = S.pairs[e].width; H = S.pairs[e].height;
                    a = {c->S[v][1 - sw], c->S[1 - v][1 - sw], W, H, S.p.maxdispdiff, S.p.maxanglediff / 180.0f,
                         v == 0 ? 1 : 0, c->tmp, nullptr};
                }, [&](const PmBatch<PmConsArgs>& b) { return pm_batch_consistency(b, S.kn, S.st); }, "batched consistency",
                   &S.launches)) != CVTPM_OK)
                return s;
            if ((s = run_phase<PmFillArgs>(ctx, S.n, PMB_ROW, S.kn, [&](int e, PmFillArgs& a, int& W, int& H) {
                    cvtpm_ctx* c = ctx->bpairs[e];
                    W = S.pairs[e].width; H = S.pairs[e].height;
                    a = {c->tmp, W, H, S.pairs[e].depthmax, v == 0 ? 1 : 0, c->tmp2};
                }, [&](const PmBatch<PmFillArgs>& b) { return pm_batch_fill_state(b, S.maxW, S.kn, S.st); }, "batched fill",
                   &S.launches)) != CVTPM_OK)
                return s;
            if ((s = phase_pd(S, v, lambda)) != CVTPM_OK) return s;
        }
        if (iter >= 5) theta = smoothstep01(((float)iter - 5.0f) / ((float)N - 5.0f)) * 1.0f;
    }
    const int fin = 1 - ((N - 1) & 1);                              /* :268-290 */
    if ((s = run_phase<PmConsArgs>(ctx, S.n, PMB_PIXEL, S.kn, [&](int e, PmConsArgs& a, int& W, int& H) {
            cvtpm_ctx* c = ctx->bpairs[e];
            W = S.pairs[e].width; H = S.pairs[e].height;
            a = {c->S[0][fin], c->S[1][fin], W, H, S.p.maxdispdiff, S.p.maxanglediff / 180.0f, 1, c->tmp, c->valid};
        }, [&](const PmBatch<PmConsArgs>& b) { return pm_batch_consistency(b, S.kn, S.st); }, "batched consistency",
           &S.launches)) != CVTPM_OK)
        return s;
    return run_phase<PmOutArgs>(ctx, S.n, PMB_ROW, S.kn, [&](int e, PmOutArgs& a, int& W, int& H) {
            cvtpm_ctx* c = ctx->bpairs[e];
            const cvtpm_pair& q = S.pairs[e];
            W = q.width; H = q.height;
            const float dscale = S.p.dscale <= 0.0f ? 1.0f / q.depthmax : S.p.dscale;
            a = {c->tmp, W, H, dscale, q.dmap, q.dmap_pitch / 4, nullptr, 0};
        }, [&](const PmBatch<PmOutArgs>& b) { return pm_batch_fill_output(b, S.maxW, S.kn, S.st); }, "batched fill output",
        &S.launches);
}

/* The batch autotuner.  The knobs do not change any result, only how the
 * launches are shaped: the persistent grid of every phase (1 or 2 times the
 * blocks resident per SM, or one block per work item) and the PD smoother's
 * tile (16 or 8 rows) and steps per launch (4 or 2, also its halo width).
 * On the batch's own data (its first pairs, up to 4 Mpx, after their prep
 * and init), it times one propagation phase of the left view per grid
 * choice, then one PD apply of 8 steps of the left view per PD tile, halo
 * and grid, and keeps the fastest. */
cvtpm_status tune_phased(PhaseState& full, PmBatchKnobs* best) {
    PhaseState S = full;
    long long px = 0;
    S.n = 0;
    while (S.n < full.n && (S.n == 0 || px < 4000000)) {
        px += (long long)full.pairs[S.n].width * full.pairs[S.n].height;
        ++S.n;
    }
    cvtpm_ctx* ctx = S.ctx;
    cvtpm_batch_info& bi = ctx->binfo;
    cvtpm_status s;
    bi.ncand = 0;
    S.kn = PmBatchKnobs{1, 16, 4};
    if ((s = phase_start(S)) != CVTPM_OK) return s;
    for (int i = 0; i < S.n; ++i) {
        cvtpm_ctx* c = ctx->bpairs[i];
        PmPassArgs& L = S.aL[i];
        L.iter = 0; L.theta = 0.0f;
        L.old = c->S[0][0]; L.out = c->S[0][1]; L.smooth = c->smooth[0];
        L.viewin = c->list[1]; L.viewsrc = c->S[1][0]; L.winners = c->win[0];
    }
    EventPair ev;
    CK(cudaEventCreate(&ev.a), "tune event");
    CK(cudaEventCreate(&ev.b), "tune event");
    cudaEvent_t t0 = ev.a, t1 = ev.b;
    auto timed = [&](auto&& body, float* ms) -> cvtpm_status {
        cvtpm_status r;
        if (cudaEventRecord(t0, S.st) != cudaSuccess) return cuda_fail(ctx, cudaGetLastError(), "tune record");
        if ((r = body()) != CVTPM_OK) return r;
        if (cudaEventRecord(t1, S.st) != cudaSuccess || cudaEventSynchronize(t1) != cudaSuccess ||
            cudaEventElapsedTime(ms, t0, t1) != cudaSuccess)
            return cuda_fail(ctx, cudaGetLastError(), "tune timing");
        return CVTPM_OK;
    };
    auto add = [&](const PmBatchKnobs& k, float ms) {
        if (bi.ncand < CVTPM_BATCH_MAX_CAND) {
            bi.cand_lanes[bi.ncand] = 0;
            bi.cand_grid_mult[bi.ncand] = k.grid_mult;
            bi.cand_pd_rows[bi.ncand] = k.pd_rows;
            bi.cand_pd_halo[bi.ncand] = k.pd_halo;
            bi.cand_ms[bi.ncand] = ms;
            ++bi.ncand;
        }
    };
    PmBatchKnobs win{1, 16, 4};
    float best_ms = -1.0f;
    s = CVTPM_OK;
    for (int g : {1, 2, 0}) {                             /* the propagation's grid */
        S.kn = PmBatchKnobs{g, 16, 4};
        float ms = 0.0f;
        s = timed([&] { return phase_propagate(S, S.aL, list0, [](cvtpm_ctx* c, int) { return (const float4*)c->S[0][1]; }, 0); }, &ms);
        if (s != CVTPM_OK) break;
        add(S.kn, ms);
        if (best_ms < 0.0f || ms < best_ms) { best_ms = ms; win.grid_mult = g; }
    }
    if (s == CVTPM_OK) {
        cvtpm_params pd = S.p;
        S.p.pd_iterations = 8;
        best_ms = -1.0f;
        for (int rows : {16, 8})
            for (int halo : {4, 2})
                for (int g : {1, 0}) {
                    S.kn = PmBatchKnobs{g, rows, halo};
                    float ms = 0.0f;
                    s = timed([&] { return phase_pd(S, 0, 5.0f); }, &ms);
                    if (s != CVTPM_OK) break;
                    add(S.kn, ms);
                    if (best_ms < 0.0f || ms < best_ms) { best_ms = ms; win.pd_rows = rows; win.pd_halo = halo; }
                }
        S.p = pd;
    }
    if (s != CVTPM_OK) return s;
    *best = win;
    return CVTPM_OK;
}

/* Captures the phase-batched schedule into one graph. */
cvtpm_status capture_phased(PhaseState& S, cudaGraphExec_t* exec, size_t* nodes) {
    cvtpm_ctx* ctx = S.ctx;
    std::vector<cvtpm_ctx*> pc(ctx->bpairs.begin(), ctx->bpairs.begin() + S.n);
    for (cvtpm_ctx* c : pc) c->no_alloc = true;
    if (cudaStreamBeginCapture(S.st, cudaStreamCaptureModeThreadLocal) != cudaSuccess) {
        for (cvtpm_ctx* c : pc) c->no_alloc = false;
        return cuda_fail(ctx, cudaGetLastError(), "begin capture");
    }
    CaptureGuard guard(S.st, pc);
    S.launches = 0;
    cvtpm_status err = phase_schedule(S, S.p.iterations);
    cudaGraph_t graph = nullptr;
    cudaError_t e = cudaStreamEndCapture(S.st, &graph);
    guard.release();
    for (cvtpm_ctx* c : pc) c->no_alloc = false;
    if (err != CVTPM_OK) { if (graph) cudaGraphDestroy(graph); return err; }
    if (e != cudaSuccess) { if (graph) cudaGraphDestroy(graph); return cuda_fail(ctx, e, "end capture"); }
    *nodes = 0;
    cudaGraphGetNodes(graph, nullptr, nodes);
    e = cudaGraphInstantiate(exec, graph, 0);
    cudaGraphDestroy(graph);
    if (e != cudaSuccess) return cuda_fail(ctx, e, "graph instantiate");
    return CVTPM_OK;
}

/* The batch mode: the phase-batched schedule (knobs S.kn) against one lane
 * of per-pair launch sequences (run_depthmap, whose smoothers overlap on its
 * side stream), each timed once on the tuner's subset (the first pairs, up
 * to 4 Mpx) for one iteration, after the lane's scratch is sized for the
 * subset.  ms[0]: phase-batched, ms[1]: one lane. */
cvtpm_status tune_mode(PhaseState& full, float ms[2]) {
    PhaseState S = full;
    long long px = 0;
    int maxW = 1, maxH = 1;
    cvtpm_ctx* ctx = S.ctx;
    cvtpm_ctx* lane = ctx->lanes[0].c;
    cvtpm_status s = cvtpm_set_memory_budget(lane, ctx->pass_budget);
    S.n = 0;
    while (S.n < full.n && (S.n == 0 || px < 4000000)) {
        PmPassArgs aL, aR;
        bool overlap;
        if (s == CVTPM_OK)
            s = plan_pass(lane, S.p, full.pairs[S.n].width, full.pairs[S.n].height, true, S.st, &aL, &aR, &overlap);
        px += (long long)full.pairs[S.n].width * full.pairs[S.n].height;
        maxW = std::max(maxW, full.pairs[S.n].width);
        maxH = std::max(maxH, full.pairs[S.n].height);
        ++S.n;
    }
    if (s == CVTPM_OK) s = ensure_buffers(lane, maxW, maxH);
    if (s != CVTPM_OK) return fail(ctx, s, lane->err);
    EventPair ev;
    CK(cudaEventCreate(&ev.a), "tune event");
    CK(cudaEventCreate(&ev.b), "tune event");
    for (int mode = 0; mode < 2; ++mode) {
        if (cudaEventRecord(ev.a, S.st) != cudaSuccess) return cuda_fail(ctx, cudaGetLastError(), "tune record");
        if (mode == 0) {
            if ((s = phase_schedule(S, 1)) != CVTPM_OK) return s;
        } else {
            for (int i = 0; i < S.n; ++i) {
                const cvtpm_pair& q = S.pairs[i];
                cvtpm_params pq = S.p;
                pq.iterations = 1;
                pq.depthmax = q.depthmax;
                lane->prm = pq;
                lane->timing = false;
                if ((s = run_depthmap(lane, pq, q.dmap, q.dmap_pitch, q.left, q.right, q.width, q.height, q.pitch,
                                      nullptr, 0, nullptr, S.st)) != CVTPM_OK)
                    return fail(ctx, s, lane->err);
            }
        }
        float t = 0.0f;
        if (cudaEventRecord(ev.b, S.st) != cudaSuccess || cudaEventSynchronize(ev.b) != cudaSuccess ||
            cudaEventElapsedTime(&t, ev.a, ev.b) != cudaSuccess)
            return cuda_fail(ctx, cudaGetLastError(), "tune timing");
        ms[mode] = t;
    }
    return CVTPM_OK;
}

}  // namespace

extern "C" {

/* The graph of k lanes of per-pair launch sequences, captured and launched. */
static cvtpm_status batch_lanes(cvtpm_ctx* ctx, const cvtpm_pair* pairs, int npairs, int k,
                                const std::vector<unsigned char>& key, cudaStream_t st) {
    cvtpm_status s;
    ctx->binfo.phased = 0;
    size_t nodes = 0;
    if ((s = capture_batch(ctx, pairs, npairs, k, ctx->prm.iterations, &ctx->bexec, &nodes)) != CVTPM_OK) return s;
    ctx->bkey = key;
    ctx->binfo.lanes = k;
    ctx->binfo.shared_windows = ctx->prm.arith == CVTPM_ARITH_FAST && ctx->pass_budget > 0 ? 1 : 0;
    ctx->binfo.graph_nodes = (long long)nodes;
    ctx->binfo.replays = 0;
    ctx->binfo.launches = 0;
    return launch_batch(ctx, ctx->bexec, st);
}

static cvtpm_status depthmap_batched(cvtpm_ctx* ctx, const cvtpm_pair* pairs, int npairs, void* stream) {
    if (!ctx) return CVTPM_ERR_INVALID_ARGUMENT;
    if (!pairs || npairs < 1) return fail(ctx, CVTPM_ERR_INVALID_ARGUMENT, "no pairs");
    cvtpm_status s;
    if ((s = check_params(ctx, ctx->prm)) != CVTPM_OK) return s;
    for (int i = 0; i < npairs; ++i)
        if ((s = check_pair(ctx, pairs[i], i)) != CVTPM_OK) return s;
    CK(cudaSetDevice(ctx->device), "cudaSetDevice");
    cudaStream_t st = (cudaStream_t)stream;
    /* the graph of the previous call is replayed when nothing changed */
    std::vector<unsigned char> key;
    auto put = [&](const void* v, size_t nb) { key.insert(key.end(), (const unsigned char*)v, (const unsigned char*)v + nb); };
    const cvtpm_params& pr = ctx->prm;          /* field by field: no padding bytes in the key */
    put(&pr.patchsize, sizeof(int)); put(&pr.depthmax, sizeof(float)); put(&pr.iterations, sizeof(int));
    put(&pr.viewsamples, sizeof(int)); put(&pr.dscale, sizeof(float)); put(&pr.maxdispdiff, sizeof(float));
    put(&pr.maxanglediff, sizeof(float)); put(&pr.thetascale, sizeof(float)); put(&pr.pd_iterations, sizeof(int));
    put(&pr.color_weight, sizeof(float)); put(&pr.color_alpha, sizeof(float)); put(&pr.color_maxdiff, sizeof(float));
    put(&pr.grad_maxdiff, sizeof(float)); put(&pr.weight_profile, sizeof(int)); put(&pr.rng, sizeof(int));
    put(&pr.seed, sizeof(uint64_t)); put(&pr.arith, sizeof(int)); put(&pr.schedule, sizeof(int));
    put(&ctx->batch_lanes, sizeof(int));
    put(&ctx->pinned_knobs, sizeof(bool));
    put(&ctx->knobs.grid_mult, sizeof(int)); put(&ctx->knobs.pd_rows, sizeof(int)); put(&ctx->knobs.pd_halo, sizeof(int));
    put(&ctx->pass_budget, sizeof(size_t));
    for (int i = 0; i < npairs; ++i) {
        const cvtpm_pair& q = pairs[i];
        put(&q.width, sizeof(int)); put(&q.height, sizeof(int)); put(&q.depthmax, sizeof(float));
    }
    const std::vector<unsigned char> tkey = key;       /* parameters and shapes */
    for (int i = 0; i < npairs; ++i) {
        const cvtpm_pair& q = pairs[i];
        put(&q.left, sizeof(void*)); put(&q.right, sizeof(void*)); put(&q.pitch, sizeof(size_t));
        put(&q.dmap, sizeof(void*)); put(&q.dmap_pitch, sizeof(size_t));
    }
    if (ctx->bexec && key == ctx->bkey) {
        ++ctx->binfo.replays;
        return launch_batch(ctx, ctx->bexec, st);
    }
    if (ctx->bexec) { cudaGraphExecDestroy(ctx->bexec); ctx->bexec = nullptr; ctx->bkey.clear(); }
    if ((s = ensure_lanes(ctx, 1)) != CVTPM_OK) return s;
    CK(cudaStreamSynchronize(st), "batch order");      /* inputs written on `st` before tuning reads them */
    if (ctx->batch_lanes == 0 && ctx->prm.schedule == CVTPM_SCHEDULE_JACOBI) {
        /* phase-batched: one launch per phase for all pairs */
        PhaseState S{ctx, pairs, npairs, ctx->prm, PmBatchKnobs{1, 16, 4}, ctx->bstream, 1, 0, {}, {}};
        if ((s = phase_prepare(S)) != CVTPM_OK) return s;
        CK(cudaStreamSynchronize(ctx->bstream), "batch prepare");
        ctx->binfo.tuned = 0;
        bool cached = false, phased = true;
        if (ctx->pinned_knobs) { S.kn = ctx->knobs; cached = true; ctx->binfo.mode_ms[0] = ctx->binfo.mode_ms[1] = 0.0f; }
        for (auto& tk : ctx->tuned_knobs)
            if (!cached && tk.key == tkey) {
                S.kn = tk.kn;
                phased = tk.phased;
                ctx->binfo.mode_ms[0] = tk.mode_ms[0];
                ctx->binfo.mode_ms[1] = tk.mode_ms[1];
                cached = true;
            }
        if (!cached) {
            const auto c0 = std::chrono::steady_clock::now();
            PmBatchKnobs best{1, 16, 4};
            if ((s = tune_phased(S, &best)) != CVTPM_OK) return s;
            S.kn = best;
            float ms[2] = {0.0f, 0.0f};
            if ((s = tune_mode(S, ms)) != CVTPM_OK) return s;
            /* one lane is the plain call sequence in a graph (it measured level
             * with a loop of plain calls); the phase-batched schedule has to
             * beat it clearly on the proxy (on a full batch it measured 1 %
             * behind where the proxy had it 1 % ahead) */
            phased = ms[0] < 0.97f * ms[1];
            ctx->binfo.tune_ms = std::chrono::duration<float, std::milli>(std::chrono::steady_clock::now() - c0).count();
            ctx->tuned_knobs.push_back({tkey, best, phased, {ms[0], ms[1]}});
            ctx->binfo.mode_ms[0] = ms[0];
            ctx->binfo.mode_ms[1] = ms[1];
            ctx->binfo.tuned = 1;
        }
        if (!phased) return batch_lanes(ctx, pairs, npairs, 1, key, st);
        size_t nodes = 0;
        if ((s = capture_phased(S, &ctx->bexec, &nodes)) != CVTPM_OK) return s;
        ctx->bkey = key;
        ctx->binfo.phased = 1;
        ctx->binfo.lanes = 0;
        ctx->binfo.grid_mult = S.kn.grid_mult;
        ctx->binfo.pd_rows = S.kn.pd_rows;
        ctx->binfo.pd_halo = S.kn.pd_halo;
        ctx->binfo.launches = S.launches;
        int nb = 0;
        for (int i = 0; i < npairs; ++i) nb += S.aL[i].costs ? 1 : 0;
        ctx->binfo.shared_windows = nb == npairs ? 1 : 0;
        ctx->binfo.graph_nodes = (long long)nodes;
        ctx->binfo.replays = 0;
        return launch_batch(ctx, ctx->bexec, st);
    }
    int k = ctx->batch_lanes > 0 ? ctx->batch_lanes : 0;
    ctx->binfo.tuned = 0;
    ctx->binfo.mode_ms[0] = ctx->binfo.mode_ms[1] = 0.0f;
    if (k <= 0) {
        if (!ctx->tkey.empty() && tkey == ctx->tkey) {   /* same shapes: keep the tuned choice */
            k = ctx->tuned_lanes;
        } else {
            if ((s = tune_batch(ctx, pairs, npairs, &k)) != CVTPM_OK) return s;
            ctx->tkey = tkey;
            ctx->tuned_lanes = k;
        }
        ctx->binfo.tuned = 1;
    }
    return batch_lanes(ctx, pairs, npairs, k, key, st);
}

/* the lane plans are sized by npairs: a failed host allocation becomes a
 * status, no exception leaves the C ABI */
cvtpm_status cvtpm_depthmap_batched(cvtpm_ctx* ctx, const cvtpm_pair* pairs, int npairs, void* stream) {
    try {
        return depthmap_batched(ctx, pairs, npairs, stream);
    } catch (const std::bad_alloc&) {
        return ctx ? fail(ctx, CVTPM_ERR_ALLOC, "host memory exhausted") : CVTPM_ERR_ALLOC;
    }
}

cvtpm_status cvtpm_set_batch_lanes(cvtpm_ctx* ctx, int lanes) {
    if (!ctx || lanes < 0 || lanes > 64) return CVTPM_ERR_INVALID_ARGUMENT;
    ctx->batch_lanes = lanes;
    return CVTPM_OK;
}

cvtpm_status cvtpm_set_batch_knobs(cvtpm_ctx* ctx, int grid_mult, int pd_rows, int pd_halo) {
    if (!ctx) return CVTPM_ERR_INVALID_ARGUMENT;
    if (grid_mult < 0) { ctx->pinned_knobs = false; return CVTPM_OK; }
    if (grid_mult > 2 || (pd_rows != 16 && pd_rows != 8) || (pd_halo != 4 && pd_halo != 2))
        return fail(ctx, CVTPM_ERR_INVALID_ARGUMENT, "batch knobs: grid_mult 0..2, pd_rows 16 or 8, pd_halo 4 or 2");
    ctx->pinned_knobs = true;
    ctx->knobs = PmBatchKnobs{grid_mult, pd_rows, pd_halo};
    return CVTPM_OK;
}

cvtpm_status cvtpm_get_batch_info(const cvtpm_ctx* ctx, cvtpm_batch_info* out) {
    if (!ctx || !out) return CVTPM_ERR_INVALID_ARGUMENT;
    *out = ctx->binfo;
    return CVTPM_OK;
}

cvtpm_status cvtpm_tool_fp32_peak(int device, void* stream, float* tflops) {
    if (!tflops) return CVTPM_ERR_INVALID_ARGUMENT;
    cudaStream_t st = (cudaStream_t)stream;
    if (cudaSetDevice(device) != cudaSuccess) return CVTPM_ERR_CUDA;
    int sms = 0;
    if (cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device) != cudaSuccess) return CVTPM_ERR_CUDA;
    const int blocks = sms * 8, iters = 1 << 16;
    float* out = nullptr;
    if (cudaMalloc(&out, sizeof(float) * blocks * 256) != cudaSuccess) return CVTPM_ERR_ALLOC;
    cudaEvent_t a, b;
    cudaEventCreate(&a);
    cudaEventCreate(&b);
    float best = 1e30f;
    cvtpm_status s = CVTPM_OK;
    for (int rep = 0; rep < 4 && s == CVTPM_OK; ++rep) {
        cudaEventRecord(a, st);
        if (pm_launch_ffma_peak(out, blocks, iters, st) != cudaSuccess) s = CVTPM_ERR_CUDA;
        cudaEventRecord(b, st);
        if (cudaEventSynchronize(b) != cudaSuccess) s = CVTPM_ERR_CUDA;
        float ms = 0.0f;
        cudaEventElapsedTime(&ms, a, b);
        if (rep > 0 && ms < best) best = ms;    /* the first launch warms up */
    }
    cudaEventDestroy(a);
    cudaEventDestroy(b);
    cudaFree(out);
    if (s != CVTPM_OK) return s;
    const double flops = 2.0 * 8.0 * (double)iters * blocks * 256.0;
    *tflops = (float)(flops / (best * 1e-3) / 1e12);
    return CVTPM_OK;
}

cvtpm_status cvtpm_tool_pd_math_check(int device, void* stream, unsigned long long* bad) {
    if (!bad) return CVTPM_ERR_INVALID_ARGUMENT;
    if (cudaSetDevice(device) != cudaSuccess) return CVTPM_ERR_CUDA;
    cudaStream_t st = (cudaStream_t)stream;
    unsigned long long* d = nullptr;
    if (cudaMalloc(&d, 4 * sizeof(*d)) != cudaSuccess) { cudaGetLastError(); return CVTPM_ERR_ALLOC; }
    cudaError_t e = cudaMemsetAsync(d, 0, 4 * sizeof(*d), st);
    if (e == cudaSuccess) e = pm_launch_pd_math_check(d, st);
    if (e == cudaSuccess) e = cudaMemcpyAsync(bad, d, 4 * sizeof(*d), cudaMemcpyDeviceToHost, st);
    if (e == cudaSuccess) e = cudaStreamSynchronize(st);
    cudaFree(d);
    return e == cudaSuccess ? CVTPM_OK : CVTPM_ERR_CUDA;
}

int cvtpm_tool_routes(const cvtpm_params* params, int width, int height) {
    if (!params || width < 1 || height < 1 || params->patchsize < 1) return -1;
    PmCostConsts k;
    memset(&k, 0, sizeof(k));
    k.W = width; k.H = height; k.P = params->patchsize;
    return (pm_tap_parallel(k) ? CVTPM_ROUTE_TAPS : 0) | (pm_tap_sweeps(k) ? CVTPM_ROUTE_TAP_SWEEPS : 0) |
           (pm_shared_windows(k) ? CVTPM_ROUTE_WINDOWS : 0) |
           (pm_tap_field(k, params->arith == CVTPM_ARITH_EXACT) ? CVTPM_ROUTE_TAP_COST : 0) |
           (pm_tap_adjoint(k, true, true) ? CVTPM_ROUTE_TAP_ADJOINT : 0);
}

cvtpm_status cvtpm_tool_pd_time(cvtpm_ctx* ctx, int steps, void* stream, float* us_per_step) {
    if (!ctx || !us_per_step || steps < 2 || (steps & 1)) return CVTPM_ERR_INVALID_ARGUMENT;
    if (!ctx->pool || ctx->capW <= 0 || ctx->capH <= 0)
        return fail(ctx, CVTPM_ERR_INVALID_ARGUMENT, "no depthMap has sized this context yet");
    if (cudaSetDevice(ctx->device) != cudaSuccess) return CVTPM_ERR_CUDA;
    cudaStream_t st = (cudaStream_t)stream;
    const int W = ctx->capW, H = ctx->capH;
    const bool timing = ctx->timing;
    ctx->timing = false;
    cudaEvent_t a = nullptr, b = nullptr;
    cudaEventCreate(&a);
    cudaEventCreate(&b);
    float best = 1e30f;
    cvtpm_status s = CVTPM_OK;
    for (int rep = 0; rep < 3 && s == CVTPM_OK; ++rep) {
        /* the left view's smoother input of the last call, warm-started from
         * its smoothed field as depthMap's own calls are, into scratch that the
         * next call rewrites before reading */
        if (cudaMemcpyAsync(ctx->tmpR, ctx->smooth[0], (size_t)W * H * 16, cudaMemcpyDeviceToDevice, st) != cudaSuccess) {
            s = CVTPM_ERR_CUDA;
            break;
        }
        cudaEventRecord(a, st);
        s = pd_apply(ctx, ctx->tmpR, ctx->tmp2, ctx->wgt[0], 5.0f, steps, W, H, st, nullptr, 1);
        cudaEventRecord(b, st);
        if (s == CVTPM_OK && cudaEventSynchronize(b) != cudaSuccess) s = CVTPM_ERR_CUDA;
        float ms = 0.0f;
        cudaEventElapsedTime(&ms, a, b);
        if (rep > 0 && ms < best) best = ms;    /* the first run warms up */
    }
    cudaEventDestroy(a);
    cudaEventDestroy(b);
    ctx->timing = timing;
    if (s != CVTPM_OK) return s;
    *us_per_step = best * 1e3f / (float)steps;
    return CVTPM_OK;
}

}  // extern "C"
