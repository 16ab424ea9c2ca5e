// C ABI of libtrips_b200: context (scratch owner), forward, backward, fused Adam and the inspection calls.
// The host logic here replaces PointRendererCache (src/lib/rendering/PointRenderer.cu:197-528) and the host
// parts of RenderFast16 / BlendBackwardsBilinearFast / MyAdam::step.
#include <algorithm>
#include <cfloat>
#include <cmath>
#include <cstdio>
#include <cstring>
#include <new>
#include <string>
#include <vector>

#include "common.cuh"
#include "list_order.h"

using namespace trips;

namespace
{
struct DevBuf
{
    void* p      = nullptr;
    size_t bytes = 0;
};

inline cudaError_t ensure(DevBuf& b, size_t bytes, double growth = 1.0)
{
    if (bytes <= b.bytes) return cudaSuccess;
    if (b.p) cudaFree(b.p);
    b.p          = nullptr;
    b.bytes      = 0;
    size_t want  = (size_t)((double)bytes * growth);
    want         = (want + 255) & ~(size_t)255;
    cudaError_t e = cudaMalloc(&b.p, want);
    if (e != cudaSuccess && want > bytes)
    {
        (void)cudaGetLastError();
        want = (bytes + 255) & ~(size_t)255;
        e    = cudaMalloc(&b.p, want);
    }
    if (e == cudaSuccess) b.bytes = want;
    return e;
}
// Optional CUDA-event timers around every stage (the reference's SAIGA_OPTIONAL_TIME_MEASURE scopes,
// RenderForward.cu:1090,1166,1238,1271, PointRenderer.cu:1338) and a launch counter per stage.
struct StageTimers
{
    bool enabled = false;
    struct Span
    {
        int stage;
        cudaEvent_t a, b;
    };
    std::vector<Span> open;                            // recorded, not yet read back
    std::vector<std::pair<cudaEvent_t, cudaEvent_t>> pool;  // reusable event pairs
    double ms[TRIPS_NUM_STAGES]        = {};
    int64_t launches[TRIPS_NUM_STAGES] = {};
    int64_t timed[TRIPS_NUM_STAGES]    = {};

    bool begin(int stage, cudaStream_t st, Span& sp)
    {
        if (!enabled) return false;
        if (pool.empty())
        {
            cudaEvent_t a, b;
            if (cudaEventCreate(&a) != cudaSuccess || cudaEventCreate(&b) != cudaSuccess) return false;
            pool.emplace_back(a, b);
        }
        sp.stage = stage;
        sp.a     = pool.back().first;
        sp.b     = pool.back().second;
        pool.pop_back();
        cudaEventRecord(sp.a, st);
        return true;
    }
    void end(const Span& sp, cudaStream_t st)
    {
        cudaEventRecord(sp.b, st);
        open.push_back(sp);
    }
    void collect()
    {
        for (const Span& sp : open)
        {
            float t = 0.f;
            if (cudaEventSynchronize(sp.b) == cudaSuccess && cudaEventElapsedTime(&t, sp.a, sp.b) == cudaSuccess)
            {
                ms[sp.stage] += t;
                timed[sp.stage] += 1;
            }
            pool.emplace_back(sp.a, sp.b);
        }
        open.clear();
    }
    void destroy()
    {
        collect();
        for (auto& pr : pool)
        {
            cudaEventDestroy(pr.first);
            cudaEventDestroy(pr.second);
        }
        pool.clear();
    }
};
}  // namespace

struct SizeKey
{
    int N, B, w, h, L, C, train;
    int layer_rule;  // which layers a point is written to (use_layer_point_size, render_points_in_all_lower_resolutions): changes the fragment count
    bool operator==(const SizeKey& o) const
    {
        return N == o.N && B == o.B && w == o.w && h == o.h && L == o.L && C == o.C && train == o.train && layer_rule == o.layer_rule;
    }
};

struct TripsContext
{
    StageTimers timers;
    int device   = 0;
    int sm_count = 148;
    std::string error;
    // forward scratch
    DevBuf heavy, cams, zeroed, bin_base, view_total, bin_cursor, entry_base, entries, offsets, view_base, frags, rec_n, records, stats, point_entry, point_state, resize_scratch, block_skip;
    size_t zero_bins = 0, zero_counts = 0;  // where bin_count and counts start inside `zeroed` (behind the work counters)
    // backward scratch
    DevBuf egrad, g_small;
    // adam
    DevBuf adam_tab;
    // pinned host mirror of DevStats and the event behind which it becomes valid when a call did not wait for it
    void* h_pinned        = nullptr;
    cudaEvent_t totals_ev = nullptr;
    bool pending          = false;  // the totals of the last forward call have not been read yet
    // shapes of the last training call, while it may be followed by one of the same shapes that does not wait for its counts
    SizeKey size_key{};
    bool have_sizes                 = false;
    unsigned long long need_entries = 0, need_frags = 0;  // of the last pass whose totals were read (training and inference)
    int entry_C                     = 0;  // channel count the entry arrays are laid out for
    bool crowded                    = false;  // the point cloud crowds into few screen tiles: use the aggregating binning kernels
    // state of the last forward call
    bool have_forward = false;
    Geom geom{};
    TripsRenderParams params{};
    int B = 0, N = 0, n_tex = 0, C = 0;
    size_t entry_cap = 0;                  // entries the two entry arrays (head | tail, in this order) are laid out for
    TripsStats host_stats{};
};

#define CU_CHECK(ctx, expr)                                                                      \
    do                                                                                           \
    {                                                                                            \
        cudaError_t _e = (expr);                                                                 \
        if (_e != cudaSuccess)                                                                   \
        {                                                                                        \
            (ctx)->error = std::string(#expr) + ": " + cudaGetErrorString(_e);                   \
            (void)cudaGetLastError();                                                            \
            return _e == cudaErrorMemoryAllocation ? TRIPS_ERR_OUT_OF_MEMORY : TRIPS_ERR_CUDA;   \
        }                                                                                        \
    } while (0)

// Runs `expr` (which launches `n` kernels of `stage`) between two events when the stage timers are on.
#define STAGE(ctx, stage, n, st, expr)                      \
    do                                                      \
    {                                                       \
        StageTimers::Span _sp;                              \
        bool _t = (ctx)->timers.begin((stage), (st), _sp);  \
        cudaError_t _se = (expr);                           \
        if (_t) (ctx)->timers.end(_sp, (st));               \
        (ctx)->timers.launches[(stage)] += (n);             \
        CU_CHECK(ctx, _se);                                 \
    } while (0)

static int fail(TripsContext* ctx, int code, const char* msg)
{
    if (ctx) ctx->error = msg;
    return code;
}

static void free_buf(DevBuf& b)
{
    if (b.p) cudaFree(b.p);
    b.p     = nullptr;
    b.bytes = 0;
}

static ScenePtrs scene_ptrs(const TripsScene* s)
{
    ScenePtrs sp;
    sp.N          = s->n_points;
    sp.n_tex      = s->n_tex;
    sp.C          = s->channels;
    sp.position   = reinterpret_cast<const float4*>(s->position);
    sp.point_size = s->point_size;
    sp.index      = s->index;
    sp.texture    = s->texture;
    sp.confidence = s->confidence;
    sp.background = s->background;
    sp.dropout    = s->dropout;
    return sp;
}

// work counters of the binning passes: one per pass and group of views
static size_t ticket_groups(int B) { return 2 * (((size_t)B + kViewGroup - 1) / kViewGroup); }
// work counter of the blend: behind those of the binning, count and collect passes, on a line of its own
static size_t blend_ticket_at(int B) { return (ticket_groups(B) + 2 * (size_t)B + 31) / 32 * 32; }

// views the point-to-entry table holds at a time
static int entry_views(int B, int N)
{
    return (int)std::min<size_t>((size_t)B, std::max<size_t>(1, kEntryTableBytes / (sizeof(uint32_t) * (size_t)std::max(1, N))));
}

// Room for what the pre-selection of a call can meet: a list has more than kHeavyList fragments, a part of a shared one at
// least half of kHeavyPart, and a call at most 4 fragments per point, layer and view.
static HeavyLists heavy_lists(int N, int L, int B, void* p)
{
    HeavyLists h;
    const unsigned long long most = 4ull * N * L * B;
    h.cap        = (unsigned)std::min<unsigned long long>(kHeavyCap, most / kHeavyList + 1);
    h.shared_cap = (unsigned)std::min<unsigned long long>(kHeavyShared, most / (kHeavyPart / 2) + 1);
    h.item       = (uint4*)p;
    h.nearest    = (uint32_t*)(h.item + h.cap);
    h.finished   = h.nearest + 16 * (size_t)h.shared_cap;
    return h;
}
static size_t heavy_bytes(const HeavyLists& h) { return sizeof(uint4) * h.cap + sizeof(uint32_t) * 17 * (size_t)h.shared_cap; }

static FwdBuffers fwd_buffers(TripsContext* c, int B)
{
    FwdBuffers fb;
    fb.bin_count  = (uint32_t*)((char*)c->zeroed.p + c->zero_bins);
    fb.bin_base   = (uint32_t*)c->bin_base.p;
    fb.view_total = (uint32_t*)c->view_total.p;
    fb.bin_cursor = (uint32_t*)c->bin_cursor.p;
    fb.entry_base = (unsigned long long*)c->entry_base.p;
    fb.ent_head   = (float4*)c->entries.p;
    fb.ent_tail   = (float*)c->entries.p + 8 * c->entry_cap;
    fb.counts     = (uint32_t*)((char*)c->zeroed.p + c->zero_counts);
    fb.offsets    = (uint32_t*)c->offsets.p;
    fb.view_base  = (unsigned long long*)c->view_base.p;
    fb.frags      = (uint4*)c->frags.p;
    fb.frag_cap   = c->frags.bytes / sizeof(uint4);
    fb.report_overflow = c->params.train;
    fb.rec_n      = (uint8_t*)c->rec_n.p;
    fb.records    = (uint2*)c->records.p;
    fb.stats      = (DevStats*)c->stats.p;
    fb.ticket         = (unsigned int*)c->zeroed.p;
    fb.ticket_count   = fb.ticket + ticket_groups(B);
    fb.ticket_collect = fb.ticket_count + B;
    fb.ticket_blend   = fb.ticket + blend_ticket_at(B);
    fb.finished       = fb.ticket_blend + 32;  // on another line than the blend's counter
    fb.list_cursor    = fb.finished + 2;
    fb.point_entry = c->params.train ? (uint32_t*)c->point_entry.p : nullptr;
    fb.entry_views = entry_views(B, c->N);
    fb.note_entry  = fb.entry_views == B ? fb.point_entry : nullptr;
    fb.point_state = c->params.train ? (float4*)c->point_state.p : nullptr;
    fb.block_skip = (const uint8_t*)c->block_skip.p;
    fb.heavy      = heavy_lists(c->N, c->geom.L, B, c->heavy.p);
    return fb;
}

// DevStats is allocated once and zeroed then; afterwards setup_cams_kernel clears its counters per call.
static cudaError_t ensure_stats(TripsContext* c, cudaStream_t st)
{
    if (c->stats.p) return cudaSuccess;
    cudaError_t e = ensure(c->stats, sizeof(DevStats));
    if (e != cudaSuccess) return e;
    return cudaMemsetAsync(c->stats.p, 0, sizeof(DevStats), st);
}

static bool valid_channels(int c) { return c == 3 || c == 4 || c == 6 || c == 8 || c == 16; }

extern "C" {

const char* trips_status_string(int status)
{
    switch (status)
    {
        case TRIPS_OK: return "ok";
        case TRIPS_ERR_INVALID_ARG: return "invalid argument";
        case TRIPS_ERR_CUDA: return "CUDA error";
        case TRIPS_ERR_OUT_OF_MEMORY: return "out of device memory";
        case TRIPS_ERR_UNSUPPORTED: return "unsupported camera model or flag";
        case TRIPS_ERR_NO_FORWARD: return "backward without a training forward pass";
        case TRIPS_ERR_TOO_LARGE: return "size beyond the supported maximum";
        default: return "unknown status";
    }
}

const char* trips_last_error(const TripsContext* ctx) { return ctx ? ctx->error.c_str() : "null context"; }

int trips_context_create(TripsContext** out, int device)
{
    if (!out) return TRIPS_ERR_INVALID_ARG;
    *out = nullptr;
    int count = 0;
    if (cudaGetDeviceCount(&count) != cudaSuccess || device < 0 || device >= count)
    {
        (void)cudaGetLastError();
        return TRIPS_ERR_CUDA;
    }
    TripsContext* c = new (std::nothrow) TripsContext();
    if (!c) return TRIPS_ERR_OUT_OF_MEMORY;
    c->device = device;
    cudaDeviceProp prop;
    if (cudaGetDeviceProperties(&prop, device) == cudaSuccess) c->sm_count = prop.multiProcessorCount;
    *out = c;
    return TRIPS_OK;
}

void trips_context_destroy(TripsContext* c)
{
    if (!c) return;
    DevBuf* all[] = {&c->heavy, &c->cams, &c->zeroed, &c->bin_base, &c->view_total, &c->bin_cursor, &c->entry_base, &c->entries, &c->offsets,
                     &c->view_base, &c->frags, &c->rec_n, &c->records, &c->stats, &c->egrad,
                     &c->point_entry, &c->point_state, &c->g_small, &c->adam_tab, &c->resize_scratch, &c->block_skip};
    for (DevBuf* b : all) free_buf(*b);
    c->timers.destroy();
    if (c->h_pinned) cudaFreeHost(c->h_pinned);
    if (c->totals_ev) cudaEventDestroy(c->totals_ev);
    delete c;
}

// Geometry of the pyramid and of the tile / bin decompositions for a (w, h, L) image.
static bool make_geom(int w, int h, int L, Geom& g)
{
    g.L = L;
    long long base = 0;
    int lw = w, lh = h;
    for (int l = 0; l < g.L; ++l)
    {
        g.W[l]    = lw;
        g.H[l]    = lh;
        g.base[l] = (int)base;
        base += (long long)lw * lh;
        lw = (lw + 1) / 2;  // ceil halving, PointRenderer.cu:385-389
        lh = (lh + 1) / 2;
    }
    double in_x = DBL_MAX, in_y = DBL_MAX;
    for (int l = 0; l < TRIPS_MAX_LAYERS; ++l)
    {
        if (l < g.L)
        {
            in_x = std::min(in_x, std::ldexp((double)(g.W[l] - 1), l));
            in_y = std::min(in_y, std::ldexp((double)(g.H[l] - 1), l));
        }
        auto below = [](double v) { return (double)(float)v > v ? std::nextafterf((float)v, 0.f) : (float)v; };
        g.inside_x[l] = below(in_x), g.inside_y[l] = below(in_y);
    }
    for (int l = g.L; l <= TRIPS_MAX_LAYERS; ++l) g.base[l] = (int)base;
    if (base > (1ll << 30)) return false;
    g.P = (int)base;
    static const int kRegTiles[5] = {0, 128, 160, 168, 170};
    g.reg_layers = g.L < 4 ? g.L : 4;
    g.reg_x      = (w + 63) / 64;
    g.reg_tiles  = kRegTiles[g.reg_layers];
    g.reg_total  = g.reg_x * ((h + 63) / 64) * g.reg_tiles;
    int tb = g.reg_total;
    for (int l = 0; l < TRIPS_MAX_LAYERS; ++l)
    {
        g.tile_base[l] = tb;
        g.tiles_x[l]   = 1;
        if (l >= g.reg_layers && l < g.L)
        {
            g.tiles_x[l] = (g.W[l] + kTileW - 1) / kTileW;
            tb += g.tiles_x[l] * ((g.H[l] + kTileH - 1) / kTileH);
        }
    }
    g.tile_base[TRIPS_MAX_LAYERS] = tb;
    g.n_tiles = tb;
    g.bins_x  = ((w - 1) >> kBinShift) + 1;
    g.bins_y  = ((h - 1) >> kBinShift) + 1;
    g.n_bins  = g.bins_x * g.bins_y;
    return true;
}

// The entry arrays (head | tail, in this order) re-laid out for at least `entries` entries.
static cudaError_t ensure_entries(TripsContext* ctx, size_t entries, int C, double growth)
{
    const size_t ES = (size_t)entry_stride(C);
    if (ctx->entries.p && ctx->entry_C == C && entries <= ctx->entry_cap) return cudaSuccess;
    const size_t want = (size_t)((double)(entries > 0 ? entries : 1) * growth) + 1;
    cudaError_t e = ensure(ctx->entries, sizeof(float) * ES * want + 16);
    if (e != cudaSuccess)
    {
        ctx->entry_cap = 0;
        return e;
    }
    ctx->entry_cap = (ctx->entries.bytes - 16) / (sizeof(float) * ES);
    ctx->entry_C   = C;
    return cudaSuccess;
}

// Totals of a forward call whose sizes were not waited for (steady-state training): read them now, publish the
// statistics, and grow the entry / fragment buffers if that call needed more than they hold (the call itself rendered
// the views that did not fit as background and raised a status bit).
static int resolve_pending(TripsContext* ctx)
{
    if (!ctx->pending) return TRIPS_OK;
    ctx->pending = false;
    CU_CHECK(ctx, cudaEventSynchronize(ctx->totals_ev));
    const DevStats* hs = (const DevStats*)ctx->h_pinned;
    ctx->need_entries  = hs->visible;
    ctx->need_frags    = hs->frag_need;
    ctx->crowded       = hs->max_key >= kHotKey;
    ctx->host_stats.visible_points      = (int64_t)hs->visible;
    ctx->host_stats.fragments           = (int64_t)hs->frag_need;
    ctx->host_stats.kept_fragments      = (int64_t)hs->kept;
    ctx->host_stats.max_list_length     = (int64_t)hs->max_len;
    ctx->host_stats.culled_point_blocks = (int64_t)hs->culled_blocks;
    return TRIPS_OK;
}

namespace
{
constexpr double kGrowth      = 1.25;  // head room of the entry / fragment buffers over the counted need
constexpr int kEvalSubBatch   = 8;     // views rendered per pass when nothing has to be kept for a backward pass
}  // namespace

// When a pass learns how many entries and fragments its views have.
enum class Sizes
{
    wait,   // before it writes them: the buffers are sized from the pass's own counts, which costs two host synchronisations (the
            // reference synchronises 2 * num_layers times per view for the same purpose, RenderForward.cu:1201-1208)
    later,  // the buffers keep the capacity found by earlier calls (need x 1.25) and nothing is waited for: the totals travel to pinned
            // host memory behind an event, and the next training call reads them
    look,   // an inference pass: everything is launched with the buffers as they are, and the totals are looked at while the GPU
            // renders.  A pass that does not fit them, or calls for other kernels, is given up on the device (place_views) and taken up
            // from where it stopped
};

// One pass over `B` views (all views of a training call; up to kEvalSubBatch views of an inference call).
static int forward_views(TripsContext* ctx, const TripsScene* scene, const TripsView* views, int B, const TripsRenderParams* params,
                         const Geom& g, float* const* out_layers, size_t out_view_offset, const float* dropout, cudaStream_t st, Sizes sizes)
{
    const size_t N    = (size_t)scene->n_points;
    const size_t P    = (size_t)g.P;
    const int C       = scene->channels;
    const size_t n_box = (N + 8191) / 8192 + 1;

    CU_CHECK(ctx, ensure(ctx->cams, sizeof(CamConst) * B));
    // everything a pass wants zeroed, in one buffer and one clear: work counters | visible points per (bin, 8x4 tile of the bin) | list lengths
    auto aligned      = [](size_t n) { return (n + 255) & ~(size_t)255; };
    ctx->zero_bins    = aligned(sizeof(unsigned) * (blend_ticket_at(B) + 32 + B + 2));
    ctx->zero_counts  = ctx->zero_bins + aligned(sizeof(uint32_t) * (size_t)g.n_bins * 32 * B);
    const size_t zero_bytes = ctx->zero_counts + sizeof(uint32_t) * P * B;
    CU_CHECK(ctx, ensure(ctx->zeroed, zero_bytes));
    CU_CHECK(ctx, ensure(ctx->bin_base, sizeof(uint32_t) * (size_t)g.n_bins * 32 * B));
    CU_CHECK(ctx, ensure(ctx->view_total, sizeof(uint32_t) * B));
    CU_CHECK(ctx, ensure(ctx->bin_cursor, sizeof(uint32_t) * (size_t)g.n_bins * B));
    CU_CHECK(ctx, ensure(ctx->entry_base, sizeof(unsigned long long) * (B + 1)));
    CU_CHECK(ctx, ensure(ctx->block_skip, (size_t)B * n_box));
    CU_CHECK(ctx, ensure(ctx->heavy, heavy_bytes(heavy_lists((int)N, g.L, B, nullptr))));
    CU_CHECK(ctx, ensure(ctx->offsets, sizeof(uint32_t) * P * B));
    CU_CHECK(ctx, ensure(ctx->view_base, sizeof(unsigned long long) * (B + 1)));
    CU_CHECK(ctx, ensure_stats(ctx, st));
    if (params->train)
    {
        CU_CHECK(ctx, ensure(ctx->rec_n, (size_t)g.n_tiles * 32 * B));
        CU_CHECK(ctx, ensure(ctx->records, sizeof(uint2) * 16 * 32 * (size_t)g.n_tiles * B));
        CU_CHECK(ctx, ensure(ctx->point_entry, sizeof(uint32_t) * N * entry_views(B, (int)N)));
        CU_CHECK(ctx, ensure(ctx->point_state, sizeof(float4) * N));
    }
    if (ctx->frags.bytes == 0) CU_CHECK(ctx, ensure(ctx->frags, 16 * 1024 * 1024));
    if (!ctx->entries.p || ctx->entry_C != C) CU_CHECK(ctx, ensure_entries(ctx, 1024, C, 1.0));
    if (!ctx->h_pinned)
    {
        CU_CHECK(ctx, cudaMallocHost(&ctx->h_pinned, sizeof(DevStats)));
        CU_CHECK(ctx, cudaEventCreateWithFlags(&ctx->totals_ev, cudaEventDisableTiming));
    }
    DevStats* h_stats = (DevStats*)ctx->h_pinned;

    ScenePtrs sp = scene_ptrs(scene);
    sp.dropout   = dropout;
    FwdBuffers fb = fwd_buffers(ctx, B);
    CU_CHECK(ctx, cudaMemsetAsync(ctx->zeroed.p, 0, zero_bytes, st));
    STAGE(ctx, TRIPS_STAGE_SETUP, (B + kViewTable - 1) / kViewTable, st,
          launch_setup_cams(views, B, scene->poses, scene->n_images, scene->intrinsics, scene->n_cameras, params->distortion,
                            params->dist_cutoff, (CamConst*)ctx->cams.p, fb.stats, st));
    const CamConst* cams = (const CamConst*)ctx->cams.p;
    unsigned long long entries = ctx->need_entries;  // as far as the host knows

    // ---- the steps of a pass ----
    auto write_lists = [&](bool sized) -> int {  // entries, list lengths, list starts; sized: the list buffer is grown behind it
        STAGE(ctx, TRIPS_STAGE_BIN_POINTS, bin_scatter_launches((int)N, B), st, launch_bin_scatter(sp, cams, g, *params, B, fb, ctx->crowded, ctx->sm_count, st));
        if (N > 0) STAGE(ctx, TRIPS_STAGE_COUNT, 1, st, launch_count(sp, g, B, fb, strict_layers(*params), entries, ctx->sm_count, st));
        FwdBuffers fscan = fb;
        if (sized) fscan.frag_cap = ~0ull;
        STAGE(ctx, TRIPS_STAGE_SCAN, 1, st, launch_list_starts(g, B, params->k_keep, fscan, st));
        CU_CHECK(ctx, cudaMemcpyAsync(h_stats, ctx->stats.p, sizeof(DevStats), cudaMemcpyDeviceToHost, st));
        return TRIPS_OK;
    };
    auto render = [&]() -> int {
        if (N > 0) STAGE(ctx, TRIPS_STAGE_COLLECT, 1, st, launch_collect(sp, g, B, fb, strict_layers(*params), entries, ctx->sm_count, st));
        LayerPtrs out{};
        for (int l = 0; l < g.L; ++l) out.p[l] = out_layers[l] + out_view_offset * (size_t)C * g.W[l] * g.H[l];
        if (second_pipeline(*params))
            STAGE(ctx, TRIPS_STAGE_SORT_BLEND, 1, st, launch_second_blend(sp, g, *params, B, fb, out, ctx->sm_count, st));
        else
            STAGE(ctx, TRIPS_STAGE_SORT_BLEND, 2, st, [&]() -> cudaError_t {
                cudaError_t e = launch_heavy_topk(g, B, fb, ctx->sm_count, st);
                return e != cudaSuccess ? e : launch_sort_blend(sp, g, *params, B, fb, out, ctx->sm_count, st);
            }());
        return TRIPS_OK;
    };
    auto grow_entries = [&]() -> int {
        CU_CHECK(ctx, ensure_entries(ctx, (size_t)h_stats->visible, C, kGrowth));
        ctx->crowded = h_stats->max_key >= kHotKey;  // this pass's own counts already know
        entries      = h_stats->visible;
        fb           = fwd_buffers(ctx, B);
        return TRIPS_OK;
    };
    auto grow_lists = [&]() -> int {
        if ((size_t)h_stats->frag_need * sizeof(uint4) > ctx->frags.bytes)
        {
            CU_CHECK(ctx, ensure(ctx->frags, (size_t)h_stats->frag_need * sizeof(uint4), kGrowth));
            fb = fwd_buffers(ctx, B);
        }
        return TRIPS_OK;
    };
#define STEP(expr)                             \
    do                                         \
    {                                          \
        const int _rc = (expr);                \
        if (_rc != TRIPS_OK) return _rc;       \
    } while (0)

    // crowded: the last pass that reported back saw more than kHotKey visible points in one (view, bin, tile) group
    STAGE(ctx, TRIPS_STAGE_BIN_POINTS, bin_count_launches((int)N, B), st,
          launch_bin_count(sp, cams, g, *params, B, fb, sizes == Sizes::wait ? ~0ull : (unsigned long long)ctx->entry_cap,
                           PassGuess{sizes == Sizes::look, ctx->crowded, entries}, ctx->sm_count, st));
    if (sizes == Sizes::wait)
    {
        CU_CHECK(ctx, cudaMemcpyAsync(h_stats, ctx->stats.p, sizeof(DevStats), cudaMemcpyDeviceToHost, st));
        CU_CHECK(ctx, cudaStreamSynchronize(st));
        STEP(grow_entries());
        STEP(write_lists(true));
        CU_CHECK(ctx, cudaStreamSynchronize(st));
        STEP(grow_lists());
        STEP(render());
    }
    else
    {
        STEP(write_lists(false));
        CU_CHECK(ctx, cudaEventRecord(ctx->totals_ev, st));
        ctx->pending = sizes == Sizes::later;
        STEP(render());
    }
    if (sizes == Sizes::look)
    {
        CU_CHECK(ctx, cudaEventSynchronize(ctx->totals_ev));
        const GivenUp given_up = h_stats->given_up;
        ctx->crowded           = h_stats->max_key >= kHotKey;
        if (given_up == kGivenUpEntries)
        {
            STEP(grow_entries());
            STAGE(ctx, TRIPS_STAGE_BIN_POINTS, 1, st, launch_place_views(B, fb, true, st));
            STEP(write_lists(true));
            CU_CHECK(ctx, cudaStreamSynchronize(st));
        }
        if (given_up != kNotGivenUp)
        {
            STEP(grow_lists());
            if (given_up == kGivenUpLists) STAGE(ctx, TRIPS_STAGE_SCAN, 1, st, launch_place_views(B, fb, false, st));
            STEP(render());
        }
    }
#undef STEP
    if (sizes != Sizes::later)
    {
        ctx->need_entries = h_stats->visible;
        ctx->need_frags   = h_stats->frag_need;
        ctx->host_stats.visible_points += (int64_t)h_stats->visible;
        ctx->host_stats.fragments += (int64_t)h_stats->frag_need;
        ctx->host_stats.kept_fragments += (int64_t)h_stats->kept;
        ctx->host_stats.max_list_length = std::max<int64_t>(ctx->host_stats.max_list_length, (int64_t)h_stats->max_len);
        ctx->host_stats.culled_point_blocks += (int64_t)h_stats->culled_blocks;
    }
    ctx->B       = B;
    return TRIPS_OK;
}

int trips_forward(TripsContext* ctx, const TripsScene* scene, const TripsView* views, int n_views,
                  const TripsRenderParams* params, float* const* out_layers, void* stream)
{
    if (!ctx) return TRIPS_ERR_INVALID_ARG;
    if (!scene || !views || !params || !out_layers || n_views < 1) return fail(ctx, TRIPS_ERR_INVALID_ARG, "null argument");
    if (params->num_layers < 1 || params->num_layers > TRIPS_MAX_LAYERS) return fail(ctx, TRIPS_ERR_INVALID_ARG, "num_layers must be 1..8");
    if (params->k_keep < 1 || params->k_keep > TRIPS_MAX_KEEP) return fail(ctx, TRIPS_ERR_INVALID_ARG, "k_keep must be 1..16");
    if (!valid_channels(scene->channels)) return fail(ctx, TRIPS_ERR_INVALID_ARG, "channels must be 3, 4, 6, 8 or 16");
    if (scene->n_points < 0 || scene->n_tex < 1 || scene->n_images < 1 || scene->n_cameras < 1)
        return fail(ctx, TRIPS_ERR_INVALID_ARG, "bad scene sizes");
    if (scene->n_points > 0 && (!scene->position || !scene->point_size)) return fail(ctx, TRIPS_ERR_INVALID_ARG, "null point arrays");
    if (!scene->texture || !scene->confidence || !scene->background || !scene->poses || !scene->intrinsics)
        return fail(ctx, TRIPS_ERR_INVALID_ARG, "null scene arrays");
    if (!scene->index && scene->n_tex < scene->n_points) return fail(ctx, TRIPS_ERR_INVALID_ARG, "identity index needs n_tex >= n_points");
    const int w = views[0].w, h = views[0].h;
    if (w < 2 || h < 2) return fail(ctx, TRIPS_ERR_INVALID_ARG, "image must be at least 2x2");
    for (int b = 0; b < n_views; ++b)
    {
        if (views[b].w != w || views[b].h != h) return fail(ctx, TRIPS_ERR_INVALID_ARG, "all views of a call must share (w, h)");
        if (views[b].camera_model_type != 0) return fail(ctx, TRIPS_ERR_UNSUPPORTED, "only the pinhole camera model is implemented");
        if (views[b].image_index < 0 || views[b].image_index >= scene->n_images || views[b].camera_index < 0 ||
            views[b].camera_index >= scene->n_cameras)
            return fail(ctx, TRIPS_ERR_INVALID_ARG, "view index out of range");
    }
    for (int l = 0; l < params->num_layers; ++l)
        if (!out_layers[l]) return fail(ctx, TRIPS_ERR_INVALID_ARG, "null output layer");
    cudaStream_t st = (cudaStream_t)stream;
    ctx->have_forward = false;
    {
        const int rs = resolve_pending(ctx);
        if (rs != TRIPS_OK) return rs;
    }
    Geom g{};
    if (!make_geom(w, h, params->num_layers, g)) return fail(ctx, TRIPS_ERR_TOO_LARGE, "pyramid has more than 2^30 pixels");
    const int B    = n_views;
    const size_t N = (size_t)scene->n_points;
    if (N * 4ull * g.L >= (1ull << 32)) return fail(ctx, TRIPS_ERR_TOO_LARGE, "a view could hold more than 2^32 fragments");
    if ((unsigned long long)B * (unsigned long long)g.n_tiles >= (1ull << 32)) return fail(ctx, TRIPS_ERR_TOO_LARGE, "too many pixel tiles");

    const SizeKey key{scene->n_points, B, w, h, params->num_layers, scene->channels, params->train,
                      (params->use_layer_point_size ? 1 : 0) | (params->render_points_in_all_lower_resolutions ? 2 : 0)};
    ctx->host_stats        = TripsStats{};
    ctx->host_stats.pixels = (int64_t)g.P * B;
    ctx->geom              = g;
    ctx->params            = *params;
    ctx->N                 = (int)N;
    ctx->n_tex             = scene->n_tex;
    ctx->C                 = scene->channels;
    if (params->train)
    {
        // Steady state of a training loop: same shapes as the previous training call.  The buffers keep the capacity that
        // call needed (x 1.25), grown here if its totals (read above, long after they were produced) say so.
        bool steady = ctx->have_sizes && key == ctx->size_key;
        if (steady)
        {
            if (ctx->need_entries > ctx->entry_cap)
                steady = ensure_entries(ctx, (size_t)ctx->need_entries, scene->channels, kGrowth) == cudaSuccess;
            if (steady && (size_t)ctx->need_frags * sizeof(uint4) > ctx->frags.bytes)
                steady = ensure(ctx->frags, (size_t)ctx->need_frags * sizeof(uint4), kGrowth) == cudaSuccess;
            (void)cudaGetLastError();
        }
        const int rc = forward_views(ctx, scene, views, B, params, g, out_layers, 0, scene->dropout, st, steady ? Sizes::later : Sizes::wait);
        if (rc != TRIPS_OK)
        {
            ctx->have_sizes = false;
            return rc;
        }
        ctx->size_key   = key;
        ctx->have_sizes = true;
    }
    else
    {
        // Nothing is kept for a backward pass: the views are rendered kEvalSubBatch at a time, so the scratch of a call
        // with many views (a batch of 64 evaluation views) is that of kEvalSubBatch views.  The inspection calls then
        // describe the last sub-batch.
        ctx->have_sizes = false;
        for (int b0 = 0; b0 < B; b0 += kEvalSubBatch)
        {
            const int nb = std::min(kEvalSubBatch, B - b0);
            // With buffers from an earlier pass at hand everything is launched at once and the sizes are looked at afterwards, while the
            // collect pass and the blend run: waiting for them in between left the GPU idle twice per pass (640x480 frame of 200 k
            // points 209 -> 185 us, 1080p frame of 6 M 774 -> 758, the latter with the binning pass made faster in between).
            const bool buffers = ctx->frags.p && ctx->entries.p && ctx->entry_C == scene->channels;
            const int rc = forward_views(ctx, scene, views + b0, nb, params, g, out_layers, (size_t)b0, nullptr, st, buffers ? Sizes::look : Sizes::wait);
            if (rc != TRIPS_OK) return rc;
        }
    }
    ctx->have_forward = true;
    return TRIPS_OK;
}

int trips_backward(TripsContext* ctx, const TripsScene* scene, const float* const* grad_layers, const TripsGrads* grads,
                   void* stream)
{
    if (!ctx) return TRIPS_ERR_INVALID_ARG;
    if (!scene || !grad_layers || !grads) return fail(ctx, TRIPS_ERR_INVALID_ARG, "null argument");
    if (!ctx->have_forward || !ctx->params.train) return fail(ctx, TRIPS_ERR_NO_FORWARD, "no training forward pass to differentiate");
    if (scene->n_points != ctx->N || scene->n_tex != ctx->n_tex || scene->channels != ctx->C)
        return fail(ctx, TRIPS_ERR_INVALID_ARG, "scene sizes differ from the forward pass");
    const Geom& g = ctx->geom;
    for (int l = 0; l < g.L; ++l)
        if (!grad_layers[l]) return fail(ctx, TRIPS_ERR_INVALID_ARG, "null gradient layer");
    cudaStream_t st = (cudaStream_t)stream;
    const int B = ctx->B, C = ctx->C;
    const size_t N = (size_t)ctx->N;

    const size_t GS = (size_t)egrad_stride(C);
    CU_CHECK(ctx, ensure(ctx->egrad, sizeof(float) * GS * ctx->entry_cap + 16));  // one row per entry the arrays can hold
    const size_t small_bytes = sizeof(double) * (TRIPS_MAX_CHANNELS + (size_t)B * 19) + sizeof(unsigned) * kTileCounters * kTileCounterPitch;  // background | per view: 6 pose, 5 pinhole, 8 distortion | work counters
    CU_CHECK(ctx, ensure(ctx->g_small, small_bytes));
    BwdBuffers bb;
    bb.egrad        = (float*)ctx->egrad.p;
    bb.g_bg         = (double*)ctx->g_small.p;
    bb.g_pose       = bb.g_bg + TRIPS_MAX_CHANNELS;
    bb.g_k          = bb.g_pose + (size_t)B * 6;
    bb.g_dis        = bb.g_k + (size_t)B * 5;
    bb.ticket       = (unsigned int*)(bb.g_dis + (size_t)B * 8);
    ScenePtrs sp  = scene_ptrs(scene);
    FwdBuffers fb = fwd_buffers(ctx, B);
    // all accumulators start from zero (timed with the gradient bookkeeping of the unpack stage)
    auto clear_accumulators = [&]() -> cudaError_t {
        cudaError_t e = cudaSuccess;
        e = cudaMemsetAsync(ctx->g_small.p, 0, small_bytes, st);
        if (grads->pose_tangent && e == cudaSuccess) e = cudaMemsetAsync(grads->pose_tangent, 0, sizeof(double) * 6 * scene->n_images, st);
        if (grads->intrinsics && e == cudaSuccess) e = cudaMemsetAsync(grads->intrinsics, 0, sizeof(float) * 13 * scene->n_cameras, st);
        if (N > 0 && e == cudaSuccess) e = launch_zero_entry_rows(C, B, fb, bb, ctx->sm_count, st);
        return e;
    };
    STAGE(ctx, TRIPS_STAGE_UNPACK, N > 0 ? 1 : 0, st, clear_accumulators());
    ConstLayerPtrs gin{};
    for (int l = 0; l < g.L; ++l) gin.p[l] = grad_layers[l];
    const bool cam_grads = grads->pose_tangent || grads->intrinsics;
    STAGE(ctx, TRIPS_STAGE_BACKWARD, 1, st,
          launch_blend_backward(sp, (const CamConst*)ctx->cams.p, g, ctx->params, B, fb, bb, gin, ctx->need_entries, ctx->sm_count, st));
    const int n_unpack = (N > 0 ? unpack_launches(B, fb.entry_views) + (cam_grads ? 1 : 0) : 0) + 1;
    STAGE(ctx, TRIPS_STAGE_UNPACK, n_unpack, st,
          launch_unpack_grads(sp, (const CamConst*)ctx->cams.p, B, fb, bb, *grads, ctx->params, ctx->sm_count, st));
    return TRIPS_OK;
}

uint32_t trips_last_status(TripsContext* ctx, void* stream)
{
    if (!ctx || !ctx->stats.p) return 0;
    DevStats s{};
    cudaStream_t st = (cudaStream_t)stream;
    if (cudaMemcpyAsync(&s, ctx->stats.p, sizeof(s), cudaMemcpyDeviceToHost, st) != cudaSuccess) return 0;
    if (cudaStreamSynchronize(st) != cudaSuccess) return 0;
    unsigned zero = 0;
    cudaMemcpyAsync((char*)ctx->stats.p + offsetof(DevStats, status), &zero, sizeof(unsigned), cudaMemcpyHostToDevice, st);
    cudaStreamSynchronize(st);
    return s.status;
}

int trips_get_stats(TripsContext* ctx, TripsStats* out, void* stream)
{
    (void)stream;
    if (!ctx || !out) return TRIPS_ERR_INVALID_ARG;
    if (!ctx->have_forward) return fail(ctx, TRIPS_ERR_NO_FORWARD, "no forward pass");
    {
        const int rs = resolve_pending(ctx);  // waits for the totals of a call that did not wait for them itself
        if (rs != TRIPS_OK) return rs;
    }
    *out = ctx->host_stats;
    return TRIPS_OK;
}

int trips_adam_step(TripsContext* ctx, const TripsAdamTensor* tensors, int n_tensors, void* stream)
{
    if (!ctx) return TRIPS_ERR_INVALID_ARG;
    if (!tensors || n_tensors < 1) return fail(ctx, TRIPS_ERR_INVALID_ARG, "no tensors");
    cudaStream_t st = (cudaStream_t)stream;
    std::vector<int64_t> start(n_tensors + 1, 0);
    for (int i = 0; i < n_tensors; ++i)
    {
        const TripsAdamTensor& t = tensors[i];
        if (t.n < 0 || (t.n > 0 && (!t.weights || !t.gradients || !t.first_moments || !t.second_moments || !t.steps)))
            return fail(ctx, TRIPS_ERR_INVALID_ARG, "null tensor in Adam group");
        start[i + 1] = start[i] + (t.n + kAdamPerBlock - 1) / kAdamPerBlock;
    }
    if (start[n_tensors] >= (1ll << 31)) return fail(ctx, TRIPS_ERR_TOO_LARGE, "too many elements for one Adam launch");
    if (n_tensors <= kAdamTable)
    {
        STAGE(ctx, TRIPS_STAGE_ADAM, 1, st, launch_adam_by_value(tensors, start.data(), n_tensors, st));
        return TRIPS_OK;
    }
    const size_t tab_bytes   = sizeof(TripsAdamTensor) * n_tensors;
    const size_t tab_aligned = (tab_bytes + 15) & ~(size_t)15;
    CU_CHECK(ctx, ensure(ctx->adam_tab, tab_aligned + sizeof(int64_t) * (n_tensors + 1)));
    CU_CHECK(ctx, cudaMemcpyAsync(ctx->adam_tab.p, tensors, tab_bytes, cudaMemcpyHostToDevice, st));
    CU_CHECK(ctx, cudaMemcpyAsync((char*)ctx->adam_tab.p + tab_aligned, start.data(), sizeof(int64_t) * (n_tensors + 1),
                                  cudaMemcpyHostToDevice, st));
    STAGE(ctx, TRIPS_STAGE_ADAM, 1, st,
          launch_adam((const TripsAdamTensor*)ctx->adam_tab.p, (const int64_t*)((char*)ctx->adam_tab.p + tab_aligned), n_tensors,
                      start[n_tensors], st));
    return TRIPS_OK;
}

int trips_resize_points(TripsContext* ctx, const int64_t* indices_to_remove, int64_t n_remove, int64_t n_points, int64_t n_new,
                        const TripsPointTensor* tensors, int n_tensors, void* stream)
{
    if (!ctx) return TRIPS_ERR_INVALID_ARG;
    if (n_points < 0 || n_remove < 0 || n_remove > n_points || n_new < n_points - n_remove) return fail(ctx, TRIPS_ERR_INVALID_ARG, "bad point counts");
    if (n_remove > 0 && !indices_to_remove) return fail(ctx, TRIPS_ERR_INVALID_ARG, "null removal list");
    if (n_tensors < 0 || n_tensors > TRIPS_MAX_POINT_TENSORS || (n_tensors > 0 && !tensors)) return fail(ctx, TRIPS_ERR_INVALID_ARG, "bad tensor table");
    if (n_points >= (1ll << 32) || n_new >= (1ll << 32)) return fail(ctx, TRIPS_ERR_TOO_LARGE, "more than 2^32 points");
    for (int i = 0; i < n_tensors; ++i)
    {
        const TripsPointTensor& t = tensors[i];
        if (t.rows < 1 || (t.elem_bytes != 4 && t.elem_bytes != 8)) return fail(ctx, TRIPS_ERR_INVALID_ARG, "rows >= 1 and 4- or 8-byte elements");
        if ((n_new > 0 && !t.dst) || (n_points > n_remove && !t.src)) return fail(ctx, TRIPS_ERR_INVALID_ARG, "null tensor");
    }
    cudaStream_t st = (cudaStream_t)stream;
    CU_CHECK(ctx, ensure_stats(ctx, st));
    CU_CHECK(ctx, ensure(ctx->resize_scratch, resize_scratch_bytes(n_points)));
    STAGE(ctx, TRIPS_STAGE_RESIZE, 5, st,
          launch_resize_points(indices_to_remove, n_remove, n_points, n_new, tensors, n_tensors, ctx->resize_scratch.p, (DevStats*)ctx->stats.p,
                               ctx->sm_count, st));
    ctx->have_forward = false;  // the scratch of the last forward pass describes the old point set
    return TRIPS_OK;
}

int trips_fused_reduce_adam(TripsContext* ctx, const float* const* grad_ptrs, float* const* param_ptrs, int world, int rank,
                            const TripsAdamSegment* segments, int n_segments, int64_t lo, int64_t hi, float* first_moments,
                            float* second_moments, int32_t* steps, void* stream)
{
    if (!ctx) return TRIPS_ERR_INVALID_ARG;
    if (!grad_ptrs || !param_ptrs || !segments) return fail(ctx, TRIPS_ERR_INVALID_ARG, "null argument");
    if (world < 1 || world > TRIPS_MAX_RANKS || rank < 0 || rank >= world) return fail(ctx, TRIPS_ERR_INVALID_ARG, "bad world / rank");
    if (n_segments < 1 || n_segments > TRIPS_MAX_SEGMENTS || segments[0].offset != 0) return fail(ctx, TRIPS_ERR_INVALID_ARG, "bad segment table");
    for (int s = 1; s < n_segments; ++s)
        if (segments[s].offset <= segments[s - 1].offset) return fail(ctx, TRIPS_ERR_INVALID_ARG, "segments must be sorted by offset");
    if (lo < 0 || hi < lo) return fail(ctx, TRIPS_ERR_INVALID_ARG, "bad slice");
    for (int r = 0; r < world; ++r)
        if (!grad_ptrs[r] || !param_ptrs[r] || (((uintptr_t)grad_ptrs[r] | (uintptr_t)param_ptrs[r]) & 15))
            return fail(ctx, TRIPS_ERR_INVALID_ARG, "flat buffers must be non-null and 16-byte aligned");
    if (hi > lo && (!first_moments || !second_moments || !steps)) return fail(ctx, TRIPS_ERR_INVALID_ARG, "null optimizer state");
    cudaStream_t st = (cudaStream_t)stream;
    STAGE(ctx, TRIPS_STAGE_FUSED_ADAM, hi > lo ? 1 : 0, st,
          launch_fused_reduce_adam(grad_ptrs, param_ptrs, world, rank, segments, n_segments, lo, hi, first_moments, second_moments,
                                   steps, ctx->sm_count, st));
    return TRIPS_OK;
}

int trips_fused_reduce_adam_multicast(TripsContext* ctx, const float* grad_multicast, float* param_multicast, const float* param_local,
                                      const TripsAdamSegment* segments, int n_segments, int64_t lo, int64_t hi, float* first_moments,
                                      float* second_moments, int32_t* steps, void* stream)
{
    if (!ctx) return TRIPS_ERR_INVALID_ARG;
    if (!grad_multicast || !param_multicast || !param_local || !segments) return fail(ctx, TRIPS_ERR_INVALID_ARG, "null argument");
    if (n_segments < 1 || n_segments > TRIPS_MAX_SEGMENTS || segments[0].offset != 0) return fail(ctx, TRIPS_ERR_INVALID_ARG, "bad segment table");
    for (int s = 1; s < n_segments; ++s)
        if (segments[s].offset <= segments[s - 1].offset) return fail(ctx, TRIPS_ERR_INVALID_ARG, "segments must be sorted by offset");
    if (lo < 0 || hi < lo || ((lo | hi) & 3)) return fail(ctx, TRIPS_ERR_INVALID_ARG, "the slice must start and end on a multiple of 4 elements");
    if (((uintptr_t)grad_multicast | (uintptr_t)param_multicast | (uintptr_t)param_local) & 15)
        return fail(ctx, TRIPS_ERR_INVALID_ARG, "flat buffers must be 16-byte aligned");
    if (hi > lo && (!first_moments || !second_moments || !steps)) return fail(ctx, TRIPS_ERR_INVALID_ARG, "null optimizer state");
    cudaStream_t st = (cudaStream_t)stream;
    STAGE(ctx, TRIPS_STAGE_FUSED_ADAM, hi > lo ? 1 : 0, st,
          launch_fused_multicast_adam(grad_multicast, param_multicast, param_local, segments, n_segments, lo, hi, first_moments,
                                      second_moments, steps, ctx->sm_count, st));
    return TRIPS_OK;
}

int trips_enable_stage_timers(TripsContext* ctx, int enable)
{
    if (!ctx) return TRIPS_ERR_INVALID_ARG;
    ctx->timers.enabled = enable != 0;
    return TRIPS_OK;
}

int trips_get_stage_times(TripsContext* ctx, double* ms, int64_t* timed_calls, int64_t* kernel_launches, int reset)
{
    if (!ctx) return TRIPS_ERR_INVALID_ARG;
    ctx->timers.collect();
    for (int i = 0; i < TRIPS_NUM_STAGES; ++i)
    {
        if (ms) ms[i] = ctx->timers.ms[i];
        if (timed_calls) timed_calls[i] = ctx->timers.timed[i];
        if (kernel_launches) kernel_launches[i] = ctx->timers.launches[i];
        if (reset)
        {
            ctx->timers.ms[i]       = 0.0;
            ctx->timers.timed[i]    = 0;
            ctx->timers.launches[i] = 0;
        }
    }
    return TRIPS_OK;
}

const char* trips_stage_name(int stage)
{
    static const char* names[TRIPS_NUM_STAGES] = {"setup_cams", "bin_points", "count", "scan", "collect", "sort_blend",
                                                  "blend_backward", "unpack_grads", "adam", "l1_loss", "fused_reduce_adam", "resize_points"};
    return (stage >= 0 && stage < TRIPS_NUM_STAGES) ? names[stage] : "?";
}

int trips_l1_loss_backward(TripsContext* ctx, const float* const* out_layers, const float* const* target_layers,
                           float* const* grad_layers, const int64_t* layer_numel, int num_layers, double* loss_out,
                           void* stream)
{
    if (!ctx) return TRIPS_ERR_INVALID_ARG;
    if (!out_layers || !target_layers || !grad_layers || !layer_numel || !loss_out || num_layers < 1 ||
        num_layers > TRIPS_MAX_LAYERS)
        return fail(ctx, TRIPS_ERR_INVALID_ARG, "bad l1 loss arguments");
    cudaStream_t st = (cudaStream_t)stream;
    L1Args a{};
    int64_t total = 0;
    for (int l = 0; l < num_layers; ++l)
    {
        if (!out_layers[l] || !target_layers[l] || !grad_layers[l] || layer_numel[l] < 0)
            return fail(ctx, TRIPS_ERR_INVALID_ARG, "null layer in l1 loss");
        a.out[l]    = out_layers[l];
        a.target[l] = target_layers[l];
        a.grad[l]   = grad_layers[l];
        a.start[l]  = total;
        total += layer_numel[l];
    }
    for (int l = num_layers; l <= TRIPS_MAX_LAYERS; ++l) a.start[l] = total;
    a.L = num_layers;
    CU_CHECK(ctx, cudaMemsetAsync(loss_out, 0, sizeof(double), st));
    STAGE(ctx, TRIPS_STAGE_LOSS, 1, st, launch_l1_loss(a, total, loss_out, ctx->sm_count, st));
    return TRIPS_OK;
}

int trips_debug_points(TripsContext* ctx, int view, float* depth, int32_t* nlayers, float* record, void* stream)
{
    if (!ctx) return TRIPS_ERR_INVALID_ARG;
    if (!ctx->have_forward) return fail(ctx, TRIPS_ERR_NO_FORWARD, "no forward pass");
    if (view < 0 || view >= ctx->B) return fail(ctx, TRIPS_ERR_INVALID_ARG, "view out of range");
    cudaStream_t st = (cudaStream_t)stream;
    const size_t N = (size_t)ctx->N, ES = 8;  // the two float4 of an entry's head
    unsigned long long eb[2];
    CU_CHECK(ctx, cudaMemcpyAsync(eb, (unsigned long long*)ctx->entry_base.p + view, sizeof(eb), cudaMemcpyDeviceToHost, st));
    CU_CHECK(ctx, cudaStreamSynchronize(st));
    const size_t n = (size_t)(eb[1] - eb[0]);
    const size_t TS = (size_t)tail_stride(ctx->C);
    std::vector<float> e(n * ES), tl(n * TS);
    if (n)
    {
        CU_CHECK(ctx, cudaMemcpyAsync(e.data(), (float*)ctx->entries.p + eb[0] * ES, sizeof(float) * n * ES, cudaMemcpyDeviceToHost, st));
        CU_CHECK(ctx, cudaMemcpyAsync(tl.data(), (float*)ctx->entries.p + 8 * ctx->entry_cap + eb[0] * TS, sizeof(float) * n * TS,
                                      cudaMemcpyDeviceToHost, st));
    }
    CU_CHECK(ctx, cudaStreamSynchronize(st));
    // the per-point arrays of the reference (depth = -1 for culled points) are rebuilt from the view's entries
    for (size_t i = 0; i < N; ++i)
    {
        if (depth) depth[i] = -1.f;
        if (nlayers) nlayers[i] = 0;
        if (record) record[4 * i] = record[4 * i + 1] = record[4 * i + 2] = record[4 * i + 3] = 0.f;
    }
    for (size_t k = 0; k < n; ++k)
    {
        const float* en = e.data() + k * ES;
        int32_t pid, nl;
        memcpy(&pid, en + 4, 4);
        memcpy(&nl, en + 7, 4);
        if (pid < 0 || (size_t)pid >= N) continue;
        if (depth) depth[pid] = en[5];
        if (nlayers) nlayers[pid] = nl;
        if (record)
        {
            record[4 * (size_t)pid + 0] = en[0];
            record[4 * (size_t)pid + 1] = en[1];
            record[4 * (size_t)pid + 2] = en[2];
            record[4 * (size_t)pid + 3] = tl[k * TS + 3];  // texture index
        }
    }
    return TRIPS_OK;
}

// List lengths of a view, its number of fragments and where the lists start in its part of the list buffer.  An error when the lists
// do not fill that part exactly.
static int read_lists(TripsContext* ctx, int view, cudaStream_t st, std::vector<uint32_t>& counts, std::vector<uint32_t>& starts, unsigned long long (&vb)[2])
{
    if (!ctx->have_forward) return fail(ctx, TRIPS_ERR_NO_FORWARD, "no forward pass");
    if (view < 0 || view >= ctx->B) return fail(ctx, TRIPS_ERR_INVALID_ARG, "view out of range");
    const size_t P = (size_t)ctx->geom.P, off = (size_t)view * P;
    counts.resize(P), starts.resize(P);
    CU_CHECK(ctx, cudaMemcpyAsync(vb, (unsigned long long*)ctx->view_base.p + view, sizeof(vb), cudaMemcpyDeviceToHost, st));
    CU_CHECK(ctx, cudaMemcpyAsync(counts.data(), (const uint32_t*)((const char*)ctx->zeroed.p + ctx->zero_counts) + off, sizeof(uint32_t) * P, cudaMemcpyDeviceToHost, st));
    CU_CHECK(ctx, cudaMemcpyAsync(starts.data(), (uint32_t*)ctx->offsets.p + off, sizeof(uint32_t) * P, cudaMemcpyDeviceToHost, st));
    CU_CHECK(ctx, cudaStreamSynchronize(st));
    if (vb[1] == vb[0])  // no fragments, or the view did not fit: the collect pass has skipped it
    {
        starts.assign(P, 0);
        return TRIPS_OK;
    }
    for (size_t i = 0; i < P; ++i) starts[i] -= counts[i];  // the collect pass advanced the starts to the list ends
    if (!lists_cover(starts.data(), counts.data(), P, vb[1] - vb[0]))
        return fail(ctx, TRIPS_ERR_CUDA, "the lists of the view overlap or leave their part of the list buffer (internal error)");
    return TRIPS_OK;
}

int trips_debug_lists(TripsContext* ctx, int view, int32_t* counts, int64_t* offsets, uint64_t* frags, int64_t* n_frags,
                      void* stream)
{
    if (!ctx) return TRIPS_ERR_INVALID_ARG;
    cudaStream_t st = (cudaStream_t)stream;
    std::vector<uint32_t> c, s;
    unsigned long long vb[2];
    const int rc = read_lists(ctx, view, st, c, s, vb);
    if (rc != TRIPS_OK) return rc;
    const unsigned long long nf = vb[1] - vb[0];
    if (n_frags) *n_frags = (int64_t)nf;
    // the lists lie in the buffer in the order in which their blocks came; here they follow one another in pixel order
    int64_t next = 0;
    for (size_t i = 0; i < c.size(); ++i)
    {
        if (counts) counts[i] = (int32_t)c[i];
        if (offsets) offsets[i] = next;
        next += c[i];
    }
    if (frags && nf)
    {
        std::vector<uint4> f(nf);
        CU_CHECK(ctx, cudaMemcpyAsync(f.data(), (uint4*)ctx->frags.p + vb[0], sizeof(uint4) * nf, cudaMemcpyDeviceToHost, st));
        CU_CHECK(ctx, cudaStreamSynchronize(st));
        for (size_t i = 0; i < c.size(); ++i)
            for (size_t k = 0; k < c[i]; ++k) *frags++ = ((uint64_t)f[s[i] + k].y << 32) | f[s[i] + k].x;
    }
    return TRIPS_OK;
}

int trips_debug_list_starts(TripsContext* ctx, int view, int64_t* starts, void* stream)
{
    if (!ctx) return TRIPS_ERR_INVALID_ARG;
    if (!starts) return fail(ctx, TRIPS_ERR_INVALID_ARG, "null argument");
    std::vector<uint32_t> c, s;
    unsigned long long vb[2];
    const int rc = read_lists(ctx, view, (cudaStream_t)stream, c, s, vb);
    if (rc != TRIPS_OK) return rc;
    std::copy(s.begin(), s.end(), starts);
    return TRIPS_OK;
}

int trips_debug_records(TripsContext* ctx, int view, int32_t* nrec, int32_t* rec_pid, float* rec_alpha, void* stream)
{
    if (!ctx) return TRIPS_ERR_INVALID_ARG;
    if (!ctx->have_forward || !ctx->params.train) return fail(ctx, TRIPS_ERR_NO_FORWARD, "no training forward pass");
    if (view < 0 || view >= ctx->B) return fail(ctx, TRIPS_ERR_INVALID_ARG, "view out of range");
    cudaStream_t st = (cudaStream_t)stream;
    const Geom& g = ctx->geom;
    const size_t T = (size_t)g.n_tiles;
    std::vector<uint8_t> n(T * 32);
    std::vector<uint2> r(T * 16 * 32);
    const size_t ES = 8;  // the two float4 of an entry's head
    unsigned long long eb[2];
    CU_CHECK(ctx, cudaMemcpyAsync(eb, (unsigned long long*)ctx->entry_base.p + view, sizeof(eb), cudaMemcpyDeviceToHost, st));
    CU_CHECK(ctx, cudaMemcpyAsync(n.data(), (uint8_t*)ctx->rec_n.p + (size_t)view * T * 32, n.size(), cudaMemcpyDeviceToHost, st));
    CU_CHECK(ctx, cudaMemcpyAsync(r.data(), (uint2*)ctx->records.p + (size_t)view * T * 16 * 32, sizeof(uint2) * r.size(), cudaMemcpyDeviceToHost, st));
    CU_CHECK(ctx, cudaStreamSynchronize(st));
    const size_t n_e = (size_t)(eb[1] - eb[0]);
    std::vector<float> e(n_e * ES);
    if (n_e) CU_CHECK(ctx, cudaMemcpyAsync(e.data(), (float*)ctx->entries.p + eb[0] * ES, sizeof(float) * n_e * ES, cudaMemcpyDeviceToHost, st));
    CU_CHECK(ctx, cudaStreamSynchronize(st));
    // the device holds the records by tile, rank and lane and with the entry index of the fragment's point; report them
    // per pixel and with the point id
    for (int l = 0; l < g.L; ++l)
        for (int y = 0; y < g.H[l]; ++y)
            for (int x = 0; x < g.W[l]; ++x)
            {
                int tile, lane;
                pixel_tile(g, l, x, y, tile, lane);
                const size_t p = (size_t)g.base[l] + (size_t)y * g.W[l] + x;
                const int m    = n[(size_t)tile * 32 + lane];
                if (nrec) nrec[p] = m;
                for (int j = 0; j < 16; ++j)
                {
                    const uint2 q   = r[((size_t)tile * 16 + j) * 32 + lane];
                    int32_t pid     = -1;
                    float a         = -1.f;
                    if (j < m)
                    {
                        if (q.x < n_e) memcpy(&pid, e.data() + (size_t)q.x * ES + 4, 4);
                        memcpy(&a, &q.y, 4);
                    }
                    if (rec_pid) rec_pid[p * 16 + j] = pid;
                    if (rec_alpha) rec_alpha[p * 16 + j] = a;
                }
            }
    return TRIPS_OK;
}

int trips_debug_nearest(TripsContext* ctx, const uint64_t* keys, int n, uint32_t* positions, int* gatherings, void* stream)
{
    if (!ctx) return TRIPS_ERR_INVALID_ARG;
    if (!keys || n < 16) return fail(ctx, TRIPS_ERR_INVALID_ARG, "at least 16 keys");
    cudaStream_t st = (cudaStream_t)stream;
    DevBuf buf;
    const size_t key_bytes = sizeof(uint64_t) * (size_t)n;
    uint32_t result[17]    = {};
    auto run = [&]() -> cudaError_t {
        cudaError_t e = ensure(buf, key_bytes + sizeof(result));
        uint32_t* out = (uint32_t*)((char*)buf.p + key_bytes);
        if (e == cudaSuccess) e = cudaMemcpyAsync(buf.p, keys, key_bytes, cudaMemcpyHostToDevice, st);
        if (e == cudaSuccess) e = launch_nearest_16((const unsigned long long*)buf.p, (uint32_t)n, out, st);
        if (e == cudaSuccess) e = cudaMemcpyAsync(result, out, sizeof(result), cudaMemcpyDeviceToHost, st);
        const cudaError_t s = cudaStreamSynchronize(st);
        return e != cudaSuccess ? e : s;
    };
    const cudaError_t e = run();
    free_buf(buf);
    CU_CHECK(ctx, e);
    if (positions) memcpy(positions, result, sizeof(uint32_t) * 16);
    if (gatherings) *gatherings = (int)result[16];
    return TRIPS_OK;
}

}  // extern "C"
