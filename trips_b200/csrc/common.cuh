// Internal declarations shared by the kernels and the C ABI of libtrips_b200.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

#include "../../include/trips_b200.h"
#include "trips_math.h"

namespace trips
{
constexpr float kAlphaCut = 0.001f;  // ALPHA_DEST_CUTOFF, RenderForward.cu:907
constexpr unsigned kFull  = 0xffffffffu;
constexpr int kBinShift   = 5;   // visible points are bucketed by 32x32-pixel screen bins of layer 0
constexpr int kTileW      = 8;   // one warp renders / differentiates an 8x4 pixel tile
constexpr int kTileH      = 4;
constexpr uint32_t kNoEntry = 0xffffffffu;  // a point that is not visible in a view
// Point-to-entry table of a training call: at most this many bytes.  It has 4 bytes per point and view, also where most points
// are visible in few of the views; a call of 20 M points reaches the limit with 53 views.
constexpr size_t kEntryTableBytes = (size_t)4 << 30;
constexpr int kViewGroup  = 16;  // views whose camera constants are in shared memory at a time in the binning passes (one launch per group)
// Lists longer than kHeavyList get their 16 nearest fragments moved to the front by a block of their own.  sort_blend, ms, at 128 /
// 256 / 512 / 1024 / 4096: 20 M points at 1440p x 2 views 1.17 / 0.89 / 0.75 / 0.80 / 0.79, 3 M points in 64x64 pixels x 4 views
// 0.54 / 0.54 / 0.54 / 0.59 / 1.31, 1.6 M points in 53x28 pixels x 8 views 0.70 / 0.71 / 0.73 / 0.79 / 1.10; 64 views of 10 M points 23.5
// at 128 and 22.9 from 256 on.
constexpr int kHeavyList  = 512;
constexpr int kHeavyPart  = 8192;     // longer ones are shared by several blocks, each with a part of at most this many fragments ...
constexpr int kHeavyParts = 256;      // ... or by this many blocks
constexpr int kHeavyCap   = 1 << 17;  // such lists and parts per call the pre-selection handles at most; beyond that the blend walks the lists itself
constexpr int kHeavyShared = 1 << 16; // parts of shared lists per call at most; beyond that a long list gets one block

// Pyramid geometry shared by all views of a call.
struct Geom
{
    int L;
    int W[TRIPS_MAX_LAYERS];            // ceil-halved layer sizes (PointRenderer.cu:385-389)
    int H[TRIPS_MAX_LAYERS];
    float inside_x[TRIPS_MAX_LAYERS];   // layer-0 positions below these have their footprint inside layers 0..l: min (W_k - 1) 2^k
    float inside_y[TRIPS_MAX_LAYERS];
    int base[TRIPS_MAX_LAYERS + 1];     // first pixel of every layer in the per-view pixel arrays (row-major)
    int P;                              // pixels per view
    // Tile order of a view: first the 64x64-pixel regions of layer 0 in row-major order, each with its tiles of
    // layers 0..reg_layers-1 (a region is (64 >> l) pixels wide on layer l), so that the entries of a region stay in L2
    // while all its fine layers are processed; then the remaining coarse layers, layer by layer.
    int reg_layers;                     // min(L, 4)
    int reg_x;                          // regions per row
    int reg_tiles;                      // tiles of one region: 128 + 32 + 8 + 2 for four layers
    int reg_total;                      // tiles of all regions of a view
    int tiles_x[TRIPS_MAX_LAYERS];      // 8x4 pixel tiles per layer row (coarse layers)
    int tile_base[TRIPS_MAX_LAYERS + 1];  // first tile of every coarse layer (layers below reg_layers: reg_total)
    int n_tiles;                        // tiles per view
    int bins_x, bins_y, n_bins;         // 32x32 screen bins of layer 0
};

// Per-view constants built on the device from the pose / intrinsics tensors (setup_cams_kernel).  First what the projection of a
// point reads.
struct CamConst
{
    float qx, qy, qz, qw;
    float tx, ty, tz, s;
    float fx, fy, cx, cy;
    float cfx, cfy, ccx, ccy;
    float r00, r01, r10, r11;
    float cenx, ceny, cs;
    int dist;                              // apply the distortion and the cut-off radius
    float R[9];
    int image_index, camera_index;
    float k1, k2, k3, k4, k5, k6, p1, p2;  // lens distortion (TripsRenderParams.distortion)
    float cut2;                            // dist_cutoff^2
};

struct LayerPtrs
{
    float* p[TRIPS_MAX_LAYERS];
};
struct ConstLayerPtrs
{
    const float* p[TRIPS_MAX_LAYERS];
};

// Where an inference pass was given up because it does not suit what it was launched with (place_views in forward.cu).
enum GivenUp : unsigned int
{
    kNotGivenUp,
    kGivenUpEntries,  // before its entries were written: they do not fit, or PassGuess was wrong
    kGivenUpLists,    // before its lists were written: they do not fit
};

// Device-side counters of one forward call.
struct DevStats
{
    unsigned long long visible;    // visible points over all views (needed entries, whether or not they fitted)
    unsigned long long kept;
    unsigned long long frag_need;  // fragments over all views (needed list slots, whether or not they fitted)
    unsigned int max_len;
    unsigned int n_heavy;          // lists longer than kHeavyList (they are pre-selected before the blend); every part of a shared one counts
    unsigned int max_key;          // largest number of visible points in one (view, screen bin, tile) group
    unsigned int n_shared;         // parts of shared lists among them
    unsigned int status;
    GivenUp given_up;            // an inference pass: its remaining kernels write nothing, the host takes it up again
    unsigned int culled_blocks;  // (view, block of consecutive points) pairs skipped by the bounding-box test, counted once per pass
};

// A visible point of one view ("entry"): everything the later stages need, gathered once and stored in screen-bin
// order so that fragments of neighbouring pixels read neighbouring entries.  The fields live in two arrays, split by
// the stage that reads them, so that a stage's gathers touch fewer bytes it does not use (DRAM is read in 64-byte
// pieces), while the binning pass still writes whole 32-byte sectors:
//   head [2 x float4]     u, v (layer-0 image position), size in pixels, confidence (all the backward pass reads) |
//                         point id (bits), view-space depth, raw point size (fills the sector: nothing reads it), number of layers
//                         written (bits)
//   tail [1 + C4/4 float4] world position x, y, z (read for the camera gradients with lens distortion only), texture index
//                         (bits) | descriptor row (C floats, padded to 4)
__host__ __device__ constexpr int tail_stride(int C) { return 4 + ((C + 3) & ~3); }
__host__ __device__ constexpr int entry_stride(int C) { return 8 + tail_stride(C); }  // floats per entry over both arrays
// Gradient accumulator of an entry: sums over its fragments of (J0 gbs, J1 gbs, bf conf lf' ga, bf lf ga) | descriptor row.
__host__ __device__ constexpr int egrad_stride(int C) { return 4 + ((C + 3) & ~3); }

// Everything the forward kernels need besides the scene (all device pointers into context scratch).
// Lists longer than kHeavyList, found by the scan.  A list of several parts has one item per part.
struct HeavyLists
{
    uint4* item;        // [cap] view, pixel, part | parts << 16 (0: empty), where the list's parts start in `nearest` and `finished`
    uint32_t* nearest;  // [shared_cap, 16] list positions of a part's nearest fragments
    uint32_t* finished; // [shared_cap] parts of the list that are done, at the list's first part
    unsigned cap, shared_cap;
};

struct FwdBuffers
{
    uint32_t* bin_count;              // [B,n_bins,32] visible points per (screen bin, 8x4 tile of the bin)
    uint32_t* bin_base;               // [B,n_bins,32] next free entry (within the view) of every (bin, tile) group
    uint32_t* view_total;             // [B] visible points per view
    uint32_t* bin_cursor;             // [B,n_bins] first entry of every bin within the view
    unsigned long long* entry_base;   // [B+1] first entry of each view
    float4* ent_head;                 // [sum V_b, 2]
    float* ent_tail;                  // [sum V_b, tail_stride]
    uint32_t* counts;                 // [B,P] list lengths
    uint32_t* offsets;                // [B,P] list start within the view, the lists in no particular order (list end after the collect pass)
    unsigned long long* view_base;    // [B+1] first fragment of each view in `frags`
    uint4* frags;                     // [frag_cap] x = point id, y = depth bits (y:x = 64-bit sort key), z = alpha bits, w = entry index within the view
    unsigned long long frag_cap;
    bool report_overflow;             // training: raise a status bit for views that do not fit; off where the host looks (place_views)
    uint8_t* rec_n;                   // [B,n_tiles,32] records kept for backward, by tile and lane (pixel of the tile)
    uint2* records;                   // [B,n_tiles,16,32] (entry index within the view, alpha bits), by tile, rank and lane: a warp's
                                      // access to one rank of its tile is 256 consecutive bytes
    DevStats* stats;
    // work counters of the persistent kernels, zeroed with bin_count and counts by one clear per forward pass
    unsigned int* ticket;             // binning passes: one per pass and group of views
    unsigned int* ticket_count;       // [B] count pass
    unsigned int* ticket_collect;     // [B] collect pass
    unsigned int* ticket_blend;
    unsigned int* finished;           // [2] blocks that are done, of the bin scan and of list_starts_kernel
    uint32_t* list_cursor;            // [B] fragments of the views as list_starts_kernel adds them up
    uint32_t* point_entry;            // training: [entry_views,N] entry (within the view) of every point, kNoEntry where it is not visible
    int entry_views;                  // B, or fewer where the table of all views would be larger than kEntryTableBytes: the backward
                                      // pass then fills it for so many views at a time
    uint32_t* note_entry;             // point_entry where the binning pass notes the entries of all views, else nullptr
    float4* point_state;              // training: [N] position and raw size of the points that were not discarded, as this pass saw them
    const uint8_t* block_skip;        // [B, ceil(N / 8192)] 1 = the block cannot hold a point visible in that view
    HeavyLists heavy;
};

struct ScenePtrs
{
    int N, n_tex, C;
    const float4* position;
    const float* point_size;
    const int32_t* index;
    const float* texture;
    const float* confidence;
    const float* background;
    const float* dropout;
};

struct BwdBuffers
{
    float* egrad;         // [sum V_b, egrad_stride] per-entry gradient accumulators
    unsigned int* ticket; // [kTileCounters x kTileCounterPitch] work counters of the tile kernel
    double* g_bg;         // [C]
    double* g_pose;       // [B,6]
    double* g_k;          // [B,5]
    double* g_dis;        // [B,8] distortion coefficients
};

// The reference has two forward pipelines (PointRenderer.cu:730-731): the second (CountTiled, CollectTiled2[Pointsize],
// FastSortAndBlendWPrep2WarpSharedWork, RenderForward.cu:1401-3674) runs when one of these flags differs from its
// default.  strict_layers: a point is written to the two layers around log2(size) only (RenderForward.cu:2291-2393).
__host__ __device__ inline bool second_pipeline(const TripsRenderParams& pr)
{
    return !(pr.use_layer_point_size && pr.render_points_in_all_lower_resolutions && !pr.combine_lists);
}
__host__ __device__ inline bool strict_layers(const TripsRenderParams& pr)
{
    return pr.use_layer_point_size && !pr.render_points_in_all_lower_resolutions;
}

// Kernels of a call follow one another on one stream.  A kernel that starts with follow_previous() may be launched by
// launch_following() while its predecessor drains: its blocks are in place when the last ones of that kernel end, and wait there
// until all of its memory operations are visible.  Every kernel waits before it does anything, so that the end of one kernel
// implies the end of all before it.  What a kernel of the same call has written is read with plain loads only: a load through
// __restrict__ or __ldg promises that nobody writes there while the kernel exists, and may be moved ahead of the wait.  14 kernels of a step, us, one after another / like this: 800 k points x 2 views 698 / 682, 2 M x 4
// 1715 / 1691, a 640x480 frame (10 kernels) 228 / 213, a 1080p frame 843 / 825, 6 M x 8 views 8823 / 8800.
__device__ __forceinline__ void follow_previous()
{
    asm volatile("griddepcontrol.wait;" ::: "memory");
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
}
template <class... Params, class... Args>
cudaError_t launch_following(void (*kernel)(Params...), dim3 grid, dim3 block, cudaStream_t st, Args&&... args)
{
    cudaLaunchAttribute overlap{};
    overlap.id                                         = cudaLaunchAttributeProgrammaticStreamSerialization;
    overlap.val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t config{};
    config.gridDim  = grid;
    config.blockDim = block;
    config.stream   = st;
    config.attrs    = &overlap;
    config.numAttrs = 1;
    return cudaLaunchKernelEx(&config, kernel, static_cast<Args&&>(args)...);
}

// ---- device helpers (op order mirrors the CPU oracle; compiled with -fmad=false) ----

__device__ __forceinline__ void transform_point(const CamConst& V, float px, float py, float pz, float& ox, float& oy,
                                                float& oz)
{
    // Sophus SE3f * p: Eigen quaternion _transformVector, then translation (PointRendererHelper.h:238)
    float ux = V.qy * pz - V.qz * py;
    float uy = V.qz * px - V.qx * pz;
    float uz = V.qx * py - V.qy * px;
    ux += ux;
    uy += uy;
    uz += uz;
    float cx = V.qy * uz - V.qz * uy;
    float cy = V.qz * ux - V.qx * uz;
    float cz = V.qx * uy - V.qy * ux;
    ox       = ((px + V.qw * ux) + cx) + V.tx;
    oy       = ((py + V.qw * uy) + cy) + V.ty;
    oz       = ((pz + V.qw * uz) + cz) + V.tz;
}

// saiga's distortNormalizedPoint restated: the 8-coefficient rational model with tangential terms (the operation order
// is the CPU oracle's).  J (optional): d(xd, yd) / d(x, y) row-major; Jk (optional): d(xd, yd) / d(k1..k6, p1, p2), two
// rows of 8.
__device__ __forceinline__ void distort_point(const CamConst& c, float x, float y, float& xd, float& yd, float* J, float* Jk)
{
    const float x2 = x * x, y2 = y * y;
    const float r2 = x2 + y2, xy2 = 2.f * x * y;
    const float r4 = r2 * r2, r6 = r4 * r2;
    const float A  = ((1.f + c.k1 * r2) + c.k2 * r4) + c.k3 * r6;
    const float B  = ((1.f + c.k4 * r2) + c.k5 * r4) + c.k6 * r6;
    const float iB = 1.f / B;
    const float radial = A * iB;
    const float tx = c.p1 * xy2 + c.p2 * (r2 + 2.f * x2);
    const float ty = c.p1 * (r2 + 2.f * y2) + c.p2 * xy2;
    xd = x * radial + tx;
    yd = y * radial + ty;
    if (J)
    {
        const float dA = (c.k1 + 2.f * c.k2 * r2) + 3.f * c.k3 * r4;
        const float dB = (c.k4 + 2.f * c.k5 * r2) + 3.f * c.k6 * r4;
        const float dr = (dA * B - A * dB) * iB * iB;  // d radial / d r2
        J[0] = radial + x * dr * (2.f * x) + (2.f * c.p1 * y + 6.f * c.p2 * x);
        J[1] = x * dr * (2.f * y) + (2.f * c.p1 * x + 2.f * c.p2 * y);
        J[2] = y * dr * (2.f * x) + (2.f * c.p1 * x + 2.f * c.p2 * y);
        J[3] = radial + y * dr * (2.f * y) + (6.f * c.p1 * y + 2.f * c.p2 * x);
    }
    if (Jk)
    {
        const float AiB2 = A * iB * iB;
        Jk[0] = x * r2 * iB, Jk[1] = x * r4 * iB, Jk[2] = x * r6 * iB;
        Jk[3] = -x * AiB2 * r2, Jk[4] = -x * AiB2 * r4, Jk[5] = -x * AiB2 * r6;
        Jk[6] = xy2, Jk[7] = r2 + 2.f * x2;
        Jk[8] = y * r2 * iB, Jk[9] = y * r4 * iB, Jk[10] = y * r6 * iB;
        Jk[11] = -y * AiB2 * r2, Jk[12] = -y * AiB2 * r4, Jk[13] = -y * AiB2 * r6;
        Jk[14] = r2 + 2.f * y2, Jk[15] = xy2;
    }
}

// ProjectPointPinholeWoNormal + crop transform + crop rotation
// (PointRendererHelper.h:232-253, RenderForward.cu:302-303,69-76).
__device__ __forceinline__ void project_point(const CamConst& c, float px, float py, float pz, float& u, float& v, float& z)
{
    float vx, vy, vz;
    transform_point(c, px, py, pz, vx, vy, vz);
    z        = fmaxf(vz, 0.f);
    float iz = 1.f / vz;
    float nx = vx * iz;
    float ny = vy * iz;
    if (c.dist)  // uniform per view
    {
        // outside the cut-off radius distortNormalizedPoint returns (100000, 100000) and the caller sets z = 0
        // (PointRendererHelper.h:246-249)
        if (nx * nx + ny * ny > c.cut2) z = 0.f;
        float xd, yd;
        distort_point(c, nx, ny, xd, yd, nullptr, nullptr);
        nx = xd, ny = yd;
    }
    float ix = (c.fx * nx + c.s * ny) + c.cx;
    float iy = c.fy * ny + c.cy;
    float jx = (c.cfx * ix + c.cs * iy) + c.ccx;
    float jy = c.cfy * iy + c.ccy;
    float dx = jx - c.cenx;
    float dy = jy - c.ceny;
    float rx = c.r00 * dx + c.r01 * dy;
    float ry = c.r10 * dx + c.r11 * dy;
    u        = rx + c.cenx;
    v        = ry + c.ceny;
}

// compute_point_size_fac (PointBlending.h:81-149); floor / ceil of log2 taken from the float's bits.
// FAST_EXP: the hardware exponential (about 2 ulp) instead of the reproducible one; only for values that do not decide
// list membership, i.e. in the backward pass (gradient tolerance 1e-4), never in the forward pass.
template <bool FAST_EXP = false>
__device__ __forceinline__ float layer_factor(float ps, int layer, int L, float* grad)
{
    int lo = 0, hi = 0;
    if (ps > 1.f)
    {
        lo = min(max(0, tm_floor_log2(ps)), L - 1);
        hi = min(max(0, tm_ceil_log2(ps)), L - 1);
    }
    if (layer < lo)
    {
        if (grad) *grad = 0.f;
        return 1.f;
    }
    float f = 1.f;
    if (hi == 0)
    {
        f = 0.75f * (FAST_EXP ? __expf(ps - 1.f) : tm_expf(ps - 1.f)) + 0.25f;
        if (grad) *grad = 0.27591f * ps;
    }
    else if (lo == hi)
    {
        if (grad) *grad = 1.f;
    }
    else
    {
        // hi = lo + 1: the layers' sizes differ by 2^lo, and a division by it is a product with its exact reciprocal
        const float l_l = (float)(1 << lo), inv = __int_as_float((127 - lo) << 23);
        f               = (ps - l_l) * inv;
        if (layer == lo) f = 1.f - f;
        if (grad) *grad = layer == lo ? -inv : inv;
    }
    return f;
}

// Pixel handled by `lane` of the warp that owns 8x4 tile `tile` of a view; p = -1 outside the image.
__device__ __forceinline__ void tile_pixel(const Geom& g, int tile, int lane, int& layer, int& gx, int& gy, int& p)
{
    int l, tx, ty;
    if (tile < g.reg_total)
    {
        const int r = tile / g.reg_tiles, k = tile - r * g.reg_tiles;
        l           = k < 128 ? 0 : (k < 160 ? 1 : (k < 168 ? 2 : 3));
        const int kk = k - (l == 0 ? 0 : (l == 1 ? 128 : (l == 2 ? 160 : 168)));
        const int ry = r / g.reg_x, rx = r - ry * g.reg_x;
        tx = rx * (8 >> l) + (kk & ((8 >> l) - 1));   // a region is 8 >> l tiles wide and 16 >> l tiles high on layer l
        ty = ry * (16 >> l) + (kk >> (3 - l));
    }
    else
    {
        l = g.reg_layers;
#pragma unroll
        for (int i = 1; i < TRIPS_MAX_LAYERS; ++i)
            if (i > g.reg_layers && i < g.L && tile >= g.tile_base[i]) l = i;
        const int t = tile - g.tile_base[l];
        ty          = t / g.tiles_x[l];
        tx          = t - ty * g.tiles_x[l];
    }
    layer        = l;
    gx           = tx * kTileW + (lane & (kTileW - 1));
    gy           = ty * kTileH + (lane >> 3);
    p            = (gx < g.W[l] && gy < g.H[l]) ? g.base[l] + gy * g.W[l] + gx : -1;
}

// The inverse: tile of a view and lane that own pixel (gx, gy) of a layer.
__host__ __device__ __forceinline__ void pixel_tile(const Geom& g, int layer, int gx, int gy, int& tile, int& lane)
{
    lane = ((gy & (kTileH - 1)) << 3) | (gx & (kTileW - 1));
    if (layer < g.reg_layers)
    {
        const int rx = gx >> (6 - layer), ry = gy >> (6 - layer);  // regions are 64 >> layer pixels wide and high
        const int tx = (gx >> 3) - rx * (8 >> layer), ty = (gy >> 2) - ry * (16 >> layer);
        const int first = layer == 0 ? 0 : (layer == 1 ? 128 : (layer == 2 ? 160 : 168));
        tile            = (ry * g.reg_x + rx) * g.reg_tiles + first + (ty << (3 - layer)) + tx;
    }
    else
        tile = g.tile_base[layer] + (gy >> 2) * g.tiles_x[layer] + (gx >> 3);
}

// Work distribution of the backward tile kernel: a warp takes one tile at a time.  One counter for all warps is a single
// address, and its returning atomics queue up behind one another and among the kernel's gradient atomics in one slice of
// L2.  kTileCounters counters on lines of their own, each over every kTileCounters-th tile, so that tiles still come in
// order; a warp whose counter has run out goes on with the next one.  blend_backward, one / four counters: 6 M points x 8
// views 3.42 / 3.11 ms, 2 M x 4 views (720p) 0.74 / 0.61 ms, 20 M x 2 views (many empty tiles) 0.89 / 0.70 ms.  The blend of
// the forward pass, which has no other atomics, is 4 % slower with four and keeps one.
constexpr int kTileCounters     = 4;
constexpr int kTileCounterPitch = 32;  // words between counters: one 128-byte line each
struct TileTickets
{
    unsigned* counters;
    unsigned n_tiles;   // of all views
    unsigned id;        // counter in use
    unsigned ahead;     // lane 0: the following ticket, requested a whole tile ahead of its use
    int left;           // counters that have not run out yet, the one in use included
    __device__ __forceinline__ void request(int lane)
    {
        if (lane == 0) ahead = atomicAdd(counters + id * kTileCounterPitch, 1u) * kTileCounters + id;
    }
    __device__ __forceinline__ void start(unsigned* c, unsigned n, unsigned warp_id, int lane)
    {
        counters = c, n_tiles = n, id = warp_id % kTileCounters, left = kTileCounters;
        request(lane);
    }
    // the next tile of the warp (all lanes call this together), or n_tiles and more when there is none
    __device__ __forceinline__ unsigned next(int lane)
    {
        unsigned t = __shfl_sync(kFull, ahead, 0);
        while (t >= n_tiles && --left > 0)
        {
            id = (id + 1) % kTileCounters;
            request(lane);
            t = __shfl_sync(kFull, ahead, 0);
        }
        if (t < n_tiles) request(lane);
        return t;
    }
};

// ---- launchers (forward.cu / backward.cu / adam.cu) ----
cudaError_t launch_setup_cams(const TripsView* h_views, int B, const double* poses, int n_images, const float* intrinsics,
                              int n_cameras, int distortion, float dist_cutoff, CamConst* cams, DevStats* stats, cudaStream_t st);
constexpr int kViewTable = 32;  // views passed to one launch of setup_cams_kernel as an argument;
// What the kernels of a pass are launched with before its counts are known.
struct PassGuess
{
    bool look;                   // the host looks at the counts while the pass runs: one that the guess does not suit is given up
    bool hot;                    // binning kernels that aggregate in shared memory (kHotKey)
    unsigned long long entries;  // the size of the window passes' tickets and grids
};
// More entries than kGuessFactor times the guess, and at least kGuessEntries: too few blocks for them.  One 1080p view taken in turn with
// one that sees less, us, with the guess of that one / its own: 7.0 M entries (6 times the guess) 1370 / 1361, (28 times) 1502 / 1361,
// 13.9 M (33 times) 2609 / 2415, 1.4 M (6 to 1000 times) 562 / 523; a pass that is given up takes 50 longer.
constexpr unsigned long long kGuessFactor = 8, kGuessEntries = 2ull << 20;
cudaError_t launch_bin_count(const ScenePtrs& sc, const CamConst* cams, const Geom& g, const TripsRenderParams& pr, int B,
                             const FwdBuffers& fb, unsigned long long entry_cap, PassGuess guess, int sm_count, cudaStream_t st);
cudaError_t launch_bin_scatter(const ScenePtrs& sc, const CamConst* cams, const Geom& g, const TripsRenderParams& pr, int B,
                               const FwdBuffers& fb, bool hot, int sm_count, cudaStream_t st);
constexpr unsigned kHotKey = 4096;  // visible points in one (view, bin, tile) group beyond which the binning passes aggregate in shared memory
int bin_count_launches(int N, int B);
int bin_scatter_launches(int N, int B);
size_t resize_scratch_bytes(int64_t n_points);
cudaError_t launch_resize_points(const int64_t* remove, int64_t n_remove, int64_t n_points, int64_t n_new, const TripsPointTensor* tensors,
                                 int n_tensors, void* scratch, DevStats* stats, int sm_count, cudaStream_t st);
cudaError_t launch_list_starts(const Geom& g, int B, int k_keep, const FwdBuffers& fb, cudaStream_t st);
cudaError_t launch_place_views(int B, const FwdBuffers& fb, bool entries, cudaStream_t st);  // of the entries, or of the lists
// strict: an entry's layers start at the layer below log2(size) instead of layer 0 (strict_layers above)
// entries_hint: the number of entries of the call as far as the host knows it (selects the size of the work tickets)
cudaError_t launch_count(const ScenePtrs& sc, const Geom& g, int B, const FwdBuffers& fb, bool strict, unsigned long long entries_hint, int sm_count,
                         cudaStream_t st);
cudaError_t launch_collect(const ScenePtrs& sc, const Geom& g, int B, const FwdBuffers& fb, bool strict, unsigned long long entries_hint, int sm_count, cudaStream_t st);
// top-K + blend by the rules of the reference's second forward pipeline (one thread per pixel)
cudaError_t launch_second_blend(const ScenePtrs& sc, const Geom& g, const TripsRenderParams& pr, int B, const FwdBuffers& fb,
                                const LayerPtrs& out, int sm_count, cudaStream_t st);
cudaError_t launch_nearest_16(const unsigned long long* d_keys, uint32_t n, uint32_t* d_result, cudaStream_t st);  // n >= 16; d_result [17]
cudaError_t launch_heavy_topk(const Geom& g, int B, const FwdBuffers& fb, int sm_count, cudaStream_t st);
cudaError_t launch_sort_blend(const ScenePtrs& sc, const Geom& g, const TripsRenderParams& pr, int B, const FwdBuffers& fb,
                              const LayerPtrs& out, int sm_count, cudaStream_t st);
cudaError_t launch_zero_entry_rows(int C, int B, const FwdBuffers& fb, const BwdBuffers& bb, int sm_count, cudaStream_t st);
cudaError_t launch_blend_backward(const ScenePtrs& sc, const CamConst* cams, const Geom& g, const TripsRenderParams& pr,
                                  int B, const FwdBuffers& fb, const BwdBuffers& bb, const ConstLayerPtrs& grad_in,
                                  unsigned long long entries_hint, int sm_count, cudaStream_t st);
int unpack_launches(int B, int entry_views);  // launches of the point gradients
cudaError_t launch_unpack_grads(const ScenePtrs& sc, const CamConst* cams, int B, const FwdBuffers& fb, const BwdBuffers& bb,
                                const TripsGrads& out, const TripsRenderParams& pr, int sm_count, cudaStream_t st);
cudaError_t launch_adam(const TripsAdamTensor* d_tensors, const int64_t* d_block_start, int n_tensors, int64_t total_blocks,
                        cudaStream_t st);
constexpr int kAdamTable = 16;  // tensors whose table travels as a kernel argument
cudaError_t launch_adam_by_value(const TripsAdamTensor* h_tensors, const int64_t* h_block_start, int n_tensors, cudaStream_t st);
cudaError_t launch_fused_reduce_adam(const float* const* grad_ptrs, float* const* param_ptrs, int world, int rank,
                                     const TripsAdamSegment* segs, int n_seg, int64_t lo, int64_t hi, float* m_state,
                                     float* v_state, int32_t* steps, int sm_count, cudaStream_t st);
cudaError_t launch_fused_multicast_adam(const float* grad_mc, float* param_mc, const float* param, const TripsAdamSegment* segs, int n_seg,
                                        int64_t lo, int64_t hi, float* m_state, float* v_state, int32_t* steps, int sm_count, cudaStream_t st);
struct L1Args
{
    const float* out[TRIPS_MAX_LAYERS];
    const float* target[TRIPS_MAX_LAYERS];
    float* grad[TRIPS_MAX_LAYERS];
    int64_t start[TRIPS_MAX_LAYERS + 1];
    int L;
};
cudaError_t launch_l1_loss(const L1Args& a, int64_t total, double* loss_out, int sm_count, cudaStream_t st);
// Pixels whose lists a block of list_starts_kernel places one after another.  Blocks come in any order: the smaller the ranges, the more
// places of the list buffer the passes behind it work on at a time.  scan / collect / sort_blend, us, of 2048 / 4096 / 8192 / 16384 pixels:
// 6 M points x 8 views 83 / 52 / 58 / 70, 1227 / 1209 / 1201 / 1191, 2287 / 2305 / 2300 / 2288 (chunk totals scanned in pixel order: 130 for
// the scan), 64 views of 10 M points 697 / 429 / 484 / 554, - / 14907 / 14770 / 14558, 22617 / 22814 / 22767 / 22590.
constexpr int kScanThreads = 1024, kScanPerLane = 16;
constexpr int kScanChunk   = kScanThreads * kScanPerLane;
constexpr int kAdamPerBlock = 1024 * 4;  // elements handled by one Adam block
}  // namespace trips
