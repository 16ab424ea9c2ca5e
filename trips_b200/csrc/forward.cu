// Forward rasterizer: project + count, scan, collect, per-pixel top-K sort and front-to-back blend.
//
// Stage map to the reference (src/lib/rendering/RenderForward.cu):
//   bin_count / bin_scan / bin_scatter kernels <- CountAndCollectTiled (:168-366)
//   list_starts_kernel    <- cub::DeviceScan + host glue (:1155-1232), no host sync
//   collect_kernel        <- SplattingPass               (:368-436)
//   sort_blend_kernel     <- FastSortFusedNew            (:474-1059)
// All views of a call are processed by one launch per stage (grid.y / ticket space spans the batch).
#include "common.cuh"

namespace trips
{
// ------------------------------------------------------------------------------------------------------------
// per-view camera constants
// ------------------------------------------------------------------------------------------------------------
// The view table travels as a kernel argument: a copy from pageable host memory costs a staging copy on the host and a
// transfer of its own on the stream.
struct ViewTable
{
    TripsView v[kViewTable];
};
__global__ void setup_cams_kernel(const __grid_constant__ ViewTable views, int b0, int B, const double* __restrict__ poses, int n_images,
                                  const float* __restrict__ intrinsics, int n_cameras, int distortion, float dist_cutoff,
                                  CamConst* __restrict__ cams, DevStats* stats)
{
    follow_previous();
    const int b = b0 + (int)threadIdx.x;
    if (b == 0)
    {
        // the counters of the call start from zero; the status word keeps the bits raised by earlier calls until
        // trips_last_status reads them
        stats->visible = stats->kept = stats->frag_need = 0ull;
        stats->max_len = stats->n_heavy = stats->max_key = stats->n_shared = stats->culled_blocks = 0u;
        stats->given_up = kNotGivenUp;
    }
    if (b >= B) return;
    const TripsView& v = views.v[threadIdx.x];
    CamConst c;
    const double* p = poses + (size_t)min(max(v.image_index, 0), n_images - 1) * 8;
    // DeviceRenderParams::Pose: SE3d cast to float (RenderConstants.h:85-88)
    c.qx = (float)p[0];
    c.qy = (float)p[1];
    c.qz = (float)p[2];
    c.qw = (float)p[3];
    c.tx = (float)p[4];
    c.ty = (float)p[5];
    c.tz = (float)p[6];
    // Eigen::Quaternion::toRotationMatrix
    float tx = 2.f * c.qx, ty = 2.f * c.qy, tz = 2.f * c.qz;
    float twx = tx * c.qw, twy = ty * c.qw, twz = tz * c.qw;
    float txx = tx * c.qx, txy = ty * c.qx, txz = tz * c.qx;
    float tyy = ty * c.qy, tyz = tz * c.qy, tzz = tz * c.qz;
    c.R[0] = 1.f - (tyy + tzz);
    c.R[1] = txy - twz;
    c.R[2] = txz + twy;
    c.R[3] = txy + twz;
    c.R[4] = 1.f - (txx + tzz);
    c.R[5] = tyz - twx;
    c.R[6] = txz - twy;
    c.R[7] = tyz + twx;
    c.R[8] = 1.f - (txx + tyy);
    const float* k = intrinsics + (size_t)min(max(v.camera_index, 0), n_cameras - 1) * 13;
    c.fx = k[0];
    c.fy = k[1];
    c.cx = k[2];
    c.cy = k[3];
    c.s  = k[4];
    bool dist = false;
    for (int i = 5; i < 13; ++i) dist |= (k[i] != 0.f);
    if (dist && !distortion) atomicOr(&stats->status, TRIPS_DEV_NONZERO_DISTORTION);  // a plain pinhole was asked for: ignored
    c.k1 = k[5], c.k2 = k[6], c.k3 = k[7], c.k4 = k[8], c.k5 = k[9], c.k6 = k[10], c.p1 = k[11], c.p2 = k[12];
    c.cut2 = dist_cutoff * dist_cutoff;
    c.dist = distortion ? 1 : 0;
    c.cfx  = v.crop_transform[0];
    c.cfy  = v.crop_transform[1];
    c.ccx  = v.crop_transform[2];
    c.ccy  = v.crop_transform[3];
    c.cs   = v.crop_transform[4];
    c.r00  = v.crop_rotation[0];
    c.r01  = v.crop_rotation[1];
    c.r10  = v.crop_rotation[2];
    c.r11  = v.crop_rotation[3];
    c.cenx = (float)(v.w / 2);  // integer division as in RenderForward.cu:303
    c.ceny = (float)(v.h / 2);
    c.image_index  = v.image_index;
    c.camera_index = v.camera_index;
    cams[b]        = c;
}

cudaError_t launch_setup_cams(const TripsView* h_views, int B, const double* poses, int n_images, const float* intrinsics,
                              int n_cameras, int distortion, float dist_cutoff, CamConst* cams, DevStats* stats, cudaStream_t st)
{
    for (int b0 = 0; b0 < B; b0 += kViewTable)
    {
        ViewTable t;
        const int n = min(kViewTable, B - b0);
        for (int k = 0; k < n; ++k) t.v[k] = h_views[b0 + k];
        for (int k = n; k < kViewTable; ++k) t.v[k] = h_views[b0];
        launch_following(setup_cams_kernel, 1, kViewTable, st, t, b0, B, poses, n_images, intrinsics, n_cameras, distortion, dist_cutoff, cams, stats);
    }
    return cudaGetLastError();
}

// ------------------------------------------------------------------------------------------------------------
// project + cull + layer select, and sort the visible points of every view by (32x32 screen bin, 8x4 tile of the bin)
//
// Kernels: bounding boxes of blocks of consecutive points and their visibility per view; (1) count the visible points
// per (view, bin, tile) with one global counter each; (2) exclusive scan of the counters; (3) project again, take a slot
// in the point's group and write its entry there (head and tail, 32 bytes each).  Replaces the projection part of
// CountAndCollectTiled (RenderForward.cu:168-366); the list lengths are counted afterwards from the entries
// (window_kernel<false>).  Both passes read every point ONCE per call and loop over the views with the point in
// registers (the camera constants of up to kViewGroup views sit in shared memory): position, size and, in the scatter
// pass, confidence and descriptor row cost N reads per call instead of N x B, and softplus(size) is evaluated
// once per point.  Projecting twice avoids writing and re-reading a per-point record for all N x B point-views.
// ------------------------------------------------------------------------------------------------------------
struct Projected
{
    float u, v, z, ps;
    bool ok;
};

// radius of a point in pixels; read with drop_out_points_by_radius only
__device__ __forceinline__ float projected_radius(const CamConst& cam, const float4& p, float z) { return cam.fx * cam.cfx * p.w / z; }

// Visibility test of one point in one view (RenderForward.cu:224-340).  `sp` caches softplus(raw) across the views of
// the point: negative = not computed yet (softplus is never negative); only visible points pay for it.
__device__ __forceinline__ Projected project_visible(const CamConst& cam, const Geom& g, const TripsRenderParams& pr, const float4& p,
                                                     float raw, float& sp)
{
    Projected r;
    const float fxc = cam.fx * cam.cfx;
    project_point(cam, p.x, p.y, p.z, r.u, r.v, r.z);
    r.ps = 0.f;
    bool ok = !(r.z <= 0.f || r.u < 0.f || r.u >= (float)(g.W[0] - 1) || r.v < 0.f || r.v >= (float)(g.H[0] - 1));
    // the first pipeline's test takes an int (RenderForward.cu:212-218), the second's the float (RenderForward.cu:1527-1531)
    if (ok && pr.drop_out_points_by_radius)
    {
        const float rad = projected_radius(cam, p, r.z);
        if ((second_pipeline(pr) ? rad : (float)(int)rad) < pr.drop_out_radius_threshold) ok = false;
    }
    if (ok)
    {
        if (sp < 0.f) sp = tm_softplus(raw);
        r.ps = fxc * sp / r.z;
    }
    r.ok = ok;
    return r;
}

// A camera as the binning kernels hold it in shared memory: on 16 bytes, so that it is read four words at a time.  (For CamConst itself
// the alignment costs point_grad_kernel registers: 753 -> 808 us on 20 M points in 2 views.)
struct alignas(16) BinCam : CamConst
{
};
static_assert(sizeof(BinCam) == sizeof(CamConst), "copied word by word");

constexpr int kBinThreads     = 256;
constexpr int kBinBlocksPerSM = 8;
constexpr int kCountMinBlocks = 4;     // 64 registers; 5 blocks of 48: the same, uncapped 74 registers
constexpr int kScatterMinBlocks = 4, kScatterMinBlocksWide = 3;  // up to 4 channels / more; measured at 3 / 4: 6 M points 1.26 / 1.23 ms (8 views), 0.346 / 0.313 ms (1 view); 8 channels 0.116 / 0.127 ms
constexpr int kBinChunk       = 8192;  // points per bounding box
constexpr int kBinTicket      = 1024;  // points per work ticket of the binning kernels; a ticket lies inside one box
constexpr int kSweep          = 4;     // views whose entry slots a thread requests before it waits for any of them
static_assert(kBinChunk % kBinTicket == 0, "a ticket must not straddle two bounding boxes");

// True when no point inside the box can pass the visibility test of project_visible for this view.  The image position
// is an affine map of (x/z, y/z); multiplied by z > 0 every image border becomes a plane through the camera centre,
// i.e. a linear function of the view-space position, and a box lies outside a plane when its 8 corners do.  The borders
// are moved out by a margin of 2 pixels (+ 1e-3 of the depth), far more than the rounding difference between this
// test and the per-point arithmetic.
__device__ __forceinline__ bool box_outside_view(const CamConst& c, const Geom& g, const float* __restrict__ box)
{
    if (!(box[3] < 3.0e38f)) return false;
    // u(nx, ny) = cu + au nx + bu ny, v likewise: evaluate the projection chain at three normalised positions
    float u0, v0, u1, v1, u2, v2;
    {
        auto img = [&](float nx, float ny, float& u, float& v) {
            const float ix = (c.fx * nx + c.s * ny) + c.cx, iy = c.fy * ny + c.cy;
            const float jx = (c.cfx * ix + c.cs * iy) + c.ccx, jy = c.cfy * iy + c.ccy;
            const float dx = jx - c.cenx, dy = jy - c.ceny;
            u = (c.r00 * dx + c.r01 * dy) + c.cenx;
            v = (c.r10 * dx + c.r11 * dy) + c.ceny;
        };
        img(0.f, 0.f, u0, v0);
        img(1.f, 0.f, u1, v1);
        img(0.f, 1.f, u2, v2);
    }
    const float au = u1 - u0, bu = u2 - u0, av = v1 - v0, bv = v2 - v0;
    const float m = 2.f, wmax = (float)(g.W[0] - 1) + m, hmax = (float)(g.H[0] - 1) + m;
    bool all_behind = true, all_left = true, all_right = true, all_up = true, all_down = true;
#pragma unroll
    for (int k = 0; k < 8; ++k)
    {
        float x, y, z;
        transform_point(c, box[(k & 1) ? 3 : 0], box[(k & 2) ? 4 : 1], box[(k & 4) ? 5 : 2], x, y, z);
        const float U = au * x + bu * y + u0 * z, V = av * x + bv * y + v0 * z;
        const float slack = 1e-3f * fabsf(z) + 1e-6f * (fabsf(x) + fabsf(y));
        all_behind &= z < -slack;
        all_left &= (U + m * z) < -slack * (fabsf(au) + fabsf(bu) + fabsf(u0) + m);
        all_right &= (wmax * z - U) < -slack * (fabsf(au) + fabsf(bu) + fabsf(u0) + wmax);
        all_up &= (V + m * z) < -slack * (fabsf(av) + fabsf(bv) + fabsf(v0) + m);
        all_down &= (hmax * z - V) < -slack * (fabsf(av) + fabsf(bv) + fabsf(v0) + hmax);
    }
    return all_behind || all_left || all_right || all_up || all_down;
}

// Bounding boxes of blocks of consecutive points and the conservative frustum test on them: the reference computes
// such boxes per 10 240 points (NeuralPointCloudCuda.cpp:339-384) but never uses them.  Point clouds stored in a
// spatially coherent order (scans, reconstructions) have compact blocks, and a block whose box lies outside a view
// is skipped by both binning passes; for a cloud in random order every box spans the scene and nothing is skipped.
// Boxes are recomputed by every forward pass (points move): one read of the positions.  skip[b * n_blocks + k] = 1 when block k of
// the point cloud cannot hold a point visible in view b (a test inside the binning kernels would cost their loops 30
// registers).
__global__ __launch_bounds__(256) void block_visibility_kernel(const float4* __restrict__ pos, int N, const CamConst* cams,
                                                               const __grid_constant__ Geom g, int B, uint8_t* skip, DevStats* stats)
{
    follow_previous();
    const int first = blockIdx.x * kBinChunk, last = min(N, first + kBinChunk);
    float lo[3] = {3.0e38f, 3.0e38f, 3.0e38f}, hi[3] = {-3.0e38f, -3.0e38f, -3.0e38f};
    bool bad = false;
    for (int i = first + threadIdx.x; i < last; i += 256)
    {
        const float4 p = pos[i];
        const float v[3] = {p.x, p.y, p.z};
#pragma unroll
        for (int k = 0; k < 3; ++k)
        {
            bad |= !(fabsf(v[k]) < 3.0e38f);  // NaN or infinite: the block is never skipped
            lo[k] = fminf(lo[k], v[k]);
            hi[k] = fmaxf(hi[k], v[k]);
        }
    }
    __shared__ float s_lo[8][3], s_hi[8][3], s_box[6];
    __shared__ int s_bad;
    if (threadIdx.x == 0) s_bad = 0;
    __syncthreads();
    if (bad) s_bad = 1;
#pragma unroll
    for (int k = 0; k < 3; ++k)
    {
#pragma unroll
        for (int o = 16; o > 0; o >>= 1)
        {
            lo[k] = fminf(lo[k], __shfl_xor_sync(kFull, lo[k], o));
            hi[k] = fmaxf(hi[k], __shfl_xor_sync(kFull, hi[k], o));
        }
        if ((threadIdx.x & 31) == 0) s_lo[threadIdx.x >> 5][k] = lo[k], s_hi[threadIdx.x >> 5][k] = hi[k];
    }
    __syncthreads();
    if (threadIdx.x < 3)
    {
        float a = s_lo[0][threadIdx.x], b = s_hi[0][threadIdx.x];
        for (int w = 1; w < 8; ++w) a = fminf(a, s_lo[w][threadIdx.x]), b = fmaxf(b, s_hi[w][threadIdx.x]);
        if (s_bad) a = -3.4e38f, b = 3.4e38f;
        s_box[threadIdx.x] = a, s_box[3 + threadIdx.x] = b;
    }
    __syncthreads();
    for (int b = threadIdx.x; b < B; b += 256)
    {
        const CamConst cam = cams[b];
        const bool out     = box_outside_view(cam, g, s_box);
        skip[(size_t)b * gridDim.x + blockIdx.x] = out ? 1 : 0;
        if (out) atomicAdd(&stats->culled_blocks, 1u);
    }
}

// Work distribution of the binning kernels: tickets of kBinTicket consecutive points from one counter, so that every SM
// is busy until the last ticket whatever the number of resident blocks is (a static split left a partial last wave).
// (A block does not ask for its next ticket before it is done: where there are fewer tickets than blocks, those that come
// first would take two each - 130 k points in 11 views 0.23 instead of 0.17 ms - and elsewhere it gains nothing.)
// Returns false when the cloud is exhausted; `skip` gets one bit per view of the group whose bounding-box test rules the
// ticket's points out.
__device__ __forceinline__ bool next_point_ticket(unsigned* ticket, int N, unsigned* s_ticket, const uint8_t* block_skip, int v0,
                                                  int nv, int& first, int& last, unsigned& skip)
{
    __syncthreads();
    if (threadIdx.x == 0) *s_ticket = atomicAdd(ticket, 1u);
    __syncthreads();
    const unsigned t = *s_ticket;
    if (t >= ((unsigned)N + kBinTicket - 1) / kBinTicket) return false;
    first = (int)(t * kBinTicket);
    last  = min(N, first + kBinTicket);
    skip  = 0;
    if (block_skip)
    {
        const int n_box = (N + kBinChunk - 1) / kBinChunk, box = first / kBinChunk;
        for (int v = 0; v < nv; ++v) skip |= (unsigned)block_skip[(size_t)(v0 + v) * n_box + box] << v;  // uniform loads
    }
    return true;
}

// Sort key of a visible point: its 32x32 screen bin, then its 8x4 pixel tile inside the bin.  Entries of a tile are
// contiguous, so the fragments a tile kernel works on refer to a short range of entries and gradient rows: the 32
// gathers (or atomics) of a warp instruction touch a handful of 128-byte lines instead of 32 different ones.
constexpr int kSubShift = 5;  // 32 tiles (4 x 8) per bin
__device__ __forceinline__ int bin_key(const Geom& g, float u, float v)
{
    const int px = __float2int_rd(u), py = __float2int_rd(v);
    const int bin = (py >> kBinShift) * g.bins_x + (px >> kBinShift);
    return (bin << kSubShift) | (((py >> 2) & 7) << 2) | ((px >> 3) & 3);
}

// discard_point_for_confidence (RenderForward.cu:122-130): viewer only, points below the stability cut-off are not drawn
template <bool ACT>
__device__ __forceinline__ bool discarded_for_confidence(const ScenePtrs& sc, const TripsRenderParams& pr, int tex)
{
    if (!pr.viewer_only || (unsigned)tex >= (unsigned)sc.n_tex) return false;
    float c = __ldg(sc.confidence + tex);
    if (ACT && pr.confidence_is_raw) c = tm_sigmoid(pr.confidence_scale * c);
    return c < pr.stability_cutoff_value;
}

// What the scatter pass reads of a point; requested one point ahead.
struct PointHead
{
    float4 p;
    float raw;
    int tex;
    __device__ __forceinline__ void fetch(const ScenePtrs& sc, int i, int last)
    {
        if (i >= last) return;
        tex = sc.index ? __ldg(sc.index + i) : i;
        p   = __ldg(sc.position + i);
        raw = __ldg(sc.point_size + i);
    }
};

// ACT: the scene tensors may be raw parameters (fused texture preparation); compiled separately so that the common case
// carries none of its code.  One launch handles the views [v0, v0 + nv).
// A thread takes four points at a time, so that a camera is read from shared memory (24 words) once for four projections and four
// points are on their way from memory at once; the radius of a point is only computed where it is asked for.  Together with the
// projections that wait in shared memory in the scatter pass and cameras read four words at a time: bin_points 1204 -> 1097 us (6 M
// points x 8 views), 241 -> 206 (2 M x 4), 1733 -> 1660 (20 M x 2), 64 views of 10 M points 16.5 -> 15.4 ms.  Issue slots bound both
// passes (57 and 69 % in use before).
template <bool ACT>
__global__ __launch_bounds__(kBinThreads, kCountMinBlocks) void bin_count_kernel(ScenePtrs sc, const CamConst* cams, const __grid_constant__ Geom g,
                                                                TripsRenderParams pr, FwdBuffers fb, int v0, int nv, unsigned* ticket)
{
    follow_previous();
    __shared__ BinCam s_cam[kViewGroup];
    __shared__ unsigned s_ticket;
    for (int k = threadIdx.x; k < nv * (int)(sizeof(CamConst) / 4); k += kBinThreads) ((int*)s_cam)[k] = ((const int*)(cams + v0))[k];
    const bool use_dropout = pr.train && sc.dropout;  // the mask applies with and without viewer_only (RenderForward.cu:224-240)
    constexpr int kPoints = kBinTicket / kBinThreads;  // of a thread: a camera is read from shared memory once for all of them
    int first, last;
    unsigned skip;
    while (next_point_ticket(ticket, sc.N, &s_ticket, fb.block_skip, v0, nv, first, last, skip))
    {
        float4 p[kPoints];
        unsigned there = 0;
#pragma unroll
        for (int k = 0; k < kPoints; ++k)
        {
            const int i = first + (int)threadIdx.x + k * kBinThreads;
            p[k]        = make_float4(0.f, 0.f, 0.f, 0.f);
            if (i >= last) continue;
            p[k] = __ldg(sc.position + i);
            if (!(pr.viewer_only && discarded_for_confidence<ACT>(sc, pr, sc.index ? __ldg(sc.index + i) : i))) there |= 1u << k;
        }
        for (int v = 0; v < nv; ++v)
        {
            if ((skip >> v) & 1u) continue;  // uniform
            const BinCam cam = s_cam[v];
            uint32_t* counters = fb.bin_count + ((size_t)(v0 + v) * g.n_bins << kSubShift);
#pragma unroll
            for (int k = 0; k < kPoints; ++k)
            {
                if (!((there >> k) & 1u)) continue;
                if (use_dropout && __ldg(sc.dropout + (size_t)(v0 + v) * sc.N + first + threadIdx.x + k * kBinThreads) == 1.f) continue;
                float sp          = 0.f;  // (the size is not asked for)
                const Projected r = project_visible(cam, g, pr, p[k], 0.f, sp);
                if (r.ok) atomicAdd(counters + bin_key(g, r.u, r.v), 1u);
            }
        }
    }
}

// One block per view: visible points per key -> first entry (within the view) of every key, and of every screen bin;
// view_total[b] = visible points of the view.  A turn of the block covers 16384 keys, 16 consecutive ones per thread (64
// bytes, vector loads and stores): the turns follow one another, and with one key per thread a 1080p view (65 k keys) took
// 64 of them, each two dependent loads and three barriers long.
// Measured on a 1080p view: 90 us with one key per thread and turn; sixteen take the whole binning stage from 0.326 to 0.270 ms.
constexpr int kScanKeys = 16;

// One of `n` blocks that end with this call: true in all threads of the last one, which then sees what the others wrote before it.
__device__ __forceinline__ bool last_block(unsigned* finished, unsigned n)
{
    __shared__ unsigned s_last;
    __threadfence();
    __syncthreads();
    if (threadIdx.x == 0) s_last = atomicAdd(finished, 1u) == n - 1 ? 1u : 0u;
    __syncthreads();
    if (s_last) __threadfence();
    return s_last != 0;
}

// Where every view starts in a buffer of `cap` places, of which view b needs totals[b]: in the entry arrays and in the list buffer, which
// are sized from an earlier pass, not for the worst case.  In a training pass a view that does not fit gets no places: it renders
// as background, the status word says so (status_bit), and the host grows the buffer behind the number that was needed.  An inference pass
// (status_bit 0) that needs more than `most` is given up: no view gets any places, so that the kernels behind have nothing to do, and the
// host takes it up again here (launch_place_views).
__device__ __forceinline__ void place_views(const uint32_t* totals, int B, unsigned long long cap, unsigned long long most, unsigned long long* base,
                                            unsigned status_bit, GivenUp where, unsigned long long* need, DevStats* stats)
{
    unsigned long long at = 0, sum = 0;
    for (int b = 0; b < B; ++b)
    {
        const uint32_t n = __ldcg(totals + b);
        base[b]          = at;
        sum += n;
        if (at + n <= cap)
            at += n;
        else if (status_bit)
            atomicOr(&stats->status, status_bit);
    }
    base[B] = at;
    *need   = sum;
    if (status_bit || sum <= most) return;
    for (int b = 0; b <= B; ++b) base[b] = 0;
    stats->given_up = where;
}

__global__ __launch_bounds__(1024) void bin_scan_kernel(const uint32_t* counts, uint32_t* key_first,
                                                        uint32_t* bin_first, int n_keys, uint32_t* view_total, unsigned long long entry_cap,
                                                        unsigned long long* entry_base, bool report, PassGuess guess, unsigned* finished, DevStats* stats)
{
    follow_previous();
    __shared__ uint32_t sm[32];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int b    = blockIdx.x;
    const uint32_t* c = counts + (size_t)b * n_keys;  // n_keys is a multiple of 32: every row and every quad is 16-byte aligned
    uint32_t* w       = key_first + (size_t)b * n_keys;
    uint32_t* o       = bin_first + (size_t)b * (n_keys >> kSubShift);
    uint32_t carry    = 0;
    for (int s = 0; s < n_keys; s += 1024 * kScanKeys)
    {
        const int i0 = s + (int)threadIdx.x * kScanKeys;
        uint4 q[kScanKeys / 4];
#pragma unroll
        for (int k = 0; k < kScanKeys / 4; ++k) q[k] = i0 + 4 * k < n_keys ? *reinterpret_cast<const uint4*>(c + i0 + 4 * k) : make_uint4(0u, 0u, 0u, 0u);
        uint32_t sum = 0, most = 0;
#pragma unroll
        for (int k = 0; k < kScanKeys / 4; ++k)
        {
            sum += (q[k].x + q[k].y) + (q[k].z + q[k].w);
            most = max(most, max(max(q[k].x, q[k].y), max(q[k].z, q[k].w)));
        }
        if (most >= kHotKey) atomicMax(&stats->max_key, most);  // crowded group: the next call uses the aggregating binning kernels
        uint32_t inc = sum;
#pragma unroll
        for (int k = 1; k < 32; k <<= 1)
        {
            const uint32_t t = __shfl_up_sync(kFull, inc, k);
            if (lane >= k) inc += t;
        }
        if (lane == 31) sm[warp] = inc;
        __syncthreads();
        const uint32_t wsum = sm[lane];
        uint32_t winc       = wsum;
#pragma unroll
        for (int k = 1; k < 32; k <<= 1)
        {
            const uint32_t t = __shfl_up_sync(kFull, winc, k);
            if (lane >= k) winc += t;
        }
        const uint32_t total = __shfl_sync(kFull, winc, 31);
        uint32_t run         = carry + __shfl_sync(kFull, winc - wsum, warp) + inc - sum;
        if (i0 < n_keys && (i0 & ((1 << kSubShift) - 1)) == 0) o[i0 >> kSubShift] = run;
#pragma unroll
        for (int k = 0; k < kScanKeys / 4; ++k)
        {
            const uint4 v = make_uint4(run, run + q[k].x, run + q[k].x + q[k].y, run + q[k].x + q[k].y + q[k].z);
            run           = v.w + q[k].w;
            if (i0 + 4 * k < n_keys) *reinterpret_cast<uint4*>(w + i0 + 4 * k) = v;
        }
        carry += total;
        __syncthreads();  // the warp sums are overwritten by the next turn
    }
    if (threadIdx.x == 0) view_total[b] = carry;
    if (!last_block(finished, gridDim.x) || threadIdx.x != 0) return;
    // An inference pass was launched with the kernels that suit the pass before.  One that calls for the other scatter kernel or has many
    // more entries is given up as well: the host now knows better.  Two views of a cloud in turn, us, with the kernels of the view before /
    // given up: 3 M points in 100x100 pixels and near by 1788 / 1615 for the pair, 20 M points after a view that sees 0.4 M of them
    // 2609 / 2450.  In passes of 8 views the scatter kernel matters less than the time it takes to give up: 13.59 / 13.73 ms for 32 views.
    unsigned long long most = entry_cap;
    if (guess.look)
    {
        most = min(most, max(kGuessFactor * guess.entries, kGuessEntries));
        if ((__ldcg(&stats->max_key) >= kHotKey) != guess.hot) most = 0;
    }
    place_views(view_total, (int)gridDim.x, entry_cap, most, entry_base, report ? TRIPS_DEV_ENTRY_OVERFLOW : 0u, kGivenUpEntries, &stats->visible, stats);
}

// One 32-byte store (sm_100 has 256-bit global stores) for the two float4 halves of a 32-byte-aligned record: half the
// store instructions of the entry scatter, each covering a whole sector.
__device__ __forceinline__ void store_entry_head(float4* dst, const float4& a, const float4& b)
{
    // Entries of one screen tile are written by many point blocks at different times.  Keeping the written lines in L2 for as
    // long as it will hold them lets neighbouring 32-byte sectors meet in one line before it goes to DRAM (measured: the
    // scatter pass 3 % faster than with the default policy, evict_first no different from the default).
    uint64_t policy;
    asm volatile("createpolicy.fractional.L2::evict_last.b64 %0, 1.0;" : "=l"(policy));
    asm volatile("st.global.L2::cache_hint.v8.f32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8}, %9;" ::"l"(dst), "f"(a.x), "f"(a.y), "f"(a.z), "f"(a.w), "f"(b.x), "f"(b.y),
                 "f"(b.z), "f"(b.w), "l"(policy)
                 : "memory");
}

// What an entry carries of its point besides the projection: fetched once per point, when it turns out visible in a view.
template <int C>
struct PointRow
{
    static constexpr int C4 = (C + 3) & ~3;
    bool fetched = false, tex_ok = false;
    int tex      = 0;
    float conf   = 0.f;
    float row[C4];
};

template <int C, bool ACT>
__device__ __forceinline__ void fetch_point_row(const ScenePtrs& sc, const TripsRenderParams& pr, const FwdBuffers& fb, int i, PointRow<C>& d)
{
    if (d.fetched) return;
    d.fetched = true;
    if (d.tex_ok)
    {
        d.conf = __ldg(sc.confidence + d.tex);
        if (ACT && pr.confidence_is_raw) d.conf = tm_sigmoid(pr.confidence_scale * d.conf);  // PrepareConfidence, NeuralTexture.h:40-43
    }
    else
        atomicOr(&fb.stats->status, TRIPS_DEV_BAD_TEXTURE_INDEX);  // the point is drawn with alpha 0
#pragma unroll
    for (int c = 0; c < PointRow<C>::C4; ++c) d.row[c] = (c < C && d.tex_ok) ? __ldg(sc.texture + (size_t)c * sc.n_tex + d.tex) : 0.f;
    if (ACT && pr.texture_abs)  // PrepareTexture, NeuralTexture.h:45-57
    {
#pragma unroll
        for (int c = 0; c < PointRow<C>::C4; ++c) d.row[c] = fabsf(d.row[c]);
    }
}

// Writes entry `at` (index into the entry arrays) of point i as projected by `r`.
template <int C>
__device__ __forceinline__ void write_entry(const FwdBuffers& fb, const Geom& g, const TripsRenderParams& pr, const CamConst& cam, unsigned long long at, int i,
                                            const float4& p, float raw, const Projected& r, const PointRow<C>& d)
{
    constexpr int TS = tail_stride(C);
    constexpr int C4 = PointRow<C>::C4;
    // layers first..hi, stopping where the 2x2 footprint leaves the layer (RenderForward.cu:342-363).  first = 0 except for
    // the strict write of the second pipeline, which starts at the layer below log2(size) (RenderForward.cu:2291-2393);
    // without use_layer_point_size every layer is written (RenderForward.cu:1611-1631).  The entry stores the NUMBER of
    // layers; the first layer of a strict entry is recomputed from its size where needed (strict_first_layer).
    int hi = 0, first = 0;
    if (!pr.use_layer_point_size)
        hi = g.L - 1;
    else if (r.ps > 1.f)
    {
        hi = min(tm_ceil_log2(r.ps), g.L - 1);
        if (!pr.render_points_in_all_lower_resolutions) first = min(tm_floor_log2(r.ps), g.L - 1);
    }
    // A point whose footprint lies inside all layers 0..hi, as nearly all do, needs no look at each of them (floor(u / 2^l) < W_l - 1
    // exactly when u < (W_l - 1) 2^l).  The walk over the layers took as many turns as the largest point of the warp has layers: bin_points,
    // us, 1080p frame of 6 M points 234 -> 221, 2 M points x 4 views 194 -> 184, 20 M x 2 1649 -> 1616, 64 views of 10 M 15530 -> 15130.
    int layer = first;
    if (first == 0 && !pr.drop_out_points_by_radius && r.u < g.inside_x[hi] && r.v < g.inside_y[hi])
        layer = hi + 1;
    else
    {
        const bool second = second_pipeline(pr);
        const float sc0   = __int_as_float((127 - first) << 23);  // 2^-first
        float x = r.u * sc0, y = r.v * sc0, rad = pr.drop_out_points_by_radius ? projected_radius(cam, p, r.z) * sc0 : 0.f;
        for (; layer < hi + 1; ++layer, x *= 0.5f, y *= 0.5f, rad *= 0.5f)
        {
            const int px = __float2int_rd(x), py = __float2int_rd(y);
            if (px < 0 || px >= g.W[layer] - 1 || py < 0 || py >= g.H[layer] - 1) break;
            if (pr.drop_out_points_by_radius && (second ? rad : (float)(int)rad) < pr.drop_out_radius_threshold) break;
        }
    }
    store_entry_head(fb.ent_head + at * 2, make_float4(r.u, r.v, r.ps, d.conf),
                     make_float4(__int_as_float(i), r.z, raw, __int_as_float(layer - first)));
    float4* e = reinterpret_cast<float4*>(fb.ent_tail + at * TS);
    if constexpr (C4 == 4)
        store_entry_head(e, make_float4(p.x, p.y, p.z, __int_as_float(d.tex_ok ? d.tex : -1)), make_float4(d.row[0], d.row[1], d.row[2], d.row[3]));
    else
    {
        e[0] = make_float4(p.x, p.y, p.z, __int_as_float(d.tex_ok ? d.tex : -1));
#pragma unroll
        for (int c = 0; c < C4; c += 4) e[1 + c / 4] = make_float4(d.row[c], d.row[c + 1], d.row[c + 2], d.row[c + 3]);
    }
}

template <int C, bool ACT>
__global__ __launch_bounds__(kBinThreads, (C <= 4 ? kScatterMinBlocks : kScatterMinBlocksWide)) void bin_scatter_kernel(ScenePtrs sc, const CamConst* cams, const __grid_constant__ Geom g,
                                                                  TripsRenderParams pr, FwdBuffers fb, int v0, int nv, unsigned* ticket)
{
    follow_previous();
    __shared__ BinCam s_cam[kViewGroup];
    __shared__ unsigned long long s_ebase[kViewGroup + 1];
    __shared__ unsigned s_ticket;
    __shared__ float4 s_proj[kSweep][kBinThreads];  // u v z ps of the thread's visible views of a sweep
    for (int k = threadIdx.x; k < nv * (int)(sizeof(CamConst) / 4); k += kBinThreads) ((int*)s_cam)[k] = ((const int*)(cams + v0))[k];
    if (threadIdx.x <= nv) s_ebase[threadIdx.x] = fb.entry_base[v0 + threadIdx.x];
    __syncthreads();
    unsigned no_room = 0;  // views without entries: nothing visible, or the view did not fit the entry arrays
    for (int v = 0; v < nv; ++v) no_room |= (s_ebase[v + 1] == s_ebase[v] ? 1u : 0u) << v;
    if (!fb.point_state && s_ebase[0] == s_ebase[nv]) return;  // nothing to write (a training pass still notes its points)
    const bool use_dropout = pr.train && sc.dropout;
    int first, last;
    unsigned skip;
    while (next_point_ticket(ticket, sc.N, &s_ticket, fb.block_skip, v0, nv, first, last, skip))
    {
        skip |= no_room;
        PointHead nx;
        nx.fetch(sc, first + threadIdx.x, last);
        for (int i = first + threadIdx.x; i < last; i += kBinThreads)
        {
            const PointHead h = nx;
            nx.fetch(sc, i + kBinThreads, last);
            PointRow<C> d;
            d.tex    = h.tex;
            d.tex_ok = (unsigned)d.tex < (unsigned)sc.n_tex;
            if (discarded_for_confidence<ACT>(sc, pr, d.tex))
            {
                if (fb.note_entry)
                    for (int v = 0; v < nv; ++v) fb.note_entry[(size_t)(v0 + v) * sc.N + i] = kNoEntry;
                continue;
            }
            const float4 p  = h.p;
            const float raw = h.raw;
            if (fb.point_state && v0 == 0) fb.point_state[i] = make_float4(p.x, p.y, p.z, raw);
            float sp        = -1.f;
            // Views are handled kSweep at a time in two sweeps: the first projects and takes the entry slots (up to kSweep
            // returning atomics in flight per thread instead of one), the second writes the entries.  Waiting for each slot before
            // the next projection made the kernel latency-bound.
            for (int vb = 0; vb < nv; vb += kSweep)
            {
                uint32_t slot[kSweep];
                unsigned vis = 0;
#pragma unroll
                for (int j = 0; j < kSweep; ++j)
                {
                    const int v = vb + j;
                    slot[j]     = kNoEntry;
                    if (v >= nv || ((skip >> v) & 1u)) continue;  // uniform
                    if (use_dropout && __ldg(sc.dropout + (size_t)(v0 + v) * sc.N + i) == 1.f) continue;
                    const Projected r = project_visible(s_cam[v], g, pr, p, raw, sp);
                    if (!r.ok) continue;
                    vis |= 1u << j;
                    s_proj[j][threadIdx.x] = make_float4(r.u, r.v, r.z, r.ps);
                    slot[j] = atomicAdd(fb.bin_base + ((size_t)(v0 + v) * g.n_bins << kSubShift) + bin_key(g, r.u, r.v), 1u);
                }
                if (vis) fetch_point_row<C, ACT>(sc, pr, fb, i, d);  // travels with the slots
#pragma unroll
                for (int j = 0; j < kSweep; ++j)
                {
                    if (!((vis >> j) & 1u)) continue;
                    const int v     = vb + j;
                    const float4 uv = s_proj[j][threadIdx.x];
                    Projected r;
                    r.u = uv.x, r.v = uv.y, r.z = uv.z, r.ps = uv.w, r.ok = true;
                    write_entry<C>(fb, g, pr, s_cam[v], s_ebase[v] + slot[j], i, p, raw, r, d);
                }
                if (fb.note_entry)  // behind the entries
#pragma unroll
                    for (int j = 0; j < kSweep; ++j)
                        if (vb + j < nv) fb.note_entry[(size_t)(v0 + vb + j) * sc.N + i] = slot[j];
            }
        }
    }
}

// ------------------------------------------------------------------------------------------------------------
// The same two passes for point clouds that crowd into a few screen tiles (a distant or tiny object: millions of points
// in a 64x64-pixel window).  There the per-(bin, tile) counters above become a handful of addresses that every thread
// of the machine updates, and same-address atomics are served one after the other.  These variants aggregate in shared
// memory first: a block takes a ticket of kHotTicket points, counts its visible point-views per key in a small hash
// table (linear probing, at most four probes; a key that finds no slot simply uses the global counter directly), and
// touches the global counter of every key it met once per ticket.  In the scatter pass that one returning atomic
// reserves a range of the key's entries for the whole ticket, and the slots inside the range come from the table.
// They run when the previous pass saw more than kHotKey visible points in one (view, bin, tile) group; the scatter pass of an inference or
// a sized call goes by its own counts (bin_scan_kernel); ordinary scenes never do and run the kernels above.
// ------------------------------------------------------------------------------------------------------------
constexpr int kHotTicket        = 2048;
constexpr int kHotSlots         = 2048;
constexpr uint32_t kHotEmpty    = 0xffffffffu;

__device__ __forceinline__ uint32_t hot_hash(uint32_t key) { return (key * 2654435761u) >> 21; }  // 11 bits

__device__ __forceinline__ int hot_find_or_insert(uint32_t* tag, uint32_t key)
{
    const uint32_t h = hot_hash(key);
#pragma unroll
    for (int probe = 0; probe < 4; ++probe)
    {
        const uint32_t s   = (h + probe) & (kHotSlots - 1);
        const uint32_t old = atomicCAS(tag + s, kHotEmpty, key);
        if (old == kHotEmpty || old == key) return (int)s;
    }
    return -1;
}

__device__ __forceinline__ int hot_find(const uint32_t* tag, uint32_t key)
{
    const uint32_t h = hot_hash(key);
#pragma unroll
    for (int probe = 0; probe < 4; ++probe)
    {
        const uint32_t s = (h + probe) & (kHotSlots - 1);
        const uint32_t t = tag[s];
        if (t == key) return (int)s;
        if (t == kHotEmpty) return -1;
    }
    return -1;
}

__device__ __forceinline__ bool next_hot_ticket(unsigned* ticket, int N, unsigned* s_ticket, int& first, int& last)
{
    __syncthreads();
    if (threadIdx.x == 0) *s_ticket = atomicAdd(ticket, 1u);
    __syncthreads();
    const unsigned t = *s_ticket;
    if (t >= ((unsigned)N + kHotTicket - 1) / kHotTicket) return false;
    first = (int)(t * kHotTicket);
    last  = min(N, first + kHotTicket);
    return true;
}

template <bool ACT>
__global__ __launch_bounds__(kBinThreads) void bin_count_hot_kernel(ScenePtrs sc, const CamConst* cams, const __grid_constant__ Geom g,
                                                                    TripsRenderParams pr, FwdBuffers fb, int v0, int nv, unsigned* ticket)
{
    follow_previous();
    __shared__ BinCam s_cam[kViewGroup];
    __shared__ uint32_t s_tag[kHotSlots], s_cnt[kHotSlots];
    __shared__ unsigned s_ticket;
    for (int k = threadIdx.x; k < nv * (int)(sizeof(CamConst) / 4); k += kBinThreads) ((int*)s_cam)[k] = ((const int*)(cams + v0))[k];
    const bool use_dropout = pr.train && sc.dropout;
    const uint32_t n_keys  = (uint32_t)g.n_bins << kSubShift;
    uint32_t* counters     = fb.bin_count + (size_t)v0 * n_keys;  // counter of (view v0 + v, key) at [v * n_keys + key]
    int first, last;
    while (next_hot_ticket(ticket, sc.N, &s_ticket, first, last))
    {
        for (int k = threadIdx.x; k < kHotSlots; k += kBinThreads) s_tag[k] = kHotEmpty, s_cnt[k] = 0u;
        __syncthreads();
        for (int i = first + threadIdx.x; i < last; i += kBinThreads)
        {
            const int tex = sc.index ? __ldg(sc.index + i) : i;
            if (discarded_for_confidence<ACT>(sc, pr, tex)) continue;
            const float4 p  = __ldg(sc.position + i);
            const float raw = __ldg(sc.point_size + i);
            float sp        = -1.f;
            for (int v = 0; v < nv; ++v)
            {
                if (use_dropout && __ldg(sc.dropout + (size_t)(v0 + v) * sc.N + i) == 1.f) continue;
                const Projected r = project_visible(s_cam[v], g, pr, p, raw, sp);
                if (!r.ok) continue;
                const uint32_t key = (uint32_t)v * n_keys + (uint32_t)bin_key(g, r.u, r.v);
                const int s        = hot_find_or_insert(s_tag, key);
                if (s >= 0)
                    atomicAdd(s_cnt + s, 1u);
                else
                    atomicAdd(counters + key, 1u);
            }
        }
        __syncthreads();
        for (int k = threadIdx.x; k < kHotSlots; k += kBinThreads)
            if (s_tag[k] != kHotEmpty) atomicAdd(counters + s_tag[k], s_cnt[k]);
    }
}

template <int C, bool ACT>
__global__ __launch_bounds__(kBinThreads) void bin_scatter_hot_kernel(ScenePtrs sc, const CamConst* cams, const __grid_constant__ Geom g,
                                                                      TripsRenderParams pr, FwdBuffers fb, int v0, int nv, unsigned* ticket)
{
    follow_previous();
    __shared__ BinCam s_cam[kViewGroup];
    __shared__ unsigned long long s_ebase[kViewGroup + 1];
    __shared__ uint32_t s_tag[kHotSlots], s_cnt[kHotSlots], s_base[kHotSlots];
    __shared__ unsigned s_ticket;
    for (int k = threadIdx.x; k < nv * (int)(sizeof(CamConst) / 4); k += kBinThreads) ((int*)s_cam)[k] = ((const int*)(cams + v0))[k];
    if (threadIdx.x <= nv) s_ebase[threadIdx.x] = fb.entry_base[v0 + threadIdx.x];
    __syncthreads();
    unsigned no_room = 0;  // views without entries: nothing visible, or the view did not fit the entry arrays
    for (int v = 0; v < nv; ++v) no_room |= (s_ebase[v + 1] == s_ebase[v] ? 1u : 0u) << v;
    if (!fb.point_state && s_ebase[0] == s_ebase[nv]) return;  // nothing to write (a training pass still notes its points)
    const bool use_dropout = pr.train && sc.dropout;
    const uint32_t n_keys  = (uint32_t)g.n_bins << kSubShift;
    uint32_t* cursors      = fb.bin_base + (size_t)v0 * n_keys;
    int first, last;
    while (next_hot_ticket(ticket, sc.N, &s_ticket, first, last))
    {
        for (int k = threadIdx.x; k < kHotSlots; k += kBinThreads) s_tag[k] = kHotEmpty, s_cnt[k] = 0u;
        __syncthreads();
        // ---- the ticket's visible point-views per key ----
        for (int i = first + threadIdx.x; i < last; i += kBinThreads)
        {
            const int tex = sc.index ? __ldg(sc.index + i) : i;
            if (discarded_for_confidence<ACT>(sc, pr, tex)) continue;
            const float4 p  = __ldg(sc.position + i);
            const float raw = __ldg(sc.point_size + i);
            if (fb.point_state && v0 == 0) fb.point_state[i] = make_float4(p.x, p.y, p.z, raw);
            float sp        = -1.f;
            for (int v = 0; v < nv; ++v)
            {
                if ((no_room >> v) & 1u) continue;  // uniform
                if (use_dropout && __ldg(sc.dropout + (size_t)(v0 + v) * sc.N + i) == 1.f) continue;
                const Projected r = project_visible(s_cam[v], g, pr, p, raw, sp);
                if (!r.ok) continue;
                const int s = hot_find_or_insert(s_tag, (uint32_t)v * n_keys + (uint32_t)bin_key(g, r.u, r.v));
                if (s >= 0) atomicAdd(s_cnt + s, 1u);
            }
        }
        __syncthreads();
        // ---- one returning atomic per key reserves the ticket's range of that key's entries ----
        for (int k = threadIdx.x; k < kHotSlots; k += kBinThreads)
            if (s_tag[k] != kHotEmpty)
            {
                s_base[k] = atomicAdd(cursors + s_tag[k], s_cnt[k]);
                s_cnt[k]  = 0u;
            }
        __syncthreads();
        // ---- the same point-views again (the same arithmetic, hence the same keys): slots from the table, entries out ----
        for (int i = first + threadIdx.x; i < last; i += kBinThreads)
        {
            PointRow<C> d;
            d.tex    = sc.index ? __ldg(sc.index + i) : i;
            d.tex_ok = (unsigned)d.tex < (unsigned)sc.n_tex;
            if (discarded_for_confidence<ACT>(sc, pr, d.tex))
            {
                if (fb.note_entry)
                    for (int v = 0; v < nv; ++v) fb.note_entry[(size_t)(v0 + v) * sc.N + i] = kNoEntry;
                continue;
            }
            const float4 p  = __ldg(sc.position + i);
            const float raw = __ldg(sc.point_size + i);
            float sp        = -1.f;
            for (int v = 0; v < nv; ++v)
            {
                uint32_t slot = kNoEntry;
                Projected r;
                if (!((no_room >> v) & 1u) && !(use_dropout && __ldg(sc.dropout + (size_t)(v0 + v) * sc.N + i) == 1.f))
                {
                    r = project_visible(s_cam[v], g, pr, p, raw, sp);
                    if (r.ok)
                    {
                        fetch_point_row<C, ACT>(sc, pr, fb, i, d);
                        const uint32_t key = (uint32_t)v * n_keys + (uint32_t)bin_key(g, r.u, r.v);
                        const int s        = hot_find(s_tag, key);
                        slot               = s >= 0 ? s_base[s] + atomicAdd(s_cnt + s, 1u) : atomicAdd(cursors + key, 1u);
                    }
                }
                if (fb.note_entry) fb.note_entry[(size_t)(v0 + v) * sc.N + i] = slot;
                if (slot == kNoEntry) continue;
                write_entry<C>(fb, g, pr, s_cam[v], s_ebase[v] + slot, i, p, raw, r, d);
            }
        }
    }
}

// Count pass of the binning stage: bounding boxes, visible points per (view, bin, tile), their exclusive scan and the
// first entry of every view.  After it fb.view_total / stats->visible say how many entries the scatter pass will write.
cudaError_t launch_bin_count(const ScenePtrs& sc, const CamConst* cams, const Geom& g, const TripsRenderParams& pr, int B,
                             const FwdBuffers& fb, unsigned long long entry_cap, PassGuess guess, int sm_count, cudaStream_t st)
{
    const bool hot     = guess.hot;
    const int n_keys   = g.n_bins << kSubShift;
    const int grid     = sm_count * kBinBlocksPerSM;
    const int n_groups = (B + kViewGroup - 1) / kViewGroup;
    if (sc.N > 0 && fb.block_skip)
        launch_following(block_visibility_kernel, (sc.N + kBinChunk - 1) / kBinChunk, 256, st, sc.position, sc.N, cams, g, B, const_cast<uint8_t*>(fb.block_skip), fb.stats);
    const bool act = pr.confidence_is_raw || pr.texture_abs;
    if (sc.N > 0)
        for (int gi = 0; gi < n_groups; ++gi)
        {
            const int v0 = gi * kViewGroup, nv = min(kViewGroup, B - v0);
            if (hot && act)
                launch_following(bin_count_hot_kernel<true>, grid, kBinThreads, st, sc, cams, g, pr, fb, v0, nv, fb.ticket + gi);
            else if (hot)
                launch_following(bin_count_hot_kernel<false>, grid, kBinThreads, st, sc, cams, g, pr, fb, v0, nv, fb.ticket + gi);
            else if (act)
                launch_following(bin_count_kernel<true>, grid, kBinThreads, st, sc, cams, g, pr, fb, v0, nv, fb.ticket + gi);
            else
                launch_following(bin_count_kernel<false>, grid, kBinThreads, st, sc, cams, g, pr, fb, v0, nv, fb.ticket + gi);
        }
    launch_following(bin_scan_kernel, B, 1024, st, fb.bin_count, fb.bin_base, fb.bin_cursor, n_keys, fb.view_total, entry_cap, fb.entry_base, fb.report_overflow, guess, fb.finished, fb.stats);
    return cudaGetLastError();
}

int bin_count_launches(int N, int B) { return 1 + (N > 0 ? 1 + (B + kViewGroup - 1) / kViewGroup : 0); }
int bin_scatter_launches(int N, int B) { return N > 0 ? (B + kViewGroup - 1) / kViewGroup : 0; }

// Scatter pass of the binning stage: writes the entries (the arrays must hold fb.entry_base[B] entries).
cudaError_t launch_bin_scatter(const ScenePtrs& sc, const CamConst* cams, const Geom& g, const TripsRenderParams& pr, int B,
                               const FwdBuffers& fb, bool hot, int sm_count, cudaStream_t st)
{
    if (sc.N <= 0) return cudaSuccess;
    const int grid     = sm_count * kBinBlocksPerSM;
    const int n_groups = (B + kViewGroup - 1) / kViewGroup;
    const bool act     = pr.confidence_is_raw || pr.texture_abs;
    for (int gi = 0; gi < n_groups; ++gi)
    {
        const int v0 = gi * kViewGroup, nv = min(kViewGroup, B - v0);
        unsigned* tk = fb.ticket + n_groups + gi;
#define TRIPS_SCATTER_CASE(CC)                                                                                    \
    case CC:                                                                                                      \
        if (hot && act)                                                                                           \
            launch_following(bin_scatter_hot_kernel<CC, true>, grid, kBinThreads, st, sc, cams, g, pr, fb, v0, nv, tk);     \
        else if (hot)                                                                                             \
            launch_following(bin_scatter_hot_kernel<CC, false>, grid, kBinThreads, st, sc, cams, g, pr, fb, v0, nv, tk);    \
        else if (act)                                                                                             \
            launch_following(bin_scatter_kernel<CC, true>, grid, kBinThreads, st, sc, cams, g, pr, fb, v0, nv, tk);         \
        else                                                                                                      \
            launch_following(bin_scatter_kernel<CC, false>, grid, kBinThreads, st, sc, cams, g, pr, fb, v0, nv, tk);        \
        break;
        switch (sc.C)
        {
            TRIPS_SCATTER_CASE(3)
            TRIPS_SCATTER_CASE(4)
            TRIPS_SCATTER_CASE(6)
            TRIPS_SCATTER_CASE(8)
            TRIPS_SCATTER_CASE(16)
            default: return cudaErrorInvalidValue;
        }
#undef TRIPS_SCATTER_CASE
    }
    return cudaGetLastError();
}

// ------------------------------------------------------------------------------------------------------------
// list starts.  The lists of a view need not follow one another in pixel order: a block scans the lengths of kScanChunk consecutive
// pixels and takes a range of the view's list buffer for them from the view's counter.  One pass over the lengths and one
// kernel; chunk totals, their scan and a second pass over the lengths, which this replaces, were three.
// ------------------------------------------------------------------------------------------------------------
__device__ __forceinline__ uint32_t warp_incl_scan(uint32_t v, int lane)
{
#pragma unroll
    for (int o = 1; o < 32; o <<= 1)
    {
        uint32_t t = __shfl_up_sync(kFull, v, o);
        if (lane >= o) v += t;
    }
    return v;
}

// A warp takes 32 consecutive lengths at a time, kScanPerLane times: the lists of neighbouring pixels are neighbours.
// cursor: [B] fragments of the views so far, zero before; finished: blocks that are done, zero before.
__global__ __launch_bounds__(kScanThreads) void list_starts_kernel(const unsigned long long* entry_base, const uint32_t* counts, int P, int k_keep, uint32_t* offsets, uint32_t* cursor,
                                                                   unsigned* finished, unsigned long long* view_base, unsigned long long frag_cap, bool report,
                                                                   DevStats* stats, HeavyLists heavy)
{
    follow_previous();
    __shared__ uint32_t s_warp[kScanThreads / 32], s_kept[kScanThreads / 32], s_most[kScanThreads / 32], s_base;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int b           = blockIdx.y;
    const uint32_t* c     = counts + (size_t)b * P;
    const int start       = blockIdx.x * kScanChunk + warp * 32 * kScanPerLane + lane;
    uint32_t v[kScanPerLane], sum = 0, kept = 0, mx = 0;
#pragma unroll
    for (int k = 0; k < kScanPerLane; ++k) v[k] = start + k * 32 < P ? c[start + k * 32] : 0u;
    // No view has an entry, in a pass that was given up above all: no lists.  The collect pass must not meet the starts of an earlier
    // pass.  (Looked at while the lengths are on their way; `stats` lies on a line that all blocks update.)
    if (entry_base[gridDim.y] == 0)
    {
        if (blockIdx.x == 0 && blockIdx.y == 0)
            for (int w = threadIdx.x; w <= (int)gridDim.y; w += kScanThreads) view_base[w] = 0;
        return;
    }
#pragma unroll
    for (int k = 0; k < kScanPerLane; ++k)
    {
        sum += v[k];
        kept += min(v[k], (uint32_t)k_keep);
        mx = max(mx, v[k]);
    }
    // lists worth a block of their own, or several (heavy_topk_kernel): a warp reserves the items of its lists together (one
    // atomic per list queued up where most lists are long: 90 k long lists of 88x88 pixels in 11 views 0.041 -> 0.025 ms)
    if (__any_sync(kFull, mx > (uint32_t)kHeavyList))
    {
        auto parts_of  = [](uint32_t n) { return n > (uint32_t)kHeavyList ? min((n - 1) / kHeavyPart + 1, (uint32_t)kHeavyParts) : 0u; };
        uint32_t items = 0, shared_items = 0;
#pragma unroll
        for (int k = 0; k < kScanPerLane; ++k)
        {
            const uint32_t parts = parts_of(v[k]);
            items += parts;
            shared_items += parts > 1 ? parts : 0u;
        }
        const uint32_t items_incl = warp_incl_scan(items, lane), shared_incl = warp_incl_scan(shared_items, lane);
        uint32_t slot = 0, shared = 0;
        if (lane == 31)
        {
            slot = atomicAdd(&stats->n_heavy, items_incl);
            if (shared_incl) shared = atomicAdd(&stats->n_shared, shared_incl);
        }
        slot   = __shfl_sync(kFull, slot, 31) + items_incl - items;
        shared = __shfl_sync(kFull, shared, 31) + shared_incl - shared_items;
#pragma unroll 1
        for (int k = 0; k < kScanPerLane; ++k)
        {
            const uint32_t n     = c[min(start + k * 32, P - 1)];
            const uint32_t parts = start + k * 32 < P ? parts_of(n) : 0u;
            // no room for its parts: one block takes the whole list, the other items stay empty
            const bool whole = parts > 1 && shared + parts > heavy.shared_cap;
            if (parts > 1 && !whole) heavy.finished[shared] = 0;
            for (uint32_t t = 0; t < parts && slot + t < heavy.cap; ++t)
                heavy.item[slot + t] = make_uint4((unsigned)b, (unsigned)(start + k * 32), whole ? (t == 0 ? 1u << 16 : 0u) : t | parts << 16, shared);
            slot += parts;
            shared += parts > 1 ? parts : 0u;
        }
    }
    sum  = __reduce_add_sync(kFull, sum);
    kept = __reduce_add_sync(kFull, kept);
    mx   = __reduce_max_sync(kFull, mx);
    if (lane == 0) s_warp[warp] = sum, s_kept[warp] = kept, s_most[warp] = mx;
    __syncthreads();
    const uint32_t w = lane < kScanThreads / 32 ? s_warp[lane] : 0u;
    if (warp == 0)  // one update of the call's counters per block
    {
        kept = __reduce_add_sync(kFull, lane < kScanThreads / 32 ? s_kept[lane] : 0u);
        mx   = __reduce_max_sync(kFull, lane < kScanThreads / 32 ? s_most[lane] : 0u);
        if (lane == 0 && mx) atomicMax(&stats->max_len, mx), atomicAdd(&stats->kept, (unsigned long long)kept);
    }
    const uint32_t w_incl = warp_incl_scan(w, lane);
    const uint32_t total  = __shfl_sync(kFull, w_incl, 31);
    if (threadIdx.x == 0) s_base = total ? atomicAdd(cursor + b, total) : 0u;
    __syncthreads();
    uint32_t run = s_base + __shfl_sync(kFull, w_incl - w, warp);
#pragma unroll
    for (int k = 0; k < kScanPerLane; ++k)
    {
        const uint32_t incl = warp_incl_scan(v[k], lane);
        if (start + k * 32 < P) offsets[(size_t)b * P + start + k * 32] = run + incl - v[k];
        run += __shfl_sync(kFull, incl, 31);
    }
    if (!last_block(finished, gridDim.x * gridDim.y) || threadIdx.x != 0) return;
    // First fragment of every view.  A view without places: the collect pass skips it and the blend treats its lists as empty.
    place_views(cursor, (int)gridDim.y, frag_cap, frag_cap, view_base, report ? TRIPS_DEV_FRAGMENT_OVERFLOW : 0u, kGivenUpLists, &stats->frag_need, stats);
}

// Takes up an inference pass that was given up (place_views); the buffer is large enough now.
__global__ void place_views_kernel(const uint32_t* totals, int B, unsigned long long* base, unsigned long long* need, unsigned* ticket_blend, DevStats* stats)
{
    follow_previous();
    place_views(totals, B, ~0ull, ~0ull, base, 0u, kNotGivenUp, need, stats);
    stats->given_up = kNotGivenUp;
    *ticket_blend   = 0;  // the blend that gave up had asked for tiles
}

cudaError_t launch_place_views(int B, const FwdBuffers& fb, bool entries, cudaStream_t st)
{
    launch_following(place_views_kernel, 1, 1, st, entries ? fb.view_total : fb.list_cursor, B, entries ? fb.entry_base : fb.view_base,
                     entries ? &fb.stats->visible : &fb.stats->frag_need, fb.ticket_blend, fb.stats);
    return cudaGetLastError();
}

cudaError_t launch_list_starts(const Geom& g, int B, int k_keep, const FwdBuffers& fb, cudaStream_t st)
{
    launch_following(list_starts_kernel, dim3((g.P + kScanChunk - 1) / kScanChunk, B), kScanThreads, st, fb.entry_base, fb.counts, g.P, k_keep, fb.offsets, fb.list_cursor, fb.finished + 1,
                                                                                    fb.view_base, fb.frag_cap, fb.report_overflow, fb.stats, fb.heavy);
    return cudaGetLastError();
}

// ------------------------------------------------------------------------------------------------------------
// count and collect: fragments into per-pixel lists, with the list counters of a screen bin held in shared memory
//
// Entries are in bin order, and every fragment of a bin's points lands inside the bin's window: on layer l the
// pixels [x0, x0 + w_l) x [y0, y0 + w_l) with x0 = (32 bx) >> l and w_l = (31 >> l) + 3 (the 2x2 footprint adds one
// pixel).  A block takes a chunk of consecutive entries, and for each bin the chunk touches it
//   count pass:   counts the fragments per window pixel with shared-memory atomics and adds every non-zero window
//                 counter to the global list length once;
//   collect pass: counts the same way, reserves for each window pixel a contiguous range of its list with ONE
//                 returning global atomic, then hands out slots inside the ranges with shared-memory atomics and
//                 writes the 16-byte fragments: the 64-bit sort key (depth bits << 32 | point id), alpha and the
//                 entry index.
// This replaces one global atomic per fragment (SplattingPass, RenderForward.cu:368-436, and the counting half of
// CountAndCollectTiled, :347-362) by one per (chunk, touched pixel).  alpha = bilinear * confidence * layer factor
// in the operation order of FastSortFusedNew (RenderForward.cu:882-899) is computed here, where every thread holds
// a whole point, and travels with the fragment.
// ------------------------------------------------------------------------------------------------------------
constexpr int kWinChunkCount   = 4096;  // entries per block ticket, counting pass
constexpr int kWinSparse       = 512;   // entries of a bin up to which the window of shared-memory counters is bypassed
constexpr int kWinChunkCountFew = 1024;  // the same when the call has too few entries for kWinTicketsPerBlock tickets of 4096 per resident block:
constexpr int kWinTicketsPerBlock = 6;   // measured count pass, tickets of 4096 / 1024: config 4 (2 views, 16 M entries) 0.58 / 0.25 ms, config 2
                                         // (4 M) 0.093 / 0.09 ms; config 3 (27 M) 0.31 / 0.52 ms, config 5 (39 M) 0.40 / 0.53 ms
constexpr int kWinChunkCollect = 1024;  // and collecting pass: the lists a chunk writes to must stay in L2 until complete (measured with tile-ordered entries: 256 1.80 ms, 512 1.46 ms, 1024 1.35 ms, 2048 1.47 ms)
// A call with fewer chunks of 1024 than resident blocks takes 512, by blocks of 128 threads: 0.5 M entries in 11 views 0.55 -> 0.50 ms,
// 3 views of 2.4 k points at 1440p 0.55 -> 0.37.  Above that they lose, on crowded clouds most: 12 M entries in 64x64 pixels 0.440 ->
// 0.478 ms, 10 M in 88x88 0.284 -> 0.296.
constexpr int kWinChunkCollectFew = 512;
// Threads of a block.  Half as many per barrier suits the counting pass (40 M entries 0.405 -> 0.380 ms, crowded clouds 0.145 ->
// 0.122 ms); the collecting pass at 1024 entries per chunk wants 256 (1.25 against 1.45 ms with 128).
constexpr int kWinThreadsCount = 128, kWinThreadsCollect = 256, kWinThreadsCollectFew = 128;
// List ranges a thread reserves before it waits for any of them: all of a window's 1659 pixels by 256 threads.  One after another
// they were most of a chunk's time (barriers and waits for atomics 13 of 20 cycles per instruction); with the search of the first bin by
// 32 lanes: collect 217 -> 201 us (2 M points x 4 views), 66 -> 60 (8 channels), 1227 -> 1196 (6 M x 8), crowded cloud 430 -> 414.
constexpr int kWinReserve      = 7;
constexpr int kWinWarpsPerSM   = 64;  // grid size of the window kernels, in warps per SM
constexpr int kWinMinWarps     = 40;  // resident warps the register allocation leaves room for
constexpr int kWinMax     = 34 * 34 + 18 * 18 + 10 * 10 + 6 * 6 + 4 * 4 + 3 * 3 * 3;  // 1659 window pixels over 8 layers

// Window of a bin: on layer l it starts at ((32 bx) >> l, (32 by) >> l) and is win_w(l) pixels wide; the counters of
// the layers follow one another in shared memory.  Everything is computed from (bx32, by32) with shifts and selects:
// arrays indexed by the layer would live in local memory.
struct Window
{
    int bx32, by32;
    __device__ __forceinline__ int x0(int l) const { return bx32 >> l; }
    __device__ __forceinline__ int y0(int l) const { return by32 >> l; }
};

__device__ __forceinline__ int win_w(int l) { return (31 >> l) + 3; }

// first counter of layer l: sum of win_w(k)^2 over k < l = 0, 1156, 1480, 1580, 1616, 1632, 1641, 1650, 1659
__device__ __forceinline__ int win_off(int l)
{
    return l < 4 ? (l < 2 ? (l == 0 ? 0 : 1156) : (l == 2 ? 1480 : 1580)) : (l < 6 ? (l == 4 ? 1616 : 1632) : (l == 6 ? 1641 : (l == 7 ? 1650 : 1659)));
}

__device__ __forceinline__ Window make_window(const Geom& g, int bin)
{
    Window w;
    const int by = bin / g.bins_x, bx = bin - by * g.bins_x;
    w.bx32 = bx << kBinShift;
    w.by32 = by << kBinShift;
    return w;
}

// window counter -> global pixel index of the view, -1 if outside the layer
__device__ __forceinline__ int window_pixel(const Geom& g, const Window& w, int i)
{
    int l = 0;
#pragma unroll
    for (int k = 1; k < TRIPS_MAX_LAYERS; ++k)
        if (i >= win_off(k)) l = k;
    const int r  = i - win_off(l);
    const int ww = win_w(l);
    const int dy = r / ww, dx = r - dy * ww;
    const int x = w.x0(l) + dx, y = w.y0(l) + dy;
    return (l < g.L && x < g.W[l] && y < g.H[l]) ? g.base[l] + y * g.W[l] + x : -1;
}

// the chunk [c0, c1) of the view's entries and the first bin it touches; false when the view has no more chunks
__device__ __forceinline__ bool next_chunk(const FwdBuffers& fb, const Geom& g, int b, unsigned* ticket, uint32_t n_entry, uint32_t* s_tmp, int kWinChunk,
                                           uint32_t& c0, uint32_t& c1, int& first_bin)
{
    __syncthreads();
    if (threadIdx.x < 32)
    {
        uint32_t t = 0;
        if (threadIdx.x == 0) t = atomicAdd(ticket + b, 1u);
        t                 = __shfl_sync(kFull, t, 0);
        const uint32_t lo = (uint32_t)min((unsigned long long)t * kWinChunk, (unsigned long long)n_entry);
        // Last bin whose first entry is <= lo (empty bins share their first entry with the next non-empty one).  The lanes probe 32
        // bins at a time: three steps for the bins of a 1080p view, where a search by halves is eleven dependent loads that the
        // whole block waits for.
        const uint32_t* bf = fb.bin_cursor + (size_t)b * g.n_bins;
        int a = 0, z = lo < n_entry ? g.n_bins : 1;  // invariant: bf[a] <= lo, and bf[z] > lo or z is the end
        while (z - a > 1)
        {
            const int step   = (z - a + 31) >> 5;
            const int probe  = a + ((int)threadIdx.x + 1) * step;  // ascending with the lane
            const bool below = probe < z && bf[probe] <= lo;
            const int n      = __popc(__ballot_sync(kFull, below));
            z                = min(z, a + (n + 1) * step);
            a += n * step;
        }
        if (threadIdx.x == 0) s_tmp[0] = lo, s_tmp[1] = (uint32_t)a;
    }
    __syncthreads();
    c0        = s_tmp[0];
    first_bin = (int)s_tmp[1];
    c1        = min(n_entry, c0 + (uint32_t)kWinChunk);
    return c0 < n_entry;
}


// Calls body(e0, e1, x, y, layer, entry) for every (entry, layer) pair of the entries [lo, hi), with (x, y) the entry's
// position on that layer.  A warp takes 32 entries at a time: layer 0 directly (every entry has it), the higher layers
// through a per-warp queue of (lane, layer) items that all 32 lanes drain together, so that an entry with many layers
// does not hold up the 31 other lanes.  WITH_E1 = false: body only needs x, y, layer.
// First layer of an entry written by the strict two-layer rule: the layer below log2(size), as write_entry computed it.
__device__ __forceinline__ int strict_first_layer(float ps, int L) { return ps > 1.f ? min(tm_floor_log2(ps), L - 1) : 0; }

// first_warp: the warp of the block that takes the first 32 entries
template <int THREADS, bool WITH_E1, bool STRICT, class Body>
__device__ __forceinline__ void for_each_footprint(const float4* head, uint32_t lo, uint32_t hi, uint8_t* queue, int L, Body&& body, unsigned first_warp = 0)
{
    const int lane = threadIdx.x & 31;
    uint32_t base  = lo + ((threadIdx.x + 32 * first_warp) & (THREADS - 32));
    float4 e0n = make_float4(0.f, 0.f, 0.f, 0.f), e1n = e0n;
    if (base + lane < hi)
    {
        e0n = head[2 * (size_t)(base + lane)];      // u v ps conf
        e1n = head[2 * (size_t)(base + lane) + 1];  // pid z raw nl
    }
    for (; base < hi; base += THREADS)
    {
        const uint32_t ei = base + lane;
        const float4 e0 = e0n, e1 = e1n;
        const int nl = ei < hi ? __float_as_int(e1.w) : 0;
        if (base + THREADS + lane < hi)  // the next round's entry travels while this one is processed
        {
            e0n = head[2 * (size_t)(ei + THREADS)];
            e1n = head[2 * (size_t)(ei + THREADS) + 1];
        }
        int first = 0;
        if constexpr (STRICT)
        {
            first = strict_first_layer(e0.z, L);
            const float sc = __int_as_float((127 - first) << 23);
            if (nl > 0) body(e0, e1, e0.x * sc, e0.y * sc, first, ei);
        }
        else if (nl > 0)
            body(e0, e1, e0.x, e0.y, 0, ei);
        const int extra = max(nl - 1, 0);
        int incl = extra;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1)
        {
            const int t = __shfl_up_sync(kFull, incl, o);
            if (lane >= o) incl += t;
        }
        const int total = __shfl_sync(kFull, incl, 31);
        if (total == 0) continue;  // uniform
        int pos = incl - extra;
        for (int l = 1; l < nl; ++l) queue[pos++] = (uint8_t)(lane | ((first + l) << 5));
        __syncwarp();
        for (int i0 = 0; i0 < total; i0 += 32)
        {
            const int i        = i0 + lane;
            const unsigned it  = i < total ? queue[i] : 0u;
            const int src = it & 31, layer = it >> 5;
            float4 s0, s1 = make_float4(0.f, 0.f, 0.f, 0.f);
            s0.x = __shfl_sync(kFull, e0.x, src);
            s0.y = __shfl_sync(kFull, e0.y, src);
            s0.z = s0.w = 0.f;
            if (WITH_E1)
            {
                s0.z = __shfl_sync(kFull, e0.z, src);
                s0.w = __shfl_sync(kFull, e0.w, src);
                s1.x = __shfl_sync(kFull, e1.x, src);
                s1.y = __shfl_sync(kFull, e1.y, src);
            }
            if (i < total)
            {
                const float sc = __int_as_float((127 - layer) << 23);  // 2^-layer: the same value as `layer` halvings
                body(s0, s1, s0.x * sc, s0.y * sc, layer, base + src);
            }
        }
        __syncwarp();
    }
}


// 16-byte store that asks L2 to keep the line: a pixel's list is written 16 bytes at a time by many threads, and a
// sector that leaves L2 half written costs a read-modify-write in DRAM.
__device__ __forceinline__ void store_frag(uint4* p, const uint4& v, uint64_t policy)
{
    asm volatile("st.global.L2::cache_hint.v4.b32 [%0], {%1, %2, %3, %4}, %5;" ::"l"(p), "r"(v.x), "r"(v.y), "r"(v.z), "r"(v.w), "l"(policy) : "memory");
}
__device__ __forceinline__ uint64_t evict_last_policy()
{
    uint64_t policy = 0;
    asm volatile("createpolicy.fractional.L2::evict_last.b64 %0, 1.0;" : "=l"(policy));
    return policy;
}

// A bin with few entries inside a ticket (sky, far ground: a ticket can span hundreds of such bins) is not worth clearing
// and flushing a window of shared-memory counters with three block barriers: its footprints go straight to the pixels'
// global counters.  (On a 2560x1440 view of 20 M points with half of the bins nearly empty, the blocks that drew the
// sparse tickets ran 12 times longer than the others.)  The bins take turns in which warp of the block gets their first 32
// entries: most sparse bins have no more, and with warp 0 in charge of all of them the rest of the block idled through such
// chunks (20 M points at 1440p: count 0.29 -> 0.17 ms, collect in chunks of 1024 0.91 -> 0.55; 4 k points in 11 views 0.67 -> 0.35
// and 1.63 -> 0.50).  Not inlined: the dense path keeps its registers.
template <int THREADS, bool COLLECT, bool STRICT>
__device__ __noinline__ void sparse_bin_footprints(const Geom& g, const float4* head, uint32_t lo, uint32_t hi, uint8_t* queue,
                                                   uint32_t* pixel_ctr, uint4* frags, uint64_t keep, unsigned first_warp)
{
    for_each_footprint<THREADS, COLLECT, STRICT>(head, lo, hi, queue, g.L, [&](const float4& e0, const float4& e1, float x, float y, int layer, uint32_t ei) {
        const int px = __float2int_rd(x), py = __float2int_rd(y);
        const int Wl = g.W[layer];
        uint32_t* c  = pixel_ctr + g.base[layer] + py * Wl + px;
        if constexpr (!COLLECT)
        {
            atomicAdd(c, 1u);
            atomicAdd(c + 1, 1u);
            atomicAdd(c + Wl, 1u);
            atomicAdd(c + Wl + 1, 1u);
        }
        else
        {
            const float conf   = e0.w;
            const uint32_t pid = __float_as_uint(e1.x), zb = __float_as_uint(e1.y);
            const float lf  = layer_factor(e0.z, layer, g.L, nullptr);
            const float dx0 = fabsf(x - (float)px), dx1 = fabsf(x - (float)(px + 1));
            const float dy0 = fabsf(y - (float)py), dy1 = fabsf(y - (float)(py + 1));
            auto alpha = [&](float dx, float dy) {
                float bl = (1.f - dx) * (1.f - dy);
                if (dx > 1.f || dy > 1.f) bl = 0.f;
                float a = bl * conf;
                a *= lf;
                return __float_as_uint(a);
            };
            const uint32_t s00 = atomicAdd(c, 1u);
            const uint32_t s10 = atomicAdd(c + 1, 1u);
            const uint32_t s01 = atomicAdd(c + Wl, 1u);
            const uint32_t s11 = atomicAdd(c + Wl + 1, 1u);
            store_frag(frags + s00, make_uint4(pid, zb, alpha(dx0, dy0), ei), keep);
            store_frag(frags + s10, make_uint4(pid, zb, alpha(dx1, dy0), ei), keep);
            store_frag(frags + s01, make_uint4(pid, zb, alpha(dx0, dy1), ei), keep);
            store_frag(frags + s11, make_uint4(pid, zb, alpha(dx1, dy1), ei), keep);
        }
    }, first_warp);
}

template <int THREADS, bool COLLECT, bool STRICT>
__global__ __launch_bounds__(THREADS, kWinMinWarps * 32 / THREADS) void window_kernel(const __grid_constant__ Geom g, FwdBuffers fb, int B, int chunk)
{
    follow_previous();
    __shared__ uint32_t s_cnt[kWinMax];
    __shared__ uint32_t s_tmp[2];
    const uint64_t keep = evict_last_policy();
    __shared__ uint8_t s_queue[THREADS / 32][32 * (TRIPS_MAX_LAYERS - 1)];
    // all blocks walk the views in the same order: the lists, counters and entries in flight belong to one view (or two,
    // where blocks cross over), which keeps the partially written list sectors of a view in L2 until they are complete
    for (int b = 0; b < B; ++b)
    {
    if (COLLECT && fb.view_base[b + 1] == fb.view_base[b]) continue;  // no fragments, or the view did not fit the list buffer
    uint32_t* pixel_ctr   = (COLLECT ? fb.offsets : fb.counts) + (size_t)b * g.P;
    uint4* frags          = fb.frags + fb.view_base[COLLECT ? b : 0];
    const uint32_t n_entry = (uint32_t)(fb.entry_base[b + 1] - fb.entry_base[b]);
    if (!COLLECT && n_entry == 0) continue;  // (no ticket is taken: the pass may be taken up again)
    const float4* head     = fb.ent_head + fb.entry_base[b] * 2;
    const uint32_t* bfirst = fb.bin_cursor + (size_t)b * g.n_bins;
    uint32_t c0, c1;
    int bin;
    while (next_chunk(fb, g, b, COLLECT ? fb.ticket_collect : fb.ticket_count, n_entry, s_tmp, chunk, c0, c1, bin))
    {
        for (; bin < g.n_bins && bfirst[bin] < c1; ++bin)
        {
            const uint32_t bin_end = (bin + 1 < g.n_bins) ? bfirst[bin + 1] : n_entry;
            const uint32_t lo = max(c0, bfirst[bin]), hi = min(c1, bin_end);
            if (lo >= hi) continue;  // uniform: all threads read the same values
            if (bin_end - bfirst[bin] <= (uint32_t)kWinSparse)  // the whole bin is sparse (a short piece of a dense bin still pays off in the window)
            {
                sparse_bin_footprints<THREADS, COLLECT, STRICT>(g, head, lo, hi, s_queue[threadIdx.x >> 5], pixel_ctr, frags, keep, (unsigned)bin);
                continue;
            }
            const Window w = make_window(g, bin);
            const int n_win = win_off(g.L);
            for (int i = threadIdx.x; i < n_win; i += THREADS) s_cnt[i] = 0;
            __syncthreads();
            // ---- fragments per window pixel ----
            for_each_footprint<THREADS, false, STRICT>(head, lo, hi, s_queue[threadIdx.x >> 5], g.L,
                                      [&](const float4&, const float4&, float x, float y, int layer, uint32_t) {
                                          const int ww = win_w(layer);
                                          uint32_t* c  = s_cnt + win_off(layer) + (__float2int_rd(y) - w.y0(layer)) * ww + (__float2int_rd(x) - w.x0(layer));
                                          atomicAdd(c, 1u);
                                          atomicAdd(c + 1, 1u);
                                          atomicAdd(c + ww, 1u);
                                          atomicAdd(c + ww + 1, 1u);
                                      });
            __syncthreads();
            // ---- one global atomic per touched pixel ----
            if constexpr (COLLECT)
            {
                // several of them on their way at a time: their results are the pixels' next free slots
                for (int i0 = threadIdx.x; i0 < n_win; i0 += THREADS * kWinReserve)
                {
                    uint32_t slot[kWinReserve];
#pragma unroll
                    for (int k = 0; k < kWinReserve; ++k)
                    {
                        const int i      = i0 + k * THREADS;
                        const uint32_t c = i < n_win ? s_cnt[i] : 0u;
                        const int pix    = c ? window_pixel(g, w, i) : -1;
                        slot[k]          = pix >= 0 ? atomicAdd(pixel_ctr + pix, c) : 0u;
                    }
#pragma unroll
                    for (int k = 0; k < kWinReserve; ++k)
                        if (i0 + k * THREADS < n_win) s_cnt[i0 + k * THREADS] = slot[k];
                }
            }
            else
            {
                for (int i = threadIdx.x; i < n_win; i += THREADS)
                {
                    const uint32_t c = s_cnt[i];
                    const int pix    = c ? window_pixel(g, w, i) : -1;
                    if (pix >= 0) atomicAdd(pixel_ctr + pix, c);
                }
            }
            __syncthreads();
            if (COLLECT)
            {
                // ---- slots inside the reserved ranges; alpha and the fragment itself ----
                for_each_footprint<THREADS, true, STRICT>(head, lo, hi, s_queue[threadIdx.x >> 5], g.L,
                                         [&](const float4& e0, const float4& e1, float x, float y, int layer, uint32_t ei) {
                                             // x, y equal (u, v) * 2^-layer exactly (power-of-two scaling)
                                             const float conf   = e0.w;
                                             const uint32_t pid = __float_as_uint(e1.x), zb = __float_as_uint(e1.y);
                                             const int px = __float2int_rd(x), py = __float2int_rd(y);
                                             const int ww = win_w(layer);
                                             const int li = win_off(layer) + (py - w.y0(layer)) * ww + (px - w.x0(layer));
                                             const float lf  = layer_factor(e0.z, layer, g.L, nullptr);
                                             const float dx0 = fabsf(x - (float)px), dx1 = fabsf(x - (float)(px + 1));
                                             const float dy0 = fabsf(y - (float)py), dy1 = fabsf(y - (float)(py + 1));
                                             auto alpha = [&](float dx, float dy) {
                                                 float bl = (1.f - dx) * (1.f - dy);
                                                 if (dx > 1.f || dy > 1.f) bl = 0.f;
                                                 float a = bl * conf;
                                                 a *= lf;
                                                 return __float_as_uint(a);
                                             };
                                             // the four slots first, then the four stores: the shared-memory atomics do not wait for one another
                                             const uint32_t s00 = atomicAdd(s_cnt + li, 1u);
                                             const uint32_t s10 = atomicAdd(s_cnt + li + 1, 1u);
                                             const uint32_t s01 = atomicAdd(s_cnt + li + ww, 1u);
                                             const uint32_t s11 = atomicAdd(s_cnt + li + ww + 1, 1u);
                                             store_frag(frags + s00, make_uint4(pid, zb, alpha(dx0, dy0), ei), keep);
                                             store_frag(frags + s10, make_uint4(pid, zb, alpha(dx1, dy0), ei), keep);
                                             store_frag(frags + s01, make_uint4(pid, zb, alpha(dx0, dy1), ei), keep);
                                             store_frag(frags + s11, make_uint4(pid, zb, alpha(dx1, dy1), ei), keep);
                                         });
                __syncthreads();  // the next bin of this chunk reuses s_cnt
            }
        }
    }
    }
}

// Too few entries for kWinTicketsPerBlock tickets of kWinChunkCount per 8 resident warps?  entries_hint: the number of
// entries of the call as far as the host knows it (the previous call's, or this call's own count)
static bool few_entries(unsigned long long entries_hint, int sm_count)
{
    return entries_hint / kWinChunkCount < (unsigned long long)kWinTicketsPerBlock * sm_count * (kWinMinWarps / 8);
}

template <int THREADS, bool COLLECT>
static void run_window(const Geom& g, int B, const FwdBuffers& fb, bool strict, int chunk, unsigned long long entries_hint, int sm_count, cudaStream_t st)
{
    // No more blocks than the call has chunks: every block asks for a ticket in every view, and with twice as many blocks of half the
    // size small calls spent longer on that than before (0.7 M entries in 11 views: count 0.063 -> 0.084 ms; 0.055 like this).  The
    // hint may be an earlier call's: four blocks per SM take whatever there is.
    const unsigned long long most = (unsigned long long)sm_count * (kWinWarpsPerSM * 32 / THREADS);
    const unsigned long long want = entries_hint / chunk + B;
    const int grid                = (int)min(most, max((unsigned long long)sm_count * 4, want));
    if (strict)
        launch_following(window_kernel<THREADS, COLLECT, true>, grid, THREADS, st, g, fb, B, chunk);
    else
        launch_following(window_kernel<THREADS, COLLECT, false>, grid, THREADS, st, g, fb, B, chunk);
}

cudaError_t launch_count(const ScenePtrs& sc, const Geom& g, int B, const FwdBuffers& fb, bool strict, unsigned long long entries_hint, int sm_count,
                         cudaStream_t st)
{
    run_window<kWinThreadsCount, false>(g, B, fb, strict, few_entries(entries_hint, sm_count) ? kWinChunkCountFew : kWinChunkCount, entries_hint, sm_count, st);
    return cudaGetLastError();
}

cudaError_t launch_collect(const ScenePtrs& sc, const Geom& g, int B, const FwdBuffers& fb, bool strict, unsigned long long entries_hint, int sm_count,
                           cudaStream_t st)
{
    if (entries_hint / kWinChunkCollect < (unsigned long long)sm_count * (kWinMinWarps * 32 / kWinThreadsCollect))
        run_window<kWinThreadsCollectFew, true>(g, B, fb, strict, kWinChunkCollectFew, entries_hint, sm_count, st);
    else
        run_window<kWinThreadsCollect, true>(g, B, fb, strict, kWinChunkCollect, entries_hint, sm_count, st);
    return cudaGetLastError();
}

// ------------------------------------------------------------------------------------------------------------
// per-pixel top-K selection + front-to-back blend
//
// One warp renders an 8x4 pixel tile of one view, lane = pixel.
//   staging: (depth, alpha, entry) of up to 16 fragments of every pixel go to shared memory with asynchronous copies, 8
//     lanes on consecutive fragments of one list; loads by lane = pixel would touch 32 lines each.
//   selection: every lane sorts its own list by depth in registers, 16 fragments at a time, with a fixed comparator
//     network (Batcher's odd-even merge sort); further chunks are merged into the 16 nearest (bitonic half-cleaner +
//     merge).  A comparator serves 32 pixels at once, so a chunk costs a few hundred instructions per WARP, whatever
//     the lists look like.  Fragments of equal depth are put into point-id order afterwards.
//   blend: the sequential transmittance recurrence and the colour sum over the kept fragments.
// Replaces FastSortFusedNew (RenderForward.cu:474-1059).
//
// What bounds it (ncu, one 1080p view of 6 M points): half of the issue slots and half of the load/store unit's wavefront
// rate in use at 20 warps per SM, the rest are waits for the gathers of list heads and descriptor rows; DRAM at 27 %.
// 184 M instructions, against 323 M when the fragments of a tile were ranked against each other with shuffles (lists of at
// most 32) or sorted by half-warps, which this replaces: sort_blend stage 0.42 -> 0.31 ms on that view, 32.1 -> 22.9 ms on
// 64 views of 10 M points (longer lists), 1.41 -> 0.75 ms on 2 1440p views of 20 M, 0.206 -> 0.070 ms on a 640x480 view of
// 200 k points (lists up to 379, K = 8).
// Loops stay rolled where they can: with the blend unrolled over 16 fragments and every network instantiated twice the
// warps spent 8.6 of 20 cycles per instruction waiting for instruction fetches, and the kernel lost to its predecessor.
// ------------------------------------------------------------------------------------------------------------
typedef unsigned long long u64;
constexpr u64 kInfKey    = 0xffffffffffffffffull;
constexpr int kSbPitch   = 17;   // row pitch (entries) of the per-pixel arrays in shared memory
constexpr uint32_t kNoDepth = 0xffffffffu;  // sorts behind every depth
constexpr int kSbThreads = 128;
constexpr int kSbWarps   = kSbThreads / 32;

// Pre-selection of very long lists.  A pixel list of thousands of fragments (many points projected into a few pixels)
// would keep one warp of the blend kernel busy on its own while the rest of the machine idles.  Here a block of 256
// threads takes one such list and moves its 16 nearest fragments to the front, in depth order, by swapping them with the
// fragments that were there - the list stays the same set of fragments.  The blend kernel then reads only the first 16
// entries of every list longer than kHeavyList.  A list longer than kHeavyPart is shared by several blocks, each of which
// selects the 16 nearest of its part; the last one to finish selects from those and swaps.  Lists and parts are found by
// list_starts_kernel; with more than kHeavyCap of them nothing is done here and the blend kernel, which sees the same
// counter, walks the lists itself.
//
// What bounds it: on long lists the two walks over the keys (8 of 16 bytes used; the second comes from L2), on lists of about
// 1000 the barriers of a list.  sort_blend stage, ms, half-warps with sorted streams and one block per list / a bound from 16
// half-warps and one block per list / this: 2 M points in 2 pixels x 8 views 1.48 / 2.5 / 0.39, 700 k points in 4 pixels x 8
// views 0.26 / 0.36 / 0.18, 3 M points in 64x64 pixels x 4 views 0.90 / 0.53 / 0.54, 20 M points at 1440p x 2 views (lists up
// to 1473) 1.39 / 0.80 / 0.79.  Parts of 4096 / 8192 / 16384 fragments: within 3 % on the longest lists, 16384 leaves more of the
// chip idle on single lists, 4096 costs 10 % on the crowded 8-view calls.
constexpr int kHeavyCand   = 128;  // fragments within the bound that are ranked at a time
constexpr int kHeavyGroups = 64;   // groups of 4 threads that each bring their nearest fragment
// Keys a thread requests before it looks at any of them, and resident blocks: 4 keys and 6 blocks suit lists of about 1000,
// 8 keys and 4 blocks the very long ones (2 M points in 2 pixels x 8 views 0.39 / 0.31 ms, 700 k points, lists up to 866, x 8
// views 1.17 / 1.23 ms).
constexpr int kHeavyBatch  = 4;
constexpr int kHeavyBlocks = 6;
struct HeavyShared
{
    u64 nearest[kHeavyGroups];
    u64 key[kHeavyCand];
    uint32_t pos[kHeavyCand];
    uint32_t win[16];  // the result: indices of the 16 smallest keys, ascending
    u64 bound;
    unsigned found;
};

// The 16 smallest of n >= 16 distinct keys, by a block of 256 threads.  Every group of 4 threads brings the smallest key of
// its share; the 16th smallest of those bounds the 16th smallest of all.  What is not beyond that bound - 18 keys expected in
// random order whatever n is, at most 64 in ascending or descending order - is gathered and ranked by counting.  If it is more
// than fits (the small keys are in the shares of fewer than 16 groups), the 16th of what did fit is a closer bound and
// the gathering is repeated; from the third time on the bound is found by bisection, so that no order takes more than 66
// repetitions.  Returns the number of times the keys were gathered.
template <class KeyAt>
__device__ int nearest_16(uint32_t n, KeyAt&& key_at, HeavyShared& sh)
{
    const uint32_t t = threadIdx.x;
    u64 k[kHeavyBatch], nearest = kInfKey;
    for (uint32_t i0 = t; i0 < n; i0 += 256 * kHeavyBatch)
    {
#pragma unroll
        for (int u = 0; u < kHeavyBatch; ++u) k[u] = i0 + 256 * u < n ? key_at(i0 + 256 * u) : kInfKey;
#pragma unroll
        for (int u = 0; u < kHeavyBatch; ++u) nearest = min(nearest, k[u]);
    }
    nearest = min(nearest, __shfl_xor_sync(kFull, nearest, 1));
    nearest = min(nearest, __shfl_xor_sync(kFull, nearest, 2));
    if ((t & 3) == 0) sh.nearest[t >> 2] = nearest;
    if (t < 16) sh.win[t] = t;
    __syncthreads();
    {
        // rank of the group's key: each of its threads counts over a quarter of the others
        unsigned r = 0;
#pragma unroll 4
        for (unsigned q0 = 0; q0 < kHeavyGroups / 4; ++q0)
        {
            const unsigned q = q0 * 4 + (t & 3);
            const u64 other  = sh.nearest[q];
            r += (other < nearest || (other == nearest && q < t >> 2)) ? 1u : 0u;
        }
        r += __shfl_xor_sync(kFull, r, 1);
        r += __shfl_xor_sync(kFull, r, 2);
        if (r == 15u && (t & 3) == 0) sh.bound = nearest;
        if (t == 0) sh.found = 0;
    }
    __syncthreads();
    u64 bound = sh.bound;
    u64 low = 0, high = bound;  // fewer than 16 keys up to low, at least 16 up to high
    const bool held = n <= 256 * kHeavyBatch;  // the threads still hold all keys
    for (int walks = 1;; ++walks)
    {
        for (uint32_t i0 = t; i0 < n; i0 += 256 * kHeavyBatch)
        {
            if (!held)
            {
#pragma unroll
                for (int u = 0; u < kHeavyBatch; ++u) k[u] = i0 + 256 * u < n ? key_at(i0 + 256 * u) : kInfKey;
            }
#pragma unroll
            for (int u = 0; u < kHeavyBatch; ++u)
                if (k[u] <= bound && i0 + 256 * u < n)
                {
                    const unsigned at = atomicAdd(&sh.found, 1u);
                    if (at < (unsigned)kHeavyCand) sh.key[at] = k[u], sh.pos[at] = i0 + 256 * u;
                }
        }
        __syncthreads();
        const unsigned found = sh.found, m = min(found, (unsigned)kHeavyCand);
        if (found >= 16u && t < m)
        {
            const u64 mine = sh.key[t];
            unsigned r     = 0;
            for (unsigned q = 0; q < m; ++q) r += sh.key[q] < mine ? 1u : 0u;
            if (r < 16u) sh.win[r] = sh.pos[t];
            if (r == 15u) sh.bound = mine;
        }
        __syncthreads();
        // all of this is uniform; keys that are not distinct (there are none) end with low and high next to each other
        if ((found >= 16u && found <= (unsigned)kHeavyCand) || (found > (unsigned)kHeavyCand && high - low <= 1)) return walks;
        if (found < 16u)
            low = bound;
        else
            high = min(bound, sh.bound);
        bound = (walks <= 2 && found >= 16u) || high - low <= 1 ? high : low + (high - low) / 2;
        if (t == 0) sh.found = 0;
        __syncthreads();
    }
}

__global__ __launch_bounds__(256, kHeavyBlocks) void heavy_topk_kernel(const __grid_constant__ Geom g, FwdBuffers fb, int B)
{
    follow_previous();
    __shared__ HeavyShared sh;
    __shared__ uint32_t s_vac[16];
    __shared__ unsigned s_last;
    const unsigned n_heavy = fb.stats->n_heavy;
    if (n_heavy == 0 || n_heavy > fb.heavy.cap) return;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, j = lane & 15;
    for (unsigned h = blockIdx.x; h < n_heavy; h += gridDim.x)
    {
        const uint4 e = fb.heavy.item[h];
        const int b   = (int)e.x;
        if (e.z == 0 || b >= B || fb.view_base[b + 1] == fb.view_base[b]) continue;  // uniform: an empty item, or the view did not fit the list buffer
        const size_t bP    = (size_t)b * g.P;
        const uint32_t cnt = fb.counts[bP + e.y];
        uint4* list        = fb.frags + fb.view_base[b] + (fb.offsets[bP + e.y] - cnt);  // offsets hold list ends after the collect pass
        auto key_at = [&](uint32_t i) {
            const uint2 k = *reinterpret_cast<const uint2*>(list + i);
            return ((u64)k.y << 32) | k.x;
        };
        const uint32_t part = e.z & 0xffffu, parts = e.z >> 16;
        const uint32_t first = (uint32_t)((u64)cnt * part / parts), last = (uint32_t)((u64)cnt * (part + 1) / parts);
        if (threadIdx.x < 16) s_vac[threadIdx.x] = threadIdx.x;
        nearest_16(last - first, [&](uint32_t i) { return key_at(first + i); }, sh);
        if (parts > 1)  // uniform
        {
            uint32_t* nearest = fb.heavy.nearest + 16 * (size_t)e.w;  // of all parts of this list
            if (threadIdx.x < 16)
            {
                nearest[16 * part + threadIdx.x] = first + sh.win[threadIdx.x];
                __threadfence();
            }
            __syncthreads();
            if (threadIdx.x == 0)
            {
                s_last = atomicAdd(fb.heavy.finished + e.w, 1u) == parts - 1 ? 1u : 0u;
                __threadfence();
            }
            __syncthreads();
            if (!s_last) continue;  // uniform
            nearest_16(16 * parts, [&](uint32_t i) { return key_at(__ldcg(nearest + i)); }, sh);
            if (threadIdx.x < 16) sh.win[threadIdx.x] = __ldcg(nearest + sh.win[threadIdx.x]);
            __syncthreads();
        }
        if (warp == 0)
        {
            // lanes 0..15 hold the 16 nearest fragments in depth order (cnt > kHeavyList >= 16: all present); swap them to the front
            const bool act    = lane < 16;
            const uint32_t wp = sh.win[j];
            uint4 winner = make_uint4(0u, 0u, 0u, 0u), front = winner;
            if (act)
            {
                winner = list[wp];
                front  = list[j];
            }
            bool front_is_winner = false;
            for (int k = 0; k < 16; ++k) front_is_winner |= (__shfl_sync(kFull, wp, k) == (uint32_t)j);
            const bool displaced = act && !front_is_winner;  // a fragment that has to leave the front
            const bool vacated   = act && wp >= 16u;         // a winner's old place outside the front
            const unsigned m_d = __ballot_sync(kFull, displaced) & 0xffffu, m_v = __ballot_sync(kFull, vacated) & 0xffffu;
            if (vacated) s_vac[__popc(m_v & ((1u << j) - 1u))] = wp;
            __syncwarp();  // every lane holds its two fragments in registers before anything is stored
            if (displaced) list[s_vac[__popc(m_d & ((1u << j) - 1u))]] = front;
            if (act) list[j] = winner;
        }
        __syncthreads();
    }
}

cudaError_t launch_heavy_topk(const Geom& g, int B, const FwdBuffers& fb, int sm_count, cudaStream_t st)
{
    launch_following(heavy_topk_kernel, sm_count * kHeavyBlocks, 256, st, g, fb, B);
    return cudaGetLastError();
}

// the selection alone, for inspection: result[0..15] the positions, result[16] the number of gatherings
__global__ __launch_bounds__(256, kHeavyBlocks) void nearest_16_kernel(const u64* __restrict__ keys, uint32_t n, uint32_t* __restrict__ result)
{
    __shared__ HeavyShared sh;
    const int walks = nearest_16(n, [&](uint32_t i) { return keys[i]; }, sh);
    if (threadIdx.x < 16) result[threadIdx.x] = sh.win[threadIdx.x];
    if (threadIdx.x == 16) result[16] = (uint32_t)walks;
}

cudaError_t launch_nearest_16(const unsigned long long* d_keys, uint32_t n, uint32_t* d_result, cudaStream_t st)
{
    nearest_16_kernel<<<1, 256, 0, st>>>(d_keys, n, d_result);
    return cudaGetLastError();
}

// 4 / 8 bytes global -> shared, asynchronous; the wait covers all of the thread's copies
__device__ __forceinline__ void copy_async_4(void* dst_shared, const void* src_global)
{
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"((unsigned)__cvta_generic_to_shared(dst_shared)), "l"(src_global) : "memory");
}
__device__ __forceinline__ void copy_async_8(void* dst_shared, const void* src_global)
{
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"((unsigned)__cvta_generic_to_shared(dst_shared)), "l"(src_global) : "memory");
}
__device__ __forceinline__ void copy_async_wait() { asm volatile("cp.async.wait_all;" ::: "memory"); }

// ---- per-lane sorting in registers: depth bits as the key, position in the list as the payload ----
__device__ __forceinline__ void order_pair(uint32_t& ka, uint32_t& kb, uint32_t& ia, uint32_t& ib)
{
    const bool swap   = kb < ka;
    const uint32_t k0 = swap ? kb : ka, k1 = swap ? ka : kb;
    const uint32_t i0 = swap ? ib : ia, i1 = swap ? ia : ib;
    ka = k0, kb = k1, ia = i0, ib = i1;
}

// Batcher's odd-even merge sort of the first N of 16 elements (ascending): 19 comparators for N = 8, 63 for 16.
template <int N>
__device__ __forceinline__ void sort_network(uint32_t (&key)[16], uint32_t (&idx)[16])
{
#pragma unroll
    for (int p = 1; p < N; p *= 2)
    {
#pragma unroll
        for (int k = p; k >= 1; k /= 2)
        {
#pragma unroll
            for (int i = 0; i + k < N; ++i)
            {
                // element i is the lower partner of a comparator of distance k when it lies in the lower half of its block of
                // 2k (counted from k mod p) and both partners lie in the same block of 2p
                const int j0 = k % p;
                if (i >= j0 && ((i - j0) % (2 * k)) < k && (i / (2 * p)) == ((i + k) / (2 * p))) order_pair(key[i], key[i + k], idx[i], idx[i + k]);
            }
        }
    }
}

// resident blocks, up to 4 channels / up to 8; measured: 4 / 5 / 6 blocks 2.84 / 2.82 / 3.35 ms (6 M points, 8 views, 4
// channels, records still by pixel; 6 spills inside the networks), and 0.142 ms at 4 against 0.176 ms at 5 with 8 channels
constexpr int kSbMinBlocks = 5, kSbMinBlocksWide = 4;
template <int C>
__global__ __launch_bounds__(kSbThreads, (C <= 4 ? kSbMinBlocks : (C <= 8 ? kSbMinBlocksWide : 1))) void sort_blend_kernel(ScenePtrs sc, const __grid_constant__ Geom g, TripsRenderParams pr,
                                                                int B, FwdBuffers fb, const __grid_constant__ LayerPtrs out,
                                                                unsigned n_tiles_total)
{
    follow_previous();
    constexpr int ES = tail_stride(C);
    __shared__ uint32_t s_key[kSbWarps][32 * kSbPitch];  // depths of a chunk of 16 fragments per pixel; later the sorted list positions, [rank][lane]
    __shared__ uint2 s_az[kSbWarps][32 * kSbPitch];      // (alpha bits, entry index) of the chunk
    const int lane = threadIdx.x & 31;
    const int warp = threadIdx.x >> 5;
    const int K    = pr.k_keep;
    float bg[C];
#pragma unroll
    for (int c = 0; c < C; ++c) bg[c] = __ldg(sc.background + c);

    const bool preselected = fb.stats->n_heavy <= fb.heavy.cap;  // heavy_topk_kernel handled every long list
    unsigned next_ticket = 0;
    if (lane == 0) next_ticket = atomicAdd(fb.ticket_blend, 1u);
    if (fb.stats->given_up != kNotGivenUp) return;  // (looked at while the first ticket is on its way)
    for (;;)
    {
        // the ticket of the following tile is requested now, a whole tile ahead of its use
        const unsigned ticket = __shfl_sync(kFull, next_ticket, 0);
        if (ticket >= n_tiles_total) break;
        if (lane == 0) next_ticket = atomicAdd(fb.ticket_blend, 1u);
        const int b          = ticket / (unsigned)g.n_tiles;
        const int tile       = ticket - b * (unsigned)g.n_tiles;
        const size_t bP      = (size_t)b * g.P;
        const uint4* frags   = fb.frags + fb.view_base[b];
        const float* entries = fb.ent_tail + fb.entry_base[b] * ES;  // (position, descriptor row) of the view's entries
        const uint32_t n_entry = (uint32_t)(fb.entry_base[b + 1] - fb.entry_base[b]);
        int layer, gx, gy, p;
        tile_pixel(g, tile, lane, layer, gx, gy, p);  // lane i owns one pixel of the tile
        uint32_t cnt = 0, start = 0;
        if (p >= 0 && fb.view_base[b + 1] != fb.view_base[b])  // (a view that did not fit the list buffer renders as background)
        {
            cnt   = fb.counts[bP + p];
            start = fb.offsets[bP + p] - cnt;  // offsets hold list ends after the collect pass
            // of a pre-selected list (heavy_topk_kernel) only the front matters: its 16 nearest fragments in depth order
            if (preselected && cnt > (uint32_t)kHeavyList) cnt = 16u;
        }
        const uint32_t max_cnt = __reduce_max_sync(kFull, cnt);
        const uint4* list      = frags + start;

        if (max_cnt <= 4)
        {
            // A tile of short lists: lane = pixel reads them in place, five comparators on depth and id sort them, and the blend
            // finds alphas and entries where a staged chunk would be.  Staging, the networks and the search for ties cost such a tile
            // more than all of the rest: 7 views of 1158x940 with 0.45 fragments per pixel 0.43 -> 0.34 ms (0.30 with the fragments of
            // a tile ranked by shuffles), 11 of 835x489 with 8 channels 0.32 -> 0.28, and nothing where lists are longer.
            // (Requesting lengths and ends of the next tile's lists ahead made this case 0.49: instructions bound it, not latency.)
            uint32_t id[4], key[4], at[4];
#pragma unroll
            for (int j = 0; j < 4; ++j)
            {
                key[j] = kNoDepth, id[j] = 0u, at[j] = j;
                if (j < (int)cnt)
                {
                    const uint4 f = list[j];
                    id[j] = f.x, key[j] = f.y;
                    s_az[warp][lane * kSbPitch + j] = make_uint2(f.z, f.w);
                }
            }
            auto sort_pair = [&](int a, int b) {
                const bool swap = key[b] < key[a] || (key[b] == key[a] && id[b] < id[a]);
                const uint32_t k0 = swap ? key[b] : key[a], k1 = swap ? key[a] : key[b];
                const uint32_t d0 = swap ? id[b] : id[a], d1 = swap ? id[a] : id[b];
                const uint32_t a0 = swap ? at[b] : at[a], a1 = swap ? at[a] : at[b];
                key[a] = k0, key[b] = k1, id[a] = d0, id[b] = d1, at[a] = a0, at[b] = a1;
            };
            if (max_cnt > 1) sort_pair(0, 1), sort_pair(2, 3), sort_pair(0, 2), sort_pair(1, 3), sort_pair(1, 2);
#pragma unroll
            for (int j = 0; j < 4; ++j) s_key[warp][32 * j + lane] = at[j];
        }
        else
        {
            // ---- selection: the 16 nearest fragments of the lane's list, nearest first.  The network for 8, 12 or 16 goes by the
            //      longest list of the tile (half of the tiles of a 720p view stay at 8; 12 instead of 16: 42 against 63 comparators) ----
            uint32_t key[16], idx[16];
            uint32_t dropped = kNoDepth;  // smallest depth among the fragments that are not kept
#pragma unroll
            for (int i = 0; i < 16; ++i) key[i] = kNoDepth, idx[i] = 0u;
#pragma unroll 1
            for (uint32_t c0 = 0; c0 < max_cnt; c0 += 16)
            {
                // 8 lanes copy 8 (16) consecutive fragments of one pixel, 4 pixels per step: the lane = pixel pattern would touch
                // 32 lines with every load
                const uint32_t left = max_cnt - c0;
                const int i8        = lane & 7;
#pragma unroll 4
                for (int q = 0; q < 8; ++q)
                {
                    const int src          = q * 4 + (lane >> 3);
                    const uint32_t n_src   = __shfl_sync(kFull, cnt, src);
                    const uint32_t beg_src = __shfl_sync(kFull, start, src);
                    const uint32_t i       = c0 + i8;
                    const uint4* f         = frags + beg_src + i;
                    uint32_t* dk           = s_key[warp] + src * kSbPitch + i8;
                    uint2* da              = s_az[warp] + src * kSbPitch + i8;
                    if (i < n_src) copy_async_4(dk, &f->y), copy_async_8(da, &f->z);
                    if (left > 8 && i + 8 < n_src) copy_async_4(dk + 8, &f[8].y), copy_async_8(da + 8, &f[8].z);
                }
                copy_async_wait();
                __syncwarp();
                uint32_t k2[16], i2[16];
                uint32_t nearest = kNoDepth;
#pragma unroll
                for (int i = 0; i < 16; ++i)
                {
                    k2[i]   = (i < 8 || left > 8) && c0 + i < cnt ? s_key[warp][lane * kSbPitch + i] : kNoDepth;
                    i2[i]   = c0 + i;
                    nearest = min(nearest, k2[i]);
                }
                __syncwarp();  // the next chunk may overwrite the staged depths
                if (!__any_sync(kFull, nearest < key[15]))  // nothing nearer in any of the 32 lists
                {
                    dropped = min(dropped, nearest);
                    continue;
                }
                if (left <= 8)
                    sort_network<8>(k2, i2);
                else if (left <= 12)
                    sort_network<12>(k2, i2);
                else
                    sort_network<16>(k2, i2);
                if (c0 == 0)
                {
#pragma unroll
                    for (int i = 0; i < 16; ++i) key[i] = k2[i], idx[i] = i2[i];
                    continue;
                }
#pragma unroll
                for (int i = 0; i < 16; ++i)
                {
                    const bool take = k2[15 - i] < key[i];
                    dropped         = min(dropped, take ? key[i] : k2[15 - i]);
                    if (take) key[i] = k2[15 - i], idx[i] = i2[15 - i];
                }
#pragma unroll
                for (int st = 8; st > 0; st >>= 1)
#pragma unroll
                    for (int i = 0; i < 16; ++i)
                        if ((i & st) == 0) order_pair(key[i], key[i + st], idx[i], idx[i + st]);
            }
            uint32_t ties = 0;  // bit j: ranks j and j + 1 are equal
#pragma unroll
            for (int j = 0; j < 15; ++j) ties |= key[j] == key[j + 1] && key[j] != kNoDepth ? 1u << j : 0u;
            const bool tie_end = dropped == key[15] && dropped != kNoDepth;
            uint32_t* order    = s_key[warp] + lane;  // list position of the fragment of rank j at order[32 * j]
#pragma unroll
            for (int j = 0; j < 16; ++j)
                if (j < 8 || max_cnt > 8) order[32 * j] = idx[j];
            // Equal depths go by point id (the total order of the lists), the ids read from the lists in place.  Some percent of the
            // tiles of a scene of surfaces have such a pair, so this goes from tie to tie and looks at nothing else: functions that
            // gather all ids and sort them in registers cost 10 % there by their registers alone.  A wall that faces the camera, all of one
            // depth: 2 M points in 640x480 (lists up to 45) 0.57 -> 0.23 ms, in 4 views of 1280x960 0.95 -> 0.76 ms, against sweeps
            // over all ranks and one scan of the list per rank.
            if (__any_sync(kFull, ties || tie_end))
            {
                if (tie_end)  // a tie across the end of the selection: of the fragments at the last kept depth those with the smallest ids stay
                {
                    const int first = 15 - __clz(~(ties << 17));  // rank of the first of them; the ranks from there on are filled in order
                    ties &= (1u << first) - 1u;
                    uint2* kept = s_az[warp] + lane * kSbPitch;  // (id, list position) at kept[rank]; not in use, the list is longer than a chunk
                    int end     = first;
                    uint32_t worst = 0xffffffffu;
#pragma unroll 4
                    for (uint32_t i = 0; i < cnt; ++i)
                    {
                        const uint2 f = *reinterpret_cast<const uint2*>(list + i);
                        if (f.y != dropped || f.x >= worst) continue;
                        int k = end < 16 ? end++ : 15;
                        for (; k > first; --k)
                        {
                            const uint2 before = kept[k - 1];
                            if (before.x < f.x) break;
                            kept[k] = before;
                        }
                        kept[k] = make_uint2(f.x, i);
                        if (end == 16) worst = kept[15].x;
                    }
                    for (int k = first; k < 16; ++k) order[32 * k] = kept[k].y;
                }
                for (uint32_t left = ties; left; left &= left - 1)  // insertion of the higher rank of every pair, lowest pair first
                {
                    int k             = __ffs(left);
                    const uint32_t at = order[32 * k], id = list[at].x;
                    do
                    {
                        const uint32_t before = order[32 * (k - 1)];
                        if (list[before].x < id) break;
                        order[32 * k] = before;
                        --k;
                    } while (k > 0 && ((ties >> (k - 1)) & 1u));
                    order[32 * k] = at;
                }
                __syncwarp();
            }
        }
        const int n           = min((int)cnt, K);
        const int n_max       = min((int)max_cnt, K);
        const uint32_t* order = s_key[warp] + lane;  // list position of the fragment of rank j at order[32 * j]

        // ---- blend.  T_j = T_{j-1} * (1 - a_{j-1}), colour summed in the order of a 16-leaf butterfly
        //      (RenderForward.cu:940-994) so that results do not depend on how lanes are assigned: four leaves per turn ----
        float run = 1.f, t_last = 1.f, tn_last = 1.f;
        int m      = 0;
        bool alive = true;
        const bool one_chunk = max_cnt <= 16;  // (alpha, entry) of all fragments are staged
        float half0[C], half1[C];              // sums of leaves 0..7 and 8..15
#pragma unroll
        for (int c = 0; c < C; ++c) half0[c] = half1[c] = 0.f;
        constexpr int kRows = (C + 3) / 4;
        float4 row[4][kRows];                   // descriptor rows of this turn's fragments
        uint2 rec[4];                           // (entry index, alpha bits)
        uint2* records = fb.records + (size_t)ticket * (16 * 32);  // tickets run over the tiles of all views
#pragma unroll 1
        for (int j0 = 0; j0 < n_max; j0 += 4)
        {
#pragma unroll
            for (int u = 0; u < 4; ++u)
                if (j0 + u < n)
                {
                    const uint32_t at = order[32 * (j0 + u)];
                    const uint2 az    = one_chunk ? s_az[warp][lane * kSbPitch + at] : *reinterpret_cast<const uint2*>(&list[at].z);
                    const bool bad    = az.y >= n_entry;  // corrupted list: draws nothing, reads in bounds
                    if (bad) atomicOr(&fb.stats->status, TRIPS_DEV_BAD_FRAGMENT);
                    rec[u]          = make_uint2(bad ? 0u : az.y, bad ? 0u : az.x);
                    const float* rp = entries + (size_t)rec[u].x * ES + 4;
#pragma unroll
                    for (int r = 0; r < kRows; ++r) row[u][r] = *reinterpret_cast<const float4*>(rp + 4 * r);
                }
            float pair[C], quad[C];
#pragma unroll
            for (int u = 0; u < 4; ++u)
            {
                float leaf[C];
#pragma unroll
                for (int c = 0; c < C; ++c) leaf[c] = 0.f;
                const int j = j0 + u;
                if (j < n)
                {
                    const float a     = __uint_as_float(rec[u].y);
                    const float T_out = (j == 0 || run >= kAlphaCut) ? run : 0.f;
                    const float w     = T_out * a;
#pragma unroll
                    for (int c = 0; c < C; ++c)
                    {
                        const float4 v4 = row[u][c / 4];
                        leaf[c]         = w * ((c & 3) == 0 ? v4.x : ((c & 3) == 1 ? v4.y : ((c & 3) == 2 ? v4.z : v4.w)));
                    }
                    if (alive && T_out >= kAlphaCut)
                    {
                        m = j + 1;
                        if (pr.train) records[j * 32 + lane] = rec[u];
                    }
                    else
                        alive = false;
                    if (j == n - 1)
                    {
                        t_last  = T_out;
                        tn_last = run * (1.f - a);
                    }
                    run = run * (1.f - a);
                }
#pragma unroll
                for (int c = 0; c < C; ++c)
                {
                    if (u == 0 || u == 2)
                        pair[c] = leaf[c];
                    else if (u == 1)
                        quad[c] = pair[c] + leaf[c];
                    else
                        quad[c] = quad[c] + (pair[c] + leaf[c]);
                }
            }
#pragma unroll
            for (int c = 0; c < C; ++c)
            {
                if (j0 < 8)
                    half0[c] = j0 == 0 ? quad[c] : half0[c] + quad[c];
                else
                    half1[c] = j0 == 8 ? quad[c] : half1[c] + quad[c];
            }
        }
        if (p >= 0)
        {
            float wb;
            if (n == 0)
                wb = 1.f;  // the reference reads a neighbouring lane here (RenderForward.cu:1002-1003): defined as pure background
            else if (pr.bg_uses_Tn)
                wb = (t_last >= kAlphaCut && tn_last >= kAlphaCut) ? tn_last : 0.f;
            else
                wb = t_last;
            const int Wl = g.W[layer], Hl = g.H[layer];
            float* o = out.p[layer] + ((size_t)b * C * Hl + gy) * Wl + gx;
#pragma unroll
            for (int c = 0; c < C; ++c)
            {
                float v = half0[c] + half1[c];
                if (wb >= kAlphaCut) v += bg[c] * (wb * 1.f);
                o[(size_t)c * Hl * Wl] = v;
            }
        }
        if (pr.train) fb.rec_n[(size_t)ticket * 32 + lane] = (uint8_t)m;
        __syncwarp();
    }
}

cudaError_t launch_sort_blend(const ScenePtrs& sc, const Geom& g, const TripsRenderParams& pr, int B, const FwdBuffers& fb,
                              const LayerPtrs& out, int sm_count, cudaStream_t st)
{
    const unsigned n_tiles = (unsigned)g.n_tiles * (unsigned)B;
    int blocks             = (int)min((unsigned)(sm_count * 16), (n_tiles + kSbWarps - 1) / kSbWarps);
    blocks     = max(blocks, 1);
    switch (sc.C)
    {
        case 3: launch_following(sort_blend_kernel<3>, blocks, kSbThreads, st, sc, g, pr, B, fb, out, n_tiles); break;
        case 4: launch_following(sort_blend_kernel<4>, blocks, kSbThreads, st, sc, g, pr, B, fb, out, n_tiles); break;
        case 6: launch_following(sort_blend_kernel<6>, blocks, kSbThreads, st, sc, g, pr, B, fb, out, n_tiles); break;
        case 8: launch_following(sort_blend_kernel<8>, blocks, kSbThreads, st, sc, g, pr, B, fb, out, n_tiles); break;
        case 16: launch_following(sort_blend_kernel<16>, blocks, kSbThreads, st, sc, g, pr, B, fb, out, n_tiles); break;
        default: return cudaErrorInvalidValue;
    }
    return cudaGetLastError();
}
}  // namespace trips
