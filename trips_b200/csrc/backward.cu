// Backward rasterizer: replays the kept fragments of every pixel and scatters gradients to descriptors,
// confidences, positions, point sizes, the background colour, the camera pose and the pinhole coefficients.
//
// Replaces BlendBackwardsBilinearTiled (src/lib/rendering/RenderBackward.cu:90-618).  Differences in structure:
//   * a warp per 8x4 pixel tile; the reference's O(K^2) inner loop (RenderBackward.cu:284-301) becomes a reverse
//     running sum over the pixel's kept fragments;
//   * fragments add image-space sums to a 32-byte row of their entry (one row per visible point and view, in screen
//     order); one thread per point then gathers the rows of the point's entries (the binning pass noted which entry a
//     point has in every view), applies the chain to position / size once per entry and writes the reference's
//     layouts (point_grad_kernel); the camera sums are a pass of their own over the entries (entry_cam_grad_kernel);
//   * pixels are enumerated with the ceil-halved layer sizes of the forward pass (the reference halves with
//     floor here, RenderBackward.cu:112-130, and thereby skips rows of odd-sized layers).
#include "common.cuh"

namespace trips
{
template <int C>
__device__ __forceinline__ void atomic_add_row(float* row, const float (&v)[C])
{
    if constexpr (C % 4 == 0)
    {
#pragma unroll
        for (int c = 0; c < C; c += 4) atomicAdd(reinterpret_cast<float4*>(row + c), make_float4(v[c], v[c + 1], v[c + 2], v[c + 3]));
    }
    else if constexpr (C % 2 == 0)
    {
#pragma unroll
        for (int c = 0; c < C; c += 2) atomicAdd(reinterpret_cast<float2*>(row + c), make_float2(v[c], v[c + 1]));
    }
    else
    {
#pragma unroll
        for (int c = 0; c < C; ++c) atomicAdd(row + c, v[c]);
    }
}

__device__ __forceinline__ double warp_sum_d(double v)
{
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(kFull, v, o);
    return v;
}

constexpr int kPad        = 17;   // row pitch (entries) of the per-pixel arrays in shared memory
constexpr int kBwdThreads = 128;  // 4 warps x (32 x 17 slots x 12 bytes + fragment table + gradient tile) = 32 KB of static shared memory
constexpr int kBwdWarps   = kBwdThreads / 32;

// One warp differentiates an 8x4 pixel tile; tiles come from a few ticket counters over all views, in the order of
// tile_pixel (region-major), so the entries and gradient rows a tile touches are a short, L2-resident range.
//   staging: the tile's records go to shared memory (lane = pixel: 256 consecutive bytes per rank).
//   phase 0 (lane = kept fragment, lanes densely packed over the tile's fragments): gather the descriptor row of
//     the fragment's entry, G_j = <col_j, g> and alpha_j go to shared memory.
//   phase 1 (lane = pixel, shared memory only): the sequential recurrences over the pixel's kept fragments:
//     transmittance T_j, w_j = T_j alpha_j, and d_j = dLoss/dalpha_j = T_j G_j - (W_bg + sum_{i>j} W_i) / (1 - alpha_j + 1e-9)
//     with W_i = G_i T_i alpha_i (RenderBackward.cu:262-303; the reference's O(K^2) inner loop becomes a reverse
//     running sum).
//   phase 2 (lane = kept fragment): descriptor gradient and the image-space sums of the fragment's entry
//     (RenderBackward.cu:335-393), accumulated with two vector atomics into the per-entry gradient rows, which are
//     in screen-bin order like the entries and therefore stay hot in L2 while a region of the image is processed.
// What bounds the kernel (ncu, one 1080p view of 6 M points): 48 % of the issue slots and 66 % of the load/store
// unit's wavefront rate are in use at 26 active warps per SM; DRAM is at 20 %.  Hence the care for lines per instruction (entries ordered by
// tile, paired atomics, coalesced staging) and for instructions per fragment (fragment table, no shuffle searches).
constexpr int kBwdBlocksPerSM = 12;  // grid size of the persistent kernel, in blocks per SM
// Resident blocks: seven, and five of the variant DENSE, with 3 and 4 channels.  Seven is what 72 registers (70 with 3 channels) and 32.5 KB
// of shared memory per block allow; the bound of six below is a minimum, and six have not been measured with this body.  The L1 that is left holds next to
// nothing then (1.7 % of the sectors of that view hit; 20.7 % in an earlier build with five blocks).  Where a tile's entries are few the
// further blocks hide more latency, where they are many its rows should stay in L1 between the fragments of neighbouring pixels.
// blend_backward, seven / five blocks, us, by visible points per pixel of layer 0: 0.8 281 / 322, 1.5 (6 M points x 8 views) 2752 / 2904,
// 1.65 206 / 209, 1.84 228 / 206, 2.05 499 / 469, 2.6 1094 / 978, 2.8 290 / 257, 3.65 718 / 586 (4 channels).  DENSE is the variant for more
// than 1.75: the table of fragments is written by an unrolled loop, and its 87 registers (84 with 3 channels) leave room for five blocks.
// That is the compiler's doing (-Xptxas -v): to be looked at again when the kernel or the compiler changes.
constexpr int kBwdMinBlocks = 6, kBwdMinBlocksDense = 5;
inline bool dense_entries(unsigned long long entries, const Geom& g, int B) { return 4 * entries > 7ull * g.W[0] * g.H[0] * B; }
// SAT: saturated_alpha_accumulation as the reference's backward pass has it (RenderBackward.cu:227-259); a separate
// instantiation, so that the common case carries none of its code or registers.
template <int C, bool SAT, bool DENSE>
__global__ __launch_bounds__(kBwdThreads, (C <= 4 ? (SAT || DENSE ? kBwdMinBlocksDense : kBwdMinBlocks) : 1)) void blend_backward_kernel(ScenePtrs sc, const CamConst* cams,
                                                                     const __grid_constant__ Geom g, TripsRenderParams pr, int B,
                                                                     FwdBuffers fb, BwdBuffers bb,
                                                                     const __grid_constant__ ConstLayerPtrs grad_in)
{
    follow_previous();
    constexpr int DS = tail_stride(C);
    constexpr int GS = egrad_stride(C);
    constexpr int C4 = (C + 3) & ~3;
    __shared__ float4 s_g[kBwdWarps][C4 / 4][32];  // image gradients of the tile's pixels, four channels together
    __shared__ float s_d[kBwdWarps][32 * kPad];   // G_j, then dA_j = G_j T_j, finally d_j
    __shared__ float s_sum[SAT ? kBwdWarps : 1][SAT ? 32 * kPad : 1];  // SAT: sum of the descriptor channels of fragment j
    __shared__ uint16_t s_map[kBwdWarps][32 * 16];
    __shared__ uint2 s_rec[kBwdWarps][32 * kPad]; // the tile's records: (entry index, alpha_j bits; after phase 1: w_j = T_j * alpha_j)
    const int lane = threadIdx.x & 31;
    const int warp = threadIdx.x >> 5;
    float bg[C];
#pragma unroll
    for (int c = 0; c < C; ++c) bg[c] = __ldg(sc.background + c);

    float* my_d          = s_d[warp] + lane * kPad;
    uint2* my_rec        = s_rec[warp] + lane * kPad;

    double acc_bg[C];
#pragma unroll
    for (int c = 0; c < C; ++c) acc_bg[c] = 0.0;

    // the tickets run over the tiles of all views: the views are processed one after the other, so the entries, gradient rows and
    // records in flight belong to one view
    const unsigned n_total = (unsigned)g.n_tiles * (unsigned)B;
    TileTickets tickets;
    tickets.start(bb.ticket, n_total, blockIdx.x * kBwdWarps + warp, lane);
    for (;;)
    {
        const unsigned ticket = tickets.next(lane);
        if (ticket >= n_total) break;
        const int b          = ticket / (unsigned)g.n_tiles;
        const unsigned tile  = ticket - b * (unsigned)g.n_tiles;
        const float* desc    = fb.ent_tail + fb.entry_base[b] * DS + 4;  // descriptor row of entry e at desc + e * DS
        const float4* head   = fb.ent_head + fb.entry_base[b] * 2;
        float* egrad         = bb.egrad + fb.entry_base[b] * GS;
        const uint32_t n_ent = (uint32_t)(fb.entry_base[b + 1] - fb.entry_base[b]);
        int layer, gx, gy, p;
        tile_pixel(g, (int)tile, lane, layer, gx, gy, p);
        const int gx0 = __shfl_sync(kFull, gx, 0), gy0 = __shfl_sync(kFull, gy, 0);  // tile origin: lane l is pixel (gx0 + (l & 7), gy0 + (l >> 3))
        int m = 0;
        float gin[C4];
#pragma unroll
        for (int c = 0; c < C4; ++c) gin[c] = 0.f;
        if (p >= 0)
        {
            m            = fb.rec_n[(size_t)ticket * 32 + lane];  // tickets run over the tiles of all views
            const int Wl = g.W[layer], Hl = g.H[layer];
            const float* gi = grad_in.p[layer] + ((size_t)b * C * Hl + gy) * Wl + gx;
#pragma unroll
            for (int c = 0; c < C; ++c) gin[c] = __ldg(gi + (size_t)c * Hl * Wl);
        }
#pragma unroll
        for (int c = 0; c < C4; c += 4) s_g[warp][c / 4][lane] = make_float4(gin[c], gin[c + 1], gin[c + 2], gin[c + 3]);
        const int m_max = (int)__reduce_max_sync(kFull, (unsigned)m);
        // lanes <-> kept fragments of the tile: exclusive prefix of the record counts
        int incl = m;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1)
        {
            int t = __shfl_up_sync(kFull, incl, o);
            if (lane >= o) incl += t;
        }
        const int rel     = incl - m;
        const int n_entry = __shfl_sync(kFull, incl, 31);
        // the tile's records (entry index, alpha) -> shared memory: lane = pixel, 256 consecutive bytes per rank
        {
            const uint2* rec = fb.records + (size_t)ticket * (16 * 32) + lane;
#pragma unroll 8
            for (int j = 0; j < m_max; ++j)
                if (j < m)
                {
                    const uint2 v = rec[j * 32];
                    my_rec[j]     = make_uint2(v.x < n_ent ? v.x : 0u, v.x < n_ent ? v.y : 0u);  // a corrupted record contributes nothing
                }
        }
        __syncwarp();
        // (pixel, slot in the padded per-pixel arrays) of the e-th kept fragment of the tile: a table written by the
        // pixels' lanes replaces a binary search over warp shuffles in every round of both fragment phases
        {
            uint16_t* mp = s_map[warp] + rel;
            if constexpr (DENSE)
            {
#pragma unroll
                for (int j = 0; j < 16; ++j)
                    if (j < m) mp[j] = (uint16_t)((lane << 10) | (lane * kPad + j));
            }
            else
            {
#pragma unroll 4
                for (int j = 0; j < m_max; ++j)
                    if (j < m) mp[j] = (uint16_t)((lane << 10) | (lane * kPad + j));
            }
        }
        __syncwarp();
        auto locate = [&](int e, int& seg, int& slot) {
            const unsigned v = e < n_entry ? s_map[warp][e] : 0u;  // lanes beyond the last fragment point at slot 0
            seg  = v >> 10;
            slot = v & 1023;
        };

        // ---- phase 0 (lane = kept fragment): G_j = <descriptor row of the entry, g>; the row of the next round is
        //      requested before the current one is consumed ----
        {
            int seg_n, j_n;
            locate(lane, seg_n, j_n);
            float4 row_n[(C + 3) / 4];
            if (lane < n_entry)
            {
                const float* rp = desc + (size_t)s_rec[warp][j_n].x * DS;
#pragma unroll
                for (int c = 0; c < (C + 3) / 4; ++c) row_n[c] = *reinterpret_cast<const float4*>(rp + 4 * c);
            }
            for (int e0 = 0; e0 < n_entry; e0 += 32)
            {
                const int seg = seg_n, j = j_n;
                float4 row[(C + 3) / 4];
#pragma unroll
                for (int c = 0; c < (C + 3) / 4; ++c) row[c] = row_n[c];
                if (e0 + 32 < n_entry)
                {
                    locate(e0 + 32 + lane, seg_n, j_n);
                    if (e0 + 32 + lane < n_entry)
                    {
                        const float* rp = desc + (size_t)s_rec[warp][j_n].x * DS;
#pragma unroll
                        for (int c = 0; c < (C + 3) / 4; ++c) row_n[c] = *reinterpret_cast<const float4*>(rp + 4 * c);
                    }
                }
                if (e0 + lane < n_entry)
                {
                    float G = 0.f;
#pragma unroll
                    for (int c = 0; c < C; c += 4)
                    {
                        const float4 v4 = row[c / 4], g4 = s_g[warp][c / 4][seg];
                        G += v4.x * g4.x;
                        if (c + 1 < C) G += v4.y * g4.y;
                        if (c + 2 < C) G += v4.z * g4.z;
                        if (c + 3 < C) G += v4.w * g4.w;
                    }
                    s_d[warp][j] = G;
                    if constexpr (SAT)
                    {
                        float S = 0.f;
#pragma unroll
                        for (int c = 0; c < C; c += 4)
                        {
                            const float4 v4 = row[c / 4];
                            S += v4.x;
                            if (c + 1 < C) S += v4.y;
                            if (c + 2 < C) S += v4.z;
                            if (c + 3 < C) S += v4.w;
                        }
                        s_sum[warp][j] = S;
                    }
                }
            }
        }
        __syncwarp();

        // ---- phase 1 (lane = pixel), forward: T_j, dA_j = G_j T_j, w_j = T_j a_j.  The alphas move to registers (the
        //      reverse sweep needs them again) and w_j takes their place in shared memory. ----
        float run = 1.f;
        if constexpr (SAT)
        {
            // RenderBackward.cu:227-259 as written.  alpha_dest starts at 1 and loses every alpha; a fragment's texture
            // gradient is weighted by its alpha while alpha_dest - alpha > 0, else by what is left (the fragment that
            // fills the pixel).  d_j starts as G_j = <colour_j, g>; the filling fragment's own d is dropped and the sum
            // of its colour channels (not weighted by g) is taken from every fragment before it.  After the filling
            // fragment alpha_dest is 0 and the replay ends, so this happens at most once per pixel, possibly for the
            // background step (colour = background, alpha = 1).
            float* my_sum = s_sum[warp] + lane * kPad;
#pragma unroll
            for (int j = 0; j < 16; ++j)
            {
                if (j >= m_max) continue;  // uniform
                if (j < m && run < kAlphaCut)
                {
                    // the replay ends where alpha_dest falls below the cut-off (RenderBackward.cu:308); records behind that
                    // point exist when the forward pass blended by transmittance, which falls more slowly
                    my_rec[j].y = 0u;
                    my_d[j]     = 0.f;
                }
                else if (j < m)
                {
                    const float a    = __uint_as_float(my_rec[j].y);
                    const bool fill  = (run - a) < 0.f && run > 0.f;
                    my_rec[j].y      = __float_as_uint((run - a) > 0.f ? a : __saturatef(run));
                    if (fill)
                    {
                        const float S = my_sum[j];
                        my_d[j]       = 0.f;
                        for (int i = 0; i < j; ++i) my_d[i] -= S;
                    }
                    run = __saturatef(run - a);
                }
            }
            if (p >= 0 && run >= kAlphaCut)
            {
                // background step: alpha 1, weight saturate(alpha_dest); it fills the pixel whenever alpha_dest < 1
                float S = 0.f;
#pragma unroll
                for (int c = 0; c < C; ++c)
                {
                    acc_bg[c] += (double)(((run - 1.f) > 0.f ? 1.f : __saturatef(run)) * gin[c]);
                    S += bg[c];
                }
                if ((run - 1.f) < 0.f && run > 0.f)
                    for (int i = 0; i < m; ++i) my_d[i] -= S;
            }
        }
        else
        {
        float al[16];
#pragma unroll
        for (int j = 0; j < 16; ++j)
        {
            al[j] = 0.f;
            if (j >= m_max) continue;  // uniform
            if (j < m)
            {
                const float a = __uint_as_float(my_rec[j].y);
                al[j]         = a;
                my_d[j]       = my_d[j] * run;
                my_rec[j].y   = __float_as_uint(run * a);
                run           = (1.f - a) * run;
            }
        }
        // background step with alpha = 1 while the transmittance is above the cut-off (RenderBackward.cu:205-210,308)
        float R = 0.f;
        if (p >= 0 && run >= kAlphaCut)
        {
#pragma unroll
            for (int c = 0; c < C; ++c)
            {
                R += gin[c] * bg[c] * run * 1.f;
                acc_bg[c] += (double)(run * 1.f * gin[c]);
            }
        }
        // ---- phase 1, reverse: d_j = dA_j - R_j / (1 - a_j + eps), R_j = W_bg + sum_{i>j} W_i, W_i = dA_i a_i ----
#pragma unroll
        for (int j = 15; j >= 0; --j)
        {
            if (j < m)
            {
                const float a   = al[j];
                const float dA  = my_d[j];
                const float dem = 1.f / (1.f - a + 1e-9f);
                my_d[j]         = dA - R * dem;
                R += dA * a;
            }
        }
        }
        __syncwarp();

        // ---- phase 2 (lane = kept fragment): the header of the next round's entry is requested early ----
        {
            int seg_n, j_n;
            locate(lane, seg_n, j_n);
            float4 e0_n = make_float4(0.f, 0.f, 0.f, 0.f);
            unsigned eidx_n = 0;
            if (lane < n_entry)
            {
                eidx_n          = s_rec[warp][j_n].x;
                e0_n            = head[2 * (size_t)eidx_n];  // u v ps conf
            }
            for (int e0 = 0; e0 < n_entry; e0 += 32)
            {
                const int seg = seg_n, j = j_n;
                const float4 e0v = e0_n;  // u v ps conf
                const float conf = e0v.w;
                const unsigned eidx = eidx_n;
                const bool valid = e0 + lane < n_entry;
                if (e0 + 32 < n_entry)
                {
                    locate(e0 + 32 + lane, seg_n, j_n);
                    if (e0 + 32 + lane < n_entry)
                    {
                        eidx_n          = s_rec[warp][j_n].x;
                        e0_n            = head[2 * (size_t)eidx_n];
                    }
                }
                const int layer_s = layer;  // a tile lies on one layer
                const int gx_s = gx0 + (seg & (kTileW - 1)), gy_s = gy0 + (seg >> 3);
                // (lanes without a fragment run through with zero weights: the exchange below needs all lanes)
                const float ga = valid ? s_d[warp][j] : 0.f;
                const float w  = valid ? __uint_as_float(s_rec[warp][j].y) : 0.f;
                // bilinear weight of this pixel and its Jacobian at uv (compute_blending_fac, PointBlending.h:216-257)
                const float fac = __int_as_float((127 - layer_s) << 23);
                const float ux = e0v.x * fac, uy = e0v.y * fac;
                const float ps = e0v.z;
                const bool nx = (float)gx_s < ux, ny = (float)gy_s < uy;  // the pixel is the near one of the two columns / rows
                const float sx = ux - floorf(ux), sy = uy - floorf(uy);
                const float wx = nx ? 1.f - sx : sx, wy = ny ? 1.f - sy : sy;
                float bf       = wx * wy;
                if (pr.combine_lists && (fabsf(ux - (float)gx_s) > 1.f || fabsf(uy - (float)gy_s) > 1.f)) bf *= 0.f;  // (fragments of other layers only)
                float lf_grad   = 0.f;
                // (without use_layer_point_size the forward pass applied no layer factor: none here, and no size gradient)
                const float lf  = pr.use_layer_point_size ? layer_factor<true>(ps, layer_s, g.L, &lf_grad) : 1.f;
                const float gbs = conf * lf * ga;  // dLoss / d(bilinear weight) (RenderBackward.cu:385)
                // image-space sums of the entry: the chain to position / size / pose is linear in them and is applied
                // once per entry by point_grad_kernel
                const float4 h0 = make_float4((nx ? -wy : wy) * gbs, (ny ? -wx : wx) * gbs, bf * conf * lf_grad * ga, bf * lf * ga);
                float gt[C4];
#pragma unroll
                for (int c = 0; c < C4; c += 4)
                {
                    const float4 g4 = s_g[warp][c / 4][seg];
                    gt[c] = w * g4.x, gt[c + 1] = w * g4.y, gt[c + 2] = w * g4.z, gt[c + 3] = w * g4.w;
                }
                if constexpr (C4 == 4)
                {
                    // The row of an entry is 32 bytes: two 16-byte atomics.  Lanes work in pairs: the even lane adds the
                    // first half and the odd lane the second half of the SAME row (first the even lane's fragment, then
                    // the odd lane's), so an atomic instruction touches 16 rows instead of 32.  The load/store unit
                    // handles one 128-byte line per cycle, and that, not DRAM or the L2 atomic rate, bounds this kernel.
                    const bool odd       = lane & 1;
                    const unsigned mine  = valid ? eidx : 0xffffffffu;
                    const unsigned other = __shfl_xor_sync(kFull, mine, 1);
                    float4 x;  // even lane receives the partner's first half, odd lane the partner's second half
                    x.x = __shfl_xor_sync(kFull, odd ? h0.x : gt[0], 1);
                    x.y = __shfl_xor_sync(kFull, odd ? h0.y : gt[1], 1);
                    x.z = __shfl_xor_sync(kFull, odd ? h0.z : gt[2], 1);
                    x.w = __shfl_xor_sync(kFull, odd ? h0.w : gt[3], 1);
                    const unsigned row_a = odd ? other : mine;  // the even lane's fragment
                    const unsigned row_b = odd ? mine : other;  // the odd lane's fragment
                    const float4 own     = odd ? make_float4(gt[0], gt[1], gt[2], gt[3]) : h0;
                    if (row_a != 0xffffffffu) atomicAdd(reinterpret_cast<float4*>(egrad + (size_t)row_a * GS + (odd ? 4 : 0)), odd ? x : own);
                    if (row_b != 0xffffffffu) atomicAdd(reinterpret_cast<float4*>(egrad + (size_t)row_b * GS + (odd ? 4 : 0)), odd ? own : x);
                }
                else if (valid)
                {
                    float* eg = egrad + (size_t)eidx * GS;
                    atomicAdd(reinterpret_cast<float4*>(eg), h0);
                    atomic_add_row<C4>(eg + 4, gt);
                }
            }
        }
        __syncwarp();
    }
    // view-level gradients: warp shuffle reduction, then one double atomic per warp
#pragma unroll
    for (int c = 0; c < C; ++c)
    {
        double v = warp_sum_d(acc_bg[c]);
        if (lane == 0 && v != 0.0) atomicAdd(bb.g_bg + c, v);
    }
}

// The gradient rows of the entries the forward pass wrote start from zero.  Their number is known on the device only
// (entry_base[B]): the host does not wait for the forward pass's counts.
__global__ __launch_bounds__(256) void zero_entry_rows_kernel(float4* egrad, const unsigned long long* entry_base, int B,
                                                              int row_f4)
{
    follow_previous();
    const unsigned long long n = entry_base[B] * (unsigned long long)row_f4;
    const float4 z             = make_float4(0.f, 0.f, 0.f, 0.f);
    for (unsigned long long i = (unsigned long long)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (unsigned long long)gridDim.x * blockDim.x)
        egrad[i] = z;
}

cudaError_t launch_zero_entry_rows(int C, int B, const FwdBuffers& fb, const BwdBuffers& bb, int sm_count, cudaStream_t st)
{
    launch_following(zero_entry_rows_kernel, sm_count * 8, 256, st, reinterpret_cast<float4*>(bb.egrad), fb.entry_base, B, egrad_stride(C) / 4);
    return cudaGetLastError();
}

cudaError_t launch_blend_backward(const ScenePtrs& sc, const CamConst* cams, const Geom& g, const TripsRenderParams& pr,
                                  int B, const FwdBuffers& fb, const BwdBuffers& bb, const ConstLayerPtrs& grad_in,
                                  unsigned long long entries_hint, int sm_count, cudaStream_t st)
{
    const int grid = (int)max(1u, min((unsigned)(sm_count * kBwdBlocksPerSM), ((unsigned)g.n_tiles * (unsigned)B + kBwdWarps - 1) / kBwdWarps));
#define TRIPS_BWD_CASE(CC)                                                                                         \
    case CC:                                                                                                       \
        if (pr.saturated_alpha_accumulation)                                                                       \
            launch_following(blend_backward_kernel<CC, true, false>, grid, kBwdThreads, st, sc, cams, g, pr, B, fb, bb, grad_in);           \
        else if (CC <= 4 && dense_entries(entries_hint, g, B))                                                     \
            launch_following(blend_backward_kernel<CC, false, (CC <= 4)>, grid, kBwdThreads, st, sc, cams, g, pr, B, fb, bb, grad_in);      \
        else                                                                                                       \
            launch_following(blend_backward_kernel<CC, false, false>, grid, kBwdThreads, st, sc, cams, g, pr, B, fb, bb, grad_in);          \
        break;
    switch (sc.C)
    {
        TRIPS_BWD_CASE(3)
        TRIPS_BWD_CASE(4)
        TRIPS_BWD_CASE(6)
        TRIPS_BWD_CASE(8)
        TRIPS_BWD_CASE(16)
        default: return cudaErrorInvalidValue;
    }
#undef TRIPS_BWD_CASE
    return cudaGetLastError();
}

// ------------------------------------------------------------------------------------------------------------
// per-entry gradient rows -> per-point gradients in the reference's output layouts (PointRenderer.cu:1423-1426)
// ------------------------------------------------------------------------------------------------------------
// View-space gradient of one entry from its image-space sums (sx, sy): crop rotation, crop transform, pinhole, lens
// distortion (DIST), division by z (ProjectPointPinholeBackward, PointRendererHelper.h:434-494).
struct ViewGrad
{
    float gv0, gv1, gv2;  // gradient of the view-space position
    float gk0, gk1;       // gradient of the image-plane position before the crop transform
    float kx, ky;         // the normalised coordinates the pinhole matrix sees
    float gn0, gn1;       // gradient of the (distorted) normalised coordinates
};

template <bool DIST>
__device__ __forceinline__ ViewGrad view_gradient(const CamConst& cam, float vx, float vy, float vz, float sx, float sy, float* Jk)
{
    ViewGrad r;
    const float iz  = 1.f / vz;
    const float gr0 = cam.r00 * sx + cam.r10 * sy;
    const float gr1 = cam.r01 * sx + cam.r11 * sy;
    r.gk0           = cam.cfx * gr0;
    r.gk1           = cam.cs * gr0 + cam.cfy * gr1;
    r.gn0           = cam.fx * r.gk0;
    r.gn1           = cam.s * r.gk0 + cam.fy * r.gk1;
    r.kx = vx * iz, r.ky = vy * iz;
    float gn0 = r.gn0, gn1 = r.gn1;
    if constexpr (DIST)
    {
        float xd, yd, Jd[4];
        distort_point(cam, r.kx, r.ky, xd, yd, Jd, Jk);
        gn0  = Jd[0] * r.gn0 + Jd[2] * r.gn1;
        gn1  = Jd[1] * r.gn0 + Jd[3] * r.gn1;
        r.kx = xd, r.ky = yd;
    }
    r.gv0 = iz * gn0;
    r.gv1 = iz * gn1;
    r.gv2 = (-vx * iz * iz) * gn0 + (-vy * iz * iz) * gn1;
    return r;
}

// One thread per point: reads the point's entry index in every view, gathers the gradient rows of those entries, applies
// the chain to the position and the softplus derivative to the size, sums over the views in view order (the same result
// every time) and writes the output layouts once.  Position and raw size are those the forward pass saw (point_state, written
// by the binning pass): the rows belong to that projection, whatever has become of the caller's tensors since.
//
// Why a gather: the rows are read once each, next to 4 B of entry index per point and view and 16 B of point data.  Adding the rows to per-point accumulators entry by entry, which this replaces, read the
// entry heads as well, needed 36 B per point cleared, updated by atomics, and read again in another order, and a spatial
// sort of the points to keep those updates in L2.
// Measured, the whole gradient bookkeeping (clearing, this kernel, camera sums), per-point accumulators / gather:
// 6 M points x 8 views 1.05 / 0.73 ms, x 1 view 0.44 / 0.27 ms, 20 M x 2 views 1.54 / 0.75 ms, 2 M x 4 views 0.22 / 0.16 ms.
// Random 32-byte reads: a row costs 127 bytes of DRAM on one view of 6 M points and 92 on 8 views of 1.5 M, and the kernel
// moves 4.8-5.4 TB/s (resident blocks of 256 threads at 3 / 4 / 5: 0.77 / 0.73 / 0.93 ms on 6 M x 8, 0.99 / 0.85 / 1.04 ms on 20 M x 2;
// 5 spill).
// With a texture index the descriptor / confidence gradients of all points sharing a column are added (atomics into
// zeroed outputs); with the identity index they are plain stores.
// ACC: adds to the outputs, for the views behind the first entry_views (identity index; with a texture index the descriptor and
// confidence gradients are added anyway).
constexpr int kGradViews = 4;   // views whose rows a thread requests before it waits for any of them
constexpr int kGradCams  = 32;  // cameras held in shared memory; further ones are read from global memory (uniform addresses)
template <int C, bool DIST, bool ACC>
__global__ __launch_bounds__(256, (C <= 4 ? 4 : 1)) void point_grad_kernel(ScenePtrs sc, FwdBuffers fb, BwdBuffers bb, const CamConst* cams, int B,
                                                         TripsGrads out, const float* __restrict__ raw_texture,
                                                         const float* __restrict__ raw_confidence, float confidence_scale)
{
    follow_previous();
    constexpr int GS = egrad_stride(C);
    constexpr int C4 = (C + 3) & ~3;
    __shared__ CamConst s_cam[kGradCams];
    for (int k = threadIdx.x; k < min(B, kGradCams) * (int)(sizeof(CamConst) / 4); k += 256) ((int*)s_cam)[k] = ((const int*)cams)[k];
    __syncthreads();
    for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < (size_t)sc.N; i += (size_t)gridDim.x * blockDim.x)
    {
        const float4 p = fb.point_state[i];  // x y z raw size
        float gp0 = 0.f, gp1 = 0.f, gp2 = 0.f, gl = 0.f, gc = 0.f;
        float gt[C4];
#pragma unroll
        for (int c = 0; c < C4; ++c) gt[c] = 0.f;
        for (int vb = 0; vb < B; vb += kGradViews)
        {
            uint32_t ent[kGradViews];
            float4 s4[kGradViews], row[kGradViews][C4 / 4];
#pragma unroll
            for (int j = 0; j < kGradViews; ++j) ent[j] = vb + j < B ? fb.point_entry[(size_t)(vb + j) * sc.N + i] : kNoEntry;
#pragma unroll
            for (int j = 0; j < kGradViews; ++j)
                if (ent[j] != kNoEntry)
                {
                    const float* eg = bb.egrad + (fb.entry_base[vb + j] + ent[j]) * GS;
                    s4[j]           = *reinterpret_cast<const float4*>(eg);  // sum J0 gbs, sum J1 gbs, sum bf conf lf' ga, sum bf lf ga
#pragma unroll
                    for (int c = 0; c < C4; c += 4) row[j][c / 4] = *reinterpret_cast<const float4*>(eg + 4 + c);
                }
#pragma unroll
            for (int j = 0; j < kGradViews; ++j)
            {
                if (ent[j] == kNoEntry) continue;
                const int v         = vb + j;
                const CamConst& cam = v < kGradCams ? s_cam[v] : cams[v];
                float vx, vy, vz;
                transform_point(cam, p.x, p.y, p.z, vx, vy, vz);
                if (vz > 0.f && (s4[j].x != 0.f || s4[j].y != 0.f || s4[j].z != 0.f))
                {
                    const ViewGrad r = view_gradient<DIST>(cam, vx, vy, vz, s4[j].x, s4[j].y, nullptr);
                    gp0 += cam.R[0] * r.gv0 + cam.R[3] * r.gv1 + cam.R[6] * r.gv2;
                    gp1 += cam.R[1] * r.gv0 + cam.R[4] * r.gv1 + cam.R[7] * r.gv2;
                    gp2 += cam.R[2] * r.gv0 + cam.R[5] * r.gv1 + cam.R[8] * r.gv2;
                    gl += (cam.fx * cam.cfx / vz) * s4[j].z;
                }
                gc += s4[j].w;
#pragma unroll
                for (int c = 0; c < C4; c += 4)
                {
                    const float4 t4 = row[j][c / 4];
                    gt[c] += t4.x, gt[c + 1] += t4.y, gt[c + 2] += t4.z, gt[c + 3] += t4.w;
                }
            }
        }
        auto put = [](float* dst, float v) { *dst = ACC ? *dst + v : v; };
        if (out.points)
        {
            float4* dst = reinterpret_cast<float4*>(out.points) + i;
            if constexpr (ACC)
            {
                const float4 before = *dst;
                gp0 += before.x, gp1 += before.y, gp2 += before.z;
            }
            *dst = make_float4(gp0, gp1, gp2, 0.f);
        }
        if (out.point_size) put(out.point_size + i, gl == 0.f ? 0.f : tm_softplus_grad(p.w) * gl);
        // fused texture preparation: chain through sigmoid(scale * raw) and |raw| (raw_* are null when the caller passes
        // activated tensors)
        const int col = sc.index ? __ldg(sc.index + i) : (int)i;
        if ((unsigned)col < (unsigned)sc.n_tex)
        {
            if (raw_confidence)
            {
                const float sg = tm_sigmoid(confidence_scale * raw_confidence[col]);
                gc             = gc * (confidence_scale * (sg * (1.f - sg)));
            }
            if (raw_texture)
            {
#pragma unroll
                for (int c = 0; c < C; ++c)
                {
                    const float w = raw_texture[(size_t)c * sc.n_tex + col];
                    gt[c]         = w > 0.f ? gt[c] : (w < 0.f ? -gt[c] : 0.f);
                }
            }
        }
        if (!sc.index)
        {
            if (out.texture)
            {
#pragma unroll
                for (int c = 0; c < C; ++c) put(out.texture + (size_t)c * sc.n_tex + i, gt[c]);
            }
            if (out.confidence) put(out.confidence + i, gc);
        }
        else if ((unsigned)col < (unsigned)sc.n_tex)
        {
            if (out.texture)
            {
#pragma unroll
                for (int c = 0; c < C; ++c)
                    if (gt[c] != 0.f) atomicAdd(out.texture + (size_t)c * sc.n_tex + col, gt[c]);
            }
            if (out.confidence && gc != 0.f) atomicAdd(out.confidence + col, gc);
        }
    }
}

// Fills the point-to-entry table of a view group from the entries (view v0 + blockIdx.y); it holds kNoEntry before.
__global__ __launch_bounds__(256) void note_entries_kernel(FwdBuffers fb, int v0, int N)
{
    follow_previous();
    const int v = v0 + blockIdx.y;
    const unsigned long long first = fb.entry_base[v], n = fb.entry_base[v + 1] - first;
    uint32_t* table = fb.point_entry + (size_t)blockIdx.y * N;
    for (unsigned long long i = (unsigned long long)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (unsigned long long)gridDim.x * blockDim.x)
    {
        const unsigned pid = __float_as_uint(fb.ent_head[(first + i) * 2 + 1].x);
        if (pid < (unsigned)N) table[pid] = (uint32_t)i;
    }
}

// Pose and intrinsics gradients, summed per view in double over the entries of the view (RenderBackward.cu:453-466,587-611).
// DIST: the view-space position comes from the entry's world position (the stored projection cannot be undistorted in
// closed form) and the eight coefficients receive J_dis_dis^T (PointRendererHelper.h:468-491).
template <int C, bool DIST>
__global__ __launch_bounds__(256) void entry_cam_grad_kernel(FwdBuffers fb, BwdBuffers bb, const CamConst* cams, int B)
{
    follow_previous();
    constexpr int GS = egrad_stride(C);
    constexpr int NA = DIST ? 19 : 11;  // 6 pose + 5 pinhole (+ 8 distortion) sums per view
    __shared__ CamConst cam;
    __shared__ double s_acc[8][NA];
    const int b = blockIdx.y;
    if (threadIdx.x < sizeof(CamConst) / 4) ((int*)&cam)[threadIdx.x] = ((const int*)&cams[b])[threadIdx.x];
    __syncthreads();
    const unsigned long long first = fb.entry_base[b], n = fb.entry_base[b + 1] - first;
    const float4* head   = fb.ent_head + first * 2;
    const float* egrad   = bb.egrad + first * GS;
    double acc[NA];
#pragma unroll
    for (int k = 0; k < NA; ++k) acc[k] = 0.0;
    for (unsigned long long i = (unsigned long long)blockIdx.x * blockDim.x + threadIdx.x; i < n;
         i += (unsigned long long)gridDim.x * blockDim.x)
    {
        const float4 s4 = *reinterpret_cast<const float4*>(egrad + i * GS);
        const float4 e1 = head[2 * i + 1];  // pid z raw nl
        const float4 e0 = head[2 * i];      // u v ps conf
        // View-space position from the stored projection: (u, v) back through crop rotation, crop transform and the
        // pinhole matrix gives the normalised coordinates, the stored depth scales them.
        float vz = e1.y;
        float vx, vy;
        if constexpr (DIST)
        {
            const float4 wp = *reinterpret_cast<const float4*>(fb.ent_tail + (first + i) * tail_stride(C));  // world xyz | texture index
            transform_point(cam, wp.x, wp.y, wp.z, vx, vy, vz);
        }
        else
        {
            const float du = e0.x - cam.cenx, dv = e0.y - cam.ceny;
            const float idet = 1.f / (cam.r00 * cam.r11 - cam.r01 * cam.r10);
            const float jx = (cam.r11 * du - cam.r01 * dv) * idet + cam.cenx;
            const float jy = (cam.r00 * dv - cam.r10 * du) * idet + cam.ceny;
            const float iy = (jy - cam.ccy) / cam.cfy;
            const float ix = (jx - cam.ccx - cam.cs * iy) / cam.cfx;
            const float ny = (iy - cam.cy) / cam.fy;
            const float nx = (ix - cam.cx - cam.s * ny) / cam.fx;
            vx = nx * vz;
            vy = ny * vz;
        }
        if (vz > 0.f && (s4.x != 0.f || s4.y != 0.f || s4.z != 0.f))
        {
            float Jk[16];
            const ViewGrad r = view_gradient<DIST>(cam, vx, vy, vz, s4.x, s4.y, DIST ? Jk : nullptr);
            if constexpr (DIST)
            {
#pragma unroll
                for (int k = 0; k < 8; ++k) acc[11 + k] += (double)(Jk[k] * r.gn0 + Jk[8 + k] * r.gn1);
            }
            acc[0] += (double)r.gv0;
            acc[1] += (double)r.gv1;
            acc[2] += (double)r.gv2;
            acc[3] += (double)(vy * r.gv2 - vz * r.gv1);
            acc[4] += (double)(vz * r.gv0 - vx * r.gv2);
            acc[5] += (double)(vx * r.gv1 - vy * r.gv0);
            acc[6] += (double)(r.kx * r.gk0);
            acc[7] += (double)(r.ky * r.gk1);
            acc[8] += (double)r.gk0;
            acc[9] += (double)r.gk1;
            acc[10] += (double)(r.ky * r.gk0);
        }
    }
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
    for (int k = 0; k < NA; ++k)
    {
        const double v = warp_sum_d(acc[k]);
        if (lane == 0) s_acc[warp][k] = v;
    }
    __syncthreads();
    if (threadIdx.x < NA)
    {
        double v = 0.0;
        for (int w = 0; w < 8; ++w) v += s_acc[w][threadIdx.x];
        if (v != 0.0)
        {
            if (threadIdx.x < 6)
                atomicAdd(bb.g_pose + (size_t)b * 6 + threadIdx.x, v);
            else if (threadIdx.x < 11)
                atomicAdd(bb.g_k + (size_t)b * 5 + (threadIdx.x - 6), v);
            else
                atomicAdd(bb.g_dis + (size_t)b * 8 + (threadIdx.x - 11), v);
        }
    }
}

// One block; a thread per component (the views of a call may share an image / camera index, so every component adds its
// views in order).  One thread for everything took 12 us longer with 4 views: 76 dependent read-modify-writes.
__global__ __launch_bounds__(64) void unpack_small_kernel(int C, int B, const CamConst* cams, const double* g_bg,
                                                          const double* g_pose, const double* g_k,
                                                          const double* g_dis, float* out_bg, double* out_pose, float* out_intr)
{
    follow_previous();
    const int t = threadIdx.x;
    if (out_bg && t < C) out_bg[t] = (float)g_bg[t];
    if (out_pose && t < 6)
        for (int b = 0; b < B; ++b) out_pose[(size_t)cams[b].image_index * 6 + t] += g_pose[b * 6 + t];
    if (out_intr && t >= 32 && t < 45)
    {
        const int k = t - 32;  // 5 pinhole values, then 8 distortion coefficients (zero without distortion)
        for (int b = 0; b < B; ++b) out_intr[(size_t)cams[b].camera_index * 13 + k] += (float)(k < 5 ? g_k[b * 5 + k] : g_dis[b * 8 + k - 5]);
    }
}

int unpack_launches(int B, int entry_views) { return entry_views < B ? 2 * ((B + entry_views - 1) / entry_views) : 1; }

cudaError_t launch_unpack_grads(const ScenePtrs& sc, const CamConst* cams, int B, const FwdBuffers& fb, const BwdBuffers& bb,
                                const TripsGrads& out, const TripsRenderParams& pr, int sm_count, cudaStream_t st)
{
    if (sc.N > 0 && (out.pose_tangent || out.intrinsics))
    {
        // the entry counts live on the device: the grid covers a fixed share of the worst case and threads stride
        const dim3 grid(max(1, min(sm_count * 8 / max(1, min(B, 8)) + 1, (sc.N + 255) / 256)), B);
#define TRIPS_CAM_CASE(CC)                                                              \
    case CC:                                                                            \
        if (pr.distortion)                                                              \
            launch_following(entry_cam_grad_kernel<CC, true>, grid, 256, st, fb, bb, cams, B);     \
        else                                                                            \
            launch_following(entry_cam_grad_kernel<CC, false>, grid, 256, st, fb, bb, cams, B);    \
        break;
        switch (sc.C)
        {
            TRIPS_CAM_CASE(3)
            TRIPS_CAM_CASE(4)
            TRIPS_CAM_CASE(6)
            TRIPS_CAM_CASE(8)
            TRIPS_CAM_CASE(16)
            default: return cudaErrorInvalidValue;
        }
#undef TRIPS_CAM_CASE
    }
    if (sc.N > 0 && (out.texture || out.confidence || out.points || out.point_size))
    {
        if (sc.index || sc.n_tex != sc.N)
        {
            // columns are accumulated (or not covered by the identity mapping): start from zero
            if (out.texture)
            {
                cudaError_t e = cudaMemsetAsync(out.texture, 0, sizeof(float) * (size_t)sc.C * sc.n_tex, st);
                if (e != cudaSuccess) return e;
            }
            if (out.confidence)
            {
                cudaError_t e = cudaMemsetAsync(out.confidence, 0, sizeof(float) * (size_t)sc.n_tex, st);
                if (e != cudaSuccess) return e;
            }
        }
        const int blocks      = max(1, (int)min((size_t)sm_count * 16, ((size_t)sc.N + 255) / 256));
        const float* raw_tex  = pr.texture_abs ? sc.texture : nullptr;
        const float* raw_conf = pr.confidence_is_raw ? sc.confidence : nullptr;
        for (int v0 = 0; v0 < B; v0 += fb.entry_views)
        {
            const int nv   = min(fb.entry_views, B - v0);
            FwdBuffers fbv = fb;
            fbv.entry_base = fb.entry_base + v0;
            if (fb.entry_views < B)
            {
                cudaError_t e = cudaMemsetAsync(fb.point_entry, 0xff, sizeof(uint32_t) * (size_t)sc.N * nv, st);  // kNoEntry
                if (e != cudaSuccess) return e;
                launch_following(note_entries_kernel, dim3(max(1, sm_count * 8 / nv), nv), 256, st, fb, v0, sc.N);
            }
#define TRIPS_POINT_LAUNCH(CC, DIST, ACC) \
    launch_following(point_grad_kernel<CC, DIST, ACC>, blocks, 256, st, sc, fbv, bb, cams + v0, nv, out, raw_tex, raw_conf, pr.confidence_scale)
#define TRIPS_POINT_CASE(CC)                                                                              \
    case CC:                                                                                              \
        if (pr.distortion)                                                                                \
            v0 ? TRIPS_POINT_LAUNCH(CC, true, true) : TRIPS_POINT_LAUNCH(CC, true, false);                \
        else                                                                                              \
            v0 ? TRIPS_POINT_LAUNCH(CC, false, true) : TRIPS_POINT_LAUNCH(CC, false, false);              \
        break;
            switch (sc.C)
            {
                TRIPS_POINT_CASE(3)
                TRIPS_POINT_CASE(4)
                TRIPS_POINT_CASE(6)
                TRIPS_POINT_CASE(8)
                TRIPS_POINT_CASE(16)
                default: return cudaErrorInvalidValue;
            }
#undef TRIPS_POINT_CASE
#undef TRIPS_POINT_LAUNCH
        }
    }
    launch_following(unpack_small_kernel, 1, 64, st, sc.C, B, cams, bb.g_bg, bb.g_pose, bb.g_k, bb.g_dis, out.background, out.pose_tangent,
                                         out.intrinsics);
    return cudaGetLastError();
}
}  // namespace trips
