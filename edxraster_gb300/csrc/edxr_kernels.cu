// CUDA kernels of the EDXRaster GB300 pipeline (sm_103a).
//
// One pass renders any number of frames (a frame = one mesh seen by one
// camera); the plain path is a pass of one frame.  Stages:
//   k_clear        zero the per-tile counters and work queues;  Renderer.cpp:120-127
//                  the vertex stage of shared-vertex meshes
//   k_setup        clip = MVP * (p, 1), clip codes, fixed-point Shader.h:40-49,
//   k_clip         setup and the post-pass per input triangle;  Clipper.h:71-189,
//                  clipping of those that straddle a plane;     RasterTriangle.h:27-153
//                  the count pass of the binning
//   k_bin_*, scan  (triangle, 16x16 tile) decisions, counted,   Renderer.cpp:161-229
//                  scanned and scattered into per-tile bins
//   k_raster       persistent work items of tiles: coverage,   Renderer.cpp:248-350,
//                  depth test and winner per pixel, then the    Rasterizer.h:32-415,
//                  winner shaded: one write of colour, depth    FrameBuffer.cpp:54-68
//                  and triangle id per pixel
#include <cuda_runtime.h>

#include "edxr_device.cuh"

namespace edxr {

constexpr int kRasterThreads = 256;    // 8 warps, each on its own work items
constexpr uint32_t kBigChunk = 128;    // unsorted-list slots a k_bin_big warp reserves at a time
constexpr uint32_t kEmptySlot = 0xFFFFFFFFu;
constexpr uint32_t kDenseEntries = 640;  // entries a tile from which a frame is dense (see by_density)
constexpr uint32_t kSplitTile = 0x80000000u;  // item tag: the tile has several items (tiles < 2^24)

// Programmatic dependent launch: the pass's kernels follow one another with the
// next one's blocks already resident.  Each kernel first lets its successor be
// scheduled (which happens once all of its own blocks run) and then waits for
// its predecessor's end and memory; nothing is read or written before the
// wait.  A kernel so starts about a microsecond after its predecessor's last
// block instead of two.
__device__ __forceinline__ void follow_on()
{
    asm volatile("griddepcontrol.launch_dependents;\n\tgriddepcontrol.wait;" ::: "memory");
}

// Clip-space position of vertex v: clip = MVP * (p, 1) (DefaultVertexShader,
// Shader.h:40-49).
__device__ __forceinline__ float4 clip_position(const FrameDesc& f, uint32_t v)
{
    const float* p = reinterpret_cast<const float*>(f.positions + (size_t)v * f.pos_stride);
    return xform_point4(f.mvp, __ldg(p), __ldg(p + 1), __ldg(p + 2));
}

// Setup record of a vertex (vertex stage, for meshes whose vertices are
// shared by several triangles): inside the view volume (clip code 0) the
// projected vertex (x, y on the subpixel grid, z / w, 1 / w); otherwise
// (kVtxOutside, clip code).
constexpr int kVtxOutside = (int)0x80000000;

__device__ __forceinline__ int4 vertex_record(const FrameDesc& f, uint32_t v)
{
    const float4 c = clip_position(f, v);
    const uint32_t code = clip_code(c);
    if (code)
        return make_int4(kVtxOutside, (int)code, 0, 0);
    int vx, vy;
    float z, iw;
    project_vertex(f, c, vx, vy, z, iw);
    return make_int4(vx, vy, __float_as_int(z), __float_as_int(iw));
}

// -------------------------------------------------------------------------
// Clear of the per-tile counters and work queues, and the vertex stage.
__global__ void k_clear(PassArgs a)
{
    follow_on();
    const uint32_t stride = gridDim.x * blockDim.x;
    if (a.vrecs)
        for (uint32_t i0 = blockIdx.x * blockDim.x + (threadIdx.x & ~31u); i0 < a.total_vertices; i0 += stride)
        {
            // the frame of the warp's first vertex, then on over the frames
            // that start at or before the lane's own
            const auto base = [](const FrameDesc& f) { return f.vtx_base; };
            uint32_t fi = find_frame_warp(a.frames, a.num_frames, i0, base);
            const uint32_t i = i0 + (threadIdx.x & 31);
            if (i >= a.total_vertices)
                break;
            while (fi + 1 < a.num_frames && a.frames[fi + 1].vtx_base <= i)
                fi++;
            const FrameDesc& f = a.frames[fi];
            a.vrecs[i] = vertex_record(f, i - f.vtx_base);
        }
    // several frames: the frame of every 256th triangle, where setup's
    // frame lookup starts (instead of a search over every frame)
    if (a.frame_of_block)
        for (uint32_t b = blockIdx.x * blockDim.x + threadIdx.x; b <= (a.total_tris >> 8); b += stride)
        {
            const uint32_t fi =
                find_frame(a.frames, a.num_frames, b << 8, [](const FrameDesc& f) { return f.tri_base; });
            const FrameDesc& f = a.frames[fi];
            a.frame_of_block[b] = { fi, fi + 1 < a.num_frames ? a.frames[fi + 1].tri_base : 0xFFFFFFFFu,
                                    f.tri_base, f.vtx_base, f.indices, f.nv, 0u };
        }
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i <= a.total_tiles; i += stride)
    {
        a.tile_count[i] = 0;
        a.tile_zocc[i] = 0xFFFFFFFFu;
        a.tile_cursor[i] = 0;
    }
    if (blockIdx.x == 0)
        for (int i = (int)threadIdx.x; i < kCounters; i += (int)blockDim.x)
            a.counters[i] = 0;
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < scan_blocks(a.total_tiles); i += stride)
        a.scan_status[i] = 0ull;
    if (blockIdx.x == 0 && threadIdx.x == 0)
    {
        a.status->overflow = 0;
        a.status->error = 0;
        a.status->bins_needed = 0;
        a.status->raster_tris = 0;
        a.status->clipped_polys = 0;
        a.status->big_tris = 0;
        a.status->bin_entries = 0;
    }
}

// -------------------------------------------------------------------------
// -------------------------------------------------------------------------
// Binning.  Every non-rejected (triangle, tile) pair is counted in its tile
// and kept as (tile, raster triangle << 2 | decision) in an unsorted list;
// after the scan of the counts, k_bin_move moves the entries into their
// bins.  Triangles the reference treats as small are binned by the thread
// that sets them up (k_setup, k_clip); the others by one warp each with the
// full decision of quad_decisions (k_bin_big).
//
// bin_count_tile counts one entry of `tile`.  Neighbouring triangles of a
// warp often land in the same tile: lanes with equal tiles share one atomic,
// issued by the lowest lane.
__device__ __forceinline__ void bin_count_tile(const PassArgs& a, uint32_t tile)
{
    const uint32_t act = __activemask();
    const uint32_t peers = __match_any_sync(act, tile);
    if ((int)(threadIdx.x & 31) == __ffs(peers) - 1)
        atomicAdd(&a.tile_count[tile], (uint32_t)__popc(peers));
}

// A small triangle's entries.  The reference rasterizes a small triangle
// with FineRasterize in every tile of its range (Renderer.cpp:173-180), so
// the decision is "fine" where the quad-aligned bounding box meets the
// screen.  Tiles where no pixel centre can be covered get no entry.
struct SmallTiles
{
    int tx0, tx1, ty0, ty1;
};

// The tile range of a small triangle's entries and their number.
__device__ __forceinline__ uint32_t small_tiles(const PassArgs& a, const FrameDesc& f, const RTri& t, const BinGeom& g,
                                               SmallTiles& st)
{
    // Without wraparound only points inside the vertices' bounding box can be
    // covered: with one sample per pixel the pixels whose centre is in it,
    // with several (each inside its own pixel) the pixels the box overlaps.
    // Otherwise the reference's quad-aligned region.
    const bool wfree = wrap_free(t);
    const bool tight = a.msaa_log2 == 0 && wfree, box = a.msaa_log2 != 0 && wfree;
    const int x0 = max(tight ? g.cx0 : box ? g.bbx0 : g.bbx0 & ~1, 0);
    const int x1 = min(tight ? g.cx1 : box ? g.bbx1 : g.bbx1 | 1, f.width - 1);
    const int y0 = max(tight ? g.cy0 : box ? g.bby0 : g.bby0 & ~1, 0);
    const int y1 = min(tight ? g.cy1 : box ? g.bby1 : g.bby1 | 1, f.height - 1);
    if (x0 > x1 || y0 > y1)
        return 0;
    st.tx0 = x0 >> kTileLog2;
    st.tx1 = x1 >> kTileLog2;
    st.ty0 = y0 >> kTileLog2;
    st.ty1 = y1 >> kTileLog2;
    return (uint32_t)((st.tx1 - st.tx0 + 1) * (st.ty1 - st.ty0 + 1));
}

// Counts a small triangle's entries in their tiles and keeps them in the
// unsorted list from `slot` on, up to its stripe's end (the caller reserved
// their number; entries past the end are dropped, the frame overflows).
__device__ __forceinline__ void bin_small(const PassArgs& a, const FrameDesc& f, uint32_t ri, const SmallTiles& st,
                                          uint64_t slot, uint64_t end)
{
    for (int ty = st.ty0; ty <= st.ty1; ty++)
        for (int tx = st.tx0; tx <= st.tx1; tx++)
        {
            const uint32_t tile = f.tile_base + (uint32_t)(ty * f.tdx + tx);
            bin_count_tile(a, tile);
            if (slot < end)
                a.bin_tmp[slot] = make_uint2(tile, (ri << 2) | kDecisionFine);
            slot++;
        }
}

// Lower bound (as a depth key) of every depth the reference computes for the
// triangle at a pixel it rasterizes, or 0 (never culled) when the triangle is
// large enough for int32 edge values to wrap.  Without wraparound the
// barycentrics of rasterized pixels are within a few ulps of [0, 1], so the
// computed depth is at least min(z) minus a few ulps of the |z| sum.
__device__ __forceinline__ uint32_t zmin_key(const RTri& t, bool wf)
{
    if (!wf)
        return 0u;
    const float zmin = fminf(t.z0, fminf(t.z1, t.z2));
    const float margin = 2e-6f * (fabsf(t.z0) + fabsf(t.z1) + fabsf(t.z2)) + 1e-30f;
    const float lo = zmin - margin;
    return (lo == lo) ? depth_key(lo) : 0u;
}

// Stripe of the unsorted bin list a warp appends to, its fill counter and
// its first slot.
__device__ __forceinline__ uint32_t warp_stripe()
{
    return ((blockIdx.x * blockDim.x + threadIdx.x) >> 5) % (uint32_t)kBinStripes;
}
__device__ __forceinline__ uint32_t* stripe_counter(const PassArgs& a, uint32_t r)
{
    return a.counters + kStripeBase + r * kStripeStride;
}
__device__ __forceinline__ uint64_t stripe_begin(const PassArgs& a, uint32_t r)
{
    return (uint64_t)r * stripe_slots(a.bin_capacity);
}

// A big triangle (bounding box over more than 2x2 reference tiles) goes to
// the list k_bin_big bins warp-cooperatively, appended to with one atomic
// per warp.
__device__ __forceinline__ void bin_big_append(const PassArgs& a, uint32_t ri, bool big)
{
    const uint32_t act = __activemask();
    const uint32_t bigs = __ballot_sync(act, big);
    if (!big)
        return;
    const uint32_t lane = threadIdx.x & 31;
    const int leader = __ffs(bigs) - 1;
    uint32_t b = 0;
    if ((int)lane == leader)
        b = atomicAdd(&a.counters[2], (uint32_t)__popc(bigs));
    b = __shfl_sync(bigs, b, leader) + (uint32_t)__popc(bigs & ((1u << lane) - 1u));
    if (b < a.big_capacity)
        a.big_list[b] = ri;
}


// Appends n slots for this lane with one atomic per warp on `counter`;
// returns the lane's first slot.  Every lane of the warp must call it.
__device__ __forceinline__ uint32_t warp_append(uint32_t* counter, int n)
{
    const uint32_t lane = threadIdx.x & 31;
    int incl = n;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1)
    {
        const int v = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= (uint32_t)o) incl += v;
    }
    const int total = __shfl_sync(0xffffffffu, incl, 31);
    uint32_t base = 0;
    if (lane == 31 && total > 0)
        base = atomicAdd(counter, (uint32_t)total);
    return __shfl_sync(0xffffffffu, base, 31) + (uint32_t)(incl - n);
}

// Frame of flattened input triangle gi: from its 256-block's frame, forward
// over the frames that start at or before it (find_frame's answer: the last
// frame whose first triangle is at or before gi).
__device__ __forceinline__ uint32_t frame_of_triangle(const PassArgs& a, uint32_t gi)
{
    if (!a.frame_of_block)
        return find_frame(a.frames, a.num_frames, gi, [](const FrameDesc& f) { return f.tri_base; });
    uint32_t fi = a.frame_of_block[gi >> 8].frame;
    while (fi + 1 < a.num_frames && a.frames[fi + 1].tri_base <= gi)
        fi++;
    return fi;
}

// Setup of the triangles that need no clipping (all clip codes zero), one
// thread per input triangle; triangles that straddle a clip plane are queued
// for k_clip, triangles outside one plane are dropped (Clipper.h:103-109).
// A small set-up triangle is binned here as well.  A set-up triangle's
// record goes to its own slot (no append); the clip queue and the warp's
// stripe of the unsorted bin list take one atomic per warp each.
// Blocks of 128: warps of culled triangles leave early, and a small block's
// place is refilled sooner.  256 batched views 147 -> 142 us at 256 threads,
// 6 blocks per SM, against 128, 12 (64, 24: 149; 48 registers without the 24
// spilled bytes: 160 and 153).
constexpr int kSetupThreads = 128;

__global__ void __launch_bounds__(kSetupThreads, 12) k_setup(PassArgs a)
{
    follow_on();
    const uint32_t gi = blockIdx.x * blockDim.x + threadIdx.x;
    const uint32_t lane = threadIdx.x & 31;
    uint32_t fi = 0, tri = 0;
    int nOut = 0;
    bool straddle = false, big = false;
    uint32_t nent = 0;
    SmallTiles st;
    RTri t;
    if (gi < a.total_tris)
    {
        // several frames: what the chain to the vertices starts from comes in
        // one record of the 256 triangles' first one, unless its frame ended
        // (setup and binning of 256 views 141.6 -> 131.9 us, of 64 views 66 -> 62)
        FrameHead h;
        if (a.frame_of_block)
            h = a.frame_of_block[gi >> 8];
        if (!a.frame_of_block || gi >= h.next_tri)
        {
            fi = frame_of_triangle(a, gi);
            const FrameDesc& d = a.frames[fi];
            h = { fi, 0u, d.tri_base, d.vtx_base, d.indices, d.nv, 0u };
        }
        fi = h.frame;
        const FrameDesc& f = a.frames[fi];
        tri = gi - h.tri_base;
        const uint32_t i0 = __ldg(h.indices + 3 * (size_t)tri);
        const uint32_t i1 = __ldg(h.indices + 3 * (size_t)tri + 1);
        const uint32_t i2 = __ldg(h.indices + 3 * (size_t)tri + 2);
        if (i0 >= h.nv || i1 >= h.nv || i2 >= h.nv)
        {
            // device-resident index buffers are checked here instead of on the host
            atomicOr(&a.status->error, 1u);  // EDXR_ERR_INVALID_ARG
        }
        else
        {
            uint32_t k0, k1, k2;
            if (a.vrecs)
            {
                // projected by the vertex stage
                const int4 r0 = a.vrecs[h.vtx_base + i0], r1 = a.vrecs[h.vtx_base + i1], r2 = a.vrecs[h.vtx_base + i2];
                k0 = r0.x == kVtxOutside ? (uint32_t)r0.y : 0u;
                k1 = r1.x == kVtxOutside ? (uint32_t)r1.y : 0u;
                k2 = r2.x == kVtxOutside ? (uint32_t)r2.y : 0u;
                if ((k0 | k1 | k2) == 0)
                {
                    const int vx[3] = { r0.x, r1.x, r2.x }, vy[3] = { r0.y, r1.y, r2.y };
                    const float zp[3] = { __int_as_float(r0.z), __int_as_float(r1.z), __int_as_float(r2.z) };
                    const float iw[3] = { __int_as_float(r0.w), __int_as_float(r1.w), __int_as_float(r2.w) };
                    nOut = setup_projected(vx, vy, zp, iw, t) ? 1 : 0;
                }
            }
            else
            {
                const float4 c0 = clip_position(f, i0);
                const float4 c1 = clip_position(f, i1);
                const float4 c2 = clip_position(f, i2);
                k0 = clip_code(c0);
                k1 = clip_code(c1);
                k2 = clip_code(c2);
                if ((k0 | k1 | k2) == 0)
                    nOut = setup_triangle(f, c0, c1, c2, t) ? 1 : 0;
            }
            if (nOut)
            {
                const BinGeom g = bin_geom(t, f);
                big = !g.small;
                if (g.small)
                    nent = small_tiles(a, f, t, g, st);
            }
            straddle = (k0 | k1 | k2) != 0 && !(k0 & k1 & k2);
        }
    }
    // A warp whose triangles are all culled has nothing to append: half the
    // warps of a frame whose mesh reaches beyond the view or turns away.
    const uint32_t kept = __ballot_sync(0xffffffffu, nOut != 0), queued = __ballot_sync(0xffffffffu, straddle);
    if (!(kept | queued))
        return;
    // places of the queued triangles and of the bin entries within the warp
    // (an entry count has five bits: at most 16 tiles), one atomic per warp on
    // the clip queue (few warps have any) and on the warp's stripe of the
    // unsorted list
    const uint32_t before = (1u << lane) - 1u;
    uint32_t eexcl = 0, etotal = 0;
#pragma unroll
    for (int o = 0; o < 5; o++)
    {
        const uint32_t bit = __ballot_sync(0xffffffffu, (nent >> o) & 1u);
        eexcl += (uint32_t)__popc(bit & before) << o;
        etotal += (uint32_t)__popc(bit) << o;
    }
    const uint32_t stripe = warp_stripe();
    uint32_t qbase = 0, ebase = 0;
    if (lane == 0)
    {
        if (kept)
            atomicAdd(stripe_counter(a, stripe) + 1, (uint32_t)__popc(kept));  // statistics
        qbase = queued ? atomicAdd(&a.counters[4], (uint32_t)__popc(queued)) : 0u;
        ebase = etotal ? atomicAdd(stripe_counter(a, stripe), etotal) : 0u;
    }
    ebase = __shfl_sync(0xffffffffu, ebase, 0);
    if (queued)
    {
        qbase = __shfl_sync(0xffffffffu, qbase, 0);
        const uint32_t q = qbase + (uint32_t)__popc(queued & before);
        if (straddle && q < a.poly_capacity)
            a.clip_list[q] = gi;
    }
    // an unclipped triangle's record sits at its flattened index
    const uint64_t sbegin = stripe_begin(a, stripe);
    const uint64_t slot = sbegin + ebase + eexcl;
    if (nOut)
    {
        t.order = tri << 4;
        t.meta |= fi << 12;
        t.poly = kUnclipped;
        store_rtri(a.rtris + gi, t);
        a.rtri_zlo[gi] = zmin_key(t, wrap_free(t));
    }
    bin_big_append(a, gi, nOut && big);
    if (nOut && nent)
        bin_small(a, a.frames[fi], gi, st, slot, sbegin + stripe_slots(a.bin_capacity));
}

// Clipping of the queued triangles (Clipper.h:107-171): Sutherland-Hodgman,
// fan triangulation, setup of each fan triangle.  Each clipped triangle
// reserves n - 2 consecutive raster-triangle slots, fan piece k - 1 (fan
// vertices 0, k - 1, k) in slot first + k - 2; a piece that setup culls
// leaves its slot unused.  Its polygon record is the one of its queue
// position.  Two ways to spread the work over the lanes, chosen by the
// queue length (the kernel is latency-bound either way):
//  - short queues (one round of the grid's 16-lane groups): a group clips
//    one triangle with one polygon vertex per lane (a polygon has at most
//    kMaxPolygon = 16 vertices), so the polygon stays in registers: per
//    plane each lane classifies its edge (its vertex and the next), emits 0,
//    1 or 2 vertices, and a scan over the group places them in the order of
//    the serial loop (Clipper::ClipPolygon, Clipper.h:235-288);
//  - long queues: the first `per` lanes of a warp (per <= kClipPer) clip one
//    triangle each with the serial loop, and the warp's fan pieces are then
//    set up one per lane.
constexpr int kClipThreads = 128;
constexpr int kClipWarps = kClipThreads / 32;
constexpr int kClipLanes = 16;
constexpr int kClipPer = 8;
static_assert(kClipLanes == kMaxPolygon, "one lane per polygon vertex");

// Bit of plane k in the order L, R, B, T, F, N.
__device__ __forceinline__ uint32_t plane_bit(int k)
{
    return k < 4 ? 1u << k : (k == 4 ? (uint32_t)kFar : (uint32_t)kNear);
}

// Clipper::ClipPolygon (Clipper.h:235-288), one lane: Sutherland-Hodgman
// against the planes in planeCode, in the order L, R, B, T, F, N, then the
// polygon is dropped when any vertex has w <= 0.  The polygon starts in buf0
// and alternates between buf0 and buf1; returns the vertex count and sets
// res to the buffer that holds the result.
__device__ __forceinline__ int clip_polygon(PolyVert* buf0, PolyVert* buf1, uint32_t planeCode, PolyVert*& res)
{
    PolyVert* src = buf0;
    PolyVert* dst = buf1;
    int n = 3;
#pragma unroll 1
    for (int k = 0; k < 6; k++)
    {
        if (!(planeCode & plane_bit(k)))
            continue;
        int m = 0;
        // edges (i, i + 1) from i = 0, the first vertex carried in registers
        PolyVert v0 = src[0];
        bool in0 = plane_inside(k, v0.p);
        for (int i = 0; i < n; i++)
        {
            const PolyVert v1 = src[(i + 1 == n) ? 0 : i + 1];
            const bool in1 = plane_inside(k, v1.p);
            if (in0)
            {
                if (m < kMaxPolygon) dst[m++] = in1 ? v1 : plane_cut(k, v0, v1);
            }
            else if (in1)
            {
                if (m < kMaxPolygon) dst[m++] = plane_cut(k, v0, v1);
                if (m < kMaxPolygon) dst[m++] = v1;
            }
            v0 = v1;
            in0 = in1;
        }
        PolyVert* t = src;
        src = dst;
        dst = t;
        n = m;
    }
    res = src;
    for (int i = 0; i < n; i++)
        if (src[i].p.w <= 0.0f)
            return 0;
    return n;
}

// Clipper.h:121-152: a polygon vertex whose weight is exactly one on a source
// vertex is that source vertex (position and attributes); the others are
// new.  Returns the source index, or -1, and makes the weights exact.
__device__ __forceinline__ int source_vertex(PolyVert& v)
{
    int sv = -1;
    if (v.w0 == 1.0f) sv = 0;
    else if (v.w1 == 1.0f) sv = 1;
    else if (v.w2 == 1.0f) sv = 2;
    if (sv >= 0)
    {
        v.w0 = (sv == 0) ? 1.f : 0.f;
        v.w1 = (sv == 1) ? 1.f : 0.f;
        v.w2 = (sv == 2) ? 1.f : 0.f;
    }
    return sv;
}

// Slots of a warp's fan pieces and the capacity checks: `pieces` is this
// lane's count (0 for lanes that hold no triangle); returns its first slot
// and clears `pieces` when a capacity is exceeded.
__device__ __forceinline__ uint32_t reserve_pieces(const PassArgs& a, int& pieces, uint32_t q)
{
    const uint32_t first = a.total_tris + warp_append(&a.counters[0], pieces);
    if (pieces && (uint64_t)first + (uint32_t)pieces > a.rtri_capacity)
    {
        atomicOr(&a.status->overflow, 2u);
        pieces = 0;
    }
    if (pieces && q >= a.poly_capacity)
    {
        atomicOr(&a.status->overflow, 4u);
        pieces = 0;
    }
    return first;
}

// Setup and binning of one fan piece (c0, c1, c2 in clip space): piece `fan`
// of input triangle `tri` of frame fi, clipped polygon `poly`, slot ri.
// Every lane of the warp calls it; lanes with has == false hold no piece.
__device__ __forceinline__ void clip_piece(const PassArgs& a, bool has, uint32_t fi, uint32_t tri, uint32_t poly,
                                           uint32_t fan, uint32_t ri, float4 c0, float4 c1, float4 c2)
{
    const FrameDesc& f = a.frames[fi];
    bool big = false, kept = false;
    uint32_t nent = 0;
    SmallTiles st;
    RTri tk;
    if (has && setup_triangle(f, c0, c1, c2, tk))
    {
        tk.order = (tri << 4) | fan;
        tk.meta |= fi << 12;
        tk.poly = (poly << 4) | (fan + 1u);
        kept = true;
        store_rtri(a.rtris + ri, tk);
        a.rtri_zlo[ri] = zmin_key(tk, wrap_free(tk));
        const BinGeom bg = bin_geom(tk, f);
        big = !bg.small;
        if (bg.small)
            nent = small_tiles(a, f, tk, bg, st);
    }
    const uint32_t kept_lanes = __ballot_sync(0xffffffffu, kept);
    if ((threadIdx.x & 31) == 0 && kept_lanes)
        atomicAdd(&a.counters[11], (uint32_t)__popc(kept_lanes));
    bin_big_append(a, ri, big);
    const uint32_t stripe = warp_stripe();
    const uint64_t sbegin = stripe_begin(a, stripe);
    const uint64_t slot = sbegin + warp_append(stripe_counter(a, stripe), (int)nent);
    if (nent)
        bin_small(a, f, ri, st, slot, sbegin + stripe_slots(a.bin_capacity));
}

// Vertex of lane `src` (within the 16-lane group) of every lane's group.
__device__ __forceinline__ PolyVert shfl_vert(const PolyVert& v, int src)
{
    PolyVert r;
    r.p.x = __shfl_sync(0xffffffffu, v.p.x, src, kClipLanes);
    r.p.y = __shfl_sync(0xffffffffu, v.p.y, src, kClipLanes);
    r.p.z = __shfl_sync(0xffffffffu, v.p.z, src, kClipLanes);
    r.p.w = __shfl_sync(0xffffffffu, v.p.w, src, kClipLanes);
    r.w0 = __shfl_sync(0xffffffffu, v.w0, src, kClipLanes);
    r.w1 = __shfl_sync(0xffffffffu, v.w1, src, kClipLanes);
    r.w2 = __shfl_sync(0xffffffffu, v.w2, src, kClipLanes);
    return r;
}
__device__ __forceinline__ float4 shfl_f4(float4 v, int src)
{
    return make_float4(__shfl_sync(0xffffffffu, v.x, src, kClipLanes), __shfl_sync(0xffffffffu, v.y, src, kClipLanes),
                       __shfl_sync(0xffffffffu, v.z, src, kClipLanes), __shfl_sync(0xffffffffu, v.w, src, kClipLanes));
}

// Short queues: one 16-lane group per triangle, q < nq <= the grid's groups.
__device__ __forceinline__ void clip_groups(const PassArgs& a, uint32_t nq)
{
    const uint32_t lane = threadIdx.x & 31;
    const int g = (int)(lane & 15u);  // vertex lane within the group
    const uint32_t gmask = 0xFFFFu << (lane & 16u);
    const uint32_t q = (blockIdx.x * kClipThreads + threadIdx.x) / kClipLanes;
    uint32_t gi = 0, fi = 0, tri = 0, code = 0;
    PolyVert v = { make_float4(0.f, 0.f, 0.f, 0.f), 0.f, 0.f, 0.f };
    int n = 0;
    if (q < nq)
    {
        gi = a.clip_list[q];
        fi = frame_of_triangle(a, gi);
        const FrameDesc& f = a.frames[fi];
        tri = gi - f.tri_base;
        n = 3;
        if (g < 3)
        {
            v.p = clip_position(f, __ldg(f.indices + 3 * (size_t)tri + g));
            v.w0 = g == 0 ? 1.f : 0.f;
            v.w1 = g == 1 ? 1.f : 0.f;
            v.w2 = g == 2 ? 1.f : 0.f;
            code = clip_code(v.p);
        }
    }
    const float4 src = v.p;  // source vertex g (g < 3)
    const uint32_t k0 = __shfl_sync(0xffffffffu, code, 0, kClipLanes);
    const uint32_t k1 = __shfl_sync(0xffffffffu, code, 1, kClipLanes);
    const uint32_t k2 = __shfl_sync(0xffffffffu, code, 2, kClipLanes);
    const uint32_t planes = (k0 ^ k1) | (k1 ^ k2) | (k2 ^ k0);
    const uint32_t any = __reduce_or_sync(0xffffffffu, planes);
#pragma unroll 1
    for (int k = 0; k < 6; k++)
    {
        const uint32_t bit = plane_bit(k);
        if (!(any & bit))
            continue;
        // edge (g, g + 1 mod n): its end vertex, the cut, the emissions
        const PolyVert v1 = shfl_vert(v, (g + 1 >= n) ? 0 : g + 1);
        const bool valid = g < n;
        const bool in0 = valid && plane_inside(k, v.p);
        const bool in1 = valid && plane_inside(k, v1.p);
        const int c = !valid ? 0 : (in0 ? 1 : (in1 ? 2 : 0));
        PolyVert e0 = v1;
        if (valid && in0 != in1)
            e0 = plane_cut(k, v, v1);
        int incl = c;
#pragma unroll
        for (int o = 1; o < kClipLanes; o <<= 1)
        {
            const int t = __shfl_up_sync(0xffffffffu, incl, o, kClipLanes);
            if (g >= o) incl += t;
        }
        const int m = min(__shfl_sync(0xffffffffu, incl, kClipLanes - 1, kClipLanes), kMaxPolygon);
        // output vertex g: emission g - excl(s) of the first lane s whose
        // inclusive count exceeds g
        int s = 0;
#pragma unroll
        for (int st = kClipLanes / 2; st >= 1; st >>= 1)
        {
            const int t = __shfl_sync(0xffffffffu, incl, s + st - 1, kClipLanes);
            if (t <= g) s += st;
        }
        const int which = g - __shfl_sync(0xffffffffu, incl - c, s, kClipLanes);
        const PolyVert first = shfl_vert(e0, s);
        const PolyVert second = shfl_vert(v1, s);
        if (planes & bit)
        {
            if (g < m)
                v = which == 0 ? first : second;
            n = m;
        }
    }
    // the polygon is dropped when any vertex has w <= 0
    if (__ballot_sync(0xffffffffu, g < n && v.p.w <= 0.0f) & gmask)
        n = 0;
    const int sv = source_vertex(v);
    const float4 sp = shfl_f4(src, sv < 0 ? 0 : sv);
    if (sv >= 0)
        v.p = sp;
    int pieces = (g == 0 && n >= 3) ? n - 2 : 0;
    const uint32_t first = __shfl_sync(0xffffffffu, reserve_pieces(a, pieces, q), 0, kClipLanes);
    pieces = __shfl_sync(0xffffffffu, pieces, 0, kClipLanes);
    if (pieces)
    {
        ClipPoly& P = a.polys[q];
        if (g < n)
        {
            P.w[g][0] = v.w0;
            P.w[g][1] = v.w1;
            P.w[g][2] = v.w2;
        }
        if (g == 0)
        {
            P.n = (uint32_t)n;
            a.tri_first[gi] = first;
        }
    }
    // lane g: piece g + 1, fan vertices 0, g + 1, g + 2
    const float4 f0 = shfl_f4(v.p, 0);
    const float4 f1 = shfl_f4(v.p, min(g + 1, kClipLanes - 1));
    const float4 f2 = shfl_f4(v.p, min(g + 2, kClipLanes - 1));
    clip_piece(a, g < pieces, fi, tri, q, (uint32_t)g + 1u, first + (uint32_t)g, f0, f1, f2);
}

// Long queues: `per` triangles per warp and round, clipped by one lane each.
__device__ __forceinline__ void clip_lanes(const PassArgs& a, uint32_t nq, float4 (*s_vc)[kMaxPolygon])
{
    const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const uint32_t nwarps = gridDim.x * kClipWarps;
    uint32_t per = 1;
    while (per < (uint32_t)kClipPer && (uint64_t)per * nwarps < nq)
        per <<= 1;
    const uint64_t span = (uint64_t)per * nwarps;
    const uint32_t rounds = (uint32_t)((nq + span - 1) / span);
    for (uint32_t r = 0; r < rounds; r++)
    {
        const uint64_t q64 = ((uint64_t)r * nwarps + blockIdx.x * kClipWarps + warp) * per + lane;
        const uint32_t q = (uint32_t)min(q64, (uint64_t)0xFFFFFFFFu);
        PolyVert buf0[kMaxPolygon], buf1[kMaxPolygon];
        PolyVert* poly = buf0;
        int n = 0;
        uint32_t gi = 0, fi = 0, tri = 0;
        if (lane < per && q64 < nq)
        {
            gi = a.clip_list[q];
            fi = frame_of_triangle(a, gi);
            const FrameDesc& f = a.frames[fi];
            tri = gi - f.tri_base;
            const float4 c0 = clip_position(f, __ldg(f.indices + 3 * (size_t)tri));
            const float4 c1 = clip_position(f, __ldg(f.indices + 3 * (size_t)tri + 1));
            const float4 c2 = clip_position(f, __ldg(f.indices + 3 * (size_t)tri + 2));
            const uint32_t k0 = clip_code(c0), k1 = clip_code(c1), k2 = clip_code(c2);
            buf0[0] = { c0, 1.f, 0.f, 0.f };
            buf0[1] = { c1, 0.f, 1.f, 0.f };
            buf0[2] = { c2, 0.f, 0.f, 1.f };
            n = clip_polygon(buf0, buf1, (k0 ^ k1) | (k1 ^ k2) | (k2 ^ k0), poly);
            const float4 src[3] = { c0, c1, c2 };
            for (int j = 0; j < n; j++)
            {
                const int sv = source_vertex(poly[j]);
                s_vc[lane][j] = sv >= 0 ? src[sv] : poly[j].p;
            }
        }
        int pieces = n >= 3 ? n - 2 : 0;
        const uint32_t first = reserve_pieces(a, pieces, q);
        if (pieces)
        {
            ClipPoly& P = a.polys[q];
            for (int j = 0; j < n; j++)
            {
                P.w[j][0] = poly[j].w0;
                P.w[j][1] = poly[j].w1;
                P.w[j][2] = poly[j].w2;
            }
            P.n = (uint32_t)n;
            a.tri_first[gi] = first;
        }
        // the warp's pieces, numbered across its lanes and taken 32 at a time
        int incl = pieces;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1)
        {
            const int v = __shfl_up_sync(0xffffffffu, incl, o);
            if (lane >= (uint32_t)o) incl += v;
        }
        const int total = __shfl_sync(0xffffffffu, incl, 31);
        __syncwarp();
        for (int base = 0; base < total; base += 32)
        {
            const int p = base + (int)lane;
            // owner: the first lane whose inclusive count exceeds p
            int j = 0;
#pragma unroll
            for (int st = 16; st >= 1; st >>= 1)
            {
                const int v = __shfl_sync(0xffffffffu, incl, j + st - 1);
                if (v <= p) j += st;
            }
            const int k = p - __shfl_sync(0xffffffffu, incl - pieces, j) + 2;
            const uint32_t jfirst = __shfl_sync(0xffffffffu, first, j);
            const uint32_t jfi = __shfl_sync(0xffffffffu, fi, j);
            const uint32_t jtri = __shfl_sync(0xffffffffu, tri, j);
            const uint32_t jq = __shfl_sync(0xffffffffu, q, j);
            const bool has = p < total;
            const float4* vj = s_vc[j & (kClipPer - 1)];
            float4 c0 = make_float4(0.f, 0.f, 0.f, 1.f), c1 = c0, c2 = c0;
            if (has)
            {
                c0 = vj[0];
                c1 = vj[k - 1];
                c2 = vj[k];
            }
            clip_piece(a, has, jfi, jtri, jq, (uint32_t)(k - 1), jfirst + (uint32_t)(k - 2), c0, c1, c2);
        }
        __syncwarp();
    }
}

__global__ void __launch_bounds__(kClipThreads) k_clip(PassArgs a)
{
    follow_on();
    __shared__ float4 s_vc[kClipWarps][kClipPer][kMaxPolygon];
    const uint32_t nq = min(*(volatile uint32_t*)&a.counters[4], a.poly_capacity);
    if (nq <= gridDim.x * (uint32_t)(kClipThreads / kClipLanes))
        clip_groups(a, nq);
    else
        clip_lanes(a, nq, s_vc[threadIdx.x >> 5]);
}

// Scatter of the unsorted entries into their bins (after the scan); empty
// slots and entries hidden behind their tile's occluder are skipped, so a
// bin holds its tile's first tile_cursor entries.
__global__ void __launch_bounds__(256) k_bin_move(PassArgs a)
{
    follow_on();
    // the filled parts of the stripes (slots past a stripe's end were
    // dropped: overflow), numbered one after another
    __shared__ uint32_t s_first[kBinStripes + 1];
    // a pass that reported an error (a scan wait that ran out, a bad index)
    // fails as a whole: its offsets may be wrong, so nothing is scattered
    if (*(volatile uint32_t*)&a.status->error)
        return;
    const uint64_t R = stripe_slots(a.bin_capacity);
    const uint32_t lane = threadIdx.x & 31;
    if (threadIdx.x < 32)
    {
        static_assert(kBinStripes == 32, "one lane per stripe");
        const uint32_t m = (uint32_t)min((uint64_t)*(volatile uint32_t*)stripe_counter(a, lane), R);
        uint32_t incl = m;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1)
        {
            const uint32_t v = __shfl_up_sync(0xffffffffu, incl, o);
            if (lane >= (uint32_t)o) incl += v;
        }
        s_first[lane] = incl - m;
        if (lane == 31)
            s_first[32] = incl;
    }
    __syncthreads();
    const uint32_t total = s_first[kBinStripes];
    const uint32_t stride = gridDim.x * blockDim.x;
    const uint32_t rounds = (total + stride - 1) / stride;
    for (uint32_t rd = 0; rd < rounds; rd++)
    {
        const uint32_t j = rd * stride + blockIdx.x * blockDim.x + threadIdx.x;
        uint2 e = make_uint2(kEmptySlot, 0u);
        uint32_t bin = 0;  // the bin's start, loaded beside the occluder bound
        if (j < total)
        {
            // stripe of entry j: the last one starting at or before it
            uint32_t r = 0;
#pragma unroll
            for (uint32_t st = 16; st >= 1; st >>= 1)
                if (s_first[r + st] <= j) r += st;
            e = a.bin_tmp[(uint64_t)r * R + (j - s_first[r])];
            // an entry wholly behind its tile's occluder is dropped: the
            // raster's depth bound would skip it at staging (its nearest
            // depth beyond min(occluder bound, clear depth))
            if (e.x != kEmptySlot)
            {
                const uint32_t zocc = a.tile_zocc[e.x];
                bin = a.tile_offset[e.x];
                const uint32_t ri = e.y >> 2;
                if (zocc != 0xFFFFFFFFu && ri < a.rtri_capacity && a.rtri_zlo[ri] > min(zocc, 0xBF800000u))
                    e.x = kEmptySlot;
            }
        }
        uint32_t base = 0;
        if (a.vrecs)
        {
            // a mesh with shared vertices: neighbouring lanes hold entries
            // of neighbouring triangles, interleaved over the same few
            // tiles; all lanes with equal tiles share one atomic
            const uint32_t peers = __match_any_sync(0xffffffffu, e.x);
            const int leader = __ffs(peers) - 1;
            if ((int)lane == leader && e.x != kEmptySlot)
                base = atomicAdd(&a.tile_cursor[e.x], (uint32_t)__popc(peers));
            base = __shfl_sync(0xffffffffu, base, leader) + (uint32_t)__popc(peers & ((1u << lane) - 1u));
        }
        else
        {
            // a triangle soup: lanes rarely share a tile, except in runs
            // of consecutive lanes, which share one atomic
            const uint32_t prev = __shfl_up_sync(0xffffffffu, e.x, 1);
            const uint32_t heads = __ballot_sync(0xffffffffu, lane == 0 || e.x != prev);
            const uint32_t upto = 0xffffffffu >> (31 - lane);  // lanes 0..lane
            const uint32_t head = 31 - __clz(heads & upto);
            if (lane == head && e.x != kEmptySlot)
            {
                const uint32_t later = heads & ~upto;
                const uint32_t end = later ? (uint32_t)__ffs(later) - 1u : 32u;
                base = atomicAdd(&a.tile_cursor[e.x], end - lane);
            }
            base = __shfl_sync(0xffffffffu, base, head) + (lane - head);
        }
        if (e.x == kEmptySlot)
            continue;
        const uint64_t pos = (uint64_t)bin + base;
        if (pos < a.bin_capacity)
            a.bins[pos] = e.y;
    }
}

// Upper bound (as a depth key) of every depth the reference computes for
// the triangle at a pixel of a 16x16 block it trivially accepts, or ~0 (no
// bound) when its edge values can wrap or its depths are not finite.  The
// block's corners are inside every edge, so are all its pixel centres: the
// barycentrics are within a few ulps of [0, 1] and the depth at most max(z)
// plus a few ulps of the |z| sum.  Every entry of the tile whose lower bound
// lies beyond it loses at every pixel to this triangle's fragment.
__device__ __forceinline__ uint32_t zmax_key(const RTri& t)
{
    if (!wrap_free(t))
        return 0xFFFFFFFFu;
    const float zmax = fmaxf(t.z0, fmaxf(t.z1, t.z2));
    const float margin = 2e-6f * (fabsf(t.z0) + fabsf(t.z1) + fabsf(t.z2)) + 1e-30f;
    const float hi = zmax + margin;
    return (hi == hi && fabsf(hi) <= 3.0e38f && fabsf(t.invDet) <= 3.0e38f) ? depth_key(hi) : 0xFFFFFFFFu;
}

// Big triangles, up to 32 at a time per warp: their (triangle, 32x32 reference
// tile) pairs are numbered across the warp and taken 32 at a time, each lane
// deciding the four quadrants of its pair's tile, so a triangle with few
// tiles does not leave lanes idle.  Each entry is counted in its tile and
// kept in the unsorted list, which the warp fills from slots it reserves
// kBigChunk at a time (one atomic on the shared counter per chunk); slots
// it leaves unused are marked empty.  Warps that share a triangle reserve what
// a round needs and no more: a chunk for each of up to 32 warps would be up to
// 4,096 slots for a thin triangle's hundred entries.
__global__ void __launch_bounds__(256, 4) k_bin_big(PassArgs a)
{
    follow_on();
    const uint32_t nb = min(*(volatile uint32_t*)&a.counters[2], a.big_capacity);
    if (!nb)
        return;  // (the divisions below, on every warp, take 0.9 us of a small frame)
    const uint32_t lane = threadIdx.x & 31;
    const uint32_t nw = (gridDim.x * blockDim.x) >> 5;
    // batches of up to 32 triangles, small enough that every warp gets one
    const uint32_t batch = min(32u, max(1u, (nb + nw - 1) / nw));
    // with few triangles, several warps share one, each taking every parts-th
    // 32 of its tiles (a triangle over the whole screen is 7 rounds for one
    // warp at 1366x769, 255 at 3840x2160)
    const uint32_t parts = min(32u, max(1u, nw / nb));
    const uint32_t gw = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const uint32_t group = gw / parts, part = gw % parts;
    if (group * batch >= nb)
        return;
    // the warp's current chunk of its stripe of the unsorted list: the stripes
    // of a triangle's parts follow one another from its group's on, so that
    // neither the parts of one triangle nor the first parts of all (the only
    // ones with work where triangles have few tiles) meet in one stripe
    const uint32_t stripe = (group + part) % (uint32_t)kBinStripes;
    const uint64_t send = stripe_begin(a, stripe) + stripe_slots(a.bin_capacity);
    uint64_t cbase = 0;
    uint32_t cleft = 0;
    auto mark_empty = [&]() {
        for (uint32_t k = lane; k < cleft; k += 32)
            if (cbase + k < send)
                a.bin_tmp[cbase + k] = make_uint2(kEmptySlot, 0u);
    };
    const bool early_cull = nb >= a.total_tiles;
    for (uint32_t b0 = group * batch; b0 < nb; b0 += max(1u, nw / parts) * batch)
    {
        // this lane's triangle of the batch and its number of 32x32 tiles
        uint32_t mine = kNoTriangle, mine_zocc = 0xFFFFFFFFu;
        int n = 0;
        if (lane < batch && b0 + lane < nb)
        {
            mine = a.big_list[b0 + lane];
            const RTri t = a.rtris[mine];
            const BinGeom g = bin_geom(t, a.frames[t.meta >> 12]);
            n = (g.t32x1 - g.t32x0 + 1) * (g.t32y1 - g.t32y0 + 1);
            mine_zocc = zmax_key(t);
        }
        int incl = n;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1)
        {
            const int v = __shfl_up_sync(0xffffffffu, incl, o);
            if (lane >= (uint32_t)o) incl += v;
        }
        const int pairs = __shfl_sync(0xffffffffu, incl, 31);
        for (int base = 32 * (int)part; base < pairs; base += 32 * (int)parts)
        {
            const int p = base + (int)lane;
            // owner: the first lane whose inclusive count exceeds p
            int j = 0;
#pragma unroll
            for (int st = 16; st >= 1; st >>= 1)
            {
                const int v = __shfl_sync(0xffffffffu, incl, j + st - 1);
                if (v <= p) j += st;
            }
            const int first = __shfl_sync(0xffffffffu, incl - n, j);
            const uint32_t ri = __shfl_sync(0xffffffffu, mine, j);
            // an accepted quadrant is covered whole: the triangle's far depth
            // bounds the tile
            const uint32_t zocc = __shfl_sync(0xffffffffu, mine_zocc, j);
            uint32_t dq = 0, tile00 = 0;
            int tdx = 0;
            if (p < pairs)
            {
                const RTri t = a.rtris[ri];
                const FrameDesc& f = a.frames[t.meta >> 12];
                const BinGeom g = bin_geom(t, f);
                const Edges e = tri_edges(t);
                const int nx = g.t32x1 - g.t32x0 + 1, local = p - first;
                const int T32y = g.t32y0 + local / nx, T32x = g.t32x0 + local - (local / nx) * nx;
                dq = quad_decisions(t, e, g, f, T32x, T32y);
                tdx = f.tdx;
                tile00 = f.tile_base + (uint32_t)(2 * T32y * f.tdx + 2 * T32x);
                // a quadrant already hidden behind its tile's occluder bound
                // (which only falls) gets no entry: the scatter would drop it.
                // Checked when big triangles outnumber tiles (deep overdraw of
                // large triangles); with few, the check's load costs more.
                const uint32_t zlo = early_cull ? zmin_key(t, wrap_free(t)) : 0u;
#pragma unroll
                for (int q = 0; q < 4; q++)
                    if (early_cull && ((dq >> (2 * q)) & 3u))
                    {
                        const uint32_t tq = tile00 + (uint32_t)((q >> 1) * tdx + (q & 1));
                        const uint32_t zocc_now = *(volatile uint32_t*)&a.tile_zocc[tq];
                        if (zocc_now != 0xFFFFFFFFu && zlo > min(zocc_now, 0xBF800000u))
                            dq &= ~(3u << (2 * q));
                    }
            }
            const uint32_t nz = (dq | (dq >> 1)) & 0x55u;
            const int cnt = __popc(nz);
            int cincl = cnt;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1)
            {
                const int v = __shfl_up_sync(0xffffffffu, cincl, o);
                if (lane >= (uint32_t)o) cincl += v;
            }
            const uint32_t h = (uint32_t)__shfl_sync(0xffffffffu, cincl, 31);
            if (h == 0)
                continue;
            if (h > cleft)
            {
                mark_empty();
                const uint32_t chunk = parts > 1 ? h : kBigChunk;
                uint32_t nbase = 0;
                if (lane == 0)
                    nbase = atomicAdd(stripe_counter(a, stripe), chunk);
                cbase = stripe_begin(a, stripe) + __shfl_sync(0xffffffffu, nbase, 0);
                cleft = chunk;
            }
            uint64_t pos = cbase + (uint32_t)(cincl - cnt);
#pragma unroll
            for (int q = 0; q < 4; q++)
            {
                const uint32_t d = (dq >> (2 * q)) & 3u;
                if (!d)
                    continue;
                const uint32_t tile = tile00 + (uint32_t)((q >> 1) * tdx + (q & 1));
                atomicAdd(&a.tile_count[tile], 1u);
                if (d == kDecisionAccept && zocc != 0xFFFFFFFFu)
                    atomicMin(&a.tile_zocc[tile], zocc);
                if (pos < send)
                    a.bin_tmp[pos] = make_uint2(tile, (ri << 2) | d);
                pos++;
            }
            cbase += h;
            cleft -= h;
        }
    }
    mark_empty();
}

// -------------------------------------------------------------------------
// Exclusive scan of the per-tile counts, each rounded up to a multiple of 4
// entries so every bin starts on a 16-byte boundary, in one pass: blocks
// take consecutive ranges of kScanBlock tiles in the order they start (a
// ticket, so every range a block waits for belongs to a block already
// running) and find their offset by looking back over the published sums of
// the ranges before them (scan_status: 0 not yet, kScanAggregate | sum of
// the range, kScanPrefix | sum of everything up to the range's end).
//
// The same pass lists the raster work items: one per tune.item_entries
// entries of a tile.  Items of at least 3/4 of that are listed from the front
// of the item array, the lighter ones from its back, and the queue hands out
// the front list first: the heavy work starts early instead of forming the
// tail.  Tiles without an entry, which only need their background, have a
// list of their own.
__device__ __forceinline__ uint32_t padded(uint32_t c) { return (c + 3u) & ~3u; }

constexpr unsigned long long kScanAggregate = 1ull << 32;
constexpr unsigned long long kScanPrefix = 2ull << 32;
constexpr int kScanSpinLimit = 1 << 22;

// Block-wide inclusive scan of one value per thread; returns the inclusive
// value and sets `total` (all threads).
__device__ __forceinline__ uint32_t block_scan(uint32_t v, uint32_t* warp_sums, uint32_t& total)
{
    const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    uint32_t incl = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1)
    {
        const uint32_t t = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= (uint32_t)o) incl += t;
    }
    if (lane == 31)
        warp_sums[warp] = incl;
    __syncthreads();
    if (warp == 0)
    {
        const uint32_t w = lane < (blockDim.x >> 5) ? warp_sums[lane] : 0u;
        uint32_t wi = w;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1)
        {
            const uint32_t t = __shfl_up_sync(0xffffffffu, wi, o);
            if (lane >= (uint32_t)o) wi += t;
        }
        warp_sums[lane] = wi - w;
        if (lane == 31)
            warp_sums[32] = wi;
    }
    __syncthreads();
    total = warp_sums[32];
    return warp_sums[warp] + incl;
}

__global__ void __launch_bounds__(kScanThreads) k_scan(PassArgs a)
{
    follow_on();
    __shared__ uint32_t warp_sums[33];
    __shared__ uint32_t s_block, s_prefix;
    __shared__ bool s_dropped, s_dense;
    const uint32_t lane = threadIdx.x & 31;
    if (threadIdx.x == 0)
        s_block = atomicAdd(&a.counters[8], 1u);
    __syncthreads();
    const uint32_t b = s_block;
    const uint32_t base = b * kScanBlock + threadIdx.x * kScanItems;
    uint32_t cnt[kScanItems], sum = 0;
#pragma unroll
    for (int k = 0; k < kScanItems; k++)
    {
        const uint32_t i = base + k;
        cnt[k] = (i < a.total_tiles) ? a.tile_count[i] : 0u;
        sum += padded(cnt[k]);
    }
    // (the last warp, for the statistics as well; loaded before the scan's
    // barriers and the look-back)
    uint32_t filled = 0, survived = 0;
    if (threadIdx.x >= kScanThreads - 32)
    {
        static_assert(kBinStripes == 32, "one lane per stripe");
        const volatile uint32_t* c = stripe_counter(a, lane);
        filled = c[0];
        survived = c[1];
        const bool over = __any_sync(0xffffffffu, filled > stripe_slots(a.bin_capacity));
        // many entries a tile: single warps rasterize them (see by_density; in
        // sixteenths, so that the sum fits 32 bits)
        const bool dense = a.dense_entries && __reduce_add_sync(0xffffffffu, filled >> 4) >
                                                  (uint64_t)a.total_tiles * (kDenseEntries >> 4);
        if (lane == 0)
        {
            s_dropped = over;
            s_dense = dense;
            if (b == 0)
                a.counters[10] = dense ? 1u : 0u;
        }
    }
    uint32_t total;
    const uint32_t incl = block_scan(sum, warp_sums, total);
    // Look back over the ranges before this one, a warp's lanes on 32 of them
    // at a time: the nearest that publishes everything up to its end, and the
    // sums of those after it.  (One thread walking them took an L2 round trip
    // per range.)
    if (threadIdx.x < 32)
    {
        // (a failure test makes one block keep its sums to itself)
        const bool publish = (int)b != a.tune.scan_stall_block && lane == 0;
        const int spin_limit = a.tune.scan_spin_limit > 0 ? a.tune.scan_spin_limit : kScanSpinLimit;
        uint32_t prefix = 0;
        if (b > 0 && publish)
            atomicExch(&a.scan_status[b], kScanAggregate | total);
        for (int j = (int)b - 1, spins = 0; j >= 0;)
        {
            const int r = j - (int)lane;
            unsigned long long st = kScanPrefix;
            if (r >= 0)
                st = *(volatile unsigned long long*)&a.scan_status[r];
            const uint32_t missing = __ballot_sync(0xffffffffu, st == 0), ends = __ballot_sync(0xffffffffu, (st & kScanPrefix) != 0);
            // lanes before the first range that is not there yet, up to the first prefix
            const uint32_t known = missing ? (missing & (0u - missing)) - 1u : 0xffffffffu;
            const uint32_t end = ends & known;
            if (!end && missing)
            {
                if (++spins >= spin_limit)
                {
                    // a range never published: report it, never hang
                    if (lane == 0)
                        atomicOr(&a.status->error, 3u);  // EDXR_ERR_TIMEOUT
                    break;
                }
                continue;
            }
            const uint32_t take = end ? (end ^ (end - 1u)) : 0xffffffffu;  // up to the first prefix
            prefix += __reduce_add_sync(0xffffffffu, (take >> lane) & 1u ? (uint32_t)st : 0u);
            if (end)
                break;
            j -= 32;
            spins = 0;
        }
        if (publish)
            atomicExch(&a.scan_status[b], kScanPrefix | (prefix + total));
        if (lane == 0)
            s_prefix = prefix;
    }
    __syncthreads();
    const uint32_t prefix = s_prefix;

    // offsets, and the items of this thread's tiles.  A frame whose entries
    // did not all fit (the unsorted list or the bins overflowed) is rendered
    // again by the host; its tiles are made empty here, so no raster item
    // reads a bin with missing entries or leaves a split tile's keys behind.
    const bool dropped = s_dropped;
    // entries per work item; items of at least 3/4 of that are heavy
    const uint32_t E = s_dense ? a.dense_entries : (uint32_t)a.tune.item_entries, heavy_min = E - E / 4;
    uint32_t run = prefix + incl - sum;
    uint32_t nheavy = 0, nlight = 0, nempty = 0;
    uint32_t start[kScanItems], n[kScanItems];
#pragma unroll
    for (int k = 0; k < kScanItems; k++)
    {
        const uint32_t i = base + k;
        start[k] = run;
        n[k] = 0;
        if (i < a.total_tiles)
        {
            a.tile_offset[i] = run;
            uint32_t c = cnt[k];
            a.tile_count[i] = 0;  // from here on: the split tile's rastered entries
            if (dropped || (uint64_t)run + c > a.bin_capacity)
                c = 0;
            n[k] = (c + E - 1) / E;
            // only the last item of a tile can be light
            const uint32_t light = c && (c - (n[k] - 1) * E) < heavy_min ? 1u : 0u;
            nlight += light;
            nheavy += n[k] - light;
            nempty += c ? 0u : 1u;
            cnt[k] = c;
        }
        run += padded(cnt[k]);
    }
    // one atomic per warp and list (light and empty counts, at most 128 each,
    // share a word)
    const uint32_t packed = nlight | (nempty << 16);
    uint32_t hincl = nheavy, pincl = packed;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1)
    {
        const uint32_t h = __shfl_up_sync(0xffffffffu, hincl, o), t = __shfl_up_sync(0xffffffffu, pincl, o);
        if (lane >= (uint32_t)o)
        {
            hincl += h;
            pincl += t;
        }
    }
    uint32_t hbase = 0, lbase = 0, ebase = 0;
    if (lane == 31)
    {
        if (hincl)
            hbase = atomicAdd(&a.counters[6], hincl);
        if (pincl & 0xFFFFu)
            lbase = atomicAdd(&a.counters[7], pincl & 0xFFFFu);
        if (pincl >> 16)
            ebase = atomicAdd(&a.counters[9], pincl >> 16);
    }
    const uint32_t pexcl = pincl - packed;
    hbase = __shfl_sync(0xffffffffu, hbase, 31) + hincl - nheavy;
    lbase = __shfl_sync(0xffffffffu, lbase, 31) + (pexcl & 0xFFFFu);
    ebase = __shfl_sync(0xffffffffu, ebase, 31) + (pexcl >> 16);
#pragma unroll
    for (int k = 0; k < kScanItems; k++)
    {
        const uint32_t i = base + k;
        if (i >= a.total_tiles)
            continue;
        if (!cnt[k])
        {
            a.empty_tiles[ebase++] = i;
            continue;
        }
        const bool light = (cnt[k] - (n[k] - 1) * E) < heavy_min;
        const uint32_t heavy = n[k] - (light ? 1u : 0u);
        const uint32_t end = start[k] + cnt[k];
        const uint32_t tag = i | (n[k] > 1 ? kSplitTile : 0u);
        for (uint32_t j = 0; j < heavy; j++, hbase++)
            if (hbase < a.item_capacity)
                a.items[hbase] = make_uint4(tag, start[k] + j * E, min(end, start[k] + (j + 1) * E), start[k]);
        if (light)
        {
            if (lbase < a.item_capacity)
                a.items[a.item_capacity - 1 - lbase] = make_uint4(tag, start[k] + (n[k] - 1) * E, end, start[k]);
            lbase++;
        }
    }

    // the range holding the last tile has the grand total
    if (a.total_tiles > 0 && b == (a.total_tiles - 1) / kScanBlock && threadIdx.x >= kScanThreads - 32)
    {
        const uint64_t grand = prefix + total;
        // the unsorted list's stripes share the capacity: the fullest decides
        const uint64_t fullest = __reduce_max_sync(0xffffffffu, filled);
        uint64_t entries = filled, survivors = survived;
        for (int o = 16; o >= 1; o >>= 1)
        {
            entries += __shfl_down_sync(0xffffffffu, entries, o);
            survivors += __shfl_down_sync(0xffffffffu, survivors, o);
        }
        if (lane != 0)
            return;
        a.tile_offset[a.total_tiles] = (uint32_t)grand;
        const uint64_t needed = max(grand, fullest * kBinStripes);
        a.status->bins_needed = needed;
        a.status->bin_entries = entries;
        a.status->raster_tris = (uint32_t)survivors + a.counters[11];
        a.status->rtri_slots = a.total_tris + a.counters[0];
        a.status->big_tris = a.counters[2];
        if ((uint64_t)a.total_tris + a.counters[0] > a.rtri_capacity)
            atomicOr(&a.status->overflow, 2u);
        if (a.counters[4] > a.poly_capacity)
            atomicOr(&a.status->overflow, 4u);
        a.status->clipped_polys = a.counters[4];  // one polygon record per queued triangle
        if (needed > a.bin_capacity)
            atomicOr(&a.status->overflow, 1u);
        if (a.counters[2] > a.big_capacity)
            atomicOr(&a.status->overflow, 8u);
    }
}

// -------------------------------------------------------------------------
// Raster: persistent warps take work items from a queue.  An item is one
// 16x16 tile's slice of at most tune.item_entries bin entries; the warp keeps one
// 64-bit key per pixel of the tile in shared memory.  The winner of the
// reference's sequential depth test at a pixel is the fragment with the
// smallest key (depth key << 32 | submission rank term): for LEQUAL the last
// fragment with the smallest depth wins, for LESS the first.  Keys can be
// combined in any order, so the bin needs no ordering and two paths share
// the work of each group of 32 entries (one staged per lane):
//  * small entries (region of at most tune.small_region pixels): their
//    (entry, pixel) pairs are spread over the lanes, merging into the key
//    array with a shared 64-bit atomicMin;
//  * the other entries are staged as tile-relative edge equations and
//    rasterized pixel-parallel by the whole warp over their region.
// Entries whose depth lower bound is behind every pixel of the tile so far
// (the tile's hierarchical depth bound) are skipped.  The winners are then
// shaded by the same warp: directly for a tile of one item; for a tile split
// into several items, by the item that finishes last, after all of them
// merged their keys in the per-pixel key buffer.
struct __align__(16) StagedTri
{
    int A0, D0, K0, A1;    // e0 = A0*lx + D0*ly + K0 (with bias); l1 = A1*lx + D1*ly + K1 (no bias)
    int D1, K1, A2, D2;
    int K2;
    uint32_t flags;        // region lx0|lx1<<5|ly0<<10|ly1<<15, accept<<20, bias1<<21, bias2<<22
    uint32_t rank;         // global rank: (frame tri_base * 16 + order) + 1
    uint32_t pad;
    float invDet, z0, z1, z2;
};

constexpr uint32_t kEmptyRegion = 16u | (16u << 10);  // lx0 = ly0 = 16 > lx1 = ly1 = 0

// Tile-relative edge equations, barycentric numerators and region of one
// bin entry.
// With MS (several samples per pixel) it also returns G[k] = B[k] + C[k]:
// sample s sits at (o, o) from the pixel centre (see kSampleOffsets), where
// edge k changes by o * G[k]; and it keeps the quad-aligned region.
template <bool MS = false>
__device__ __forceinline__ void stage_tri(const PassArgs& a, uint32_t entry, uint32_t nr, uint32_t rank_base,
                                          int tileX, int tileY,
                                          StagedTri& s, uint32_t& zkey, int* G = nullptr,
                                          bool* wrapfree = nullptr)
{
    const uint32_t ri = entry >> 2;
    if (ri >= nr)
    {
        // never written by a consistent pass; an empty region keeps it inert
        s.flags = kEmptyRegion;
        zkey = 0xFFFFFFFFu;
        return;
    }
    const bool accept = (entry & 3u) == kDecisionAccept;
    const RTri t = load_rtri(a.rtris + ri);
    const Edges e = tri_edges(t);
    // pixel (lx, ly) of the tile samples at (16*(16*tileX + lx) + 8, ...)
    const int ox = (tileX << 8) + 8, oy = (tileY << 8) + 8;
    int A[3], D[3], K[3], bias[3];
#pragma unroll
    for (int k = 0; k < 3; k++)
    {
        const int n = (k + 1) % 3;
        bias[k] = tl_pixel(e.vx[k], e.vy[k], e.vx[n], e.vy[n]);
        A[k] = wmul(16, e.B[k]);
        D[k] = wmul(16, e.C[k]);
        K[k] = wadd(wmul(e.B[k], wsub(ox, e.vx[k])), wmul(e.C[k], wsub(oy, e.vy[k])));
    }
    s.A0 = A[0]; s.D0 = D[0]; s.K0 = wadd(K[0], bias[0]);
    // the barycentric numerators of RasterTriangle.h:335-336 are edges 1
    // and 2 measured from v2, equal to the unbiased edge values
    s.A1 = A[1]; s.D1 = D[1]; s.K1 = K[1];
    s.A2 = A[2]; s.D2 = D[2]; s.K2 = K[2];
    if (MS)
    {
#pragma unroll
        for (int k = 0; k < 3; k++)
            G[k] = wadd(e.B[k], e.C[k]);
    }
    // wrap-free: covered pixel centres lie in the vertices' bounding box (the
    // tight region, single sample only: an off-centre sample can be covered
    // where the centre is not), and the depth bound below holds at every
    // covered sample
    const bool wfree = wrap_free(t);
    if (MS)
        *wrapfree = wfree;
    const bool wf = !MS && wfree;
    int lx0 = 0, lx1 = 15, ly0 = 0, ly1 = 15;
    if (!accept)
    {
        // FineRasterize's quad-aligned bounding box (Rasterizer.h:132-140),
        // or only the pixels whose centre is in the vertices' bounding box
        // when no edge function can wrap (no other centre can be covered)
        const int minx = min(t.v0x, min(t.v1x, t.v2x)), maxx = max(t.v0x, max(t.v1x, t.v2x));
        const int miny = min(t.v0y, min(t.v1y, t.v2y)), maxy = max(t.v0y, max(t.v1y, t.v2y));
        // with several samples, each inside its own pixel (offsets -8..7 in
        // 1/16 pixel): the pixels the wrap-free triangle's box overlaps
        const bool box = MS && wfree;
        const int bbx0 = wf ? centre_lo(minx) : box ? minx >> 4 : (minx >> 4) & ~1;
        const int bbx1 = wf ? centre_hi(maxx) : box ? maxx >> 4 : (maxx >> 4) | 1;
        const int bby0 = wf ? centre_lo(miny) : box ? miny >> 4 : (miny >> 4) & ~1;
        const int bby1 = wf ? centre_hi(maxy) : box ? maxy >> 4 : (maxy >> 4) | 1;
        lx0 = max(0, bbx0 - (tileX << 4));
        lx1 = min(15, bbx1 - (tileX << 4));
        ly0 = max(0, bby0 - (tileY << 4));
        ly1 = min(15, bby1 - (tileY << 4));
        if (lx1 < lx0 || ly1 < ly0) { lx0 = 16; lx1 = 0; ly0 = 16; ly1 = 0; }
    }
    s.flags = (uint32_t)lx0 | ((uint32_t)lx1 << 5) | ((uint32_t)ly0 << 10) | ((uint32_t)ly1 << 15) |
              (accept ? (1u << 20) : 0u) | (bias[1] ? (1u << 21) : 0u) | (bias[2] ? (1u << 22) : 0u);
    s.invDet = t.invDet;
    s.z0 = t.z0; s.z1 = t.z1; s.z2 = t.z2;
    // submission order within the frame, offset by the frame's first input
    // triangle, so the winner's record is found from the rank alone
    s.rank = rank_base + t.order + 1u;
    zkey = zmin_key(t, wfree);
}

// Key of the fragment of staged triangle s at tile pixel (lx, ly), or false
// when the pixel is not covered (FineRasterize's edge test; trivially
// accepted entries skip it) or the depth is NaN (never passes).
__device__ __forceinline__ bool fragment_key(const StagedTri& s, int lx, int ly, bool less, uint64_t& key)
{
    // (no early exit: the lanes of a warp test different pixels, and the
    // arithmetic of an uncovered one costs the warp nothing extra)
    const uint32_t fl = s.flags;
    const int l1 = wadd(wadd(wmul(s.A1, lx), wmul(s.D1, ly)), s.K1);
    const int l2 = wadd(wadd(wmul(s.A2, lx), wmul(s.D2, ly)), s.K2);
    const int e0 = wadd(wadd(wmul(s.A0, lx), wmul(s.D0, ly)), s.K0);
    const int e1 = wadd(l1, (fl & (1u << 21)) ? -1 : 0);
    const int e2 = wadd(l2, (fl & (1u << 22)) ? -1 : 0);
    const bool inside = (fl & (1u << 20)) || (e0 | e1 | e2) >= 0;
    // TriangleSSE::CalcBarycentricCoord / GetDepth (RasterTriangle.h:324-337)
    const float L0 = fmul(__int2float_rn(l1), s.invDet);
    const float L1 = fmul(__int2float_rn(l2), s.invDet);
    const float L2 = fsub(fsub(1.0f, L0), L1);
    const float d = fadd(fadd(fmul(L0, s.z0), fmul(L1, s.z1)), fmul(L2, s.z2));
    key = ((uint64_t)depth_key(d) << 32) | (less ? s.rank : ~s.rank);
    return inside && d == d;
}

constexpr int kRasterWarps = kRasterThreads / 32;

// A staged entry padded to 80 bytes: lanes reading different entries hit
// different shared-memory banks.
struct __align__(16) StagedSlot
{
    StagedTri s;
    uint4 pad;
};

// The next work item of a persistent raster warp: after the first (item
// number = the warp's index in the grid, no claim), items first_items,
// first_items + 1, ... are claimed one at a time.
__device__ __forceinline__ uint32_t claim_item(const PassArgs& a, uint32_t first_items)
{
    uint32_t q = 0;
    if ((threadIdx.x & 31) == 0)
        q = first_items + atomicAdd(&a.counters[3], 1u);
    return __shfl_sync(0xffffffffu, q, 0);
}

// Raster triangle of the fragment with submission rank `rank` (0: none), or
// kNoTriangle.  rank - 1 = flattened input triangle * 16 + fan field: 0 for a
// triangle that was not clipped, whose record sits at its flattened index;
// piece `fan` of a clipped triangle otherwise, in slot tri_first + fan - 1
// (each clipped triangle reserves a slot per fan piece, in fan order).
__device__ __forceinline__ uint32_t raster_triangle_of(const PassArgs& a, uint32_t rank, uint32_t nr)
{
    if (rank == 0)
        return kNoTriangle;
    const uint32_t gi = (rank - 1u) >> 4, fan = (rank - 1u) & 15u;
    if (fan == 0)
        return gi < a.total_tris ? gi : kNoTriangle;
    const uint32_t ri = gi < a.total_tris ? a.tri_first[gi] + fan - 1u : kNoTriangle;
    return ri < nr ? ri : kNoTriangle;
}

// *p += v at device scope with acquire-release semantics; returns the old
// value.  A split tile's items count its rastered entries with it (see k_raster).
__device__ __forceinline__ uint32_t atomic_add_acq_rel(uint32_t* p, uint32_t v)
{
    uint32_t old;
    asm volatile("atom.acq_rel.gpu.global.add.u32 %0, [%1], %2;\n" : "=r"(old) : "l"(p), "r"(v) : "memory");
    return old;
}

// Depth of raster triangle t at 1/16-pixel position (x, y)
// (RasterTriangle.h:324-337).
__device__ __forceinline__ float depth_at(const RTri& t, int x, int y, float& L0, float& L1)
{
    const Edges e = tri_edges(t);
    const int n1 = wadd(wmul(e.B[1], wsub(x, t.v2x)), wmul(e.C[1], wsub(y, t.v2y)));
    const int n2 = wadd(wmul(e.B[2], wsub(x, t.v2x)), wmul(e.C[2], wsub(y, t.v2y)));
    L0 = fmul(__int2float_rn(n1), t.invDet);
    L1 = fmul(__int2float_rn(n2), t.invDet);
    const float L2 = fsub(fsub(1.0f, L0), L1);
    return fadd(fadd(fmul(L0, t.z0), fmul(L1, t.z1)), fmul(L2, t.z2));
}

// The one write of a pixel (Renderer::FragmentProcessing / UpdateFrameBuffer,
// Renderer.cpp:272-350, shade every fragment and keep the last; only the
// winner is shaded here): its barycentrics and depth are recomputed exactly
// (RasterTriangle.h:324-337), then interpolated and shaded.  Inlined: a
// call per pixel cost more than the registers it spills in the raster loop.
struct PixelOut
{
    const RTri* rtris;
    const ClipPoly* polys;
    float4* color;
    float* depth;
    uint32_t* tri_id;
};

// The per-vertex-attribute shaders (Blinn-Phong, Lambertian with or without
// albedo) at barycentrics (L0, L1) of raster triangle t: perspective-correct
// weights, the vertices' attributes, the shading model.  No call inside.
static __device__ __forceinline__ float3 shade_common(const FrameDesc& f, const RTri& t, const ClipPoly* polys,
                                                      float L0, float L1, const uint32_t* vi = nullptr)
{
    float b0 = L0, b1 = L1;
    float b2 = fsub(fsub(1.0f, b0), b1);
    b0 = fmul(b0, t.invW0);
    b1 = fmul(b1, t.invW1);
    b2 = fmul(b2, t.invW2);
    const float invB = __frcp_rn(fadd(fadd(b0, b1), b2));
    b0 = fmul(b0, invB);
    b1 = fmul(b1, invB);
    b2 = fsub(fsub(1.0f, b0), b1);
    const ShadeVerts v = shade_verts(f, t, polys, vi);
    return shade_model(f, lerp3(b0, v.p[0], b1, v.p[1], b2, v.p[2]), lerp3(b0, v.n[0], b1, v.n[1], b2, v.n[2]),
                       lerp3(b0, v.a[0], b1, v.a[1], b2, v.a[2]));
}

// Is the frame shaded out of line (the reference Blinn-Phong and the textured
// shaders)?
__device__ __forceinline__ bool slow_shading(const FrameDesc& f) { return f.ps_kind == 1 || f.ps_kind == 4; }

static __device__ __forceinline__ void write_pixel(const PixelOut a, const FrameDesc& f, uint32_t ri, uint64_t pix, int px,
                                                int py)
{
    if (ri == kNoTriangle)
    {
        a.color[pix] = make_float4(0.f, 0.f, 0.f, 0.f);
        a.depth[pix] = 1.0f;
        a.tri_id[pix] = kNoTriangle;
        return;
    }
    const RTri t = load_rtri(a.rtris + ri);
    const Edges e = tri_edges(t);
    const int cx = (px << 4) + 8, cy = (py << 4) + 8;
    const int n1 = wadd(wmul(e.B[1], wsub(cx, t.v2x)), wmul(e.C[1], wsub(cy, t.v2y)));
    const int n2 = wadd(wmul(e.B[2], wsub(cx, t.v2x)), wmul(e.C[2], wsub(cy, t.v2y)));
    const float L0 = fmul(__int2float_rn(n1), t.invDet);
    const float L1 = fmul(__int2float_rn(n2), t.invDet);
    const float L2 = fsub(fsub(1.0f, L0), L1);
    const float d = fadd(fadd(fmul(L0, t.z0), fmul(L1, t.z1)), fmul(L2, t.z2));
    const float3 c = shade_fragment(f, t, a.rtris + ri, a.polys, L0, L1, px, py);
    a.color[pix] = make_float4(c.x, c.y, c.z, 1.0f);
    a.depth[pix] = d;
    a.tri_id[pix] = t.order >> 4;
}

// The one write of a pixel for the per-vertex-attribute shaders: no call
// inside.
static __device__ __forceinline__ void write_pixel_fast(const PixelOut a, const FrameDesc& f, uint32_t ri,
                                                        uint64_t pix, int px, int py, uint32_t rank)
{
    if (ri == kNoTriangle)
    {
        a.color[pix] = make_float4(0.f, 0.f, 0.f, 0.f);
        a.depth[pix] = 1.0f;
        a.tri_id[pix] = kNoTriangle;
        return;
    }
    // the rank names the input triangle: its indices load beside its record
    const uint32_t tri = ((rank - 1u) >> 4) - f.tri_base;
    const uint32_t* idx = f.indices + 3 * (size_t)tri;
    const uint32_t vi[3] = { __ldg(idx), __ldg(idx + 1), __ldg(idx + 2) };
    const RTri t = load_rtri(a.rtris + ri);
    float L0, L1;
    const float d = depth_at(t, (px << 4) + 8, (py << 4) + 8, L0, L1);
    const float3 c = shade_common(f, t, a.polys, L0, L1, vi);
    a.color[pix] = make_float4(c.x, c.y, c.z, 1.0f);
    a.depth[pix] = d;
    a.tri_id[pix] = tri;
}

// A tile shaded by the reference Blinn-Phong or the textured shader
// (slow_shading): out of line, pixel by pixel, so that the common shaders' loop
// keeps its registers.
static __device__ __noinline__ void shade_tile_slow(const PixelOut out, const FrameDesc& f,
                                                    const unsigned long long* key, int first, int step, int tileX,
                                                    int tileY, bool less, uint32_t nr, const uint32_t* tri_first,
                                                    uint32_t total_tris)
{
#pragma unroll 1
    for (int p = first; p < 256; p += step)
    {
        const int px = (tileX << 4) + (p & 15), py = (tileY << 4) + (p >> 4);
        if (px >= f.width || py >= f.height)
            continue;
        const uint32_t low = (uint32_t)key[p];
        const uint32_t rank = less ? low : ~low;
        uint32_t ri = kNoTriangle;
        if (rank)
        {
            // raster_triangle_of on the pass's tables
            const uint32_t gi = (rank - 1u) >> 4, fan = (rank - 1u) & 15u;
            if (gi < total_tris)
                ri = fan == 0 ? gi : tri_first[gi] + fan - 1u;
            if (ri >= nr)
                ri = kNoTriangle;
        }
        write_pixel(out, f, ri, f.pix_base + (uint64_t)py * (uint32_t)f.width + (uint32_t)px, px, py);
    }
}

// The background of a tile, written by `threads` threads.
static __device__ __forceinline__ void clear_tile(const PassArgs& a, const FrameDesc& f, uint32_t tile, int thread,
                                                  int threads)
{
    const uint32_t lt = tile - f.tile_base;
    const int tileX = (int)(lt % (uint32_t)f.tdx), tileY = (int)(lt / (uint32_t)f.tdx);
    const int w = f.width, h = f.height;
    const uint64_t base = f.pix_base;
    for (int p = thread; p < 256; p += threads)
    {
        const int px = (tileX << 4) + (p & 15), py = (tileY << 4) + (p >> 4);
        if (px < w && py < h)
        {
            const uint64_t pix = base + (uint64_t)py * (uint32_t)w + (uint32_t)px;
            a.color[pix] = make_float4(0.f, 0.f, 0.f, 0.f);
            a.depth[pix] = 1.0f;
            a.tri_id[pix] = kNoTriangle;
        }
    }
}

// The pass's status word, final once the raster kernel runs, written to the
// host (page-locked memory) by its first thread: no copy follows the pass.
__device__ __forceinline__ void report_status(const PassArgs& a)
{
    if (a.status_host && blockIdx.x == 0 && threadIdx.x == 0)
        *a.status_host = *a.status;
}

// Entries a warp stages at a time when `warps` warps share n: the least that
// takes as few rounds as chunks of `most` do, so that the last round is shared
// evenly too.
__device__ __forceinline__ uint32_t even_chunk(uint32_t n, uint32_t warps, uint32_t most = 32u)
{
    const uint32_t rounds = (n + most * warps - 1u) / (most * warps), shares = max(rounds, 1u) * warps;
    return max(1u, (n + shares - 1u) / shares);
}

// Barrier of the Group warps that share an item: the warp's own lanes
// (Group 1), the whole block (Group 8), or a named barrier per group.
template <int Group>
__device__ __forceinline__ void group_sync(int group)
{
    if (Group == 1)
        __syncwarp();
    else if (Group == kRasterWarps)
        __syncthreads();
    else
    {
        __syncwarp();
        asm volatile("bar.sync %0, %1;\n" ::"r"(group + 1), "r"(Group * 32) : "memory");
    }
}

// Group warps share an item (1: a warp per item; 4 or 8 where the frame has
// too few tiles to give every warp one, see raster_group).
// 3 blocks per SM: the 80 registers a thread hold the shading without spills.
// At 5 blocks (48 registers, 156 bytes spilled) the raster stage took 119
// instead of 100 us on the terrain (2,097,152 triangles, 1920x1080), 235
// instead of 217 on the binning stress (3840x2160), 67 instead of 55 on a
// 301x301-quad terrain at 1366x769; at 4 blocks 109, 219 and 61; at 2 blocks
// (124 registers) 111, 250 and 53.
template <int Group, bool One>
__global__ void __launch_bounds__(kRasterThreads, 3) k_raster(PassArgs a)
{
    follow_on();
    constexpr int kGroups = kRasterWarps / Group;   // groups of a block
    constexpr int kThreads = 32 * Group;            // threads of a group
    constexpr int kPixels = 256 / kThreads;         // pixels of the tile per thread
    __shared__ unsigned long long s_key[kGroups][256];
    __shared__ StagedSlot s_tri[kRasterWarps][32];
    __shared__ uint32_t s_next[kGroups], s_done[kGroups], s_staged[kRasterWarps], s_bound[kRasterWarps];
    report_status(a);
    if (*(volatile uint32_t*)&a.status->error)
        return;  // the pass failed (see k_bin_move); every thread of the block leaves
    if (a.dense_entries && (*(volatile uint32_t*)&a.counters[10] != 0) != (Group == 1))
        return;  // the pass's other raster kernel takes the frame
    // ceil(65536 / w): ((p * s_recip[w]) >> 16) == p / w for 0 <= p < 256 and
    // 1 <= w <= 16, the row of pixel p of a region w pixels wide
    __shared__ uint32_t s_recip[17];
    // A pass of one frame (One) keeps its descriptor in shared memory: the
    // shading reads some twenty of its fields a pixel, and stores to the images
    // keep the compiler from holding them (raster stage: terrain 95 -> 93 us,
    // binning stress 219 -> 211).  With several frames each warp keeps its
    // item's, copied when the frame changes: 256 views at 512x512 695 -> 678 us,
    // 64 views at 256x256 110 -> 107.
    __shared__ FrameDesc s_frames[One ? 1 : kRasterWarps];
    FrameDesc& s_frame = s_frames[One ? 0 : threadIdx.x >> 5];
    uint32_t in_shared = 0xFFFFFFFFu;  // several frames: the one whose descriptor the warp holds
    if (One)
        copy_frame(s_frame, a.frames, threadIdx.x, kRasterThreads);
    if (threadIdx.x >= 1 && threadIdx.x <= 16)
        s_recip[threadIdx.x] = (65536u + threadIdx.x - 1u) / threadIdx.x;
    __syncthreads();
    const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int group = (int)warp / Group;
    const uint32_t gwarp = warp % Group;             // warp within the group
    const int gthread = (int)(threadIdx.x % kThreads);
    unsigned long long* key = s_key[group];
    StagedSlot* staged = s_tri[warp];
    // raster-triangle slots in use: one per input triangle, then the fan pieces
    const uint32_t nr = (uint32_t)min((uint64_t)a.total_tris + *(volatile uint32_t*)&a.counters[0],
                                      (uint64_t)a.rtri_capacity);
    const uint32_t nheavy = *(volatile uint32_t*)&a.counters[6];
    const uint32_t nitems = (uint32_t)min((uint64_t)nheavy + *(volatile uint32_t*)&a.counters[7], a.item_capacity);
    const int small_region = min(a.tune.small_region, 64);
    const uint32_t before = (1u << lane) - 1u;  // lanes before this one
    const PixelOut out = { a.rtris, a.polys, a.color, a.depth, a.tri_id };
    // The work: the items, then the tiles without an entry, a few at a time.
    // Each group's first piece is its own (the heaviest items, no claim), the
    // rest are claimed one at a time; nothing is claimed when every piece is
    // some group's first (a claim on the one counter by every warp of the
    // grid takes 3 to 6 us).  The empty tiles at the end fill the tail.  Where
    // the items outnumber the groups, each item writes `share` of the empty
    // tiles first, so that the background's stores overlap other warps'
    // rasterization: 256 views at 512x512 768 -> 728 us.
    const uint32_t nempty = *(volatile uint32_t*)&a.counters[9], ngroups = gridDim.x * kGroups;
    const uint32_t share = nitems >= 2u * ngroups ? min(nempty / nitems, 4u) : 0u;
    const uint32_t shared_tiles = share * nitems;
    const uint32_t bulk = min(8u, max(1u, (nempty - shared_tiles) / ngroups));
    const uint32_t nwork = nitems + (nempty - shared_tiles + bulk - 1) / bulk;
    // the frame of a tile
    auto frame_index = [&](uint32_t tile) -> uint32_t {
        return a.tiles_per_frame ? tile / a.tiles_per_frame
                                 : find_frame(a.frames, a.num_frames, tile,
                                              [](const FrameDesc& f) { return f.tile_base; });
    };
    auto frame_of = [&](uint32_t tile) -> const FrameDesc& {
        if (One)
            return s_frame;
        return a.frames[frame_index(tile)];
    };
    auto next_item = [&]() -> uint32_t {
        if (ngroups >= nwork)
            return nwork;
        if (Group == 1)
            return claim_item(a, ngroups);
        if (gthread == 0)
            s_next[group] = ngroups + atomicAdd(&a.counters[3], 1u);
        group_sync<Group>(group);
        return s_next[group];
    };
    for (uint32_t q = blockIdx.x * kGroups + group; q < nwork; q = next_item())
    {
        if (q >= nitems)
        {
            const uint32_t i0 = shared_tiles + (q - nitems) * bulk, i1 = min(nempty, i0 + bulk);
            for (uint32_t i = i0; i < i1; i++)
                clear_tile(a, frame_of(a.empty_tiles[i]), a.empty_tiles[i], gthread, kThreads);
            if (Group > 1)
                group_sync<Group>(group);
            continue;
        }
        const uint4 item = a.items[q < nheavy ? q : (uint32_t)(a.item_capacity - 1 - (q - nheavy))];
        for (uint32_t i = 0; i < share; i++)
            clear_tile(a, frame_of(a.empty_tiles[q * share + i]), a.empty_tiles[q * share + i], gthread, kThreads);
        const uint32_t tile = item.x & ~kSplitTile;
        if (!One)
        {
            const uint32_t fi = frame_index(tile);
            if (fi != in_shared)
            {
                in_shared = fi;
                __syncwarp();
                copy_frame(s_frame, a.frames + fi, lane, 32u);
                __syncwarp();
            }
        }
        const FrameDesc& f = s_frame;
        const uint32_t lt = tile - f.tile_base;
        const int tileX = (int)(lt % (uint32_t)f.tdx), tileY = (int)(lt / (uint32_t)f.tdx);
        const bool less = f.depth_func == 1;
        // (a frame whose entries overflowed has empty items: rendered again by the host)
        bool split = (item.x & kSplitTile) != 0;
        // the item's range within the entries its bin kept (the scatter drops
        // entries hidden behind the tile's occluder)
        uint32_t e0 = item.y, e1 = item.z, kept = 0;
        // entries a warp stages at a time: 32, fewer where not every warp of
        // the group would get some
        const uint32_t per = Group == 1 ? 32u : even_chunk(e1 - e0, (uint32_t)Group);
        const uint32_t c0 = e0 + per * gwarp, cstep = per * (uint32_t)Group;
        uint32_t next = lane < per && c0 + lane < e1 ? a.bins[c0 + lane] : 0u;
        if (e0 != e1)
        {
            const uint32_t bin0 = item.w;
            kept = a.tile_cursor[tile];
            e1 = min(e1, bin0 + kept);
            e0 = min(e0, e1);
            if (split && e0 == e1)
            {
                if (item.y != bin0 || kept != 0)
                {
                    // the tile's kept entries are in its other items
                    if (Group > 1)
                        group_sync<Group>(group);
                    continue;
                }
                split = false;  // it kept none: its first item writes the background
            }
        }
        if (e0 == e1 && !split)
        {
            // every entry was hidden behind the clear depth: the background, with no key
            clear_tile(a, f, tile, gthread, kThreads);
            if (Group > 1)
                group_sync<Group>(group);
            continue;
        }

        // clear depth 1.0 with no triangle: rank term ~0 (LEQUAL) or 0 (LESS)
        const unsigned long long clear = ((unsigned long long)0xBF800000u << 32) | (less ? 0u : 0xFFFFFFFFu);
#pragma unroll
        for (int k = 0; k < kPixels; k++)
            key[gthread + kThreads * k] = clear;
        group_sync<Group>(group);
        // depth bound of the tile: the nearest triangle that covers it whole,
        // then the largest depth key of its pixels so far
        const uint32_t tzocc = min(0xBF800000u, a.tile_zocc[tile]);
        uint32_t tzmax = tzocc;

        // each chunk's bin entries load while the previous chunk is rasterized
        for (uint32_t c = c0, cg = e0; cg < e1; c += cstep, cg += cstep)
        {
            const uint32_t m = c < e1 ? min(per, e1 - c) : 0u;
            const uint32_t entry = next;
            if (lane < per && c + cstep + lane < e1)
                next = a.bins[c + cstep + lane];
            int nsmall = 0;
            bool big = false;
            StagedTri s;
            if (lane < m)
            {
                uint32_t zk;
                stage_tri(a, entry, nr, f.tri_base << 4, tileX, tileY, s, zk);
                const uint32_t fl = s.flags;
                const int rx0 = fl & 31, rx1 = (fl >> 5) & 31, ry0 = (fl >> 10) & 31, ry1 = (fl >> 15) & 31;
                if (zk <= tzmax && rx0 <= rx1 && ry0 <= ry1)
                {
                    const int area = (rx1 - rx0 + 1) * (ry1 - ry0 + 1);
                    if (!(fl & (1u << 20)) && area <= small_region)
                        nsmall = area;
                    else
                        big = true;
                }
            }
            // staged: the small entries, then the others
            const uint32_t smalls = __ballot_sync(0xffffffffu, nsmall > 0), bigs = __ballot_sync(0xffffffffu, big);
            const int nsm = __popc(smalls), nst = nsm + __popc(bigs);
            if (nsmall > 0)
                staged[__popc(smalls & before)].s = s;
            else if (big)
                staged[nsm + __popc(bigs & before)].s = s;
            // Small entries: their (entry, pixel) pairs are numbered across
            // the warp and taken 32 at a time, so lanes do not idle while
            // one lane walks a larger region.  A lane finds its pair's entry
            // from the entries that begin in the 32 pairs at hand, a lane mask
            // (one warp-wide OR instead of five dependent shuffles of a
            // search: terrain 102 -> 98 us).
            int incl = nsmall;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1)
            {
                const int v = __shfl_up_sync(0xffffffffu, incl, o);
                if (lane >= (uint32_t)o) incl += v;
            }
            const int pairs = __shfl_sync(0xffffffffu, incl, 31);
            __syncwarp();
            int started = -1, carry = 0;  // the last entry begun so far, and its pairs already taken
            for (int base = 0; base < pairs; base += 32)
            {
                // the entries that begin in this window, as a lane mask
                const uint32_t begin = (uint32_t)(incl - nsmall - base);
                const uint32_t heads = __reduce_or_sync(0xffffffffu, nsmall > 0 && begin < 32u ? 1u << begin : 0u);
                const uint32_t upto = heads & (before | (1u << lane));
                const int j = started + __popc(upto);
                const int local = upto ? (int)lane - (31 - __clz(upto)) : carry + (int)lane;
                started += __popc(heads);
                carry = heads ? 32 - (31 - __clz(heads)) : carry + 32;
                if (base + (int)lane < pairs)
                {
                    const StagedTri s = staged[j].s;
                    const uint32_t fl = s.flags;
                    const int rx0 = fl & 31, rx1 = (fl >> 5) & 31, ry0 = (fl >> 10) & 31;
                    const int rw = rx1 - rx0 + 1;
                    const int dy = (int)(((uint32_t)local * s_recip[rw]) >> 16);
                    const int x = rx0 + local - dy * rw, y = ry0 + dy;
                    uint64_t k;
                    // a plain read first: most fragments of deep overdraw lose
                    const bool hit = fragment_key(s, x, y, less, k);
                    const unsigned long long cur = key[y * 16 + x];
                    if (hit && k < cur)
                        atomicMin(&key[y * 16 + x], (unsigned long long)k);
                }
            }
            __syncwarp();
            // Other entries, a warp alone: the whole warp over each region in
            // turn.
            for (int j = nsm; Group == 1 && j < nst; j++)
            {
                const StagedTri s = staged[j].s;
                const uint32_t fl = s.flags;
                const int rx0 = fl & 31, rx1 = (fl >> 5) & 31, ry0 = (fl >> 10) & 31, ry1 = (fl >> 15) & 31;
                const int rw = rx1 - rx0 + 1;
                const int area = rw * (ry1 - ry0 + 1);
                const uint32_t inv = s_recip[rw];
                // each pixel of the region belongs to one lane for this entry
                for (int p = (int)lane; p < area; p += 32)
                {
                    const int dy = (int)(((uint32_t)p * inv) >> 16);
                    const int x = rx0 + p - dy * rw, y = ry0 + dy;
                    uint64_t k;
                    const bool hit = fragment_key(s, x, y, less, k);
                    const unsigned long long cur = key[y * 16 + x];
                    if (hit && k < cur)
                        key[y * 16 + x] = k;
                }
                __syncwarp();
            }
            // Several warps: each thread over its own pixels (the ones it
            // shades) and every warp's staged entries, so no key is shared and
            // none needs an atomic.
            if (Group > 1)
            {
                if (lane == 0)
                    s_staged[warp] = (uint32_t)nsm | ((uint32_t)nst << 8);
                group_sync<Group>(group);  // every warp's entries staged, its small ones rasterized
                unsigned long long mine[kPixels];
                const int x = gthread & 15, row = gthread >> 4;
#pragma unroll
                for (int k = 0; k < kPixels; k++)
                    mine[k] = key[gthread + kThreads * k];
                for (int w = 0; w < Group; w++)
                {
                    const uint32_t range = s_staged[group * Group + w];
                    for (uint32_t j = range & 255u; j < range >> 8; j++)
                    {
                        const StagedTri& t = s_tri[group * Group + w][j].s;
                        const uint32_t fl = t.flags;
                        const int rx0 = fl & 31, rx1 = (fl >> 5) & 31, ry0 = (fl >> 10) & 31, ry1 = (fl >> 15) & 31;
#pragma unroll
                        for (int k = 0; k < kPixels; k++)
                        {
                            const int y0 = 2 * (int)gwarp + (kThreads >> 4) * k;  // the warp's two rows
                            if (y0 + 1 < ry0 || y0 > ry1)
                                continue;
                            const int y = row + (kThreads >> 4) * k;
                            uint64_t kk;
                            const bool hit = fragment_key(t, x, y, less, kk);
                            if (hit && x >= rx0 && x <= rx1 && y >= ry0 && y <= ry1 && kk < mine[k])
                                mine[k] = kk;
                        }
                    }
                }
                uint32_t mz = 0;
#pragma unroll
                for (int k = 0; k < kPixels; k++)
                {
                    key[gthread + kThreads * k] = mine[k];
                    mz = max(mz, (uint32_t)(mine[k] >> 32));
                }
                mz = __reduce_max_sync(0xffffffffu, mz);
                if (lane == 0)
                    s_bound[warp] = mz;
                group_sync<Group>(group);  // before the entries are staged over
                if (cg + cstep < e1)
                {
                    uint32_t b = 0;
                    for (int w = 0; w < Group; w++)
                        b = max(b, s_bound[group * Group + w]);
                    tzmax = min(tzocc, b);
                }
            }
            else if (c + cstep < e1)
            {
                uint32_t mz = 0;
#pragma unroll
                for (int k = 0; k < 8; k++)
                    mz = max(mz, (uint32_t)(key[lane + 32 * k] >> 32));
                tzmax = min(tzocc, __reduce_max_sync(0xffffffffu, mz));
            }
        }

        // A tile split into several items merges its keys in the key buffer;
        // the item that finishes last (the one whose entries bring the tile's
        // rastered count, zeroed by the scan, to the entries its bin kept)
        // shades the tile.
        bool shade = true;
        if (split)
        {
#pragma unroll
            for (int k = 0; k < kPixels; k++)
            {
                const int p = gthread + kThreads * k;
                const int px = (tileX << 4) + (p & 15), py = (tileY << 4) + (p >> 4);
                const unsigned long long kk = key[p];
                if (px < f.width && py < f.height && kk < clear)
                    atomicMax(&a.keybuf[f.pix_base + (uint64_t)py * (uint32_t)f.width + (uint32_t)px], ~kk);
            }
            // The count is one acquire-release atomic: the group's merges
            // happen before it (barrier, then its first thread's release),
            // and the item that completes the tile acquires every other
            // item's merges before it reads them back.
            group_sync<Group>(group);
            if (Group == 1)
            {
                uint32_t done = 0;
                if (lane == 0)
                    done = atomic_add_acq_rel(&a.tile_count[tile], e1 - e0) + (e1 - e0);
                shade = __shfl_sync(0xffffffffu, done, 0) == kept;
                __syncwarp();  // lane 0's acquire, then every lane's reads
            }
            else
            {
                if (gthread == 0)
                    s_done[group] = atomic_add_acq_rel(&a.tile_count[tile], e1 - e0) + (e1 - e0);
                group_sync<Group>(group);
                shade = s_done[group] == kept;
            }
            if (shade)
            {
#pragma unroll
                for (int k = 0; k < kPixels; k++)
                {
                    const int p = gthread + kThreads * k;
                    const int px = (tileX << 4) + (p & 15), py = (tileY << 4) + (p >> 4);
                    if (px < f.width && py < f.height)
                    {
                        // read and leave zero for the next pass
                        const unsigned long long m = atomicExch(
                            &a.keybuf[f.pix_base + (uint64_t)py * (uint32_t)f.width + (uint32_t)px], 0ull);
                        key[p] = m ? ~m : clear;
                    }
                }
            }
        }
        if (shade && slow_shading(f))
            shade_tile_slow(out, f, key, gthread, kThreads, tileX, tileY, less, nr, a.tri_first, a.total_tris);
        else if (shade)
        {
#pragma unroll 1
            for (int k = 0; k < kPixels; k++)
            {
                const int p = gthread + kThreads * k;
                const int px = (tileX << 4) + (p & 15), py = (tileY << 4) + (p >> 4);
                const uint32_t low = (uint32_t)key[p];
                const uint32_t rank = less ? low : ~low;
                const uint32_t ri = raster_triangle_of(a, rank, nr);
                if (px < f.width && py < f.height)
                    write_pixel_fast(out, f, ri, f.pix_base + (uint64_t)py * (uint32_t)f.width + (uint32_t)px, px, py,
                                     rank);
            }
        }
        group_sync<Group>(group);
    }
}

// -------------------------------------------------------------------------
// Multisampling (Renderer::SetMSAAMode, Renderer.cpp:94-98).
//
// FrameBuffer::MultiSampleOffsets (FrameBuffer.cpp:107-191): the reference's
// table of 1/16-pixel sample offsets per sample-count log2.  Its rasterizer
// reads sample s as `const Vector2i& sampleOffset = MultiSampleOffsets[level]
// [2 * s]` (Rasterizer.h:247, 382): the int goes through Vector2i's scalar
// constructor, so the sample sits at (o, o) with o = table[level][2 s].
constexpr int kSampleOffsets[kMaxMsaaLog2 + 1][64] = {
    { 0, 0 },
    { 4, 4, -4, -4 },
    { -2, -6, 6, -2, -6, 2, 2, 6 },
    { 1, -3, -1, 3, 5, 1, -3, -5, -5, 5, -7, -1, 3, 7, 7, -7 },
    { 1, 1, -1, -3, -3, 2, 4, -1, -5, -2, 2, 5, 5, 3, 3, -5,
      -2, 6, 0, -7, -4, -6, -6, 4, -8, 0, 7, -4, 6, 7, -7, -8 },
    { 1, 1, -1, -3, -3, 2, 4, -1, -5, -2, 2, 5, 5, 3, 3, -5,
      -2, 6, 0, -7, -4, -6, -6, 4, -8, 0, 7, -4, 6, 7, -7, -8,
      1, 3, -3, -3, -3, 0, 6, -2, -7, -1, 3, 4, 7, 3, 3, -6,
      -2, 7, 0, -4, -2, -5, -7, 6, -8, 3, 4, -1, 2, 7, 4, -8 }
};

// The offsets of samples 16 * half .. of a level, 4 bits each (offset + 8):
// an immediate where the sample loop is unrolled, two shifts where it is not,
// instead of a constant-memory load per sample.
constexpr unsigned long long sample_pack(int level, int half)
{
    unsigned long long bits = 0;
    for (int s = 0; s < 16 && 16 * half + s < (1 << level); s++)
        bits |= (unsigned long long)(kSampleOffsets[level][2 * (16 * half + s)] + 8) << (4 * s);
    return bits;
}
constexpr int log2_of(int S) { return S <= 1 ? 0 : 1 + log2_of(S / 2); }

template <int S>
struct SamplePack
{
    static constexpr unsigned long long lo = sample_pack(log2_of(S), 0), hi = sample_pack(log2_of(S), 1);
};

template <int S>
__device__ __forceinline__ int sample_offset(int s)
{
    return (int)(((s < 16 ? SamplePack<S>::lo : SamplePack<S>::hi) >> (4 * (s & 15))) & 15u) - 8;
}

// A staged entry with several samples: the fields of StagedTri, the change G
// of each edge per 1/16 pixel along the diagonal the samples sit on, and Q,
// the edge constants raised to the largest value any sample of a pixel can
// see.  112 bytes: 16-byte loads of eight consecutive entries hit eight
// different bank groups.
struct __align__(16) StagedMs
{
    int A0, D0, Q0, A1;
    int D1, Q1, A2, D2;
    int Q2;
    uint32_t flags, rank;
    int K0;
    int K1, K2, G0, G1;
    int G2;
    float invDet, z0, z1;
    float z2;
    uint32_t pad[7];
};
static_assert(sizeof(StagedMs) == 112, "odd multiple of 16 bytes");

// Can any sample of pixel (lx, ly) be covered?  (Always, flag bit 23, where
// the entry is accepted whole or its edge values can wrap.)
__device__ __forceinline__ bool pixel_possible(const StagedMs& st, int lx, int ly)
{
    const int q0 = wadd(wadd(wmul(st.A0, lx), wmul(st.D0, ly)), st.Q0);
    const int q1 = wadd(wadd(wmul(st.A1, lx), wmul(st.D1, ly)), st.Q1);
    const int q2 = wadd(wadd(wmul(st.A2, lx), wmul(st.D2, ly)), st.Q2);
    return (st.flags & (1u << 23)) || (q0 | q1 | q2) >= 0;
}

// Float -> 8 bits as Color4b::FromFloats: clamp, scale by 255, round half up.
__device__ __forceinline__ uint32_t to_byte(float v)
{
    v = fminf(fmaxf(v, 0.0f), 1.0f);
    return (uint32_t)fadd(fmul(v, 255.0f), 0.5f);
}


// The output of one pixel with S samples: per sample the winner's id and its
// depth at the sample; the colour is the reference's resolve
// (FrameBuffer::Resolve, FrameBuffer.cpp:70-87): each sample stores its
// winner's colour shaded at the pixel centre as 8 bits (Renderer.cpp:
// 295-350), the samples are averaged in float (alpha 1 per covered sample,
// 0 for the clear value).
// The pixel's keys (key[s * 256], shared memory) are worked off winner by
// winner: the first open sample's winner is shaded, then every sample it wins
// is written and its 8-bit colour left in the key's low word for the average
// in sample order.  A warp so runs the shading once per distinct winner of
// its busiest pixel (one to three) instead of once per sample at which any of
// its pixels changes winner: 8 samples of the sphere at 1280x720, 94 -> 72 us.
// The depth comes out of the key.  Common: the per-vertex-attribute shaders,
// inline (no call); otherwise shade_fragment (the reference and textured shaders
// out of line).
template <int S, bool Common>
static __device__ __forceinline__ void write_pixel_ms(const PassArgs& a, const FrameDesc& f,
                                                   unsigned long long* key, bool less, uint32_t nr,
                                                   uint64_t pix, int px, int py)
{
    const uint64_t plane = a.total_pixels;
    uint32_t* low_words = reinterpret_cast<uint32_t*>(key);  // sample s: words 512 s (rank term), 512 s + 1 (depth)
    uint32_t todo = S == 32 ? 0xFFFFFFFFu : (1u << (S & 31)) - 1u, covered = 0;
    while (todo)
    {
        // the next sample's winner, shaded once for every sample it wins
        const uint32_t low = low_words[512 * (__ffs(todo) - 1)];
        const uint32_t rank = less ? low : ~low;
        const uint32_t ri = raster_triangle_of(a, rank, nr);
        uint32_t id = kNoTriangle, rgb = 0;
        if (ri != kNoTriangle)
        {
            // the rank names the input triangle: its indices load beside its record
            id = ((rank - 1u) >> 4) - f.tri_base;
            uint32_t vi[3];
            if (Common)
            {
                const uint32_t* idx = f.indices + 3 * (size_t)id;
                vi[0] = __ldg(idx); vi[1] = __ldg(idx + 1); vi[2] = __ldg(idx + 2);
            }
            const RTri t = load_rtri(a.rtris + ri);
            float L0, L1;
            depth_at(t, (px << 4) + 8, (py << 4) + 8, L0, L1);
            const float3 c = Common ? shade_common(f, t, a.polys, L0, L1, vi)
                                    : shade_fragment(f, t, a.rtris + ri, a.polys, L0, L1, px, py);
            rgb = to_byte(c.x) | (to_byte(c.y) << 8) | (to_byte(c.z) << 16);
        }
#pragma unroll (S <= 8 ? S : 4)
        for (int s = 0; s < S; s++)
        {
            if (!((todo >> s) & 1u) || low_words[512 * s] != low)
                continue;
            todo &= ~(1u << s);
            float d = 1.0f;
            if (ri != kNoTriangle)
            {
                covered |= 1u << s;
                low_words[512 * s] = rgb;
                d = key_depth(low_words[512 * s + 1]);
                if (d == 0.0f)
                {
                    // the key does not keep the sign of a zero
                    const int o = sample_offset<S>(s);
                    float L0, L1;
                    d = depth_at(a.rtris[ri], (px << 4) + 8 + o, (py << 4) + 8 + o, L0, L1);
                }
            }
            a.depth[s * plane + pix] = d;
            a.tri_id[s * plane + pix] = id;
        }
    }
    // the samples' 8-bit colours, averaged in sample order
    float acc[3] = { 0.f, 0.f, 0.f }, cf[3] = { 0.f, 0.f, 0.f };
    uint32_t last = 0;
#pragma unroll 1
    for (uint32_t m = covered; m; m &= m - 1u)
    {
        const uint32_t rgb = low_words[512 * (__ffs(m) - 1)];
        if (rgb != last)
        {
            last = rgb;
#pragma unroll
            for (int q = 0; q < 3; q++)
                cf[q] = fdiv((float)((rgb >> (8 * q)) & 255u), 255.0f);
        }
#pragma unroll
        for (int q = 0; q < 3; q++)
            acc[q] = fadd(acc[q], cf[q]);
    }
    const float inv = fdiv(1.0f, (float)S);
    a.color[pix] = make_float4(fmul(acc[0], inv), fmul(acc[1], inv), fmul(acc[2], inv),
                               fmul((float)__popc(covered), inv));
}

// A multisampled tile shaded by the reference or the textured shader: out of line,
// so that the common shaders' loop keeps its registers.  (`a` is the
// kernel's grid-constant parameter: passed by address, it is not copied.)
template <int S>
static __device__ __noinline__ void shade_tile_ms_slow(const PassArgs& a, const FrameDesc& f,
                                                       unsigned long long* key, int first, int step, int tileX,
                                                       int tileY, bool less, uint32_t nr)
{
#pragma unroll 1
    for (int p = first; p < 256; p += step)
    {
        const int px = (tileX << 4) + (p & 15), py = (tileY << 4) + (p >> 4);
        if (px >= f.width || py >= f.height)
            continue;
        write_pixel_ms<S, false>(a, f, key + p, less, nr, f.pix_base + (uint64_t)py * (uint32_t)f.width + (uint32_t)px,
                                 px, py);
    }
}

// The background of a tile with S samples, written by `threads` threads.
template <int S>
static __device__ __forceinline__ void clear_tile_ms(const PassArgs& a, const FrameDesc& f, uint32_t tile, int thread,
                                                     int threads)
{
    const uint32_t lt = tile - f.tile_base;
    const int tileX = (int)(lt % (uint32_t)f.tdx), tileY = (int)(lt / (uint32_t)f.tdx);
    const int w = f.width, h = f.height;
    const uint64_t base = f.pix_base, plane = a.total_pixels;
    for (int p = thread; p < 256; p += threads)
    {
        const int px = (tileX << 4) + (p & 15), py = (tileY << 4) + (p >> 4);
        if (px >= w || py >= h)
            continue;
        const uint64_t pix = base + (uint64_t)py * (uint32_t)w + (uint32_t)px;
        a.color[pix] = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
        for (int s = 0; s < S; s++)
        {
            a.depth[s * plane + pix] = 1.0f;
            a.tri_id[s * plane + pix] = kNoTriangle;
        }
    }
}

// Raster with S samples per pixel: persistent blocks on the same work items as
// k_raster.  A block's W warps share one tile and its keys [sample][pixel] in
// dynamic shared memory: with a tile per warp the keys (2 KiB per sample) left
// room for 12 warps per SM at 8 samples and 3 at 32, and a tile's chain of
// dependent loads and tests ran on one warp (7.8 % of the warps active on the
// sphere at 8 samples).  Each warp stages its own chunks of 32 entries; their
// (entry, pixel) pairs are spread over the lanes, the pixels where no sample
// can be covered are dropped by one conservative test, and the rest are queued
// and take the S samples 32 pixels at a time.  Entries behind the tile's
// samples are skipped.  Split tiles merge per sample in the key buffer (S
// planes).
// Raster and shading, a warp per tile -> a block per tile: terrain of 2,097,152
// triangles at 1920x1080, 4 samples 350-364 -> 270 us, 8 samples 702 -> 373;
// sphere at 1280x720, 4 samples 88 -> 55, 8 samples 139 -> 72; 512x512-quad
// terrain at 1280x720, 16 samples 1104 -> 317, 32 samples 3146 -> 717.
// With the pixel queue, even shares and one shading per winner: terrain 4 samples
// 222, sphere 8 samples 49, the 16 and 32 samples 235 and 513.
// W and the blocks per SM (registers a thread): 4 warps at 8 blocks (64, some
// spilled) against 5 (96, none) measured 270 and 313 us on the terrain at 4
// samples, 55 and 51 on the sphere; 2 warps 291 and 59, 8 warps 350 and 61.
// The shared memory (ms_smem) admits all 8 blocks up to 4 samples, 7 at 8
// samples, 3 at 16 and 2 at 32: there 8 warps each.  The register caps are not
// fitted to that (ms_blocks asks for 8 at 8 samples and 3 at 32).
constexpr int kMsWarpBytes = 32 * (int)sizeof(StagedMs) + 64 * 2;

__host__ __device__ constexpr int ms_warps(int S) { return S <= 8 ? 4 : 8; }
__host__ __device__ constexpr int ms_blocks(int S) { return S <= 8 ? 8 : 3; }

template <int S>
__global__ void __launch_bounds__(32 * ms_warps(S), ms_blocks(S)) k_raster_ms(const __grid_constant__ PassArgs a)
{
    follow_on();
    constexpr int W = ms_warps(S);
    constexpr int kThreads = 32 * W;
    extern __shared__ unsigned long long ms_shared[];
    __shared__ uint32_t s_next, s_done, s_bound[W];
    report_status(a);
    if (*(volatile uint32_t*)&a.status->error)
        return;  // the pass failed (see k_bin_move); every thread of the block leaves
    // ceil(65536 / w): ((p * s_recip[w]) >> 16) == p / w for 0 <= p < 256
    // and 1 <= w <= 16, the row of pixel p of a region w pixels wide
    __shared__ uint32_t s_recip[17];
    // (several samples: one frame, its descriptor as in k_raster)
    __shared__ FrameDesc s_frame;
    copy_frame(s_frame, a.frames, threadIdx.x, kThreads);
    const FrameDesc& f = s_frame;
    if (threadIdx.x >= 1 && threadIdx.x <= 16)
        s_recip[threadIdx.x] = (65536u + threadIdx.x - 1u) / threadIdx.x;
    __syncthreads();
    const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const uint32_t before = (1u << lane) - 1u;  // lanes before this one
    unsigned long long* key = ms_shared;
    unsigned char* mine = reinterpret_cast<unsigned char*>(ms_shared + 256 * S) + warp * kMsWarpBytes;
    StagedMs* staged = reinterpret_cast<StagedMs*>(mine);
    uint16_t* queue = reinterpret_cast<uint16_t*>(mine + 32 * sizeof(StagedMs));  // up to 63 pixels
    // raster-triangle slots in use: one per input triangle, then the fan pieces
    const uint32_t nr = (uint32_t)min((uint64_t)a.total_tris + *(volatile uint32_t*)&a.counters[0],
                                      (uint64_t)a.rtri_capacity);
    const uint32_t nheavy = *(volatile uint32_t*)&a.counters[6];
    const uint32_t nitems = (uint32_t)min((uint64_t)nheavy + *(volatile uint32_t*)&a.counters[7], a.item_capacity);
    const uint64_t plane = a.total_pixels;
    const uint32_t nempty = *(volatile uint32_t*)&a.counters[9];
    const bool dense = S <= 4 && *(volatile uint32_t*)&a.counters[10] != 0;
    const uint32_t bulk = min(8u, max(1u, nempty / gridDim.x));
    const uint32_t nwork = nitems + (nempty + bulk - 1) / bulk;
    // the items, then the tiles without an entry, as in k_raster
    auto next_item = [&]() -> uint32_t {
        if (gridDim.x >= nwork)
            return nwork;
        if (threadIdx.x == 0)
            s_next = gridDim.x + atomicAdd(&a.counters[3], 1u);
        __syncthreads();
        return s_next;
    };
    // each block's first item is its own (the heaviest ones, no claim), the
    // rest are claimed one at a time
    for (uint32_t q = blockIdx.x; q < nwork; q = next_item())
    {
        if (q >= nitems)
        {
            const uint32_t i0 = (q - nitems) * bulk, i1 = min(nempty, i0 + bulk);
            for (uint32_t i = i0; i < i1; i++)
                clear_tile_ms<S>(a, f, a.empty_tiles[i], (int)threadIdx.x, kThreads);
            __syncthreads();
            continue;
        }
        const uint4 item = a.items[q < nheavy ? q : (uint32_t)(a.item_capacity - 1 - (q - nheavy))];
        const uint32_t tile = item.x & ~kSplitTile;
        const uint32_t lt = tile - f.tile_base;
        const int tileX = (int)(lt % (uint32_t)f.tdx), tileY = (int)(lt / (uint32_t)f.tdx);
        const bool less = f.depth_func == 1;
        // (a frame whose entries overflowed has empty items: rendered again by the host)
        bool split = (item.x & kSplitTile) != 0;
        // the item's range within the entries its bin kept (the scatter drops
        // entries hidden behind the tile's occluder)
        uint32_t e0 = item.y, e1 = item.z, kept = 0;
        if (e0 != e1)
        {
            const uint32_t bin0 = item.w;
            kept = a.tile_cursor[tile];
            e1 = min(e1, bin0 + kept);
            e0 = min(e0, e1);
            if (split && e0 == e1)
            {
                if (item.y != bin0 || kept != 0)
                {
                    __syncthreads();
                    continue;  // the tile's kept entries are in its other items
                }
                split = false;  // it kept none: its first item writes the background
            }
        }
        if (e0 == e1 && !split)
        {
            // every entry was hidden behind the clear depth: the background, with no key
            clear_tile_ms<S>(a, f, tile, (int)threadIdx.x, kThreads);
            __syncthreads();
            continue;
        }
        const unsigned long long clear = ((unsigned long long)0xBF800000u << 32) | (less ? 0u : 0xFFFFFFFFu);
        for (int k = (int)threadIdx.x; k < 256 * S; k += kThreads)
            key[k] = clear;
        if (lane == 0)
            s_bound[warp] = 0xFFFFFFFFu;
        __syncthreads();

        // depth bound of the tile: the nearest triangle that covers it whole
        // (every sample), then the largest depth key of its samples so far
        const uint32_t tzocc = min(0xBF800000u, a.tile_zocc[tile]);
        uint32_t tzmax = tzocc;
        // one queued pixel: entry << 8 | pixel of the tile, its samples tested
        auto test_samples = [&](uint32_t e) {
            const StagedMs& st = staged[e >> 8];
            const int p = (int)(e & 255u), x = p & 15, y = p >> 4;
            const uint32_t fl = st.flags;
            const int c0 = wadd(wadd(wmul(st.A0, x), wmul(st.D0, y)), st.K0);
            const int c1 = wadd(wadd(wmul(st.A1, x), wmul(st.D1, y)), st.K1);
            const int c2 = wadd(wadd(wmul(st.A2, x), wmul(st.D2, y)), st.K2);
            const int b1 = (fl & (1u << 21)) ? -1 : 0, b2 = (fl & (1u << 22)) ? -1 : 0;
            const bool accept = (fl & (1u << 20)) != 0;
            const uint32_t rank = less ? st.rank : ~st.rank;
            const int G0 = st.G0, G1 = st.G1, G2 = st.G2;
            const float invDet = st.invDet, z0 = st.z0, z1 = st.z1, z2 = st.z2;
#pragma unroll (S <= 8 ? S : 8)
            for (int s = 0; s < S; s++)
            {
                // FineRasterize_MultiSample / TrivialAcceptTriangle_MultiSample
                // (Rasterizer.h:202-300, 355-415): the biased pixel-centre
                // edge values plus o * G decide coverage (accepted entries
                // skip the test), the barycentrics and depth come from the
                // unbiased values at the sample
                const int o = sample_offset<S>(s);
                const int e0 = wadd(c0, wmul(o, G0)), l1 = wadd(c1, wmul(o, G1)), l2 = wadd(c2, wmul(o, G2));
                const bool inside = accept || (e0 | wadd(l1, b1) | wadd(l2, b2)) >= 0;
                const float L0 = fmul(__int2float_rn(l1), invDet);
                const float L1 = fmul(__int2float_rn(l2), invDet);
                const float L2 = fsub(fsub(1.0f, L0), L1);
                const float d = fadd(fadd(fmul(L0, z0), fmul(L1, z1)), fmul(L2, z2));
                const unsigned long long k = ((uint64_t)depth_key(d) << 32) | rank;
                unsigned long long* slot = &key[s * 256 + p];
                const unsigned long long cur = *slot;
                if (inside && d == d && k < cur)
                    atomicMin(slot, k);
            }
        };
        // entries a warp stages at a time: 32, fewer where all W would not get
        // some (100,000 stress triangles at 1920x1080, a handful of large ones
        // a tile: 8 samples 447 -> 326 us, 4 samples 296 -> 224).  Of a dense
        // frame's hundreds of entries a tile most lie behind the others: 16 at
        // a time, so that the tile's bound is taken twice as often (4 samples,
        // 100,000 stress triangles at 300x200 431 -> 336 us a frame, 215,347 at
        // 216x129 656 -> 541, 845,117 at 271x229 1435 -> 1286; the
        // 1024x1024-quad terrain at 320x180 185 -> 197)
        const uint32_t per = even_chunk(e1 - e0, (uint32_t)W, dense ? 16u : 32u);
        for (uint32_t c = e0 + per * warp; c < e1; c += per * (uint32_t)W)
        {
            const uint32_t m = min(per, e1 - c);
            int area = 0;
            StagedTri st;
            int G[3];
            bool wfree = false;
            if (lane < m)
            {
                uint32_t zk;
                stage_tri<true>(a, a.bins[c + lane], nr, f.tri_base << 4, tileX, tileY, st, zk, G, &wfree);
                const uint32_t fl = st.flags;
                const int rx0 = fl & 31, rx1 = (fl >> 5) & 31, ry0 = (fl >> 10) & 31, ry1 = (fl >> 15) & 31;
                if (zk <= tzmax && rx0 <= rx1 && ry0 <= ry1)
                    area = (rx1 - rx0 + 1) * (ry1 - ry0 + 1);
            }
            const uint32_t live = __ballot_sync(0xffffffffu, area > 0);
            if (area > 0)
            {
                StagedMs& t = staged[__popc(live & before)];
                t.A0 = st.A0; t.D0 = st.D0; t.A1 = st.A1; t.D1 = st.D1; t.A2 = st.A2; t.D2 = st.D2;
                t.K0 = st.K0; t.K1 = st.K1; t.K2 = st.K2;
                t.G0 = G[0]; t.G1 = G[1]; t.G2 = G[2];
                // the largest o * G over the offsets [-8, 7] of any sample table
                t.Q0 = wadd(st.K0, G[0] > 0 ? wmul(7, G[0]) : wmul(-8, G[0]));
                t.Q1 = wadd(st.K1, G[1] > 0 ? wmul(7, G[1]) : wmul(-8, G[1]));
                t.Q2 = wadd(st.K2, G[2] > 0 ? wmul(7, G[2]) : wmul(-8, G[2]));
                t.flags = st.flags | ((st.flags & (1u << 20)) || !wfree ? (1u << 23) : 0u);
                t.rank = st.rank;
                t.invDet = st.invDet; t.z0 = st.z0; t.z1 = st.z1; t.z2 = st.z2;
            }
            // (entry, pixel) pairs numbered across the warp and taken 32 at a
            // time (as in k_raster), so lanes do not idle on entries of a few
            // pixels; pixels with a sample that may be covered are queued
            // and, 32 at a time again, their S samples tested
            int incl = area;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1)
            {
                const int v = __shfl_up_sync(0xffffffffu, incl, o);
                if (lane >= (uint32_t)o) incl += v;
            }
            const int pairs = __shfl_sync(0xffffffffu, incl, 31);
            __syncwarp();
            int queued = 0, started = -1, carry = 0;
            for (int base = 0; base < pairs; base += 32)
            {
                const uint32_t begin = (uint32_t)(incl - area - base);
                const uint32_t heads = __reduce_or_sync(0xffffffffu, area > 0 && begin < 32u ? 1u << begin : 0u);
                const uint32_t upto = heads & (before | (1u << lane));
                const int j = started + __popc(upto);
                const int local = upto ? (int)lane - (31 - __clz(upto)) : carry + (int)lane;
                started += __popc(heads);
                carry = heads ? 32 - (31 - __clz(heads)) : carry + 32;
                bool keep = false;
                uint32_t e = 0;
                if (base + (int)lane < pairs)
                {
                    const StagedMs& st = staged[j];
                    const uint32_t fl = st.flags;
                    const int rx0 = fl & 31, rx1 = (fl >> 5) & 31, ry0 = (fl >> 10) & 31;
                    const int rw = rx1 - rx0 + 1;
                    const int dy = (int)(((uint32_t)local * s_recip[rw]) >> 16);
                    const int x = rx0 + local - dy * rw, y = ry0 + dy;
                    e = ((uint32_t)j << 8) | (uint32_t)(y * 16 + x);
                    keep = pixel_possible(st, x, y);
                }
                if (S == 2)
                {
                    // (two samples cost about what queueing does)
                    if (keep)
                        test_samples(e);
                    continue;
                }
                const uint32_t kept_lanes = __ballot_sync(0xffffffffu, keep);
                if (keep)
                    queue[queued + __popc(kept_lanes & before)] = (uint16_t)e;
                queued += __popc(kept_lanes);
                __syncwarp();
                if (queued >= 32)
                {
                    queued -= 32;
                    test_samples(queue[queued + lane]);
                    __syncwarp();
                }
            }
            if ((int)lane < queued)
                test_samples(queue[lane]);
            __syncwarp();
            if (c + per * (uint32_t)W < e1)
            {
                // each warp takes the bound of its share of the keys again
                // and combines it with the others' last ones (keys only fall:
                // an old bound is a valid, larger one)
                uint32_t mz = 0;
                for (int k = (int)threadIdx.x; k < 256 * S; k += kThreads)
                    mz = max(mz, (uint32_t)(key[k] >> 32));
                mz = __reduce_max_sync(0xffffffffu, mz);
                if (lane == 0)
                    *(volatile uint32_t*)&s_bound[warp] = mz;
                __syncwarp();
#pragma unroll
                for (int w = 0; w < W; w++)
                    mz = max(mz, *(volatile uint32_t*)&s_bound[w]);
                tzmax = min(tzocc, mz);
            }
        }
        __syncthreads();

        bool shade = true;
        if (split)
        {
            for (int k = (int)threadIdx.x; k < 256 * S; k += kThreads)
            {
                const int s = k >> 8, p = k & 255;
                const int px = (tileX << 4) + (p & 15), py = (tileY << 4) + (p >> 4);
                const unsigned long long kk = key[k];
                if (px < f.width && py < f.height && kk < clear)
                    atomicMax(&a.keybuf[s * plane + f.pix_base + (uint64_t)py * (uint32_t)f.width + (uint32_t)px], ~kk);
            }
            // acquire-release count, as in k_raster
            __syncthreads();
            if (threadIdx.x == 0)
                s_done = atomic_add_acq_rel(&a.tile_count[tile], e1 - e0) + (e1 - e0);
            __syncthreads();
            shade = *(volatile uint32_t*)&s_done == kept;
            if (shade)
            {
                for (int k = (int)threadIdx.x; k < 256 * S; k += kThreads)
                {
                    const int s = k >> 8, p = k & 255;
                    const int px = (tileX << 4) + (p & 15), py = (tileY << 4) + (p >> 4);
                    if (px < f.width && py < f.height)
                    {
                        const unsigned long long m = atomicExch(
                            &a.keybuf[s * plane + f.pix_base + (uint64_t)py * (uint32_t)f.width + (uint32_t)px], 0ull);
                        key[k] = m ? ~m : clear;
                    }
                }
                __syncthreads();
            }
        }
        if (shade && slow_shading(f))
            shade_tile_ms_slow<S>(a, f, key, (int)threadIdx.x, kThreads, tileX, tileY, less, nr);
        else if (shade)
        {
#pragma unroll 1
            for (int p = (int)threadIdx.x; p < 256; p += kThreads)
            {
                const int px = (tileX << 4) + (p & 15), py = (tileY << 4) + (p >> 4);
                if (px >= f.width || py >= f.height)
                    continue;
                write_pixel_ms<S, true>(a, f, key + p, less, nr,
                                        f.pix_base + (uint64_t)py * (uint32_t)f.width + (uint32_t)px, px, py);
            }
        }
        __syncthreads();
    }
}

static size_t ms_smem(int S) { return (size_t)256 * S * sizeof(unsigned long long) + (size_t)ms_warps(S) * kMsWarpBytes; }

// -------------------------------------------------------------------------
// Renderer::GetBackBuffer compatibility: RGBA8, bottom-up (FrameBuffer.cpp:41).
__global__ void k_back_buffer(const float4* color, uchar4* out, int width, int height)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= width * height)
        return;
    const int x = i % width, y = i / width;
    const float4 c = color[i];
    // Color4b::FromFloats for one sample (alpha 1 or 0), Color4b(Color) of
    // the resolve with several (alpha = covered share)
    out[(size_t)(height - 1 - y) * width + x] =
        make_uchar4(to_byte(c.x), to_byte(c.y), to_byte(c.z), to_byte(c.w));
}

// -------------------------------------------------------------------------

// Resident blocks per SM of k_raster<Group>.
template <int Group>
static int raster_occupancy()
{
    static int per_sm = 0;
    if (!per_sm)
    {
        int n = 0;
        if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, k_raster<Group, false>, kRasterThreads, 0) != cudaSuccess || n < 1)
            n = 1;
        per_sm = n;
    }
    return per_sm;
}

// Launches a kernel of the pass; `follows`: right behind the pass's previous
// kernel (see follow_on).
template <typename Kernel>
static cudaError_t launch(Kernel kernel, unsigned blocks, unsigned threads, size_t smem, cudaStream_t s, bool follows,
                          const PassArgs& a)
{
    cudaLaunchConfig_t c = {};
    c.gridDim = dim3(blocks);
    c.blockDim = dim3(threads);
    c.dynamicSmemBytes = smem;
    c.stream = s;
    cudaLaunchAttribute at;
    at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at.val.programmaticStreamSerializationAllowed = 1;
    c.attrs = &at;
    c.numAttrs = follows ? 1 : 0;
    return cudaLaunchKernelEx(&c, kernel, a);
}

template <int Group>
static cudaError_t launch_raster(int sms, const PassArgs& a, cudaStream_t s, bool follows)
{
    int per = raster_occupancy<Group>();
    if (a.tune.raster_blocks_per_sm > 0 && a.tune.raster_blocks_per_sm < per)
        per = a.tune.raster_blocks_per_sm;
    return launch((a.num_frames == 1 ? k_raster<Group, true> : k_raster<Group, false>), (unsigned)(sms * per), kRasterThreads, 0, s, follows, a);
}

// Warps per raster item.  A warp alone takes 10 to 25 us for a tile (a chain
// of dependent loads, then eight rounds of shading), so a frame with fewer
// tiles than resident warps (24 per SM) leaves most of the chip idle for that
// long; more warps per tile shorten it.  Against it stand the barriers and that
// every warp looks at every large region, so frames with several tiles per
// warp keep one.  Raster stage with 1 / 2 / 4 / 8 warps, us:
//   sphere (4,032 triangles) 320x180, 240 tiles      28.0 / 18.4 / 16.4 / 16.0
//   96x96-quad terrain 480x270, 510 tiles            42.0 / 30.7 / 23.6 / 20.5
//   10,000 stress triangles 480x270                  56.3 / 46.1 / 31.8 / 33.1
//   128x128-quad terrain 640x400, 1,000 tiles        41.0 / 30.4 / 25.6 / 23.6
//   sphere 1280x720, 3,600 tiles                     23.6 / 24.2 / 19.1 / 20.1
//   256x256-quad terrain 1280x720, textured          69.3 / 61.1 / 56.3 / 63.5
//   301x301-quad terrain 1366x769, 4,214 tiles       53.6 / 46.8 / 45.1 / 56.0
//   100,000 stress triangles 1600x900, 5,700 tiles   64.2 / 71.7 / 73.7 / 96.6
//   512x512-quad terrain 1760x990, 6,820 tiles       67.9 / 68.6 / 69.3 / 87.1
//   sphere (16,256 triangles) 1920x1080, 8,160 tiles 31.1 / 26.6 / 26.6 / 32.8
//   terrain (2,097,152 triangles) 1920x1080          93.9 / 102  / 103  / 123
// Two warps are best nowhere; above 30 tiles per SM four pay only where the
// triangles are few, so that most tiles have a handful of large regions or none.
static int raster_group(const PassArgs& a, int sms)
{
    const uint64_t tiles = a.total_tiles, n = (uint64_t)sms;
    if (a.tune.raster_variant == 0)
        return 1;
    if (8 * tiles <= 27 * n)
        return 8;
    return tiles <= 30 * n || (tiles <= 60 * n && a.total_tris <= 120 * n) ? 4 : 1;
}

// Several warps rasterize an item's large regions together, each its own
// pixels, so every warp looks at every one: where a tile has hundreds of
// entries, most of them large, single warps are faster (raster stage,
// several / one warp per item: 111,605 stress triangles at 427x394, 891 entries
// a tile, 138 / 92 us; 30,000 at 320x180, 2,690 a tile, 66 / 53; but 10,000
// there, 896 a tile, 51 / 49; the 1024x1024-quad terrain at 320x180, 543 a tile,
// 27 / 40).  The entries are known after binning, so where the triangles allow
// that many both kernels are launched, the scan decides and the other one
// returns at once (1 us).
static bool by_density(const PassArgs& a, int sms)
{
    return a.msaa_log2 == 0 && a.total_tris >= 64ull * a.total_tiles && raster_group(a, sms) > 1;
}

// Resident blocks per SM of k_raster_ms with 2^level samples (the dynamic
// shared-memory limit raised first).
template <int S>
static int ms_occupancy_of()
{
    int n = 0;
    if (cudaFuncSetAttribute(k_raster_ms<S>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)ms_smem(S)) !=
            cudaSuccess ||
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, k_raster_ms<S>, 32 * ms_warps(S), ms_smem(S)) !=
            cudaSuccess ||
        n < 1)
        n = 1;
    return n;
}

static int ms_occupancy(int level)
{
    static int per_sm[kMaxMsaaLog2 + 1] = {};
    if (!per_sm[level])
    {
        switch (level)
        {
        case 1: per_sm[1] = ms_occupancy_of<2>(); break;
        case 2: per_sm[2] = ms_occupancy_of<4>(); break;
        case 3: per_sm[3] = ms_occupancy_of<8>(); break;
        case 4: per_sm[4] = ms_occupancy_of<16>(); break;
        default: per_sm[5] = ms_occupancy_of<32>(); break;
        }
    }
    return per_sm[level];
}

void prepare_kernels()
{
    raster_occupancy<1>();
    raster_occupancy<4>();
    raster_occupancy<8>();
    for (int level = 1; level <= kMaxMsaaLog2; level++)
        ms_occupancy(level);
}

Tuning default_tuning()
{
    Tuning t;
    t.small_region = 32;
    t.raster_variant = 1;
    t.bin_blocks_per_sm = 8;
    t.raster_blocks_per_sm = 0;
    t.item_entries = (int)kItemEntries;
    t.scan_stall_block = -1;
    t.scan_spin_limit = 0;
    return t;
}

cudaError_t launch_pipeline(const PassArgs& pass, cudaStream_t s, cudaEvent_t* ev)
{
    PassArgs a = pass;
    const int sms = a.num_sms > 0 ? a.num_sms : 148;
    // With several samples a block of warps shares an item, so an item takes
    // more entries (twice, four times with 8 warps): 4 samples of the terrain
    // 309 -> 303 us, 16 samples 381 -> 317.
    if (a.msaa_log2 > 0)
    {
        a.tune.item_entries = min(1024, a.tune.item_entries * (a.msaa_log2 <= 3 ? 2 : 4));
        // (the items stay; k_raster_ms takes smaller chunks of a dense frame's)
        if (a.msaa_log2 <= 2)
            a.dense_entries = (uint32_t)a.tune.item_entries;
    }
    else
    {
        // Several warps share an item; and with many small frames, four tiles
        // and more per warp, the last items are a small part of the pass, so
        // fewer tiles need splitting (raster stage, 128 / 256 entries: 256
        // views at 512x512 722 / 709 us, 64 views of a torus at 256x256 122 /
        // 113, 90 views at 300x200 96 / 92; 12 views there 25 / 30; the frames
        // of one mesh, terrain 92 / 103, binning stress 200 / 203).
        const bool many = a.num_frames > 1 && (uint64_t)a.total_tiles >= 96ull * (uint64_t)sms;
        if (by_density(a, sms))
            a.dense_entries = (uint32_t)a.tune.item_entries;
        a.tune.item_entries = min(1024, a.tune.item_entries * (many ? 2 : raster_group(a, sms)));
    }
    const uint32_t nscan = scan_blocks(a.total_tiles);
    auto mark = [&](int i) {
        if (ev) cudaEventRecord(ev[i], s);
    };
    cudaError_t e = cudaSuccess;
    // (stage events between the kernels keep them apart)
    bool follows = false;
    auto go = [&](auto kernel, uint64_t blocks, unsigned threads, size_t smem) {
        if (e == cudaSuccess)
            e = launch(kernel, (unsigned)blocks, threads, smem, s, follows, a);
        follows = !ev;
    };
    if (a.frames_host)
        e = cudaMemcpyAsync(const_cast<FrameDesc*>(a.frames), a.frames_host, sizeof(FrameDesc) * a.num_frames,
                            cudaMemcpyHostToDevice, s);
    mark(0);
    const uint32_t clear_items = max(a.total_tiles + 1, a.vrecs ? a.total_vertices : 0u);
    go(k_clear, (clear_items + 255) / 256 + 1, 256, 0);
    mark(1);
    if (a.total_tris)
    {
        go(k_setup, (a.total_tris + kSetupThreads - 1) / kSetupThreads, kSetupThreads, 0);
        // (no more blocks than one 16-lane group per triangle fills)
        go(k_clip, min((uint32_t)sms * 8u, (a.total_tris + 7u) / 8u), kClipThreads, 0);
    }
    go(k_bin_big, sms * 4, 256, 0);
    mark(2);
    go(k_scan, nscan, kScanThreads, 0);
    mark(3);
    // (two blocks per SM at least, more by about two entries per triangle)
    const uint32_t move = (uint32_t)sms * (uint32_t)(a.tune.bin_blocks_per_sm > 0 ? a.tune.bin_blocks_per_sm : 8);
    go(k_bin_move, min(move, max((uint32_t)sms * 2u, a.total_tris / 128u)), 256, 0);
    mark(4);
    if (a.msaa_log2 > 0)
    {
        const int level = min(a.msaa_log2, kMaxMsaaLog2), S = 1 << level;
        // Not behind its predecessor's end (follow_on): blocks that become
        // resident while others still run are placed under the shared-memory
        // split those left, a few per SM, and as they stay until the work is
        // done, the rest find no room (2 samples, 48,873 stress triangles at
        // 164x125 427 -> 292 us a frame, 300,000 at 800x450 439 -> 350; terrain
        // and sphere unchanged).
        follows = false;
        const unsigned blocks = (unsigned)(sms * ms_occupancy(level)), threads = 32u * (unsigned)ms_warps(S);
        switch (level)
        {
        case 1: go(k_raster_ms<2>, blocks, threads, ms_smem(2)); break;
        case 2: go(k_raster_ms<4>, blocks, threads, ms_smem(4)); break;
        case 3: go(k_raster_ms<8>, blocks, threads, ms_smem(8)); break;
        case 4: go(k_raster_ms<16>, blocks, threads, ms_smem(16)); break;
        default: go(k_raster_ms<32>, blocks, threads, ms_smem(32)); break;
        }
    }
    else if (e == cudaSuccess)
    {
        const int group = raster_group(a, sms);
        if (a.tune.raster_variant == 2)
            a.tune.small_region = 0;
        switch (group)
        {
        case 8: e = launch_raster<8>(sms, a, s, follows); break;
        case 4: e = launch_raster<4>(sms, a, s, follows); break;
        default: e = launch_raster<1>(sms, a, s, follows); break;
        }
        if (e == cudaSuccess && a.dense_entries)
            e = launch_raster<1>(sms, a, s, follows);
    }
    mark(5);
    const cudaError_t last = cudaGetLastError();
    return e != cudaSuccess ? e : last;
}

int kernels_per_pass(const PassArgs& a)
{
    return 5 + (a.total_tris ? 2 : 0) + (by_density(a, a.num_sms > 0 ? a.num_sms : 148) ? 1 : 0);
}

__global__ void k_mip_level(const float4* src, int sw, int sh, float4* dst, int dw, int dh)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= dw * dh)
        return;
    const int x = i % dw, y = i / dw;
    const int x0 = min(2 * x, sw - 1), x1 = min(2 * x + 1, sw - 1);
    const int y0 = min(2 * y, sh - 1), y1 = min(2 * y + 1, sh - 1);
    const float4 a = src[(size_t)y0 * sw + x0], b = src[(size_t)y0 * sw + x1];
    const float4 c = src[(size_t)y1 * sw + x0], d = src[(size_t)y1 * sw + x1];
    auto avg = [](float p, float q, float r, float t) { return fmul(fadd(fadd(fadd(p, q), r), t), 0.25f); };
    dst[i] = make_float4(avg(a.x, b.x, c.x, d.x), avg(a.y, b.y, c.y, d.y), avg(a.z, b.z, c.z, d.z),
                         avg(a.w, b.w, c.w, d.w));
}

cudaError_t launch_mip_level(const float4* src, int sw, int sh, float4* dst, int dw, int dh, cudaStream_t s)
{
    const int n = dw * dh;
    k_mip_level<<<(n + 255) / 256, 256, 0, s>>>(src, sw, sh, dst, dw, dh);
    return cudaGetLastError();
}

cudaError_t launch_back_buffer(const float4* color, uint8_t* rgba8, int width, int height, cudaStream_t s)
{
    const int n = width * height;
    k_back_buffer<<<(n + 255) / 256, 256, 0, s>>>(color, reinterpret_cast<uchar4*>(rgba8), width, height);
    return cudaGetLastError();
}

}  // namespace edxr
