// kernels.cu - the per-frame stage kernels of Voxel ReSTIR on sm_103a, plus the
// one-time world kernels (uber grid, light table).
//
// Memory layout in HBM (per view):
//   G-buffer   vd[2]  uint2  (voxel | side << 24, bits(dist))   current / previous frame
//              seed   uint32 per-pixel xorshift32 state
//   reservoirs C, H   uint4 + float4 planes (see Res in device.cuh), 32 B/pixel each:
//              C = candidate+temporal output, H = spatial output = temporal history
//   frame      float4 (rgb, dist); accum float4 (running mean, the output image)
// and per batch of views (a single view holds two sets and takes the other one as each
// frame begins, so its candidate passes can run beside the previous frame's shading):
//   hits       uint32 list of (view << 27 | pixel) whose primary ray hit a voxel
//   queue      float4 x 2 per entry: shadow-ray requests (origin | entry, dir | light)
//   counters   uint32[kCounters]: list lengths and work-queue cursors (kernels.hpp)
// The reference cycles two 80-byte reservoir buffers through three roles per frame
// (world.cpp:2209-2219) and copies the shaded reservoir at the end of shading
// (ris.cl:412). Here the spatial pass writes H in place of the previous history,
// which the candidate pass has finished reading, and shading patches H on a failed
// visibility test; H is then next frame's history without any copy.
//
// Work decomposition: the reference runs one work item per pixel through each whole
// kernel, so sky pixels idle beside terrain pixels and every warp waits for its
// longest shadow ray. Here every stage is one launch over a table of views (one view,
// or a batch of up to 16 independent views with their own worlds, resolutions and
// light models): pixel stages are persistent blocks pulling screen tiles from a work queue;
// the candidate loop, the temporal step and the shading request run over a compacted
// list of hit pixels; and every shadow ray goes through one persistent tracer whose
// lanes take a new ray as soon as theirs ends and whose warps walk bricks together. Each
// pixel's arithmetic is unchanged, so results are the same bit for bit whatever order
// pixels and rays are processed in.
#include <algorithm>
#include <cstdint>
#include <map>
#include <mutex>
#include <cuda_runtime.h>

#include "device.cuh"
#include "kernels.hpp"
#include "proposal.hpp"

namespace vxr {
namespace dev {

__device__ __forceinline__ void raise_error(uint32_t* err, uint32_t code) { atomicOr(err, code); }
__global__ void clear_flags_kernel(uint32_t* err, uint32_t flags) { atomicAnd(err, ~flags); }

// The start of every kernel that launch_next may launch: waits until the kernel before it in the
// stream has ended and its writes are seen (nothing, for a kernel launched plainly).
__device__ __forceinline__ void follow_previous() { asm volatile("griddepcontrol.wait;" ::: "memory"); }

// Light centre/emission from the reference records (tools.cl:600-607, phat.cl:8-12): n records
// of WORDS words, (position, voxel, size) first.
template <int WORDS>
__global__ void build_light_table_kernel(const uint32_t* __restrict__ raw, uint32_t n, float4* geom, float4* emit) {
    follow_previous();
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const uint32_t* r = raw + (size_t)i * WORDS;
    const uint4 l = WORDS == 4 ? *reinterpret_cast<const uint4*>(r) : make_uint4(r[0], r[1], r[2], 0u);
    const uint32_t y = l.x / (1024u * 1024u), z = (l.x / 1024u) % 1024u, x = l.x % 1024u;
    const float size = (float)l.z;
    const float half = 0.5f * size;
    geom[i] = make_float4((float)x + half, (float)y + half, (float)z + half, size);
    const float3 c = to_rgb(l.y);
    const float m = strength(l.y);
    const float INVPI = 0.31830988618379067153777f;
    emit[i] = make_float4((c.x * m) * INVPI, (c.y * m) * INVPI, (c.z * m) * INVPI, __uint_as_float(l.x));
}

// Per brick the boxes of its opaque voxels (type nibble 15) and of its non-zero voxels,
// packed as World::bbox describes, and its masks of both (World::bmask, bmask0): one warp per
// brick, 16 voxels a lane, min / max reductions over the warp, a ballot per mask word.
__device__ __forceinline__ uint32_t warp_box(bool any, const uint32_t lo[3], const uint32_t hi[3]) {
    const bool anyw = __any_sync(0xffffffffu, any);
    uint32_t box = 0u;
    for (int a = 0; a < 3; a++) {
        box |= __reduce_min_sync(0xffffffffu, lo[a]) << (3 * a);
        box |= __reduce_max_sync(0xffffffffu, hi[a]) << (9 + 3 * a);
    }
    return anyw ? box : kNoOpaque;
}
// (list: the bricks to do, or null for bricks 0 .. n - 1; bmask and bmask0 may be null)
__global__ void build_brick_boxes_kernel(const uint32_t* __restrict__ bricks, const uint32_t* __restrict__ list,
                                         uint32_t n, uint32_t* __restrict__ bbox, uint32_t* __restrict__ bbox0,
                                         uint32_t* __restrict__ bmask, uint32_t* __restrict__ bmask0) {
    follow_previous();
    const size_t item = ((size_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    if (item >= n) return;   // whole warps leave together (blockDim a multiple of 32)
    const size_t brick = list ? (size_t)__ldg(list + item) : item;
    const uint32_t lane = threadIdx.x & 31u;
    uint32_t lo[3] = {7u, 7u, 7u}, hi[3] = {0u, 0u, 0u}, lo0[3] = {7u, 7u, 7u}, hi0[3] = {0u, 0u, 0u};
    bool any = false, any0 = false;
    for (uint32_t i = 0; i < 16; i++) {
        const uint32_t e = i * 32u + lane;   // coalesced: a warp reads 32 consecutive voxels
        const uint32_t v = __ldg(bricks + brick * 512u + e);
        const uint32_t c[3] = {e & 7u, (e >> 3) & 7u, e >> 6};
        const bool opaque = ((v & 0xf000u) >> 12) == 15u;
        const uint32_t word = __ballot_sync(0xffffffffu, opaque), word0 = __ballot_sync(0xffffffffu, v != 0u);
        if (bmask && lane == i) {
            bmask[brick * 16u + i] = word;
            bmask0[brick * 16u + i] = word0;
        }
        if (opaque) {
            for (int a = 0; a < 3; a++) { lo[a] = min(lo[a], c[a]); hi[a] = max(hi[a], c[a]); }
            any = true;
        }
        if (v != 0u) {
            for (int a = 0; a < 3; a++) { lo0[a] = min(lo0[a], c[a]); hi0[a] = max(hi0[a], c[a]); }
            any0 = true;
        }
    }
    const uint32_t box = warp_box(any, lo, hi), box0 = warp_box(any0, lo0, hi0);
    if (lane == 0u) {
        bbox[brick] = box;
        bbox0[brick] = box0;
    }
}

// commit (kernels.cl:448-477): staged brick i (512 voxels after the index list) to its
// place in the pool; one block of 128 threads per brick, 16 bytes a thread
__global__ void commit_bricks_kernel(const uint32_t* __restrict__ list, const uint32_t* __restrict__ voxels,
                                     uint32_t* __restrict__ bricks) {
    const uint32_t b = __ldg(list + blockIdx.x);
    const uint4 v = __ldg(reinterpret_cast<const uint4*>(voxels + (size_t)blockIdx.x * 512u) + threadIdx.x);
    reinterpret_cast<uint4*>(bricks + (size_t)b * 512u)[threadIdx.x] = v;
}

// The tables that follow from the grid and the brick boxes, two warps per uber cell, a lane
// per grid cell:
//   uber    updateUberGrid (kernels.cl:498-513): 1 when any of the 4^3 grid cells is non-empty
//   ucell   World::ucell; ucell0 World::ucell0 (with the box: brick-less non-zero cells count
//           whole, bricks with their non-zero box)
//   gbox, gbox0   World::gbox, gbox0, unless null
// bbox, bbox0 null: no brick boxes (every brick may hold anything); nbricks, err: a grid cell
// that points past nbricks bricks raises flag 16 (err null: not checked). With one thread
// per uber cell reading its 64 cells in turn this took 59 us for 107,384 bricks (and the
// uber grid 12, the cell boxes 9, each a launch); 13 us this way.
struct CellTables {
    uint8_t* uber;
    unsigned long long* ucell;
    uint4* ucell0;
    uint2 *gbox, *gbox0;
};
__global__ void __launch_bounds__(256) build_cells_kernel(const uint32_t* __restrict__ grid, const uint32_t* __restrict__ bbox,
                                                          const uint32_t* __restrict__ bbox0, const CellTables out,
                                                          uint32_t nbricks, uint32_t* err) {
    __shared__ uint32_t s_mask[8], s_mask0[8], s_lo[8][3], s_hi[8][3];
    __shared__ bool s_occ[8];
    follow_previous();
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const uint32_t u = blockIdx.x * 4u + (uint32_t)(warp >> 1);            // x + z*32 + y*1024
    const uint32_t b = (uint32_t)(warp & 1) * 32u + (uint32_t)lane;        // x + z*4 + y*16 inside it
    const uint32_t cx = b & 3u, cz = (b >> 2) & 3u, cy = b >> 4;
    const uint32_t i = ((u & 31u) * 4u + cx) + (((u >> 5) & 31u) * 4u + cz) * 128u + ((u >> 10) * 4u + cy) * 16384u;
    const uint32_t c = __ldg(grid + i);
    const bool brick = c & 1u;
    const bool bad = err && brick && (c >> 1) >= nbricks;
    if (bad) atomicOr(err, kBadGrid);
    const uint32_t box = brick && bbox && !bad ? __ldg(bbox + (c >> 1)) : 0u,
                   box0 = brick && bbox0 && !bad ? __ldg(bbox0 + (c >> 1)) : 0u;
    if (out.gbox) out.gbox[i] = make_uint2(c, box);
    if (out.gbox0) out.gbox0[i] = make_uint2(c, box0);
    const bool stops = brick ? box != kNoOpaque : (((c >> 1) & 0xf000u) >> 12) == 15u;
    const bool stops0 = c != 0u && !(brick && box0 == kNoOpaque);
    const uint32_t m = __ballot_sync(0xffffffffu, stops), m0 = __ballot_sync(0xffffffffu, stops0);
    const bool occ = __any_sync(0xffffffffu, c != 0u);
    const uint32_t at[3] = {cx * 8u, cy * 8u, cz * 8u};
    uint32_t lo[3], hi[3];
    for (int a = 0; a < 3; a++) {
        const uint32_t l = brick && bbox0 ? (box0 >> (3 * a)) & 7u : 0u, h = brick && bbox0 ? (box0 >> (9 + 3 * a)) & 7u : 7u;
        lo[a] = __reduce_min_sync(0xffffffffu, stops0 ? at[a] + l : 31u);
        hi[a] = __reduce_max_sync(0xffffffffu, stops0 ? at[a] + h : 0u);
    }
    if (lane == 0) {
        s_mask[warp] = m;
        s_mask0[warp] = m0;
        s_occ[warp] = occ;
        for (int a = 0; a < 3; a++) { s_lo[warp][a] = lo[a]; s_hi[warp][a] = hi[a]; }
    }
    __syncthreads();
    if (lane == 0 && !(warp & 1)) {
        const bool any = s_occ[warp] || s_occ[warp + 1];
        uint32_t k[2] = {s_mask[warp], s_mask[warp + 1]}, k0[2] = {s_mask0[warp], s_mask0[warp + 1]};
        uint32_t ubox = 0u;
        for (int a = 0; a < 3; a++)
            ubox |= (min(s_lo[warp][a], s_lo[warp + 1][a]) << (5 * a)) | (max(s_hi[warp][a], s_hi[warp + 1][a]) << (15 + 5 * a));
        if (!(k0[0] | k0[1])) ubox = kNoOpaque;
        if (any && !(k[0] | k[1])) k[0] = 1u;
        if (any && !(k0[0] | k0[1])) k0[0] = 1u;
        out.uber[u] = any ? 1 : 0;
        out.ucell[u] = k[0] | ((unsigned long long)k[1] << 32);
        out.ucell0[u] = make_uint4(k0[0], k0[1], ubox, 0u);
    }
}

// ---- work distribution --------------------------------------------------------------------
// VARIANT of a launch: 0 one view with area lights, 1 one view with point lights (the
// view is read from the kernel parameter), 2 a table of views in device memory, light
// model per view.
constexpr uint32_t kPixMask = (1u << 27) - 1u;

template <int VARIANT>
__device__ __forceinline__ const ViewDev* view_of(const BatchDev& bd, uint32_t v) {
    if (VARIANT < 2) return &bd.one;
    return bd.views + v;
}
// pixel of a hit-list or request entry (a single view's entries are the bare pixel index,
// so a single view may hold more than 2^27 pixels)
template <int VARIANT>
__device__ __forceinline__ uint32_t pix_of(uint32_t e) {
    return VARIANT < 2 ? e : (e & kPixMask);
}
template <int VARIANT>
__device__ __forceinline__ bool point_of(const ViewDev* V) {
    return VARIANT == 1 || (VARIANT == 2 && V->point);
}

// warp-aggregated append to a list: one atomic per group of lanes that call it together
__device__ __forceinline__ uint32_t append_slot(uint32_t* counter) {
    const unsigned m = __activemask();
    const int lane = threadIdx.x & 31;
    const int leader = __ffs(m) - 1;
    uint32_t base = 0;
    if (lane == leader) base = atomicAdd(counter, (uint32_t)__popc(m));
    base = __shfl_sync(m, base, leader);
    return base + (uint32_t)__popc(m & ((1u << lane) - 1u));
}

// Block-aggregated append: one atomic per block and call instead of one per warp, so a
// list filled by a short kernel is not serialised on its counter. Every thread of the
// block, which has whole warps (the ballot waits for all 32 lanes), calls it (flag = this
// thread appends); returns this thread's slot when flag.
__device__ __forceinline__ uint32_t block_append(uint32_t* counter, bool flag) {
    __shared__ uint32_t s_warp[32];
    __shared__ uint32_t s_base;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = (int)((blockDim.x + 31) >> 5);
    const unsigned m = __ballot_sync(0xffffffffu, flag);
    if (lane == 0) s_warp[warp] = (uint32_t)__popc(m);
    __syncthreads();
    if (threadIdx.x == 0) {
        uint32_t tot = 0;
        for (int w = 0; w < nw; w++) {
            const uint32_t c = s_warp[w];
            s_warp[w] = tot;
            tot += c;
        }
        s_base = tot ? atomicAdd(counter, tot) : 0u;
    }
    __syncthreads();
    const uint32_t slot = s_base + s_warp[warp] + (uint32_t)__popc(m & ((1u << lane) - 1u));
    __syncthreads();   // the shared words are reused by the next call
    return slot;
}

// appends a shadow-ray request; every thread of the block calls it
__device__ __forceinline__ void append_ray(const BatchDev& bd, int counter, bool want, float4 ra, float4 rb) {
    const uint32_t slot = block_append(bd.counters + counter, want);
    if (want) {
        bd.qA[slot] = ra;
        bd.qB[slot] = rb;
    }
}

// Next tile of the batch for this block: with bd.persistent, resident blocks pull tiles
// from the queue cursor `ctr` until it is drained; otherwise the launch has one block per
// tile and the hardware block scheduler balances them. `round` counts calls (starts at 0).
__device__ __forceinline__ bool next_tile(const BatchDev& bd, uint32_t* ctr, uint32_t* tile, uint32_t& round) {
    if (bd.halt && (*bd.halt & kBadGrid)) return false;
    if (!bd.persistent) {
        *tile = blockIdx.x;
        return round++ == 0;
    }
    __shared__ uint32_t s_tile;
    __syncthreads();
    if (threadIdx.x == 0) s_tile = atomicAdd(ctr, 1u);
    __syncthreads();
    *tile = s_tile;
    return s_tile < bd.totalTiles;
}

// View of a batch tile and the pixel of this thread in it. RAYS: a warp takes 8 x 4 pixels of
// the tile where its sides allow (else, and for stages that read and write planes, rows
// in order): the primary rays of a compact block cross the same cells longer than those of
// 16 x 2 pixels (1080p, 65,536 emitters: 393 us against 413).
template <int VARIANT, bool RAYS = false>
__device__ __forceinline__ const ViewDev* tile_pixel(const BatchDev& bd, uint32_t tile, int* x, int* y) {
    uint32_t v = 0;
    if (VARIANT == 2)
        while (v + 1 < bd.nviews && bd.views[v + 1].tileBase <= tile) v++;
    const ViewDev* V = view_of<VARIANT>(bd, v);
    const uint32_t lt = tile - V->tileBase;
    const uint32_t tx = lt % V->tilesX, ty = lt / V->tilesX;
    uint32_t ix = threadIdx.x % (uint32_t)bd.tx, iy = threadIdx.x / (uint32_t)bd.tx;
    if (RAYS && (((uint32_t)bd.tx & 7u) | ((uint32_t)bd.ty & 3u)) == 0u) {
        const uint32_t warp = threadIdx.x >> 5, across = (uint32_t)bd.tx >> 3;
        ix = (warp % across) * 8u + (threadIdx.x & 7u);
        iy = (warp / across) * 4u + ((threadIdx.x >> 3) & 3u);
    }
    *x = (int)(tx * (uint32_t)bd.tx + ix);
    *y = (int)(ty * (uint32_t)bd.ty + iy);
    return V;
}

// ---- stage 1: primary rays / G-buffer (renderAlbedo, ris.cl:295-389) --------------------
template <bool BITS>
__device__ __forceinline__ uint32_t albedo_px(const World& w, const Frame& k, uint2* __restrict__ vd, uint32_t* __restrict__ seeds,
                                          int x, int y) {
    const uint32_t seed = wang_hash((uint32_t)x * 171u + (uint32_t)y * 1773u + k.R0);
    const float3 D = camera_ray(k, x, y);
    uint32_t side = 0;
    float dist = 0.0f;
    uint32_t voxel = trace_primary<BITS>(w, k.E, D, &dist, &side);
    float alpha = alphaf(voxel);
    float3 outc = mul(to_rgb(voxel), alpha);
    float total = 0.0f;
    // translucency: continue through non-opaque voxels (ris.cl:321-377)
    float remvis = 1.0f - alphaf(voxel);
    int iteration = 0;
    uint32_t prevSide = 0, prevHit = 0;
    while (prevHit != voxel && remvis > 0.0f) {
        prevHit = voxel;
        prevSide = side;
        total += dist + 0.01f;
        const float3 o = f3(k.E.x + total * D.x, k.E.y + total * D.y, k.E.z + total * D.z);
        voxel = trace<2>(w, o.x, o.y, o.z, D.x, D.y, D.z, 999999, voxel, 0x00FFFFu, &dist, &side);
        const float3 c = to_rgb(voxel);
        alpha = alphaf(voxel);
        outc = add(outc, mul(mul(c, remvis), alpha));
        remvis = remvis * (1.0f - alpha);
        if (++iteration == 25) remvis = 0.0f;
        if (dist <= 0.001f) break;
    }
    if (voxel != 0u) total += dist;
    else side = prevSide;
    const uint32_t enc = from_rgba(outc, 1.0f - remvis, (uint32_t)strength(voxel));
    const size_t i = (size_t)y * k.W + x;
    vd[i] = make_uint2(enc | (side << 24), __float_as_uint(total));
    seeds[i] = seed;
    return (enc & 0x00FFFFFFu) != 0u ? min(side, 2u) : 3u;
}

// Ranks a block's threads of three groups, one group after the other (group 0, 1 or 2, or 3 for
// no rank): this thread's rank; *total: how many have one, plus, with a counter, where their
// slots of a list begin. (Blocks of whole warps, at most kMaxTileThreads: the first warp adds
// the warps' counts up.)
static_assert(kMaxTileThreads <= 256, "8 warps a group");
__device__ __forceinline__ uint32_t block_rank_grouped(uint32_t group, uint32_t* counter, uint32_t* total) {
    __shared__ uint32_t s_first[32];   // 8 group + warp: the warp's count, then its first rank; 31: the total
    const uint32_t warp = threadIdx.x >> 5, lane = threadIdx.x & 31u;
    uint32_t rank = 0;
    for (uint32_t g = 0; g < 3; g++) {
        const unsigned m = __ballot_sync(0xffffffffu, group == g);
        if (group == g) rank = (uint32_t)__popc(m & ((1u << lane) - 1u));
        if (lane == g) s_first[8u * g + warp] = (uint32_t)__popc(m);
    }
    __syncthreads();
    if (warp == 0) {
        const uint32_t c = lane < 24u && (lane & 7u) < (blockDim.x >> 5) ? s_first[lane] : 0u;
        uint32_t sum = c;
        for (uint32_t d = 1; d < 32; d <<= 1) {
            const uint32_t o = __shfl_up_sync(0xffffffffu, sum, d);
            if (lane >= d) sum += o;
        }
        uint32_t first = 0;
        if (counter && lane == 31u && sum) first = atomicAdd(counter, sum);
        s_first[lane] = __shfl_sync(0xffffffffu, first, 31) + sum - c;   // lane 31 has no count
    }
    __syncthreads();
    const uint32_t slot = s_first[8u * min(group, 2u) + warp] + rank;
    *total = s_first[31];
    __syncthreads();   // the shared words are reused by the next call
    return slot;
}
__device__ __forceinline__ uint32_t block_append_grouped(uint32_t* counter, uint32_t group) {
    uint32_t total;
    return block_rank_grouped(group, counter, &total);
}

// Where pixel i of the view (number v of its batch) goes after its primary ray: a pixel that hit
// a face of axis `face` to the hit list, the others (3) get the empty reservoir (ris.cl:34,123).
// A block's hits are listed axis by axis, so that most warps of the candidate pass have
// pixels of one face, where that pays (GROUPED: bd.grouped). Every thread of a block calls it together.
template <bool GROUPED>
__device__ __forceinline__ void list_pixel(const BatchDev& bd, const ViewDev* V, uint32_t v, uint32_t i, bool in, uint32_t face) {
    const uint32_t slot = GROUPED ? block_append_grouped(bd.counters + kCtrHits, face) : block_append(bd.counters + kCtrHits, face < 3u);
    if (face < 3u) {
        bd.hits[slot] = (v << 27) | i;
    } else if (in) {
        V->b.cA[i] = make_uint4(0u, 6u << 29, 0u, 0u);
        V->b.cB[i] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    }
}

// Bound by instruction issue; 4 blocks of 256 threads a SM (64 registers) measured faster than
// 3 (1080p: 413 us against 446) and 5 (455). trace_first's cell masks and packed cells, these
// blocks and compact warps: 1080p, 65,536 emitters 544 -> 393 us, 3840 x 2160 with 1,048,576
// emitters 3,099 -> 2,103 us.
// LISTS: the kernel also fills the hit list (2: grouped), in tile order (compact_hits_kernel
// reads the G-buffer back for it: 333 x 187 271 -> 267 us a frame; at 1080p no difference).
template <int VARIANT, int LISTS, bool BITS>
__global__ void __launch_bounds__(kMaxTileThreads, 4) albedo_kernel(const __grid_constant__ BatchDev bd) {
    follow_previous();
    uint32_t tile, round = 0;
    while (next_tile(bd, bd.counters + kCtrAlbedo, &tile, round)) {
        int x, y;
        const ViewDev* V = tile_pixel<VARIANT, true>(bd, tile, &x, &y);
        const Frame& k = V->k;
        const bool in = x < k.W && y < k.H;
        uint32_t face = 3u;
        if (in) {
            const World w = V->w;
            face = albedo_px<BITS>(w, k, V->b.vd[V->cur], V->b.seed, x, y);
        }
        if (LISTS) list_pixel<LISTS == 2>(bd, V, VARIANT < 2 ? 0u : (uint32_t)(V - bd.views), (uint32_t)y * (uint32_t)k.W + (uint32_t)x, in, face);
    }
}

// ---- ground truth: renderPathTracer / render_di_gfxexp (kernels.cl:177-260, GFXEXP 1) ----
// One-bounce estimate of the direct light: the primary hit's own emission plus the
// emission met along one uniform hemisphere direction (stratified on a 16 x 16 grid by the
// frame counter), weighted by 2 pi N.L and the BRDF, into the frame buffer as (rgb,
// distance); no hit: (0, 0, 0, 1e20). Sky sampling is off (no sky texture). cos and sin
// are the correctly rounded FP64 results rounded to FP32, the oracle's choice for the
// implementation-defined OpenCL builtins.
__device__ __forceinline__ float3 uniform_sample_hemisphere(float r1, float r2, float3 N) {   // tools.cl:31-51
    float3 Nt;
    if (fabsf(N.x) > fabsf(N.y)) {
        const float l = sqrtf(N.x * N.x + N.z * N.z);
        Nt = f3(N.z / l, 0.0f / l, -N.x / l);
    } else {
        const float l = sqrtf(N.y * N.y + N.z * N.z);
        Nt = f3(0.0f / l, -N.z / l, N.y / l);
    }
    const float3 Nb = f3(N.y * Nt.z - N.z * Nt.y, N.z * Nt.x - N.x * Nt.z, N.x * Nt.y - N.y * Nt.x);
    const float sinTheta = sqrtf(1.0f - r1 * r1);
    const float phi = 6.28318530717958647692528f * r2;
    double sd, cd;
    sincos((double)phi, &sd, &cd);            // one argument reduction for both
    const float x = sinTheta * (float)cd;
    const float z = sinTheta * (float)sd;
    return f3((x * Nb.x + r1 * N.x) + z * Nt.x, (x * Nb.y + r1 * N.y) + z * Nt.y, (x * Nb.z + r1 * N.z) + z * Nt.z);
}

// What a pixel's first half leaves to its second (the hemisphere ray).
struct PathRay {
    float3 o, R;
    float ndotl, dist;
    uint32_t voxel, pixel;
};
// the primary ray and the direction; the axis of the face it hit, or 3 (and the finished pixel)
__device__ __forceinline__ uint32_t path_first(const World& w, const Frame& k, int x, int y, float4* frame, PathRay* p) {
    uint32_t seed = wang_hash((uint32_t)x * 171u + (uint32_t)y * 1773u + k.R0);
    const float3 D = camera_ray(k, x, y);
    float dist = 0.0f;
    uint32_t side = 0;
    const uint32_t voxel = trace_primary(w, k.E, D, &dist, &side);
    p->pixel = (uint32_t)y * (uint32_t)k.W + (uint32_t)x;
    if (voxel == 0u) {
        frame[p->pixel] = make_float4(0.0f, 0.0f, 0.0f, 1e20f);
        return 3u;
    }
    const float3 I = f3(k.E.x + D.x * dist, k.E.y + D.y * dist, k.E.z + D.z * dist);
    const int sx = (int)(k.frame & 15u), sy = (int)(k.frame >> 4);
    const float r0 = (float)sx * 0.0625f + rnd(seed) * 0.0625f;
    const float r1 = (float)sy * 0.0625f + rnd(seed) * 0.0625f;
    const float s = side_sign(side, D);
    const float3 N = side_normal(side, s);
    p->R = uniform_sample_hemisphere(r0, r1, N);
    p->ndotl = fmaxf(0.0f, (N.x * p->R.x + N.y * p->R.y) + N.z * p->R.z);
    p->o = f3(I.x + 0.1f * N.x, I.y + 0.1f * N.y, I.z + 0.1f * N.z);
    p->dist = dist;
    p->voxel = voxel;
    return min(side, 2u);
}
__device__ __forceinline__ void path_second(const World& w, const PathRay& p, float4* frame) {
    float dist2 = 0.0f;
    uint32_t side2 = 0;
    // (by the bricks' masks: 8 samples at 1080p 9.15 ms -> 8.92; the primary ray by masks too 8.96)
    const uint32_t voxel2 = trace_first<1, true, true>(w, p.o.x, p.o.y, p.o.z, p.R.x, p.R.y, p.R.z, 128, &dist2, &side2);
    const float INVPI = 0.31830988618379067153777f;
    const float3 rgb = to_rgb(p.voxel);
    const float es = (float)((p.voxel & 0xff0000u) >> 16);
    const float3 contribution = mul(mul(rgb, es), INVPI);
    const float3 brdf = f3(INVPI * rgb.x, INVPI * rgb.y, INVPI * rgb.z);
    const float3 sampleL = mul(mul(to_rgb(voxel2), (float)((voxel2 & 0xff0000u) >> 16)), INVPI);
    const float TWOPI = 6.28318530717958647692528f;
    frame[p.pixel] = make_float4(((sampleL.x * TWOPI) * p.ndotl) * brdf.x + contribution.x,
                                 ((sampleL.y * TWOPI) * p.ndotl) * brdf.y + contribution.y,
                                 ((sampleL.z * TWOPI) * p.ndotl) * brdf.z + contribution.z, p.dist);
}
// The directions of a sample are drawn from one cell of a 16 x 16 grid over the hemisphere, so
// rays of one face are alike and those of another face are not: a block of whole warps deals
// its second rays out again, axis by axis (8 samples at 1080p: 8.92 ms -> 8.77). Bound by
// instruction issue (76 % active); 64 registers: 48 take 9.26 ms, 80 10.2.
__global__ void __launch_bounds__(kMaxTileThreads, 4) path_trace_kernel(const __grid_constant__ BatchDev bd) {
    __shared__ PathRay s_ray[kMaxTileThreads];
    uint32_t tile, round = 0;
    while (next_tile(bd, bd.counters + kCtrAlbedo, &tile, round)) {
        int x, y;
        const ViewDev* V = tile_pixel<0, true>(bd, tile, &x, &y);
        const Frame& k = V->k;
        PathRay p;
        const uint32_t face = x < k.W && y < k.H ? path_first(V->w, k, x, y, V->b.frame, &p) : 3u;
        bool ray = face < 3u;
        if (blockDim.x % 32u == 0u) {
            uint32_t rays;
            const uint32_t slot = block_rank_grouped(face, nullptr, &rays);
            if (ray) s_ray[slot] = p;
            __syncthreads();
            ray = threadIdx.x < rays;
            if (ray) p = s_ray[threadIdx.x];
        }
        if (ray) path_second(V->w, p, V->b.frame);
    }
}

// Hit list of the frame over every view (blockIdx.y = view), for frames run stage by stage
// (whole frames fill it in the primary rays' kernel).
template <int VARIANT, bool GROUPED>
__global__ void __launch_bounds__(256) compact_hits_kernel(const __grid_constant__ BatchDev bd) {
    const ViewDev* V = view_of<VARIANT>(bd, blockIdx.y);
    const uint32_t n = (uint32_t)V->k.W * (uint32_t)V->k.H;
    const uint2* vd = V->b.vd[V->cur];
    // every thread of a block runs the same iterations (list_pixel needs all of them)
    for (uint32_t i0 = blockIdx.x * blockDim.x; i0 < n; i0 += gridDim.x * blockDim.x) {
        const uint32_t i = i0 + threadIdx.x;
        const bool in = i < n;
        const uint32_t word = in ? vd[i].x : 0u;
        list_pixel<GROUPED>(bd, V, blockIdx.y, i, in, (word & 0x00FFFFFFu) != 0u ? min(word >> 24, 2u) : 3u);
    }
}

// ---- visibility (isLightOccluded, ris.cl:1-17) -----------------------------------------
// Persistent shadow tracer over the batch's request queue. Requests:
// qA = (origin, bits(view << 27 | pixel)), qB = (dir, bits(light)). Budget GRIDWIDTH = 128
// steps (ris.cl:10); a miss leaves dist/side at 0 (the fixed convention for the
// reference's uninitialised locals); visible iff the hit voxel (hit point - 0.1 N,
// truncated) lies in the emitter cube [pos, pos + size) (GridCoordinatesFromHit /
// Uint3CubeEquals, tools.cl:452-472). An occluded request zeroes sumOfWeights of its
// pixel in reservoir plane C (plane 0) or H (plane 1) of its view (W follows:
// ris.cl:79-80, 248-250).
__device__ __forceinline__ bool shadow_visible(float3 o, float3 L, float d2, uint32_t s2, uint32_t pos, uint32_t size) {
    const float ns = side_sign(s2, L);
    const float hx = L.x * d2 + o.x, hy = L.y * d2 + o.y, hz = L.z * d2 + o.z;
    const uint32_t vx = f2u(hx - (s2 == 0 ? ns * 0.1f : 0.0f));
    const uint32_t vy = f2u(hy - (s2 == 1 ? ns * 0.1f : 0.0f));
    const uint32_t vz = f2u(hz - (s2 == 2 ? ns * 0.1f : 0.0f));
    const uint32_t ey = pos / (1024u * 1024u), ez = (pos / 1024u) % 1024u, ex = pos % 1024u;
    return ex <= vx && ex + size > vx && ey <= vy && ey + size > vy && ez <= vz && ez + size > vz;
}

// Whether a candidate's ray towards emitter li has to be traced at all. 24 % of the candidate
// rays of the 1080p frame with 65,536 emitters run out of budget far from their emitter, after
// 29 % of all cell visits (49 and 56 % with 1,048,576 emitters). (Shading's rays, most of which
// found their emitter before, are not asked: next to none is ruled out.)
__device__ __forceinline__ bool ray_in_reach(const World& w, float3 o, float3 L, uint32_t li) {
    return shadow_can_reach(w.uber, o, L, __float_as_uint(__ldg(&w.lemit[li].w)), (uint32_t)__ldg(&w.lgeom[li].w), 128);
}

// Rays and queues of one warp of the tracer below (shared memory).
constexpr uint32_t kCellQueue = 256, kBrickQueue = 64;   // powers of two
constexpr int kBurst = 4;      // grid visits between two appends to the cell queue (at most 4)
constexpr uint32_t kSolidCell = 0xFFFFFFFFu;
struct ShadowWarp {
    float4 a[32];                  // per lane its ray: (origin, clipped distance)
    float4 v[32];                  // (direction, bits(view << 1 | 1 when not the request's own numbers))
    float4 r[32];                  // (1 / direction, bits(request))
    uint2 light[32];               // (position, size) of the emitter
    uint2 cell[kCellQueue];        // (bits(t), packed cell | last << 21 | lane << 23)
    uint2 walk[kBrickQueue];       // the same, of cells that have to be walked
    float out[kBrickQueue];        // crossing behind which the ray has left their opaque voxels' box
    uint32_t brick[kBrickQueue];   // their brick, kSolidCell for an opaque brick-less cell
    uint32_t first[32];            // per lane: first hit of a batch, task lane << 1 | visible
};

// The tracer: each lane walks one ray's uber and grid cells (GridWalk) and appends the cells
// that could stop it to the warp's cell queue; 32 queued cells at a time are tested by the
// whole warp (brick-box test), the survivors' bricks queue again and 32 at a time are
// walked by the whole warp. Queues are first in, first out, so a ray's earliest hit is the
// first one seen; its lane takes the answer and any later tasks of it are dropped. A lane
// is refilled from the request queue once `refill` lanes are done, after both queues
// have been emptied (an ended walk is a miss only when none of its tasks hit): half as many as
// the tuning says for candidates, a quarter for shading, whose rays are more alike. Passes in
// us at 8, 4, 3, 2 and 1 idle lanes: 720p candidates 319, 312, 311, 311, 317, shading 304, 291,
// 288, 285, 279; 1080p 515, 511, 510, 515, 543 and 616, 606, 605, 601, 601.
// Bound by instruction issue (70 % active at 960 x 540), not by memory (25 MB of DRAM reads):
// a walker that also steps through bricks keeps 9 of 32 threads busy per instruction, since
// some lane is always in a brick; with the bricks taken out of the walk and packed densely
// 18 are, and a ray costs 387 warp instructions instead of 860. 1,894,052 candidate rays of
// the 1080p frame with 65,536 emitters: 1,563 us before, 728 us now, 515 for the three quarters
// of them in reach (shading's 1,801,412: 1,330 and 601 us); 58,047 rays of a 333 x 187
// frame, bound by the longest ray: 77 and 45 us. 7 blocks a SM (72 registers): 6 took 768 us, 8 (64 registers, spills) 755 us.
// BOX: 1 the world has cell boxes and opacity masks, 2 brick boxes only, 0 neither (cells and
// voxels are read).
template <int VARIANT, int BOX, int MINB>
__global__ void __launch_bounds__(128, MINB) shadow_kernel(const __grid_constant__ BatchDev bd, int countIdx, int fetchIdx,
                                                           int planeSel) {
    follow_previous();
    __shared__ ShadowWarp s_warp[4];
    const int refill = max(bd.refill >> (planeSel ? 2 : 1), 1);
    ShadowWarp& q = s_warp[threadIdx.x >> 5];
    const int lane = threadIdx.x & 31;
    const unsigned below = (1u << lane) - 1u;
    const uint32_t n = bd.counters[countIdx];
    uint32_t* fetch = bd.counters + fetchIdx;
    q.first[lane] = 0xFFFFFFFFu;
    GridWalk k;
    const unsigned long long* ucell = bd.one.w.ucell;
    int st = GW_IDLE;
    bool exhausted = false;
    uint32_t h1 = 0, n1 = 0, h2 = 0, n2 = 0;   // queue heads and lengths, the same in every lane
    auto ray = [&](int owner) {
        const float4 a = q.a[owner], v = q.v[owner], r = q.r[owner];
        return ShadowRay{a.x, a.y, a.z, a.w, v.x, v.y, v.z, r.x, r.y, r.z};
    };
    auto view = [&](int owner) { return view_of<VARIANT>(bd, VARIANT < 2 ? 0u : __float_as_uint(q.v[owner].w) >> 1); };
    // answer of the ray of lane `owner`: a hit at distance d on axis side, or (0, 0) for a miss
    auto visible = [&](int owner, float d, uint32_t side) {
        float4 a = q.a[owner], b = q.v[owner];
        if (__float_as_uint(b.w) & 1u) {
            const uint32_t req = __float_as_uint(q.r[owner].w);
            a = __ldg(bd.qA + req);
            b = __ldg(bd.qB + req);
        }
        const uint2 e = q.light[owner];
        return shadow_visible(f3(a.x, a.y, a.z), f3(b.x, b.y, b.z), d, side, e.x, e.y);
    };
    auto occlude = [&]() {
        const uint32_t e = __float_as_uint(__ldg(&bd.qA[__float_as_uint(q.r[lane].w)].w));
        const ViewDev* V = view_of<VARIANT>(bd, e >> 27);
        reinterpret_cast<uint32_t*>(planeSel ? V->b.hA : V->b.cA)[(size_t)pix_of<VARIANT>(e) * 4u + 2u] = 0u;
    };
    // the first 32 tasks of the brick queue, one per lane
    auto walk_batch = [&]() {
        const uint32_t cnt = min(n2, 32u);
        const uint32_t slot = (h2 + (uint32_t)lane) & (kBrickQueue - 1u);
        const unsigned alive = __ballot_sync(0xffffffffu, st != GW_IDLE);
        bool hit = false;
        if ((uint32_t)lane < cnt) {
            const uint2 rec = q.walk[slot];
            const int owner = (int)(rec.y >> 23);
            if ((alive >> owner) & 1u) {
                const ShadowRay g = ray(owner);
                const uint32_t brick = q.brick[slot];
                const float t = __uint_as_float(rec.x);
                float d = t * 8.0f;
                uint32_t side = (rec.y >> 21) & 3u;
                hit = brick == kSolidCell || brick_task<BOX == 1>(view(owner)->w, brick, rec.y, t, q.out[slot], side, g, &d, &side);
                if (hit) atomicMin(&q.first[owner], (uint32_t)(lane << 1) | (visible(owner, d + g.to, side) ? 1u : 0u));
            }
        }
        h2 += cnt;
        n2 -= cnt;
        if (__any_sync(0xffffffffu, hit)) {
            __syncwarp();
            const uint32_t f = q.first[lane];
            if (f != 0xFFFFFFFFu) {
                q.first[lane] = 0xFFFFFFFFu;
                if (!(f & 1u)) occlude();
                st = GW_IDLE;
            }
        }
        __syncwarp();
    };
    while (true) {
        const unsigned idle = __ballot_sync(0xffffffffu, st == GW_IDLE);
        if (!exhausted) {
            uint32_t base = 0;
            if (lane == 0) base = atomicAdd(fetch, (uint32_t)__popc(idle));
            base = __shfl_sync(0xffffffffu, base, 0);
            if (base + (uint32_t)__popc(idle) >= n) exhausted = true;
            const uint32_t i = base + (uint32_t)__popc(idle & below);
            if (st == GW_IDLE && i < n) {
                const float4 a = __ldg(bd.qA + i), b = __ldg(bd.qB + i);
                const uint32_t vi = VARIANT < 2 ? 0u : __float_as_uint(a.w) >> 27, li = __float_as_uint(b.w);
                const World& w = view_of<VARIANT>(bd, vi)->w;
                q.light[lane] = make_uint2(__float_as_uint(__ldg(&w.lemit[li].w)), (uint32_t)__ldg(&w.lgeom[li].w));
                if (VARIANT == 2) ucell = w.ucell;
                ShadowRay g;
                const bool walks = gw_init(k, g, ucell, a.x, a.y, a.z, b.x, b.y, b.z, 128);
                const bool own = walks && g.ax == a.x && g.ay == a.y && g.az == a.z && g.vx == b.x && g.vy == b.y && g.vz == b.z;
                q.a[lane] = make_float4(g.ax, g.ay, g.az, g.to);
                q.v[lane] = make_float4(g.vx, g.vy, g.vz, __uint_as_float((vi << 1) | (own ? 0u : 1u)));
                q.r[lane] = make_float4(g.rx, g.ry, g.rz, __uint_as_float(i));
                st = walks ? GW_UBER : GW_END;
            }
            __syncwarp();
        }
        if (!__any_sync(0xffffffffu, st != GW_IDLE)) {
            if (exhausted) break;
            continue;
        }
        bool flush;
        do {
            if (st == GW_UBER) st = gw_enter(k, ray(lane), ucell);
            // kBurst grid visits; the cells they report go to the queue together, each lane's
            // in its order (slots by prefix sums over the lanes' counts, one ballot a bit)
            for (int s = 0; s < bd.burst && n1 <= kCellQueue - 32u * kBurst; s += kBurst) {
                float ct[kBurst];
                uint32_t cp[kBurst], found = 0;
#pragma unroll
                for (int u = 0; u < kBurst; u++) {
                    bool task = false;
                    if (st == GW_GRID) {
                        if (gw_visit(k, &task)) {
                            ct[u] = k.t;
                            cp[u] = (k.p & 0x1FFFFFu) | (k.last << 21);
                            if (task) found |= 1u << u;
                            if (!gw_step(k)) st = GW_UBER;
                        } else {
                            st = GW_END;
                        }
                    }
                }
                const uint32_t c = (uint32_t)__popc(found);
                const unsigned b0 = __ballot_sync(0xffffffffu, c & 1u), b1 = __ballot_sync(0xffffffffu, c & 2u),
                               b2 = __ballot_sync(0xffffffffu, c & 4u);
                uint32_t slot = h1 + n1 + (uint32_t)(__popc(b0 & below) + 2 * __popc(b1 & below) + 4 * __popc(b2 & below));
                n1 += (uint32_t)(__popc(b0) + 2 * __popc(b1) + 4 * __popc(b2));
#pragma unroll
                for (int u = 0; u < kBurst; u++)
                    if (found & (1u << u))
                        q.cell[slot++ & (kCellQueue - 1u)] = make_uint2(__float_as_uint(ct[u]), cp[u] | ((uint32_t)lane << 23));
            }
            const unsigned busy = __ballot_sync(0xffffffffu, st == GW_UBER || st == GW_GRID);
            flush = busy == 0u || (!exhausted && 32 - __popc(busy) >= refill);
            __syncwarp();
            while (n1 >= 32u || (flush && n1 > 0u)) {
                const uint32_t cnt = min(n1, 32u);
                const unsigned alive = __ballot_sync(0xffffffffu, st != GW_IDLE);
                int kind = 0;
                float out = 0.0f;
                uint32_t brick = kSolidCell;
                uint2 rec = make_uint2(0u, 0u);
                if ((uint32_t)lane < cnt) {
                    rec = q.cell[(h1 + (uint32_t)lane) & (kCellQueue - 1u)];
                    const int owner = (int)(rec.y >> 23);
                    if ((alive >> owner) & 1u) {
                        const World& w = view(owner)->w;
                        const uint32_t i = rec.y & 0x1FFFFFu;
                        uint2 o = BOX == 1 ? __ldg(w.gbox + i) : make_uint2(__ldg(w.grid + i), 0u);
                        if (BOX == 2 && (o.x & 1u)) o.y = __ldg(w.bbox + (o.x >> 1));
                        kind = grid_task<BOX != 0>(o.x, o.y, rec.y, ray(owner), &out);
                        if (kind == 2) brick = o.x >> 1;
                    }
                }
                const unsigned m = __ballot_sync(0xffffffffu, kind != 0);
                if (kind != 0) {
                    const uint32_t slot = (h2 + n2 + (uint32_t)__popc(m & below)) & (kBrickQueue - 1u);
                    q.walk[slot] = rec;
                    q.out[slot] = out;
                    q.brick[slot] = brick;
                }
                n2 += (uint32_t)__popc(m);
                h1 += cnt;
                n1 -= cnt;
                __syncwarp();
                if (n2 >= 32u) walk_batch();
            }
            if (flush)
                while (n2 > 0u) walk_batch();
        } while (!flush);
        // both queues are empty: a walk that ended without a hit is a miss
        if (st == GW_END) {
            if (!visible(lane, 0.0f, 0u)) occlude();
            st = GW_IDLE;
        }
    }
}

// The same rays through the resumable walker, one cell of any level per lane and step: the
// form that the tuning's walker options (schedule, early-out, brick cache) belong to. Lanes
// refill from the queue as soon as enough are idle. With the early-out a walk stops, as
// occluded, once its budget cannot reach the emitter (walk_target).
__device__ __forceinline__ void shadow_finish(const World& w, int st, const Walker& wk, float3 o, float3 L, uint32_t* plane,
                                              uint32_t pix, uint32_t li) {
    const bool hit = st == WALK_HIT;
    if (!shadow_visible(o, L, hit ? wk.dist : 0.0f, hit ? wk.side : 0u, __float_as_uint(__ldg(&w.lemit[li].w)),
                        (uint32_t)__ldg(&w.lgeom[li].w)))
        plane[(size_t)pix * 4u + 2u] = 0u;
}

// MINB > 0 caps registers so that MINB blocks of 128 threads fit on an SM (more warps to
// hide L2 latency, at the price of a few spills); chosen by the launch tuning.
// CACHE = 1 (single views): blocks of 512 threads, brick walks through the cache walk: with
// a brick cache (bd.bcLog2 > 0) every block first copies the table and the opacity masks
// into shared memory; with bd.bcCount set they count brick walks (calibration).
// EARLY = 1: walks stop as occluded once their budget cannot reach the emitter.
template <int VARIANT, int MINB, int CACHE, int EARLY>
__global__ void __launch_bounds__(CACHE ? 512 : 128, CACHE ? 1 : MINB) shadow_walker_kernel(const __grid_constant__ BatchDev bd,
                                                                                    int countIdx, int fetchIdx,
                                                                                    int planeSel) {
    follow_previous();
    const int refill = bd.refill, burst = bd.burst, schedule = bd.schedule;
    const uint32_t n = bd.counters[countIdx];
    uint32_t* fetch = bd.counters + fetchIdx;
    const int lane = threadIdx.x & 31;
    Walker wk;
    World wt;   // a table batch: the world of this lane's ray; one view: the parameter's
    if (CACHE) {
        extern __shared__ __align__(16) uint32_t bcs[];
        wt = bd.one.w;
        wt.bcCount = bd.bcCount;
        wt.bcLog2 = bd.bcLog2;
        if (bd.bcLog2 > 0) {
            const uint32_t nk = 1u << bd.bcLog2, nm = (nk >> 1) * 16u;
            for (uint32_t i = threadIdx.x; i < nk; i += blockDim.x) bcs[i] = __ldg(bd.bcKeys + i);
            for (uint32_t i = threadIdx.x; i < nm / 4u; i += blockDim.x)
                reinterpret_cast<uint4*>(bcs + nk)[i] = __ldg(reinterpret_cast<const uint4*>(bd.bcMask) + i);
            wt.bcKeys = bcs;
            wt.bcMask = bcs + nk;
        }
        __syncthreads();
    }
    const World& w = (VARIANT < 2 && !CACHE) ? bd.one.w : wt;
    uint32_t* plane = nullptr;
    bool active = false, exhausted = false;
    float3 o = f3(0.0f, 0.0f, 0.0f), L = f3(0.0f, 0.0f, 0.0f);
    uint32_t pix = 0, li = 0;
    while (true) {
        const unsigned idle = __ballot_sync(0xffffffffu, !active);
        if (!exhausted && (idle == 0xffffffffu || __popc(idle) >= refill)) {
            uint32_t base = 0;
            if (lane == 0) base = atomicAdd(fetch, (uint32_t)__popc(idle));
            base = __shfl_sync(0xffffffffu, base, 0);
            if (base + (uint32_t)__popc(idle) >= n) exhausted = true;
            if (!active) {
                const uint32_t r = base + (uint32_t)__popc(idle & ((1u << lane) - 1u));
                if (r < n) {
                    const float4 a = __ldg(bd.qA + r), b = __ldg(bd.qB + r);
                    o = f3(a.x, a.y, a.z);
                    L = f3(b.x, b.y, b.z);
                    const uint32_t e = __float_as_uint(a.w);
                    const ViewDev* V = view_of<VARIANT>(bd, e >> 27);
                    pix = pix_of<VARIANT>(e);
                    li = __float_as_uint(b.w);
                    if (VARIANT == 2) wt = V->w;
                    plane = reinterpret_cast<uint32_t*>(planeSel ? V->b.hA : V->b.cA);
                    const int st = walk_init(wk, w, o.x, o.y, o.z, L.x, L.y, L.z, 128);
                    if (st == WALK_CONTINUE) {
                        if (EARLY)
                            walk_target(wk, __float_as_uint(__ldg(&w.lemit[li].w)), (uint32_t)__ldg(&w.lgeom[li].w));
                        active = true;
                    } else {
                        shadow_finish(w, st, wk, o, L, plane, pix, li);
                    }
                }
            }
        }
        if (!__any_sync(0xffffffffu, active)) {
            if (exhausted) break;
            continue;
        }
        // schedule 1: only the lanes at the DDA level most lanes are at take this round
        // (one level's code per round instead of all three), and stop when they leave it
        int sel = -1;
        if (schedule) {
            const int n2 = __popc(__ballot_sync(0xffffffffu, active && wk.level == 2));
            const int n1 = __popc(__ballot_sync(0xffffffffu, active && wk.level == 1));
            const int n0 = __popc(__ballot_sync(0xffffffffu, active && wk.level == 0));
            sel = n2 >= n1 ? (n2 >= n0 ? 2 : 0) : (n1 >= n0 ? 1 : 0);
        }
        if (active && (sel < 0 || wk.level == sel)) {
#pragma unroll 1
            for (int s = 0; s < burst; s++) {
                const int st = walk_step<(CACHE ? kWalkCache : 0) | (EARLY ? kWalkEarly : 0)>(wk, w);
                if (st != WALK_CONTINUE) {
                    shadow_finish(w, st, wk, o, L, plane, pix, li);
                    active = false;
                    break;
                }
                if (sel >= 0 && wk.level != sel) break;
            }
        }
    }
}

// ---- stage 2a: candidates (perPixelInitialSampling, ris.cl:20-82) ---------------------------
// Over the hit list. Ends with AdjustWeight(res, res.pHat) (implied by the stored
// sumW, pHat, M) and a shadow-ray request for the selected sample when sumW > 0 (when
// sumW == 0 the discard of ris.cl:79-80 changes nothing).
// Bound by instruction issue (80 % active, the ALU pipe 66 %): area_candidate's branch-free
// roots and quotients take a candidate from 761 to 497 warp instructions, 1,894,057 hit
// pixels x 32 candidates from 1,563 to 914 us, x 4 learned ones from 281 to 166 us.
// LEARNED: the light index and its source pdf p come from the learned proposal (drawn
// by the inference kernel) instead of GenerateLightCandidate's uniform 1 / N.
//
// Emitters behind the shading point's surface have weight 0: such a candidate only counts and
// draws. Where they are many, a lane first scans its candidates, leaping over the 14 draws that
// follow the light's, and keeps the random states of those in front; then it works those out
// one after the other, so that a warp takes as many rounds as its lane with the most of them.
// A scanned candidate costs a sixth of a worked-out one, so a warp scans on only when a third
// of its lanes' first two candidates lie behind. SCAN: views that scan (kReachEmitters).
// 1080p frames scanning and not, us, with 8, 12, 16 and 32 candidates: 1,048,576 emitters 1,724
// and 1,742, 1,852 and 1,896, 1,973 and 2,042, 2,419 and 2,584; 65,536 emitters 2,061 and
// 2,053, 2,200 and 2,194, 2,326 and 2,322, 2,795 and 2,797: from 16 on it gains more than it costs.
constexpr uint32_t kScanMin = 16, kScanMax = 32;   // candidates of a pixel (more: no room)
struct FrontScan {
    uint32_t jump[128];               // xs_jump(14)
    uint32_t state[kScanMax][128];    // per thread
};
__device__ const XsJump kJump14 = xs_jump(14);

template <bool POINT, bool LEARNED, bool SCAN>
__device__ __forceinline__ Res ris_reservoir(const ViewDev* V, uint32_t i, uint32_t j, FrontScan* scan, float3* origin) {
    const World w = V->w;
    const Frame& k = V->k;
    const int x = (int)(i % (uint32_t)k.W), y = (int)(i / (uint32_t)k.W);
    const uint2 g = V->b.vd[V->cur][i];
    const uint32_t voxel = g.x & 0x00FFFFFFu, side = g.x >> 24;
    const float dist = __uint_as_float(g.y);
    Res res = res_zero();
    uint32_t seed = V->b.seed[i];
    const float3 D = camera_ray(k, x, y);
    const float nsign = side_sign(side, D);
    const float3 brdf = mul(to_rgb(voxel), 0.31830988618379067153777f);
    const float3 sp = f3(D.x * dist + k.E.x, D.y * dist + k.E.y, D.z * dist + k.E.z);
    const float3 spo = f3(sp.x + (side == 0 ? 0.1f * nsign : 0.0f), sp.y + (side == 1 ? 0.1f * nsign : 0.0f),
                          sp.z + (side == 2 ? 0.1f * nsign : 0.0f));
    const uint32_t nL = k.nlights;
    const float puni = 1.0f / (float)nL;
    // x / (1 / N) is exactly x * N when N is a power of two (1 / N is then exact, and both
    // are the rounding of the same real number)
    const bool pow2 = !LEARNED && (nL & (nL - 1u)) == 0u;
    const float nLf = (float)nL;
    uint32_t count = k.ncand, end = 0;
    bool front = false;
    if (SCAN && !POINT && !LEARNED && count >= kScanMin && count <= kScanMax) {
        const float at = side == 0 ? sp.x : (side == 1 ? sp.y : sp.z);
        uint32_t s = seed, n = 0;
        for (uint32_t c = 0; c < k.ncand; c++) {
            scan->state[n][threadIdx.x] = s;
            const int li = min(max(f2i(rnd(s) * nLf), 0), (int)nL - 1);
            const float4 lg = __ldg(w.lgeom + li);
            // (the sampled point's rounding is below 0.001)
            const float to = nsign * ((side == 0 ? lg.x : (side == 1 ? lg.y : lg.z)) - at) + 0.5f * lg.w;
            if (!(to < -0.01f && lg.w <= 1024.0f)) n++;
            s = xs_leap(scan->jump, s);
            if (c == 1) {
                const unsigned m = __activemask();
                if (3u * __reduce_add_sync(m, n) > 4u * (uint32_t)__popc(m)) break;
                front = true;
            }
        }
        if (front) {
            count = n;
            end = s;
        }
    }
    for (uint32_t c = 0; c < count; c++) {
        int li;
        float p = puni;
        if (front) seed = scan->state[c][threadIdx.x];
        if (LEARNED) {
            const uint2 cq = __ldg(V->ll.cand + (size_t)c * V->ll.stride + j);
            li = (int)cq.x;
            p = __uint_as_float(cq.y);
            // an entry the inference did not write (it gave up and raised its error flag):
            // a uniform candidate instead, so no index leaves the light table
            if (cq.x >= nL || !(p > 0.0f && p <= 1.0f)) {
                li = min(max(f2i(rnd(seed) * (float)nL), 0), (int)nL - 1);
                p = puni;
            }
        } else {
            // GenerateLightCandidate (tools.cl:593-598)
            li = min(max(f2i(rnd(seed) * (float)nL), 0), (int)nL - 1);
        }
        const float4 lg = __ldg(w.lgeom + li);
        const float4 le = __ldg(w.lemit + li);
        float3 pos;
        float inv, ph;
        uint32_t nc;
        if (POINT) {
            pos = f3(lg.x, lg.y, lg.z);
            inv = 1.0f;
            nc = 6;
            ph = phat<true>(pos, nc, sp, side, nsign, brdf, le, lg.w) * inv;
        } else {
            const uint32_t seed0 = seed;
            if (!area_candidate(lg, le, sp, spo, side, nsign, brdf, seed, &ph, &pos, &inv, &nc)) {
                seed = seed0;
                pos = sample_area_light(lg, spo, seed, &inv, &nc);
                ph = phat<false>(pos, nc, sp, side, nsign, brdf, le, lg.w) * inv;
            }
        }
        res_update(res, pow2 ? ph * nLf : ph / p, ph, (uint32_t)li, rnd(seed), pos, inv, nc);
    }
    if (front) {
        seed = end;
        res.M = k.ncand;
    }
    V->b.seed[i] = seed;
    *origin = spo;
    return res;
}

template <bool POINT, bool LEARNED>
__device__ __forceinline__ void ris_item(const BatchDev& bd, const ViewDev* V, uint32_t e, uint32_t i, uint32_t j) {
    float3 o;
    const Res res = ris_reservoir<POINT, LEARNED, false>(V, i, j, nullptr, &o);
    if (res.sumW > 0.0f) {   // (no candidates: sumW is 0)
        const float3 L = normalize3(sub(res.pos, o));
        const uint32_t slot = append_slot(bd.counters + kCtrQ1);
        bd.qA[slot] = make_float4(o.x, o.y, o.z, __uint_as_float(e));
        bd.qB[slot] = make_float4(L.x, L.y, L.z, __uint_as_float(res.idx));
    }
    res_store(V->b.cA, V->b.cB, i, res);
}

template <int VARIANT, bool LEARNED, int MINB>
__global__ void __launch_bounds__(128, MINB) ris_kernel(const __grid_constant__ BatchDev bd) {
    follow_previous();
    const uint32_t nh = bd.counters[kCtrHits];
    for (uint32_t j = blockIdx.x * blockDim.x + threadIdx.x; j < nh; j += gridDim.x * blockDim.x) {
        const uint32_t e = bd.hits[j];
        const ViewDev* V = view_of<VARIANT>(bd, e >> 27);
        if (point_of<VARIANT>(V)) ris_item<true, LEARNED>(bd, V, e, pix_of<VARIANT>(e), j);
        else ris_item<false, LEARNED>(bd, V, e, pix_of<VARIANT>(e), j);
    }
}

// The same with no request for a ray that cannot reach its emitter.
template <int VARIANT, bool LEARNED, int MINB>
__global__ void __launch_bounds__(128, MINB) ris_reach_kernel(const __grid_constant__ BatchDev bd) {
    FrontScan* scan = nullptr;
    if constexpr (VARIANT != 1 && !LEARNED) {
        __shared__ FrontScan s_scan;
        s_scan.jump[threadIdx.x] = kJump14.w[threadIdx.x];   // 128 threads
        __syncthreads();
        scan = &s_scan;
    }
    follow_previous();
    const uint32_t nh = bd.counters[kCtrHits];
    const uint32_t j = blockIdx.x * blockDim.x + threadIdx.x;
    if ((j & ~31u) >= nh) return;   // whole warps
    const bool in = j < nh;
    uint32_t e = 0, i = 0;
    const ViewDev* V = nullptr;
    Res res = res_zero();
    float3 o = f3(0.0f, 0.0f, 0.0f), L = o;
    if (in) {
        e = bd.hits[j];
        V = view_of<VARIANT>(bd, e >> 27);
        i = pix_of<VARIANT>(e);
        res = point_of<VARIANT>(V) ? ris_reservoir<true, LEARNED, true>(V, i, j, scan, &o)
                                   : ris_reservoir<false, LEARNED, true>(V, i, j, scan, &o);
    }
    // the warp's requests together: lanes that appended as they came out of the walk would pay
    // an atomic each (learned, 4 candidates: 354 us against 253)
    __syncwarp();
    bool ray = res.sumW > 0.0f, out = false;
    if (ray) {
        L = normalize3(sub(res.pos, o));
        out = !ray_in_reach(V->w, o, L, res.idx);
        if (out) res.sumW = 0.0f;   // as the tracer does for an occluded request
    }
    __syncwarp();
    ray = ray && !out;
    const uint32_t outs = __ballot_sync(0xFFFFFFFFu, out), rays = __ballot_sync(0xFFFFFFFFu, ray);
    const uint32_t lane = threadIdx.x & 31u;
    uint32_t slot = 0;
    if (lane == 0) {
        if (outs) atomicAdd(bd.counters + kCtrOut1, (uint32_t)__popc(outs));
        if (rays) slot = atomicAdd(bd.counters + kCtrQ1, (uint32_t)__popc(rays));
    }
    slot = __shfl_sync(0xFFFFFFFFu, slot, 0) + (uint32_t)__popc(rays & ((1u << lane) - 1u));
    if (ray) {
        bd.qA[slot] = make_float4(o.x, o.y, o.z, __uint_as_float(e));
        bd.qB[slot] = make_float4(L.x, L.y, L.z, __uint_as_float(res.idx));
    }
    if (in) res_store(V->b.cA, V->b.cB, i, res);
}

// ---- stage 2c: temporal reuse (ris.cl:84-119) over the hit list, after visibility ------------
template <bool POINT>
__device__ __forceinline__ void temporal_item(const ViewDev* V, uint32_t i) {
    const Frame& k = V->k;
    if (!(k.restirtemporalframe > 0 && k.temporal)) return;
    // loads are issued as early as their addresses are known (before the tests that may
    // make them unneeded), so the item waits for three rounds of memory instead of five
    const uint4 ca = __ldg(V->b.cA + i);
    const float4 cb = __ldg(V->b.cB + i);
    const uint32_t seed0 = V->b.seed[i];
    const int x = (int)(i % (uint32_t)k.W), y = (int)(i / (uint32_t)k.W);
    const uint2 g = V->b.vd[V->cur][i];
    const uint32_t voxel = g.x & 0x00FFFFFFu, side = g.x >> 24;
    const float dist = __uint_as_float(g.y);
    const float3 D = camera_ray(k, x, y);
    const float3 sp = f3(D.x * dist + k.E.x, D.y * dist + k.E.y, D.z * dist + k.E.z);
    const float dl = ((sp.x * k.Nl.x + sp.y * k.Nl.y) + sp.z * k.Nl.z) - k.Nl.w;
    const float dr = ((sp.x * k.Nr.x + sp.y * k.Nr.y) + sp.z * k.Nr.z) - k.Nr.w;
    const float dt = ((sp.x * k.Nt.x + sp.y * k.Nt.y) + sp.z * k.Nt.z) - k.Nt.w;
    const float db = ((sp.x * k.Nb.x + sp.y * k.Nb.y) + sp.z * k.Nb.z) - k.Nb.w;
    const float up = (float)k.W * (dl / (dl + dr));
    const float vp = (float)k.H * (dt / (dt + db));
    const float ru = roundf(up), rv = roundf(vp);
    if (!(ru == ru && rv == rv)) return;
    const int px = f2i(ru), py = f2i(rv);
    if (px < 0 || py < 0 || px >= k.W || py >= k.H) return;
    const size_t jp = (size_t)py * k.W + px;
    const uint2 pg = __ldg(V->b.vd[V->cur ^ 1] + jp);
    Res prev = res_load(V->b.hA, V->b.hB, jp);
    const float pdist = __uint_as_float(pg.y);
    if ((pg.x >> 24) != side || !(fabsf(dist - pdist) <= 0.1f * dist)) return;
    const uint32_t pm = min(k.maxTemporal * k.ncand, prev.M);
    if (pm == 0u) return;
    uint32_t pli = prev.idx;
    if (pli >= k.nlights) { raise_error(V->b.err, 2u); pli = 0; }
    const float nsign = side_sign(side, D);
    const float3 brdf = mul(to_rgb(voxel), 0.31830988618379067153777f);
    const float4 pg4 = __ldg(V->w.lgeom + pli), pe4 = __ldg(V->w.lemit + pli);
    const float pph = phat<POINT>(prev.pos, prev.ncode, sp, side, nsign, brdf, pe4, pg4.w) * prev.inv;
    const float W = res_W(prev);
    res_reweigh(prev, W, pph, pm);
    Res res;
    res.idx = ca.x;
    res.M = ca.y & 0x1FFFFFFFu;
    res.ncode = ca.y >> 29;
    res.sumW = __uint_as_float(ca.z);
    res.pHat = __uint_as_float(ca.w);
    res.pos = f3(cb.x, cb.y, cb.z);
    res.inv = cb.w;
    uint32_t seed = seed0;
    res_combine(res, prev, rnd(seed));
    // AdjustWeight(res, pHat of the selected sample here) equals res.pHat
    res_store(V->b.cA, V->b.cB, i, res);
    V->b.seed[i] = seed;
}

template <int VARIANT>
__global__ void __launch_bounds__(128) temporal_kernel(const __grid_constant__ BatchDev bd) {
    follow_previous();
    const uint32_t nh = bd.counters[kCtrHits];
    for (uint32_t j = blockIdx.x * blockDim.x + threadIdx.x; j < nh; j += gridDim.x * blockDim.x) {
        const uint32_t e = bd.hits[j];
        const ViewDev* V = view_of<VARIANT>(bd, e >> 27);
        if (point_of<VARIANT>(V)) temporal_item<true>(V, pix_of<VARIANT>(e));
        else temporal_item<false>(V, pix_of<VARIANT>(e));
    }
}

// 4a: the shadow-ray request of a hit pixel whose reservoir has W > 0 and M > 0; false without
__device__ __forceinline__ bool shade_ray(const ViewDev* V, uint32_t e, int x, int y, uint2 g, uint32_t li, uint32_t M,
                                          float sumW, float pHat, float3 pos, float4* ra, float4* rb) {
    const Frame& k = V->k;
    const float W = sumW / fmaxf(1e-5f, pHat * (float)M);
    if (!(W > 0.0f && M > 0u)) return false;
    const uint32_t side = g.x >> 24;
    const float dist = __uint_as_float(g.y);
    const float3 D = camera_ray(k, x, y);
    const float nsign = side_sign(side, D);
    const float3 sp = f3(D.x * dist + k.E.x, D.y * dist + k.E.y, D.z * dist + k.E.z);
    const float3 spo = f3(sp.x + (side == 0 ? 0.1f * nsign : 0.0f), sp.y + (side == 1 ? 0.1f * nsign : 0.0f),
                          sp.z + (side == 2 ? 0.1f * nsign : 0.0f));
    if (li >= k.nlights) { raise_error(V->b.err, 8u); li = 0; }
    const float3 L = normalize3(sub(pos, spo));
    *ra = make_float4(spo.x, spo.y, spo.z, __uint_as_float(e));
    *rb = make_float4(L.x, L.y, L.z, __uint_as_float(li));
    return true;
}
// ---- stage 3: spatial reuse (perPixelSpatialResampling, ris.cl:126-151,
//      spatialSampling.cl:2-66) -------------------------------------------------------
// Returns the pixel's reservoir and G-buffer word.
template <bool POINT>
__device__ __forceinline__ Res spatial_px(const ViewDev* V, int x, int y, uint2* gout) {
    const Frame& k = V->k;
    const size_t i = (size_t)y * k.W + x;
    const uint4* cA = V->b.cA;
    const float4* cB = V->b.cB;
    const uint2* vd = V->b.vd[V->cur];
    Res res = res_load(cA, cB, i);
    const uint2 g = vd[i];
    *gout = g;
    const uint32_t voxel = g.x & 0x00FFFFFFu;
    if (voxel != 0u && k.spatial) {
        const uint32_t side = g.x >> 24;
        const float dist = __uint_as_float(g.y);
        uint32_t seed = V->b.seed[i];
        const float3 D = camera_ray(k, x, y);
        const float nsign = side_sign(side, D);
        const float3 brdf = mul(to_rgb(voxel), 0.31830988618379067153777f);
        const float3 sp = f3(D.x * dist + k.E.x, D.y * dist + k.E.y, D.z * dist + k.E.z);
        const float rad = (float)(k.radius - 1u);
        for (uint32_t t = 0; t < k.taps; t++) {
            const float angle = rnd(seed) * 6.28318530717958647692528f;
            const float radius = rad * sqrtf(rnd(seed)) + 1.0f;
            float sn, cs;
            sincos_vx(angle, &sn, &cs);
            const int nx = x + f2i(cs * radius), ny = y + f2i(sn * radius);
            if ((nx == x && ny == y) || nx < 0 || ny < 0 || nx >= k.W || ny >= k.H) continue;
            const size_t j = (size_t)ny * k.W + nx;
            Res nb = res_load(cA, cB, j);
            const uint2 ng = __ldg(vd + j);
            // the light record is fetched with the tests still pending (it is needed when
            // they pass), one round of memory fewer per combined tap
            const uint32_t nli = nb.idx < k.nlights ? nb.idx : 0u;
            const float4 lg = __ldg(V->w.lgeom + nli), le = __ldg(V->w.lemit + nli);
            if (nb.M > 0u) {
                const float ndist = __uint_as_float(ng.y);
                if ((ng.x >> 24) == side && fabsf(dist - ndist) <= 0.1f * dist) {
                    if (nb.idx >= k.nlights) raise_error(V->b.err, 4u);
                    const float ph = phat<POINT>(nb.pos, nb.ncode, sp, side, nsign, brdf, le, lg.w) * nb.inv;
                    const float W = res_W(nb);
                    res_reweigh(nb, W, ph, nb.M);
                    res_combine(res, nb, rnd(seed));
                }
            }
        }
        // AdjustWeight(res, res.pHat): implied by the stored (sumW, pHat, M)
        V->b.seed[i] = seed;
    }
    res_store(V->b.hA, V->b.hB, i, res);
    return res;
}

// LISTS: the pixel's shading request too, from the reservoir at hand (requests_with_spatial).
template <int VARIANT, bool LISTS>
__global__ void __launch_bounds__(kMaxTileThreads) spatial_kernel(const __grid_constant__ BatchDev bd) {
    follow_previous();
    uint32_t tile, round = 0;
    while (next_tile(bd, bd.counters + kCtrSpatial, &tile, round)) {
        int x, y;
        const ViewDev* V = tile_pixel<VARIANT>(bd, tile, &x, &y);
        bool want = false;
        float4 ra = make_float4(0.0f, 0.0f, 0.0f, 0.0f), rb = ra;
        if (x < V->k.W && y < V->k.H) {
            uint2 g;
            const Res r = point_of<VARIANT>(V) ? spatial_px<true>(V, x, y, &g) : spatial_px<false>(V, x, y, &g);
            if (LISTS && (g.x & 0x00FFFFFFu) != 0u) {
                const uint32_t v = VARIANT < 2 ? 0u : (uint32_t)(V - bd.views);
                want = shade_ray(V, (v << 27) | ((uint32_t)y * (uint32_t)V->k.W + (uint32_t)x), x, y, g, r.idx, r.M, r.sumW,
                                 r.pHat, r.pos, &ra, &rb);
            }
        }
        if (LISTS) append_ray(bd, kCtrQ2, want, ra, rb);
    }
}

// ---- stage 4: shading (renderRIS / render_di_ris, ris.cl:155-293, 391-413) ------------------
// (small whole frames append their requests in the spatial pass instead)
template <int VARIANT>
__global__ void __launch_bounds__(128) shade_request_kernel(const __grid_constant__ BatchDev bd) {
    follow_previous();
    const uint32_t nh = bd.counters[kCtrHits];
    // every thread of a block runs the same iterations (append_ray needs all of them)
    for (uint32_t j0 = blockIdx.x * blockDim.x; j0 < nh; j0 += gridDim.x * blockDim.x) {
        const uint32_t j = j0 + threadIdx.x;
        bool want = false;
        float4 ra = make_float4(0.0f, 0.0f, 0.0f, 0.0f), rb = ra;
        if (j < nh) {
            const uint32_t e = bd.hits[j];
            const ViewDev* V = view_of<VARIANT>(bd, e >> 27);
            const uint32_t i = pix_of<VARIANT>(e);
            const Res r = res_load(V->b.hA, V->b.hB, i);
            want = shade_ray(V, e, (int)(i % (uint32_t)V->k.W), (int)(i / (uint32_t)V->k.W), V->b.vd[V->cur][i], r.idx, r.M,
                             r.sumW, r.pHat, r.pos, &ra, &rb);
        }
        append_ray(bd, kCtrQ2, want, ra, rb);
    }
}

// ---- sky dome (tools.cl:6-15, 21-28, 54-70, 130-144) --------------------------------
// acos, atan2, sin and cos are the correctly rounded binary32 values (through double).

// SampleSky with SphericalTheta / SphericalPhi: bilinear lookup of direction (tx, ty, tz)
// in the z-up sky texture
__device__ __forceinline__ float3 sample_sky(const Sky& s, float tx, float ty, float tz) {
    const float PI = 3.14159265358979323846264f;
    const float INV2PI = 0.15915494309189533576888f, INVPI = 0.31830988618379067153777f;
    const float theta = (float)acos((double)fminf(fmaxf(tz, -1.0f), 1.0f));
    float phi = (float)atan2((double)ty, (double)tx);
    phi = phi < 0.0f ? phi + 2.0f * PI : phi;
    const float u = ((float)s.w * phi) * INV2PI - 0.5f;
    const float v = ((float)s.h * theta) * INVPI - 0.5f;
    const float fu = u - floorf(u), fv = v - floorf(v);
    const uint32_t iu = (uint32_t)f2i(u), iv = (uint32_t)f2i(v), n = s.w * s.h;
    const float4 a = __ldg(s.tex + (iu + iv * s.w) % n), b = __ldg(s.tex + (iu + 1u + iv * s.w) % n);
    const float4 c = __ldg(s.tex + (iu + (iv + 1u) * s.w) % n), d = __ldg(s.tex + (iu + 1u + (iv + 1u) * s.w) % n);
    const float gu = 1.0f - fu, gv = 1.0f - fv;
    return f3((((a.x * gu) * gv + (b.x * fu) * gv) + (c.x * gu) * fv) + (d.x * fu) * fv,
              (((a.y * gu) * gv + (b.y * fu) * gv) + (c.y * gu) * fv) + (d.y * fu) * fv,
              (((a.z * gu) * gv + (b.z * fu) * gv) + (c.z * gu) * fv) + (d.z * fu) * fv);
}

// blueNoiseSampler: E. Heitz's ranked, scrambled sequence, sample `idx`, dimension `dim`
__device__ __forceinline__ float blue_noise(const uint32_t* bn, int x, int y, int idx, int dim) {
    x &= 127, y &= 127, idx &= 255, dim &= 255;
    const int ranked = (idx ^ (int)__ldg(bn + dim + (x + y * 128) * 8 + 65536 * 3)) & 255;
    int value = (int)__ldg(bn + dim + ranked * 256);
    value ^= (int)__ldg(bn + (dim & 7) + (x + y * 128) * 8 + 65536);
    float r = (0.5f + (float)value) * (1.0f / 256.0f);
    if (r >= 1.0f) r -= 1.0f;
    return r;
}

// DiffuseReflectionCosWeighted: cosine-weighted direction around N
__device__ __forceinline__ float3 cos_weighted(float r0, float r1, float3 N) {
    const float3 T = normalize3(cross3(N, fabsf(N.y) > 0.99f ? f3(1.0f, 0.0f, 0.0f) : f3(0.0f, 1.0f, 0.0f)));
    const float3 B = cross3(T, N);
    const float term1 = 6.28318530717958647692528f * r0, term2 = sqrtf(1.0f - r1);
    double sd, cd;
    sincos((double)term1, &sd, &cd);          // one argument reduction for both
    const float c = (float)cd, s = (float)sd;
    const float ct = c * term2, st = s * term2, sr = sqrtf(r1);
    return f3((ct * T.x + st * B.x) + sr * N.x, (ct * T.y + st * B.y) + sr * N.y, (ct * T.z + st * B.z) + sr * N.z);
}

// skyLight entry of an axis normal (ris.cl:279-285: the last matching test wins)
__device__ __forceinline__ float4 sky_light(const Sky& s, float3 M) {
    float4 l = s.light[0];
    if (M.x > 0.9f) l = s.light[1];
    if (M.y < -0.9f) l = s.light[2];
    if (M.y > 0.9f) l = s.light[3];
    if (M.z < -0.9f) l = s.light[4];
    if (M.z > 0.9f) l = s.light[5];
    return l;
}

// accumulatorFinalizer (kernels.cl:304-326): running mean over `framecount` frames
__device__ __forceinline__ void accumulate_px(const ViewDev* V, size_t i, float4 px) {
    const Frame& k = V->k;
    const int n = (int)k.framecount * k.accumulate;
    float4 prev = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    if (n > 0) prev = V->b.accum[i];
    const float cw = 1.0f / (float)(1 + n);
    V->b.accum[i] = make_float4((1.0f - cw) * prev.x + cw * px.x, (1.0f - cw) * prev.y + cw * px.y,
                                (1.0f - cw) * prev.z + cw * px.z, 1.0f);
}

// 4c: colour per pixel once visibility has zeroed the occluded reservoirs; optionally
// fused with the accumulator. SKY: the frame may carry a sky dome (the sky-less
// instantiation keeps the common case's registers).
template <bool POINT, bool SKY>
__device__ __forceinline__ void shade_finish_px(const ViewDev* V, int x, int y, int fuse) {
    const Frame& k = V->k;
    const size_t i = (size_t)y * k.W + x;
    const uint2 g = V->b.vd[V->cur][i];
    const uint32_t voxel = g.x & 0x00FFFFFFu;
    const float dist = __uint_as_float(g.y);
    const float INVPI = 0.31830988618379067153777f;
    float3 color = f3(0.0f, 0.0f, 0.0f);
    const Sky* sky = SKY ? k.sky : nullptr;
    if (sky && voxel == 0u) {
        // background (ris.cl:197-202); the sky-light term adds its incoming light times a
        // zero BRDF, which leaves non-negative sums as they are
        const float3 D = camera_ray(k, x, y);
        color = sample_sky(*sky, D.x, D.z, D.y);
        const float4 l = sky_light(*sky, side_normal(g.x >> 24, side_sign(g.x >> 24, D)));
        color = add(color, f3((0.0f + sky->lightScale * l.x) * 0.0f, (0.0f + sky->lightScale * l.y) * 0.0f,
                              (0.0f + sky->lightScale * l.z) * 0.0f));
    }
    if (voxel != 0u) {
        float3 skyC = f3(0.0f, 0.0f, 0.0f);   // sky seen through a translucent voxel (ris.cl:206-211)
        if (sky && ((voxel & 0xf000u) >> 12) != 15u) {
            const float3 D = camera_ray(k, x, y);
            skyC = sample_sky(*sky, D.x, D.z, D.y);
        }
        if (emitter(voxel)) {
            const float3 c = to_rgb(voxel);
            const float m = strength(voxel);
            color = add(color, f3((c.x * m) * INVPI, (c.y * m) * INVPI, (c.z * m) * INVPI));
        }
        const uint4 qa = V->b.hA[i];
        const uint32_t M = qa.y & 0x1FFFFFFFu;
        const float W = __uint_as_float(qa.z) / fmaxf(1e-5f, __uint_as_float(qa.w) * (float)M);
        if (W > 0.0f && M > 0u) {   // visible: occluded reservoirs were zeroed by the tracer
            const uint32_t side = g.x >> 24;
            const float4 qb = __ldg(V->b.hB + i);
            const float3 D = camera_ray(k, x, y);
            const float nsign = side_sign(side, D);
            const float3 sp = f3(D.x * dist + k.E.x, D.y * dist + k.E.y, D.z * dist + k.E.z);
            const uint32_t li = qa.x < k.nlights ? qa.x : 0u;
            const float4 lg = __ldg(V->w.lgeom + li), le = __ldg(V->w.lemit + li);
            const float3 brdf = mul(to_rgb(voxel), INVPI);
            bool zero;
            const float3 inc = phat_full<POINT>(f3(qb.x, qb.y, qb.z), qa.y >> 29, sp, side, nsign, brdf, le, lg.w, &zero);
            color = add(color, f3((inc.x * W) * qb.w, (inc.y * W) * qb.w, (inc.z * W) * qb.w));
        }
        const float a = alphaf(voxel);
        color = f3(color.x + ((a * color.x) + ((1.0f - a) * skyC.x)), color.y + ((a * color.y) + ((1.0f - a) * skyC.y)),
                   color.z + ((a * color.z) + ((1.0f - a) * skyC.z)));
        if (sky) {
            // sky light (ris.cl:258-290): one cosine-weighted ray, 10 steps, opaque voxels
            // only; lit by the sky light of the normal it ends on
            const uint32_t side = g.x >> 24;
            const float3 D = camera_ray(k, x, y);
            const float3 N = side_normal(side, side_sign(side, D));
            const float r0 = blue_noise(sky->blueNoise, x, y, (int)k.frame, 0);
            const float r1 = blue_noise(sky->blueNoise, x, y, (int)k.frame, 1);
            const float3 R = cos_weighted(r0, r1, N);
            const float3 sp = f3(D.x * dist + k.E.x, D.y * dist + k.E.y, D.z * dist + k.E.z);
            float dist2 = 0.0f;
            uint32_t side2 = 0;
            const uint32_t voxel2 = trace_first<1, true, true, true>(V->w, sp.x + 0.1f * N.x, sp.y + 0.1f * N.y, sp.z + 0.1f * N.z,
                                                                     R.x, R.y, R.z, 10 /* GRIDWIDTH / 12 */, &dist2, &side2);
            float3 toAdd = f3(sky->lightScale, sky->lightScale, sky->lightScale), M = N;
            if (voxel2 != 0u) {
                const float3 c2 = to_rgb(voxel2);
                toAdd = f3(toAdd.x * (INVPI * c2.x), toAdd.y * (INVPI * c2.y), toAdd.z * (INVPI * c2.z));
                M = side_normal(side2, side_sign(side2, R));
            }
            const float4 l = sky_light(*sky, M);
            const float3 inc = f3(0.0f + toAdd.x * l.x, 0.0f + toAdd.y * l.y, 0.0f + toAdd.z * l.z);
            const float3 brdf = mul(to_rgb(voxel), INVPI);
            color = add(color, mulv(inc, brdf));
        }
    }
    const float4 px = make_float4(color.x, color.y, color.z, dist);
    V->b.frame[i] = px;
    if (fuse) accumulate_px(V, i, px);
}

// SKY: bound by the 10-step ray's chain of loads, which more warps hide: 1080p 297 us with
// trace<1> (64 registers), by masks 240 with 80 registers, 204 with 48 (the frame 3.25, 3.17
// and 3.14 ms). A batch's table variant spills more and keeps 80.
template <int VARIANT, bool SKY>
__global__ void __launch_bounds__(kMaxTileThreads, SKY ? (VARIANT < 2 ? 5 : 3) : 1) shade_finish_kernel(const __grid_constant__ BatchDev bd) {
    follow_previous();
    uint32_t tile, round = 0;
    while (next_tile(bd, bd.counters + kCtrFinish, &tile, round)) {
        int x, y;
        const ViewDev* V = tile_pixel<VARIANT>(bd, tile, &x, &y);
        if (x < V->k.W && y < V->k.H) {
            if (point_of<VARIANT>(V)) shade_finish_px<true, SKY>(V, x, y, bd.fuse);
            else shade_finish_px<false, SKY>(V, x, y, bd.fuse);
        }
    }
}

// stage 5 on its own
template <int VARIANT>
__global__ void __launch_bounds__(kMaxTileThreads) accumulate_kernel(const __grid_constant__ BatchDev bd) {
    uint32_t tile, round = 0;
    while (next_tile(bd, bd.counters + kCtrAccum, &tile, round)) {
        int x, y;
        const ViewDev* V = tile_pixel<VARIANT>(bd, tile, &x, &y);
        if (x < V->k.W && y < V->k.H) {
            const size_t i = (size_t)y * V->k.W + x;
            accumulate_px(V, i, V->b.frame[i]);
        }
    }
}

}  // namespace dev
}  // namespace vxr

// ---- launchers -------------------------------------------------------------------------
namespace vxr {

static int g_sms = 0;
static int sm_count() {
    if (!g_sms) {
        int dev = 0;
        cudaGetDevice(&dev);
        cudaDeviceGetAttribute(&g_sms, cudaDevAttrMultiProcessorCount, dev);
        if (g_sms <= 0) g_sms = 1;
    }
    return g_sms;
}
// grid-stride kernels over a list of at most n items
static unsigned list_blocks(size_t n, int threads, int per_sm) {
    const size_t need = (n + threads - 1) / threads;
    const size_t cap = (size_t)sm_count() * per_sm;
    return (unsigned)std::max<size_t>(1, std::min(need, cap));
}
// Persistent kernels: as many blocks as fit on the machine at once (occupancy query per
// kernel and block size, cached), never more than there are tiles.
static unsigned resident_blocks(const void* kernel, int threads) {
    static std::mutex mu;
    static std::map<std::pair<const void*, int>, int> cache;
    std::lock_guard<std::mutex> lock(mu);
    auto it = cache.find({kernel, threads});
    if (it == cache.end()) {
        int per = 0;
        if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, kernel, threads, 0) != cudaSuccess || per < 1) per = 1;
        it = cache.emplace(std::make_pair(kernel, threads), per).first;
    }
    return (unsigned)(sm_count() * it->second);
}
// brackets one kernel launch with the attached timer's events
struct Timed {
    const BatchDev& bd;
    int id;
    cudaStream_t s;
    Timed(const BatchDev& b, int i, cudaStream_t st) : bd(b), id(i), s(st) {
        if (bd.timer) bd.timer->mark(id, false, s);
    }
    ~Timed() {
        if (bd.timer) bd.timer->mark(id, true, s);
    }
};

// A kernel whose launch is made ready while the kernel before it in the stream still runs
// (programmatic stream serialization; follow_previous is what keeps the order). Frames, us,
// without and with it: 256 x 144 without allocation 222 and 203, 333 x 187 217 and 212, 640 x 360
// 329 and 325; large ones do not change. Its blocks are not placed before the others' are done
// (griddepcontrol.launch_dependents at the kernels' start): they would hold places that the
// blocks still to come then share unevenly (241, 230 and 326 us).
template <class... P, class... A>
static void launch_next(bool follow, void (*kernel)(P...), unsigned blocks, unsigned threads, cudaStream_t s, const A&... args) {
    cudaLaunchAttribute at;
    at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at.val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(blocks);
    cfg.blockDim = dim3(threads);
    cfg.stream = s;
    cfg.attrs = &at;
    cfg.numAttrs = follow ? 1 : 0;
    cudaLaunchKernelEx(&cfg, kernel, args...);
}
// whole frames of single views (a batch's are captured, and its chains overlap on their own)
static bool follows(const BatchDev& bd) { return bd.lists && bd.nviews == 1; }

template <class K>
static void launch_tiles(K kernel, const BatchDev& bd, int ctr, cudaStream_t s, int id) {
    const int threads = bd.tx * bd.ty;
    unsigned nb = std::max(1u, bd.totalTiles);
    if (bd.persistent) {
        if (!bd.lists) cudaMemsetAsync(bd.counters + ctr, 0, sizeof(uint32_t), s);
        nb = std::max(1u, std::min(resident_blocks((const void*)kernel, threads), bd.totalTiles));
    }
    Timed tm(bd, id, s);
    if (id == K_ACCUM) kernel<<<nb, threads, 0, s>>>(bd);
    else launch_next(follows(bd), kernel, nb, threads, s, bd);
}

void apply_tuning(BatchDev& bd, const Tuning& tu) {
    bd.tx = tu.bx;
    bd.ty = tu.by;
    bd.persistent = tu.persistent;
    bd.refill = tu.refill;
    bd.burst = tu.burst;
    bd.listPerSm = tu.listPerSm;
    bd.schedule = tu.schedule;
    bd.earlyOut = tu.earlyOut;
}

// Rays are tested for their reach when the emitters are at least as many as the map's uber
// cells: walks then cross few empty ones, and the budget runs out. Candidates and their rays,
// us without and with the test: 65,536 emitters at 1080p 914 + 728 and 1,001 + 521, learned
// 166 + 738 and 253 + 415; 1,048,576 at 4K 3,568 + 2,330 and 3,892 + 1,108. Worlds with fewer
// lose: 4,096 emitters at 720p 417 + 320 and 460 + 280, 1,024 in a 512^3 world 411 + 266 and
// 435 + 266. Whole 720p frames with the test and without, us: 1024-voxel worlds of 8,192
// emitters 1,277 and 1,281, 16,384 1,277 and 1,293, 32,768 1,291 and 1,319, 65,536 1,320 and
// 1,363; 256-voxel ones of 16,384 1,189 and 1,179, 32,768 1,233 and 1,237, 65,536 1,189 and
// 1,223 (the scan's gain). It loses where rays end within their budget: 512-voxel worlds of
// 32,768 emitters 1,319 and 1,292, of 65,536 1,386 and 1,361, and small frames (333 x 187, 8
// candidates: 204 and 201) - 1 to 2 %, for which a rule would need the emitters' extent.
// Single views only: a batch's views share a launch.
// The area-light candidates of these views are also scanned for those in front of the surface
// (FrontScan), and their hits listed by the axis of their face: at 4K, where 63 % of the
// candidates lie behind, 3,902 us -> 3,061 (3,592 with hits in tile order, as neighbouring
// pixels see different faces), at 1080p, where 21 % do, 1,003 -> 1,005. In worlds of fewer
// emitters, whose light tables L1 holds, the scan's shared memory takes that place: 4,096
// emitters at 720p 418 -> 439 us, 1,024 412 -> 429; and listing by axis costs a small frame
// 1 % (333 x 187: 211.9 -> 213.2 us).
constexpr uint32_t kReachEmitters = 32768;
BatchDev single_batch(const dev::World& w, const dev::Frame& k, const ViewBuffers& b, int cur, bool point, const Tuning& tu) {
    BatchDev bd;
    bd.one.w = w;
    bd.one.k = k;
    bd.one.b = b;
    bd.one.cur = cur;
    bd.one.point = point ? 1 : 0;
    bd.one.tileBase = 0;
    bd.one.tilesX = (uint32_t)((k.W + tu.bx - 1) / tu.bx);
    bd.nviews = 1;
    bd.sky = k.sky != nullptr ? 1 : 0;
    bd.totalPixels = (uint32_t)k.W * (uint32_t)k.H;
    bd.totalTiles = bd.one.tilesX * (uint32_t)((k.H + tu.by - 1) / tu.by);
    apply_tuning(bd, tu);
    bd.grouped = !point && k.nlights >= kReachEmitters && k.ncand >= dev::kScanMin && k.ncand <= dev::kScanMax &&
                 tu.bx * tu.by % 32 == 0;   // (block_append_grouped needs whole warps)
    bd.hits = b.hits;
    bd.qA = b.qA;
    bd.qB = b.qB;
    bd.counters = b.counters;
    return bd;
}

void launch_build_light_table(const uint32_t* raw, int words, uint32_t n, float4* geom, float4* emit, cudaStream_t s) {
    const unsigned nb = (n + 255u) / 256u;
    if (n && words == 4) launch_next(true, dev::build_light_table_kernel<4>, nb, 256, s, raw, n, geom, emit);
    else if (n) launch_next(true, dev::build_light_table_kernel<3>, nb, 256, s, raw, n, geom, emit);
}

void launch_build_brick_boxes(const uint32_t* bricks, const uint32_t* list, uint32_t n, uint32_t* bbox, uint32_t* bbox0,
                              uint32_t* bmask, uint32_t* bmask0, cudaStream_t s) {
    const size_t threads = (size_t)n * 32u;
    if (threads)
        launch_next(true, dev::build_brick_boxes_kernel, (unsigned)((threads + 255u) / 256u), 256, s, bricks, list, n, bbox, bbox0, bmask,
                    bmask0);
}

void launch_clear_flags(uint32_t* err, uint32_t flags, cudaStream_t s) { dev::clear_flags_kernel<<<1, 1, 0, s>>>(err, flags); }

void launch_commit_bricks(const uint32_t* list, const uint32_t* voxels, uint32_t n, uint32_t* bricks, cudaStream_t s) {
    if (n) dev::commit_bricks_kernel<<<n, 128, 0, s>>>(list, voxels, bricks);
}

void launch_build_cells(const uint32_t* grid, const uint32_t* bbox, const uint32_t* bbox0, uint8_t* uber,
                        unsigned long long* ucell, uint4* ucell0, uint2* gbox, uint2* gbox0, uint32_t nbricks, uint32_t* err,
                        cudaStream_t s) {
    const dev::CellTables out{uber, ucell, ucell0, gbox, gbox0};
    launch_next(true, dev::build_cells_kernel, 32 * 32 * 32 / 4, 256, s, grid, bbox, bbox0, out, nbricks, err);
}

void launch_path_trace(const BatchDev& bd, cudaStream_t s) {
    BatchDev b = bd;
    b.timer = nullptr;
    launch_tiles(dev::path_trace_kernel, b, kCtrAlbedo, s, K_ALBEDO);
}

// Views of at most this many pixels walk bricks by the masks of their non-zero voxels: small
// frames wait for their longest ray, whose brick walk reads a line instead of a sector a row
// (333 x 187: 42.5 us -> 35.3, 640 x 360: 41.7 -> 36.3, 1280 x 720: 153 -> 144); larger ones are
// bound by instructions, of which a mask takes more (1080p: 393 -> 405, 3840 x 2160: 2,106 ->
// 2,176). Whole frames with masks and without, us, 4,096 and 65,536 emitters: 960 x 540 759 and
// 788, 814 and 838; 1120 x 630 969 and 976, 1,040 and 1,045; 1280 x 720 1,231 and 1,237, 1,320
// and 1,325; 1440 x 810 1,525 and 1,531, 1,637 and 1,639; 1600 x 900 1,851 and 1,855, 1,987 and
// 1,988; 1080p 2,608 and 2,612, 2,798 and 2,795: alike from a million pixels on.
constexpr uint32_t kBitsPixels = 1u << 20;
void launch_batch_albedo(const BatchDev& bd, int variant, cudaStream_t s) {
    const bool bits = variant != 2 && bd.totalPixels <= kBitsPixels && bd.one.w.bmask0;
    if (bd.lists) {
        // all of the frame's list lengths and cursors at once
        if (!bd.cleared) cudaMemsetAsync(bd.counters, 0, kCounters * sizeof(uint32_t), s);
        if (variant == 2) launch_tiles(dev::albedo_kernel<2, 1, false>, bd, kCtrAlbedo, s, K_ALBEDO);
        else if (bd.grouped) launch_tiles(bits ? dev::albedo_kernel<0, 2, true> : dev::albedo_kernel<0, 2, false>, bd, kCtrAlbedo, s, K_ALBEDO);
        else launch_tiles(bits ? dev::albedo_kernel<0, 1, true> : dev::albedo_kernel<0, 1, false>, bd, kCtrAlbedo, s, K_ALBEDO);
    } else {
        if (variant == 2) launch_tiles(dev::albedo_kernel<2, 0, false>, bd, kCtrAlbedo, s, K_ALBEDO);
        else launch_tiles(bits ? dev::albedo_kernel<0, 0, true> : dev::albedo_kernel<0, 0, false>, bd, kCtrAlbedo, s, K_ALBEDO);
    }
}

constexpr int kShadowMinBlocks = 7;   // of shadow_kernel: 728 us against 768 at 6 and 755 at 8 (see there)
template <class K>
static void launch_shadow_rays(K kernel, const BatchDev& bd, int countIdx, int planeSel, cudaStream_t s) {
    const size_t rb = resident_blocks((const void*)kernel, 128);
    const unsigned nb = (unsigned)std::max<size_t>(1, std::min<size_t>(rb, ((size_t)bd.totalPixels + 127) / 128));
    Timed tm(bd, planeSel ? K_SHADOW_SHADE : K_SHADOW_CAND, s);
    launch_next(follows(bd), kernel, nb, 128, s, bd, countIdx, countIdx + 1, planeSel);
}
// shared memory of the brick-cache variant: 2^log2 keys and 2^(log2 - 1) masks of 64 bytes
size_t brick_cache_smem(int log2) { return log2 > 0 ? ((size_t)4 << log2) + ((size_t)64 << (log2 - 1)) : 0; }
template <int EARLY>
static void launch_shadow_cached(const BatchDev& bd, int countIdx, int planeSel, cudaStream_t s) {
    const void* fn = (const void*)dev::shadow_walker_kernel<0, 0, 1, EARLY>;
    const size_t sm = brick_cache_smem(bd.bcLog2);
    if (sm > 48 * 1024) cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm);
    int per = 0;
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, fn, 512, sm);
    const size_t rb = (size_t)std::max(per, 1) * (size_t)sm_count();
    const unsigned nb = (unsigned)std::max<size_t>(1, std::min<size_t>(rb, ((size_t)bd.totalPixels + 511) / 512));
    Timed tm(bd, planeSel ? K_SHADOW_SHADE : K_SHADOW_CAND, s);
    dev::shadow_walker_kernel<0, 0, 1, EARLY><<<nb, 512, sm, s>>>(bd, countIdx, countIdx + 1, planeSel);
}
template <int VARIANT>
static void launch_shadow(const BatchDev& bd, int countIdx, int planeSel, cudaStream_t s) {
    const bool early = bd.earlyOut != 0;
    if (VARIANT < 2 && (bd.bcLog2 > 0 || bd.bcCount)) {
        if (early) launch_shadow_cached<1>(bd, countIdx, planeSel, s);
        else launch_shadow_cached<0>(bd, countIdx, planeSel, s);
    } else if (early) {
        launch_shadow_rays(dev::shadow_walker_kernel<VARIANT, 8, 0, 1>, bd, countIdx, planeSel, s);
    } else if (bd.schedule) {
        launch_shadow_rays(dev::shadow_walker_kernel<VARIANT, 8, 0, 0>, bd, countIdx, planeSel, s);
    } else {
        if constexpr (VARIANT == 0) {
            if (!bd.one.w.bmask) {   // a caller's bricks (vxr_render_frame_noalloc): no masks
                launch_shadow_rays(bd.one.w.bbox ? dev::shadow_kernel<0, 2, kShadowMinBlocks> : dev::shadow_kernel<0, 0, kShadowMinBlocks>,
                                   bd, countIdx, planeSel, s);
                return;
            }
        }
        launch_shadow_rays(dev::shadow_kernel<VARIANT, 1, kShadowMinBlocks>, bd, countIdx, planeSel, s);
    }
}
// 64 registers: at 1080p 914 us against 937 (7 blocks a SM), 988 (6) and 987 (5)
constexpr int kRisMinBlocks = 8;
// A block per 128 pixels of the batch, those past the hit list's end leaving at once: a warp's
// candidates take long enough that the block scheduler balances them better than resident
// blocks striding over the list (1080p, 7 blocks a SM: 937 us against 1,005).
template <int VARIANT, bool LEARNED>
static void launch_ris(const BatchDev& bd, cudaStream_t s) {
    const unsigned nb = (unsigned)(((size_t)bd.totalPixels + 127) / 128);
    Timed tm(bd, K_RIS, s);
    if constexpr (VARIANT < 2) {
        if (bd.one.k.nlights >= kReachEmitters) {
            launch_next(follows(bd), dev::ris_reach_kernel<VARIANT, LEARNED, kRisMinBlocks>, nb, 128, s, bd);
            return;
        }
    }
    launch_next(follows(bd), dev::ris_kernel<VARIANT, LEARNED, kRisMinBlocks>, nb, 128, s, bd);
}

template <int VARIANT>
static void candidates_v(const BatchDev& bd, const LearnedHook* learned, cudaStream_t s, cudaStream_t tail,
                         cudaEvent_t ev) {
    const size_t n = bd.totalPixels;
    if (!bd.lists) {
        cudaMemsetAsync(bd.counters + kCtrHits, 0, 4 * sizeof(uint32_t), s);   // hits, q1 requests, q1 fetch, decided rays
        const uint32_t maxPx = VARIANT < 2 ? bd.totalPixels : (uint32_t)(n / bd.nviews + 1);
        Timed tm(bd, K_COMPACT, s);
        const dim3 nb(list_blocks(maxPx, 256, 8), bd.nviews);
        if (VARIANT < 2 && bd.grouped) dev::compact_hits_kernel<VARIANT < 2 ? 0 : 2, true><<<nb, 256, 0, s>>>(bd);
        else dev::compact_hits_kernel<VARIANT < 2 ? 0 : 2, false><<<nb, 256, 0, s>>>(bd);
    }
    const unsigned nb = list_blocks(n, 128, bd.listPerSm);
    bool learnedDone = false;
    if constexpr (VARIANT < 2) {
        if (learned) {
            BatchDev lb = bd;
            lb.one.ll.cand = learned->cand;
            lb.one.ll.stride = (uint32_t)n;
            prop::InferArgs ia = learned->infer;
            ia.k = bd.one.k;
            ia.vd = bd.one.b.vd[bd.one.cur];
            ia.hits = bd.hits;
            ia.count = bd.counters + kCtrHits;
            ia.ncand = bd.one.k.ncand;
            ia.cand = learned->cand;
            ia.clOff = learned->clOff;
            ia.clMembers = learned->clMembers;
            ia.lightCluster = learned->lightCluster;
            ia.nlights = bd.one.k.nlights;
            ia.candStride = (uint32_t)n;
            ia.err = bd.one.b.err;
            ia.samples = nullptr;
            ia.probs = nullptr;
            if (bd.one.k.ncand > 0) {
                Timed tm(bd, K_INFER, s);
                if (learned->rows) {
                    cudaMemsetAsync(learned->rowCount, 0, sizeof(uint32_t), s);
                    prop::launch_pair_rows(ia.k, ia.vd, ia.hits, ia.count, (uint32_t)n, learned->group,
                                           learned->pairDist, learned->rows, learned->rowCount, s);
                    ia.rows = learned->rows;
                    ia.rowCount = learned->rowCount;
                }
                prop::launch_infer(ia, (uint32_t)n, s);
            }
            launch_ris<VARIANT, true>(lb, s);
            learnedDone = true;
        }
    }
    if (!learnedDone) launch_ris<VARIANT, false>(bd, s);
    launch_shadow<VARIANT < 2 ? 0 : 2>(bd, kCtrQ1, 0, s);
    if (tail && tail != s) {
        cudaEventRecord(ev, s);
        cudaStreamWaitEvent(tail, ev, 0);
        s = tail;
    }
    // a single view without temporal reuse this frame skips the launch (a table checks per view)
    if (VARIANT == 2 || (bd.one.k.restirtemporalframe > 0 && bd.one.k.temporal)) {
        Timed tm(bd, K_TEMPORAL, s);
        launch_next(follows(bd), dev::temporal_kernel<VARIANT>, nb, 128, s, bd);
    }
}

void launch_batch_candidates(const BatchDev& bd, int variant, const LearnedHook* learned, cudaStream_t s,
                             cudaStream_t tail, cudaEvent_t ev) {
    if (variant == 0) candidates_v<0>(bd, learned, s, tail, ev);
    else if (variant == 1) candidates_v<1>(bd, learned, s, tail, ev);
    else candidates_v<2>(bd, nullptr, s, tail, ev);
}

// A whole frame's shading requests come from the spatial pass while the frame is small: that
// saves a launch and a pass. In larger frames the pass, with the registers and barriers that
// appending costs it, holds back the next frame's primary rays, which start at its end and
// run beside the separate kernel. Frames in us with the pass appending and with the kernel:
// one after the other 480 x 270 169 and 172 (4,096 emitters 302 and 304), 640 x 360 230 and 232
// (423 and 427), 720 x 405 261 and 256 (494 and 472), 800 x 450 299 and 293 (577 and 555),
// 960 x 540 384 and 378 (759 and 743), 1280 x 720 614 and 612 (1,237 and 1,231); each waited
// for, the pass stays ahead: 640 x 360 268 and 271, 720 x 405 298 and 303 (533 and 537),
// 960 x 540 426 and 431 (803 and 807). Batches, whose frames do not overlap, are within 1 %
// either way.
constexpr uint32_t kSpatialRequests = 1u << 18;
static bool requests_with_spatial(const BatchDev& bd) { return bd.lists && bd.totalPixels <= kSpatialRequests; }

template <bool LISTS>
static void spatial_v(const BatchDev& bd, int variant, cudaStream_t s) {
    if (variant == 0) launch_tiles(dev::spatial_kernel<0, LISTS>, bd, kCtrSpatial, s, K_SPATIAL);
    else if (variant == 1) launch_tiles(dev::spatial_kernel<1, LISTS>, bd, kCtrSpatial, s, K_SPATIAL);
    else launch_tiles(dev::spatial_kernel<2, LISTS>, bd, kCtrSpatial, s, K_SPATIAL);
}
void launch_batch_spatial(const BatchDev& bd, int variant, cudaStream_t s) {
    if (requests_with_spatial(bd)) spatial_v<true>(bd, variant, s);
    else spatial_v<false>(bd, variant, s);
}

template <int VARIANT>
static void shade_v(const BatchDev& bd, cudaStream_t s) {
    if (!requests_with_spatial(bd)) {
        if (!bd.lists) cudaMemsetAsync(bd.counters + kCtrQ2, 0, 2 * sizeof(uint32_t), s);   // q2 requests, q2 fetch
        Timed tm(bd, K_SHADE_REQ, s);
        launch_next(follows(bd), dev::shade_request_kernel<VARIANT < 2 ? 0 : 2>, list_blocks(bd.totalPixels, 128, bd.listPerSm), 128, s, bd);
    }
    launch_shadow<VARIANT < 2 ? 0 : 2>(bd, kCtrQ2, 1, s);
    if (bd.sky) launch_tiles(dev::shade_finish_kernel<VARIANT, true>, bd, kCtrFinish, s, K_SHADE_FINISH);
    else launch_tiles(dev::shade_finish_kernel<VARIANT, false>, bd, kCtrFinish, s, K_SHADE_FINISH);
}

void launch_batch_shade(const BatchDev& bd, int variant, cudaStream_t s) {
    if (variant == 0) shade_v<0>(bd, s);
    else if (variant == 1) shade_v<1>(bd, s);
    else shade_v<2>(bd, s);
}

void launch_batch_accumulate(const BatchDev& bd, int variant, cudaStream_t s) {
    if (variant == 2) launch_tiles(dev::accumulate_kernel<2>, bd, kCtrAccum, s, K_ACCUM);
    else launch_tiles(dev::accumulate_kernel<0>, bd, kCtrAccum, s, K_ACCUM);
}

}  // namespace vxr

// ---- converged reference and error metric ----------------------------------------------
namespace vxr {
namespace dev {

// FP64 running sum of the shaded frame's rgb (converged reference render).
__global__ void __launch_bounds__(256) sum64_add_kernel(const float4* __restrict__ frame, double* __restrict__ sum,
                                                        uint32_t n) {
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        const float4 f = frame[i];
        sum[3 * (size_t)i + 0] += (double)f.x;
        sum[3 * (size_t)i + 1] += (double)f.y;
        sum[3 * (size_t)i + 2] += (double)f.z;
    }
}

// CalculateMSE / CalculateRMAE (mse.cpp:33-65): the ground truth is the FP64 mean
// rounded to float (the reference compares float images); per pixel the squared and
// absolute channel errors are summed in float as mse.cpp does, then accumulated in FP64.
__global__ void __launch_bounds__(256) error_kernel(const float4* __restrict__ img, const double* __restrict__ sum,
                                                    double inv_count, uint32_t n, double* out) {
    double se = 0.0, ae = 0.0;
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        const float4 x = img[i];
        const float gx = (float)(sum[3 * (size_t)i + 0] * inv_count);
        const float gy = (float)(sum[3 * (size_t)i + 1] * inv_count);
        const float gz = (float)(sum[3 * (size_t)i + 2] * inv_count);
        const float dx = gx - x.x, dy = gy - x.y, dz = gz - x.z;
        se += (double)((dx * dx + dy * dy) + dz * dz);
        ae += (double)((fabsf(dx) + fabsf(dy)) + fabsf(dz));
    }
    for (int o = 16; o > 0; o >>= 1) {
        se += __shfl_down_sync(0xffffffffu, se, o);
        ae += __shfl_down_sync(0xffffffffu, ae, o);
    }
    __shared__ double s_se[8], s_ae[8];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    if (lane == 0) { s_se[warp] = se; s_ae[warp] = ae; }
    __syncthreads();
    if (threadIdx.x == 0) {
        double a = 0.0, b = 0.0;
        for (int i = 0; i < (int)(blockDim.x >> 5); i++) { a += s_se[i]; b += s_ae[i]; }
        atomicAdd(&out[0], a);
        atomicAdd(&out[1], b);
    }
}

}  // namespace dev

void launch_sum64_add(const float4* frame, double* sum, uint32_t n, cudaStream_t s) {
    dev::sum64_add_kernel<<<list_blocks(n, 256, 8), 256, 0, s>>>(frame, sum, n);
}

void launch_error(const float4* img, const double* sum, double inv_count, uint32_t n, double* out, cudaStream_t s) {
    dev::error_kernel<<<list_blocks(n, 256, 4), 256, 0, s>>>(img, sum, inv_count, n, out);
}

}  // namespace vxr
