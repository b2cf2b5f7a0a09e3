// Fused RGB-D TSDF integration for sm_100a: block allocation from a depth frame
// and the running weighted average of sdf / colour / weight per cell.
//
// It replaces the ~40 torch launches per frame of TSDFFusion.fuse_frame
// (demo/rgbd_fusion.py:199-254) and project_points_to_rgbd (:76-110), the temporary
// hash set of SparseDenseGrid.spatial_init_ (ash/grid.py:121-159) and the
// third-party depth unprojection (demo/rgbd_fusion.py:57-74) with two launches and
// no host synchronisation:
//
//   touch     one CTA per 32 x 16 pixels: unproject with the pinhole model, take the
//             block of each point, and for every block of the (2*dilation+1)^3
//             neighbourhood insert-if-absent into the grid's hash table, record the
//             block coordinate and stamp the block as touched by this frame.  Blocks
//             and neighbours that repeat within the CTA are dropped in shared memory.
//   integrate resident CTAs walk the compact list of touched blocks (without a list: one CTA
//             per embedding row, those of untouched rows exit at once).  The 10 KB of a block (512
//             cells x 5 floats) come into shared memory by bulk copies (by 16-byte loads where
//             rows do not allow them), every cell is projected into the frame and fused, and
//             the block leaves the same way.
//
// A sequence goes in batches of frames: the allocation pass marks which frames touch each block and the
// fusion pass applies them to a block in their order.
#include <algorithm>
#include <cmath>
#include <mutex>

#include "hashmap.cuh"

// Scratch of ashb_tsdf_fuse_frame_static: per block one stamp word and one int32x3
// coordinate.  It lives in the library image, so no allocation is ever made for it; every
// GPU that loads the library holds these bytes until the process exits.
#define ASHB_TSDF_STATIC_MAX_BLOCKS 262144
static __device__ __align__(256) unsigned char g_tsdf_static_scratch[ASHB_TSDF_STATIC_MAX_BLOCKS * 16];

namespace ashb {

// A frame as one of the two passes sees it.
struct View {
    float K[9];     // intrinsic, row major
    float pose[12]; // rows of [R | t]: camera -> world for the allocation, world -> camera for the fusion
    const float* depth;
    const float* color;
};

// Frames of one launch.  A sequence goes in batches of this many (a bit each in a block's word): a launch of one frame spends
// more time starting and running dry than at work (a 640 x 480 frame is 3,400 blocks for 1,184 resident CTAs), and a
// block that several frames see is loaded and stored once.  100 frames of 640 x 480: 35 us a frame with the allocation
// beside the fusion of the frame before on a second stream; in batches of 8, 16, 32: 25.6, 23.5, 22.3.
constexpr int kBatch = 32;
template <int N>
struct Views {
    View view[N];
};

// Every product and sum below is individually rounded (no fused multiply-add), so the
// block a point falls in and the pixel a cell projects to are bit-reproducible.
__device__ __forceinline__ float affine3(const float* r, float x, float y, float z) {
    return __fadd_rn(__fadd_rn(__fadd_rn(__fmul_rn(r[0], x), __fmul_rn(r[1], y)), __fmul_rn(r[2], z)), r[3]);
}
__device__ __forceinline__ float dot3(const float* r, float x, float y, float z) {
    return __fadd_rn(__fadd_rn(__fmul_rn(r[0], x), __fmul_rn(r[1], y)), __fmul_rn(r[2], z));
}

// ---- touch -------------------------------------------------------------------------
struct TouchTarget {
    int32_t* heap;
    int32_t* counter;
    int32_t capacity;
    int lo_off, hi_off;  // neighbourhood offsets per axis: [-dilation, dilation] or [0, dilation]
    int3 lo, hi;         // admissible block coordinates (half open) when bounded
    int bounded;
    int32_t* grid_coords;
    uint32_t* touched;
    uint32_t stamp;
    int32_t* touched_list;
    int32_t* touched_count;
    uint32_t* frames;   // of a batch: bit f of a block's word is set when frame f touches it; null for a single frame
};

// Row of a block that another thread of this launch is inserting, once that thread has published it; -1 when it found no
// free row.  The owner waits for nothing between its claim and the row; the wait is bounded all the same.
__device__ __noinline__ int index_of_pending(const Table16& t, int kx, int ky, int kz) {
    uint32_t s = hash_key(kx, ky, kz, 0) & t.mask, probe = 0;
    for (int spin = 0; probe <= t.mask;) {
        const Entry e = t.read_fresh(s);
        if (e.val == kEmpty) return -1;
        if (e.val != kTomb && key_match(e, kx, ky, kz, 0)) {
            if (e.val >= 0) return e.val;
            if (++spin == kSpinLimit) {
                atomicOr(t.status, ASHB_STATUS_SPIN);
                return -1;
            }
            continue;
        }
        s = (s + 1) & t.mask;
        ++probe;
    }
    return -1;
}

// Insert-if-absent of block (kx, ky, kz), its coordinate recorded and its stamp (of a batch: the bit of `frame`) set;
// appended to the compact list by the first toucher of the call.
template <bool BATCH>
__device__ __forceinline__ void touch_block(const Table16& t, const TouchTarget& tt, int kx, int ky, int kz, int frame) {
    if (tt.bounded && (kx < tt.lo.x || ky < tt.lo.y || kz < tt.lo.z || kx >= tt.hi.x || ky >= tt.hi.y || kz >= tt.hi.z))
        return;
    // fast path: the block exists already (probe at L2: this launch mutates the table)
    int idx = -1;
    {
        uint32_t s = hash_key(kx, ky, kz, 0) & t.mask;
        for (uint32_t probe = 0; probe <= t.mask; ++probe) {
            const Entry e = t.read_fresh(s);
            if (e.val == kEmpty) break;
            if (e.val >= 0 && key_match(e, kx, ky, kz, 0)) {
                idx = e.val;
                break;
            }
            s = (s + 1) & t.mask;
        }
    }
    if (idx < 0) {
        bool present = false;
        const int64_t slot = emplace(t, kx, ky, kz, 0, kPending, &present);
        if (slot < 0) {
            // another thread of this launch owns it and stamps it -- for its own frame
            if (!BATCH || !present) return;
            idx = index_of_pending(t, kx, ky, kz);
            if (idx < 0) return;
        } else {
            const int top = atomicAdd(tt.counter, 1);
            if (top >= tt.capacity) {
                atomicSub(tt.counter, 1);
                *reinterpret_cast<volatile int*>(t.val_ptr((uint32_t)slot)) = kTomb;
                atomicOr(t.status, ASHB_STATUS_CAPACITY);
                return;
            }
            idx = tt.heap[top];
            *reinterpret_cast<volatile int*>(t.val_ptr((uint32_t)slot)) = idx;
        }
    }
    // many pixels of a frame fall in the same few thousand blocks: whoever finds the block already
    // stamped by this call has nothing left to do (the first toucher recorded it)
    const uint32_t bit = 1u << frame;
    if (BATCH ? (__ldcg(&tt.frames[idx]) & bit) != 0u : __ldcg(&tt.touched[idx]) == tt.stamp) return;
    // the coordinate is recorded for blocks allocated by other means too
    tt.grid_coords[3 * idx] = kx;
    tt.grid_coords[3 * idx + 1] = ky;
    tt.grid_coords[3 * idx + 2] = kz;
    if (BATCH) {
        if (atomicOr(&tt.frames[idx], bit) == 0u) tt.touched_list[atomicAdd(tt.touched_count, 1)] = idx;
    } else if (tt.touched_list) {
        // first toucher of the call appends the block to the compact work list
        if (atomicExch(&tt.touched[idx], tt.stamp) != tt.stamp) tt.touched_list[atomicAdd(tt.touched_count, 1)] = idx;
    } else {
        tt.touched[idx] = tt.stamp;
    }
}

// The blocks that the points of a CTA fall in, and the neighbours that were already taken care of.
// A tile of pixels sees a handful of blocks whose neighbourhoods are mostly the same ones; probing each
// neighbour of each block of each WARP's 32 pixels was 780,000 probes of a 640 x 480 frame where
// 3,500 blocks are touched.  The pass is a chain of L2 round trips: what it costs is probes per thread.
// 21.1 -> 7.4 us for that frame into a volume that holds its blocks.
constexpr int kTouchPoints = 512;   // points of a CTA of 256 threads
constexpr int kSeenSlots = 2048;
struct TouchTile {
    uint32_t seen[kSeenSlots];
    int3 blocks[kTouchPoints];
    int n_blocks;
    int has_origin;
    int3 origin;
};

// False when `word` (not 0) is in the set already.  In a crowded set it gives up and says true: touching a
// block twice costs time only.
__device__ __forceinline__ bool first_seen(uint32_t* seen, uint32_t word) {
    uint32_t s = (word * 0x9E3779B1u) >> 21;
#pragma unroll 1
    for (int k = 0; k < 8; ++k) {
        const uint32_t old = atomicCAS(seen + s, 0u, word);
        if (old == 0u) return true;
        if (old == word) return false;
        s = (s + 1) & (kSeenSlots - 1);
    }
    return true;
}

// Offset from the tile's origin as one word, or 0 when an axis is too far off.  `tag` keeps the two uses apart.
__device__ __forceinline__ uint32_t tile_word(const int3& o, int x, int y, int z, uint32_t tag) {
    const uint32_t dx = (uint32_t)x - (uint32_t)o.x + 512u, dy = (uint32_t)y - (uint32_t)o.y + 512u,
                   dz = (uint32_t)z - (uint32_t)o.z + 512u;
    return (dx | dy | dz) < 1024u ? dx | dy << 10 | dz << 20 | tag : 0u;
}

// Points in any order are a block each: 512 x 27 neighbours that the set is too small for, and that it costs more to ask than
// to probe.  From this many blocks on, warps take blocks and their lanes the neighbours as they come: spatial_init_ of
// 100k points in a cube with 27 and 125 neighbours 212 -> 130 and 518 -> 235 us.  The pixels of
// a frame are not in any order: it keeps to the set (small voxels, 140k blocks: 80 us with it, 90 without).
constexpr int kCrowded = 64;

// Called by ALL 256 threads of a CTA, each with two points (`valid` ones carry a block), in no order if SCATTERED.
// `slices` (a power of two) CTAs may be given the same points: `slice` of them takes the blocks whose coordinates say so.
template <bool SCATTERED, bool BATCH>
__device__ __forceinline__ void touch_neighbourhoods(const Table16& t, const TouchTarget& tt, const bool* valid,
                                                     const int3* block, unsigned slices, unsigned slice, int frame) {
    constexpr uint32_t kOwnTag = 1u << 30, kNeighbourTag = 1u << 31;
    __shared__ TouchTile tile;
    for (int i = threadIdx.x; i < kSeenSlots; i += 256) tile.seen[i] = 0u;
    if (threadIdx.x == 0) tile.n_blocks = tile.has_origin = 0;
    __syncthreads();
    bool ok[2];
#pragma unroll
    for (int j = 0; j < 2; ++j) {
        const int3 b = block[j];
        // a point whose own block is out of bounds contributes nothing (ash/grid.py:134-135)
        ok[j] = valid[j] && !(tt.bounded && (b.x < tt.lo.x || b.y < tt.lo.y || b.z < tt.lo.z || b.x >= tt.hi.x ||
                                             b.y >= tt.hi.y || b.z >= tt.hi.z));
        const unsigned any = __ballot_sync(0xffffffffu, ok[j]);
        if (any && (int)(threadIdx.x & 31) == __ffs(any) - 1 && atomicExch(&tile.has_origin, 1) == 0) tile.origin = b;
    }
    __syncthreads();
    if (!tile.has_origin) return;
    const int3 o = tile.origin;
#pragma unroll
    for (int j = 0; j < 2; ++j) {
        const int3 b = block[j];
        const uint32_t word = ok[j] ? tile_word(o, b.x, b.y, b.z, kOwnTag) : 0u;
        // one lane per distinct block of the warp asks the set
        const unsigned peers = __match_any_sync(0xffffffffu, word);
        const bool ask = ok[j] && (word == 0u || (int)(threadIdx.x & 31) == __ffs(peers) - 1) &&
                         (((unsigned)b.x + 3u * (unsigned)b.y + 5u * (unsigned)b.z) & (slices - 1)) == slice;
        if (ask && (word == 0u || first_seen(tile.seen, word))) tile.blocks[atomicAdd(&tile.n_blocks, 1)] = b;
    }
    __syncthreads();
    const int w = tt.hi_off - tt.lo_off + 1, n_nb = w * w * w;
    if (SCATTERED && w > 2 && tile.n_blocks > kCrowded) {
        for (int which = threadIdx.x >> 5; which < tile.n_blocks; which += 8) {
            const int3 b = tile.blocks[which];
            for (int k = threadIdx.x & 31; k < n_nb; k += 32)
                touch_block<BATCH>(t, tt, b.x + tt.lo_off + k % w, b.y + tt.lo_off + (k / w) % w, b.z + tt.lo_off + k / (w * w),
                                   frame);
            __syncwarp();
        }
        return;
    }
    const int n = tile.n_blocks * n_nb;
    for (int i = threadIdx.x; i < n; i += 256) {
        const int which = i / n_nb, k = i - which * n_nb;
        const int x = tile.blocks[which].x + tt.lo_off + k % w, y = tile.blocks[which].y + tt.lo_off + (k / w) % w,
                  z = tile.blocks[which].z + tt.lo_off + k / (w * w);
        const uint32_t word = tile_word(o, x, y, z, kNeighbourTag);
        if (word == 0u || first_seen(tile.seen, word)) touch_block<BATCH>(t, tt, x, y, z, frame);
    }
}

// world -> cell -> block as the Python layer does on a CUDA tensor: multiply by the float
// reciprocals (ash/grid.py:132-134, :756, :846)
__device__ __forceinline__ int block_of(float w, float org, float inv_cell, float inv_G) {
    return (int)floorf(__fmul_rn(__fmul_rn(__fsub_rn(w, org), inv_cell), inv_G));
}

// CTAs (x, f) are those of frame f of the N of a batch.
template <int N>
__global__ void __launch_bounds__(256, 6) tsdf_touch_kernel(Table16 t, TouchTarget tt, const __grid_constant__ Views<N> views,
                                                            int H, int W, float depth_max, float inv_cell, float3 origin,
                                                            float inv_G) {
    const View& cam = views.view[N == 1 ? 0 : blockIdx.y];
    bool valid[2];
    int3 block[2];
    const unsigned tiles_x = ((unsigned)W + 31) / 32;
    const int u = (int)(blockIdx.x % tiles_x) * 32 + (int)(threadIdx.x & 31);
#pragma unroll
    for (int j = 0; j < 2; ++j) {
        const int v = (int)(blockIdx.x / tiles_x) * 16 + j * 8 + (int)(threadIdx.x >> 5);
        const float d = u < W && v < H ? __ldg(cam.depth + (int64_t)v * W + u) : 0.f;
        valid[j] = d > 0.f && d < depth_max;
        block[j] = make_int3(0, 0, 0);
        if (valid[j]) {
            // camera point of pixel (u, v) at depth d for K = [fx 0 cx; 0 fy cy; 0 0 1]
            const float xc = __fdiv_rn(__fmul_rn(__fsub_rn((float)u, cam.K[2]), d), cam.K[0]);
            const float yc = __fdiv_rn(__fmul_rn(__fsub_rn((float)v, cam.K[5]), d), cam.K[4]);
            block[j] = make_int3(block_of(affine3(cam.pose, xc, yc, d), origin.x, inv_cell, inv_G),
                                 block_of(affine3(cam.pose + 4, xc, yc, d), origin.y, inv_cell, inv_G),
                                 block_of(affine3(cam.pose + 8, xc, yc, d), origin.z, inv_cell, inv_G));
        }
    }
    touch_neighbourhoods<false, (N > 1)>(t, tt, valid, block, 1, 0, N == 1 ? 0 : (int)blockIdx.y);
}

// SparseDenseGrid.spatial_init_ (ash/grid.py:121-159) without its temporary hash set: two points per thread.
__global__ void __launch_bounds__(256, 6) points_touch_kernel(Table16 t, TouchTarget tt, const float* __restrict__ pts,
                                                              int64_t n, float inv_cell, float3 origin, float inv_G) {
    bool valid[2];
    int3 block[2];
#pragma unroll
    for (int j = 0; j < 2; ++j) {
        const int64_t i = (int64_t)blockIdx.x * kTouchPoints + j * 256 + threadIdx.x;
        valid[j] = i < n;
        block[j] = make_int3(0, 0, 0);
        if (valid[j])
            block[j] = make_int3(block_of(pts[3 * i], origin.x, inv_cell, inv_G),
                                 block_of(pts[3 * i + 1], origin.y, inv_cell, inv_G),
                                 block_of(pts[3 * i + 2], origin.z, inv_cell, inv_G));
    }
    touch_neighbourhoods<true, false>(t, tt, valid, block, gridDim.y, blockIdx.y, 0);
}

// ---- integrate ---------------------------------------------------------------------
// Bound by instructions (205 a cell and view) and by the latency of the image loads.  A thread has four cells of a column in
// flight: 100 frames 2235 us in all, 2290 with two or one.
constexpr int kIntegrateSlots = 1024, kCellGroup = 4;   // threads of an SM, cells of a thread in flight

// Threads of a CTA whose tiles take `bytes`: few CTAs fit an SM where the tiles are large, so each takes more threads.  16
// frames of 640 x 480 at 128, 256, 512 threads: block edge 10 (five CTAs fit) 726, 666, 816 us, edge 12 (three) 1390, 1130,
// 1216, edge 16 (two) 4930, 3500, 2640; edge 8 with 8 channels (six) 485, 505, 660, with 13 (four) 615, 600, 630, with 16
// (three) 810, 828, 930, but a single frame of these 84, 80, 88 us: a batch has the frames of a block to overlap.
// pitch: pixels between neighbouring cells at the largest depth, or nearly.  From two on a cell reads image lines of its own,
// and a single frame waits for them: 256 threads, six CTAs an SM.  Whole frames of 640 columns at 128 and 256 threads, means:
// pitch 3.2 23.6 and 20.1 us, 2.1 27.0 and 24.4, 1.6 30.5 and 29.8 (single ones 7 % slower), of 320 columns at 1.1 23.2
// and 23.7, of 160 at 0.5 25.6 and 26.8.
static int integrate_threads(size_t bytes, int G, bool batch, float pitch) {
    constexpr size_t kSharedOfSm = 228 * 1024, kSharedOfCta = 1024;   // what a CTA takes beside its own
    const int fit = (int)(kSharedOfSm / (bytes + kSharedOfCta));
    if (G == 8) return batch || (fit >= 6 && !(pitch >= 2.f)) ? 128 : 256;
    return fit >= 6 ? 128 : fit >= 3 ? 256 : 512;
}
constexpr float kRound = 12582912.f;   // 1.5 * 2^23

struct IntegrateFrame {
    int H, W;
    float depth_max, cell_size;
    float3 origin;
    int G, cells;
    float trunc;
    int sdf_ch, rgb_ch, w_ch;
    int D;
    int G_shift;   // log2(G), or -1
    float u_end, v_end;   // W and H above kRound
    int usual;   // every intrinsic is [fx 0 cx; 0 fy cy; 0 0 1], and W and H are at most 2^22
    uint32_t* frames;   // of a batch: which frames touched a block, set back to none here; null for a single frame
    uint32_t* touched;  // of a batch: a block is given the stamp of its last frame
    uint32_t first_stamp;
};

// What a view observes at a cell.
struct Observation {
    float d, depth, r, g, b;
    bool seen;
};

// The pixel that camera coordinates (x, y, z) project to, and its loads.  USUAL: see IntegrateFrame; the general product
// gives the same pixels, as products with the intrinsic's zeros change no sum that passes the tests below.
template <bool USUAL>
__device__ __forceinline__ Observation observe(float x, float y, float z, const IntegrateFrame& f, const View& view) {
    Observation o{z, 0.f, 0.f, 0.f, 0.f, false};
    float un, vn;
    int u = 0, v = 0;
    if (USUAL) {
        un = __fadd_rn(__fmul_rn(view.K[0], x), __fmul_rn(view.K[2], z));
        vn = __fadd_rn(__fmul_rn(view.K[4], y), __fmul_rn(view.K[5], z));
    } else {
        un = dot3(view.K, x, y, z);
        vn = dot3(view.K + 3, x, y, z);
        o.d = dot3(view.K + 6, x, y, z);
    }
    // torch.round of the quotients: half to even.  A numerator beyond what the shared division is exact for has a quotient that
    // rounds to 0, or beyond every image, either way.  Adding kRound rounds and leaves the whole number in the low
    // bits where it is below 2^22 (conversions run at a quarter of the rate).
    const SharedDivisor by(o.d);
    if (USUAL && by.plain) {
        const float um = __fadd_rn(by.quotient(un), kRound), vm = __fadd_rn(by.quotient(vn), kRound);
        o.seen = um >= kRound && vm >= kRound && um < f.u_end && vm < f.v_end;
        u = __float_as_int(um) - __float_as_int(kRound), v = __float_as_int(vm) - __float_as_int(kRound);
    } else if (o.d > 0.f) {
        const float uf = rintf(__fdiv_rn(un, o.d)), vf = rintf(__fdiv_rn(vn, o.d));
        o.seen = uf >= 0.f && vf >= 0.f && uf < (float)f.W && vf < (float)f.H;
        u = (int)uf, v = (int)vf;
    }
    if (o.seen) {
        const int64_t pixel = (int64_t)v * f.W + u;
        const float* color = view.color + pixel * 3;
        o.depth = __ldg(view.depth + pixel);
        o.r = __ldg(color), o.g = __ldg(color + 1), o.b = __ldg(color + 2);
    }
    return o;
}

// The observation fused into its cell (D floats at `cell`).
__device__ __forceinline__ void fuse_cell(float* cell, const Observation& o, const IntegrateFrame& f) {
    // outside the image or behind the camera the observation has weight 0 and its
    // value does not matter (demo/rgbd_fusion.py:93-108)
    float w = 0.f, sdf = 0.f;
    if (o.seen) {
        sdf = __fsub_rn(o.depth, o.d);
        if (o.depth > 0.f && o.depth < f.depth_max && sdf >= -f.trunc) w = 1.f;
        if (sdf >= f.trunc) sdf = f.trunc;
    }
    float* rgb = cell + f.rgb_ch;
    const float w_sum = cell[f.w_ch];
    // demo/rgbd_fusion.py:247-249: mean' = (mean * w_sum + obs * w) / (w_sum + w + 1e-6); obs * w is exact
    const float w_new = __fadd_rn(w_sum, w);
    const float den = __fadd_rn(w_new, 1e-6f);
    auto sum = [&](float mean, float obs) { return __fmaf_rn(obs, w, __fmul_rn(mean, w_sum)); };
    float mean[4] = {sum(cell[f.sdf_ch], sdf), sum(rgb[0], o.r), sum(rgb[1], o.g), sum(rgb[2], o.b)};
    // A cell that no frame has observed has sums of zero, and zero over a positive number keeps its sign.
    if (!(all_zero(mean[0], mean[1], mean[2], mean[3]) && den > 0.f)) SharedDivisor(den).divide(mean);
    cell[f.sdf_ch] = mean[0];
    rgb[0] = mean[1];
    rgb[1] = mean[2];
    rgb[2] = mean[3];
    cell[f.w_ch] = w_new;
}

// One view fused into every cell of block (gx, gy, gz), whose rows sit in `tile` (cells * D floats).
// GT: the block edge where it is known when compiling, 0 otherwise.  T: threads of the CTA.  Where these cover whole
// layers of the block (GT of 4, 8) a thread stays in one column of cells and the x and y parts of its camera
// coordinates are formed once.
template <int GT, int T, bool USUAL>
__device__ __forceinline__ void integrate_cells(float* tile, int gx, int gy, int gz, const IntegrateFrame& f, const View& view) {
    constexpr int kLayers = GT ? T / (GT * GT) : 0;   // that the CTA covers at once
    const int G = GT ? GT : f.G;
    // cell_to_world: (block * G + cell) * cell_size (+ origin for bounded grids)
    auto world = [&](int b, int c, float origin) { return __fadd_rn(__fmul_rn((float)(b * G + c), f.cell_size), origin); };
    const float* E = view.pose;
    if constexpr (kLayers > 0) {
        constexpr int kEach = GT / kLayers > 0 ? GT / kLayers : 1, kGroup = kEach < kCellGroup ? kEach : kCellGroup;
        const int t = threadIdx.x, cx = t % G, cy = t / G % G, cz0 = t / (G * G);
        if (cz0 >= G) return;
        const float px = world(gx, cx, f.origin.x), py = world(gy, cy, f.origin.y);
        float xy[3];   // affine3 as far as it does not depend on z
#pragma unroll
        for (int k = 0; k < 3; ++k) xy[k] = __fadd_rn(__fmul_rn(E[4 * k], px), __fmul_rn(E[4 * k + 1], py));
#pragma unroll 1
        for (int j = 0; j < kEach; j += kGroup) {
            Observation o[kGroup];
#pragma unroll
            for (int i = 0; i < kGroup; ++i) {
                const float pz = world(gz, cz0 + (j + i) * kLayers, f.origin.z);
                float p[3];
#pragma unroll
                for (int k = 0; k < 3; ++k) p[k] = __fadd_rn(__fadd_rn(xy[k], __fmul_rn(E[4 * k + 2], pz)), E[4 * k + 3]);
                o[i] = observe<USUAL>(p[0], p[1], p[2], f, view);
            }
#pragma unroll
            for (int i = 0; i < kGroup; ++i) fuse_cell(tile + (t + (j + i) * T) * f.D, o[i], f);
        }
    } else {
        for (int c = threadIdx.x; c < f.cells; c += blockDim.x) {
            int cx, cy, cz;
            if (f.G_shift >= 0) {   // three divisions would be a quarter of a cell's instructions
                cx = c & (G - 1), cy = (c >> f.G_shift) & (G - 1), cz = c >> (2 * f.G_shift);
            } else {
                cx = c % G, cy = (c / G) % G, cz = c / (G * G);
            }
            const float px = world(gx, cx, f.origin.x), py = world(gy, cy, f.origin.y), pz = world(gz, cz, f.origin.z);
            fuse_cell(tile + c * f.D,
                      observe<USUAL>(affine3(E, px, py, pz), affine3(E + 4, px, py, pz), affine3(E + 8, px, py, pz), f, view), f);
        }
    }
}

// The frames of `frames` in their order.  A thread's cells are its own: nothing to wait for between two frames.
template <int GT, int N, int T>
__device__ __forceinline__ void fuse_frames(float* tile, const int32_t* coords, uint32_t frames, const IntegrateFrame& f,
                                            const Views<N>& views) {
    const int gx = coords[0], gy = coords[1], gz = coords[2];
#pragma unroll 1
    for (; frames; frames &= frames - 1) {
        const View& view = views.view[N == 1 ? 0 : __ffs(frames) - 1];
        if (f.usual) integrate_cells<GT, T, true>(tile, gx, gy, gz, f, view);
        else integrate_cells<0, T, false>(tile, gx, gy, gz, f, view);
        if (N == 1) break;
    }
}

// One thread, after the CTA has read the block's word.
__device__ __forceinline__ void finish_block(int64_t idx, uint32_t frames, const IntegrateFrame& f, unsigned long long* n_integrated) {
    if (f.frames) {
        f.frames[idx] = 0u;
        f.touched[idx] = f.first_stamp + (31 - __clz(frames));
    }
    if (n_integrated) atomicAdd(n_integrated, (unsigned long long)__popc(frames));
}

template <int GT, int N, int T>
__global__ void __launch_bounds__(T, kIntegrateSlots / T) tsdf_integrate_kernel(
        float* __restrict__ emb, const int32_t* __restrict__ grid_coords, const uint32_t* __restrict__ touched,
        uint32_t stamp, const __grid_constant__ IntegrateFrame f, const __grid_constant__ Views<N> views,
        unsigned long long* n_integrated, int64_t n_emb, const int32_t* __restrict__ touched_list,
        const int32_t* __restrict__ touched_count) {
    extern __shared__ float tile[];  // cells * D floats
    // Work items: the compact list written by the touch kernel (a few persistent CTAs walk it),
    // or, without a list, every embedding row whose stamp matches (one CTA per row).
    const int64_t n_items = touched_list ? (int64_t)*touched_count : n_emb;
    for (int64_t item = blockIdx.x; item < n_items; item += gridDim.x) {
        const int64_t idx = touched_list ? (int64_t)touched_list[item] : item;
        if (!touched_list && touched[idx] != stamp) continue;
        const int n_float = f.cells * f.D;
        float* block = emb + idx * (int64_t)n_float;
        // rows are 16-byte aligned when cells * D * 4 is a multiple of 16
        const bool vec_ok = (n_float & 3) == 0 && (((uintptr_t)block) & 15) == 0;
        if (vec_ok) {
            for (int i = threadIdx.x; i < n_float / 4; i += blockDim.x)
                reinterpret_cast<float4*>(tile)[i] = reinterpret_cast<const float4*>(block)[i];
        } else {
            for (int i = threadIdx.x; i < n_float; i += blockDim.x) tile[i] = block[i];
        }
        __syncthreads();
        const uint32_t frames = N > 1 ? f.frames[idx] : 1u;
        fuse_frames<GT, N, T>(tile, grid_coords + 3 * idx, frames, f, views);
        __syncthreads();
        if (threadIdx.x == 0) finish_block(idx, frames, f, n_integrated);
        if (vec_ok) {
            for (int i = threadIdx.x; i < n_float / 4; i += blockDim.x)
                reinterpret_cast<float4*>(block)[i] = reinterpret_cast<const float4*>(tile)[i];
        } else {
            for (int i = threadIdx.x; i < n_float; i += blockDim.x) block[i] = tile[i];
        }
        __syncthreads();  // the tile is reused by the next item
    }
}

// Number of waits of the bulk-copy variant below that ran out (0 in any healthy run): read with
// ashb_tsdf_copy_timeouts.
__device__ unsigned int g_tsdf_copy_timeouts = 0;

__device__ __forceinline__ uint32_t smem_address(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }

// Waits, with a limit, for phase `parity` of the mbarrier at `bar`; false when the limit ran out.
__device__ __forceinline__ bool wait_phase(uint32_t bar, uint32_t parity) {
    for (int spin = 0; spin < (1 << 18); ++spin) {
        uint32_t done;
        asm volatile(
                "{\n\t.reg .pred p;\n\t"
                "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
                "selp.u32 %0, 1, 0, p;\n\t}"
                : "=r"(done)
                : "r"(bar), "r"(parity)
                : "memory");
        if (done) return true;
    }
    return false;
}

// The same pass over a work list with the block rows moved by the copy engine: a persistent CTA keeps
// two tiles in shared memory; while it fuses the observation into one, the next block's rows arrive in
// the other (cp.async.bulk global -> shared, completion on an mbarrier) and the finished tile leaves
// as one bulk store (shared -> global), so loading, arithmetic and storing overlap instead of taking
// turns.  A block's rows are one contiguous, 16-byte aligned stretch of cells * D * 4 bytes (a multiple
// of 16: checked by the host).  Every wait has an iteration limit; a CTA whose wait runs out counts it
// in g_tsdf_copy_timeouts, waits for its own stores and stops.
template <int GT, int N, int T>
__global__ void __launch_bounds__(T, kIntegrateSlots / T) tsdf_integrate_bulk_kernel(
        float* __restrict__ emb, const int32_t* __restrict__ grid_coords, const __grid_constant__ IntegrateFrame f,
        const __grid_constant__ Views<N> views, unsigned long long* n_integrated, const int32_t* __restrict__ touched_list,
        const int32_t* __restrict__ touched_count) {
    extern __shared__ __align__(128) float tiles[];  // 2 tiles of cells * D floats
    __shared__ __align__(8) unsigned long long full[2];
    const int n_float = f.cells * f.D;
    const uint32_t bytes = (uint32_t)n_float * 4u;
    const int64_t n_items = (int64_t)*touched_count;
    const bool boss = threadIdx.x == 0;
    if (boss) {
        asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(smem_address(&full[0])) : "memory");
        asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(smem_address(&full[1])) : "memory");
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    __syncthreads();
    auto fetch = [&](int64_t item, int buf) {   // thread 0 only
        const float* src = emb + (int64_t)touched_list[item] * n_float;
        const uint32_t bar = smem_address(&full[buf]);
        asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
        asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
                             smem_address(tiles + (int64_t)buf * n_float)),
                     "l"(src), "r"(bytes), "r"(bar)
                     : "memory");
    };
    if (boss && (int64_t)blockIdx.x < n_items) fetch(blockIdx.x, 0);
    int round = 0;
    for (int64_t item = blockIdx.x; item < n_items; item += gridDim.x, ++round) {
        const int buf = round & 1;
        const int64_t next = item + gridDim.x;
        if (boss && next < n_items) {
            // the other tile was handed to a bulk store one round ago: it may be refilled once that store has read it
            asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory");
            fetch(next, buf ^ 1);
        }
        const bool arrived = wait_phase(smem_address(&full[buf]), (uint32_t)(round >> 1) & 1u);
        if (!__syncthreads_and(arrived)) {
            if (boss) {
                atomicAdd(&g_tsdf_copy_timeouts, 1u);
                // the copy already requested for the next round must not land in a dead CTA's memory
                if (next < n_items) wait_phase(smem_address(&full[buf ^ 1]), (uint32_t)((round + 1) >> 1) & 1u);
            }
            break;
        }
        float* tile = tiles + (int64_t)buf * n_float;
        const int64_t idx = touched_list[item];
        const uint32_t frames = N > 1 ? f.frames[idx] : 1u;
        fuse_frames<GT, N, T>(tile, grid_coords + 3 * idx, frames, f, views);
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");   // the tile as written, visible to the copy engine
        __syncthreads();
        if (boss) {
            asm volatile("cp.async.bulk.global.shared::cta.bulk_group [%0], [%1], %2;" ::"l"(emb + idx * (int64_t)n_float),
                         "r"(smem_address(tile)), "r"(bytes)
                         : "memory");
            asm volatile("cp.async.bulk.commit_group;" ::: "memory");
            finish_block(idx, frames, f, n_integrated);
        }
    }
    if (boss) asm volatile("cp.async.bulk.wait_group 0;" ::: "memory");   // stores complete before the CTA's memory goes
}

}  // namespace ashb

using namespace ashb;

extern "C" {

static int make_touch_target(ashb_map* m, int dilation, int bidirectional, const int32_t* bound_lo,
                             const int32_t* bound_hi, int32_t* grid_coords, uint32_t* touched, uint32_t stamp,
                             int32_t* touched_list, int32_t* touched_count, TouchTarget* out) {
    ASHB_REQUIRE(m != nullptr && m->slots != nullptr, "null or destroyed map");
    ASHB_REQUIRE(m->key_dim == 3, "block allocation needs a 3-D map");
    ASHB_REQUIRE(grid_coords && touched, "null buffer");
    ASHB_REQUIRE(dilation >= 0 && dilation <= 4, "dilation %d not in 0..4", dilation);
    ASHB_REQUIRE(stamp != 0, "stamp 0 is reserved for 'never touched'");
    ASHB_REQUIRE((touched_list == nullptr) == (touched_count == nullptr),
                 "pass both the list and its counter, or neither");
    TouchTarget tt{};
    tt.heap = m->heap;
    tt.counter = m->counter;
    tt.capacity = (int32_t)m->capacity;
    tt.lo_off = bidirectional ? -dilation : 0;
    tt.hi_off = dilation;
    tt.bounded = bound_lo != nullptr && bound_hi != nullptr;
    if (tt.bounded) {
        tt.lo = make_int3(bound_lo[0], bound_lo[1], bound_lo[2]);
        tt.hi = make_int3(bound_hi[0], bound_hi[1], bound_hi[2]);
    }
    tt.grid_coords = grid_coords;
    tt.touched = touched;
    tt.stamp = stamp;
    tt.touched_list = touched_list;
    tt.touched_count = touched_count;
    *out = tt;
    return ASHB_OK;
}

// The allocation pass of n_frames frames (bits of the n_words `frames`, a counter behind them included; or a single one).
static int touch_impl(ashb_map* m, int n_frames, const float* const* depths, int H, int W, const float* intrinsics,
                      const float* cam_to_worlds, float depth_max, double cell_size, const float* origin, int G,
                      int dilation, const int32_t* bound_lo, const int32_t* bound_hi, int32_t* grid_coords,
                      uint32_t* touched, uint32_t stamp, int32_t* touched_list, int32_t* touched_count, uint32_t* frames,
                      int64_t n_words, void* stream) {
    TouchTarget tt;
    if (int rc = make_touch_target(m, dilation, 1, bound_lo, bound_hi, grid_coords, touched, stamp, touched_list,
                                   touched_count, &tt))
        return rc;
    tt.frames = frames;
    ASHB_REQUIRE(intrinsics && cam_to_worlds && origin, "null buffer");
    ASHB_REQUIRE(H > 0 && W > 0 && G > 0 && cell_size > 0.0, "bad frame or grid geometry");
    DeviceGuard guard(m->device);
    Views<kBatch> views;   // the first n_frames are set
    for (int f = 0; f < n_frames; ++f) {
        View& v = views.view[f];
        for (int i = 0; i < 9; ++i) v.K[i] = intrinsics[9 * f + i];
        for (int i = 0; i < 12; ++i) v.pose[i] = cam_to_worlds[12 * f + i];
        v.depth = depths[f];
        ASHB_REQUIRE(v.depth != nullptr, "null buffer");
        ASHB_REQUIRE(v.K[0] != 0.f && v.K[4] != 0.f && v.K[1] == 0.f && v.K[3] == 0.f,
                     "intrinsic must be a skew-free pinhole matrix");
    }
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    // The fusion pass takes back every word of `frames` that it works off; one of a CTA whose copies ran out would stay, and
    // its block would not be listed again: zeros for every batch.  A counter right behind the words is cleared with them (100
    // frames of a volume of 160,000 blocks: 7 us less than by two fills a batch).
    if (frames) ASHB_CUDA_TRY(cudaMemsetAsync(frames, 0, (size_t)n_words * sizeof(uint32_t), st));
    if (touched_count && !(frames && reinterpret_cast<uint32_t*>(touched_count) == frames + n_words - 1))
        ASHB_CUDA_TRY(cudaMemsetAsync(touched_count, 0, sizeof(int32_t), st));
    const dim3 grid((unsigned)(((int64_t)W + 31) / 32 * (((int64_t)H + 15) / 16)), (unsigned)n_frames);
    const float3 org = make_float3(origin[0], origin[1], origin[2]);
    const float inv_cell = (float)(1.0 / cell_size), inv_G = 1.0f / (float)G;
    if (frames)
        tsdf_touch_kernel<kBatch><<<grid, 256, 0, st>>>(table16_of(m), tt, views, H, W, depth_max, inv_cell, org, inv_G);
    else
        tsdf_touch_kernel<1><<<grid, 256, 0, st>>>(table16_of(m), tt, Views<1>{{views.view[0]}}, H, W, depth_max, inv_cell,
                                                   org, inv_G);
    ASHB_LAUNCH_CHECK();
    return ASHB_OK;
}

int ashb_tsdf_touch(ashb_map* m, const float* depth, int H, int W, const float* intrinsic,
                    const float* cam_to_world, float depth_max, double cell_size, const float* origin, int G,
                    int dilation, const int32_t* bound_lo, const int32_t* bound_hi, int32_t* grid_coords,
                    uint32_t* touched, uint32_t stamp, int32_t* touched_list, int32_t* touched_count,
                    void* stream) {
    return touch_impl(m, 1, &depth, H, W, intrinsic, cam_to_world, depth_max, cell_size, origin, G, dilation, bound_lo,
                      bound_hi, grid_coords, touched, stamp, touched_list, touched_count, nullptr, 0, stream);
}

int ashb_grid_spatial_init(ashb_map* m, const float* points, int64_t n, double cell_size, const float* origin, int G,
                           int dilation, int bidirectional, const int32_t* bound_lo, const int32_t* bound_hi,
                           int32_t* grid_coords, uint32_t* touched, uint32_t stamp, int32_t* touched_list,
                           int32_t* touched_count, void* stream) {
    TouchTarget tt;
    if (int rc = make_touch_target(m, dilation, bidirectional, bound_lo, bound_hi, grid_coords, touched, stamp,
                                   touched_list, touched_count, &tt))
        return rc;
    ASHB_REQUIRE(n >= 0 && G > 0 && cell_size > 0.0, "bad point count or grid geometry");
    DeviceGuard guard(m->device);
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    if (touched_count) ASHB_CUDA_TRY(cudaMemsetAsync(touched_count, 0, sizeof(int32_t), st));
    if (n == 0) return ASHB_OK;
    ASHB_REQUIRE(points != nullptr, "null points");
    const float3 org = origin ? make_float3(origin[0], origin[1], origin[2]) : make_float3(0.f, 0.f, 0.f);
    // With less than a wave of CTAs the blocks of the same points are shared out among several: a chain of L2 round trips
    // per block, eight blocks side by side in a CTA.
    const unsigned ctas = (unsigned)((n + kTouchPoints - 1) / kTouchPoints);
    const int w = tt.hi_off - tt.lo_off + 1;
    unsigned slices = 1;
    while (w > 2 && slices < 8 && (int64_t)ctas * slices * 2 <= 6 * sm_count()) slices *= 2;
    points_touch_kernel<<<dim3(ctas, slices), 256, 0, st>>>(table16_of(m), tt, points, n, (float)(1.0 / cell_size), org,
                                                            1.0f / (float)G);
    ASHB_LAUNCH_CHECK();
    return ASHB_OK;
}

// The fusion pass of n_frames frames: the blocks of a batch's `frames` words, or those of a single stamp.
static int integrate_impl(void* embeddings, int64_t n_emb, int G, int64_t D, const int32_t* grid_coords,
                          uint32_t* touched, uint32_t stamp, int n_frames, const float* const* depths,
                          const float* const* colors, int H, int W, const float* intrinsics, const float* world_to_cams,
                          float depth_max, double cell_size, const float* origin, float trunc, int sdf_channel,
                          int rgb_channel, int weight_channel, unsigned long long* n_integrated_dev,
                          const int32_t* touched_list, const int32_t* touched_count, uint32_t* frames, void* stream) {
    ASHB_REQUIRE((touched_list == nullptr) == (touched_count == nullptr), "pass both the list and its counter, or neither");
    ASHB_REQUIRE(embeddings && grid_coords && touched && intrinsics && world_to_cams && origin, "null buffer");
    ASHB_REQUIRE(n_emb >= 1 && G >= 1 && G <= 16 && H > 0 && W > 0, "bad sizes");
    ASHB_REQUIRE(D >= 5 && D <= 16, "embedding_dim %lld cannot hold sdf + rgb + weight", (long long)D);
    ASHB_REQUIRE(sdf_channel >= 0 && sdf_channel < D && weight_channel >= 0 && weight_channel < D &&
                         rgb_channel >= 0 && rgb_channel + 2 < D,
                 "channel layout out of range");
    Views<kBatch> views;   // the first n_frames are set
    int usual = W <= 1 << 22 && H <= 1 << 22;
    for (int f = 0; f < n_frames; ++f) {
        View& v = views.view[f];
        for (int i = 0; i < 9; ++i) v.K[i] = intrinsics[9 * f + i];
        for (int i = 0; i < 12; ++i) v.pose[i] = world_to_cams[12 * f + i];
        v.depth = depths[f];
        v.color = colors[f];
        ASHB_REQUIRE(v.depth && v.color, "null buffer");
        usual &= v.K[1] == 0.f && v.K[3] == 0.f && v.K[6] == 0.f && v.K[7] == 0.f && v.K[8] == 1.f;
    }
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    const int cells = G * G * G;
    const size_t smem = (size_t)cells * D * sizeof(float);
    ASHB_REQUIRE(smem <= 200 * 1024, "block of %zu bytes does not fit in shared memory", smem);
    const IntegrateFrame frame{H, W, depth_max, (float)cell_size, make_float3(origin[0], origin[1], origin[2]), G, cells,
                               trunc, sdf_channel, rgb_channel, weight_channel, (int)D,
                               (G & (G - 1)) == 0 ? 31 - __builtin_clz((unsigned)G) : -1, kRound + (float)W,
                               kRound + (float)H, usual, frames, touched, stamp};
    // The copy-engine variant needs a work list, 16-byte aligned rows of a multiple of 16 bytes, and room
    // for two tiles per CTA; everything else takes the plain kernel.
    const bool bulk = touched_list != nullptr && smem % 16 == 0 && ((uintptr_t)embeddings & 15) == 0 && 2 * smem <= 96 * 1024;
    // with a work list: exactly the CTAs that are resident at once walk it (more would queue behind them
    // as a partly filled second wave); without: one CTA per row
#define ASHB_TSDF_LAUNCH(GT, N, T, VIEWS)                                                                  \
    {                                                                                                      \
        const void* fn = bulk ? (const void*)tsdf_integrate_bulk_kernel<GT, N, T> : (const void*)tsdf_integrate_kernel<GT, N, T>; \
        if (dyn > 48 * 1024)                                                                               \
            ASHB_CUDA_TRY(cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)dyn)); \
        int per_sm = 0;                                                                                    \
        ASHB_CUDA_TRY(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, fn, T, dyn));                 \
        const int64_t resident = (int64_t)sm_count() * (per_sm > 0 ? per_sm : 1);                          \
        const unsigned ctas = (unsigned)(touched_list && n_emb > resident ? resident : n_emb);             \
        if (bulk)                                                                                          \
            tsdf_integrate_bulk_kernel<GT, N, T><<<ctas, T, dyn, st>>>(                                    \
                    static_cast<float*>(embeddings), grid_coords, frame, VIEWS, n_integrated_dev, touched_list, touched_count); \
        else                                                                                               \
            tsdf_integrate_kernel<GT, N, T><<<ctas, T, dyn, st>>>(                                         \
                    static_cast<float*>(embeddings), grid_coords, touched, stamp, frame, VIEWS, n_integrated_dev, n_emb, \
                    touched_list, touched_count);                                                          \
    }
#define ASHB_TSDF_LAUNCH_N(GT, T)                                                                          \
    {                                                                                                      \
        if (frames) ASHB_TSDF_LAUNCH(GT, kBatch, T, views)                                                 \
        else ASHB_TSDF_LAUNCH(GT, 1, T, Views<1>{{views.view[0]}})                                         \
    }
    const size_t dyn = bulk ? 2 * smem : smem;
    const float pitch = std::max(std::fabs(views.view[0].K[0]), std::fabs(views.view[0].K[4])) * (float)cell_size / depth_max;
    const int threads = integrate_threads(dyn, G, frames != nullptr, pitch);
    if (G == 8 && threads == 128) ASHB_TSDF_LAUNCH_N(8, 128)
    else if (G == 8) ASHB_TSDF_LAUNCH(8, 1, 256, Views<1>{{views.view[0]}})
    else if (G == 4) ASHB_TSDF_LAUNCH_N(4, 128)
    else if (threads == 128) ASHB_TSDF_LAUNCH_N(0, 128)
    else if (threads == 256) ASHB_TSDF_LAUNCH_N(0, 256)
    else ASHB_TSDF_LAUNCH_N(0, 512)
#undef ASHB_TSDF_LAUNCH_N
#undef ASHB_TSDF_LAUNCH
    ASHB_LAUNCH_CHECK();
    return ASHB_OK;
}

int ashb_tsdf_integrate(void* embeddings, int64_t n_emb, int G, int64_t D, const int32_t* grid_coords,
                        const uint32_t* touched, uint32_t stamp, const float* depth, const float* color, int H,
                        int W, const float* intrinsic, const float* world_to_cam, float depth_max,
                        double cell_size, const float* origin, float trunc, int sdf_channel, int rgb_channel,
                        int weight_channel, unsigned long long* n_integrated_dev, const int32_t* touched_list,
                        const int32_t* touched_count, void* stream) {
    return integrate_impl(embeddings, n_emb, G, D, grid_coords, const_cast<uint32_t*>(touched), stamp, 1, &depth, &color, H,
                          W, intrinsic, world_to_cam, depth_max, cell_size, origin, trunc, sdf_channel, rgb_channel,
                          weight_channel, n_integrated_dev, touched_list, touched_count, nullptr, stream);
}

// Device address of g_tsdf_static_scratch on the current device.  In host code the array's
// name is only a handle; the address the kernels need comes from cudaGetSymbolAddress, looked
// up once per device with that device current.
static int static_scratch_for_current_device(unsigned char** out) {
    constexpr int kMaxDevices = 64;
    static std::mutex mu;
    static unsigned char* cached[kMaxDevices] = {};
    int dev = -1;
    ASHB_CUDA_TRY(cudaGetDevice(&dev));
    ASHB_REQUIRE(dev >= 0 && dev < kMaxDevices, "device ordinal %d out of range", dev);
    std::lock_guard<std::mutex> lock(mu);
    if (cached[dev] == nullptr) {
        void* p = nullptr;
        ASHB_CUDA_TRY(cudaGetSymbolAddress(&p, g_tsdf_static_scratch));
        ASHB_REQUIRE(p != nullptr, "static scratch has no device address");
        cached[dev] = static_cast<unsigned char*>(p);
    }
    *out = cached[dev];
    return ASHB_OK;
}

int ashb_tsdf_fuse_frame(ashb_map* m, void* embeddings, int64_t n_emb, int G, int64_t D, const float* depth,
                         const float* color, int H, int W, const float* intrinsic, const float* world_to_cam,
                         const float* cam_to_world, float depth_max, double cell_size, const float* origin,
                         int dilation, const int32_t* bound_lo, const int32_t* bound_hi, float trunc, int sdf_channel,
                         int rgb_channel, int weight_channel, int32_t* grid_coords, uint32_t* touched, uint32_t stamp,
                         int32_t* touched_list, int32_t* touched_count, unsigned long long* n_integrated_dev,
                         void* stream) {
    if (int rc = ashb_tsdf_touch(m, depth, H, W, intrinsic, cam_to_world, depth_max, cell_size, origin, G, dilation,
                                 bound_lo, bound_hi, grid_coords, touched, stamp, touched_list, touched_count, stream))
        return rc;
    DeviceGuard guard(m->device);
    return ashb_tsdf_integrate(embeddings, n_emb, G, D, grid_coords, touched, stamp, depth, color, H, W, intrinsic,
                               world_to_cam, depth_max, cell_size, origin, trunc, sdf_channel, rgb_channel,
                               weight_channel, n_integrated_dev, touched_list, touched_count, stream);
}

int ashb_tsdf_fuse_frames(ashb_map* m, void* embeddings, int64_t n_emb, int G, int64_t D, int n_frames,
                          const float* const* depths, const float* const* colors, int H, int W,
                          const float* intrinsics, const float* world_to_cams, const float* cam_to_worlds,
                          float depth_max, double cell_size, const float* origin, int dilation, const int32_t* bound_lo,
                          const int32_t* bound_hi, float trunc, int sdf_channel, int rgb_channel, int weight_channel,
                          int32_t* grid_coords, uint32_t* touched, uint32_t first_stamp, int32_t* touched_list,
                          int32_t* touched_count, int batched, unsigned long long* n_integrated_dev,
                          void* stream) {
    ASHB_REQUIRE(n_frames >= 0 && (n_frames == 0 || (depths && colors && intrinsics && world_to_cams && cam_to_worlds)),
                 "null frame tables");
    ASHB_REQUIRE((uint64_t)first_stamp + (uint64_t)n_frames <= 0x7FFFFFFFull && first_stamp != 0, "stamps would wrap");
    ASHB_REQUIRE(m != nullptr && m->slots != nullptr, "null or destroyed map");
    if (!batched || touched_list == nullptr || touched_count == nullptr || n_frames < 2) {
        for (int f = 0; f < n_frames; ++f) {
            if (int rc = ashb_tsdf_fuse_frame(m, embeddings, n_emb, G, D, depths[f], colors[f], H, W, intrinsics + 9 * f,
                                              world_to_cams + 12 * f, cam_to_worlds + 12 * f, depth_max, cell_size,
                                              origin, dilation, bound_lo, bound_hi, trunc, sdf_channel, rgb_channel,
                                              weight_channel, grid_coords, touched, first_stamp + (uint32_t)f,
                                              touched_list, touched_count, n_integrated_dev, stream))
                return rc;
        }
        return ASHB_OK;
    }
    // Batches: one allocation pass marks which frames of the batch touch each block, one fusion pass applies them to
    // it in their order.
    DeviceGuard guard(m->device);
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    uint32_t* frames = reinterpret_cast<uint32_t*>(touched_list + n_emb);
    const int64_t words = n_emb + (touched_list + 2 * n_emb == touched_count);
    for (int f = 0; f < n_frames; f += kBatch) {
        const int n = n_frames - f < kBatch ? n_frames - f : kBatch;
        const uint32_t stamp = first_stamp + (uint32_t)f;
        if (int rc = touch_impl(m, n, depths + f, H, W, intrinsics + 9 * f, cam_to_worlds + 12 * f, depth_max, cell_size,
                                origin, G, dilation, bound_lo, bound_hi, grid_coords, touched, stamp, touched_list,
                                touched_count, frames, words, st))
            return rc;
        if (int rc = integrate_impl(embeddings, n_emb, G, D, grid_coords, touched, stamp, n, depths + f, colors + f, H, W,
                                    intrinsics + 9 * f, world_to_cams + 12 * f, depth_max, cell_size, origin, trunc,
                                    sdf_channel, rgb_channel, weight_channel, n_integrated_dev, touched_list,
                                    touched_count, frames, st))
            return rc;
    }
    return ASHB_OK;
}

int ashb_tsdf_static_max_blocks(void) { return ASHB_TSDF_STATIC_MAX_BLOCKS; }

int ashb_tsdf_copy_timeouts(unsigned int* out) {
    ASHB_REQUIRE(out != nullptr, "out is null");
    ASHB_CUDA_TRY(cudaMemcpyFromSymbol(out, g_tsdf_copy_timeouts, sizeof(unsigned int)));
    return ASHB_OK;
}

int ashb_tsdf_fuse_frame_static(ashb_map* m, void* embeddings, int64_t n_emb, int G, int64_t D,
                                const float* depth, const float* color, int H, int W, const float* intrinsic,
                                const float* world_to_cam, const float* cam_to_world, float depth_max,
                                double cell_size, const float* origin, int dilation, const int32_t* bound_lo,
                                const int32_t* bound_hi, float trunc, int sdf_channel, int rgb_channel,
                                int weight_channel, void* stream) {
    ASHB_REQUIRE(m != nullptr && m->slots != nullptr, "null or destroyed map");
    ASHB_REQUIRE(n_emb >= 1 && n_emb <= ASHB_TSDF_STATIC_MAX_BLOCKS,
                 "ashb_tsdf_fuse_frame_static handles at most %d blocks (got %lld); use ashb_tsdf_touch + "
                 "ashb_tsdf_integrate with caller-provided scratch for larger grids",
                 ASHB_TSDF_STATIC_MAX_BLOCKS, (long long)n_emb);
    ASHB_REQUIRE(n_emb == m->capacity, "n_emb must equal the map's capacity");
    DeviceGuard guard(m->device);
    unsigned char* scratch = nullptr;
    if (int rc = static_scratch_for_current_device(&scratch)) return rc;
    uint32_t* touched = reinterpret_cast<uint32_t*>(scratch);
    int32_t* coords = reinterpret_cast<int32_t*>(scratch + (size_t)ASHB_TSDF_STATIC_MAX_BLOCKS * 4);
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    // The array is shared by every call and keeps the previous call's stamps: start from zero.
    ASHB_CUDA_TRY(cudaMemsetAsync(touched, 0, (size_t)n_emb * sizeof(uint32_t), st));
    const uint32_t stamp = 1;
    if (int rc = ashb_tsdf_touch(m, depth, H, W, intrinsic, cam_to_world, depth_max, cell_size, origin, G, dilation,
                                 bound_lo, bound_hi, coords, touched, stamp, nullptr, nullptr, stream))
        return rc;
    return ashb_tsdf_integrate(embeddings, n_emb, G, D, coords, touched, stamp, depth, color, H, W, intrinsic,
                               world_to_cam, depth_max, cell_size, origin, trunc, sdf_channel, rgb_channel,
                               weight_channel, nullptr, nullptr, nullptr, stream);
}

}  // extern "C"
