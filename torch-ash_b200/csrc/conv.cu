// Depth-wise window convolution over the sparse-dense structure (sm_100a),
// driven by the radius-R neighbour lookup tables of ash/grid.py:494-502.
// Semantics follow ash/src/grid.cu:951-1043: out[g, c, :] = sum over the K window
// taps k of in[neighbour_k(g, c), :] * w[k, :], skipping taps whose block is absent.
//
// One CTA works on one active block: its row of the block-neighbour table is
// staged in shared memory once, and a group of lanes shares each output cell
// (lane j owns VEC channels) so that every tap is one coalesced vector load.
#include "common.cuh"

namespace ashb {

constexpr int kMaxGridNbs = 125;  // block window of radius <= 2

template <typename T, int VEC>
__global__ void __launch_bounds__(256) conv_forward_kernel(
        const T* __restrict__ in, const T* __restrict__ w, const uint8_t* __restrict__ masks,
        const int64_t* __restrict__ grid_indices, const int64_t* __restrict__ cell_indices,
        const int64_t* __restrict__ g2g, const int64_t* __restrict__ c2c, const int64_t* __restrict__ c2g,
        T* __restrict__ out, int num_cell_nbs, int num_grid_nbs, int64_t cells_per_grid, int D, int lane_shift,
        int64_t n_emb) {
    __shared__ int64_t nb_block[kMaxGridNbs];
    const int64_t grid_i = blockIdx.x;
    const int64_t grid_idx = grid_indices[grid_i];
    const bool block_ok = grid_idx >= 0 && grid_idx < n_emb;
    for (int k = threadIdx.x; k < num_grid_nbs; k += blockDim.x)
        nb_block[k] = block_ok ? g2g[grid_idx * num_grid_nbs + k] : -1;
    __syncthreads();
    if (!block_ok) return;

    const int lanes = 1 << lane_shift;
    const int lane = threadIdx.x & (lanes - 1);
    const int ch = lane * VEC;
    if (ch >= D) return;
    const int cells_per_pass = blockDim.x >> lane_shift;
    for (int64_t cell_i = threadIdx.x >> lane_shift; cell_i < cells_per_grid; cell_i += cells_per_pass) {
        if (!masks[grid_i * cells_per_grid + cell_i]) continue;  // grid.cu:968-969
        const int64_t cell_idx = cell_indices[cell_i];
        const int64_t* nb_cell = c2c + (int64_t)num_cell_nbs * cell_idx;
        const int64_t* nb_cg = c2g + (int64_t)num_cell_nbs * cell_idx;
        T acc[VEC];
#pragma unroll
        for (int v = 0; v < VEC; ++v) acc[v] = 0;
        for (int k = 0; k < num_cell_nbs; ++k) {
            const int64_t gnb = __ldg(nb_cg + k);
            const int64_t g = (gnb >= 0 && gnb < num_grid_nbs) ? nb_block[gnb] : -1;
            if (g < 0 || g >= n_emb) continue;
            const T* src = in + (g * cells_per_grid + __ldg(nb_cell + k)) * D + ch;
            const T* wk = w + (int64_t)k * D + ch;
#pragma unroll
            for (int v = 0; v < VEC; ++v) acc[v] += __ldg(src + v) * __ldg(wk + v);
        }
        T* dst = out + (grid_idx * cells_per_grid + cell_idx) * D + ch;
#pragma unroll
        for (int v = 0; v < VEC; ++v) dst[v] = acc[v];
    }
}

// ---- shared-memory tiled variant ---------------------------------------------------------
// For the window the Python layer actually builds (radius R <= G, two-sided, block window 3^3)
// the two per-cell tables are pure arithmetic, so the kernel needs only the 27-entry block
// row.  One CTA per active block stages the block plus its R-cell halo ((G+2R)^3 cells, CH
// channels at a time) in shared memory -- neighbour blocks are read with coalesced 16-byte
// loads, absent ones count as zero -- and the K^3 weights beside it.  Each thread then
// produces XT outputs that are adjacent in x from one sliding row segment held in registers, so
// a tile value is read from shared memory once per XT outputs and a weight once per XT outputs.
// Taps are accumulated in the reference's order (x fastest, then y, then z).
// RT > 0 fixes the radius at compile time (fully unrolled taps, row segment in registers);
// RT == 0 takes it at run time.
template <int CH, int XT, int RT>
__global__ void __launch_bounds__(256) conv_tiled_kernel(const float* __restrict__ in, const float* __restrict__ w,
                                                         const int64_t* __restrict__ grid_indices,
                                                         const int64_t* __restrict__ g2g27, float* __restrict__ out,
                                                         int G, int R_arg, int D, int64_t n_emb) {
    extern __shared__ float smem[];
    const int R = RT > 0 ? RT : R_arg;
    const int S = 2 * R + 1, T = G + 2 * R;
    const int cells = G * G * G, taps = S * S * S, tile_cells = T * T * T;
    float* tile = smem;                       // [tile_cells][CH]
    float* wsm = smem + (size_t)tile_cells * CH;  // [taps][CH]
    __shared__ int64_t nb[27];
    const int64_t gidx = grid_indices[blockIdx.x];
    const bool ok = gidx >= 0 && gidx < n_emb;
    if (threadIdx.x < 27) nb[threadIdx.x] = ok ? g2g27[gidx * 27 + threadIdx.x] : -1;
    __syncthreads();
    if (!ok) return;
    const int xt_per_row = G / XT;
    const int n_items = G * G * xt_per_row;  // (z, y, x-chunk) work items
    for (int ch0 = 0; ch0 < D; ch0 += CH) {
        for (int k = threadIdx.x; k < taps * CH; k += blockDim.x) wsm[k] = w[(int64_t)(k / CH) * D + ch0 + (k % CH)];
        for (int h = threadIdx.x; h < tile_cells; h += blockDim.x) {
            const int hx = h % T, hy = (h / T) % T, hz = h / (T * T);
            const int cx = hx - R, cy = hy - R, cz = hz - R;            // cell coordinate relative to this block
            const int bx = cx < 0 ? -1 : (cx >= G ? 1 : 0), by = cy < 0 ? -1 : (cy >= G ? 1 : 0),
                      bz = cz < 0 ? -1 : (cz >= G ? 1 : 0);
            const int64_t g = nb[(bx + 1) + (by + 1) * 3 + (bz + 1) * 9];
            float v[CH];
#pragma unroll
            for (int c = 0; c < CH; ++c) v[c] = 0.f;
            if (g >= 0 && g < n_emb) {
                const int lin = (cx - bx * G) + ((cy - by * G) + (cz - bz * G) * G) * G;
                const float* src = in + (g * cells + lin) * D + ch0;
                if (CH == 4) {
                    const float4 t4 = __ldg(reinterpret_cast<const float4*>(src));
                    v[0] = t4.x, v[1] = t4.y, v[2] = t4.z, v[3] = t4.w;
                } else {
#pragma unroll
                    for (int c = 0; c < CH; ++c) v[c] = __ldg(src + c);
                }
            }
#pragma unroll
            for (int c = 0; c < CH; ++c) tile[(size_t)h * CH + c] = v[c];
        }
        __syncthreads();
        for (int item = threadIdx.x; item < n_items; item += blockDim.x) {
            const int xc = item % xt_per_row, y = (item / xt_per_row) % G, z = item / (xt_per_row * G);
            const int x0 = xc * XT;
            float acc[XT][CH];
#pragma unroll
            for (int o = 0; o < XT; ++o)
#pragma unroll
                for (int c = 0; c < CH; ++c) acc[o][c] = 0.f;
            for (int kz = 0; kz < S; ++kz)
                for (int ky = 0; ky < S; ++ky) {
                    const float* row = tile + ((size_t)((z + kz) * T + (y + ky)) * T + x0) * CH;
                    const float* wrow = wsm + (size_t)((kz * S + ky) * S) * CH;
                    // sliding window along x: XT outputs share the S + XT - 1 inputs of this row
                    if constexpr (RT > 0) {
                        constexpr int SS = 2 * RT + 1;
                        float seg[SS + XT - 1][CH];
#pragma unroll
                        for (int i = 0; i < SS + XT - 1; ++i)
#pragma unroll
                            for (int c = 0; c < CH; ++c) seg[i][c] = row[i * CH + c];
#pragma unroll
                        for (int kx = 0; kx < SS; ++kx) {
                            float wv[CH];
#pragma unroll
                            for (int c = 0; c < CH; ++c) wv[c] = wrow[kx * CH + c];
#pragma unroll
                            for (int o = 0; o < XT; ++o)
#pragma unroll
                                for (int c = 0; c < CH; ++c) acc[o][c] += seg[o + kx][c] * wv[c];
                        }
                    } else {
                        for (int kx = 0; kx < S; ++kx) {
                            float wv[CH];
#pragma unroll
                            for (int c = 0; c < CH; ++c) wv[c] = wrow[kx * CH + c];
#pragma unroll
                            for (int o = 0; o < XT; ++o)
#pragma unroll
                                for (int c = 0; c < CH; ++c) acc[o][c] += row[(o + kx) * CH + c] * wv[c];
                        }
                    }
                }
#pragma unroll
            for (int o = 0; o < XT; ++o) {
                float* dst = out + (gidx * cells + (x0 + o) + (y + z * G) * G) * D + ch0;
#pragma unroll
                for (int c = 0; c < CH; ++c) dst[c] = acc[o][c];
            }
        }
        __syncthreads();
    }
}

// The blocks to filter: `grid_indices` with one CTA each, or the first *count rows of `list`, which the CTAs
// of eight waves share out (27,000 blocks: 251 us; one wave 264, a CTA per possible row 282).
struct FilterBlocks {
    const int64_t* __restrict__ grid_indices;
    const int32_t* __restrict__ list;
    const int32_t* __restrict__ count;
};

// Separable window: weights[z][y][x][c] = wz[z][c] * wy[y][c] * wx[x][c] (a Gaussian is one).  The
// same halo tile is staged, then three 1-D passes run inside shared memory -- along x over the
// whole (G+2R)^2 cross-section, along y over the (G+2R) slabs that remain, along z -- so a
// (2R+1)^3 window costs 3 (2R+1) multiply-adds per cell and channel instead of (2R+1)^3, and the
// intermediate sums never exist for cells outside the tile (absent neighbour blocks count as zero
// exactly as in the full window).  w1: [3][S][D], axis 0 = x.
template <int CH>
__global__ void __launch_bounds__(256) conv_separable_kernel(const float* __restrict__ in, const float* __restrict__ w1,
                                                             FilterBlocks blocks,
                                                             const int64_t* __restrict__ g2g27, float* __restrict__ out,
                                                             int G, int R, int D, int64_t n_emb) {
    extern __shared__ float smem[];
    const int S = 2 * R + 1, T = G + 2 * R;
    const int cells = G * G * G, tile_cells = T * T * T;
    float* tile = smem;                                   // [T][T][T][CH]; reused for the y-pass sums [T][G][G][CH]
    float* t1 = smem + (size_t)tile_cells * CH;           // x-pass sums [T][T][G][CH]
    float* wsm = t1 + (size_t)T * T * G * CH;             // [3][S][CH]
    __shared__ int64_t nb[27];
    if (blocks.list && (int)blockIdx.x >= *blocks.count) return;
    const int64_t gidx = blocks.list ? blocks.list[blockIdx.x] : blocks.grid_indices[blockIdx.x];
    const bool ok = gidx >= 0 && gidx < n_emb;
    if (threadIdx.x < 27) nb[threadIdx.x] = ok ? g2g27[gidx * 27 + threadIdx.x] : -1;
    __syncthreads();
    if (!ok) return;
    for (int ch0 = 0; ch0 < D; ch0 += CH) {
        for (int k = threadIdx.x; k < 3 * S * CH; k += blockDim.x) wsm[k] = w1[(int64_t)(k / CH) * D + ch0 + (k % CH)];
        for (int h = threadIdx.x; h < tile_cells; h += blockDim.x) {
            const int hx = h % T, hy = (h / T) % T, hz = h / (T * T);
            const int cx = hx - R, cy = hy - R, cz = hz - R;
            const int bx = cx < 0 ? -1 : (cx >= G ? 1 : 0), by = cy < 0 ? -1 : (cy >= G ? 1 : 0),
                      bz = cz < 0 ? -1 : (cz >= G ? 1 : 0);
            const int64_t g = nb[(bx + 1) + (by + 1) * 3 + (bz + 1) * 9];
            float v[CH];
#pragma unroll
            for (int c = 0; c < CH; ++c) v[c] = 0.f;
            if (g >= 0 && g < n_emb) {
                const int lin = (cx - bx * G) + ((cy - by * G) + (cz - bz * G) * G) * G;
                const float* src = in + (g * cells + lin) * D + ch0;
                if (CH == 4) {
                    const float4 t4 = __ldg(reinterpret_cast<const float4*>(src));
                    v[0] = t4.x, v[1] = t4.y, v[2] = t4.z, v[3] = t4.w;
                } else {
#pragma unroll
                    for (int c = 0; c < CH; ++c) v[c] = __ldg(src + c);
                }
            }
#pragma unroll
            for (int c = 0; c < CH; ++c) tile[(size_t)h * CH + c] = v[c];
        }
        __syncthreads();
        // along x: t1[z'][y'][x] = sum_k wx[k] * tile[z'][y'][x + k]
        for (int i = threadIdx.x; i < T * T * G; i += blockDim.x) {
            const int x = i % G, zy = i / G;
            const float* row = tile + ((size_t)zy * T + x) * CH;
            float acc[CH];
#pragma unroll
            for (int c = 0; c < CH; ++c) acc[c] = 0.f;
            for (int k = 0; k < S; ++k)
#pragma unroll
                for (int c = 0; c < CH; ++c) acc[c] += row[k * CH + c] * wsm[k * CH + c];
#pragma unroll
            for (int c = 0; c < CH; ++c) t1[(size_t)i * CH + c] = acc[c];
        }
        __syncthreads();
        // along y: t2[z'][y][x] = sum_k wy[k] * t1[z'][y + k][x]   (t2 takes the tile's place)
        float* t2 = tile;
        for (int i = threadIdx.x; i < T * G * G; i += blockDim.x) {
            const int x = i % G, y = (i / G) % G, zp = i / (G * G);
            const float* col = t1 + ((size_t)(zp * T + y) * G + x) * CH;
            float acc[CH];
#pragma unroll
            for (int c = 0; c < CH; ++c) acc[c] = 0.f;
            for (int k = 0; k < S; ++k)
#pragma unroll
                for (int c = 0; c < CH; ++c) acc[c] += col[(size_t)k * G * CH + c] * wsm[(S + k) * CH + c];
#pragma unroll
            for (int c = 0; c < CH; ++c) t2[(size_t)i * CH + c] = acc[c];
        }
        __syncthreads();
        // along z: out[z][y][x] = sum_k wz[k] * t2[z + k][y][x]
        for (int i = threadIdx.x; i < cells; i += blockDim.x) {
            const float* col = t2 + (size_t)i * CH;
            float acc[CH];
#pragma unroll
            for (int c = 0; c < CH; ++c) acc[c] = 0.f;
            for (int k = 0; k < S; ++k)
#pragma unroll
                for (int c = 0; c < CH; ++c) acc[c] += col[(size_t)k * G * G * CH + c] * wsm[(2 * S + k) * CH + c];
            float* dst = out + (gidx * cells + i) * D + ch0;
            if (CH == 4) {
                *reinterpret_cast<float4*>(dst) = make_float4(acc[0], acc[1], acc[2], acc[3]);
            } else {
#pragma unroll
                for (int c = 0; c < CH; ++c) dst[c] = acc[c];
            }
        }
        __syncthreads();
    }
}

// The same filter for the block edges and radii that are compiled in (G of 4, 8, 16 and R of 1, 2, 3).
// Bound by the halo's way from L2 (61 M sectors of 27,000 blocks in 254 us) since the tile is touched as little as possible (two
// channels per multiply-add, a third of the instructions less, are no faster):
// a thread takes one line of the tile (one channel of a row, a column or a pillar), reads it once into
// registers, slides the window over it there and writes the sums back in the line's own place.  A line
// is read and written by its own thread alone, so one buffer serves all three passes (47 KB at G = 8,
// R = 3, four channels: four CTAs per SM instead of three with the 70 KB of conv_separable_kernel) and a
// tile value costs one access per pass instead of 2R + 1.  Rows are T + 1 cells apart: T is even, so eight
// rows start in different bank groups.  The halo arrives by cp.async, absent blocks as zero-filled copies.
// Every sum has the terms and the order of conv_separable_kernel, which stays for all other sizes.
template <int BYTES>
__device__ __forceinline__ void copy_async(float* dst, const float* src, bool present) {
    const uint32_t d = (uint32_t)__cvta_generic_to_shared(dst);
    if constexpr (BYTES == 16)   // past L1: a CTA reads a cell once
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(d), "l"(src), "r"(present ? 16 : 0) : "memory");
    else
        asm volatile("cp.async.ca.shared.global [%0], [%1], %2, %3;" ::"r"(d), "l"(src), "n"(BYTES), "r"(present ? BYTES : 0)
                     : "memory");
}

// store(o, sum over k of w[k] * line[o + k]) for N sums of a line whose values are STRIDE floats apart.
template <int N, int S, int STRIDE, class Store>
__device__ __forceinline__ void filter_line(const float* line, const float* w, Store&& store) {
    float v[N + S - 1];
#pragma unroll
    for (int i = 0; i < N + S - 1; ++i) v[i] = line[i * STRIDE];
#pragma unroll
    for (int o = 0; o < N; ++o) {
        float acc = 0.f;
#pragma unroll
        for (int k = 0; k < S; ++k) acc += v[o + k] * w[k];
        store(o, acc);
    }
}

template <int CH, int G, int R>
__global__ void __launch_bounds__(256) conv_separable_lines_kernel(const float* __restrict__ in,
                                                                   const float* __restrict__ w1, FilterBlocks blocks,
                                                                   const int64_t* __restrict__ g2g27,
                                                                   float* __restrict__ out, int D, int64_t n_emb) {
    constexpr int S = 2 * R + 1, T = G + 2 * R, ROW = (T + 1) * CH, SLAB = T * ROW, CELLS = G * G * G;
    constexpr int WIDE = T <= 8 ? 8 : (T <= 16 ? 16 : 32);
    extern __shared__ __align__(16) float tile[];   // [T][T][T + 1][CH]
    __shared__ float wsm[3 * S * CH];
    __shared__ const float* nb[27];
    const int n_items = blocks.list ? *blocks.count : (int)gridDim.x;
    for (int item = blockIdx.x; item < n_items; item += gridDim.x) {
        const int64_t gidx = blocks.list ? blocks.list[item] : blocks.grid_indices[item];
        if (gidx < 0 || gidx >= n_emb) continue;
        if (threadIdx.x < 27) {
            const int64_t g = g2g27[gidx * 27 + threadIdx.x];
            nb[threadIdx.x] = g >= 0 && g < n_emb ? in + g * CELLS * D : nullptr;
        }
        __syncthreads();
        for (int ch0 = 0; ch0 < D; ch0 += CH) {
            // a thread keeps its (x, y) of the tile and walks the slabs: the three blocks it reads are three pointers
            for (int hy = threadIdx.x / WIDE; hy < T; hy += blockDim.x / WIDE) {
                const int hx = threadIdx.x % WIDE;
                if (hx >= T) break;
                const int bx = (hx >= R) + (hx >= G + R), by = (hy >= R) + (hy >= G + R);
                const int xy = (hx + G - R) % G + (hy + G - R) % G * G;
                const float* from[3];
                bool present[3];
#pragma unroll
                for (int bz = 0; bz < 3; ++bz) {
                    const float* block = nb[bx + by * 3 + bz * 9];
                    present[bz] = block != nullptr;
                    from[bz] = (present[bz] ? block : in) + xy * D + ch0;
                }
                float* to = tile + hy * ROW + hx * CH;
#pragma unroll
                for (int hz = 0; hz < T; ++hz) {
                    const int bz = (hz >= R) + (hz >= G + R);
                    copy_async<CH * 4>(to + hz * SLAB, from[bz] + (hz + G - R) % G * (G * G) * D, present[bz]);
                }
            }
            for (int k = threadIdx.x; k < 3 * S * CH; k += blockDim.x) wsm[k] = w1[(int64_t)(k / CH) * D + ch0 + (k % CH)];
            asm volatile("cp.async.wait_all;" ::: "memory");
            __syncthreads();
            // the block size is a multiple of CH: a thread stays with one channel and its weights
            const int c = threadIdx.x % CH;
            float w[S];
#pragma unroll
            for (int k = 0; k < S; ++k) w[k] = wsm[k * CH + c];
            for (int i = threadIdx.x; i < T * T * CH; i += blockDim.x) {   // rows, along x
                float* line = tile + (i / CH) * ROW + c;
                filter_line<G, S, CH>(line, w, [&](int o, float v) { line[o * CH] = v; });
            }
#pragma unroll
            for (int k = 0; k < S; ++k) w[k] = wsm[(S + k) * CH + c];
            __syncthreads();
            for (int i = threadIdx.x; i < T * G * CH; i += blockDim.x) {   // columns, along y
                float* line = tile + (i / (G * CH)) * SLAB + i % (G * CH);
                filter_line<G, S, ROW>(line, w, [&](int o, float v) { line[o * ROW] = v; });
            }
#pragma unroll
            for (int k = 0; k < S; ++k) w[k] = wsm[(2 * S + k) * CH + c];
            __syncthreads();
            for (int i = threadIdx.x; i < G * G * CH; i += blockDim.x) {   // pillars, along z
                const int xy = i / CH;
                const float* line = tile + (xy / G) * ROW + i % (G * CH);
                float* dst = out + (gidx * CELLS + xy) * D + ch0 + c;
                filter_line<G, S, SLAB>(line, w, [&](int o, float v) { dst[(int64_t)o * G * G * D] = v; });
            }
            __syncthreads();
        }
    }
}

// values[row] = filtered[row] for the active rows (whose own entry of the block table is the row itself), zero for
// the others: the second half of an in-place filter.  `vec` 16-byte words (or floats) a row.
template <typename V>
__global__ void __launch_bounds__(256) restore_rows_kernel(V* __restrict__ values, const V* __restrict__ filtered,
                                                           const int64_t* __restrict__ g2g27, int64_t n_emb, int vec) {
    for (int64_t row = blockIdx.x; row < n_emb; row += gridDim.x) {
        const bool active = g2g27[row * 27 + 13] == row;
        V* to = values + row * vec;
        const V* from = filtered + row * vec;
        if (active) {
            for (int i = threadIdx.x; i < vec; i += blockDim.x) to[i] = __ldcs(from + i);
        } else {
            for (int i = threadIdx.x; i < vec; i += blockDim.x) to[i] = V{};
        }
    }
}

}  // namespace ashb

using namespace ashb;

extern "C" {

int ashb_conv_forward(int dtype, const void* inputs, const void* weights, const uint8_t* masks,
                      const int64_t* grid_indices, const int64_t* cell_indices, const int64_t* g2g,
                      const int64_t* c2c, const int64_t* c2g, void* outputs, int zero_output,
                      int64_t num_grids, int64_t n_emb, int64_t cells_per_grid, int64_t D,
                      int64_t num_cell_nbs, int64_t num_grid_nbs, void* stream) {
    ASHB_REQUIRE(dtype == ASHB_F32 || dtype == ASHB_F64, "unknown dtype code %d", dtype);
    ASHB_REQUIRE(D >= 1 && D <= 16, "embedding_dim %lld not in 1..16", (long long)D);
    ASHB_REQUIRE(num_grid_nbs >= 1 && num_grid_nbs <= kMaxGridNbs, "block window of %lld neighbours unsupported",
                 (long long)num_grid_nbs);
    ASHB_REQUIRE(num_grids >= 0 && n_emb >= 1 && cells_per_grid >= 1 && num_cell_nbs >= 1, "bad sizes");
    ASHB_REQUIRE(outputs != nullptr, "null outputs");
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    const size_t elem = dtype == ASHB_F32 ? 4 : 8;
    if (zero_output)  // grid.cu:1016: rows of inactive blocks stay zero
        ASHB_CUDA_TRY(cudaMemsetAsync(outputs, 0, (size_t)n_emb * cells_per_grid * D * elem, st));
    if (num_grids == 0) return ASHB_OK;
    ASHB_REQUIRE(inputs && weights && masks && grid_indices && cell_indices && g2g && c2c && c2g, "null buffer");
    int shift = 0;
    while ((1 << shift) < D) ++shift;
    const unsigned grid = (unsigned)num_grids;
    if (dtype == ASHB_F32)
        conv_forward_kernel<float, 1><<<grid, 256, 0, st>>>(
                static_cast<const float*>(inputs), static_cast<const float*>(weights), masks, grid_indices,
                cell_indices, g2g, c2c, c2g, static_cast<float*>(outputs), (int)num_cell_nbs, (int)num_grid_nbs,
                cells_per_grid, (int)D, shift, n_emb);
    else
        conv_forward_kernel<double, 1><<<grid, 256, 0, st>>>(
                static_cast<const double*>(inputs), static_cast<const double*>(weights), masks, grid_indices,
                cell_indices, g2g, c2c, c2g, static_cast<double*>(outputs), (int)num_cell_nbs,
                (int)num_grid_nbs, cells_per_grid, (int)D, shift, n_emb);
    ASHB_LAUNCH_CHECK();
    return ASHB_OK;
}

int ashb_conv_forward_tiled(const float* inputs, const float* weights, const int64_t* grid_indices,
                            const int64_t* lut_grid_nb27, float* outputs, int zero_output, int64_t num_grids,
                            int64_t n_emb, int G, int radius, int64_t D, void* stream) {
    ASHB_REQUIRE(D >= 1 && D <= 16, "embedding_dim %lld not in 1..16", (long long)D);
    ASHB_REQUIRE(G >= 1 && G <= 16 && radius >= 1 && radius <= G, "window radius %d must be within one block (G=%d)",
                 radius, G);
    ASHB_REQUIRE(num_grids >= 0 && n_emb >= 1 && outputs != nullptr, "bad sizes");
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    const int64_t cells = (int64_t)G * G * G;
    if (zero_output) ASHB_CUDA_TRY(cudaMemsetAsync(outputs, 0, (size_t)n_emb * cells * D * sizeof(float), st));
    if (num_grids == 0) return ASHB_OK;
    ASHB_REQUIRE(inputs && weights && grid_indices && lut_grid_nb27, "null buffer");
    const int ch = (D % 4 == 0 && (((uintptr_t)inputs) & 15) == 0) ? 4 : (D % 2 == 0 ? 2 : 1);
    const int T = G + 2 * radius, S = 2 * radius + 1;
    const size_t smem = ((size_t)T * T * T + (size_t)S * S * S) * ch * sizeof(float);
    ASHB_REQUIRE(smem <= 200 * 1024, "halo tile of %zu bytes does not fit in shared memory", smem);
    const int xt = G % 4 == 0 ? 4 : (G % 2 == 0 ? 2 : 1);
    const int items = G * G * (G / xt);
    const int threads = items >= 256 ? 256 : (items >= 128 ? 128 : 64);
#define ASHB_CONV_LAUNCH(CH, XT, RT)                                                                        \
    {                                                                                                       \
        if (smem > 48 * 1024)                                                                               \
            ASHB_CUDA_TRY(cudaFuncSetAttribute(conv_tiled_kernel<CH, XT, RT>,                               \
                                               cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));   \
        conv_tiled_kernel<CH, XT, RT><<<(unsigned)num_grids, threads, smem, st>>>(                          \
                inputs, weights, grid_indices, lut_grid_nb27, outputs, G, radius, (int)D, n_emb);           \
    }
#define ASHB_CONV_RADIUS(CH, XT)                                   \
    switch (radius) {                                              \
        case 1: ASHB_CONV_LAUNCH(CH, XT, 1) break;                 \
        case 2: ASHB_CONV_LAUNCH(CH, XT, 2) break;                 \
        case 3: ASHB_CONV_LAUNCH(CH, XT, 3) break;                 \
        default: ASHB_CONV_LAUNCH(CH, XT, 0)                       \
    }
    if (ch == 4 && xt == 4) ASHB_CONV_RADIUS(4, 4)
    else if (ch == 4 && xt == 2) ASHB_CONV_RADIUS(4, 2)
    else if (ch == 4) ASHB_CONV_RADIUS(4, 1)
    else if (ch == 2 && xt == 4) ASHB_CONV_RADIUS(2, 4)
    else if (ch == 2 && xt == 2) ASHB_CONV_RADIUS(2, 2)
    else if (ch == 2) ASHB_CONV_RADIUS(2, 1)
    else if (xt == 4) ASHB_CONV_RADIUS(1, 4)
    else if (xt == 2) ASHB_CONV_RADIUS(1, 2)
    else ASHB_CONV_RADIUS(1, 1)
#undef ASHB_CONV_RADIUS
#undef ASHB_CONV_LAUNCH
    ASHB_LAUNCH_CHECK();
    return ASHB_OK;
}

}  // extern "C"

// Filter the blocks of `grid_indices` (num_grids of them) or of `list` (at most n_emb, counted on the device).
static int separable_impl(const float* inputs, const float* weights_1d, const int64_t* grid_indices, const int32_t* list,
                          const int32_t* list_count, const int64_t* lut_grid_nb27, float* outputs, int64_t num_grids,
                          int64_t n_emb, int G, int radius, int64_t D, cudaStream_t st) {
    const uintptr_t bits = (uintptr_t)inputs | (uintptr_t)outputs;
    const int ch = D % 4 == 0 && (bits & 15) == 0 ? 4 : (D % 2 == 0 && (bits & 7) == 0 ? 2 : 1);
    const int T = G + 2 * radius, S = 2 * radius + 1;
    const FilterBlocks blocks{grid_indices, list, list_count};
#define ASHB_SEP_LINES(CH, GG, RR)                                                                                      \
    if (ch == CH && G == GG && radius == RR) {                                                                          \
        constexpr int TT = GG + 2 * RR, threads = GG == 4 ? 128 : 256;                                                  \
        constexpr size_t bytes = (size_t)TT * TT * (TT + 1) * CH * sizeof(float);                                       \
        const auto fn = conv_separable_lines_kernel<CH, GG, RR>;                                                        \
        if (bytes > 48 * 1024)                                                                                          \
            ASHB_CUDA_TRY(cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes));           \
        int64_t ctas = num_grids;                                                                                       \
        if (list) {                                                                                                     \
            int per_sm = 0;                                                                                             \
            ASHB_CUDA_TRY(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, fn, threads, bytes));                  \
            const int64_t resident = (int64_t)sm_count() * (per_sm > 0 ? per_sm : 1);                                   \
            ctas = n_emb < 8 * resident ? n_emb : 8 * resident;                                                         \
        }                                                                                                               \
        fn<<<(unsigned)ctas, threads, bytes, st>>>(inputs, weights_1d, blocks, lut_grid_nb27, outputs, (int)D, n_emb);  \
        ASHB_LAUNCH_CHECK();                                                                                            \
        return ASHB_OK;                                                                                                 \
    }
#define ASHB_SEP_LINES_R(CH, GG) ASHB_SEP_LINES(CH, GG, 1) ASHB_SEP_LINES(CH, GG, 2) ASHB_SEP_LINES(CH, GG, 3)
#define ASHB_SEP_LINES_G(CH) ASHB_SEP_LINES_R(CH, 4) ASHB_SEP_LINES_R(CH, 8) ASHB_SEP_LINES_R(CH, 16)
    ASHB_SEP_LINES_G(4)
    ASHB_SEP_LINES_G(2)
    ASHB_SEP_LINES_G(1)
#undef ASHB_SEP_LINES_G
#undef ASHB_SEP_LINES_R
#undef ASHB_SEP_LINES
    const size_t smem = ((size_t)T * T * T + (size_t)T * T * G + (size_t)3 * S) * ch * sizeof(float);
    ASHB_REQUIRE(smem <= 200 * 1024, "halo tile of %zu bytes does not fit in shared memory", smem);
    const unsigned ctas = (unsigned)(list ? n_emb : num_grids);
#define ASHB_SEP_LAUNCH(CH)                                                                                   \
    {                                                                                                         \
        if (smem > 48 * 1024)                                                                                 \
            ASHB_CUDA_TRY(cudaFuncSetAttribute(conv_separable_kernel<CH>,                                     \
                                               cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));     \
        conv_separable_kernel<CH><<<ctas, 256, smem, st>>>(inputs, weights_1d, blocks, lut_grid_nb27, outputs, \
                                                            G, radius, (int)D, n_emb);                        \
    }
    if (ch == 4) ASHB_SEP_LAUNCH(4)
    else if (ch == 2) ASHB_SEP_LAUNCH(2)
    else ASHB_SEP_LAUNCH(1)
#undef ASHB_SEP_LAUNCH
    ASHB_LAUNCH_CHECK();
    return ASHB_OK;
}

extern "C" {

int ashb_conv_forward_separable(const float* inputs, const float* weights_1d, const int64_t* grid_indices,
                                const int64_t* lut_grid_nb27, float* outputs, int zero_output, int64_t num_grids,
                                int64_t n_emb, int G, int radius, int64_t D, void* stream) {
    ASHB_REQUIRE(D >= 1 && D <= 16, "embedding_dim %lld not in 1..16", (long long)D);
    ASHB_REQUIRE(G >= 1 && G <= 16 && radius >= 1 && radius <= G, "window radius %d must be within one block (G=%d)",
                 radius, G);
    ASHB_REQUIRE(num_grids >= 0 && n_emb >= 1 && outputs != nullptr, "bad sizes");
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    const int64_t cells = (int64_t)G * G * G;
    if (zero_output) ASHB_CUDA_TRY(cudaMemsetAsync(outputs, 0, (size_t)n_emb * cells * D * sizeof(float), st));
    if (num_grids == 0) return ASHB_OK;
    ASHB_REQUIRE(inputs && weights_1d && grid_indices && lut_grid_nb27, "null buffer");
    return separable_impl(inputs, weights_1d, grid_indices, nullptr, nullptr, lut_grid_nb27, outputs, num_grids, n_emb, G,
                          radius, D, st);
}

int ashb_filter_separable_inplace(float* values, float* scratch, const float* weights_1d, const int32_t* list,
                                  const int32_t* list_count, const int64_t* lut_grid_nb27, int64_t n_emb, int G,
                                  int radius, int64_t D, void* stream) {
    ASHB_REQUIRE(D >= 1 && D <= 16, "embedding_dim %lld not in 1..16", (long long)D);
    ASHB_REQUIRE(G >= 1 && G <= 16 && radius >= 1 && radius <= G, "window radius %d must be within one block (G=%d)",
                 radius, G);
    ASHB_REQUIRE(n_emb >= 1 && n_emb <= 0x7fffffffll, "bad sizes");
    ASHB_REQUIRE(values && scratch && weights_1d && list && list_count && lut_grid_nb27, "null buffer");
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    if (int rc = separable_impl(values, weights_1d, nullptr, list, list_count, lut_grid_nb27, scratch, 0, n_emb, G, radius, D,
                                st))
        return rc;
    const int64_t row = (int64_t)G * G * G * D;
    const unsigned ctas = (unsigned)(n_emb < sm_count() * 8ll ? n_emb : sm_count() * 8ll);
    if (row % 4 == 0 && (((uintptr_t)values | (uintptr_t)scratch) & 15) == 0)
        restore_rows_kernel<float4><<<ctas, 256, 0, st>>>(reinterpret_cast<float4*>(values),
                                                          reinterpret_cast<const float4*>(scratch), lut_grid_nb27, n_emb,
                                                          (int)(row / 4));
    else
        restore_rows_kernel<float><<<ctas, 256, 0, st>>>(values, scratch, lut_grid_nb27, n_emb, (int)row);
    ASHB_LAUNCH_CHECK();
    return ASHB_OK;
}

}  // extern "C"
