// Triangle mesh of the iso-surface over the sparse-dense structure (sm_100a): marching cubes
// in four launches and ONE host read.  Stages and validity rules follow ash/src/grid.cu:607-946:
// a cube sits at every cell of a listed block whose own weight and the weights of its 8 corners
// (the cell and its +x/+y/+z neighbours through the lookup tables) reach the threshold and whose
// neighbour blocks all exist; corner c is inside when sdf - iso < 0; every cut edge of a valid
// cube gets one vertex, owned by the cell at the edge's lower corner, placed by linear
// interpolation; triangles index those vertices.
//
//   check      whether the cell tables are the usual ones, which classify then need not read
//   classify   per tile of blocks: corner pattern -> codes[]; each cut edge is requested at its owner
//              as one bit of a byte per cell, so the number of distinct vertices is counted in the
//              same pass, as is the number of triangles
//   (host reads the two counts and allocates)
//   vertices   per 1024 cells (256 in short lists): requested edges get consecutive slots and positions
//   triangles  likewise: triangles get consecutive slots, vertex ids looked up at the owners
//
// The last three are bound by instructions and latency, not bytes: what they shed is work per CELL where only one
// cell in twelve carries surface.  24,000 blocks of 8^3 on a B200: 444 + 114 + 107 us when every cell
// read its eight corners through the tables, each warp bumped the shared counters and an edge took
// four bytes of a 147 MB table that had to be filled, written and read; 60 + 39 + 57 us now.
//
// The triangulation table is this repository's own (mc_tables.h, derived by gen_mc_tables.py):
// the reference's table is not reproduced, so which diagonal splits an ambiguous pattern, the
// order of a triangle's corners and the output order are not comparable with the reference;
// vertex positions are.
#include <algorithm>

#include "common.cuh"

#define ASHB_MC_TABLE static __device__ const
#include "mc_tables.h"

namespace ashb {

// Scratch of a surface (ashb200.h: edge_vertex): the id of the first vertex of every cell, then one byte
// per cell -- bits 0..2: the edge along x / y / z leaving the cell is cut by a valid cube; bit 3: its
// vertices have ids -- and a word that says the cell tables are not the usual ones.
constexpr uint32_t kHasVertices = 8;
struct McEdges {
    int* __restrict__ first_vertex;
    uint8_t* __restrict__ wanted;
    uint32_t* __restrict__ odd_tables;
};

struct McLuts {
    const int64_t* __restrict__ grid_indices;
    const int64_t* __restrict__ g2g;
    const int64_t* __restrict__ c2c;
    const int64_t* __restrict__ c2g;
    int64_t cells, n_emb, len;
    int shift;  // log2(cells), or -1

    // Position in the block list and cell of the i-th cell of the list.
    __device__ __forceinline__ void split(int64_t i, int64_t& pos, int64_t& cell) const {
        if (shift >= 0) {   // a 64-bit division costs more than the rest of an inactive cell
            pos = i >> shift;
            cell = i & (cells - 1);
        } else {
            pos = i / cells;
            cell = i - pos * cells;
        }
    }
};

// Flat (embedding row * cells + cell) address of corner c of the cube at (grid_idx, cell_idx), or -1.
__device__ __forceinline__ int64_t corner_address(const McLuts& L, int64_t grid_idx, int64_t cell_idx, int c) {
    const int64_t g = L.g2g[grid_idx * 8 + (L.c2g[cell_idx * 8 + c] & 7)];
    if (g < 0 || g >= L.n_emb) return -1;
    const int64_t cc = L.c2c[cell_idx * 8 + c];
    if (cc < 0 || cc >= L.cells) return -1;
    return g * L.cells + cc;
}

__device__ __forceinline__ int edge_lower_corner(int e) {
    const int d = e >> 2, j = e & 3;
    return ((j & 1) << ((d + 1) % 3)) | ((j >> 1) << ((d + 2) % 3));
}

// Requests edges (bits 0..2 of `bits`) of the cell at flat address `a`; returns how many are new.
__device__ __forceinline__ int request_edges(uint8_t* wanted, int64_t a, uint32_t bits) {
    const int at = (int)(a & 3) * 8;
    const uint32_t old = atomicOr(reinterpret_cast<uint32_t*>(wanted + (a - (a & 3))), bits << at);
    return __popc(bits & ~(old >> at));
}

// Marks the vertices of the requested cells among the four at flat address `a` (a multiple of 4) as placed; returns the
// requests (bits 0..2 of each byte) that this call marked first: a block may be listed twice.
__device__ __forceinline__ uint32_t claim_vertices(uint8_t* wanted, int64_t a, uint32_t cells) {
    uint32_t* word = reinterpret_cast<uint32_t*>(wanted + a);
    const uint32_t want = *word & 0x07070707u & cells;
    if (want == 0u) return 0u;
    const uint32_t marks = ((want | want >> 1 | want >> 2) & 0x01010101u) << 3;
    return want & ~((atomicOr(word, marks) >> 3 & 0x01010101u) * 7u);
}

// Raises odd_tables unless corner k of cell (x, y, z) is, in both cell tables, the cell at + k's offsets.
__global__ void __launch_bounds__(256) mc_check_tables_kernel(McLuts L, McEdges edges, int G) {
    const int e = blockIdx.x * blockDim.x + threadIdx.x;
    if (e >= L.cells * 8) return;
    const int cell = e >> 3;
    const int x = cell % G + (e & 1), y = cell / G % G + ((e >> 1) & 1), z = cell / (G * G) + ((e >> 2) & 1);
    const int nb = (x == G) | (y == G) << 1 | (z == G) << 2;
    const int at = x % G + (y % G + z % G * G) * G;
    if ((L.c2g[e] & 7) != nb || L.c2c[e] != at) atomicExch(edges.odd_tables, 1u);
}

constexpr int kMaxTileBlocks = 32;
constexpr int kMaxFastEdge = 16;
constexpr int kMaxTileRows = (kMaxFastEdge + 1) * (kMaxFastEdge + 1);   // no less than 256
constexpr int kClassifyCtas = 6;   // per SM

// Bits 0..3 to the low bits of four bytes.
__device__ __forceinline__ uint32_t spread_bits(uint32_t bits) { return (bits & 15u) * 0x00204081u & 0x01010101u; }

// A CTA walks tiles of blocks: as many as have 256 rows of cells between them, counting the layer of rows that a block's
// upper neighbours add, (G + 1)^2 a block.  A row of G cells and the neighbour's first one is two words of bits, observed
// and inside, made by one thread from wide loads (1.42 values a cell at G = 8: the upper neighbours' layer too); a
// cube, an edge and whether it is cut are then the same bit of a few such words, for all cells of a row at once.  Only
// cubes with surface are looked at one by one, for their code.  Requested edges leave as a word of four cells; the
// two counters see one atomic per CTA.  Bound by latency and the values' traffic: 24,000 blocks of 8^3 60 us, 130 with a
// state byte per cell, eight of them read per cube and the edges requested corner by corner; a warp per block of
// 8^3 instead of a CTA per three 56, but 2,000 and 200 blocks 11.5 and 10.6 us for 8.1 and 6.1.
// GT: the block edge where it is known when compiling, 0 otherwise.  wide: rows and codes are aligned for GT's loads and
// stores.  Cell tables that are not the usual ones (odd_tables), and edges beyond kMaxFastEdge (G = 0), take the
// corners from the tables.
template <int GT>
__global__ void __launch_bounds__(256, kClassifyCtas) mc_classify_kernel(const float* __restrict__ sdfs,
                                                          const float* __restrict__ weights, McLuts L,
                                                          uint8_t* __restrict__ codes, McEdges edges,
                                                          unsigned long long* __restrict__ counters, float iso_value,
                                                          float weight_thr, int G_arg, int64_t num_grids,
                                                          bool wide) {
    // behind the last row: what the rows above it read, and then mask
    __shared__ uint32_t inside[kMaxTileRows + kMaxFastEdge + 1], observed[kMaxTileRows + kMaxFastEdge + 1];
    __shared__ uint32_t cubes[kMaxTileRows];   // whose eight corners are observed
    __shared__ int64_t rows[kMaxTileBlocks * 8];
    __shared__ uint8_t tri_count[256];
    const int tid = threadIdx.x;
    tri_count[tid] = kMcTriCount[tid];   // launched with 256 threads
    __syncthreads();
    int n_vertices = 0, n_triangles = 0;
    const int G = GT ? GT : G_arg;
    if (G == 0 || *edges.odd_tables != 0) {
        for (int64_t i = (int64_t)blockIdx.x * 256 + tid; i < L.len; i += (int64_t)gridDim.x * 256) {
            int64_t pos, cell_idx, corner[8];
            L.split(i, pos, cell_idx);
            const int64_t grid_idx = L.grid_indices[pos];
            bool valid = grid_idx >= 0 && grid_idx < L.n_emb;
            int code = 0;
#pragma unroll
            for (int c = 0; c < 8; ++c) {
                corner[c] = valid ? corner_address(L, grid_idx, cell_idx, c) : -1;
                valid = valid && corner[c] >= 0;
            }
            if (valid) {
#pragma unroll
                for (int c = 0; c < 8; ++c) {
                    valid = valid && weights[corner[c]] >= weight_thr;
                    code |= (int)((sdfs[corner[c]] - iso_value) < 0.f) << c;
                }
            }
            if (!valid || code == 255) code = 0;
            codes[i] = (uint8_t)code;
            const int mask = kMcEdgeMask[code];
#pragma unroll
            for (int e = 0; e < 12; ++e)
                if (mask & (1 << e)) n_vertices += request_edges(edges.wanted, corner[edge_lower_corner(e)], 1u << (e >> 2));
            n_triangles += tri_count[code];
        }
    } else {
        const int H = G + 1, HH = H * H, cells = G * G * G;
        const uint32_t all_cells = (1u << G) - 1u;
        const int per_tile = min(max(256 / HH, 1), kMaxTileBlocks);
        const int64_t n_tiles = (num_grids + per_tile - 1) / per_tile;
        // embedding row of one of a tile's blocks or of one of its upper neighbours, or -1
        auto row_of = [&](int64_t tile) -> int64_t {
            const int64_t at = tile * per_tile + (tid >> 3);
            if (tid >= per_tile * 8 || at >= num_grids) return -1;
            const int64_t g = L.grid_indices[at];
            const int64_t nb = g >= 0 && g < L.n_emb ? L.g2g[g * 8 + (tid & 7)] : -1;
            return nb < L.n_emb ? nb : -1;
        };
        // the block of the tile that row r of the tile's halo is in, its y and z there, which neighbour (and the next in x) owns
        // the row and the flat place of its first cell within a block
        struct Row {
            int b, y, z, nb, at;
        };
        auto halo_row = [&](int r) {
            const int b = r / HH, q = r - b * HH, z = q / H, y = q - z * H;
            return Row{b, y, z, (y == G) << 1 | (z == G) << 2, ((y == G ? 0 : y) + (z == G ? 0 : z) * G) * G};
        };
        int64_t row = row_of(blockIdx.x);
        for (int64_t tile = blockIdx.x; tile < n_tiles; tile += gridDim.x) {
            const int64_t first = tile * per_tile;
            const int blocks = per_tile == 1 ? 1 : (int)min((int64_t)per_tile, num_grids - first);
            if (tid < per_tile * 8) rows[tid] = row;
            __syncthreads();
            row = row_of(tile + gridDim.x);   // two dependent loads that the rest of the tile covers
            for (int r = tid; r < blocks * HH; r += 256) {
                const Row h = halo_row(r);
                const int64_t own = rows[h.b * 8 + h.nb], next = rows[h.b * 8 + h.nb + 1];
                uint32_t in = 0, seen = 0;
                auto cell = [&](int x, float d, float w) {
                    in |= (uint32_t)(d - iso_value < 0.f) << x;
                    seen |= (uint32_t)(w >= weight_thr) << x;
                };
                if (next >= 0) cell(G, sdfs[next * cells + h.at], weights[next * cells + h.at]);
                if (own >= 0) {
                    const float *d = sdfs + own * cells + h.at, *w = weights + own * cells + h.at;
                    if (GT && wide) {
#pragma unroll
                        for (int x = 0; x < GT; x += 4) {
                            const float4 d4 = *reinterpret_cast<const float4*>(d + x), w4 = *reinterpret_cast<const float4*>(w + x);
                            cell(x, d4.x, w4.x), cell(x + 1, d4.y, w4.y), cell(x + 2, d4.z, w4.z), cell(x + 3, d4.w, w4.w);
                        }
                    } else {
                        for (int x = 0; x < G; ++x) cell(x, d[x], w[x]);
                    }
                }
                inside[r] = in;
                observed[r] = seen;
                if (h.y == G || h.z == G) cubes[r] = 0;
            }
            __syncthreads();
            for (int c = tid; c < blocks * G * G; c += 256) {   // a row of cubes
                const int b = c / (G * G), yz = c - b * G * G, z = yz / G, y = yz - z * G, r = b * HH + y + z * H;
                const uint32_t i0 = inside[r], i1 = inside[r + 1], i2 = inside[r + H], i3 = inside[r + H + 1];
                uint32_t seen = observed[r] & observed[r + 1] & observed[r + H] & observed[r + H + 1];
                seen &= seen >> 1 & all_cells;
                cubes[r] = seen;
                const uint32_t any = i0 | i1 | i2 | i3, all = i0 & i1 & i2 & i3;
                uint32_t surface = (any | any >> 1) & ~(all & all >> 1) & seen;
                uint8_t* to = codes + first * cells + (int64_t)b * cells + yz * G;
                constexpr int kWords = GT ? GT / 4 : 1;
                uint32_t words[kWords] = {};
                if (!(GT && wide))
                    for (int x = 0; x < G; ++x) to[x] = 0;
                for (; surface; surface &= surface - 1) {
                    const int x = __ffs(surface) - 1;
                    const uint32_t code = (i0 >> x & 3u) | (i1 >> x & 3u) << 2 | (i2 >> x & 3u) << 4 | (i3 >> x & 3u) << 6;
                    n_triangles += tri_count[code];
                    if (GT && wide) {
#pragma unroll
                        for (int k = 0; k < kWords; ++k)
                            if (x >> 2 == k) words[k] |= code << (8 * (x & 3));
                    } else {
                        to[x] = (uint8_t)code;
                    }
                }
                if (GT && wide) {
                    if constexpr (kWords == 1) *reinterpret_cast<uint32_t*>(to) = words[0];
#pragma unroll
                    for (int k = 0; k + 1 < kWords; k += 2) *reinterpret_cast<uint2*>(to + 4 * k) = make_uint2(words[k], words[k + 1]);
                }
            }
            __syncthreads();
            for (int r = tid; r < blocks * HH; r += 256) {   // the edges that leave a row's cells, cut and in a cube
                const Row h = halo_row(r);
                const uint32_t v = cubes[r], vy = h.y > 0 ? cubes[r - 1] : 0u, vz = h.z > 0 ? cubes[r - H] : 0u,
                               vyz = h.y > 0 && h.z > 0 ? cubes[r - H - 1] : 0u;
                if ((v | vy | vz | vyz) == 0u) continue;
                const uint32_t i = inside[r], cy = v | vz, cz = v | vy;
                const uint32_t wx = (i ^ i >> 1) & (v | vy | vz | vyz), wy = (i ^ inside[r + 1]) & (cy | cy << 1),
                               wz = (i ^ inside[r + H]) & (cz | cz << 1);
                if ((wx | wy | wz) == 0u) continue;
                const int64_t a = rows[h.b * 8 + h.nb] * cells + h.at;
                if (GT) {
                    uint32_t bits[GT ? GT / 4 : 1], old[GT ? GT / 4 : 1];
#pragma unroll
                    for (int k = 0; k < GT / 4; ++k) {   // all on their way before the first is waited for
                        bits[k] = spread_bits(wx >> 4 * k) | spread_bits(wy >> 4 * k) << 1 | spread_bits(wz >> 4 * k) << 2;
                        old[k] = 0;
                        if (bits[k]) old[k] = atomicOr(reinterpret_cast<uint32_t*>(edges.wanted + a + 4 * k), bits[k]);
                    }
#pragma unroll
                    for (int k = 0; k < GT / 4; ++k) n_vertices += __popc(bits[k] & ~old[k]);
                } else {
                    for (uint32_t left = (wx | wy | wz) & all_cells; left; left &= left - 1) {
                        const int x = __ffs(left) - 1;
                        n_vertices += request_edges(edges.wanted, a + x, (wx >> x & 1u) | (wy >> x & 1u) << 1 | (wz >> x & 1u) << 2);
                    }
                }
                const uint32_t last = (wy >> G & 1u) << 1 | (wz >> G & 1u) << 2;   // of the next block's first cell
                if (last) n_vertices += request_edges(edges.wanted, rows[h.b * 8 + h.nb + 1] * cells + h.at, last);
            }
            __syncthreads();   // rows and the words are used again
        }
    }
    __shared__ int sums[2];
    if (tid < 2) sums[tid] = 0;
    __syncthreads();
    n_vertices = __reduce_add_sync(0xffffffffu, n_vertices);
    n_triangles = __reduce_add_sync(0xffffffffu, n_triangles);
    if ((tid & 31) == 0) {
        if (n_vertices) atomicAdd(sums, n_vertices);
        if (n_triangles) atomicAdd(sums + 1, n_triangles);
    }
    __syncthreads();
    if (tid < 2 && sums[tid]) atomicAdd(counters + tid, (unsigned long long)sums[tid]);
}

// Cells of a thread in the two passes below: four in large lists, one up to here, where CTAs of 1024 cells would be less
// than two per SM, each working off a list of round trips (grid.marching_cubes of 125 and of 343 blocks of 8^3 full of
// surface: 212 -> 169 and 214 -> 171 us).
constexpr int kFewCells = 300000;

// Exclusive prefix of `mine` over the CTA of 256 threads, and the start of its range of `cursor`.
__device__ __forceinline__ int reserve_range(int mine, unsigned long long* cursor, int& total, int64_t& base) {
    __shared__ int warp_total[8];
    __shared__ unsigned long long start;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    int incl = mine;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const int u = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= o) incl += u;
    }
    if (lane == 31) warp_total[warp] = incl;
    __syncthreads();
    int before = 0;
    total = 0;
#pragma unroll
    for (int w = 0; w < 8; ++w) {
        if (w < warp) before += warp_total[w];
        total += warp_total[w];
    }
    if (threadIdx.x == 0 && total) start = atomicAdd(cursor, (unsigned long long)total);
    __syncthreads();
    base = total ? (int64_t)start : 0;
    return before + incl - mine;
}

// The threads read the request bytes of their cells; the requested edges of the CTA are listed in shared
// memory and the list is worked off by all threads, so positions are computed without idle lanes
// and leave as one contiguous run.
template <int EACH>
__global__ void __launch_bounds__(256) mc_vertex_kernel(const float* __restrict__ sdfs, McLuts L,
                                                        const int32_t* __restrict__ grid_coords,
                                                        const int32_t* __restrict__ cell_coords, McEdges edges,
                                                        unsigned long long* __restrict__ cursor,
                                                        float* __restrict__ vertices, int64_t max_vertices,
                                                        float iso_value, int grid_dim) {
    __shared__ uint16_t list[3 * 256 * EACH];
    const int64_t i0 = (int64_t)blockIdx.x * 256 * EACH;
    uint32_t bits[EACH];
    int64_t address[EACH];
    int mine = 0;
    // block and cell of the thread's j-th cell as its flat address, or -1
    auto address_of = [&](int j) -> int64_t {
        const int64_t i = i0 + EACH * threadIdx.x + j;
        if (i >= L.len) return -1;
        int64_t pos, cell_idx;
        L.split(i, pos, cell_idx);
        const int64_t grid_idx = L.grid_indices[pos];
        return grid_idx >= 0 && grid_idx < L.n_emb ? grid_idx * L.cells + cell_idx : -1;
    };
    if (EACH == 4 && (L.cells & 3) == 0) {   // one word of one block
        const int64_t a = address_of(0);
        const uint32_t want = a >= 0 ? claim_vertices(edges.wanted, a, ~0u) : 0u;
#pragma unroll
        for (int j = 0; j < EACH; ++j) {
            address[j] = a + j;
            bits[j] = (want >> (8 * j)) & 7u;
        }
    } else {
#pragma unroll
        for (int j = 0; j < EACH; ++j) {
            const int64_t a = address[j] = address_of(j);
            const int at = (int)(a & 3) * 8;
            bits[j] = a >= 0 ? claim_vertices(edges.wanted, a - (a & 3), 0xFFu << at) >> at : 0u;
        }
    }
#pragma unroll
    for (int j = 0; j < EACH; ++j) mine += __popc(bits[j]);
    int total;
    int64_t base;
    int at = reserve_range(mine, cursor, total, base);
    if (total == 0) return;
#pragma unroll
    for (int j = 0; j < EACH; ++j) {
        if (bits[j] == 0) continue;
        edges.first_vertex[address[j]] = (int)(base + at);
#pragma unroll
        for (int d = 0; d < 3; ++d)
            if (bits[j] & (1u << d)) list[at++] = (uint16_t)((EACH * threadIdx.x + j) * 4 + d);
    }
    __syncthreads();
    for (int e = threadIdx.x; e < total; e += 256) {
        const int d = list[e] & 3;
        int64_t pos, cell_idx;
        L.split(i0 + (list[e] >> 2), pos, cell_idx);
        const int64_t grid_idx = L.grid_indices[pos], o = base + e;
        const int64_t nb = corner_address(L, grid_idx, cell_idx, 1 << d);
        if (o >= max_vertices || nb < 0) continue;  // cannot happen for edges a valid cube requested
        const float self_iso = sdfs[grid_idx * L.cells + cell_idx] - iso_value;
        const float nb_iso = sdfs[nb] - iso_value;
        const float ratio = self_iso / (self_iso - nb_iso);
#pragma unroll
        for (int k = 0; k < 3; ++k) {
            const int self_pos = grid_coords[grid_idx * 3 + k] * grid_dim + cell_coords[cell_idx * 3 + k];
            vertices[o * 3 + k] = (float)self_pos + (k == d ? ratio : 0.f);
        }
    }
}

// The same for triangles: the CTA lists them, then a thread per corner looks its vertex up.
template <int EACH>
__global__ void __launch_bounds__(256) mc_triangle_kernel(McLuts L, const uint8_t* __restrict__ codes, McEdges edges,
                                                          unsigned long long* __restrict__ cursor,
                                                          int32_t* __restrict__ triangles, int64_t max_triangles) {
    __shared__ uint16_t list[ASHB_MC_MAX_TRIS * 256 * EACH];
    __shared__ uint8_t code_of[256 * EACH];
    const int64_t i0 = (int64_t)blockIdx.x * 256 * EACH;
    int count[EACH];
    int mine = 0;
#pragma unroll
    for (int j = 0; j < EACH; ++j) {
        const int64_t i = i0 + EACH * threadIdx.x + j;
        const int code = i < L.len ? codes[i] : 0;
        count[j] = code ? (int)kMcTriCount[code] : 0;
        code_of[EACH * threadIdx.x + j] = (uint8_t)code;
        mine += count[j];
    }
    int total;
    int64_t base;
    int at = reserve_range(mine, cursor, total, base);
    if (total == 0) return;
#pragma unroll
    for (int j = 0; j < EACH; ++j)
        for (int t = 0; t < count[j]; ++t) list[at++] = (uint16_t)((EACH * threadIdx.x + j) * 8 + t);
    __syncthreads();
    for (int m = threadIdx.x; m < 3 * total; m += 256) {
        const int t = m / 3, v = m - 3 * t;
        if (base + t >= max_triangles) return;
        const int local = list[t] >> 3;
        const int e = kMcTris[code_of[local]][3 * (list[t] & 7) + v];
        int64_t pos, cell_idx;
        L.split(i0 + local, pos, cell_idx);
        const int64_t owner = corner_address(L, L.grid_indices[pos], cell_idx, edge_lower_corner(e));
        int id = -1;   // the owner's block is not listed
        if (owner >= 0) {
            const uint32_t bits = edges.wanted[owner];
            if (bits & kHasVertices) id = edges.first_vertex[owner] + __popc(bits & ((1u << (e >> 2)) - 1));
        }
        triangles[base * 3 + m] = id;
    }
}

}  // namespace ashb

using namespace ashb;

static McLuts mc_luts(const int64_t* grid_indices, const int64_t* g2g, const int64_t* c2c, const int64_t* c2g, int64_t cells,
                      int64_t n_emb, int64_t num_grids) {
    int shift = 0;
    while ((1ll << shift) < cells) ++shift;
    return McLuts{grid_indices, g2g, c2c, c2g, cells, n_emb, num_grids * cells, (1ll << shift) == cells ? shift : -1};
}

// Five bytes per cell and the word behind them, in the caller's twelve bytes per cell.
static McEdges mc_edges(int32_t* scratch, int64_t n) {
    uint8_t* wanted = reinterpret_cast<uint8_t*>(scratch + n);
    return McEdges{scratch, wanted, reinterpret_cast<uint32_t*>(wanted + (n + 3) / 4 * 4)};
}

extern "C" {

int ashb_marching_cubes_count(const float* sdfs, const float* weights, const int64_t* grid_indices,
                              const int64_t* lut_grid_nb2grid_idx, const int64_t* lut_cell_nb2cell_idx,
                              const int64_t* lut_cell_nb2grid_nb, uint8_t* codes, int32_t* edge_vertex,
                              void* counters_dev, float iso_value, float weight_thr, int64_t cells_per_grid,
                              int64_t n_emb, int64_t num_grids, int64_t* n_vertices, int64_t* n_triangles,
                              void* stream) {
    ASHB_REQUIRE(n_vertices && n_triangles && counters_dev, "null counter");
    ASHB_REQUIRE(num_grids >= 0 && cells_per_grid >= 1 && n_emb >= 1, "bad sizes");
    *n_vertices = *n_triangles = 0;
    if (num_grids == 0) return ASHB_OK;
    ASHB_REQUIRE(sdfs && weights && grid_indices && lut_grid_nb2grid_idx && lut_cell_nb2cell_idx &&
                         lut_cell_nb2grid_nb && codes && edge_vertex,
                 "null buffer");
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    unsigned long long* counters = static_cast<unsigned long long*>(counters_dev);
    ASHB_CUDA_TRY(cudaMemsetAsync(counters, 0, 2 * sizeof(unsigned long long), st));
    const int64_t n = n_emb * cells_per_grid;
    const McEdges edges = mc_edges(edge_vertex, n);
    ASHB_CUDA_TRY(cudaMemsetAsync(edges.wanted, 0, (size_t)(n + 3) / 4 * 4 + sizeof(uint32_t), st));
    const McLuts L = mc_luts(grid_indices, lut_grid_nb2grid_idx, lut_cell_nb2cell_idx, lut_cell_nb2grid_nb, cells_per_grid,
                             n_emb, num_grids);
    int G = 2;
    while (G < kMaxFastEdge && (int64_t)G * G * G < cells_per_grid) ++G;
    if ((int64_t)G * G * G != cells_per_grid) G = 0;
    if (G) {
        mc_check_tables_kernel<<<(unsigned)((cells_per_grid * 8 + 255) / 256), 256, 0, st>>>(L, edges, G);
        ASHB_LAUNCH_CHECK();
    }
    // persistent: one resident set of CTAs shares out the tiles (9 each at 24,000 blocks)
    const unsigned grid = (unsigned)std::min<int64_t>((L.len + 255) / 256, (int64_t)sm_count() * kClassifyCtas);
    const bool wide = (((uintptr_t)sdfs | (uintptr_t)weights) & 15) == 0 && ((uintptr_t)codes & 7) == 0;
    auto kernel = G == 8 ? mc_classify_kernel<8> : G == 4 ? mc_classify_kernel<4> : G == 16 ? mc_classify_kernel<16>
                                                                                        : mc_classify_kernel<0>;
    kernel<<<grid, 256, 0, st>>>(sdfs, weights, L, codes, edges, counters, iso_value, weight_thr, G, num_grids, wide);
    ASHB_LAUNCH_CHECK();
    unsigned long long host[2] = {0, 0};
    ASHB_CUDA_TRY(cudaMemcpyAsync(host, counters, sizeof(host), cudaMemcpyDeviceToHost, st));
    ASHB_CUDA_TRY(cudaStreamSynchronize(st));
    *n_vertices = (int64_t)host[0];
    *n_triangles = (int64_t)host[1];
    return ASHB_OK;
}

int ashb_marching_cubes_fill(const float* sdfs, const int64_t* grid_indices, const int32_t* grid_coords_table,
                             const int64_t* lut_grid_nb2grid_idx, const int32_t* cell_coords_table,
                             const int64_t* lut_cell_nb2cell_idx, const int64_t* lut_cell_nb2grid_nb,
                             const uint8_t* codes, int32_t* edge_vertex, void* counters_dev, float* vertices,
                             int64_t n_vertices, int32_t* triangles, int64_t n_triangles, float iso_value,
                             int grid_dim, int64_t cells_per_grid, int64_t n_emb, int64_t num_grids, void* stream) {
    ASHB_REQUIRE(num_grids >= 0 && cells_per_grid >= 1 && n_emb >= 1 && n_vertices >= 0 && n_triangles >= 0,
                 "bad sizes");
    if (num_grids == 0 || (n_vertices == 0 && n_triangles == 0)) return ASHB_OK;
    ASHB_REQUIRE(sdfs && grid_indices && grid_coords_table && lut_grid_nb2grid_idx && cell_coords_table &&
                         lut_cell_nb2cell_idx && lut_cell_nb2grid_nb && codes && edge_vertex && counters_dev,
                 "null buffer");
    ASHB_REQUIRE((n_vertices == 0 || vertices) && (n_triangles == 0 || triangles), "null output");
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    unsigned long long* counters = static_cast<unsigned long long*>(counters_dev);
    ASHB_CUDA_TRY(cudaMemsetAsync(counters, 0, 2 * sizeof(unsigned long long), st));
    const McLuts L = mc_luts(grid_indices, lut_grid_nb2grid_idx, lut_cell_nb2cell_idx, lut_cell_nb2grid_nb, cells_per_grid,
                             n_emb, num_grids);
    const McEdges edges = mc_edges(edge_vertex, n_emb * cells_per_grid);
    const bool few = L.len < kFewCells;
    const int64_t pass_cells = few ? 256 : 1024;
    const unsigned grid = (unsigned)((L.len + pass_cells - 1) / pass_cells);
    (few ? mc_vertex_kernel<1> : mc_vertex_kernel<4>)<<<grid, 256, 0, st>>>(
            sdfs, L, grid_coords_table, cell_coords_table, edges, counters, vertices, n_vertices, iso_value, grid_dim);
    ASHB_LAUNCH_CHECK();
    (few ? mc_triangle_kernel<1> : mc_triangle_kernel<4>)<<<grid, 256, 0, st>>>(L, codes, edges, counters + 1, triangles,
                                                                                n_triangles);
    ASHB_LAUNCH_CHECK();
    return ASHB_OK;
}

}  // extern "C"
