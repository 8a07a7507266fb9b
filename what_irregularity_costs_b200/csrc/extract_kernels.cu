// Extract: marching-tetrahedra triangle soup over every allocated block.
//
// Reference: cpp/src/marching_tets.cpp:31-245 (CPU arm) and
// cpp/src/marching_tets_cuda.cu:33-167 (CUDA arm: one CTA per block, one
// thread per cube, a full hash probe for each of the 8 corners of every cube
// and one global atomic per emitting tetrahedron).
//
// B200 design. A resident grid of 128-thread CTAs takes one block after the
// other (the block count is read on the device). The 7 neighbour blocks are
// looked up once per block and the 9x9x9 halo of corner samples (mean TSDF,
// mean colour) is staged in shared memory, three rows of nine a warp, so that
// two ballots give the rows' validity and below-iso bits. One warp finds the
// cubes with a sign change from those bits, a row of eight cubes at a time
// (about 45 of a block's 512), counts their triangles, reserves the block's
// output range with one atomic and lists the triangles in a fixed order
// (cube, then tetrahedron). Each warp then takes 32 triangles at a time, stages
// their vertices and writes them out by itself.
//
// What bounds it: the latency of its instructions (36 M warp instructions for
// 6,243 blocks and 1.34 M triangles, issue slots 47 % used at the 40 warps an SM
// that the registers allow). A 512-thread CTA per block with a thread per cube
// took 57 M and 120 us on a room of 8,468 blocks and 5.35 M vertices, against
// 90; a quarter of its instructions listed triangles cube by cube, another
// looked up the cases and ordered the corners of every edge. Looking the next
// block up ahead of time changed nothing (90.5).
//
// Arithmetic follows the reference operation for operation, unfused, so a
// volume whose voxels match bit-for-bit extracts bit-identical vertices.
#include <algorithm>
#include <mutex>

#include "volume.h"

namespace osn_b200 {
namespace {

constexpr int kExtractThreads = 128;
constexpr int kExtractWarps = kExtractThreads / 32;
constexpr int kResetThreads = 128;
constexpr int kHalo = 9;
constexpr int kHaloRows = kHalo * kHalo;  // rows of nine cells along x
constexpr int kHaloCells = kHaloRows * kHalo;

// marching_tets.cpp:37-40: six tetrahedra around the 0-7 diagonal.
__host__ __device__ constexpr int tet_corner(int k, int i) {
    constexpr int corners[6][4] = {
        {0, 5, 1, 7}, {0, 1, 3, 7}, {0, 3, 2, 7}, {0, 6, 4, 7}, {0, 4, 5, 7}, {0, 2, 6, 7},
    };
    return corners[k][i];
}

// A tetrahedron's case code (bit i: its corner i is below iso) gives its
// crossing (marching_tets.cpp:165-182): none (0000, 1111), one triangle from
// the corner on its own side (one or three bits set), or a quad split in two
// (two bits set).
constexpr int popc4(int x) { return (x & 1) + ((x >> 1) & 1) + ((x >> 2) & 1) + ((x >> 3) & 1); }
constexpr int tris_of_code(int code) { return (popc4(code) & 1) ? 1 : (popc4(code) == 2 ? 2 : 0); }
constexpr int tet_code(int below, int k) {
    int code = 0;
    for (int i = 0; i < 4; ++i) code |= ((below >> tet_corner(k, i)) & 1) << i;
    return code;
}

constexpr int corner_offset(int c) { return (c & 1) + ((c >> 1) & 1) * kHalo + ((c >> 2) & 1) * kHaloRows; }
// The corner with the smaller position (x, then y, then z) comes first in an
// interpolation (marching_tets.cpp:59-80). Corner positions are increasing
// functions of the corner's offset bits on each axis (same cube), so comparing
// the offsets (x, y, z) as a 3-bit number orders the positions exactly.
constexpr int corner_rank(int c) { return ((c & 1) << 2) | (c & 2) | ((c >> 2) & 1); }

// Tables the kernel stages in shared memory (constant-bank reads with lane-
// dependent indices would serialise):
//   kinds[below]     the six tetrahedra's triangle counts (2 bits each) of a
//                    cube whose corners below iso are the bits of `below`;
//   first[k][code]   the first of tetrahedron k's triangles in `tri`;
//   tri[n]           a triangle's three edges, each as its two corners in
//                    interpolation order: .x, .y their offsets in the halo (one
//                    byte each), .z their offset bits (3 each).
constexpr int kTetTris = 20;  // 8 codes of one triangle, 6 of two
struct alignas(16) TetTables {
    uint4 tri[6 * kTetTris];
    uint16_t kinds[256];
    uint8_t first[6][16];
};
static_assert(sizeof(TetTables) % 4 == 0, "copied by words");
constexpr int case_perm(int code) {  // (a, b, c, d) as positions in the tetrahedron
    switch (code) {
        case 0x01: case 0x0E: case 0x03: return 0 | 1 << 2 | 2 << 4 | 3 << 6;
        case 0x02: case 0x0D: return 1 | 0 << 2 | 2 << 4 | 3 << 6;
        case 0x04: case 0x0B: return 2 | 0 << 2 | 1 << 4 | 3 << 6;
        case 0x08: case 0x07: return 3 | 0 << 2 | 1 << 4 | 2 << 6;
        case 0x0C: return 2 | 3 << 2 | 0 << 4 | 1 << 6;
        case 0x05: return 0 | 2 << 2 | 1 << 4 | 3 << 6;
        case 0x0A: return 1 | 3 << 2 | 0 << 4 | 2 << 6;
        case 0x06: return 1 | 2 << 2 | 0 << 4 | 3 << 6;
        case 0x09: return 0 | 3 << 2 | 1 << 4 | 2 << 6;
        default: return 0;
    }
}
constexpr uint4 make_tri(const int (&edges)[3][2]) {
    uint32_t off[2] = {0u, 0u}, bits = 0u;
    for (int e = 0; e < 3; ++e) {
        const bool swap = corner_rank(edges[e][1]) < corner_rank(edges[e][0]);
        for (int i = 0; i < 2; ++i) {
            const int c = edges[e][swap ? 1 - i : i], n = 2 * e + i;
            off[n / 4] |= (uint32_t)corner_offset(c) << (8 * (n % 4));
            bits |= (uint32_t)c << (3 * n);
        }
    }
    return uint4{off[0], off[1], bits, 0u};
}
constexpr TetTables make_tet_tables() {
    TetTables t{};
    for (int b = 0; b < 256; ++b) {
        int v = 0;
        for (int k = 0; k < 6; ++k) v |= tris_of_code(tet_code(b, k)) << (2 * k);
        t.kinds[b] = (uint16_t)v;
    }
    int n = 0;
    for (int k = 0; k < 6; ++k) {
        for (int code = 0; code < 16; ++code) {
            const int p = case_perm(code);
            const int a = tet_corner(k, p & 3), b = tet_corner(k, (p >> 2) & 3), c = tet_corner(k, (p >> 4) & 3),
                      d = tet_corner(k, (p >> 6) & 3);
            t.first[k][code] = (uint8_t)n;
            // marching_tets.cpp:142-163: a single triangle (a-b, a-c, a-d), or
            // the quad's two (a-c, a-d, b-d) and (a-c, b-d, b-c).
            if (tris_of_code(code) == 1) {
                const int e[3][2] = {{a, b}, {a, c}, {a, d}};
                t.tri[n++] = make_tri(e);
            } else if (tris_of_code(code) == 2) {
                const int e0[3][2] = {{a, c}, {a, d}, {b, d}};
                const int e1[3][2] = {{a, c}, {b, d}, {b, c}};
                t.tri[n++] = make_tri(e0);
                t.tri[n++] = make_tri(e1);
            }
        }
    }
    return t;
}
__constant__ TetTables c_tet_tables = make_tet_tables();
static_assert(make_tet_tables().kinds[0] == 0 && make_tet_tables().kinds[255] == 0, "no crossing");
static_assert(make_tet_tables().kinds[1] == 0x555, "corner 0 alone: one triangle in every tetrahedron");
static_assert(make_tet_tables().first[5][15] == 6 * kTetTris, "every triangle has its place");

// The block's 9^3 corner samples; colours only when the caller wants them.
template <bool COL>
struct Halo {
    float val[kHaloCells];
    float col[COL ? 3 : 1][COL ? kHaloCells : 1];
    uint32_t row[kHaloRows];  // bit x: cell x is valid; bit 16 + x: valid and below iso
};

// The eight cubes of row (ly, lz): bit x set where every corner of cube x is
// valid and some but not all of them lie below iso.
template <bool COL>
__device__ __forceinline__ unsigned crossing_cubes(const Halo<COL>& h, int row) {
    const int r0 = (row >> 3) * kHalo + (row & 7);
    const uint32_t a = h.row[r0], b = h.row[r0 + 1], c = h.row[r0 + kHalo], d = h.row[r0 + kHalo + 1];
    const uint32_t all = a & b & c & d, any = a | b | c | d;
    const uint32_t both = all & (all >> 1), some = any | (any >> 1);
    return (both & (some >> 16) & ~(both >> 16)) & 0xFFu;
}

// The corners of a cube that lie below iso (bit c: corner c).
template <bool COL>
__device__ __forceinline__ unsigned below_iso(const Halo<COL>& h, int cube) {
    const int r0 = (cube >> 6) * kHalo + ((cube >> 3) & 7), x = 16 + (cube & 7);
    return ((h.row[r0] >> x) & 3u) | ((h.row[r0 + 1] >> x) & 3u) << 2 | ((h.row[r0 + kHalo] >> x) & 3u) << 4 |
           ((h.row[r0 + kHalo + 1] >> x) & 3u) << 6;
}

struct Cube {
    float lo[3], hi[3];  // voxel centres of corner 0 and corner 7 (marching_tets.cpp:126-128)
    int h0;              // halo index of corner 0
};

struct Vert {
    float p[3];
    float c[3];
};

// marching_tets.cpp:59-80: position-ordered interpolation between two corners,
// given by their halo indices and offset bits (first corner: bits 0-2).
template <bool COL>
__device__ __forceinline__ Vert interp(const Halo<COL>& h, const Cube& q, float iso, int h0, int h1, unsigned bits) {
    const float v0 = h.val[h0], v1 = h.val[h1];
    const float den = __fsub_rn(v1, v0);
    const float t = fabsf(den) < 1e-12f ? 0.5f : __fdiv_rn(__fsub_rn(iso, v0), den);
    const float tc = fminf(fmaxf(t, 0.0f), 1.0f);
    Vert o;
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        const float p0 = (bits >> k) & 1u ? q.hi[k] : q.lo[k], p1 = (bits >> (3 + k)) & 1u ? q.hi[k] : q.lo[k];
        o.p[k] = __fadd_rn(p0, __fmul_rn(tc, __fsub_rn(p1, p0)));
    }
    if constexpr (COL) {
#pragma unroll
        for (int k = 0; k < 3; ++k) {
            const float c0 = h.col[k][h0], c1 = h.col[k][h1];
            o.c[k] = __fadd_rn(c0, __fmul_rn(tc, __fsub_rn(c1, c0)));
        }
    }
    return o;
}

// A warp's 32 triangles in shared memory, as they go to the output: 96
// vertices of six floats (and 96 colours of three bytes), shifted by the
// output's offset inside its 16-byte (4-byte) group so that the copy-out is
// aligned on both sides.
constexpr int kStageFloats = 32 * 18;
constexpr int kStageBytes = 32 * 9;
template <bool COL>
struct VertexStage {
    alignas(16) float f[4 + kStageFloats];
    alignas(4) uint8_t c[COL ? 4 + kStageBytes : 4];
};

// n elements of T staged at s[pad ...] to out, whose first element lies pad
// elements into an aligned group of sizeof(V): whole groups as one V, the
// partial first and last ones by element.
template <typename V, typename T>
__device__ __forceinline__ void copy_out(T* out, const T* s, int pad, int n, int lane) {
    constexpr int kPer = (int)(sizeof(V) / sizeof(T));
    const int head = min(n, (kPer - pad) & (kPer - 1));  // elements before the first whole group
    const int groups = (n - head) / kPer, tail = n - head - groups * kPer;
    const V* from = reinterpret_cast<const V*>(s + pad + head);
    V* to = reinterpret_cast<V*>(out + head);
#pragma unroll 5
    for (int g = lane; g < groups; g += 32) __stcs(to + g, from[g]);
    if (lane < head) out[lane] = s[pad + lane];
    if (lane < tail) out[n - tail + lane] = s[pad + n - tail + lane];
}

template <bool COL>
__device__ __forceinline__ void stage_triangle(const Vert& a, const Vert& b, const Vert& c, float* f, uint8_t* col) {
    // marching_tets.cpp:206-218: face normal of the emitted triangle.
    const float e1[3] = {__fsub_rn(b.p[0], a.p[0]), __fsub_rn(b.p[1], a.p[1]), __fsub_rn(b.p[2], a.p[2])};
    const float e2[3] = {__fsub_rn(c.p[0], a.p[0]), __fsub_rn(c.p[1], a.p[1]), __fsub_rn(c.p[2], a.p[2])};
    float nx = __fsub_rn(__fmul_rn(e1[1], e2[2]), __fmul_rn(e1[2], e2[1]));
    float ny = __fsub_rn(__fmul_rn(e1[2], e2[0]), __fmul_rn(e1[0], e2[2]));
    float nz = __fsub_rn(__fmul_rn(e1[0], e2[1]), __fmul_rn(e1[1], e2[0]));
    const float len =
        __fsqrt_rn(__fadd_rn(__fadd_rn(__fmul_rn(nx, nx), __fmul_rn(ny, ny)), __fmul_rn(nz, nz)));
    if (len > 1e-20f) {
        nx = __fdiv_rn(nx, len);
        ny = __fdiv_rn(ny, len);
        nz = __fdiv_rn(nz, len);
    }
    const Vert* vs[3] = {&a, &b, &c};
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        float* dst = f + 6 * k;
        dst[0] = vs[k]->p[0];
        dst[1] = vs[k]->p[1];
        dst[2] = vs[k]->p[2];
        dst[3] = nx;
        dst[4] = ny;
        dst[5] = nz;
        if constexpr (COL) {
#pragma unroll
            for (int j = 0; j < 3; ++j) col[3 * k + j] = (uint8_t)fminf(fmaxf(vs[k]->c[j], 0.0f), 255.0f);
        }
    }
}

// Triangles listed at a time (a few hundred are usual; an unusually dense
// block takes several passes): room for 32 cubes of 6 tetrahedra x 2.
constexpr int kListItems = 1024;
static_assert(kListItems >= 32 * 12, "32 cubes fit the list");

__device__ __forceinline__ int tri_count(unsigned kinds) { return __popc(kinds & 0x555u) + 2 * __popc(kinds & 0xAAAu); }

// List the triangles of cubes[from ...] in output order (cube, tetrahedron,
// triangle), 32 cubes at a time while the list has room, by one warp. Returns
// the first cube left; listed: the triangles listed. An item is cube |
// triangle in the table << 9.
template <bool COL>
__device__ __forceinline__ int list_triangles(const Halo<COL>& h, const TetTables& tab, const uint16_t* cubes, int from,
                                              int n_cubes, uint16_t* items, int& listed, int lane) {
    int n = 0, c0 = from;
    for (; c0 < n_cubes; c0 += 32) {
        const int cube = c0 + lane < n_cubes ? cubes[c0 + lane] : -1;
        const unsigned bl = cube >= 0 ? below_iso(h, cube) : 0u;
        const unsigned kinds = tab.kinds[bl];
        const int tris = tri_count(kinds);
        int upto = tris;
        for (int o = 1; o < 32; o <<= 1) {
            const int y = __shfl_up_sync(0xffffffffu, upto, o);
            if (lane >= o) upto += y;
        }
        const int here = __shfl_sync(0xffffffffu, upto, 31);
        if (n + here > kListItems) break;  // warp-uniform
        int pos = n + upto - tris;
#pragma unroll
        for (int k = 0; k < 6; ++k) {
            const unsigned kind = (kinds >> (2 * k)) & 3u;
            if (kind == 0u) continue;
            const unsigned code = ((bl >> tet_corner(k, 0)) & 1u) | ((bl >> tet_corner(k, 1)) & 1u) << 1 |
                                  ((bl >> tet_corner(k, 2)) & 1u) << 2 | ((bl >> tet_corner(k, 3)) & 1u) << 3;
            const unsigned item = (unsigned)cube | (unsigned)tab.first[k][code] << 9;
            items[pos++] = (uint16_t)item;
            if (kind == 2u) items[pos++] = (uint16_t)(item + (1u << 9));
        }
        n += here;
    }
    listed = n;
    return min(c0, n_cubes);
}

// Resident CTAs per SM the registers are sized for: 10 (48 registers; 90 us on
// the room mesh, 99 at 11 and 100 at 12, which spill); with colours 7.
#ifndef OSN_EXTRACT_MIN_BLOCKS
#define OSN_EXTRACT_MIN_BLOCKS 10
#endif
#ifndef OSN_EXTRACT_COL_MIN_BLOCKS
#define OSN_EXTRACT_COL_MIN_BLOCKS 7
#endif
// Blocks: pool indices 0 .. *count - 1, or the *count entries of a list.
template <int S, bool COL>
__global__ void __launch_bounds__(kExtractThreads, COL ? OSN_EXTRACT_COL_MIN_BLOCKS : OSN_EXTRACT_MIN_BLOCKS)
extract_kernel(DevVolume v, const int32_t* list, const int32_t* count, float min_w, float iso, float* out_posnor,
               uint8_t* out_rgb, int32_t cap, int32_t* ctl) {
    __shared__ Halo<COL> h;
    __shared__ TetTables s_tab;
    __shared__ uint16_t s_items[kListItems];
    __shared__ uint16_t s_cubes[kBlockVoxels];  // the block's cubes with a sign change, ascending
    __shared__ VertexStage<COL> s_stage[kExtractWarps];
    __shared__ uint16_t s_cell[kHaloRows];  // first voxel of a halo row in its block | neighbour << 9
    __shared__ int s_nb[8];
    __shared__ int s_base, s_tris, s_next;
    __shared__ int s_cube_count, s_listed, s_upto;  // cubes, triangles listed, cubes they cover

    const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
    for (int k = t; k < (int)(sizeof(TetTables) / 4); k += kExtractThreads)
        reinterpret_cast<uint32_t*>(&s_tab)[k] = reinterpret_cast<const uint32_t*>(&c_tet_tables)[k];
    if (t < kHaloRows) {
        const int hy = t % kHalo, hz = t / kHalo;
        s_cell[t] = (uint16_t)(((hz & 7) * kBlockDim + (hy & 7)) * kBlockDim | (hy >> 3) << 10 | (hz >> 3) << 11);
    }
    const int32_t n_blocks = min(*count, v.pool_capacity);
    const int row3 = lane / kHalo, hx = lane - row3 * kHalo;  // this lane's place among three halo rows
    // The warp that lists: not the same one in every CTA, whose warps of one
    // number share a scheduler.
    const int lister = blockIdx.x % kExtractWarps;

    for (int32_t at = blockIdx.x; at < n_blocks;) {
        const int b = list ? list[at] : at;  // the block's pool index
        const BlockCoord bc = v.block_coord[b];
        int next = 0;
        if (t < 8) {
            const int nx = bc.x + (t & 1), ny = bc.y + ((t >> 1) & 1), nz = bc.z + ((t >> 2) & 1);
            s_nb[t] = t == 0 ? b : find_block(v, nx, ny, nz, pack_key(nx, ny, nz));
        } else if (t == 32) {
            next = (int)gridDim.x + atomicAdd(&ctl[2], 1);  // blocks differ in work: dealt out one by one
        }
        __syncthreads();  // also: every warp is done with the previous block

        // Stage the halo: corner samples of this block plus the +x/+y/+z faces,
        // edges and corner of its neighbours (volume.cpp:306-329 per sample).
#pragma unroll
        for (int i = 0; i < (kHaloRows / 3 + kExtractWarps - 1) / kExtractWarps; ++i) {
            const int r = 3 * (warp + i * kExtractWarps);
            if (r >= kHaloRows) break;  // warp-uniform
            const int row = r + row3;
            bool valid = false, below = false;
            if (row3 < 3) {
                const int cell = s_cell[row];
                const int nb = s_nb[(cell >> 9) | (hx >> 3)];
                float val = 0.0f;
                if (nb >= 0) {
                    const size_t idx = (size_t)nb * kBlockVoxels + (size_t)((cell & 511) | (hx & 7));
                    // Weight and stored TSDF loaded together (one round trip).
                    const float w = weight_at<S>(v, idx);
                    const float m = mean_from<S>(v, idx, w);
                    valid = !(w < min_w || w <= 0.0f);
                    below = valid && m < iso;
                    if (valid) {
                        val = m;
                        if constexpr (COL) {
                            const int k = row * kHalo + hx;
                            if constexpr (S == kStoreF32) {
                                const float inv = __fdiv_rn(1.0f, w);
                                h.col[0][k] = __fmul_rn(v.r[idx], inv);
                                h.col[1][k] = __fmul_rn(v.g[idx], inv);
                                h.col[2][k] = __fmul_rn(v.b[idx], inv);
                            } else {
                                // No colour arrays: every contribution is grey.
                                h.col[0][k] = 128.0f;
                                h.col[1][k] = 128.0f;
                                h.col[2][k] = 128.0f;
                            }
                        }
                    }
                }
                h.val[row * kHalo + hx] = val;
            }
            const unsigned vb = __ballot_sync(0xffffffffu, valid), bb = __ballot_sync(0xffffffffu, below);
            if (lane < 3)
                h.row[r + lane] = ((vb >> (kHalo * lane)) & 0x1FFu) | ((bb >> (kHalo * lane)) & 0x1FFu) << 16;
        }
        if (t == 32) s_next = next;
        __syncthreads();

        // The list, by one warp: cubes with a sign change in ascending order
        // (two rows of cubes per lane), then their triangles.
        if (warp == lister) {
            const unsigned m0 = crossing_cubes(h, 2 * lane), m1 = crossing_cubes(h, 2 * lane + 1);
            unsigned cubes = m0 | m1 << 8;
            int incl = __popc(cubes);
            const int own = incl;
            for (int o = 1; o < 32; o <<= 1) {
                const int y = __shfl_up_sync(0xffffffffu, incl, o);
                if (lane >= o) incl += y;
            }
            const int n_cubes = __shfl_sync(0xffffffffu, incl, 31);
            for (int pos = incl - own; cubes != 0u; cubes &= cubes - 1u, ++pos)
                s_cubes[pos] = (uint16_t)(16 * lane + __ffs(cubes) - 1);
            __syncwarp();
            int n_tris = 0;
            for (int c0 = 0; c0 < n_cubes; c0 += 32) {
                const unsigned kinds = c0 + lane < n_cubes ? s_tab.kinds[below_iso(h, s_cubes[c0 + lane])] : 0u;
                n_tris += __reduce_add_sync(0xffffffffu, tri_count(kinds));
            }
            int base = 0;
            if (lane == 0 && n_tris > 0) base = atomicAdd(&ctl[0], 3 * n_tris);
            int listed;
            const int upto = list_triangles(h, s_tab, s_cubes, 0, n_cubes, s_items, listed, lane);
            if (lane == 0) {
                if ((int64_t)base + 3 * n_tris > (int64_t)cap) {
                    atomicExch(&ctl[1], 1);
                    base = -1;
                }
                s_base = base;
                s_tris = n_tris;
                s_cube_count = n_cubes;
                s_listed = listed;
                s_upto = upto;
            }
        }
        __syncthreads();
        at = s_next;
        const int base = s_base;
        if (s_tris == 0 || base < 0) continue;  // uniform: nothing here, or the block's vertices do not fit

        for (int from = 0;;) {  // one pass, unless the block's list is longer than the stage
            const int listed = s_listed, cubes_done = s_upto;
            // One thread per triangle, 32 consecutive ones per warp.
            VertexStage<COL>& stage = s_stage[warp];
            for (int j0 = 32 * warp; j0 < listed; j0 += kExtractThreads) {
                float* const out = out_posnor + ((int64_t)base + 3 * (from + j0)) * 6;
                uint8_t* const out_c = COL ? out_rgb + ((int64_t)base + 3 * (from + j0)) * 3 : nullptr;
                // The caller's buffers are aligned to their elements only.
                const int pad = (int)((reinterpret_cast<uintptr_t>(out) >> 2) & 3);
                const int pad_c = (int)(reinterpret_cast<uintptr_t>(out_c) & 3);
                if (j0 + lane < listed) {
                    const int item = s_items[j0 + lane];
                    const int cube = item & (kBlockVoxels - 1);
                    const uint4 tri = s_tab.tri[item >> 9];
                    const int cc[3] = {cube & 7, (cube >> 3) & 7, cube >> 6};
                    const int bo[3] = {bc.x, bc.y, bc.z};
                    Cube q;
#pragma unroll
                    for (int a = 0; a < 3; ++a) {
                        const int vox = bo[a] * kBlockDim + cc[a];
                        q.lo[a] = __fmul_rn(__fadd_rn((float)vox, 0.5f), v.voxel_size);
                        q.hi[a] = __fmul_rn(__fadd_rn((float)(vox + 1), 0.5f), v.voxel_size);
                    }
                    q.h0 = (cc[2] * kHalo + cc[1]) * kHalo + cc[0];
                    const Vert v0 = interp(h, q, iso, q.h0 + (int)(tri.x & 255u), q.h0 + (int)((tri.x >> 8) & 255u), tri.z);
                    const Vert v1 = interp(h, q, iso, q.h0 + (int)((tri.x >> 16) & 255u), q.h0 + (int)(tri.x >> 24), tri.z >> 6);
                    const Vert v2 = interp(h, q, iso, q.h0 + (int)(tri.y & 255u), q.h0 + (int)(tri.y >> 8), tri.z >> 12);
                    stage_triangle<COL>(v0, v1, v2, stage.f + pad + 18 * lane, stage.c + pad_c + 9 * lane);
                }
                __syncwarp();
                const int n = min(32, listed - j0);
                copy_out<float4>(out, stage.f, pad, 18 * n, lane);
                if constexpr (COL) copy_out<uint32_t>(out_c, stage.c, pad_c, 9 * n, lane);
                __syncwarp();  // the stage is rewritten
            }
            if (cubes_done >= s_cube_count) break;  // uniform
            __syncthreads();
            from += listed;
            if (warp == lister) {
                int n;
                const int upto = list_triangles(h, s_tab, s_cubes, cubes_done, s_cube_count, s_items, n, lane);
                if (lane == 0) {
                    s_listed = n;
                    s_upto = upto;
                }
            }
            __syncthreads();
        }
    }
}

__global__ void reset_table_kernel(HashEntry* table, uint32_t count, long long key) {
    for (uint32_t k = blockIdx.x * blockDim.x + threadIdx.x; k < count; k += gridDim.x * blockDim.x) {
        table[k].key = key;
        table[k].block_idx = -1;
        table[k].pad = 0;
    }
}

// Every occupied slot of the table (slot-index layout: the slot is the
// block's pool index), appended warp by warp.
__global__ void list_blocks_kernel(const HashEntry* table, uint32_t size, int32_t* out, int32_t* count) {
    for (uint32_t base = blockIdx.x * blockDim.x; base < size; base += gridDim.x * blockDim.x) {
        const uint32_t k = base + threadIdx.x;
        bool occ = false;
        if (k < size) {
            const int4 raw = reinterpret_cast<const int4*>(table)[k];
            const long long key = ((long long)(unsigned)raw.y << 32) | (unsigned)raw.x;
            occ = key >= 0 && raw.z == (int)k;
        }
        const unsigned m = __ballot_sync(0xffffffffu, occ);
        int at = 0;
        if ((threadIdx.x & 31) == 0 && m) at = atomicAdd(count, __popc(m));
        at = __shfl_sync(0xffffffffu, at, 0);
        if (occ) out[at + __popc(m & lanemask_lt())] = (int32_t)k;
    }
}

// Zero one 512-voxel block's span of an array of ELEM-byte voxels, by the
// whole CTA in 16-byte stores.
template <int ELEM>
__device__ __forceinline__ void zero_block(void* arr, int32_t b) {
    constexpr int kVec = kBlockVoxels * ELEM / 16;
    float4* p = reinterpret_cast<float4*>(arr) + (size_t)b * kVec;
    for (int k = threadIdx.x; k < kVec; k += blockDim.x) p[k] = make_float4(0.f, 0.f, 0.f, 0.f);
}

// Reset: the allocated blocks' voxels to zero (pool indices 0..*count-1, or
// the *count entries of a list), then the table's slots to empty. The count
// is read on the device, so the host need not wait for it first. Bound by
// the stores: 16 bytes per slot and 20 (FP32) per voxel of the blocks.
template <int S>
__global__ void __launch_bounds__(kResetThreads) reset_kernel(DevVolume v, const int32_t* list, const int32_t* count) {
    const int32_t n = min(*count, v.pool_capacity);
    for (int32_t i = blockIdx.x; i < n; i += gridDim.x) {
        const int32_t b = list ? list[i] : i;
        zero_block<tsdf_bytes(S)>(v.tsdf, b);
        zero_block<weight_bytes(S)>(v.weight, b);
        if constexpr (S == kStoreF32) {
            zero_block<4>(v.r, b);
            zero_block<4>(v.g, b);
            zero_block<4>(v.b, b);
        }
    }
    const uint32_t size = v.hash_mask + 1;
    for (uint32_t k = blockIdx.x * blockDim.x + threadIdx.x; k < size; k += gridDim.x * blockDim.x)
        reinterpret_cast<int4*>(v.table)[k] = make_int4(-1, -1, -1, 0);  // kEmptyKey, no index
}
static_assert(kEmptyKey == -1, "an empty slot's key is all ones");

}  // namespace

template <int S, bool COL>
static cudaError_t launch_extract_as(const DevVolume& v, const int32_t* list, const int32_t* count, float min_w,
                                     float iso, float* posnor, uint8_t* rgb, int32_t cap, int32_t* ctl, int sm_count,
                                     cudaStream_t s) {
    static int per_sm = 0;
    static std::once_flag once;
    std::call_once(once, [] {
        if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, extract_kernel<S, COL>, kExtractThreads, 0) !=
                cudaSuccess ||
            per_sm < 1)
            per_sm = 1;
    });
    return launch_now(extract_kernel<S, COL>, per_sm * sm_count, kExtractThreads, s, v, list, count, min_w, iso, posnor,
                      rgb, cap, ctl);
}

cudaError_t launch_extract(const DevVolume& v, const int32_t* list, const int32_t* count, float min_w, float iso,
                           float* posnor, uint8_t* rgb, int32_t cap, int32_t* ctl, int sm_count, cudaStream_t s) {
    // Colours in a separate instance: without them the halo holds a quarter
    // of the shared memory and the kernel fewer registers.
    const bool col = rgb != nullptr;
    switch (v.storage) {
        case kStoreF16U16:
            return col ? launch_extract_as<kStoreF16U16, true>(v, list, count, min_w, iso, posnor, rgb, cap, ctl, sm_count, s)
                       : launch_extract_as<kStoreF16U16, false>(v, list, count, min_w, iso, posnor, nullptr, cap, ctl, sm_count, s);
        case kStoreF64:
            return col ? launch_extract_as<kStoreF64, true>(v, list, count, min_w, iso, posnor, rgb, cap, ctl, sm_count, s)
                       : launch_extract_as<kStoreF64, false>(v, list, count, min_w, iso, posnor, nullptr, cap, ctl, sm_count, s);
        default:
            return col ? launch_extract_as<kStoreF32, true>(v, list, count, min_w, iso, posnor, rgb, cap, ctl, sm_count, s)
                       : launch_extract_as<kStoreF32, false>(v, list, count, min_w, iso, posnor, nullptr, cap, ctl, sm_count, s);
    }
}

cudaError_t launch_reset_table(HashEntry* first, uint32_t count, long long key, cudaStream_t s) {
    if (count == 0) return cudaSuccess;
    const int grid = (int)std::min<uint32_t>((count + 255) / 256, 148u * 16u);
    return launch_now(reset_table_kernel, grid, 256, s, first, count, key);
}

cudaError_t launch_list_blocks(const DevVolume& v, int32_t* out, int32_t* count, cudaStream_t s) {
    const uint32_t size = v.hash_mask + 1;
    const int grid = (int)std::min<uint32_t>((size + 255) / 256, 148u * 8u);
    return launch_now(list_blocks_kernel, grid, 256, s, v.table, size, out, count);
}

cudaError_t launch_reset(const DevVolume& v, const int32_t* list, const int32_t* count, cudaStream_t s) {
    // One wave of 16 CTAs per SM, striding over the blocks and the slots.
    const int grid = 148 * 16;
    switch (v.storage) {
        case kStoreF16U16: return launch_now(reset_kernel<kStoreF16U16>, grid, kResetThreads, s, v, list, count);
        case kStoreF64: return launch_now(reset_kernel<kStoreF64>, grid, kResetThreads, s, v, list, count);
        default: return launch_now(reset_kernel<kStoreF32>, grid, kResetThreads, s, v, list, count);
    }
}

}  // namespace osn_b200
