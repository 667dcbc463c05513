// The passes behind every change of a world's words, in two launches:
//   brick_pass_kernel  changes the words (removeSphere, placeVoxel, an upload from device
//                      memory, the reference's level, or nothing), and rebuilds the brick masks of the box in the same
//                      pass, with the region and super masks' bits, the solid bounding box
//                      and the depth-field flag;
//   node_pass_kernel   everything that follows from them, as independent tiles of one launch:
//                      the directed brick distances, the region distances and the depth
//                      field (fixDepthField, render.cpp:226-253).
//
// The node pass is bit-parallel: a row of 32 nodes along x is one 32-bit word.  The masks
// already hold a bit per voxel (brick masks) and per brick (region masks), 4 bits of a row in
// each 64-bit mask, so a tile of rows with its halo is put together in shared memory from the
// few KB of masks that it spans, and the neighbourhood work of 32 nodes is done by one
// instruction.
//
// Both are latency chains for an edit (a few dozen CTAs): removeSphere(8) in the 512 x 256 x 512
// world, edits in a row, host included, takes 9.4 us, where ten launches of a few microseconds
// each took 88 us.
#include <cuda_runtime.h>

#include <algorithm>
#include <climits>
#include <cmath>
#include <cstring>
#include <utility>

#include "vrt_internal.h"

namespace vrt {

struct BrickPass {
    int32_t* words;
    int32_t* words_z;            // the z-major copy, or NULL: it follows later (see change_words)
    const int32_t* src;          // kCopyWords: words [first, first + count) come from here
    uint64_t first, count;
    uint64_t* bricks;
    uint64_t* regions;
    uint64_t* supers;            // may be NULL (stop masks)
    int* boxes;                  // one record per CTA: solid box (min x,y,z, max x,y,z), depth flag, 0
    Layout L;
    int bx0, by0, bz0, bx1;      // the bricks' box (its ends in y and z follow from ny and tasks)
    int g0;                      // first group of 8 bricks along x
    unsigned ng, ny, tasks;      // groups along x, bricks along y, groups in all
    int x, y, z, r;              // kRemoveSphere: centre and radius; kPlaceVoxel: the voxel
    int32_t word;                // kPlaceVoxel
};

constexpr int kFixLevels = 36;

struct FixPass {
    int32_t* words;
    int32_t* words_z;            // as in BrickPass
    const uint64_t* bricks;
    Layout L;
    int x0, y0, z0, x1, y1, z1;  // the voxels to refresh, within the world
    int cx, cy, cz, r2;          // r2 > 0: of those, the ones inside this sphere
    int small;                   // tiles of 8 x 8 rows instead of 16 x 16
    int tx0, ty0, tz0, ntx, nty; // the tiles that cover the box
    int32_t word[kFixLevels + 1];
};

struct NodePass {
    const uint64_t* regions;
    uint16_t* bdir;              // directed distances, the two x directions of an octant pair to a value
    const uint64_t* supers;
    uint8_t* rdist;
    int* aabb;                   // solid box, then the depth-field flag
    const int* boxes;
    Layout L;
    int n_fix, n_dir, n_reg, n_boxes;            // tiles of each kind; records to merge
    int dx0, dy0, dz0, ndx, ndy;                 // distance tiles of 32 x 8 x 8 bricks
    int rx0, ry0, rz0, nrx, nry;                 // and of 32 x 8 x 8 regions
    int reset_box, reset_flag;
    FixPass fix;
};

// ------------------------------------------------------------------ depth field
//
// fixDepthField gives an air voxel the largest d over the solid voxels within radius 7,
// where an offset's d is -sqrt(s), s = the sum over the axes of max(|o| - 1, 0)^2, and
// only offsets with d > -6 (s < 36) count (computeDepthIndices, render.cpp:66-100: the
// running value starts at -6, and a d above -2 becomes 0, which is not written).  So the
// word depends on the smallest s alone: s < 4 leaves the word as it is, 4..35 writes
// -sqrt(s), no solid neighbour writes -6.
//
// The offsets are taken row by row: for the row (dy, dz) away, an offset |x| <= k adds up
// to at most c + max(k - 1, 0)^2 with c the share of dy and dz, and |x| may go up to
// sqrt(49 - dy^2 - dz^2).  With D_k(row) = the bits within k of a solid bit of that row, the
// voxels whose smallest s is at most S are the OR of D_k over the rows and their k at level
// S.  Going up the levels, each (row, k) pair is ORed in once: about 600 ORs for 32 voxels,
// where testing the 1413 offsets voxel by voxel took 45,000 loads.

constexpr int kFixX = 32;                          // voxels per tile along x: one row word
constexpr int kFixHalo = 7;                        // DEPTH_FIELD_RADIUS, render.hpp:7
constexpr int kFixK = 6;                           // D_1 .. D_6 (|x| = 7 alone gives s = 36)

// A tile of SIDE x SIDE rows by 256 threads: one thread per row of 16 x 16, or four per row of
// 8 x 8, which take a fourth of the levels each.  The large tile reads the least halo per voxel.
// The small one is for an edit's few tiles, whose time is one tile's chain: some 600 reads of
// shared memory by each of 8 warps at 16 x 16, 150 at 8 x 8.
template <int SIDE>
struct FixTile {
    static constexpr int kShift = SIDE == 16 ? 4 : 3;
    static constexpr int kRows = SIDE + 2 * kFixHalo;  // rows per axis with the halo
    // Row pitch of a D_k plane: a warp's lanes are SIDE rows in y of 32 / SIDE z, so a pitch of SIDE
    // modulo 32 puts them into 32 different banks.
    static constexpr int kPitch = SIDE + 32, kPlane = kRows * kPitch;
    static constexpr int kSpan = SIDE / 4 + 4;         // bricks spanned in y and z; 8 + 2 x 2 in x
    static constexpr int kNodes = 12 * kSpan * kSpan;
    static constexpr int kParts = 256 / (SIDE * SIDE);  // threads of a row
    struct Smem {
        uint64_t nodes[kNodes];
        uint32_t d[kFixK * kPlane];
        uint32_t out[7][SIDE * SIDE];              // per row: the 6 bits of s, and the voxels to write
        uint32_t part[kParts > 1 ? kParts - 1 : 1][7][kParts > 1 ? SIDE * SIDE : 1];  // the other threads' bits and found
        int32_t word[kFixLevels + 1];              // the depth-field word of each s; [36]: no solid neighbour
    };
};

// Offsets (into Smem::d, from a row's own place in D_1) of the planes that level S adds.
// Level 3 stands for every s <= 3, whose voxels all keep their word.
struct FixLevel {
    int n = 0;
    int off[160] = {};
};
template <class T>
constexpr FixLevel fix_level(int S) {
    FixLevel r;
    for (int dz = -7; dz <= 7; dz++)
        for (int dy = -7; dy <= 7; dy++) {
            const int rr = 49 - dy * dy - dz * dz;
            if (rr < 0) continue;
            const int ay = (dy < 0 ? -dy : dy) - 1, az = (dz < 0 ? -dz : dz) - 1;
            const int c = (ay > 0 ? ay * ay : 0) + (az > 0 ? az * az : 0);
            int best = 0;
            for (int k = 1; k <= kFixK; k++) {
                if (k * k > rr) break;
                const int s = c + (k - 1) * (k - 1);
                if (S == 3 ? s <= 3 : s == S) best = k;
            }
            if (best) r.off[r.n++] = (best - 1) * T::kPlane + dz * T::kPitch + dy;
        }
    return r;
}

template <class T, int S>
struct FixTable {
    static constexpr FixLevel L = fix_level<T>(S);
};

// The first level of a row's part g of n: parts of about as many reads each.
constexpr int fix_part(int g, int n) {
    int total = 0, sum = 0, S = 3;
    for (int i = 3; i < kFixLevels; i++) total += fix_level<FixTile<16>>(i).n;
    while (S < kFixLevels && sum * n < total * g) sum += fix_level<FixTile<16>>(S++).n;
    return S;
}
constexpr int kFixPart1 = fix_part(1, 4), kFixPart2 = fix_part(2, 4), kFixPart3 = fix_part(3, 4);

template <class T, int S, int... I>
__device__ __forceinline__ uint32_t fix_or(const uint32_t* d, std::integer_sequence<int, I...>) {
    uint32_t f = 0;
    ((f |= d[std::integral_constant<int, FixTable<T, S>::L.off[I]>::value]), ...);
    return f;
}

// Add level S (and the levels after it) to a row: found = voxels whose smallest s is known.
// Now and then the warp looks whether every air voxel of its rows has been found.
template <class T, int S, int END>
__device__ __forceinline__ void fix_levels(const uint32_t* d, uint32_t air, uint32_t& found, uint32_t (&bit)[6]) {
    if constexpr (S < END) {
        if constexpr (S == 5 || S == 10 || S == 17 || S == 26)
            if (!__any_sync(0xffffffffu, (air & ~found) != 0)) return;
        if constexpr (FixTable<T, S>::L.n > 0) {
            const uint32_t now = fix_or<T, S>(d, std::make_integer_sequence<int, FixTable<T, S>::L.n>{}) & ~found;
            found |= now;
            if (S & 1) bit[0] |= now;
            if (S & 2) bit[1] |= now;
            if (S & 4) bit[2] |= now;
            if (S & 8) bit[3] |= now;
            if (S & 16) bit[4] |= now;
            if (S & 32) bit[5] |= now;
        }
        fix_levels<T, S + 1, END>(d, air, found, bit);
    }
}

// One 32 x SIDE x SIDE tile.  Only the air voxels of P.box (and of
// the sphere, if there is one) are written; only solidity is read, which no thread changes.
template <int SIDE>
__device__ void fix_tile(const FixPass& P, int tile, typename FixTile<SIDE>::Smem& s) {
    using T = FixTile<SIDE>;
    const Layout& L = P.L;
    const int tx = tile % P.ntx, ty = (tile / P.ntx) % P.nty, tz = tile / (P.ntx * P.nty);
    const int x0 = (P.tx0 + tx) * kFixX, y0 = (P.ty0 + ty) * SIDE, z0 = (P.tz0 + tz) * SIDE;
    const int t = threadIdx.x, row = t & (SIDE * SIDE - 1);
    const int part = T::kParts == 1 ? 0 : t >> 2 * T::kShift;  // the same for a warp's lanes

    // the bricks the tile and its halo span; bricks beyond the grid hold no solid voxel
    const int bx0 = x0 / 4 - 2, by0 = y0 / 4 - 2, bz0 = z0 / 4 - 2;
    bool solid = false;
    for (int i = t; i < T::kNodes; i += 256) {
        const int bx = bx0 + i % 12, by = by0 + (i / 12) % T::kSpan, bz = bz0 + i / (12 * T::kSpan);
        uint64_t m = 0;
        if (bx >= 0 && by >= 0 && bz >= 0 && bx < L.BWp && by < L.BHp && bz < L.BWp)
            m = P.bricks[brick_index(L, bx, by, bz)];
        s.nodes[i] = m;
        solid |= m != 0;
    }
    if (t <= kFixLevels) s.word[t] = P.word[t];
    const bool any_solid = __syncthreads_or(solid);

    // this thread's own row, and the voxels of it that may be written
    const int ly = row & (SIDE - 1), lz = row >> T::kShift, y = y0 + ly, z = z0 + lz;
    const uint32_t* n32 = reinterpret_cast<const uint32_t*>(s.nodes);
    uint32_t air = 0;
    if (y >= P.y0 && y < P.y1 && z >= P.z0 && z < P.z1) {
        const int node = ((y >> 2) - by0) * 12 + ((z >> 2) - bz0) * 12 * T::kSpan;
        uint32_t own = 0;
        for (int i = 0; i < 8; i++)
            own |= (n32[2 * (node + 2 + i) + ((z & 3) >> 1)] >> (4 * (y & 3) + 16 * (z & 1)) & 15) << (4 * i);
        const int lo = max(P.x0 - x0, 0), hi = min(P.x1 - x0, 32);  // lo < 32 and hi > 0: the tile meets the box
        air = ~own & (0xffffffffu << lo) & (0xffffffffu >> (32 - hi));
    }
    if (!__syncthreads_or(air != 0)) return;  // nothing to write (solid ground)

    uint32_t found = 0, bit[6] = {0, 0, 0, 0, 0, 0};
    if (any_solid) {
        // D_1 .. D_6 of every row: window bits [8, 40) are the tile's voxels
        for (int i = t; i < T::kRows * T::kRows; i += 256) {
            const int ry = i % T::kRows, rz = i / T::kRows;
            const int py = ry + 1, pz = rz + 1;  // rows start at y0 - 7 = 4 * by0 + 1
            const int node = (py >> 2) * 12 + (pz >> 2) * 12 * T::kSpan, half = (pz & 3) >> 1;
            const int shift = 4 * (py & 3) + 16 * (pz & 1);
            uint64_t w = 0;
#pragma unroll
            for (int j = 0; j < 12; j++)
                w |= (uint64_t)(n32[2 * (node + j) + half] >> shift & 15) << (4 * j);
            uint32_t* d = s.d + rz * T::kPitch + ry;
            uint32_t c = (uint32_t)(w >> 8);
#pragma unroll
            for (int k = 1; k <= kFixK; k++) {
                c |= (uint32_t)(w >> (8 + k)) | (uint32_t)(w >> (8 - k));
                d[(k - 1) * T::kPlane] = c;
            }
        }
        __syncthreads();
        if (__any_sync(0xffffffffu, air != 0)) {
            const uint32_t* d = s.d + (lz + kFixHalo) * T::kPitch + ly + kFixHalo;
            if constexpr (T::kParts == 1) {
                fix_levels<T, 3, kFixLevels>(d, air, found, bit);
            } else {
                switch (part) {
                    case 0: fix_levels<T, 3, kFixPart1>(d, air, found, bit); break;
                    case 1: fix_levels<T, kFixPart1, kFixPart2>(d, air, found, bit); break;
                    case 2: fix_levels<T, kFixPart2, kFixPart3>(d, air, found, bit); break;
                    default: fix_levels<T, kFixPart3, kFixLevels>(d, air, found, bit); break;
                }
            }
        }
    }
    if constexpr (T::kParts > 1) {  // the nearer part's answer counts
        static_assert(T::kParts == 4 || T::kParts == 1);
        if (part) {
#pragma unroll
            for (int k = 0; k < 6; k++) s.part[part - 1][k][row] = bit[k];
            s.part[part - 1][6][row] = found;
        }
        __syncthreads();
        if (part == 0) {
#pragma unroll
            for (int g = 0; g < T::kParts - 1; g++) {
                const uint32_t now = s.part[g][6][row] & ~found;
                found |= now;
#pragma unroll
                for (int k = 0; k < 6; k++) bit[k] |= s.part[g][k][row] & now;
            }
        }
    }
    // s <= 3 was recorded as 3: those voxels keep their word
    const uint32_t keep = found & ~(bit[2] | bit[3] | bit[4] | bit[5]);
    if (part == 0) {
#pragma unroll
        for (int k = 0; k < 6; k++) s.out[k][row] = bit[k];
        s.out[6][row] = air & ~keep;
    }
    __syncthreads();

    // write: four voxels of a row per thread, one 16-byte store where all four change
    const bool vec = (L.W & 3) == 0;
    const int seg = 4 * (t & 7);
    for (int row = t >> 3; row < SIDE * SIDE; row += 32) {
        uint32_t wr = s.out[6][row] >> seg & 15;
        if (!wr) continue;
        const int ry = y0 + (row & (SIDE - 1)), rz = z0 + (row >> T::kShift), rx = x0 + seg;
        uint32_t b[6];
#pragma unroll
        for (int k = 0; k < 6; k++) b[k] = s.out[k][row] >> seg;
        int32_t v[4];
#pragma unroll
        for (int e = 0; e < 4; e++) {
            int sq = 0;
#pragma unroll
            for (int k = 0; k < 6; k++) sq |= (int)(b[k] >> e & 1) << k;
            // every recorded s is at least 3, so 0 says that no solid voxel was found
            v[e] = s.word[sq ? sq : kFixLevels];
            if (P.r2 > 0) {
                const int ox = rx + e - P.cx, oy = ry - P.cy, oz = rz - P.cz;
                if (ox * ox + oy * oy + oz * oz >= P.r2 * P.r2) wr &= ~(1u << e);
            }
        }
        int32_t* q = P.words + ((uint64_t)rx + (uint64_t)L.W * ry + (uint64_t)L.W * L.H * rz);
        if (vec && wr == 15) {
            *reinterpret_cast<int4*>(q) = make_int4(v[0], v[1], v[2], v[3]);
        } else {
#pragma unroll
            for (int e = 0; e < 4; e++)
                if (wr >> e & 1) q[e] = v[e];
        }
        if (P.words_z)
            for (int e = 0; e < 4; e++)
                if (wr >> e & 1) P.words_z[rz + (uint64_t)L.W * ry + (uint64_t)L.W * L.H * (rx + e)] = v[e];
    }
}

// ------------------------------------------------------------------ directed brick distances
//
// D(b) = the largest r <= 15 for which the cube of r^3 bricks from b into the octant is empty.
// With E_r = "that cube is empty" as a bit per brick, E_1 is the complement of the occupancy,
// and for a + c <= 2a the cube of side a + c is the union of the cubes of side a at the eight
// corners {0, c}^3.  So E_2, E_4 and E_8 follow from each other, every other E_r is an AND of
// eight shifted copies of one of them, and D is the number of r with E_r set.  The AND over x
// is one shift of the row word, over y and z it is four rows.  (Three passes, one per axis, of
// up to 16 byte minima per brick and octant took 92 us for the 512 x 96 x 512 level, and
// three more for the regions 19 us; this whole launch takes 19 us, bound by its instructions.)
//
// One tile: 32 x 8 x 8 bricks and the two octants of one y and one z direction.  Rows are held
// as 64-bit windows from 16 bricks before the tile, so no carry between words is needed: a
// window end spoils at most 14 bits, which end before the tile's own.  Smaller tiles in y and
// z would read more halo (14 rows each); four directions to a CTA made an edit's few tiles,
// whose latency is the edit's, twice as long.

constexpr int kDirRows = 22;  // 8 + 14 rows along the octant's y and z
constexpr int kDirNodes = 16 * 6 * 6;

struct alignas(16) DirSmem {
    uint64_t nodes[kDirNodes];  // region masks; later the distance bit planes
    uint64_t e1[kDirRows * kDirRows];
    ulonglong2 e2[21 * 21];  // .x toward +x, .y toward -x; later the output
    ulonglong2 e4[19 * 19];
    ulonglong2 e8[15 * 15];
};

// The 64-bit row window at row (py, pz) of 16 x NY x n masks held in shared memory.
template <int NY>
__device__ __forceinline__ uint64_t row_window(const uint32_t* n32, int py, int pz) {
    const uint32_t* n = n32 + 2 * ((py >> 2) * 16 + (pz >> 2) * 16 * NY) + ((pz & 3) >> 1);
    const int shift = 4 * (py & 3) + 16 * (pz & 1);
    uint64_t w = 0;
#pragma unroll
    for (int j = 0; j < 16; j++) w |= (uint64_t)(n[2 * j] >> shift & 15) << (4 * j);
    return w;
}

__device__ __forceinline__ ulonglong2 and4(const ulonglong2* e, int pitch, int o) {
    const ulonglong2 a = e[0], b = e[o], c = e[o * pitch], d = e[o * pitch + o];
    return make_ulonglong2(a.x & b.x & c.x & d.x, a.y & b.y & c.y & d.y);
}

// E_(a+o) of one row and x direction (word 0: +x, word 1: -x) from E_a of side-a cubes.
template <int PITCH, int O>
__device__ __forceinline__ uint32_t corners(const ulonglong2* e, int word, bool plus) {
    const uint64_t* q = reinterpret_cast<const uint64_t*>(e) + word;
    const uint64_t v = q[0] & q[2 * O] & q[2 * O * PITCH] & q[2 * (O * PITCH + O)];
    return (uint32_t)((v & (plus ? v >> O : v << O)) >> 16);
}

// bit i of x -> bit 0 of byte i, for the low 4 bits
__device__ __forceinline__ uint32_t spread4(uint32_t x) { return (x * 0x00204081u) & 0x01010101u; }

// 4 nodes' values, one per byte, from the bit planes at bit position sh
__device__ __forceinline__ uint32_t plane_bytes(uint4 p, int sh) {
    return spread4(p.x >> sh & 15) | spread4(p.y >> sh & 15) << 1 | spread4(p.z >> sh & 15) << 2 |
           spread4(p.w >> sh & 15) << 3;
}

// r is the value of the nodes in `now`
__device__ __forceinline__ void add_planes(uint4& p, int r, uint32_t now) {
    if (r & 1) p.x |= now;
    if (r & 2) p.y |= now;
    if (r & 4) p.z |= now;
    if (r & 8) p.w |= now;
}

__device__ void dir_tile(const NodePass& P, int tile, DirSmem& s) {
    const Layout& L = P.L;
    const int ys = tile & 1, zs = tile >> 1 & 1;  // 1: toward +
    tile >>= 2;
    const int x0 = (P.dx0 + tile % P.ndx) * 32, y0 = (P.dy0 + tile / P.ndx % P.ndy) * 8;
    const int z0 = (P.dz0 + tile / (P.ndx * P.ndy)) * 8;
    const int t = threadIdx.x;

    // the regions the tile and its halo span; beyond the grid everything is empty
    const int rx0 = x0 / 4 - 4, ry0 = y0 / 4 - (ys ? 0 : 4), rz0 = z0 / 4 - (zs ? 0 : 4);
    for (int i = t; i < kDirNodes; i += 256) {
        const int rx = rx0 + (i & 15), ry = ry0 + (i >> 4) % 6, rz = rz0 + i / 96;
        uint64_t m = 0;
        if (rx >= 0 && ry >= 0 && rz >= 0 && rx < L.RWp && ry < L.RHp && rz < L.RWp)
            m = P.regions[region_index(L, rx, ry, rz)];
        s.nodes[i] = m;
    }
    __syncthreads();
    // E_1: rows (ly, lz) along the octants' directions, 0..7 the tile's own
    const uint32_t* n32 = reinterpret_cast<const uint32_t*>(s.nodes);
    for (int i = t; i < kDirRows * kDirRows; i += 256) {
        const int ly = i % kDirRows, lz = i / kDirRows;
        s.e1[i] = ~row_window<6>(n32, ys ? ly : 23 - ly, zs ? lz : 23 - lz);
    }
    __syncthreads();
    for (int i = t; i < 21 * 21; i += 256) {
        const uint64_t* e = s.e1 + i / 21 * kDirRows + i % 21;
        const uint64_t v = e[0] & e[1] & e[kDirRows] & e[kDirRows + 1];
        s.e2[i] = make_ulonglong2(v & v >> 1, v & v << 1);
    }
    __syncthreads();
    for (int i = t; i < 19 * 19; i += 256) {
        const ulonglong2 v = and4(&s.e2[i % 19 + i / 19 * 21], 21, 2);
        s.e4[i] = make_ulonglong2(v.x & v.x >> 2, v.y & v.y << 2);
    }
    __syncthreads();
    if (t < 15 * 15) {
        const ulonglong2 v = and4(&s.e4[t % 15 + t / 15 * 19], 19, 4);
        s.e8[t] = make_ulonglong2(v.x & v.x >> 4, v.y & v.y << 4);
    }
    __syncthreads();
    // One of the tile's 64 rows, one of the two octants and the lower or upper half of the
    // levels per thread
    uint4* planes = reinterpret_cast<uint4*>(s.nodes);  // [half][x direction][row]
    {
        const int ya = t & 7, za = t >> 3 & 7, xs = t >> 6 & 1, half = t >> 7;
        const int ly = ys ? ya : 7 - ya, lz = zs ? za : 7 - za;
        const ulonglong2* e2 = s.e2 + lz * 21 + ly;
        const ulonglong2* e4 = s.e4 + lz * 19 + ly;
        const ulonglong2* e8 = s.e8 + lz * 15 + ly;
        const int word = xs ? 0 : 1;
        const bool plus = xs != 0;
        uint4 p = make_uint4(0, 0, 0, 0);
        uint32_t cur = 0xffffffffu;
        auto level = [&](int r, uint32_t e) {  // E_r: the nodes that end here have D = r - 1
            add_planes(p, r < 2 ? 0 : r - 2, cur & ~e);
            cur = e;
        };
        if (half == 0) {
            level(1, (uint32_t)(s.e1[lz * kDirRows + ly] >> 16));
            level(2, corners<21, 0>(e2, word, plus));
            level(3, corners<21, 1>(e2, word, plus));
            level(4, corners<19, 0>(e4, word, plus));
            level(5, corners<19, 1>(e4, word, plus));
            level(6, corners<19, 2>(e4, word, plus));
            level(7, corners<19, 3>(e4, word, plus));
            level(8, corners<15, 0>(e8, word, plus));
        } else {
            cur = corners<15, 0>(e8, word, plus);
            level(9, corners<15, 1>(e8, word, plus));
            level(10, corners<15, 2>(e8, word, plus));
            level(11, corners<15, 3>(e8, word, plus));
            level(12, corners<15, 4>(e8, word, plus));
            level(13, corners<15, 5>(e8, word, plus));
            level(14, corners<15, 6>(e8, word, plus));
            level(15, corners<15, 7>(e8, word, plus));
            add_planes(p, kDistCap - 1, cur);
        }
        planes[t] = p;
    }
    __syncthreads();
    // planes -> one byte per octant: 8 bricks of one row per thread, two octants to 16 bits
    uint16_t* out = reinterpret_cast<uint16_t*>(s.e2);  // 64 rows x 32 bricks
    {
        const int row = t >> 2, seg = t & 3;
        const uint4 u0 = planes[row], v0 = planes[128 + row], u1 = planes[64 + row], v1 = planes[192 + row];
        const uint4 p0 = make_uint4(u0.x | v0.x, u0.y | v0.y, u0.z | v0.z, u0.w | v0.w);
        const uint4 p1 = make_uint4(u1.x | v1.x, u1.y | v1.y, u1.z | v1.z, u1.w | v1.w);
#pragma unroll
        for (int g = 0; g < 2; g++) {
            const int sh = 8 * seg + 4 * g;
            const uint32_t a0 = plane_bytes(p0, sh) << 2, a1 = plane_bytes(p1, sh) << 2;
            *reinterpret_cast<uint2*>(out + 32 * row + sh) =
                make_uint2(__byte_perm(a0, a1, 0x5140), __byte_perm(a0, a1, 0x7362));
        }
    }
    __syncthreads();
    const int lane = t & 31;
    if (x0 + lane < L.BWp)
        for (int row = t >> 5; row < 64; row += 8)  // BHp and BWp are multiples of 16: y and z lie in the grid
            P.bdir[4 * brick_index(L, x0 + lane, y0 + (row & 7), z0 + (row >> 3)) + ys + 2 * zs] = out[32 * row + lane];
}

// ------------------------------------------------------------------ region distances
//
// The same for the centred distances of the regions: D(r) = the number of k in [0, 15) for
// which the cube of side 2k + 1 around r is empty, from E_1, E_2, E_4, E_8 and E_16 of cubes
// that start at a node and reach toward +.  One tile: 32 x 8 x 8 regions.

constexpr int kRegNodes = 16 * 10 * 10;

struct alignas(16) RegSmem {
    uint64_t e1[36 * 36];
    union {
        uint64_t nodes[kRegNodes];  // done with when E_1 is
        struct {
            uint64_t e2[35 * 35], e4[33 * 33], e8[29 * 29], e16[21 * 21];
        };
    };
    uint32_t planes[64][4];
};

template <int PITCH, int O>
__device__ __forceinline__ uint64_t cube_from(const uint64_t* e) {
    const uint64_t v = e[0] & e[O] & e[O * PITCH] & e[O * PITCH + O];
    return v & v >> O;
}

// Whether the cube of radius K around the row's nodes is empty; (a, b) the row in the tile.
template <int K>
__device__ __forceinline__ uint32_t centred(const RegSmem& s, int a, int b) {
    const int z = a + 14 - K, y = b + 14 - K;
    uint64_t v;
    if constexpr (K == 0) v = s.e1[y * 36 + z];
    else if constexpr (K < 2) v = cube_from<35, 2 * K + 1 - 2>(s.e2 + y * 35 + z);
    else if constexpr (K < 4) v = cube_from<33, 2 * K + 1 - 4>(s.e4 + y * 33 + z);
    else if constexpr (K < 8) v = cube_from<29, 2 * K + 1 - 8>(s.e8 + y * 29 + z);
    else v = cube_from<21, 2 * K + 1 - 16>(s.e16 + y * 21 + z);
    return (uint32_t)(v >> (16 - K));
}

// The distances K0 .. K0 + 3 of a row
template <int K0>
__device__ __forceinline__ uint4 centred_planes(const RegSmem& s, int a0, int b0) {
    uint4 p = make_uint4(0, 0, 0, 0);
    uint32_t prev = 0xffffffffu;
    if constexpr (K0 > 0) prev = centred<K0 - 1>(s, a0, b0);
    const uint32_t a = centred<K0>(s, a0, b0), b = centred<K0 + 1>(s, a0, b0), c = centred<K0 + 2>(s, a0, b0);
    uint32_t d = 0;  // 15: "15 or more"
    if constexpr (K0 + 3 < kDistCap) d = centred<K0 + 3>(s, a0, b0);
    add_planes(p, K0, prev & ~a);
    add_planes(p, K0 + 1, a & ~b);
    add_planes(p, K0 + 2, b & ~c);
    add_planes(p, K0 + 3, c & ~d);
    return p;
}

// E of side 2 STEP from E of side STEP; a thread keeps its place z along a row of the plane.
template <int N, int PREV, int STEP>
__device__ __forceinline__ void cube_level(uint64_t* out, const uint64_t* in, int z, int y0) {
    if (z < N)
        for (int y = y0; y < N; y += 7) out[y * N + z] = cube_from<PREV, STEP>(in + y * PREV + z);
    __syncthreads();
}

__device__ void region_tile(const NodePass& P, int tile, RegSmem& s) {
    const Layout& L = P.L;
    const int x0 = (P.rx0 + tile % P.nrx) * 32, y0 = (P.ry0 + tile / P.nrx % P.nry) * 8;
    const int z0 = (P.rz0 + tile / (P.nrx * P.nry)) * 8;
    const int t = threadIdx.x;
    // the super blocks the tile and its halo span: 16 x 10 x 10; beyond the grid all is empty
    const int sx0 = x0 / 4 - 4, sy0 = y0 / 4 - 4, sz0 = z0 / 4 - 4;
    for (int i = t; i < kRegNodes; i += 256) {
        const int sx = sx0 + (i & 15), sy = sy0 + (i >> 4) % 10, sz = sz0 + i / 160;
        uint64_t m = 0;
        if (sx >= 0 && sy >= 0 && sz >= 0 && sx < L.SW && sy < L.SH && sz < L.SW)
            m = P.supers[super_index(L, sx, sy, sz)];
        s.nodes[i] = m;
    }
    __syncthreads();
    const uint32_t* n32 = reinterpret_cast<const uint32_t*>(s.nodes);
    // 36 threads along z, 7 rows of them along y (4 threads idle); rows beyond the grid in y, more
    // than half of them in flat worlds, are skipped by whole warps
    const int tz = t % 36, ty = t / 36;
    if (ty < 7)
        for (int y = ty; y < 36; y += 7)
            s.e1[y * 36 + tz] = (unsigned)(y0 - 14 + y) < (unsigned)L.RHp ? ~row_window<10>(n32, y + 2, tz + 2) : ~0ull;
    (&s.planes[0][0])[t] = 0;
    __syncthreads();
    const int first = ty < 7 ? ty : 99;
    cube_level<35, 36, 1>(s.e2, s.e1, tz, first);
    cube_level<33, 35, 2>(s.e4, s.e2, tz, first);
    cube_level<29, 33, 4>(s.e8, s.e4, tz, first);
    cube_level<21, 29, 8>(s.e16, s.e8, tz, first);
    const int row = t & 63, lz = row & 7, ly = row >> 3;
    const int part = t >> 6;  // four distances of the row each; warp-uniform
    const uint4 p = part == 0 ? centred_planes<0>(s, lz, ly)
                              : (part == 1 ? centred_planes<4>(s, lz, ly)
                                           : (part == 2 ? centred_planes<8>(s, lz, ly) : centred_planes<12>(s, lz, ly)));
    atomicOr(&s.planes[row][0], p.x);
    atomicOr(&s.planes[row][1], p.y);
    atomicOr(&s.planes[row][2], p.z);
    atomicOr(&s.planes[row][3], p.w);
    __syncthreads();
    const int r2 = t >> 2, z = z0 + (r2 & 7), y = y0 + (r2 >> 3);
    const uint4 q = *reinterpret_cast<const uint4*>(s.planes[r2]);
    for (int g = 0; g < 2; g++) {
        const int sh = 8 * (t & 3) + 4 * g;  // RWp is a multiple of 4: all four regions or none
        if (x0 + sh < L.RWp && y < L.RHp && z < L.RWp)
            *reinterpret_cast<uint32_t*>(P.rdist + region_linear(L, x0 + sh, y, z)) = plane_bytes(q, sh);
    }
}

// The solid bounding box and the depth-field flag: the brick pass left one record per CTA.
__device__ void merge_boxes(const NodePass& P, int* box) {
    const int t = threadIdx.x;
    if (t < 7) box[t] = t < 3 ? (P.reset_box ? INT_MAX : P.aabb[t])
                              : (t < 6 ? (P.reset_box ? INT_MIN : P.aabb[t]) : (P.reset_flag ? 0 : P.aabb[6]));
    __syncthreads();
    int v[7] = {INT_MAX, INT_MAX, INT_MAX, INT_MIN, INT_MIN, INT_MIN, 0};
    for (int i = t; i < P.n_boxes; i += 256) {
        const int4 a = *reinterpret_cast<const int4*>(P.boxes + 8 * i), b = *reinterpret_cast<const int4*>(P.boxes + 8 * i + 4);
        v[0] = min(v[0], a.x); v[1] = min(v[1], a.y); v[2] = min(v[2], a.z);
        v[3] = max(v[3], a.w); v[4] = max(v[4], b.x); v[5] = max(v[5], b.y); v[6] |= b.z;
    }
    for (int k = 0; k < 3; k++) atomicMin(box + k, v[k]);
    for (int k = 3; k < 6; k++) atomicMax(box + k, v[k]);
    atomicOr(box + 6, v[6]);
    __syncthreads();
    if (t < 7) P.aabb[t] = box[t];
}

// ------------------------------------------------------------------ launches

template <int SIDE>
union NodeSmem {
    DirSmem dir;
    RegSmem reg;
    typename FixTile<SIDE>::Smem fix;
    int box[8];
};

// The kinds of work lie one after the other in the grid, the longest first.  All of them only
// read what the brick pass wrote, and write different arrays.
// SIDE is that of the depth-field tiles.  8 stands for few CTAs, which an edit has: their time is
// one CTA's chain, and with the 94 registers that the compiler takes without a minimum of CTAs
// per SM it is shorter than with the 80 of a minimum of 3, with which a whole world's passes
// are faster.  That takes 0.5 us off an edit of radius 8, and with the small tiles 2.5 us off one of
// radius 7 with its depth field (1.4 of them by the tiles).
template <int SIDE>
__global__ void __launch_bounds__(256, SIDE == 8 ? 1 : 3) node_pass_kernel(const __grid_constant__ NodePass P) {
    __shared__ NodeSmem<SIDE> s;
    cudaTriggerProgrammaticLaunchCompletion();
    cudaGridDependencySynchronize();  // the brick pass before it
    int b = blockIdx.x;
    if (b < P.n_fix) return fix_tile<SIDE>(P.fix, b, s.fix);
    b -= P.n_fix;
    if (b < P.n_dir) return dir_tile(P, b, s.dir);
    b -= P.n_dir;
    if (b < P.n_reg) return region_tile(P, b, s.reg);
    merge_boxes(P, s.box);
}

// The depth field alone (fixDepthField over a box): without the distance tiles' 80 registers
// a fourth CTA fits on each SM.
__global__ void __launch_bounds__(256, 4) fix_depth_field_kernel(const __grid_constant__ FixPass P) {
    __shared__ FixTile<16>::Smem s;
    cudaTriggerProgrammaticLaunchCompletion();
    cudaGridDependencySynchronize();
    fix_tile<16>(P, blockIdx.x, s);
}

// ------------------------------------------------------------------ brick pass
//
// A warp takes 8 bricks in a row along x: lane (b, q) the four rows at z = q of brick b, one
// 16-byte load each, so that a load instruction covers four whole 128-byte lines.  The words
// are read once and written only where they change; the masks come from the same registers.
// The reference's level is made in this pass too: 33 us, bound by its stores and the trees'
// arithmetic, where layers, trees and masks took 131 us in three launches.
// Bound by the words' HBM reads: the 512 x 96 x 512 level takes 25 us (4 TB/s), where the masks
// of the three levels took 58 us in three launches.  An upload from device memory copies and
// masks in this one pass.  CTAs loop over their bricks and keep the bounding box in registers, which leaves one record
// per CTA instead of six atomics per warp.

// Four voxels of the reference's level (initVoxels, level.cpp:82-138) along x: stone, dirt
// and grass layers (:85-128), then the holes that placeBush and placeTrunk punch near the
// origin by calling destroyVoxel with relative coordinates (:11, :64) -- (0, 0..5, 0) from the
// trunks and the x, y, z >= 0 part of the radius-6 ball from the bushes -- and a tree at every
// x % 30 == 0, z % 25 == 0 of [10, W - 10) (:130-137): trunk, then bush, which wins where
// both are.  Trees are 30 x 25 voxels apart and 12 wide, so at most one reaches a voxel.
// (y is the same for a whole warp, so the layers' branches do not diverge.)
__device__ __forceinline__ void level_row(int (&v)[4], int x0, int y, int z, int W) {
    const bool any_tree = W - 10 > 30;  // the first ones stand at x = 30 and z = 25
    if (y <= 36) {
        // 5 * ((x + y + z) % 3) on top of every channel of stone, red and green of dirt, green of grass
        const int base = y <= 25 ? 0x5A5A5A : (y <= 33 ? 0x786400 : 0x0A820A);
        const int step = y <= 25 ? 0x050505 : (y <= 33 ? 0x050500 : 0x000500);
        const int m = (x0 + y + z) % 3, n = m == 2 ? 0 : m + 1, o = n == 2 ? 0 : n + 1;
        v[0] = v[3] = base + m * step;
        v[1] = base + n * step;
        v[2] = base + o * step;
        if (any_tree && y < 6 && x0 < 6 && z < 6)
            for (int e = 0; e < 4; e++)
                if ((x0 + e == 0 && z == 0) || (x0 + e < 6 && (x0 + e) * (x0 + e) + y * y + z * z < 36)) v[e] = -1;
    }
    if (any_tree && y >= 36 && y < 52) {
        const int tz = (z + 6) / 25 * 25, lean = tz % 7, oz = z - tz;  // level.cpp:133-134
        if (tz == 0 || tz >= W - 10 || oz >= 6) return;
        for (int e = 0; e < 4; e++) {
            const int tx = (x0 + e - lean + 6) / 30 * 30;
            const int ox = x0 + e - lean - tx;  // from the bush's centre, (tx + tz % 7, 46, tz)
            if (tx <= 0 || tx >= W - 10 || ox >= 6) continue;
            // placeTrunk(ivec3(bush x + 1, 36, tz), ivec3(128,100,15), 6): x, z in [-2,1), y in [0,6)
            const int ux = ox - 1, uy = y - 36, oy = y - 46;
            if (ux >= -2 && ux < 1 && oz >= -2 && oz < 1 && uy < 6) {
                const int d = (ux + oz) % 2 * 10;
                v[e] = ((((128 - d) << 8) + 100 - d) << 8) + 15;
            }
            // placeBush(ivec3(bush x, 46, tz), ivec3(15,128,15), 6): offsets in [-6,6)^3, |o|^2 < 36
            if (oy >= -6 && ox * ox + oy * oy + oz * oz < 36) v[e] = (((15 << 8) + 128 - (ox + oy + oz) % 3 * 20) << 8) + 15;
        }
    }
}

template <int OP, int MIN_CTAS>
// 64 registers, so that 4 CTAs of a large pass fit on each SM; an edit's few CTAs take 101 (MIN_CTAS
// 1: 0.2 us off an edit of radius 8, but 101.8 -> 116.8 us at radius 200).
__global__ void __launch_bounds__(256, MIN_CTAS) brick_pass_kernel(const __grid_constant__ BrickPass P) {
    cudaTriggerProgrammaticLaunchCompletion();  // the node pass may be put in place behind this
    cudaGridDependencySynchronize();
    const Layout& L = P.L;
    const int lane = threadIdx.x & 31, b = lane >> 2, q = lane & 3;
    const bool vec = (L.W & 3) == 0;
    int bx_lo = INT_MAX, by_lo = INT_MAX, bz_lo = INT_MAX, bx_hi = INT_MIN, by_hi = INT_MIN, bz_hi = INT_MIN;
    bool depth = false;
    for (unsigned task = blockIdx.x * 8 + (threadIdx.x >> 5); task < P.tasks; task += gridDim.x * 8) {
        const int by = P.by0 + (int)(task / P.ng % P.ny), bz = P.bz0 + (int)(task / P.ng / P.ny);
        const int bx = 8 * (P.g0 + (int)(task % P.ng)) + b;
        const bool in = bx >= P.bx0 && bx < P.bx1;
        const int x0 = 4 * bx, z = 4 * bz + q;
        const uint64_t slot = brick_index(L, bx, by, bz);
        uint64_t old = 0;
        if (in && q == 0) old = P.bricks[slot];
        int v[4][4];
#pragma unroll
        for (int dy = 0; dy < 4; dy++) {
            const int y = 4 * by + dy;
            const uint64_t at = ((uint64_t)z * L.H + y) * L.W + x0;
            v[dy][0] = v[dy][1] = v[dy][2] = v[dy][3] = -1;
            if (!(in && y < L.H && z < L.W)) continue;
            if (OP == kInitLevel) {
                level_row(v[dy], x0, y, z, L.W);
                if (!vec)
                    for (int e = 0; e < 4; e++)
                        if (x0 + e >= L.W) v[dy][e] = -1;
                continue;
            }
            if (vec) {
                const int32_t* from = P.words + at;
                if (OP == kCopyWords && at >= P.first && at + 4 <= P.first + P.count) {
                    const int32_t* src = P.src + (at - P.first);
                    if (((uintptr_t)src & 15) == 0) {
                        from = src;
                    } else {
                        for (int e = 0; e < 4; e++) v[dy][e] = src[e];
                        from = nullptr;
                    }
                }
                if (from) {
                    const int4 w = *reinterpret_cast<const int4*>(from);
                    v[dy][0] = w.x; v[dy][1] = w.y; v[dy][2] = w.z; v[dy][3] = w.w;
                }
            } else {
                for (int e = 0; e < 4; e++)
                    if (x0 + e < L.W) v[dy][e] = P.words[at + e];
            }
        }
        uint32_t chunk = 0;  // the 16 voxels at z = q, bit x + 4y
#pragma unroll
        for (int dy = 0; dy < 4; dy++) {
            const int y = 4 * by + dy;
            const bool row = in && y < L.H && z < L.W;
            if (OP != kReadWords && OP != kStopWords && row) {
                const uint64_t at = ((uint64_t)z * L.H + y) * L.W + x0;
                bool changed[4];
#pragma unroll
                for (int e = 0; e < 4; e++) {
                    changed[e] = false;
                    if (OP == kRemoveSphere) {
                        const int ox = x0 + e - P.x, oy = y - P.y, oz = z - P.z;
                        if (v[dy][e] != -1 && ox * ox + oy * oy + oz * oz < P.r * P.r) {
                            v[dy][e] = -1;
                            changed[e] = true;
                        }
                    } else if (OP == kPlaceVoxel) {
                        if (x0 + e == P.x && y == P.y && z == P.z) {
                            v[dy][e] = P.word;
                            changed[e] = true;
                        }
                    } else if (OP == kInitLevel) {
                        changed[e] = x0 + e < L.W;
                    } else {
                        const uint64_t i = at + e;
                        if (x0 + e < L.W && i >= P.first && i < P.first + P.count) {
                            if (!(vec && at >= P.first && at + 4 <= P.first + P.count)) v[dy][e] = P.src[i - P.first];
                            changed[e] = true;
                        }
                    }
                }
                if (vec && (changed[0] | changed[1] | changed[2] | changed[3])) {
                    *reinterpret_cast<int4*>(P.words + at) = make_int4(v[dy][0], v[dy][1], v[dy][2], v[dy][3]);
                } else if (!vec) {
                    for (int e = 0; e < 4; e++)
                        if (changed[e] && x0 + e < L.W) P.words[at + e] = v[dy][e];
                }
                if ((OP == kRemoveSphere || OP == kPlaceVoxel) && P.words_z)
                    for (int e = 0; e < 4; e++)
                        if (changed[e]) P.words_z[z + (uint64_t)L.W * y + (uint64_t)L.W * L.H * (x0 + e)] = v[dy][e];
            }
#pragma unroll
            for (int e = 0; e < 4; e++) {
                if (OP == kStopWords ? v[dy][e] != -1 : v[dy][e] >= 0) chunk |= 1u << (4 * dy + e);
                if (OP != kInitLevel) depth |= v[dy][e] < -1;
            }
        }
        uint32_t half = chunk << (16 * (q & 1));
        half |= __shfl_xor_sync(0xffffffffu, half, 1);
        const uint32_t other = __shfl_xor_sync(0xffffffffu, half, 2);
        const uint64_t m = (uint64_t)other << 32 | half;  // right in lanes q = 0
        if (in && q == 0) {
            if (m != old) P.bricks[slot] = m;
            if ((m != 0) != (old != 0)) {  // the brick's own bit of its region
                unsigned long long* r = reinterpret_cast<unsigned long long*>(
                    P.regions + region_index(L, bx >> 2, by >> 2, bz >> 2));
                const unsigned long long bit = 1ull << ((bx & 3) + 4 * (by & 3) + 16 * (bz & 3));
                // The region's own bit in its super block flips whenever the region's mask becomes
                // or stops being 0.  Flips of one region by several warps may arrive in any order:
                // their number alone decides the bit, which sets and clears would not.
                const unsigned long long was = m ? atomicOr(r, bit) : atomicAnd(r, ~bit);
                if (was == (m ? 0 : bit) && P.supers)
                    atomicXor(reinterpret_cast<unsigned long long*>(P.supers + super_index(L, bx >> 4, by >> 4, bz >> 4)),
                              1ull << ((bx >> 2 & 3) + 4 * (by >> 2 & 3) + 16 * (bz >> 2 & 3)));
            }
        }
        const unsigned solid = __ballot_sync(0xffffffffu, in && q == 0 && m != 0);
        if (solid) {
            const int first = bx - b;  // the warp's first brick
            bx_lo = min(bx_lo, first + (__ffs(solid) - 1) / 4);
            bx_hi = max(bx_hi, first + (31 - __clz(solid)) / 4);
            by_lo = min(by_lo, by); by_hi = max(by_hi, by);
            bz_lo = min(bz_lo, bz); bz_hi = max(bz_hi, bz);
        }
    }
    if (OP == kStopWords) return;
    __shared__ int box[8];
    if (threadIdx.x < 8) box[threadIdx.x] = threadIdx.x < 3 ? INT_MAX : (threadIdx.x < 6 ? INT_MIN : 0);
    __syncthreads();
    if (__any_sync(0xffffffffu, depth) && lane == 0) box[6] = 1;
    if (lane == 0 && bx_lo != INT_MAX) {
        atomicMin(box, 4 * bx_lo); atomicMin(box + 1, 4 * by_lo); atomicMin(box + 2, 4 * bz_lo);
        atomicMax(box + 3, 4 * bx_hi + 3); atomicMax(box + 4, 4 * by_hi + 3); atomicMax(box + 5, 4 * bz_hi + 3);
    }
    __syncthreads();
    if (threadIdx.x < 8) P.boxes[8 * blockIdx.x + threadIdx.x] = box[threadIdx.x];
}

// The brick box [b0, b1) of a voxel box, clipped to the world; false when it is empty.
static bool brick_box(const Layout& L, const int64_t v[6], int b[6]) {
    const int dim[3] = {L.W, L.H, L.W};
    for (int a = 0; a < 3; a++) {
        const int64_t lo = std::max<int64_t>(v[a], 0), hi = std::min<int64_t>(v[3 + a], dim[a]);
        if (lo >= hi) return false;
        b[a] = (int)(lo >> 2);
        b[3 + a] = (int)((hi + 3) >> 2);
    }
    return true;
}

template <int OP>
static int run_brick_pass(BrickPass& P, int num_sms, cudaStream_t s, bool behind, int* blocks) {
    // Whole worlds: as many CTAs as fit at once, each looping over its share
    const unsigned need = (P.tasks + 7) / 8;
    *blocks = (int)std::min<unsigned>(need, (unsigned)num_sms * kBrickCtasPerSm);
    constexpr int kFew = OP == kRemoveSphere || OP == kPlaceVoxel ? 1 : 4;
    VRT_CUDA(launch_behind(behind, *blocks <= 2 * num_sms ? brick_pass_kernel<OP, kFew> : brick_pass_kernel<OP, 4>,
                           dim3(*blocks), 256, s, P));
    return VRT_OK;
}

static BrickPass brick_pass_of(vrt_world* w, const int b[6]) {
    BrickPass P{};
    P.words = w->d_words;
    P.bricks = w->d_bricks;
    P.regions = w->d_regions;
    P.supers = w->d_supers;
    P.boxes = w->d_boxes;
    P.L = w->L;
    P.bx0 = b[0]; P.by0 = b[1]; P.bz0 = b[2]; P.bx1 = b[3];
    P.g0 = b[0] >> 3;
    P.ng = (unsigned)(((b[3] + 7) >> 3) - P.g0);
    P.ny = (unsigned)(b[4] - b[1]);
    P.tasks = P.ng * P.ny * (unsigned)(b[5] - b[2]);
    return P;
}

// Distance tiles of every brick (region) within kDistCap of the changed box.
static void node_tiles(NodePass& P, const int b[6]) {
    const Layout& L = P.L;
    int lo[3], hi[3], rlo[3], rhi[3];
    const int bdim[3] = {L.BWp, L.BHp, L.BWp}, rdim[3] = {L.RWp, L.RHp, L.RWp};
    for (int a = 0; a < 3; a++) {
        lo[a] = std::max(b[a] - kDistCap, 0);
        hi[a] = std::min(b[3 + a] + kDistCap, bdim[a]);
        rlo[a] = std::max((b[a] >> 2) - kDistCap, 0);
        rhi[a] = std::min(((b[3 + a] + 3) >> 2) + kDistCap, rdim[a]);
    }
    P.dx0 = lo[0] >> 5; P.ndx = ((hi[0] + 31) >> 5) - P.dx0;
    P.dy0 = lo[1] >> 3; P.ndy = ((hi[1] + 7) >> 3) - P.dy0;
    P.dz0 = lo[2] >> 3; P.n_dir = 4 * P.ndx * P.ndy * (((hi[2] + 7) >> 3) - P.dz0);
    P.rx0 = rlo[0] >> 5; P.nrx = ((rhi[0] + 31) >> 5) - P.rx0;
    P.ry0 = rlo[1] >> 3; P.nry = ((rhi[1] + 7) >> 3) - P.ry0;
    P.rz0 = rlo[2] >> 3; P.n_reg = P.nrx * P.nry * (((rhi[2] + 7) >> 3) - P.rz0);
}

static bool fix_tiles(NodePass& N, vrt_world* w, const int64_t v[6], int cx, int cy, int cz, int r2) {
    FixPass& P = N.fix;
    const int dim[3] = {w->L.W, w->L.H, w->L.W};
    int lo[3], hi[3];
    for (int a = 0; a < 3; a++) {
        const int64_t l = std::max<int64_t>(v[a], 0), h = std::min<int64_t>(v[3 + a], dim[a]);
        if (l >= h) return false;
        lo[a] = (int)l;
        hi[a] = (int)h;
    }
    P.words = w->d_words;
    P.bricks = w->d_bricks;
    P.L = w->L;
    P.x0 = lo[0]; P.y0 = lo[1]; P.z0 = lo[2];
    P.x1 = hi[0]; P.y1 = hi[1]; P.z1 = hi[2];
    P.cx = cx; P.cy = cy; P.cz = cz; P.r2 = r2;
    for (int i = 0; i <= kFixLevels; i++) {
        // render.cpp:81: -sqrt(int) through double sqrt, stored as float; nothing found: the
        // running value's start, -DEPTH_FIELD_RADIUS + 1
        const float d = i < kFixLevels ? (float)(-std::sqrt((double)i)) : -6.0f;
        std::memcpy(&P.word[i], &d, 4);
    }
    // small tiles where they don't outnumber the SMs; larger boxes pay for their halo, and the depth
    // field alone (no brick pass ahead) always covers large ones
    for (int side = 8;; side = 16) {
        P.small = side == 8;
        P.tx0 = P.x0 / kFixX; P.ty0 = P.y0 / side; P.tz0 = P.z0 / side;
        P.ntx = (P.x1 - 1) / kFixX - P.tx0 + 1;
        P.nty = (P.y1 - 1) / side - P.ty0 + 1;
        N.n_fix = P.ntx * P.nty * ((P.z1 - 1) / side - P.tz0 + 1);
        if (side == 16 || (N.n_boxes > 0 && N.n_fix <= w->num_sms)) break;
    }
    return true;
}

static int run_node_pass(const NodePass& P, int num_sms, cudaStream_t s, bool behind) {
    const int blocks = P.n_fix + P.n_dir + P.n_reg + (P.n_boxes > 0 ? 1 : 0);
    if (blocks > 0 && blocks == P.n_fix) VRT_CUDA(launch_behind(behind, fix_depth_field_kernel, dim3(blocks), 256, s, P.fix));
    else if (blocks > 0)
        VRT_CUDA(launch_behind(behind, (P.n_fix ? P.fix.small : blocks <= 2 * num_sms) ? node_pass_kernel<8> : node_pass_kernel<16>,
                               dim3(blocks), 256, s, P));
    return VRT_OK;
}

// The voxels of a box, clipped to the world.
static int64_t volume(const Layout& L, const int64_t v[6]) {
    const int dim[3] = {L.W, L.H, L.W};
    int64_t n = 1;
    for (int a = 0; a < 3; a++) n *= std::max<int64_t>(std::min<int64_t>(v[3 + a], dim[a]) - std::max<int64_t>(v[a], 0), 0);
    return n;
}

// Edits of at most this many voxels keep the z-major copy up to date word by word, which
// saves the next frame a launch (3.6 us); each such word is a store of its own sector, so
// larger changes leave the copy to the next word-kernel render, which copies the box in one launch.
constexpr int64_t kWriteThrough = 1 << 16;

int change_words(vrt_world* w, const WordChange& c, cudaStream_t s) {
    const Layout& L = w->L;
    const bool behind = mark_changed(w, s);
    const bool through = w->d_words_z && (c.op == kRemoveSphere || c.op == kPlaceVoxel) &&
                         volume(L, c.box) <= kWriteThrough && (!c.fix || volume(L, c.fix_box) <= kWriteThrough);
    NodePass N{};
    N.L = L;
    N.regions = w->d_regions;
    N.bdir = reinterpret_cast<uint16_t*>(w->d_bdir);
    N.supers = w->d_supers;
    N.rdist = w->d_rdist;
    N.aabb = w->d_aabb;
    N.boxes = w->d_boxes;
    int b[6];
    if (brick_box(L, c.box, b)) {
        mark_words(w, c.box, !through);
        BrickPass P = brick_pass_of(w, b);
        P.words_z = through ? w->d_words_z : nullptr;
        P.src = c.src; P.first = c.first; P.count = c.count;
        P.x = c.x; P.y = c.y; P.z = c.z; P.r = c.r; P.word = c.word;
        int st = VRT_OK;
        switch (c.op) {
            case kReadWords: st = run_brick_pass<kReadWords>(P, w->num_sms, s, behind, &N.n_boxes); break;
            case kRemoveSphere: st = run_brick_pass<kRemoveSphere>(P, w->num_sms, s, behind, &N.n_boxes); break;
            case kInitLevel: st = run_brick_pass<kInitLevel>(P, w->num_sms, s, behind, &N.n_boxes); break;
            case kPlaceVoxel: st = run_brick_pass<kPlaceVoxel>(P, w->num_sms, s, behind, &N.n_boxes); break;
            default: st = run_brick_pass<kCopyWords>(P, w->num_sms, s, behind, &N.n_boxes); break;
        }
        if (st) return st;
        node_tiles(N, b);
        // a pass over the whole world knows the solid bounding box; a partial one only grows it
        N.reset_box = b[0] == 0 && b[1] == 0 && b[2] == 0 && 4 * b[3] >= L.W && 4 * b[4] >= L.H && 4 * b[5] >= L.W;
        N.reset_flag = c.reset_flag;
    }
    if (c.fix && fix_tiles(N, w, c.fix_box, c.x, c.y, c.z, c.fix_r)) {
        N.fix.words_z = through ? w->d_words_z : nullptr;
        mark_words(w, c.fix_box, !through);
    }
    return run_node_pass(N, w->num_sms, s, behind);
}

int refresh_stop_masks(vrt_world* w, cudaStream_t s, bool behind) {
    const Layout& L = w->L;
    const int64_t v[6] = {0, 0, 0, L.W, L.H, L.W};
    int b[6], blocks = 0;
    brick_box(L, v, b);
    BrickPass P = brick_pass_of(w, b);
    P.bricks = w->d_stop;
    P.regions = w->d_stop_regions;
    P.supers = nullptr;
    const int st = run_brick_pass<kStopWords>(P, w->num_sms, s, behind, &blocks);
    if (st) return st;
    NodePass N{};
    N.L = L;
    node_tiles(N, b);
    N.regions = w->d_stop_regions;
    N.bdir = reinterpret_cast<uint16_t*>(w->d_sdir);
    N.n_reg = 0;
    return run_node_pass(N, w->num_sms, s, behind);
}

}  // namespace vrt
