// Bit-parallel passes over the occupancy masks: the depth field (fixDepthField,
// render.cpp:226-253).
//
// A row of 32 voxels along x is one 32-bit word here.  The masks already hold a bit per
// voxel, 4 bits of a row in each brick, so a tile of rows with its halo is put together in
// shared memory from the few KB of masks it spans, and the neighbourhood work of 32
// voxels is done by one instruction.
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstring>
#include <utility>

#include "vrt_internal.h"

namespace vrt {

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

constexpr int kFixX = 32, kFixY = 16, kFixZ = 16;  // voxels per tile: one row word x 16 x 16 rows
constexpr int kFixHalo = 7;                        // DEPTH_FIELD_RADIUS, render.hpp:7
constexpr int kFixRows = kFixY + 2 * kFixHalo;     // rows per axis with the halo
// Row pitch of a D_k plane: a warp's lanes are 16 rows in y of two z, so a pitch of 16
// modulo 32 puts them into 32 different banks.
constexpr int kFixPitch = 48;
constexpr int kFixPlane = kFixRows * kFixPitch;
constexpr int kFixK = 6;               // D_1 .. D_6 (|x| = 7 alone gives s = 36)
constexpr int kFixNodes = 12 * 8 * 8;  // bricks spanned: 8 + 2 x 2 in x, 4 + 2 x 2 in y and z
constexpr int kFixLevels = 36;

struct FixSmem {
    uint64_t nodes[kFixNodes];
    uint32_t d[kFixK * kFixPlane];
    uint32_t out[7][kFixY * kFixZ];  // per row: the 6 bits of s, and the voxels to write
    int32_t word[kFixLevels + 1];    // the depth-field word of each s; [36]: no solid neighbour
};

// Offsets (into FixSmem::d, from a row's own place in D_1) of the planes that level S adds.
// Level 3 stands for every s <= 3, whose voxels all keep their word.
struct FixLevel {
    int n = 0;
    int off[160] = {};
};
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
            if (best) r.off[r.n++] = (best - 1) * kFixPlane + dz * kFixPitch + dy;
        }
    return r;
}

template <int S>
struct FixTable {
    static constexpr FixLevel L = fix_level(S);
};

template <int S, int... I>
__device__ __forceinline__ uint32_t fix_or(const uint32_t* d, std::integer_sequence<int, I...>) {
    uint32_t f = 0;
    ((f |= d[std::integral_constant<int, FixTable<S>::L.off[I]>::value]), ...);
    return f;
}

// Add level S (and the levels after it) to a row: found = voxels whose smallest s is known.
template <int S>
__device__ __forceinline__ void fix_levels(const uint32_t* d, uint32_t& found, uint32_t (&bit)[6]) {
    if constexpr (S < kFixLevels) {
        if constexpr (FixTable<S>::L.n > 0) {
            const uint32_t now = fix_or<S>(d, std::make_integer_sequence<int, FixTable<S>::L.n>{}) & ~found;
            found |= now;
            if (S & 1) bit[0] |= now;
            if (S & 2) bit[1] |= now;
            if (S & 4) bit[2] |= now;
            if (S & 8) bit[3] |= now;
            if (S & 16) bit[4] |= now;
            if (S & 32) bit[5] |= now;
        }
        fix_levels<S + 1>(d, found, bit);
    }
}

struct FixPass {
    int32_t* words;
    const uint64_t* bricks;
    Layout L;
    int x0, y0, z0, x1, y1, z1;  // the voxels to refresh, within the world
    int cx, cy, cz, r2;          // r2 > 0: of those, the ones inside this sphere
    int tx0, ty0, tz0, ntx, nty; // the tiles that cover the box
    int32_t word[kFixLevels + 1];
};

// One 32 x 16 x 16 tile by 256 threads, one row each.  Only the air voxels of P.box (and of
// the sphere, if there is one) are written; only solidity is read, which no thread changes.
__device__ void fix_tile(const FixPass& P, int tile, FixSmem& s) {
    const Layout& L = P.L;
    const int tx = tile % P.ntx, ty = (tile / P.ntx) % P.nty, tz = tile / (P.ntx * P.nty);
    const int x0 = (P.tx0 + tx) * kFixX, y0 = (P.ty0 + ty) * kFixY, z0 = (P.tz0 + tz) * kFixZ;
    const int t = threadIdx.x;

    // the bricks the tile and its halo span; bricks beyond the grid hold no solid voxel
    const int bx0 = x0 / 4 - 2, by0 = y0 / 4 - 2, bz0 = z0 / 4 - 2;
    bool solid = false;
    for (int i = t; i < kFixNodes; i += 256) {
        const int bx = bx0 + i % 12, by = by0 + (i / 12) % 8, bz = bz0 + i / 96;
        uint64_t m = 0;
        if (bx >= 0 && by >= 0 && bz >= 0 && bx < L.BWp && by < L.BHp && bz < L.BWp)
            m = P.bricks[brick_index(L, bx, by, bz)];
        s.nodes[i] = m;
        solid |= m != 0;
    }
    if (t <= kFixLevels) s.word[t] = P.word[t];
    const bool any_solid = __syncthreads_or(solid);

    // this thread's own row, and the voxels of it that may be written
    const int y = y0 + (t & 15), z = z0 + (t >> 4);
    const uint32_t* n32 = reinterpret_cast<const uint32_t*>(s.nodes);
    uint32_t air = 0;
    if (y >= P.y0 && y < P.y1 && z >= P.z0 && z < P.z1) {
        const int node = ((y >> 2) - by0) * 12 + ((z >> 2) - bz0) * 96;
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
        for (int i = t; i < kFixRows * kFixRows; i += 256) {
            const int ry = i % kFixRows, rz = i / kFixRows;
            const int py = ry + 1, pz = rz + 1;  // rows start at y0 - 7 = 4 * by0 + 1
            const int node = (py >> 2) * 12 + (pz >> 2) * 96, half = (pz & 3) >> 1;
            const int shift = 4 * (py & 3) + 16 * (pz & 1);
            uint64_t w = 0;
#pragma unroll
            for (int j = 0; j < 12; j++)
                w |= (uint64_t)(n32[2 * (node + j) + half] >> shift & 15) << (4 * j);
            uint32_t* d = s.d + rz * kFixPitch + ry;
            uint32_t c = (uint32_t)(w >> 8);
#pragma unroll
            for (int k = 1; k <= kFixK; k++) {
                c |= (uint32_t)(w >> (8 + k)) | (uint32_t)(w >> (8 - k));
                d[(k - 1) * kFixPlane] = c;
            }
        }
        __syncthreads();
        if (air) fix_levels<3>(s.d + ((t >> 4) + kFixHalo) * kFixPitch + (t & 15) + kFixHalo, found, bit);
    }
    // s <= 3 was recorded as 3: those voxels keep their word
    const uint32_t keep = found & ~(bit[2] | bit[3] | bit[4] | bit[5]);
#pragma unroll
    for (int k = 0; k < 6; k++) s.out[k][t] = bit[k];
    s.out[6][t] = air & ~keep;
    __syncthreads();

    // write: a warp per row, a lane per voxel
    const int lane = t & 31;
    for (int row = t >> 5; row < kFixY * kFixZ; row += 8) {
        const uint32_t wr = s.out[6][row];
        if (!(wr >> lane & 1)) continue;
        const int ry = y0 + (row & 15), rz = z0 + (row >> 4), rx = x0 + lane;
        if (P.r2 > 0) {
            const int ox = rx - P.cx, oy = ry - P.cy, oz = rz - P.cz;
            if (ox * ox + oy * oy + oz * oz >= P.r2 * P.r2) continue;
        }
        int sq = 0;
#pragma unroll
        for (int k = 0; k < 6; k++) sq |= (int)(s.out[k][row] >> lane & 1) << k;
        // every recorded s is at least 3, so 0 says that no solid voxel was found
        P.words[(uint64_t)rx + (uint64_t)L.W * ry + (uint64_t)L.W * L.H * rz] = s.word[sq ? sq : kFixLevels];
    }
}

__global__ void __launch_bounds__(256) fix_depth_field_kernel(const __grid_constant__ FixPass P) {
    __shared__ FixSmem s;
    fix_tile(P, blockIdx.x, s);
}

int launch_fix_depth_field(vrt_world* w, int x0, int y0, int z0, int x1, int y1, int z1, int cx, int cy, int cz,
                           int r2, cudaStream_t s) {
    FixPass P{};
    P.words = w->d_words;
    P.bricks = w->d_bricks;
    P.L = w->L;
    P.x0 = std::max(x0, 0); P.y0 = std::max(y0, 0); P.z0 = std::max(z0, 0);
    P.x1 = std::min(x1, w->L.W); P.y1 = std::min(y1, w->L.H); P.z1 = std::min(z1, w->L.W);
    if (P.x0 >= P.x1 || P.y0 >= P.y1 || P.z0 >= P.z1) return VRT_OK;
    P.cx = cx; P.cy = cy; P.cz = cz; P.r2 = r2;
    for (int i = 0; i <= kFixLevels; i++) {
        // render.cpp:81: -sqrt(int) through double sqrt, stored as float; nothing found: the
        // running value's start, -DEPTH_FIELD_RADIUS + 1
        const float d = i < kFixLevels ? (float)(-std::sqrt((double)i)) : -6.0f;
        std::memcpy(&P.word[i], &d, 4);
    }
    P.tx0 = P.x0 / kFixX; P.ty0 = P.y0 / kFixY; P.tz0 = P.z0 / kFixZ;
    P.ntx = (P.x1 - 1) / kFixX - P.tx0 + 1;
    P.nty = (P.y1 - 1) / kFixY - P.ty0 + 1;
    const int ntz = (P.z1 - 1) / kFixZ - P.tz0 + 1;
    fix_depth_field_kernel<<<P.ntx * P.nty * ntz, 256, 0, s>>>(P);
    VRT_CUDA(cudaGetLastError());
    return VRT_OK;
}

}  // namespace vrt
