// Internal declarations shared by the translation units of libvrt.so.
#pragma once

#include <cuda_runtime.h>

#include <climits>
#include <cstdint>
#include <cstdio>
#include <string>

#include "vrt_host.h"

namespace vrt {

// ---- error plumbing: every C entry point returns a status and records a message ----
int cuda_error(cudaError_t e, const char* what);

#define VRT_CUDA(call)                                       \
    do {                                                     \
        cudaError_t e_ = (call);                             \
        if (e_ != cudaSuccess) return ::vrt::cuda_error(e_, #call); \
    } while (0)

// ---- occupancy hierarchy ----
// Three levels of 64-bit masks over the voxel words (a 64-ary tree):
//   brick  (4x4x4 voxels):   bit (x&3) + 4*(y&3) + 16*(z&3) set when that voxel is solid
//   region (16x16x16):       bit per brick (bx&3) + 4*(by&3) + 16*(bz&3) set when the brick has a solid voxel
//   super  (64x64x64):       bit per region, same layout, set when the region has a solid voxel
// Bricks are stored linearly, bx + BWp*(by + BHp*bz), so a ray's box lookup computes its
// brick's slot with two multiply-adds; regions are stored super-major (64 regions of a
// super block = 512 contiguous bytes).  Voxels outside the world count as empty.
struct Layout {
    int W, H;           // voxel dims: x,z in [0,W), y in [0,H)
    int RW, RH;         // regions per axis (x/z, y): ceil(W/16), ceil(H/16)
    int SW, SH;         // super blocks per axis: ceil(W/64), ceil(H/64)
    int RWp, RHp;       // regions per axis padded to a multiple of 4 (= 4*SW, 4*SH)
    int BWp, BHp;       // bricks per axis, padded (= 16*SW, 16*SH)
    uint64_t n_words;   // W*H*W
    uint64_t n_bricks;  // 64 * RWp*RHp*RWp
    uint64_t n_regions; // 64 * SW*SH*SW
    uint64_t n_supers;  // SW*SH*SW
};

// Empty-space distance fields (capped Chebyshev distance, in nodes, to the nearest
// non-empty node; 0 = the node itself holds a solid voxel).  Values are capped (never
// larger than the truth) and recomputed whenever solids may be added.
//   region distance: uint8 per region, linear index rx + RWp*(ry + RHp*rz).  A region at
//   distance d >= 1 has every region within Chebyshev radius d-1 empty, so the cube of
//   those regions is a box a ray can cross without reading voxels.
constexpr int kDistCap = 15;

// Directed brick distances: 8 bytes per brick, stored like the brick masks.  Byte o
// (octant o: bit a set = the + direction along axis a, x=0 y=1 z=2) holds, as the
// dist_code that a lookup adds to a box, the capped Chebyshev distance from the brick to
// the nearest non-empty brick n in that octant (n_a >= b_a where bit a is set, n_a <= b_a
// where it is clear).  At distance d >= 1
// the cube of bricks from b to b + (d-1) in the octant's directions is empty: a ray
// moving into that octant leaves its brick only through that cube's far faces, so the
// cube bounds it as well as a centred cube of the same radius would, while solids
// behind or beside the ray no longer shrink it.  The code is the cells of the cube beyond the
// brick itself: 4 (d - 1), and 0 for a non-empty brick.
constexpr int dist_code(int d) { return d > 0 ? 4 * (d - 1) : 0; }

__host__ __device__ inline uint64_t region_linear(const Layout& L, int rx, int ry, int rz) {
    return (uint64_t)rx + (uint64_t)L.RWp * ((uint64_t)ry + (uint64_t)L.RHp * rz);
}

__host__ __device__ inline uint64_t super_index(const Layout& L, int sx, int sy, int sz) {
    return (uint64_t)sx + (uint64_t)L.SW * ((uint64_t)sy + (uint64_t)L.SH * sz);
}
// region (rx,ry,rz) -> slot in the region array
__host__ __device__ inline uint64_t region_index(const Layout& L, int rx, int ry, int rz) {
    return super_index(L, rx >> 2, ry >> 2, rz >> 2) * 64 + ((rx & 3) + 4 * (ry & 3) + 16 * (rz & 3));
}
// brick (bx,by,bz) -> slot in the brick array (and the brick distance field)
__host__ __device__ inline uint64_t brick_index(const Layout& L, int bx, int by, int bz) {
    return (uint64_t)bx + (uint64_t)L.BWp * ((uint64_t)by + (uint64_t)L.BHp * bz);
}

Layout make_layout(int W, int H);

}  // namespace vrt

namespace vrt {
// When a structure that renders derive from the words was last rebuilt: renders on other streams wait
// for that.  A rebuild within a stream capture belongs to its graph, so it is known by the capture, up to
// the next change, and leaves the state of the plain launches as it is.
struct Derived {
    cudaEvent_t ready = nullptr;     // recorded after each plain rebuild
    cudaEvent_t captured = nullptr;  // recorded after the rebuild within capture `capture`
    unsigned long long capture = 0;  // 0: none since the last change
};
}  // namespace vrt

struct vrt_world {
    vrt::Layout L;
    int32_t* d_words = nullptr;
    uint64_t* d_bricks = nullptr;
    uint64_t* d_regions = nullptr;
    uint64_t* d_supers = nullptr;
    uint8_t* d_rdist = nullptr;     // region distance field (linear, RWp*RHp*RWp)
    uint8_t* d_bdir = nullptr;      // directed brick distances (8 bytes per brick, linear)
    uint64_t* d_stop = nullptr;     // depth-field worlds: brick masks of the cells a ray stops at
                                    // (word != -1: solid or depth-field), made on first use
    uint8_t* d_sdir = nullptr;      // directed brick distances over the stop masks
    vrt::Derived stop;              // when the stop structures were rebuilt
    bool stop_stale = true;         // they predate the last change of the words
    bool stop_cleared = false;      // they started from 0
    int32_t* d_words_z = nullptr;   // the word kernel's second copy of the words with x and z swapped
                                    // (index z + W*y + W*H*x), made on first use
    vrt::Derived z;                 // when the copy was brought up to date
    bool z_filled = false;          // it has been filled once
    int z_dirty[6] = {0, 0, 0, 0, 0, 0};  // box [x0,x1)x[y0,y1)x[z0,z1) of words changed since the
                                    // copy was last brought up to date (empty: x0 >= x1)
    uint64_t* d_stop_regions = nullptr;  // region masks of the stop masks
    int* d_boxes = nullptr;         // the brick pass's record per CTA (8 ints: solid box, flag, 0)
    int* d_aabb = nullptr;          // bounding box of the solid voxels, brick-granular and
                                    // never smaller than the truth: min x,y,z then max x,y,z;
                                    // [6] the has-depth-field flag
    int h_aabb[6] = {0, 0, 0, -1, -1, -1};  // host copy passed to the render kernels; kept a
                                    // superset of the device box (read back after uploads)
    int has_depth_field = 0;        // host copy (as of the last sync)
    int graph_box[6] = {INT_MAX, INT_MAX, INT_MAX, INT_MIN, INT_MIN, INT_MIN};  // a world that captured
    int graph_depth = 0;            // graphs change: the voxels and the flag that their runs may bring,
                                    // part of both host copies from then on (note_added)
    uint64_t device_bytes = 0;
    int device = 0;
    int num_sms = 0;
    uint64_t stamp = 0;             // a new one with every change of what renders read (mark_changed),
                                    // 0 for a world with a change in a captured graph
    bool in_graph = false;          // such a graph's runs change the words unseen: the masks and distances
                                    // with them, but neither the stop structures nor a large change's
                                    // z-major copy, which every frame that reads them rebuilds then
    bool reads_pageable = false;    // kernels read pageable host memory through the host's page tables
};

namespace vrt {
// A change of a world's words and what follows from it (world_passes.cu).
enum { kReadWords, kRemoveSphere, kPlaceVoxel, kCopyWords, kInitLevel, kStopWords };
struct WordChange {
    int op;                 // kReadWords: the words changed already, or are to be looked at again;
                            // kInitLevel: the reference's level (initVoxels, level.cpp:82-138)
    int64_t box[6];         // the words concerned: [x0,y0,z0, x1,y1,z1), clipped to the world; may be empty
    const int32_t* src;     // kCopyWords: words [first, first + count) are copied from here
    uint64_t first, count;
    int x, y, z, r;         // kRemoveSphere: |v - c|^2 < r^2 becomes air; kPlaceVoxel: the voxel
    int32_t word;           // kPlaceVoxel
    bool reset_flag;        // whole-world boxes: the depth-field flag starts from 0
    bool fix;               // then fixDepthField (render.cpp:226-253) over fix_box, and with
    int64_t fix_box[6];     // fix_r > 0 only over its voxels with |v - c|^2 < fix_r^2 (removeSphere's
    int fix_r;              // second loop, level.cpp:43-55)
};
// Change the words, and bring the masks, distances, solid box and flag up to date: at most two
// launches.
int change_words(vrt_world* w, const WordChange& c, cudaStream_t s);
// The address at which the brick pass reads an upload's words, or NULL where only a copy may take
// them: at src, whose attributes are at, for a world on GPU `device`.  A copy takes, or refuses, any
// address, another GPU's memory included, which a kernel without peer access faults on.
inline const int32_t* upload_view(const int32_t* src, bool from_host, const cudaPointerAttributes& at, int device,
                                  bool reads_pageable) {
    if ((uintptr_t)src & 3) return nullptr;  // the pass loads whole words
    if (!from_host) return at.type == cudaMemoryTypeDevice && at.device == device ? src : nullptr;
    // Page-locked memory is mapped; where the device walks the host's page tables (Grace), so is every
    // other page of the host.  The words then cross the host link once, in the pass that masks them,
    // without the copy's staging: 64 MiB in 369 us from pageable memory seen before and 409 us from
    // fresh pages, where the copy and a mask pass took 428 and 472 us.
    if (at.type == cudaMemoryTypeDevice) return nullptr;  // not host memory: the copy says so
    if (reads_pageable) return src;
    return at.type == cudaMemoryTypeHost && !((uintptr_t)at.devicePointer & 3)
               ? static_cast<const int32_t*>(at.devicePointer)
               : nullptr;
}
// The stream's capture: its id, or 0 where launches run.  *plain: no capture is known to be in the way
// of a launch as a programmatic dependent.
unsigned long long capture_of(cudaStream_t s, bool* plain);
// Called with every launch that changes the words, or what plain launches derive from them for
// renders.  False under capture, and for a world that a captured graph changes: its launches are
// plain ones.
bool mark_changed(vrt_world* w, cudaStream_t s);
// A launch that may begin, as far as its cudaGridDependencySynchronize, while the kernel ahead on
// the stream runs, from when all CTAs of that one have begun or let it
// (cudaTriggerProgrammaticLaunchCompletion); not dependent: a plain launch.  World changes and
// probes wait before their first access, which hides the launch itself: 0.6 us of each edit of
// a row, 2.4 us of probe, edit and frame, 5 us of the level built with four edits.  Kernels launched so read what others wrote by plain loads, never
// the read-only path, whose lines need not be those of after the wait.
// A kernel that triggers before its own wait lets what is behind it begin while the kernels ahead
// of it still run: it may write nothing that a kernel without a wait before its reads (an
// overlapped frame) goes by.  World changes keep to that by the stamp, which makes the next frame
// wait; a frame that waits first triggers behind its wait.
template <class... Params, class... Args>
cudaError_t launch_behind(bool dependent, void (*kern)(Params...), dim3 grid, int threads, cudaStream_t s,
                          const Args&... args) {
    cudaLaunchAttribute pdl{};
    pdl.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    pdl.val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = grid;
    cfg.blockDim = dim3(threads);
    cfg.stream = s;
    cfg.attrs = &pdl;
    cfg.numAttrs = dependent ? 1 : 0;
    return cudaLaunchKernelEx(&cfg, kern, args...);
}
// Note that the words of the box changed: the stop masks follow, and there the z-major copy
// if it has not been changed with them.
void mark_words(vrt_world* w, const int64_t box[6], bool z_copy);
// CTAs of a brick pass per SM, at most
constexpr int kBrickCtasPerSm = 4;
// Rebuild the stop masks and their directed distances from the words.
int refresh_stop_masks(vrt_world* w, cudaStream_t s, bool behind);
// Bring the stop masks and their directed distances up to date (allocated on first use),
// and make stream s wait until they are: the rebuild may have run on another stream.
int refresh_stop(vrt_world* w, cudaStream_t s);
// Bring the z-major copy of the words up to date (allocated and filled on first use, then
// only the box changed since), and make stream s wait until it is: the update may have
// run on another stream.
int refresh_words_z(vrt_world* w, cudaStream_t s);
// vrt_render_batch without the box-lookup counter: the launch that stores no side output
// and counts no lookups, a burst of requests in 2755 us instead of 2830.
int render_batch_rays(vrt_renderer* r, const vrt_view* views, int32_t count, void* stream);
}  // namespace vrt
