// Device-resident worlds: the voxel words (the reference's SSBO), the derived occupancy
// hierarchy, and the edit kernels that replace the reference's CPU world code:
//   removeSphere  level.cpp:30-56        -> change_words (world_passes.cu)
//   fixDepthField render.cpp:226-253     -> change_words
//   placeVoxel    render.cpp:256-262     -> change_words
//   initVoxels    level.cpp:82-138       -> change_words
//   updateGeometry/updatePartialGeometry render.cpp:199-223 -> vrt_world_upload -> change_words
#include <cuda_runtime.h>

#include <algorithm>
#include <atomic>
#include <climits>
#include <cstdio>
#include <cstring>
#include <vector>

#include "vrt_internal.h"

namespace vrt {

Layout make_layout(int W, int H) {
    Layout L{};
    L.W = W;
    L.H = H;
    L.RW = (W + 15) / 16;
    L.RH = (H + 15) / 16;
    L.SW = (W + 63) / 64;
    L.SH = (H + 63) / 64;
    L.RWp = 4 * L.SW;
    L.RHp = 4 * L.SH;
    L.BWp = 16 * L.SW;
    L.BHp = 16 * L.SH;
    L.n_words = (uint64_t)W * H * W;
    L.n_supers = (uint64_t)L.SW * L.SH * L.SW;
    L.n_regions = 64 * L.n_supers;
    L.n_bricks = 64 * L.n_regions;
    return L;
}

static inline unsigned blocks_for(uint64_t n, int threads) { return (unsigned)((n + threads - 1) / threads); }

unsigned long long capture_of(cudaStream_t s, bool* plain) {
    cudaStreamCaptureStatus status = cudaStreamCaptureStatusNone;
    unsigned long long id = 0;
    const bool known = cudaStreamGetCaptureInfo(s, &status, &id) == cudaSuccess;
    if (!known) cudaGetLastError();  // the legacy stream beside a capture: launches on it are refused
    *plain = known && status == cudaStreamCaptureStatusNone;
    return known && status == cudaStreamCaptureStatusActive ? id : 0;
}

bool mark_changed(vrt_world* w, cudaStream_t s) {
    static std::atomic<uint64_t> next{1};
    bool plain = false;
    if (capture_of(s, &plain)) w->in_graph = true;
    w->stamp = w->in_graph ? 0 : next++;
    return plain && !w->in_graph;
}

// Whether stream s may read a derived structure as it is: the last rebuild that its launches see is
// waited for.  fresh: the plain launches' one is up to date, as far as the host knows.
static int see_derived(const vrt_world* w, const Derived& d, bool fresh, unsigned long long capture, cudaStream_t s,
                       bool* seen) {
    const bool here = capture && d.capture == capture;
    *seen = here || (fresh && !w->in_graph);
    if (here) VRT_CUDA(cudaStreamWaitEvent(s, d.captured, 0));
    // the last rebuild, on whichever stream; in_graph: another one follows, which writes the same arrays
    else if (d.ready && (*seen || (w->in_graph && !capture))) VRT_CUDA(cudaStreamWaitEvent(s, d.ready, 0));
    return VRT_OK;
}

// Note a rebuild that was launched on stream s.
static int derived_now(Derived& d, unsigned long long capture, cudaStream_t s) {
    if (!capture) {
        VRT_CUDA(cudaEventRecord(d.ready, s));
        return VRT_OK;
    }
    VRT_CUDA(cudaEventRecord(d.captured, s));
    d.capture = capture;
    return VRT_OK;
}

static cudaError_t make_events(Derived& d) {
    cudaError_t e = cudaEventCreateWithFlags(&d.ready, cudaEventDisableTiming);
    if (e == cudaSuccess) e = cudaEventCreateWithFlags(&d.captured, cudaEventDisableTiming);
    return e;
}

static void destroy_events(Derived& d) {
    if (d.ready) cudaEventDestroy(d.ready);
    if (d.captured) cudaEventDestroy(d.captured);
    d = Derived{};
}

int refresh_stop(vrt_world* w, cudaStream_t s) {
    bool plain = false, seen = false;
    const unsigned long long capture = capture_of(s, &plain);
    int st = see_derived(w, w->stop, !w->stop_stale, capture, s, &seen);
    if (st || seen) return st;
    const Layout& L = w->L;
    const bool behind = !capture && mark_changed(w, s);
    if (!w->d_stop) {
        cudaError_t e = cudaMalloc(&w->d_stop, L.n_bricks * 8);
        if (e == cudaSuccess) e = cudaMalloc(&w->d_sdir, L.n_bricks * 8);
        if (e == cudaSuccess) e = cudaMalloc(&w->d_stop_regions, L.n_regions * 8);
        if (e == cudaSuccess) e = make_events(w->stop);
        if (e != cudaSuccess) {
            cudaGetLastError();
            cudaFree(w->d_stop);
            cudaFree(w->d_sdir);
            cudaFree(w->d_stop_regions);
            destroy_events(w->stop);
            w->d_stop = nullptr;
            w->d_sdir = nullptr;
            w->d_stop_regions = nullptr;
            return set_error(VRT_ENOMEM, "stop masks: %s", cudaGetErrorString(e));
        }
        w->device_bytes += L.n_bricks * 16 + L.n_regions * 8;
    }
    if (!w->stop_cleared) {
        VRT_CUDA(cudaMemsetAsync(w->d_stop, 0, L.n_bricks * 8, s));
        VRT_CUDA(cudaMemsetAsync(w->d_stop_regions, 0, L.n_regions * 8, s));
    }
    st = refresh_stop_masks(w, s, behind);
    if (!st) st = derived_now(w->stop, capture, s);
    if (st || capture) return st;
    w->stop_cleared = true;
    w->stop_stale = false;
    return VRT_OK;
}

void mark_words(vrt_world* w, const int64_t v[6], bool z_copy) {
    const int dim[3] = {w->L.W, w->L.H, w->L.W};
    int lo[3], hi[3];
    for (int a = 0; a < 3; a++) {
        const int64_t l = std::max<int64_t>(v[a], 0), h = std::min<int64_t>(v[3 + a], dim[a]);
        if (l >= h) return;
        lo[a] = (int)l;
        hi[a] = (int)h;
    }
    w->stop_stale = true;
    w->stop.capture = 0;
    if (!z_copy || !w->d_words_z) return;
    w->z.capture = 0;
    int* b = w->z_dirty;
    const bool empty = b[0] >= b[3];
    for (int a = 0; a < 3; a++) {
        b[a] = empty ? lo[a] : std::min(b[a], lo[a]);
        b[3 + a] = empty ? hi[a] : std::max(b[3 + a], hi[a]);
    }
}

// Whole-world copy with x and z swapped, through 64x64 tiles of the (x, z) plane of each y
// so that both the reads (along x) and the writes (along z) are whole lines.  All 16 loads
// of a thread are in flight before the first is needed: 512 x 96 x 512 words in 30 us (6.6
// TB/s of reads and writes), 70 us with 32x32 tiles and four loads in a loop.
__global__ void __launch_bounds__(256) words_z_transpose_kernel(const int32_t* __restrict__ in,
                                                                 int32_t* __restrict__ out, Layout L) {
    __shared__ int32_t tile[64][65];
    const uint64_t W = L.W, WH = (uint64_t)L.W * L.H;
    const int y = blockIdx.z, x0 = blockIdx.x * 64, z0 = blockIdx.y * 64;
    const int i = threadIdx.x & 63, j = threadIdx.x >> 6;
    int32_t v[16];
#pragma unroll
    for (int k = 0; k < 16; k++) {  // read: x along the threads
        const int x = x0 + i, z = z0 + j + 4 * k;
        v[k] = x < L.W && z < L.W ? in[x + W * y + WH * z] : 0;
    }
#pragma unroll
    for (int k = 0; k < 16; k++) tile[j + 4 * k][i] = v[k];
    __syncthreads();
#pragma unroll
    for (int k = 0; k < 16; k++) {  // write: z along the threads
        const int z = z0 + i, x = x0 + j + 4 * k;
        if (x < L.W && z < L.W) out[z + W * y + WH * x] = tile[i][j + 4 * k];
    }
}

// The same for the words of one box (edit-sized), one thread per word.
__global__ void words_z_box_kernel(const int32_t* __restrict__ in, int32_t* __restrict__ out, Layout L, int x0,
                                   int y0, int z0, int nx, int ny, int nz) {
    const uint64_t t = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= (uint64_t)nx * ny * nz) return;
    const uint64_t W = L.W, WH = (uint64_t)L.W * L.H;
    const uint64_t x = x0 + t % nx, y = y0 + (t / nx) % ny, z = z0 + t / ((uint64_t)nx * ny);
    out[z + W * y + WH * x] = in[x + W * y + WH * z];
}

int refresh_words_z(vrt_world* w, cudaStream_t s) {
    const Layout& L = w->L;
    int* b = w->z_dirty;
    bool plain = false, seen = false;
    const unsigned long long capture = capture_of(s, &plain);
    const int st = see_derived(w, w->z, w->z_filled && b[0] >= b[3], capture, s, &seen);
    if (st || seen) return st;
    if (!capture) mark_changed(w, s);
    if (!w->d_words_z) {
        cudaError_t e = cudaMalloc(&w->d_words_z, L.n_words * sizeof(int32_t));
        if (e == cudaSuccess) e = make_events(w->z);
        if (e != cudaSuccess) {
            cudaGetLastError();
            cudaFree(w->d_words_z);
            destroy_events(w->z);
            w->d_words_z = nullptr;
            return set_error(VRT_ENOMEM, "z-major words: %s", cudaGetErrorString(e));
        }
        w->device_bytes += L.n_words * sizeof(int32_t);
    }
    if (!w->z_filled || w->in_graph || capture) {  // a graph's run may follow changes outside the box
        dim3 grid((L.W + 63) / 64, (L.W + 63) / 64, L.H);
        words_z_transpose_kernel<<<grid, 256, 0, s>>>(w->d_words, w->d_words_z, L);
    } else {
        const uint64_t n = (uint64_t)(b[3] - b[0]) * (b[4] - b[1]) * (b[5] - b[2]);
        words_z_box_kernel<<<blocks_for(n, 256), 256, 0, s>>>(w->d_words, w->d_words_z, L, b[0], b[1], b[2],
                                                               b[3] - b[0], b[4] - b[1], b[5] - b[2]);
    }
    VRT_CUDA(cudaGetLastError());
    const int noted = derived_now(w->z, capture, s);
    if (noted || capture) return noted;
    w->z_filled = true;
    b[0] = b[3] = 0;
    return VRT_OK;
}

// The box of the words [first, first + count): planes, rows or part of a row.
static void words_box(const Layout& L, uint64_t first, uint64_t count, int64_t v[6]) {
    const uint64_t last = first + count - 1, plane = (uint64_t)L.W * L.H;
    const int64_t z0 = first / plane, z1 = last / plane;
    const int64_t y0 = first % plane / L.W, y1 = last % plane / L.W;
    const int64_t x0 = first % L.W, x1 = last % L.W;
    const bool rows = z0 != z1, cells = !rows && y0 == y1;
    v[0] = cells ? x0 : 0;
    v[1] = rows ? 0 : y0;
    v[2] = z0;
    v[3] = cells ? x1 + 1 : L.W;
    v[4] = rows ? L.H : y1 + 1;
    v[5] = z1 + 1;
}

static WordChange whole_world(const Layout& L) {
    WordChange c{};
    c.op = kReadWords;
    c.box[3] = L.W; c.box[4] = L.H; c.box[5] = L.W;
    return c;
}

// Copy the solid bounding box and the depth-field flag to the host copies the render
// launches go by (synchronises the stream).
static int read_state(vrt_world* w, int& flag, cudaStream_t s) {
    int st[8];
    VRT_CUDA(cudaMemcpyAsync(st, w->d_aabb, sizeof(st), cudaMemcpyDeviceToHost, s));
    VRT_CUDA(cudaStreamSynchronize(s));
    for (int i = 0; i < 3; i++) {
        w->h_aabb[i] = std::min(st[i], w->graph_box[i]);
        w->h_aabb[3 + i] = std::max(st[3 + i], w->graph_box[3 + i]);
    }
    flag = st[6] | w->graph_depth;
    return VRT_OK;
}

// A change that was launched brings depth-field words (depth), or solid voxels within the box [lo, hi]:
// the host copies of the flag and the solid box hold them from now on, and for a world that captured
// graphs change, whose runs may bring them at any time, past the next look at the words as well.
static void note_added(vrt_world* w, bool depth, const int* lo, const int* hi) {
    if (depth) {
        w->has_depth_field = 1;
        if (w->in_graph) w->graph_depth = 1;
    }
    for (int i = 0; lo && i < 3; i++) {
        for (int* box : {w->h_aabb, w->in_graph ? w->graph_box : w->h_aabb}) {
            box[i] = std::min(box[i], lo[i]);
            box[3 + i] = std::max(box[3 + i], hi[i]);
        }
    }
}

// Reads that a kernel ahead may have written, behind the wait: no __restrict__, which would let
// them go through the read-only path.
__global__ void probe_kernel(const int32_t* words, Layout L, const int32_t* xyz, int n, int32_t* out) {
    cudaTriggerProgrammaticLaunchCompletion();
    cudaGridDependencySynchronize();
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const int x = xyz[3 * i], y = xyz[3 * i + 1], z = xyz[3 * i + 2];
    const bool in = x >= 0 && y >= 0 && z >= 0 && x < L.W && y < L.H && z < L.W;
    out[i] = in ? words[(uint64_t)x + (uint64_t)L.W * y + (uint64_t)L.W * L.H * z] : -1;
}

}  // namespace vrt

using namespace vrt;

static inline cudaStream_t S(void* s) { return reinterpret_cast<cudaStream_t>(s); }

extern "C" {

int vrt_world_create(int32_t width, int32_t height, vrt_world** out) {
    if (!out) return set_error(VRT_EINVAL, "out is NULL");
    *out = nullptr;
    if (width < 1 || height < 1 || width > 65536 || height > 65536)
        return set_error(VRT_EINVAL, "world %d x %d x %d out of range", width, height, width);
    uint64_t n = (uint64_t)width * height * width;
    if (n > (1ull << 31)) return set_error(VRT_ERANGE, "world of %llu voxels exceeds 2^31", (unsigned long long)n);
    const Layout L = make_layout(width, height);
    if (L.n_bricks * 8 >= (1ull << 32))  // the render kernels index bricks in 32 bits
        return set_error(VRT_ERANGE, "world %d x %d x %d: brick grid too large", width, height, width);
    vrt_world* w = new vrt_world();
    w->L = L;
    cudaGetDevice(&w->device);
    cudaDeviceGetAttribute(&w->num_sms, cudaDevAttrMultiProcessorCount, w->device);
    int pages = 0, tables = 0;
    cudaDeviceGetAttribute(&pages, cudaDevAttrPageableMemoryAccess, w->device);
    cudaDeviceGetAttribute(&tables, cudaDevAttrPageableMemoryAccessUsesHostPageTables, w->device);
    w->reads_pageable = pages && tables;
    const uint64_t box_bytes = (uint64_t)w->num_sms * kBrickCtasPerSm * 8 * sizeof(int);
    uint64_t bytes = w->L.n_words * 4 + (w->L.n_bricks + w->L.n_regions + w->L.n_supers) * 8 + 8 * w->L.n_bricks +
                     (uint64_t)w->L.RWp * w->L.RHp * w->L.RWp + box_bytes + 256;
    cudaError_t e = cudaMalloc(&w->d_words, w->L.n_words * 4);
    if (e == cudaSuccess) e = cudaMalloc(&w->d_bricks, w->L.n_bricks * 8);
    if (e == cudaSuccess) e = cudaMalloc(&w->d_regions, w->L.n_regions * 8);
    if (e == cudaSuccess) e = cudaMalloc(&w->d_supers, w->L.n_supers * 8);
    const uint64_t rbytes = ((uint64_t)w->L.RWp * w->L.RHp * w->L.RWp + 15) & ~(uint64_t)15;  // staged as uint4
    if (e == cudaSuccess) e = cudaMalloc(&w->d_rdist, rbytes);
    if (e == cudaSuccess) e = cudaMalloc(&w->d_bdir, w->L.n_bricks * 8);
    if (e == cudaSuccess) e = cudaMalloc(&w->d_boxes, box_bytes);
    if (e == cudaSuccess) e = cudaMalloc(&w->d_aabb, 8 * sizeof(int));
    if (e == cudaSuccess) e = cudaMemset(w->d_words, 0xFF, w->L.n_words * 4);  // air = -1 (render.cpp:349-351)
    if (e == cudaSuccess) e = cudaMemset(w->d_bricks, 0, w->L.n_bricks * 8);
    if (e == cudaSuccess) e = cudaMemset(w->d_regions, 0, w->L.n_regions * 8);
    if (e == cudaSuccess) e = cudaMemset(w->d_supers, 0, w->L.n_supers * 8);
    if (e == cudaSuccess) e = cudaMemset(w->d_bdir, dist_code(kDistCap), w->L.n_bricks * 8);  // an all-air world
    if (e == cudaSuccess) e = cudaMemset(w->d_rdist, kDistCap, rbytes);
    if (e == cudaSuccess) {  // an all-air world: empty box (min > max), no depth-field word
        const int empty[8] = {INT_MAX, INT_MAX, INT_MAX, INT_MIN, INT_MIN, INT_MIN, 0, 0};
        e = cudaMemcpy(w->d_aabb, empty, sizeof(empty), cudaMemcpyHostToDevice);
        for (int i = 0; i < 6; i++) w->h_aabb[i] = empty[i];
    }
    if (e == cudaSuccess) e = cudaDeviceSynchronize();
    if (e != cudaSuccess) {
        cudaGetLastError();
        vrt_world_destroy(w);
        return e == cudaErrorMemoryAllocation ? set_error(VRT_ENOMEM, "world allocation: %s", cudaGetErrorString(e))
                                              : cuda_error(e, "vrt_world_create");
    }
    w->device_bytes = bytes;
    mark_changed(w, nullptr);
    *out = w;
    return VRT_OK;
}

int vrt_world_destroy(vrt_world* w) {
    if (!w) return VRT_OK;
    cudaFree(w->d_words);
    cudaFree(w->d_bricks);
    cudaFree(w->d_regions);
    cudaFree(w->d_supers);
    cudaFree(w->d_rdist);
    cudaFree(w->d_bdir);
    cudaFree(w->d_stop);
    cudaFree(w->d_sdir);
    destroy_events(w->stop);
    cudaFree(w->d_words_z);
    destroy_events(w->z);
    cudaFree(w->d_stop_regions);
    cudaFree(w->d_boxes);
    cudaFree(w->d_aabb);
    delete w;
    return VRT_OK;
}

int vrt_world_get_info(const vrt_world* w, vrt_world_info* out) {
    if (!w || !out) return set_error(VRT_EINVAL, "NULL argument");
    out->width = w->L.W;
    out->height = w->L.H;
    out->num_words = w->L.n_words;
    out->d_words = w->d_words;
    out->d_brick_mask = w->d_bricks;
    out->d_region_mask = w->d_regions;
    out->has_depth_field = w->has_depth_field;
    out->device_bytes = w->device_bytes;
    return VRT_OK;
}

static int upload_common(vrt_world* w, const int32_t* src, uint64_t first, uint64_t count, void* stream,
                         cudaMemcpyKind kind) {
    if (!w || (!src && count)) return set_error(VRT_EINVAL, "NULL argument");
    if (first > w->L.n_words || count > w->L.n_words - first)
        return set_error(VRT_ERANGE, "words [%llu, %llu) beyond the world's %llu", (unsigned long long)first,
                         (unsigned long long)(first + count), (unsigned long long)w->L.n_words);
    if (count == 0) return VRT_OK;
    WordChange c{};
    words_box(w->L, first, count, c.box);
    cudaPointerAttributes at{};
    if (cudaPointerGetAttributes(&at, src) != cudaSuccess) {
        (void)cudaGetLastError();  // not a pointer the runtime knows
        at.type = cudaMemoryTypeUnregistered;
    }
    const int32_t* seen = upload_view(src, kind == cudaMemcpyHostToDevice, at, w->device, w->reads_pageable);
    if (seen) {  // copied by the pass that makes the masks
        c.op = kCopyWords;
        c.src = seen;
        c.first = first;
        c.count = count;
    } else {
        c.op = kReadWords;
        VRT_CUDA(cudaMemcpyAsync(w->d_words + first, src, count * 4, kind, S(stream)));
    }
    int flag = 0, st = change_words(w, c, S(stream));
    // the kernel choice depends on the depth-field flag: read it back now
    if (!st) st = read_state(w, flag, S(stream));
    if (st) {
        if (seen) cudaStreamSynchronize(S(stream));  // the caller's memory has no reader after the return
        return st;
    }
    w->has_depth_field |= flag;
    return VRT_OK;
}

int vrt_world_upload(vrt_world* w, const int32_t* host_words, uint64_t first, uint64_t count, void* stream) {
    return upload_common(w, host_words, first, count, stream, cudaMemcpyHostToDevice);
}

int vrt_world_upload_device(vrt_world* w, const int32_t* d_words, uint64_t first, uint64_t count, void* stream) {
    return upload_common(w, d_words, first, count, stream, cudaMemcpyDeviceToDevice);
}

int vrt_world_download(const vrt_world* w, int32_t* host_words, uint64_t first, uint64_t count, void* stream) {
    if (!w || (!host_words && count)) return set_error(VRT_EINVAL, "NULL argument");
    if (first > w->L.n_words || count > w->L.n_words - first) return set_error(VRT_ERANGE, "range beyond the world");
    if (count == 0) return VRT_OK;
    VRT_CUDA(cudaMemcpyAsync(host_words, w->d_words + first, count * 4, cudaMemcpyDeviceToHost, S(stream)));
    VRT_CUDA(cudaStreamSynchronize(S(stream)));
    return VRT_OK;
}

int vrt_world_download_masks(const vrt_world* w, uint64_t* bricks, uint64_t* regions, uint64_t* supers,
                             void* stream) {
    if (!w) return set_error(VRT_EINVAL, "NULL world");
    if (bricks)
        VRT_CUDA(cudaMemcpyAsync(bricks, w->d_bricks, w->L.n_bricks * 8, cudaMemcpyDeviceToHost, S(stream)));
    if (regions)
        VRT_CUDA(cudaMemcpyAsync(regions, w->d_regions, w->L.n_regions * 8, cudaMemcpyDeviceToHost, S(stream)));
    if (supers)
        VRT_CUDA(cudaMemcpyAsync(supers, w->d_supers, w->L.n_supers * 8, cudaMemcpyDeviceToHost, S(stream)));
    VRT_CUDA(cudaStreamSynchronize(S(stream)));
    return VRT_OK;
}

int vrt_world_download_distances(const vrt_world* w, uint8_t* brick_dir, uint8_t* region_dist, void* stream) {
    if (!w) return set_error(VRT_EINVAL, "NULL world");
    std::vector<uint64_t> masks;  // the stored codes are 0 for distances 0 and 1: the masks tell them apart
    if (brick_dir) {
        masks.resize(w->L.n_bricks);
        VRT_CUDA(cudaMemcpyAsync(brick_dir, w->d_bdir, w->L.n_bricks * 8, cudaMemcpyDeviceToHost, S(stream)));
        VRT_CUDA(cudaMemcpyAsync(masks.data(), w->d_bricks, w->L.n_bricks * 8, cudaMemcpyDeviceToHost, S(stream)));
    }
    if (region_dist)
        VRT_CUDA(cudaMemcpyAsync(region_dist, w->d_rdist, (uint64_t)w->L.RWp * w->L.RHp * w->L.RWp,
                                 cudaMemcpyDeviceToHost, S(stream)));
    VRT_CUDA(cudaStreamSynchronize(S(stream)));
    for (size_t i = 0; i < masks.size(); i++)
        for (int o = 0; o < 8; o++) brick_dir[8 * i + o] = masks[i] ? 0 : (uint8_t)(brick_dir[8 * i + o] / 4 + 1);
    return VRT_OK;
}

// The brick pass raises the flag whenever it sees a word < -1 and never lowers it; a pass
// over the whole world that starts it from 0 gives the exact current state.
int vrt_world_sync_flags(vrt_world* w, void* stream) {
    if (!w) return set_error(VRT_EINVAL, "NULL world");
    WordChange c = whole_world(w->L);
    c.reset_flag = true;
    int st = change_words(w, c, S(stream));
    if (st) return st;
    int flag = 0;
    st = read_state(w, flag, S(stream));
    if (st) return st;
    w->has_depth_field = flag;
    return VRT_OK;
}

int vrt_world_probe(const vrt_world* w, const int32_t* d_xyz, int32_t n, int32_t* d_words, void* stream) {
    if (!w || n < 0 || (n > 0 && (!d_xyz || !d_words))) return set_error(VRT_EINVAL, "bad probe arguments");
    if (n == 0) return VRT_OK;
    bool plain = false;
    capture_of(S(stream), &plain);
    VRT_CUDA(launch_behind(plain, probe_kernel, dim3(blocks_for((uint64_t)n, 256)), 256, S(stream),
                           (const int32_t*)w->d_words, w->L, d_xyz, (int)n, d_words));
    return VRT_OK;
}

static const int32_t kWorldMagic = 0x57525456;  // "VRTW" little-endian

int vrt_world_save(const vrt_world* w, const char* path, void* stream) {
    if (!w || !path) return set_error(VRT_EINVAL, "NULL argument");
    std::vector<int32_t> host(w->L.n_words);
    int st = vrt_world_download(w, host.data(), 0, w->L.n_words, stream);
    if (st) return st;
    FILE* f = std::fopen(path, "wb");
    if (!f) return set_error(VRT_EINVAL, "cannot open %s for writing", path);
    const int32_t head[4] = {kWorldMagic, 1, w->L.W, w->L.H};
    bool ok = std::fwrite(head, sizeof(head), 1, f) == 1 &&
              std::fwrite(host.data(), sizeof(int32_t), host.size(), f) == host.size();
    ok = (std::fclose(f) == 0) && ok;
    return ok ? VRT_OK : set_error(VRT_EINVAL, "short write to %s", path);
}

int vrt_world_load(const char* path, vrt_world** out, void* stream) {
    if (!path || !out) return set_error(VRT_EINVAL, "NULL argument");
    *out = nullptr;
    FILE* f = std::fopen(path, "rb");
    if (!f) return set_error(VRT_EINVAL, "cannot open %s", path);
    int32_t head[4] = {0, 0, 0, 0};
    if (std::fread(head, sizeof(head), 1, f) != 1 || head[0] != kWorldMagic || head[1] != 1) {
        std::fclose(f);
        return set_error(VRT_EINVAL, "%s is not a version-1 world file", path);
    }
    vrt_world* w = nullptr;
    int st = vrt_world_create(head[2], head[3], &w);
    if (st) {
        std::fclose(f);
        return st;
    }
    std::vector<int32_t> host(w->L.n_words);
    const bool ok = std::fread(host.data(), sizeof(int32_t), host.size(), f) == host.size();
    std::fclose(f);
    if (!ok) {
        vrt_world_destroy(w);
        return set_error(VRT_EINVAL, "%s is truncated", path);
    }
    st = vrt_world_upload(w, host.data(), 0, host.size(), stream);
    if (st) {
        vrt_world_destroy(w);
        return st;
    }
    *out = w;
    return VRT_OK;
}

int vrt_place_voxel(vrt_world* w, int32_t x, int32_t y, int32_t z, int32_t word, void* stream) {
    if (!w) return set_error(VRT_EINVAL, "NULL world");
    if (x < 0 || y < 0 || z < 0 || x >= w->L.W || y >= w->L.H || z >= w->L.W) return VRT_OK;  // render.cpp:259
    WordChange ch{};
    ch.op = kPlaceVoxel;
    ch.x = x; ch.y = y; ch.z = z; ch.word = word;
    const int64_t box[6] = {x, y, z, x + 1, y + 1, z + 1};
    std::memcpy(ch.box, box, sizeof(box));
    const int st = change_words(w, ch, S(stream));
    if (st) return st;
    const int lo[3] = {x & ~3, y & ~3, z & ~3}, hi[3] = {lo[0] + 3, lo[1] + 3, lo[2] + 3};  // its brick
    note_added(w, word < -1, word >= 0 ? lo : nullptr, hi);
    return VRT_OK;
}

int vrt_fix_depth_field_box(vrt_world* w, int32_t x0, int32_t y0, int32_t z0, int32_t x1, int32_t y1, int32_t z1,
                            void* stream) {
    if (!w) return set_error(VRT_EINVAL, "NULL world");
    // the depth field changes air words only, so the occupancy structures stay as they are
    WordChange c{};
    const int64_t box[6] = {x0, y0, z0, x1, y1, z1};
    std::memcpy(c.fix_box, box, sizeof(box));
    c.fix = true;
    const int dim[3] = {w->L.W, w->L.H, w->L.W};
    for (int a = 0; a < 3; a++)
        if (std::max<int64_t>(box[a], 0) >= std::min<int64_t>(box[3 + a], dim[a])) return VRT_OK;
    const int st = change_words(w, c, S(stream));
    note_added(w, true, nullptr, nullptr);
    return st;
}

int vrt_remove_sphere(vrt_world* w, int32_t cx, int32_t cy, int32_t cz, int32_t radius, int32_t refresh_depth_field,
                      void* stream) {
    if (!w) return set_error(VRT_EINVAL, "NULL world");
    if (radius < 0 || radius > 1024) return set_error(VRT_ERANGE, "radius %d outside [0, 1024]", radius);
    const int64_t at[3] = {cx, cy, cz};
    WordChange c{};
    c.op = kRemoveSphere;
    c.x = cx; c.y = cy; c.z = cz; c.r = radius;
    for (int a = 0; a < 3; a++) {
        c.box[a] = at[a] - radius;
        c.box[3 + a] = at[a] + radius;
    }
    if (refresh_depth_field) {
        c.fix = true;
        c.fix_r = radius + (7 >> 1);  // DEPTH_FIELD_RADIUS >> 1, level.cpp:43
        for (int a = 0; a < 3; a++) {
            c.fix_box[a] = at[a] - c.fix_r;
            c.fix_box[3 + a] = at[a] + c.fix_r;
        }
    }
    const int st = change_words(w, c, S(stream));
    note_added(w, c.fix, nullptr, nullptr);
    return st;
}

int vrt_world_init_reference(vrt_world* w, void* stream) {
    if (!w) return set_error(VRT_EINVAL, "NULL world");
    WordChange c = whole_world(w->L);
    c.op = kInitLevel;
    c.reset_flag = true;
    w->has_depth_field = w->graph_depth;
    int flag = 0;
    int st = change_words(w, c, S(stream));
    if (st) return st;
    return read_state(w, flag, S(stream));
}

}  // extern "C"
