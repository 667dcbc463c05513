// Render kernels: the per-pixel path of Berry2460/voxel-rt src/fshader.glsl.
//
// render_word_kernel  one thread per pixel; every DDA step reads the 4-byte voxel word,
//                     follows depth-field jumps (fshader.glsl:114-121).  Exact on every
//                     world, including worlds built by fixDepthField.  Steps along z read
//                     a z-major copy of the words; tiles run heaviest first by the last
//                     frame's costs.
// render_mask_kernel  persistent warps over ray tiles; traversal reads the 64-ary
//                     occupancy hierarchy (64^3 -> 16^3 -> 4^3 -> voxel, one uint64
//                     per node) and keeps the current brick's 64 voxel bits in
//                     registers, so a step inside a known box touches no memory; the
//                     colour word is fetched once, at the primary hit.  Lanes whose ray
//                     ends are refilled (next shadow ray of their pixel, or a new
//                     pixel from the warp's tile queue) together, once refill_min lanes
//                     are idle, which keeps the warp's lanes busy although ray lengths
//                     vary from 1 to thousands of steps.
// Both perform every per-cell floating-point add of the shader in its order, so hit
// voxels, step counts and shadow bits are those of the CPU oracle bit for bit.
#include <cuda_runtime.h>

#include <algorithm>
#include <climits>
#include <cstring>
#include <mutex>
#include <vector>

#include "shade_common.cuh"
#include "vrt_internal.h"

namespace vrt {

// The pixels of an image's tiles, without integer divisions: 80 of the instructions that each
// warp spent before its first ray.  A quotient by a constant n is a multiplication by
// ceil(2^k / n), exact for the few bits of a thread's index, and at most 1 too large for a
// tile's (tiles < 2^32: the error is below tile / 2^32).
struct TileMap {
    int tw, th;        // pixels of a tile, one thread each (tw * th <= 128)
    int tiles_x;       // tiles in a row of the image
    uint32_t tw_mul;   // ceil(2^16 / tw)
    uint32_t row_mul;  // ceil(2^32 / tiles_x), or 0 for tiles_x = 1
    float inv_w, inv_h;  // 1 / width and 1 / height, rounded to nearest: primary_dir's divisions
    __device__ __forceinline__ void pixel(int tile, int thread, int& px, int& py) const {
        int row = row_mul ? (int)__umulhi((uint32_t)tile, row_mul) : tile;
        int col = tile - row * tiles_x;
        if (col < 0) {
            row--;
            col += tiles_x;
        }
        const int ty = (int)((uint32_t)thread * tw_mul >> 16);
        px = col * tw + (thread - ty * tw);
        py = row * th + ty;
    }
};
static TileMap tile_map(int width, int height, int tw, int th) {
    TileMap m;
    m.tw = tw;
    m.th = th;
    m.tiles_x = (width + tw - 1) / tw;
    m.tw_mul = (65536u + tw - 1) / tw;
    m.row_mul = m.tiles_x == 1 ? 0 : (uint32_t)(((1ull << 32) + m.tiles_x - 1) / m.tiles_x);
    m.inv_w = 1.0f / (float)width;
    m.inv_h = 1.0f / (float)height;
    return m;
}

// ====================================================================== word kernel

struct WordParams {
    vrt_uniforms u;
    int width, height;
    uint8_t* rgba;
    vrt_debug_out dbg;
    unsigned long long* stats;
    int bb[6];   // solid bounding box: min x,y,z, max x,y,z (never smaller than the truth)
    int exact;   // 1: every DDA iteration of the shader runs (step counts asked for)
    TileMap map;  // pixel tiles of a CTA each
    const int32_t* words;    // x + W*y + W*H*z
    const int32_t* words_z;  // the same words with x and z swapped: z + W*y + W*H*x
    // The tile order (see tile_class): the last frame's tiles by cost class, or NULL (CTA
    // (x, y) renders tile (x, y)); this frame's classes, appended to; the counts zeroed for
    // the frame after.
    const int* class_count_in;
    const int* class_list_in;
    int* class_count_out;
    int* class_list_out;
    int* class_count_clear;
    int tiles;
    int wait_first;  // 1: the kernel ahead may be changing the words (see frame_launch)
};

// The word kernel's tile order.  The frame's length is set by its heaviest tiles: on the
// reference scene the tiles along the horizon, whose pixels all run 80-170 iterations of
// depth-field jumps and steps, hold about 90 % of the frame's instructions, and each
// such CTA runs a latency-bound chain for tens of microseconds.  Launched in row order
// they start a quarter of the way into the frame and end it.  So each CTA, when it ends,
// appends its tile to the list of its cost class (its slowest pixel's DDA iterations, in
// half octaves), and the next frame of the same grid launches the tiles class by class,
// heaviest first.  A tile's pixels are computed the same way wherever it runs, so the
// order changes no result, only when each tile runs.  No kernel or host work is added:
// the lists are written and read by the render kernels themselves.
constexpr int kTileClasses = 16;
constexpr int kClassReuses = 31;  // overlapped frames that may go by one frame's classes

// Costs 0-7 -> class 0, 8-11 -> 1, 12-15 -> 2, 16-23 -> 3, ..., 768-1023 -> 14, >= 1024 -> 15.
__device__ __forceinline__ int tile_class(int cost) {
    if (cost < 8) return 0;
    const int e = 31 - __clz(cost);  // 2^e <= cost < 2^(e+1), e >= 3
    return min(kTileClasses - 1, 2 * (e - 3) + ((cost >> (e - 1)) & 1) + 1);
}

// fl(i / 255) for i = 0..255: the shader's channel scale (fshader.glsl:184-186), filled on
// each device by init_div255_kernel with the same IEEE division, so a table read gives
// the quotient bit for bit.
__device__ float g_div255[256];

__global__ void init_div255_kernel() { g_div255[threadIdx.x] = fdiv((float)threadIdx.x, 255.0f); }

// pack_color of the tile kernel: the channel quotients come from g_div255.
__device__ __forceinline__ uint32_t pack_color_tab(const vrt_uniforms& u, bool hit, int32_t word, float mr,
                                                   float mg, float mb, int primary_steps) {
    float c0, c1, c2;
    if (u.viewDepthField == 1) {
        c0 = c1 = c2 = fdiv((float)primary_steps, 100.0f);
    } else if (hit) {
        c0 = fmul(__ldg(g_div255 + ((word & 0x00FF0000) >> 16)), mr);
        c1 = fmul(__ldg(g_div255 + ((word & 0x0000FF00) >> 8)), mg);
        c2 = fmul(__ldg(g_div255 + (word & 0x000000FF)), mb);
    } else {
        c0 = 0.6f; c1 = 0.7f; c2 = 0.8f;
    }
    return to_u8(c0) | (to_u8(c1) << 8) | (to_u8(c2) << 16) | (to_u8(1.0f) << 24);
}

// The local lights that may be in range of some lane of the warp, as a warp-uniform bit
// mask: lane l < 16 tests light l's cube of half-size R1 + 1 against the integer
// bounding box of the warp's hit points (every lane must call this).  A light a lane
// would accept (every |L - hitPos| component within R1, fshader.glsl:168-171 with the
// pre-reject above) lies within that box grown by R1 + 1, so no candidate is lost; an
// inactive light (a coordinate < 0, :167) never is one.
__device__ __forceinline__ unsigned warp_light_candidates(const vrt_uniforms& u, bool lit, V3 hp) {
    const unsigned full = 0xffffffffu;
    if (!__any_sync(full, lit)) return 0;  // a warp of sky
    const int x0 = __reduce_min_sync(full, lit ? (int)floorf(hp.x) : INT_MAX);
    const int y0 = __reduce_min_sync(full, lit ? (int)floorf(hp.y) : INT_MAX);
    const int z0 = __reduce_min_sync(full, lit ? (int)floorf(hp.z) : INT_MAX);
    const int x1 = __reduce_max_sync(full, lit ? (int)floorf(hp.x) + 1 : INT_MIN);
    const int y1 = __reduce_max_sync(full, lit ? (int)floorf(hp.y) + 1 : INT_MIN);
    const int z1 = __reduce_max_sync(full, lit ? (int)floorf(hp.z) + 1 : INT_MIN);
    const int lane = threadIdx.x & 31;
    bool c = false;
    if (x0 != INT_MAX && lane < VRT_MAX_LOCAL_LIGHTS) {
        const float* L = u.localLights[lane];
        if (L[0] >= 0 && L[1] >= 0 && L[2] >= 0) {
            const float g = fabsf(u.localLightDist) * 1.0009765625f + 2.0f;
            c = L[0] + g >= (float)x0 && L[0] - g <= (float)x1 && L[1] + g >= (float)y0 && L[1] - g <= (float)y1 &&
                L[2] + g >= (float)z0 && L[2] - g <= (float)z1;
        }
    }
    return __ballot_sync(full, c);
}

// t = t + d (round to nearest) where p holds, else t unchanged: one predicated PTX add,
// which the compiler cannot turn into a branch or a select.
__device__ __forceinline__ void pred_fadd(float& t, float d, bool p) {
    asm("{.reg .pred q; setp.ne.b32 q, %1, 0; @q add.rn.f32 %0, %0, %2;}" : "+f"(t) : "r"((int)p), "f"(d));
}

// The cell of a position and its intersects, fshader.glsl:69-79 and :117-120:
// t = (float(cell + (s > 0)) - start) / dir.  inv = frcp of dir's components; fast: they lie
// in div_by's range, and the ray's first start is no NaN (a jump's NaN shows in every component).
__device__ __forceinline__ void enter_cell(RaySetup& r, V3 start, V3 dir, V3 inv, bool fast) {
    if (fast && fminf(fminf(start.x, start.y), start.z) >= kDivMinA &&
        fmaxf(fmaxf(start.x, start.y), start.z) < 4194304.0f) {
        // int(x) and float(int(x)) of 0 <= x < 2^22 from x + 2^23 rounded toward zero, on
        // the FMA pipe instead of six conversions at an eighth of its rate
        const float mx = __fadd_rz(start.x, 8388608.0f), my = __fadd_rz(start.y, 8388608.0f),
                    mz = __fadd_rz(start.z, 8388608.0f);
        r.cx = __float_as_int(mx) - 0x4B000000;
        r.cy = __float_as_int(my) - 0x4B000000;
        r.cz = __float_as_int(mz) - 0x4B000000;
        // the next cell's bound: (mx - 2^23) + 1 or + 0 is mx - (2^23 - 1) or mx - 2^23, both exact
        r.tx = div_by(fsub(fsub(mx, r.sx > 0 ? 8388607.0f : 8388608.0f), start.x), dir.x, inv.x);
        r.ty = div_by(fsub(fsub(my, r.sy > 0 ? 8388607.0f : 8388608.0f), start.y), dir.y, inv.y);
        r.tz = div_by(fsub(fsub(mz, r.sz > 0 ? 8388607.0f : 8388608.0f), start.z), dir.z, inv.z);
    } else {
        r.cx = f2i(start.x); r.cy = f2i(start.y); r.cz = f2i(start.z);
        r.tx = fdiv(fsub((float)(r.cx + (r.sx > 0)), start.x), dir.x);
        r.ty = fdiv(fsub((float)(r.cy + (r.sy > 0)), start.y), dir.y);
        r.tz = fdiv(fsub((float)(r.cz + (r.sz > 0)), start.z), dir.z);
    }
}

// Whether the words a warp's rays are about to read lie in HBM rather than in L2: one load 40 cell
// lengths ahead of the camera, timed.  A frame that follows others finds its words in L2; one
// whose words were never read or were displaced waits for HBM at every new line, and then
// prefetching 24 cell lengths ahead pays for its ten instructions an iteration, which cost an
// 800x600 level frame with three lights 11 us otherwise.  L2 flushed before each frame: 107 and
// 124 us without prefetching, 89 and 99 with it (two cameras), the app's first frame 92 and 75;
// frames in a row 44.9 -> 46.6 and 34.4 -> 35.7 us.  The limit lies where both hold: at 420
// cycles the frames in a row take 47.3 and 36.8 us, at 600 (46.1 and 35.4) the app's first frame
// takes 81 to 91 us after a flush.
constexpr float kPrefetchCells = 24.0f, kProbeCells = 40.0f;
constexpr uint32_t kFarCycles = 480;
__device__ __forceinline__ bool words_are_far(const Layout& L, const WordParams& p, V3 cam, V3 dir) {
    const int x = min(max(f2i(fadd(fmul(dir.x, kProbeCells), cam.x)), 0), L.W - 1);
    const int y = min(max(f2i(fadd(fmul(dir.y, kProbeCells), cam.y)), 0), L.H - 1);
    const int z = min(max(f2i(fadd(fmul(dir.z, kProbeCells), cam.z)), 0), L.W - 1);
    uint32_t from, to;
    int32_t v;
    asm volatile("mov.u32 %0, %%clock;" : "=r"(from));
    asm volatile("ld.global.b32 %0, [%1];" : "=r"(v) : "l"(p.words + (x + L.W * y + L.W * L.H * z)));
    // the clock is read under a condition on the word, so behind its arrival
    asm volatile("{.reg .pred q;\n\tsetp.eq.s32 q, %1, 0x7fffffff;\n\t@q mov.u32 %0, 0;\n\t@!q mov.u32 %0, %%clock;}"
                 : "=r"(to) : "r"(v));
    return to - from > kFarCycles;
}

struct WordRay {
    int32_t hit;   // voxel index or -1
    float cd;      // currDist at the hit
    int axis, s;   // axis and step sign of the last DDA step (hitNormal)
    V3 start;      // start position after depth-field jumps (hitPos uses it)
    int steps;
};

// castRay, fshader.glsl:59-129, over the voxel words.  A cell outside the world ends the
// ray, getVoxelIndex == -1 (:123-125).  Inexact launches also end a ray that cannot hit
// anything: a cell in [lo_y, lo_y + span_y) along y stays alive, beyond the solid box the
// ray moves away from (or does not move along) along y ends it, since every later cell
// stays beyond it.  Depth-field jumps move the start forward along dir, so they keep that
// true.  (Only y: in terrain worlds the solid box spans x and z, and two registers per
// ray are what this latency-bound kernel can spare.)
//
// What bounds it: instruction issue (75 % of the slots while an SM is busy), 47 M warp
// instructions for an 800x600 frame of the level with three lights.  An iteration is about 35
// instructions, a jump 45 more, a ray's set-up and shading 400.  On that frame, one by one, the
// intersect adds in the shadow of the load, and not behind it for the iterations that turn out
// not to jump, save 4.5 us of 67.2, the ray's six reciprocals by rcp_near another 0.9, and in
// frames that overlap the load predicated instead of branched around 2.9 of 47.8.
__device__ WordRay cast_word(const Layout& L, const WordParams& p, V3 start, V3 dir, int dist, int maxSteps,
                             bool far) {
    WordRay o;
    o.hit = -1; o.cd = 0.0f; o.axis = 2; o.s = 0; o.steps = 0;
    RaySetup r;
    // The divisions by the ray's direction, here and at each jump: see div_by.
    const V3 b{fadd(dir.x, 0.000001f), fadd(dir.y, 0.000001f), fadd(dir.z, 0.000001f)};
    const float lo = min3_nan(start.x, start.y, start.z);
    const bool fast = all_within(dir, kDivMinB, kDivMaxB) & all_within(b, kDivMinB, 2.5f) & (lo == lo);
    r.sx = isign(dir.x); r.sy = isign(dir.y); r.sz = isign(dir.z);
    V3 inv{0.0f, 0.0f, 0.0f};
    if (fast) {
        inv = V3{rcp_near(dir.x), rcp_near(dir.y), rcp_near(dir.z)};
        r.dx = rcp_near(fabsf(b.x)); r.dy = rcp_near(fabsf(b.y)); r.dz = rcp_near(fabsf(b.z));
    } else {
        r.dx = frcp(fabsf(b.x)); r.dy = frcp(fabsf(b.y)); r.dz = frcp(fabsf(b.z));
    }
    enter_cell(r, start, dir, inv, fast);
    int lo_y = 0, span_y = L.H;
    if (!p.exact) {
        if (r.sy > 0) {
            span_y = max(0, min(L.H, p.bb[4] + 1));
        } else {
            lo_y = min(max(0, p.bb[1]), L.H);
            span_y = L.H - lo_y;
        }
    }
    float travelled = 0.0f;
    const float lim = fminf((float)dist, (float)maxSteps);
    const int W = L.W, WH = L.W * L.H;
    const unsigned ax = (unsigned)f2i(fmul(dir.x, kPrefetchCells)), ay = (unsigned)f2i(fmul(dir.y, kPrefetchCells)),
                   az = (unsigned)f2i(fmul(dir.z, kPrefetchCells));
    const unsigned ahead = ax + (unsigned)W * ay + (unsigned)WH * az, ahead_z = az + (unsigned)W * ay + (unsigned)WH * ax;
    while (travelled < lim) {
        o.steps++;
        travelled = fadd(travelled, 1.0f);
        // The shader's axis choice (strict <, ties to z); each axis' move is predicated, not a
        // divergent branch.
        const bool bx = (r.tx < r.ty) & (r.tx < r.tz);
        const bool by = (r.ty < r.tx) & (r.ty < r.tz);  // false whenever bx holds, NaN included
        const bool bz = !(bx | by);
        if (bx) r.cx += r.sx;
        if (by) r.cy += r.sy;
        if (bz) r.cz += r.sz;
        // The intersect moves on before the word is there: the adds run in the load's shadow,
        // and a jump, which they don't concern, sets all three anew.
        const float cd = bx ? r.tx : (by ? r.ty : r.tz);
        pred_fadd(r.tx, r.dx, bx);
        pred_fadd(r.ty, r.dy, by);
        pred_fadd(r.tz, r.dz, bz);
        // Outside the world (getVoxelIndex == -1), or no solid voxel ahead: the ray ends as at a
        // solid voxel (word 0), without a hit.
        const bool in = (max((unsigned)r.cx, (unsigned)r.cz) < (unsigned)L.W) &
                        ((unsigned)(r.cy - lo_y) < (unsigned)span_y);
        // A step along z reads the copy in which z is the fastest index: a run of z steps then
        // reads consecutive words instead of one cache line per step (W*H words apart).  That
        // run is the longest ray of the reference's own frame: the shader's x == y tie sends a
        // ray along z for hundreds of steps, which set the frame's length.
        // One load, predicated: the compiler's branch around it parts and joins the lanes again in
        // every iteration.
        int32_t v = 0;
        {
            const int wy = W * r.cy;
            asm("{.reg .pred pz, pi; .reg .b64 q;\n\t"
                "setp.ne.b32 pz, %3, 0; setp.ne.b32 pi, %4, 0;\n\t"
                "mad.wide.s32 q, %1, 4, %5;\n\t"
                "@pz mad.wide.s32 q, %2, 4, %6;\n\t"
                "@pi ld.global.b32 %0, [q];}"
                : "+r"(v)
                : "r"(r.cx + wy + WH * r.cz), "r"(r.cz + wy + WH * r.cx), "r"((int)bz), "r"((int)in), "l"(p.words),
                  "l"(p.words_z));
        }
        if (far) {  // the word some way ahead in both copies (any word at all where the sum leaves them)
            const unsigned n = (unsigned)L.n_words, wy = (unsigned)W * (unsigned)r.cy;
            const unsigned i = (unsigned)r.cx + wy + (unsigned)WH * (unsigned)r.cz + ahead;
            const unsigned iz = (unsigned)r.cz + wy + (unsigned)WH * (unsigned)r.cx + ahead_z;
            if (i < n) asm volatile("prefetch.global.L2 [%0];" ::"l"(p.words + i));
            if (iz < n) asm volatile("prefetch.global.L2 [%0];" ::"l"(p.words_z + iz));
        }
        if (v != -1) {
            if (v >= 0) {
                if (in) {
                    o.hit = r.cx + W * r.cy + WH * r.cz;
                    o.cd = cd;
                    o.axis = bx ? 0 : (by ? 1 : 2);
                    o.s = bx ? r.sx : (by ? r.sy : r.sz);
                    o.start = start;
                }
                break;
            }
            // depth-field jump
            const float toJump = -__int_as_float(v);
            travelled = fadd(travelled, toJump);
            start = add3(mul3s(dir, fadd(cd, toJump)), start);
            enter_cell(r, start, dir, inv, fast);
        }
    }
    return o;
}

// A minimum of 4 CTAs per SM gives the compiler up to 128 registers; it takes 72 (7 CTAs
// per SM).
template <bool DEBUG>
__global__ void __launch_bounds__(128, 4) render_word_kernel(const int32_t* words, Layout L,
                                                          const __grid_constant__ WordParams p) {
    __shared__ int s_cost, s_done, s_tile;
    // In this order: a frame behind this one may be overlapped, and reads the words and the tile
    // classes without waiting.  It begins once all CTAs have triggered, so when each of them has
    // seen the end of the change, or of the recording frame, ahead.
    if (p.wait_first) cudaGridDependencySynchronize();
    cudaTriggerProgrammaticLaunchCompletion();  // see frame_launch
    if (threadIdx.x < 32) {
        const int b = (int)(blockIdx.x + gridDim.x * blockIdx.y), lane = threadIdx.x;
        int tile = b;
        if (p.class_count_in) {  // the b-th tile of the last frame's classes, heaviest class first
            const int c = kTileClasses - 1 - lane;  // lane l: class 15 - l, and how many lie before it
            const int n = lane < kTileClasses ? p.class_count_in[c] : 0;
            int end = n;
            for (int o = 1; o < kTileClasses; o *= 2) {
                const int u = __shfl_up_sync(0xffffffffu, end, o);
                if (lane >= o) end += u;
            }
            if (b < end && b >= end - n) tile = p.class_list_in[c * p.tiles + (b - (end - n))];
            const unsigned found = __ballot_sync(0xffffffffu, b < end && b >= end - n);
            tile = __shfl_sync(0xffffffffu, tile, found ? __ffs(found) - 1 : 0);
        }
        if (b == 0 && p.class_count_clear && lane < kTileClasses) p.class_count_clear[lane] = 0;
        if (lane == 0) {
            s_tile = tile;
            s_cost = 0;
            s_done = 0;
        }
    }
    __syncthreads();
    const int tile = s_tile;
    int px, py;
    p.map.pixel(tile, (int)threadIdx.x, px, py);
    const bool valid = px < p.width && py < p.height;
    PixelResult res{};
    const vrt_uniforms& u = p.u;
    const V3 cam{u.camPos[0], u.camPos[1], u.camPos[2]};
    bool far = false;
    V3 rd{0.f, 0.f, 0.f};
    WordRay pr;
    pr.hit = -1; pr.cd = 0.f; pr.axis = 2; pr.s = 0; pr.start = cam; pr.steps = 0;
    if (valid) {
        rd = primary_dir(u, px, py, p.width, p.height, p.map.inv_w, p.map.inv_h);
        far = words_are_far(L, p, cam, rd);
        pr = cast_word(L, p, cam, rd, u.maxSteps, u.maxSteps, far);
    }
    const bool lit = valid && pr.hit >= 0 && u.viewDepthField != 1;
    const V3 hp = lit ? add3(mul3s(rd, pr.cd), pr.start) : V3{0.f, 0.f, 0.f};
    const unsigned cand = warp_light_candidates(u, lit, hp);
    if (valid) {
        res.hit = pr.hit;
        res.steps = pr.steps;
        res.primary_steps = pr.steps;
        float mr = u.ambient, mg = u.ambient, mb = u.ambient;
        int32_t word = 0;
        if (u.viewDepthField == 1) {
            mr = mg = mb = fdiv((float)pr.steps, 100.0f);
        } else if (pr.hit >= 0) {
            V3 hn = axis_normal(pr.axis, pr.s);
            V3 lp{u.lightPos[0], u.lightPos[1], u.lightPos[2]};
            V3 toLight = norm3(sub3(lp, hp));
            WordRay sr = cast_word(L, p, add3(hp, mul3s(toLight, 0.001f)), toLight, u.maxSteps, u.maxSteps, far);
            res.steps += sr.steps;
            res.cast |= 1u;
            if (sr.hit < 0) {
                float c = fmul(u.diffuse, fmax0(dot3(hn, toLight)));
                mr = fadd(mr, c); mg = fadd(mg, c); mb = fadd(mb, c);
            } else {
                res.occ |= 1u;
            }
            // the warp's candidate local lights in ascending order, the overbright test before
            // each and once more after the last if the shader's loop had iterations left
            // (the same reasoning as in the tile kernel)
            const float ob = u.maxOverbright, R = u.localLightDist;
            const float R1 = fadd(fmul(fabsf(R), 1.0009765625f), 1.0f);
            unsigned todo = cand;
            int last = -1;
            bool clamped = false;
            while (todo) {
                const int i = __ffs(todo) - 1;
                todo &= todo - 1;
                last = i;
                if (mr >= ob && mg >= ob && mb >= ob) {
                    mr = mg = mb = ob;
                    clamped = true;
                    break;
                }
                V3 Lp{u.localLights[i][0], u.localLights[i][1], u.localLights[i][2]};
                const V3 dl = sub3(Lp, hp);
                if (fabsf(dl.x) > R1 || fabsf(dl.y) > R1 || fabsf(dl.z) > R1) continue;
                float ld = len3(dl);
                if (ld <= R) {
                    V3 tl = norm3(dl);
                    WordRay lr = cast_word(L, p, add3(hp, mul3s(tl, 0.001f)), tl, f2i(fadd(ld, 1.0f)),
                                           u.maxSteps, far);
                    res.steps += lr.steps;
                    res.cast |= 2u << i;
                    if (lr.hit < 0) {
                        float nl = fmax0(dot3(hn, tl));
                        float fall = fdiv(fsub(R, ld), R);
                        float a = u.localLights[i][3];
                        mr = fadd(mr, fmul(fmul(fmul(a, u.localLightColor[i][0]), nl), fall));
                        mg = fadd(mg, fmul(fmul(fmul(a, u.localLightColor[i][1]), nl), fall));
                        mb = fadd(mb, fmul(fmul(fmul(a, u.localLightColor[i][2]), nl), fall));
                    } else {
                        res.occ |= 2u << i;
                    }
                }
            }
            if (!clamped && last < VRT_MAX_LOCAL_LIGHTS - 1 && mr >= ob && mg >= ob && mb >= ob) mr = mg = mb = ob;
            word = words[pr.hit];
        }
        res.mr = mr; res.mg = mg; res.mb = mb;
        res.rgba = pack_color_tab(u, pr.hit >= 0, word, mr, mg, mb, pr.steps);
    }
    cudaGridDependencySynchronize();  // nothing is written before the frame ahead has ended
    if (valid) {
        if (DEBUG) store_pixel(p.dbg, p.rgba, (uint64_t)py * p.width + px, res);
        else reinterpret_cast<uint32_t*>(p.rgba)[(uint64_t)py * p.width + px] = res.rgba;
    }
    const int wmax = __reduce_max_sync(0xffffffffu, valid ? res.steps : 0);
    // The CTA's last warp to end appends the tile; nobody waits for it.
    if ((threadIdx.x & 31) == 0 && p.class_list_out) {
        atomicMax(&s_cost, wmax);
        __threadfence_block();
        if (atomicAdd(&s_done, 1) == (int)blockDim.x / 32 - 1) {
            __threadfence_block();
            const int c = tile_class(atomicMax(&s_cost, 0));
            p.class_list_out[c * p.tiles + atomicAdd(p.class_count_out + c, 1)] = tile;
        }
    }
    if (p.stats) {
        unsigned rays = valid ? 1u + __popc(res.cast) : 0u;
        unsigned steps = valid ? (unsigned)res.steps : 0u;
        unsigned hits = valid && res.hit >= 0 ? 1u : 0u;
        unsigned pix = valid ? 1u : 0u;
        rays = __reduce_add_sync(0xffffffffu, rays);
        unsigned long long s64 = steps;  // a warp's steps can pass 2^32 at large step caps
        for (int off = 16; off > 0; off >>= 1) s64 += __shfl_down_sync(0xffffffffu, s64, off);
        hits = __reduce_add_sync(0xffffffffu, hits);
        pix = __reduce_add_sync(0xffffffffu, pix);
        if ((threadIdx.x & 31) == 0) {
            atomicAdd(p.stats + VRT_STAT_RAYS, (unsigned long long)rays);
            atomicAdd(p.stats + VRT_STAT_STEPS, s64);
            atomicAdd(p.stats + VRT_STAT_HITS, (unsigned long long)hits);
            atomicAdd(p.stats + VRT_STAT_PIXELS, (unsigned long long)pix);
        }
    }
}

// ====================================================================== mask kernel

struct ViewDev {
    vrt_uniforms u;
    int width, height;
    TileMap map;
    int tile_begin;  // first global tile of this view
    int refill_min;  // lanes parked before a warp runs its slow phase (tile's view decides)
    int exact;       // 1: step every ray to its end (step counts asked for); 0: end rays that cannot hit
    uint8_t* rgba;
    vrt_debug_out dbg;
    unsigned long long* stats;
};

struct MaskParams {
    const int32_t* words;
    const uint64_t* bricks;
    const uint8_t* bdir;   // directed brick distances, 8 bytes per brick (one per octant)
    const uint8_t* rdist;
    int bb[6];             // solid bounding box: min x,y,z, max x,y,z (never smaller than the truth)
    int cl[6];             // tile kernel: boxes are clipped to [cl[0],cl[3]) x [cl[1],cl[4]) x [cl[2],cl[5])
    int tile0;             // tile kernel: the launch covers tiles [tile0, tile0 + gridDim.x)
    int one, four, sixteen;  // 1, 4, 16: multipliers the compiler cannot fold (see cast_box)
    int4 clip_k[27];       // tile kernel: see enter_box_lean
    int4 oct_k[16];        // tile kernel: see cast_lean
    Layout L;
    const ViewDev* views;  // nviews entries (device); NULL when nviews == 1 (v0 is used)
    int nviews;
    int total_tiles;
    int region_bytes16;    // region distance bytes rounded up to 16 (staged in shared memory when small)
    unsigned int* tile_counter;
    ViewDev v0;
};

enum { M_RUN = 0, M_BOX = 1, M_HIT = 2, M_MISS = 3, M_IDLE = 4, M_DONE = 5 };
enum { PH_PRIMARY = 0, PH_GLOBAL = 1, PH_LOCAL0 = 2 };
enum { T_LIVE = 0, T_HIT = 1, T_MISS = 2 };

// Per-lane pixel state kept in shared memory (structure of arrays, 256 lanes): it is
// touched only between rays, so the traversal loop keeps only the ray in registers.
enum {
    F_PIX, F_VID, F_HPX, F_HPY, F_HPZ, F_MR, F_MG, F_MB, F_HIT, F_CAST, F_OCC, F_STEPS, F_PSTEPS, F_HN,
    F_ST_VID, F_ST_RAYS, F_ST_HITS, F_ST_PIX, F_ST_STEPS_LO, F_ST_STEPS_HI, F_ST_REFILLS, NF
};
constexpr int kThreads = 256;
constexpr int kUnroll = 4;

__device__ __forceinline__ const ViewDev& view_of(const MaskParams& P, int v) {
    return P.nviews == 1 ? P.v0 : P.views[v];
}

struct Ray {
    int cx, cy, cz;
    int sx, sy, sz;
    int ex, ey, ez;  // cell coordinate at which the ray leaves its known box, per axis
    int rem;         // DDA iterations left
    int la;          // axis of the parked step
    float tx, ty, tz;
    float dx, dy, dz;
    uint64_t m;      // voxel bits of the current brick (0 inside an empty box)
};

// Start a ray at o along d with loop bound n (fshader.glsl:64-79).  The known box is
// empty: every exit coordinate is the first cell a step along that axis reaches, so the
// first step always parks the lane for a refill.
__device__ __forceinline__ int start_ray(Ray& r, V3 o, V3 d, int n, int maxSteps) {
    RaySetup s;
    ray_setup(o, d, s);
    r.cx = s.cx; r.cy = s.cy; r.cz = s.cz;
    r.sx = s.sx; r.sy = s.sy; r.sz = s.sz;
    r.tx = s.tx; r.ty = s.ty; r.tz = s.tz;
    r.dx = s.dx; r.dy = s.dy; r.dz = s.dz;
    r.rem = max(0, min(n, maxSteps));
    r.ex = s.cx + s.sx; r.ey = s.cy + s.sy; r.ez = s.cz + s.sz;
    r.m = 0;
    r.la = 2;
    return r.rem;
}

// A ray in cell c cannot hit anything if, along some axis, c lies beyond the solid
// bounding box and the ray moves away from it or parallel to it: every later cell stays
// beyond the box along that axis.
__device__ __forceinline__ bool beyond_solids(const MaskParams& P, int cx, int cy, int cz, int sx, int sy, int sz) {
    return (cx < P.bb[0] && sx <= 0) || (cy < P.bb[1] && sy <= 0) || (cz < P.bb[2] && sz <= 0) ||
           (cx > P.bb[3] && sx >= 0) || (cy > P.bb[4] && sy >= 0) || (cz > P.bb[5] && sz >= 0);
}

// The parked step moved the ray into cell c outside its box: bound the largest known
// box around c from the distance fields, or load the brick's voxel bits.
template <bool SMEM>
__device__ __forceinline__ int refill(Ray& r, const MaskParams& P, const uint8_t* rdist, bool exact) {
    const Layout& L = P.L;
    if ((unsigned)r.cx >= (unsigned)L.W || (unsigned)r.cy >= (unsigned)L.H || (unsigned)r.cz >= (unsigned)L.W)
        return T_MISS;  // getVoxelIndex == -1 (fshader.glsl:123-125)
    if (!exact && beyond_solids(P, r.cx, r.cy, r.cz, r.sx, r.sy, r.sz)) return T_MISS;
    const int rx = r.cx >> 4, ry = r.cy >> 4, rz = r.cz >> 4;
    const uint64_t rl = region_linear(L, rx, ry, rz);
    const int dr = SMEM ? (int)rdist[rl] : (int)__ldg(rdist + rl);
    int lox, loy, loz, hix, hiy, hiz;
    uint64_t m = 0;
    if (dr > 0) {  // every region within Chebyshev radius dr-1 is empty
        const int k = dr - 1;
        lox = (rx - k) << 4; loy = (ry - k) << 4; loz = (rz - k) << 4;
        hix = (rx + k + 1) << 4; hiy = (ry + k + 1) << 4; hiz = (rz + k + 1) << 4;
    } else {
        const int bx = r.cx >> 2, by = r.cy >> 2, bz = r.cz >> 2;
        const uint64_t bi = brick_index(L, bx, by, bz);
        m = __ldg(P.bricks + bi);
        const int oct = (r.sx > 0) | ((r.sy > 0) << 1) | ((r.sz > 0) << 2);
        const int k = __ldg(P.bdir + bi * 8 + oct) >> 2;  // 0 for a non-empty brick
        lox = (bx - k) << 2; loy = (by - k) << 2; loz = (bz - k) << 2;
        hix = (bx + k + 1) << 2; hiy = (by + k + 1) << 2; hiz = (bz + k + 1) << 2;
    }
    lox = max(lox, 0); loy = max(loy, 0); loz = max(loz, 0);
    hix = min(hix, L.W); hiy = min(hiy, L.H); hiz = min(hiz, L.W);
    r.ex = r.sx > 0 ? hix : (r.sx < 0 ? lox - 1 : INT_MIN);
    r.ey = r.sy > 0 ? hiy : (r.sy < 0 ? loy - 1 : INT_MIN);
    r.ez = r.sz > 0 ? hiz : (r.sz < 0 ? loz - 1 : INT_MIN);
    r.m = m;
    const int bit = (r.cx & 3) | ((r.cy & 3) << 2) | ((r.cz & 3) << 4);
    return ((m >> bit) & 1) ? T_HIT : T_LIVE;
}

template <bool SMEM, int MINB>
__global__ void __launch_bounds__(kThreads, MINB) render_mask_kernel(const __grid_constant__ MaskParams P) {
    extern __shared__ __align__(16) uint8_t smem[];
    const uint8_t* rdist = P.rdist;
    uint32_t* ls = reinterpret_cast<uint32_t*>(smem);
    if (SMEM) {
        const uint4* src = reinterpret_cast<const uint4*>(P.rdist);
        uint4* dst = reinterpret_cast<uint4*>(smem);
        for (int i = threadIdx.x; i < P.region_bytes16 / 16; i += kThreads) dst[i] = __ldg(src + i);
        rdist = smem;
        ls = reinterpret_cast<uint32_t*>(smem + P.region_bytes16);
    }
#define LSU(f) ls[(f) * kThreads + threadIdx.x]
#define LSF(f) reinterpret_cast<float*>(ls)[(f) * kThreads + threadIdx.x]
    LSU(F_ST_VID) = 0xffffffffu;
    LSU(F_ST_RAYS) = 0; LSU(F_ST_HITS) = 0; LSU(F_ST_PIX) = 0; LSU(F_ST_STEPS_LO) = 0; LSU(F_ST_STEPS_HI) = 0;
    LSU(F_ST_REFILLS) = 0;
    if (SMEM) __syncthreads();
    unsigned n_slow = 0, n_fast = 0;  // warp-uniform diagnostics

    const int lane = threadIdx.x & 31;
    const unsigned lt = (1u << lane) - 1u;
    const unsigned FULL = 0xffffffffu;

    // warp tile queue (uniform across the warp)
    int q_pos = 0, q_size = 0, q_vid = 0, q_x0 = 0, q_y0 = 0, q_w = 0, q_h = 0, q_tw = 1, q_thr = 8;
    bool q_empty = false;

    int mode = M_IDLE, phase = PH_PRIMARY;
    Ray r;
    r.cx = r.cy = r.cz = 0; r.sx = r.sy = r.sz = 0; r.ex = r.ey = r.ez = 0; r.rem = 0; r.la = 2;
    r.tx = r.ty = r.tz = 0.f; r.dx = r.dy = r.dz = 0.f; r.m = 0;

    for (;;) {
        // ================= slow phase =================
        // (a) parked box exits: refill from the hierarchy, finish the parked step
        n_slow++;
        if (mode == M_BOX) {
            LSU(F_ST_REFILLS) += 1u;
            const int t = refill<SMEM>(r, P, rdist, view_of(P, (int)LSU(F_VID)).exact != 0);
            if (t == T_LIVE) {
                if (r.la == 0) r.tx = fadd(r.tx, r.dx);
                else if (r.la == 1) r.ty = fadd(r.ty, r.dy);
                else r.tz = fadd(r.tz, r.dz);
                mode = r.rem == 0 ? M_MISS : M_RUN;
            } else {
                mode = t == T_HIT ? M_HIT : M_MISS;
            }
        }
        // (b) ended rays: fold the result into the pixel, pick the pixel's next ray
        bool want = false;
        V3 o{0.f, 0.f, 0.f}, d{0.f, 0.f, 0.f};
        int n = 0;
        if (mode == M_HIT || mode == M_MISS) {
            const int vid = (int)LSU(F_VID), pix = (int)LSU(F_PIX);
            const ViewDev& V = view_of(P, vid);
            const vrt_uniforms& u = V.u;
            int steps = (int)LSU(F_STEPS) - r.rem;  // iterations this ray did not use
            float mr = LSF(F_MR), mg = LSF(F_MG), mb = LSF(F_MB);
            int32_t hit = (int32_t)LSU(F_HIT);
            uint32_t cast = LSU(F_CAST), occ = LSU(F_OCC);
            int psteps = (int)LSU(F_PSTEPS);
            V3 hp{LSF(F_HPX), LSF(F_HPY), LSF(F_HPZ)};
            bool done = false;
            int next = VRT_MAX_LOCAL_LIGHTS;
            if (phase == PH_PRIMARY) {
                psteps = steps;
                if (mode == M_HIT) {
                    const float cd = r.la == 0 ? r.tx : (r.la == 1 ? r.ty : r.tz);
                    hit = r.cx + P.L.W * r.cy + P.L.W * P.L.H * r.cz;
                    const int px = pix % V.width, py = pix / V.width;
                    V3 rd = primary_dir(u, px, py, V.width, V.height, V.map.inv_w, V.map.inv_h);
                    hp = add3(mul3s(rd, cd), V3{u.camPos[0], u.camPos[1], u.camPos[2]});
                    const int s = r.la == 0 ? r.sx : (r.la == 1 ? r.sy : r.sz);
                    LSU(F_HN) = (uint32_t)(r.la | ((s + 1) << 2));
                }
                if (u.viewDepthField == 1) {
                    mr = mg = mb = fdiv((float)psteps, 100.0f);
                    done = true;
                } else if (hit < 0) {
                    done = true;
                } else {
                    V3 toLight = norm3(sub3(V3{u.lightPos[0], u.lightPos[1], u.lightPos[2]}, hp));
                    o = add3(hp, mul3s(toLight, 0.001f));
                    d = toLight;
                    n = u.maxSteps;
                    want = true;
                    phase = PH_GLOBAL;
                }
            } else {
                const uint32_t hn_code = LSU(F_HN);
                const V3 hn = axis_normal((int)(hn_code & 3), (int)(hn_code >> 2) - 1);
                if (phase == PH_GLOBAL) {
                    cast |= 1u;
                    if (mode == M_HIT) {
                        occ |= 1u;
                    } else {
                        V3 toLight = norm3(sub3(V3{u.lightPos[0], u.lightPos[1], u.lightPos[2]}, hp));
                        const float c = fmul(u.diffuse, fmax0(dot3(hn, toLight)));
                        mr = fadd(mr, c); mg = fadd(mg, c); mb = fadd(mb, c);
                    }
                    next = 0;
                } else {
                    const int i = phase - PH_LOCAL0;
                    cast |= 2u << i;
                    if (mode == M_HIT) {
                        occ |= 2u << i;
                    } else {
                        const V3 Lp{u.localLights[i][0], u.localLights[i][1], u.localLights[i][2]};
                        const float ld = len3(sub3(Lp, hp));
                        const V3 tl = norm3(sub3(Lp, hp));
                        const float nl = fmax0(dot3(hn, tl));
                        const float fall = fdiv(fsub(u.localLightDist, ld), u.localLightDist);
                        const float a = u.localLights[i][3];
                        mr = fadd(mr, fmul(fmul(fmul(a, u.localLightColor[i][0]), nl), fall));
                        mg = fadd(mg, fmul(fmul(fmul(a, u.localLightColor[i][1]), nl), fall));
                        mb = fadd(mb, fmul(fmul(fmul(a, u.localLightColor[i][2]), nl), fall));
                    }
                    next = i + 1;
                }
                // fshader.glsl:159-181: overbright test before each light, then the range test
                const float ob = u.maxOverbright;
                for (int i = next; i < VRT_MAX_LOCAL_LIGHTS; i++) {
                    if (mr >= ob && mg >= ob && mb >= ob) {
                        mr = mg = mb = ob;
                        break;
                    }
                    if (u.localLights[i][0] >= 0 && u.localLights[i][1] >= 0 && u.localLights[i][2] >= 0) {
                        const V3 Lp{u.localLights[i][0], u.localLights[i][1], u.localLights[i][2]};
                        const float ld = len3(sub3(Lp, hp));
                        if (ld <= u.localLightDist) {
                            const V3 tl = norm3(sub3(Lp, hp));
                            o = add3(hp, mul3s(tl, 0.001f));
                            d = tl;
                            n = f2i(fadd(ld, 1.0f));
                            want = true;
                            phase = PH_LOCAL0 + i;
                            break;
                        }
                    }
                }
                done = !want;
            }
            if (done) {
                const int32_t word = hit >= 0 ? __ldg(P.words + hit) : 0;
                PixelResult res;
                res.rgba = pack_color(u, hit >= 0, word, mr, mg, mb, psteps);
                res.hit = hit; res.cast = cast; res.occ = occ;
                res.steps = steps; res.primary_steps = psteps;
                res.mr = mr; res.mg = mg; res.mb = mb;
                store_pixel(V.dbg, V.rgba, (uint64_t)pix, res);
                if (V.stats) {
                    if (LSU(F_ST_VID) != (uint32_t)vid) {
                        if (LSU(F_ST_VID) != 0xffffffffu) {  // the lane moves to another view: flush
                            unsigned long long* s = view_of(P, (int)LSU(F_ST_VID)).stats;
                            atomicAdd(s + VRT_STAT_RAYS, (unsigned long long)LSU(F_ST_RAYS));
                            atomicAdd(s + VRT_STAT_STEPS, ((unsigned long long)LSU(F_ST_STEPS_HI) << 32) | LSU(F_ST_STEPS_LO));
                            atomicAdd(s + VRT_STAT_HITS, (unsigned long long)LSU(F_ST_HITS));
                            atomicAdd(s + VRT_STAT_PIXELS, (unsigned long long)LSU(F_ST_PIX));
                            atomicAdd(s + VRT_STAT_REFILLS, (unsigned long long)LSU(F_ST_REFILLS));
                            LSU(F_ST_RAYS) = 0; LSU(F_ST_HITS) = 0; LSU(F_ST_PIX) = 0;
                            LSU(F_ST_STEPS_LO) = 0; LSU(F_ST_STEPS_HI) = 0; LSU(F_ST_REFILLS) = 0;
                        }
                        LSU(F_ST_VID) = (uint32_t)vid;
                    }
                    LSU(F_ST_RAYS) += 1u + __popc(cast);
                    const unsigned long long s64 =
                        (((unsigned long long)LSU(F_ST_STEPS_HI) << 32) | LSU(F_ST_STEPS_LO)) + (unsigned)steps;
                    LSU(F_ST_STEPS_LO) = (uint32_t)s64;
                    LSU(F_ST_STEPS_HI) = (uint32_t)(s64 >> 32);
                    LSU(F_ST_HITS) += hit >= 0;
                    LSU(F_ST_PIX) += 1u;
                }
                mode = M_IDLE;
            } else {
                LSF(F_MR) = mr; LSF(F_MG) = mg; LSF(F_MB) = mb;
                LSU(F_HIT) = (uint32_t)hit; LSU(F_CAST) = cast; LSU(F_OCC) = occ;
                LSU(F_PSTEPS) = (uint32_t)psteps;
                LSF(F_HPX) = hp.x; LSF(F_HPY) = hp.y; LSF(F_HPZ) = hp.z;
            }
            LSU(F_STEPS) = (uint32_t)steps;
        }

        // (c) hand new pixels to idle lanes from the warp's tile queue
        unsigned need = __ballot_sync(FULL, mode == M_IDLE);
        while (need && !q_empty) {
            if (q_pos >= q_size) {
                unsigned t = 0;
                if (lane == 0) t = atomicAdd(P.tile_counter, 1u);
                t = __shfl_sync(FULL, t, 0);
                if (t >= (unsigned)P.total_tiles) {
                    q_empty = true;
                    break;
                }
                int v = 0;
                if (P.nviews > 1) {
                    while (v + 1 < P.nviews && P.views[v + 1].tile_begin <= (int)t) v++;
                }
                const ViewDev& V = view_of(P, v);
                const int lt_idx = (int)t - V.tile_begin;
                q_vid = v;
                q_tw = V.map.tw;
                q_x0 = (lt_idx % V.map.tiles_x) * V.map.tw;
                q_y0 = (lt_idx / V.map.tiles_x) * V.map.th;
                q_w = V.width;
                q_h = V.height;
                q_thr = V.refill_min;
                q_pos = 0;
                q_size = V.map.tw * V.map.th;
            }
            const int rank = __popc(need & lt);
            const int take = min(__popc(need), q_size - q_pos);
            if (((need >> lane) & 1) && rank < take) {
                const int pos = q_pos + rank;
                const int px = q_x0 + pos % q_tw, py = q_y0 + pos / q_tw;
                if (px < q_w && py < q_h) {
                    const vrt_uniforms& u = view_of(P, q_vid).u;
                    LSU(F_VID) = (uint32_t)q_vid;
                    LSU(F_PIX) = (uint32_t)(py * q_w + px);
                    LSU(F_HIT) = 0xffffffffu;
                    LSU(F_CAST) = 0; LSU(F_OCC) = 0; LSU(F_STEPS) = 0; LSU(F_PSTEPS) = 0;
                    LSF(F_MR) = u.ambient; LSF(F_MG) = u.ambient; LSF(F_MB) = u.ambient;
                    LSF(F_HPX) = 0.f; LSF(F_HPY) = 0.f; LSF(F_HPZ) = 0.f;
                    LSU(F_HN) = 2u | (1u << 2);
                    o = V3{u.camPos[0], u.camPos[1], u.camPos[2]};
                    d = primary_dir(u, px, py, q_w, q_h, view_of(P, q_vid).map.inv_w, view_of(P, q_vid).map.inv_h);
                    n = u.maxSteps;
                    want = true;
                    phase = PH_PRIMARY;
                    mode = M_RUN;
                }
            }
            q_pos += take;
            need = __ballot_sync(FULL, mode == M_IDLE);
        }
        if (mode == M_IDLE && q_empty) mode = M_DONE;

        // (d) set up the new rays together
        if (want) {
            const int vid = (int)LSU(F_VID);
            const int rem = start_ray(r, o, d, n, view_of(P, vid).u.maxSteps);
            LSU(F_STEPS) += (uint32_t)rem;
            mode = rem == 0 ? M_MISS : M_RUN;
        }

        const unsigned act = __ballot_sync(FULL, mode != M_DONE);
        if (act == 0) break;

        // ================= fast phase: DDA steps in registers =================
        const int thr = min(q_thr, __popc(act));
        for (;;) {
            n_fast++;
#pragma unroll
            for (int k = 0; k < kUnroll; k++) {
                if (mode == M_RUN) {
                    // one iteration of castRay's loop (fshader.glsl:83-126) inside a known box
                    const bool bx = (r.tx < r.ty) & (r.tx < r.tz);
                    const bool by = (!bx) & (r.ty < r.tx) & (r.ty < r.tz);
                    const bool bz = !(bx | by);
                    if (bx) r.cx += r.sx;
                    if (by) r.cy += r.sy;
                    if (bz) r.cz += r.sz;
                    r.rem -= 1;
                    const bool out = (r.cx == r.ex) | (r.cy == r.ey) | (r.cz == r.ez);
                    const int bit = (r.cx & 3) | ((r.cy & 3) << 2) | ((r.cz & 3) << 4);
                    const bool hb = (r.m >> bit) & 1;
                    if (out | hb | (r.rem == 0)) {
                        r.la = bx ? 0 : (by ? 1 : 2);
                        mode = out ? M_BOX : (hb ? M_HIT : M_MISS);
                    } else {
                        if (bx) r.tx = fadd(r.tx, r.dx);
                        if (by) r.ty = fadd(r.ty, r.dy);
                        if (bz) r.tz = fadd(r.tz, r.dz);
                    }
                }
            }
            const unsigned parked = __ballot_sync(FULL, mode != M_RUN && mode != M_DONE);
            if (__popc(parked) >= thr) break;
        }
    }

    if (LSU(F_ST_VID) != 0xffffffffu) {
        unsigned long long* s = view_of(P, (int)LSU(F_ST_VID)).stats;
        atomicAdd(s + VRT_STAT_RAYS, (unsigned long long)LSU(F_ST_RAYS));
        atomicAdd(s + VRT_STAT_STEPS, ((unsigned long long)LSU(F_ST_STEPS_HI) << 32) | LSU(F_ST_STEPS_LO));
        atomicAdd(s + VRT_STAT_HITS, (unsigned long long)LSU(F_ST_HITS));
        atomicAdd(s + VRT_STAT_PIXELS, (unsigned long long)LSU(F_ST_PIX));
        atomicAdd(s + VRT_STAT_REFILLS, (unsigned long long)LSU(F_ST_REFILLS));
    }
    if (lane == 0 && view_of(P, q_vid).stats) {
        atomicAdd(view_of(P, q_vid).stats + VRT_STAT_SLOW, (unsigned long long)n_slow);
        atomicAdd(view_of(P, q_vid).stats + VRT_STAT_FAST, (unsigned long long)n_fast);
    }
#undef LSU
#undef LSF
}

// ---------------------------------------------------------------- tile kernel, one thread per pixel

// Where a ray stands inside its known box.  Per axis: k = further steps along that axis
// that stay inside the box (the step that makes k negative leaves it), e = the box's last
// cell along that axis, the one k further steps reach, so the current cell is always
// e - s*k (one multiply-add).  An axis the ray does not move along (s == 0) has
// k = INT_MAX and e = its fixed cell.
struct BoxRay {
    float tx, ty, tz;
    float dx, dy, dz;
    int kx, ky, kz;
    int ex, ey, ez;
    int sx, sy, sz;
    int sc;          // sign code (sx+1) + 3(sy+1) + 9(sz+1): the ray's entry of clip_k
    int lb;          // lb + kx + ky + kz = DDA iterations left after the current one (negative on
                     // the last allowed one): every iteration lowers exactly one k
    int bi;          // bit of the current cell in m (valid while m != 0)
    uint64_t m;      // voxel bits of the current brick, 0 inside an empty box
};

// kmax limits k: a box is cut short so that the ray leaves it by its last allowed
// iteration (see cast_box).  e = c + s * k is the last cell before the (possibly nearer)
// far face; k = s * (ee - c) - 1 and e are multiply-adds, which issue on the FMA pipe
// rather than the integer/logic pipe.
__device__ __forceinline__ void set_axis(int c, int s, int lo, int hi, int kmax, int& k, int& e) {
    const int ee = s > 0 ? hi : lo - 1;
    k = min(s != 0 ? s * (ee - c) - 1 : INT_MAX, kmax);
    e = s * k + c;
}

// Per-octant alive ranges of a launch, one (lo, span) pair per octant and axis: a cell
// whose coordinate c has (unsigned)(c - lo) >= span along some axis ends the ray.  Exact
// launches hold the world, [0, dim): getVoxelIndex == -1 (fshader.glsl:123-125).
// Inexact launches also end rays that cannot hit anything: moving + along an axis (octant
// bit set), a cell beyond the solid box's upper face will only move further from it, so
// the range is [0, min(dim, bb_hi + 1)); moving - or not at all, [max(0, bb_lo), dim).
// (A ray that does not move along the axis could also end beyond the upper face; it is
// left to walk, which costs time, not exactness.)  Kept in shared memory: three 8-byte
// loads per lookup replace a dozen integer compares.
__device__ __forceinline__ void fill_alive_ranges(int2* alive, const MaskParams& P, bool exact) {
    if (threadIdx.x < 24) {
        const int o = threadIdx.x / 3, a = threadIdx.x % 3;
        const int dim = a == 1 ? P.L.H : P.L.W;
        int lo = 0, span = dim;
        if (!exact) {
            if ((o >> a) & 1) {
                span = max(0, min(dim, P.bb[3 + a] + 1));
            } else {
                lo = min(max(0, P.bb[a]), dim);
                span = dim - lo;
            }
        }
        alive[threadIdx.x] = make_int2(lo, span);
    }
}

// The ray stands in cell c, outside any known box: load c's brick and its directed
// distance for the ray's octant.  A non-empty brick becomes the box (its voxel bits are
// tested step by step); an empty one at directed distance d gives the cube of bricks from
// it d-1 bricks ahead.  (Region-level cubes are not consulted: with directed brick cubes
// they would shorten the walk by well under 1 % of lookups, less than their own cost.)
// left: the ray's iterations left after the current one.  The box is cut to at most
// left / 3 further steps per axis, so the ray leaves it by its last allowed iteration:
// the step cap is then tested only when a box is left.
// Returns T_LIVE, T_HIT (c is solid) or T_MISS (c is outside the alive ranges).
__device__ __forceinline__ int enter_box(BoxRay& r, int cx, int cy, int cz, const MaskParams& P,
                                         const int2* alive, const int4* clip_k, int left) {
    const Layout& L = P.L;
    const int oct = clip_k[r.sc].w;
    const int2 ax = alive[oct * 3], ay = alive[oct * 3 + 1], az = alive[oct * 3 + 2];
    if ((unsigned)(cx - ax.x) >= (unsigned)ax.y || (unsigned)(cy - ay.x) >= (unsigned)ay.y ||
        (unsigned)(cz - az.x) >= (unsigned)az.y)
        return T_MISS;
    const int bx = cx >> 2, by = cy >> 2, bz = cz >> 2;
    // slots in 32 bits: a world holds at most 2^31 voxels, so 8 * n_bricks < 2^32
    const uint32_t bidx = (uint32_t)bx + (uint32_t)L.BWp * ((uint32_t)by + (uint32_t)L.BHp * (uint32_t)bz);
    // the two loads are independent: issue them together, wait once
    const uint64_t m = __ldg(P.bricks + bidx);
    const int k = __ldg(P.bdir + (bidx * 8u + oct)) >> 2;  // 0 for a non-empty brick
    // clip to the world, and for inexact launches to the solid box too: a ray that
    // leaves the solid box along its direction of travel then ends at the next lookup.
    // (Multiplies by a kernel parameter equal to 4 rather than shifts: FMA pipe.)
    const int four = P.four;
    const int lox = max((bx - k) * four, P.cl[0]), loy = max((by - k) * four, P.cl[1]),
              loz = max((bz - k) * four, P.cl[2]);
    const int hix = min((bx + k + 1) * four, P.cl[3]), hiy = min((by + k + 1) * four, P.cl[4]),
              hiz = min((bz + k + 1) * four, P.cl[5]);
    const int kmax = (int)__umulhi((unsigned)max(left, 0), 0x55555556u);  // floor(left / 3)
    set_axis(cx, r.sx, lox, hix, kmax, r.kx, r.ex);
    set_axis(cy, r.sy, loy, hiy, kmax, r.ky, r.ey);
    set_axis(cz, r.sz, loz, hiz, kmax, r.kz, r.ez);
    r.lb = left - (r.kx + r.ky + r.kz);
    r.m = m;
    r.bi = (cx & 3) | ((cy & 3) << 2) | ((cz & 3) << 4);
    return ((m >> r.bi) & 1) ? T_HIT : T_LIVE;
}

// enter_box for worlds without depth-field words, where a ray only ever moves forward
// along each axis.  cast_box checks the ray's first cell against the near side of the
// world (and of the clip box along an axis the ray does not move along) once; every later
// cell lies on the inner side of those bounds, so here only the far side of the clip box
// [cl[0], cl[3]) x [cl[1], cl[4]) x [cl[2], cl[5]) can end the ray:
//   kclip = s > 0 ? hi - 1 - c : (s < 0 ? c - lo : INT_MAX)   (steps before the far clip face)
//         = A - s * c,   A = hi - 1, -lo or INT_MAX
// A depends only on the ray's signs: clip_k holds it for each of the 27 sign codes (with
// the octant, which indexes the directed distances), so the three terms are one shared
// load and three multiply-adds.  kclip < 0 along some axis: the cell is beyond that face
// (outside the world, or beyond the solid box in the direction of travel), which ends the
// ray as a miss.  Otherwise the box along each axis is the rest of the brick plus 4 cells
// per further brick of an empty cube, cut at the clip face and the step cap:
//   k = min((s > 0 ? 3 - (c & 3) : c & 3) + 4 kk, kclip, kmax)
// which is enter_box's box without its near-side bounds.  (An axis the ray does not move
// along steps only when its intersect is -inf or NaN; its cell stays put and its k only
// decides how often the box is looked up again.)  A lookup runs in about a quarter of the
// loop's warp iterations, with some 25 lanes at once, so each instruction here counts.
__device__ __forceinline__ int enter_box_lean(BoxRay& r, int cx, int cy, int cz, const MaskParams& P,
                                              const int4* clip_k, int left) {
    const Layout& L = P.L;
    const int4 A = clip_k[r.sc];
    const int kcx = A.x - r.sx * cx, kcy = A.y - r.sy * cy, kcz = A.z - r.sz * cz;
    if ((kcx | kcy | kcz) < 0) return T_MISS;
    const int bx = cx >> 2, by = cy >> 2, bz = cz >> 2;
    const uint32_t bidx = (uint32_t)bx + (uint32_t)L.BWp * ((uint32_t)by + (uint32_t)L.BHp * (uint32_t)bz);
    const uint64_t m = __ldg(P.bricks + bidx);
    const int kk4 = __ldg(P.bdir + (bidx * 8u + A.w));  // 0 for a non-empty brick: its own box
    const int kmax = (int)__umulhi((unsigned)max(left, 0), 0x55555556u);  // floor(left / 3)
    r.kx = min(min((((r.sx > 0) ? ~cx : cx) & 3) + kk4, kcx), kmax);
    r.ky = min(min((((r.sy > 0) ? ~cy : cy) & 3) + kk4, kcy), kmax);
    r.kz = min(min((((r.sz > 0) ? ~cz : cz) & 3) + kk4, kcz), kmax);
    r.ex = r.sx * r.kx + cx;
    r.ey = r.sy * r.ky + cy;
    r.ez = r.sz * r.kz + cz;
    r.lb = left - (r.kx + r.ky + r.kz);
    r.m = m;
    r.bi = (cx & 3) | ((cy & 3) << 2) | ((cz & 3) << 4);
    return ((m >> r.bi) & 1) ? T_HIT : T_LIVE;
}

// castRay (fshader.glsl:59-129) over the occupancy hierarchy.  Every iteration makes the
// shader's comparison and its one intersect add, in the shader's order; memory is read
// only when the ray leaves its known box.  On a hit, cd / axis / sgn / cell describe the
// last step (currDist, hitNormal, the voxel).
// DF (worlds with depth-field words): the masks mark every cell the shader's loop stops
// at (word != -1).  At such a cell the word decides: solid is a hit; a depth-field word is
// the shader's jump (:114-121): distTravelled and currDist grow by the jump, the start
// moves to dir * currDist + start, and the walk restarts from its cell.  The step cap is
// then the shader's float test distTravelled < min(dist, RENDER_DIST) (:83), kept as a
// float because the jumps make distTravelled fractional.  start_out receives the start
// the hit position is measured from.
template <bool DF, bool COUNT>
__device__ __forceinline__ int cast_box(const MaskParams& P, const int2* alive, const int4* clip_k,
                                        const RaySetup& s, V3 o, V3 d, int n, int maxSteps,
                                        float& cd, int& axis, int& sgn, int& steps, int32_t& hit_index,
                                        unsigned& refills, V3& start_out) {
    start_out = o;
    BoxRay r;
    r.tx = s.tx; r.ty = s.ty; r.tz = s.tz;
    r.dx = s.dx; r.dy = s.dy; r.dz = s.dz;
    r.sx = s.sx; r.sy = s.sy; r.sz = s.sz;
    r.sc = (s.sx + 1) + 3 * (s.sy + 1) + 9 * (s.sz + 1);
    const int n0 = max(0, min(n, maxSteps));
    if (n0 == 0) return T_MISS;
    // The bit-index update and the box-counter decrements are multiply-adds by kernel
    // parameters equal to 1, 4 and 16.  The compiler cannot turn them into plain adds, so
    // they issue on the FMA pipe, which the intersect adds leave mostly idle, instead of
    // the integer/logic pipe that bounds this loop.  (The counters as multiply-adds lost
    // while the loop still branched on each axis; with the branch-free adds they took the
    // 1080p frame from 202.4 M to 183.3 M warp instructions and 0.193 to 0.185 ms.
    // Packing the three counters and the bit index into one word, one add per step, took
    // 3.7 % of the instructions away but was slower: all of its work lands on the integer
    // pipe.)
    const int one = P.one, four = P.four, sixteen = P.sixteen;
    const int sy4 = r.sy * four, sz16 = r.sz * sixteen;  // the bit-index moves along y and z
    // The step cap.  An iteration lowers exactly one of kx, ky, kz, so lb + kx + ky + kz
    // counts the iterations left after the current one without a counter of its own; it is
    // negative on the last allowed iteration.  Every box is cut so that the ray leaves it
    // by that iteration (enter_box), so the cap is tested only where a box is left.  With
    // DF the float test decides instead, and the count only counts (it cannot reach 0
    // first: caps are at most 2^24).
    constexpr int kCount = 1 << 30;
    const int left0 = DF ? kCount - 1 : n0 - 1;
    r.lb = left0;
    int left_end = left0;  // the count at the breaking iteration
    float travelled = 0.0f;
    const float lim = DF ? fminf((float)n, (float)maxSteps) : 0.0f;
    V3 start = o;
    if (!DF) {
        // The first cell (the start cell stepped along the first iteration's axis) must lie on
        // the inner side of the near world bound along every axis the ray moves along, and
        // within the clip box along an axis it does not move along; the ray then stays there
        // (lookups test only the far side).  Otherwise it ends at its first iteration, as the
        // shader's getVoxelIndex == -1 (or, for inexact launches, no solid voxel ahead) does.
        const bool fx = (s.tx < s.ty) & (s.tx < s.tz);
        const bool fy = (s.ty < s.tx) & (s.ty < s.tz);
        const int c1x = s.cx + (fx ? s.sx : 0), c1y = s.cy + (fy ? s.sy : 0), c1z = s.cz + ((fx | fy) ? 0 : s.sz);
        const bool dead =
            (s.sx > 0 ? c1x < 0 : (s.sx < 0 ? c1x >= P.L.W : (c1x < P.cl[0] || c1x >= P.cl[3]))) ||
            (s.sy > 0 ? c1y < 0 : (s.sy < 0 ? c1y >= P.L.H : (c1y < P.cl[1] || c1y >= P.cl[4]))) ||
            (s.sz > 0 ? c1z < 0 : (s.sz < 0 ? c1z >= P.L.W : (c1z < P.cl[2] || c1z >= P.cl[5])));
        if (dead) {
            steps += 1;
            return T_MISS;
        }
    }
    // no box yet: the first step along any axis (even one with s == 0) triggers a lookup
    r.kx = 0; r.ky = 0; r.kz = 0;
    r.ex = s.cx; r.ey = s.cy; r.ez = s.cz;
    r.m = 0;
    r.bi = 0;
    int result = T_MISS;
    // Two iterations per trip of the loop for worlds without depth-field words: one
    // backward branch per two iterations, and the compiler schedules the two bodies
    // together (0.1789 -> 0.1727 ms on the 1080p frame, 0.439 -> 0.427 ms on the stress
    // camera over a 1024-wide world; 3 and 4 measured no better).  The depth-field
    // variant, whose jumps restart the walk, ran 1 % slower unrolled and is left as is.
#pragma unroll(DF ? 1 : 2)
    for (;;) {
        const bool bx = (r.tx < r.ty) & (r.tx < r.tz);
        const bool by = (r.ty < r.tx) & (r.ty < r.tz);  // false whenever bx holds, NaN included
        const bool bz = !(bx | by);
        if (bx) r.kx = r.kx * one - 1;
        if (by) r.ky = r.ky * one - 1;
        if (bz) r.kz = r.kz * one - 1;
        bool last = false;  // DF: no iteration follows this one
        if (DF) {
            travelled = fadd(travelled, 1.0f);
            last = !(travelled < lim);
        }
        // The cell's bit, meaningful only while the step stays in the box; in an empty box
        // (m == 0) it is 0.  Testing it without a branch on m pays: nearly every warp has a
        // lane inside a non-empty brick, so the branch would be taken anyway.  The index
        // moves by sx, 4 sy or 16 sz: three multiply-adds predicated on the axis, on the FMA
        // pipe, where a chain of two selects and one multiply-add put two instructions on
        // the integer/logic pipe that bounds this loop (0.1850 -> 0.1809 ms on the 1080p
        // frame, with the predicated intersect adds below 0.1789 ms).
        if (bx) r.bi = r.bi * one + r.sx;
        if (by) r.bi = r.bi * one + sy4;
        if (bz) r.bi = r.bi * one + sz16;
        // PTX's shr.b64 clamps a shift count above 63 to 64 (a zero result): no mask of bi is
        // needed.  bi leaves [0, 63] only in an empty box, where m is 0, or on a step out of
        // the box, which the box test takes first.
        uint64_t mb;
        asm("shr.b64 %0, %1, %2;" : "=l"(mb) : "l"(r.m), "r"(r.bi));
        const bool hb = mb & 1;
        if (((r.kx | r.ky | r.kz) < 0) | hb | last) {
            const int a = bx ? 0 : (by ? 1 : 2);
            const bool out = (r.kx | r.ky | r.kz) < 0;
            const int left = r.lb + r.kx + r.ky + r.kz;
            left_end = left;
            if (out) {
                if (COUNT) refills++;  // box lookups, counted only for launches that report counters
                const int cx = r.ex - r.sx * r.kx, cy = r.ey - r.sy * r.ky, cz = r.ez - r.sz * r.kz;
                const int t = DF ? enter_box(r, cx, cy, cz, P, alive, clip_k, left)
                                 : enter_box_lean(r, cx, cy, cz, P, clip_k, left);
                result = t;  // T_LIVE, T_HIT or T_MISS, taken as is: no branch on it
                hit_index = t == T_HIT ? cx + P.L.W * cy + P.L.W * P.L.H * cz : hit_index;
            } else if (hb) {
                result = T_HIT;
                const int cx = r.ex - r.sx * r.kx, cy = r.ey - r.sy * r.ky, cz = r.ez - r.sz * r.kz;
                hit_index = cx + P.L.W * cy + P.L.W * P.L.H * cz;
            } else {
                result = T_MISS;  // DF: the float cap, this was the last iteration
            }
            if (DF && result == T_HIT) {
                const int32_t v = __ldg(P.words + hit_index);
                if (v < 0) {  // a depth-field word: jump (fshader.glsl:114-121)
                    const float toJump = -__int_as_float(v);
                    travelled = fadd(travelled, toJump);
                    const float cdj = fadd(a == 0 ? r.tx : (a == 1 ? r.ty : r.tz), toJump);
                    start = add3(mul3s(d, cdj), start);
                    const int ncx = f2i(start.x), ncy = f2i(start.y), ncz = f2i(start.z);
                    r.tx = fdiv(fsub((float)(ncx + (r.sx > 0)), start.x), d.x);
                    r.ty = fdiv(fsub((float)(ncy + (r.sy > 0)), start.y), d.y);
                    r.tz = fdiv(fsub((float)(ncz + (r.sz > 0)), start.z), d.z);
                    // no box yet: the first step from the new cell looks one up
                    r.kx = 0; r.ky = 0; r.kz = 0;
                    r.lb = left;
                    r.ex = ncx; r.ey = ncy; r.ez = ncz;
                    r.m = 0;
                    r.bi = 0;
                    hit_index = -1;
                    if (!(travelled < lim)) {
                        result = T_MISS;
                        break;
                    }
                    continue;  // the jump replaced this iteration's intersect add
                }
            }
            if (result != T_LIVE) {
                axis = a;
                cd = a == 0 ? r.tx : (a == 1 ? r.ty : r.tz);
                sgn = a == 0 ? r.sx : (a == 1 ? r.sy : r.sz);
                break;
            }
            if (DF ? last : left < 0) { result = T_MISS; break; }  // entered a box on the last iteration
        }
        // The intersect add of the stepped axis (the shader's one add per iteration), as
        // three adds predicated on the axis, written in PTX so that they stay predicated
        // instructions on the FMA pipe.  Plain conditional adds compile to branches (0.2055
        // ms on the 1080p frame), and adding -0.0 to the axes not stepped (exact, but a
        // select per axis on the integer/logic pipe) took 0.1850 ms; predicated: 0.1809 ms.
        // The axis not stepped keeps its value as is, exactly as in the shader.
        pred_fadd(r.tx, r.dx, bx);
        pred_fadd(r.ty, r.dy, by);
        pred_fadd(r.tz, r.dz, bz);
    }
    steps += left0 - left_end;  // left_end = left0 - 1 - (index of the breaking iteration)
    start_out = start;
    return result;
}

// cast_box for a ray that moves along every axis and whose set-up held only ordinary numbers
// (ray_setup_lean): practically all of them.  Such a ray only moves forward, so it is walked
// in coordinates mirrored where it moves backward: q = c, or M - 1 - c with M the padded size
// of the axis, a multiple of 4, so that bricks stay aligned.  Every step adds 1 to q, the rest
// of a brick is 3 - (q & 3), the far side of the clip box and the slot of a brick need no sign
// and no select, and the first cell is checked by one subtraction per axis.
// oct_k: per octant {far clip side of q per axis, the brick slot of q = 0}, then {near side of
// the world in q per axis, 63 ^ the bit flips of the mirrored axes}, from the host.
//
// The frame is bound by its instructions (86 % of the issue slots): on a 1080p frame of 191 M
// warp instructions, 3.7 M warp iterations took 22 each, 0.8 M lookups 80, and 65 K pixels'
// and 130 K rays' frame work the rest.  Mirrored, with the rays' reciprocals and quotients as
// rcp_near and div_by and the octants' constants from the host: 182 M, 203.6 -> 192.3 us; 4K
// grazing 574 -> 550, 64 views 4008 -> 3792, every side output of 853x479 89.4 -> 83.3.
// Three ways to step several axes at once while a whole warp is in empty boxes (74-88 % of
// the iterations, 1.8-2.4 steps a trip) lost by 1 to 25 %: the votes that keep the warp
// together cost more per lookup than the trips save.
template <bool COUNT>
__device__ __forceinline__ int cast_lean(const MaskParams& P, const int4* oct_k, const RaySetup& s, int n,
                                         int maxSteps, float& cd, int& axis, int& sgn, int& steps,
                                         int32_t& hit_index, unsigned& refills) {
    const Layout& L = P.L;
    float tx = s.tx, ty = s.ty, tz = s.tz;
    const int n0 = max(0, min(n, maxSteps));
    if (n0 == 0) return T_MISS;
    const int one = P.one, four = P.four, sixteen = P.sixteen;
    const int sx = s.sx, sy4 = s.sy * four, sz16 = s.sz * sixteen;  // the bit-index moves along x, y and z
    const int by_step = s.sy * L.BWp, bz_step = s.sz * L.BWp * L.BHp;
    const int oct = (sx > 0) | ((s.sy > 0) << 1) | ((s.sz > 0) << 2);
    int ex = sx > 0 ? s.cx : 4 * L.BWp - 1 - s.cx;
    int ey = s.sy > 0 ? s.cy : 4 * L.BHp - 1 - s.cy;
    int ez = s.sz > 0 ? s.cz : 4 * L.BWp - 1 - s.cz;
    int flip;
    {   // the first cell lies before the near side of the world: getVoxelIndex == -1
        const int4 near = oct_k[8 + oct];
        flip = near.w;
        const bool fx = (tx < ty) & (tx < tz), fy = (ty < tx) & (ty < tz);
        if (((ex + fx - near.x) | (ey + fy - near.y) | (ez + !(fx | fy) - near.z)) < 0) {
            steps += 1;
            return T_MISS;
        }
    }
    const int left0 = n0 - 1;
    int lb = left0, left_end = left0;
    int kx = 0, ky = 0, kz = 0;  // no box yet: the first step along any axis triggers a lookup
    uint64_t m = 0;
    int bi = 0, result = T_MISS;
#pragma unroll 2
    for (;;) {
        const bool bx = (tx < ty) & (tx < tz);
        const bool by = (ty < tx) & (ty < tz);
        const bool bz = !(bx | by);
        if (bx) kx = kx * one - 1;
        if (by) ky = ky * one - 1;
        if (bz) kz = kz * one - 1;
        if (bx) bi = bi * one + sx;
        if (by) bi = bi * one + sy4;
        if (bz) bi = bi * one + sz16;
        uint64_t mb;
        asm("shr.b64 %0, %1, %2;" : "=l"(mb) : "l"(m), "r"(bi));
        const bool hb = mb & 1;
        if (((kx | ky | kz) < 0) | hb) {
            const int left = lb + kx + ky + kz;
            left_end = left;
            const int qx = ex - kx, qy = ey - ky, qz = ez - kz;
            result = T_HIT;
            if ((kx | ky | kz) < 0) {
                if (COUNT) refills++;
                const int4 A = oct_k[oct];
                const int cx = A.x - qx, cy = A.y - qy, cz = A.z - qz;  // steps before the far clip side
                result = T_MISS;
                if ((cx | cy | cz) >= 0) {
                    const uint32_t slot = (uint32_t)(A.w + sx * (qx >> 2) + by_step * (qy >> 2) + bz_step * (qz >> 2));
                    m = __ldg(P.bricks + slot);
                    const int far4 = __ldg(P.bdir + (slot * 8u + oct));  // 4 cells per further brick of the cube
                    // floor(left / 3); on the last iteration (left = -1) the box does not matter
                    const int kmax = (int)__umulhi((unsigned)left, 0x55555556u);
                    const int rx = ~qx & 3, ry = ~qy & 3, rz = ~qz & 3;
                    kx = min(min(rx + far4, cx), kmax);
                    ky = min(min(ry + far4, cy), kmax);
                    kz = min(min(rz + far4, cz), kmax);
                    ex = qx + kx; ey = qy + ky; ez = qz + kz;
                    lb = left - (kx + ky + kz);
                    bi = (rx + four * ry + sixteen * rz) ^ flip;
                    result = ((m >> bi) & 1) ? T_HIT : T_LIVE;
                }
            }
            if (result != T_LIVE) {
                axis = bx ? 0 : (by ? 1 : 2);
                cd = bx ? tx : (by ? ty : tz);
                sgn = bx ? s.sx : (by ? s.sy : s.sz);
                const int x = sx > 0 ? qx : 4 * L.BWp - 1 - qx, y = s.sy > 0 ? qy : 4 * L.BHp - 1 - qy,
                          z = s.sz > 0 ? qz : 4 * L.BWp - 1 - qz;
                hit_index = x + L.W * y + L.W * L.H * z;
                break;
            }
            if (left < 0) { result = T_MISS; break; }  // entered a box on the last iteration
        }
        pred_fadd(tx, s.dx, bx);
        pred_fadd(ty, s.dy, by);
        pred_fadd(tz, s.dz, bz);
    }
    steps += left0 - left_end;  // left_end = left0 - 1 - (index of the breaking iteration)
    return result;
}

// ray_setup of a ray whose direction lies in div_by's range along every axis and that starts
// at 2^-60 <= o < 2^22 along each: the cell by a truncating add, reciprocals and quotients
// without the IEEE routines' range tests.  False, with nothing usable in s, for any other ray.
__device__ __forceinline__ bool ray_setup_lean(V3 o, V3 d, RaySetup& s) {
    const V3 b{fadd(d.x, 0.000001f), fadd(d.y, 0.000001f), fadd(d.z, 0.000001f)};
    const bool ok = all_within(d, kDivMinB, kDivMaxB) & all_within(b, kDivMinB, 2.5f) &
                    (min3_nan(o.x, o.y, o.z) >= kDivMinA) & (max3_nan(o.x, o.y, o.z) < 4194304.0f);
    s.sx = d.x > 0.0f ? 1 : -1; s.sy = d.y > 0.0f ? 1 : -1; s.sz = d.z > 0.0f ? 1 : -1;
    s.dx = rcp_near(fabsf(b.x)); s.dy = rcp_near(fabsf(b.y)); s.dz = rcp_near(fabsf(b.z));
    const float mx = __fadd_rz(o.x, 8388608.0f), my = __fadd_rz(o.y, 8388608.0f), mz = __fadd_rz(o.z, 8388608.0f);
    s.cx = __float_as_int(mx) - 0x4B000000; s.cy = __float_as_int(my) - 0x4B000000; s.cz = __float_as_int(mz) - 0x4B000000;
    s.tx = div_by(fsub(fsub(mx, s.sx > 0 ? 8388607.0f : 8388608.0f), o.x), d.x, rcp_near(d.x));
    s.ty = div_by(fsub(fsub(my, s.sy > 0 ? 8388607.0f : 8388608.0f), o.y), d.y, rcp_near(d.y));
    s.tz = div_by(fsub(fsub(mz, s.sz > 0 ? 8388607.0f : 8388608.0f), o.z), d.z, rcp_near(d.z));
    return ok;
}

template <bool DF, bool COUNT>
__device__ __forceinline__ int cast_ray(const MaskParams& P, const int2* alive, const int4* clip_k, const int4* oct_k,
                                        V3 o, V3 d, int n, int maxSteps, float& cd, int& axis, int& sgn, int& steps,
                                        int32_t& hit_index, unsigned& refills, V3& start_out) {
    RaySetup s;
    if (!DF && ray_setup_lean(o, d, s)) {
        start_out = o;
        return cast_lean<COUNT>(P, oct_k, s, n, maxSteps, cd, axis, sgn, steps, hit_index, refills);
    }
    ray_setup(o, d, s);
    return cast_box<DF, COUNT>(P, alive, clip_k, s, o, d, n, maxSteps, cd, axis, sgn, steps, hit_index, refills, start_out);
}

__device__ __forceinline__ int view_of_tile(const MaskParams& P, int t) {
    if (P.nviews == 1) return 0;
    int lo = 0, hi = P.nviews - 1;
    while (lo < hi) {  // the last view whose first tile is <= t
        const int mid = (lo + hi + 1) >> 1;
        if (P.views[mid].tile_begin <= t) lo = mid;
        else hi = mid - 1;
    }
    return lo;
}

// One CTA per ray tile (tile_w x tile_h pixels, tile_w*tile_h == blockDim.x) over the tile
// space of every view of the launch: a single frame, or a batch of cameras of any sizes.
// EXACT launches (any view asking for step counts) step every ray to its end; DEBUG
// launches (any view with a debug output or counters) write the per-pixel side outputs
// and count box lookups; DF launches render a world with depth-field words (the masks are
// its stop masks).
template <bool EXACT, bool DEBUG, bool DF>
// A minimum of 7 CTAs of 128 threads per SM lets the compiler use up to 73 registers; it takes
// 63 or 64 for every variant (so 8 CTAs still fit per SM), and the code it makes for the
// unrolled loop is faster than under a minimum of 8 (1080p frame 0.1706 against 0.1727 ms, the
// stress camera 0.423 against 0.427 ms when measured).
__global__ void __launch_bounds__(128, 7) render_tiles_kernel(const __grid_constant__ MaskParams P) {
    __shared__ int2 alive[24];  // read by enter_box, i.e. only with depth-field words
    __shared__ int4 clip_s[27];  // enter_box's octants
    __shared__ int4 oct_k[16];   // cast_lean's constants
    cudaTriggerProgrammaticLaunchCompletion();  // see frame_launch
    const int4* clip_k = DF ? clip_s : P.clip_k;
    if (DF) {
        fill_alive_ranges(alive, P, EXACT);
        if (threadIdx.x < 27) clip_s[threadIdx.x] = P.clip_k[threadIdx.x];
    } else if (threadIdx.x < 16) {
        oct_k[threadIdx.x] = P.oct_k[threadIdx.x];
    }
    __syncthreads();
    const int tile = (int)blockIdx.x + P.tile0;
    const ViewDev& V = view_of(P, view_of_tile(P, tile));
    const int lt = tile - V.tile_begin;
    int px, py;
    V.map.pixel(lt, (int)threadIdx.x, px, py);
    const bool valid = px < V.width && py < V.height;
    PixelResult res{};
    unsigned refills = 0;
    const vrt_uniforms& u = V.u;
    const V3 cam{u.camPos[0], u.camPos[1], u.camPos[2]};
    V3 rd{0.f, 0.f, 0.f};
    float cd = 0.f, c2 = 0.f;
    int axis = 2, sgn = 0, steps = 0, a2 = 0, s2 = 0;
    int32_t hit = -1, dummy = -1;
    int pr = T_MISS;
    V3 from = cam, from2;  // the start a hit position is measured from (moved by depth-field jumps)
    if (valid) {
        rd = primary_dir(u, px, py, V.width, V.height, V.map.inv_w, V.map.inv_h);
        pr = cast_ray<DF, DEBUG>(P, alive, clip_k, oct_k, cam, rd, u.maxSteps, u.maxSteps, cd, axis, sgn, steps, hit, refills, from);
        res.primary_steps = steps;
    }
    const bool lit = valid && pr == T_HIT && u.viewDepthField != 1;
    const V3 hp = lit ? add3(mul3s(rd, cd), from) : V3{0.f, 0.f, 0.f};
    const unsigned cand = warp_light_candidates(u, lit, hp);
    if (valid) {
        float mr = u.ambient, mg = u.ambient, mb = u.ambient;
        int32_t word = 0;
        if (u.viewDepthField == 1) {
            mr = mg = mb = fdiv((float)steps, 100.0f);
        } else if (pr == T_HIT) {
            const V3 hn = axis_normal(axis, sgn);
            const float ob = u.maxOverbright, R = u.localLightDist;
            // R1 = |R|(1 + 2^-10) + 1 exceeds R by more than the rounding of any computed length
            const float R1 = fadd(fmul(fabsf(R), 1.0009765625f), 1.0f);
            // The shadow rays in the shader's order, through one traversal call site: j = -1
            // is the global light (fshader.glsl:147-156), then the warp's candidate local
            // lights in ascending order (:159-181).  The shader tests for overbright before
            // every local light; the colour changes only at lights that are cast, so testing
            // before each candidate, and once more after the last candidate if the shader's
            // loop had iterations left, gives the same clamp.
            unsigned todo = cand;
            int last = -1;
            bool clamped = false;
            for (int j = -1;;) {
                V3 dir{0.f, 0.f, 0.f};
                int n = 0;
                float ld = 0.f;
                bool cast = true;
                if (j < 0) {
                    dir = norm3(sub3(V3{u.lightPos[0], u.lightPos[1], u.lightPos[2]}, hp));
                    n = u.maxSteps;
                } else {
                    if (mr >= ob && mg >= ob && mb >= ob) {
                        mr = mg = mb = ob;
                        clamped = true;
                        break;
                    }
                    const float* Lj = u.localLights[j];
                    const V3 dl = sub3(V3{Lj[0], Lj[1], Lj[2]}, hp);
                    // a component beyond R1 puts the computed length beyond R too: out of range
                    cast = !(fabsf(dl.x) > R1 || fabsf(dl.y) > R1 || fabsf(dl.z) > R1);
                    if (cast) {
                        ld = len3(dl);
                        cast = ld <= R;
                    }
                    if (cast) {
                        dir = norm3(dl);
                        n = f2i(fadd(ld, 1.0f));
                    }
                }
                if (cast) {
                    const int sr = cast_ray<DF, DEBUG>(P, alive, clip_k, oct_k, add3(hp, mul3s(dir, 0.001f)), dir, n, u.maxSteps, c2, a2,
                                                s2, steps, dummy, refills, from2);
                    const unsigned bit = 1u << (j + 1);
                    res.cast |= bit;
                    if (sr == T_HIT) {
                        res.occ |= bit;
                    } else {
                        const float nl = fmax0(dot3(hn, dir));
                        if (j < 0) {
                            const float c = fmul(u.diffuse, nl);
                            mr = fadd(mr, c); mg = fadd(mg, c); mb = fadd(mb, c);
                        } else {
                            const float fall = fdiv(fsub(R, ld), R);
                            const float a = u.localLights[j][3];
                            mr = fadd(mr, fmul(fmul(fmul(a, u.localLightColor[j][0]), nl), fall));
                            mg = fadd(mg, fmul(fmul(fmul(a, u.localLightColor[j][1]), nl), fall));
                            mb = fadd(mb, fmul(fmul(fmul(a, u.localLightColor[j][2]), nl), fall));
                        }
                    }
                }
                if (!todo) break;
                j = __ffs(todo) - 1;
                todo &= todo - 1;
                last = j;
            }
            if (!clamped && last < VRT_MAX_LOCAL_LIGHTS - 1 && mr >= ob && mg >= ob && mb >= ob) mr = mg = mb = ob;
            word = __ldg(P.words + hit);
        }
        res.hit = pr == T_HIT ? hit : -1;
        res.steps = steps;
        res.mr = mr; res.mg = mg; res.mb = mb;
        res.rgba = pack_color_tab(u, pr == T_HIT, word, mr, mg, mb, res.primary_steps);
    }
    cudaGridDependencySynchronize();  // nothing is written before the frame ahead has ended
    if (valid) {
        if (DEBUG) store_pixel(V.dbg, V.rgba, (uint64_t)py * V.width + px, res);
        else reinterpret_cast<uint32_t*>(V.rgba)[(uint64_t)py * V.width + px] = res.rgba;
    }
    if (V.stats) {
        unsigned rays = valid ? 1u + __popc(res.cast) : 0u;
        unsigned hits = valid && res.hit >= 0 ? 1u : 0u;
        unsigned pix = valid ? 1u : 0u;
        unsigned long long s64 = valid ? (unsigned)res.steps : 0u;
        unsigned long long r64 = refills;
        for (int off = 16; off > 0; off >>= 1) {
            s64 += __shfl_down_sync(0xffffffffu, s64, off);
            r64 += __shfl_down_sync(0xffffffffu, r64, off);
        }
        rays = __reduce_add_sync(0xffffffffu, rays);
        hits = __reduce_add_sync(0xffffffffu, hits);
        pix = __reduce_add_sync(0xffffffffu, pix);
        if ((threadIdx.x & 31) == 0) {
            atomicAdd(V.stats + VRT_STAT_RAYS, (unsigned long long)rays);
            atomicAdd(V.stats + VRT_STAT_STEPS, s64);
            atomicAdd(V.stats + VRT_STAT_HITS, (unsigned long long)hits);
            atomicAdd(V.stats + VRT_STAT_PIXELS, (unsigned long long)pix);
            atomicAdd(V.stats + VRT_STAT_REFILLS, r64);
        }
    }
}

// ====================================================================== L2 probe

__global__ void l2_read_kernel(const uint4* __restrict__ buf, size_t n16, int iters, unsigned* sink) {
    unsigned acc = 0;
    size_t stride = (size_t)gridDim.x * blockDim.x;
    for (int it = 0; it < iters; it++)
        for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < n16; i += stride) {
            uint4 v = __ldcg(buf + i);
            acc ^= v.x ^ v.y ^ v.z ^ v.w;
        }
    if (acc == 0x9e3779b9u) *sink = acc;  // keeps the loads alive
}

}  // namespace vrt

// ====================================================================== host side

using namespace vrt;

struct vrt_renderer {
    int device = 0;
    int num_sms = 0;
    ViewDev* d_views = nullptr;
    int views_cap = 0;
    unsigned int* d_counter = nullptr;
    uint8_t* d_staging = nullptr;
    size_t staging_bytes = 0;
    cudaStream_t copy_stream = nullptr;   // vrt_render_to_host: band copies
    cudaStream_t band_stream[8] = {};     // vrt_render_to_host: one render stream per band
    cudaEvent_t start = nullptr;          // the caller's stream reached the render
    cudaEvent_t band_done[8] = {};        // a band's render finished
    cudaEvent_t copies_done = nullptr;    // the last band copy finished (copy stream)
    // word kernel tile order: 3 x kTileClasses counts, 2 x kTileClasses lists of tile_cap tiles
    int* d_class_count = nullptr;
    int* d_class_list = nullptr;
    int tile_cap = 0;
    int tile_gx = 0, tile_gy = 0;         // the grid of the frames recorded (0: none)
    uint64_t tile_frames = 0;             // word-kernel frames that recorded classes on that grid
    int tile_reuses = 0;                  // frames since then that went by the same classes
    // the last frame's world (its stamp) and stream: see frame_launch
    std::mutex seen_mu;
    uint64_t seen_stamp = 0;
    cudaStream_t seen_stream = nullptr;
};

struct Tuning {
    int tile_w, tile_h, refill_min, blocks_per_sm, exact_steps;
};

struct vrt_batch_graph {
    cudaGraph_t graph = nullptr;
    cudaGraphExec_t exec = nullptr;
    ViewDev* d_views = nullptr;
    unsigned int* d_counter = nullptr;
    cudaStream_t capture_stream = nullptr;
    // what the launch was captured from, for the next capture: its parameters hold the world's solid box
    const vrt_world* world = nullptr;
    int box[6] = {};
    std::vector<ViewDev> views;
    int total = 0;
    Tuning t{};
    bool tiles = true;
    vrt_renderer shape;  // only its device and SM count are read
};

static inline cudaStream_t S(void* s) { return reinterpret_cast<cudaStream_t>(s); }

// The shader counts the distance a ray travelled in a float (fshader.glsl:82-85), which
// stops growing at 2^24: a ray stuck on a zero direction component would never reach a
// larger cap, so caps above 2^24 are refused.
constexpr int kMaxSteps = 1 << 24;

static int check_uniforms(const vrt_uniforms* u) {
    if (!u) return set_error(VRT_EINVAL, "NULL uniforms");
    if (u->maxSteps < 0 || u->maxSteps > kMaxSteps)
        return set_error(VRT_EINVAL, "maxSteps %d outside [0, 2^24]", u->maxSteps);
    return VRT_OK;
}

static Tuning tuning_of(const vrt_render_opts* o) {
    Tuning t{8, 4, 8, 4, 0};
    if (o) {
        t.exact_steps = o->exact_steps != 0;
        if (o->tile_w > 0) t.tile_w = o->tile_w;
        if (o->tile_h > 0) t.tile_h = o->tile_h;
        if (o->refill_min > 0) t.refill_min = std::min(o->refill_min, 32);
        if (o->blocks_per_sm > 0) t.blocks_per_sm = std::min(o->blocks_per_sm, 8);
    }
    return t;
}

// Ray tiles of the tile kernel: one CTA each, tile_w * tile_h threads (a multiple of 32,
// at most 128); 8x16 unless the options name another shape (the fastest of 8x4 ... 128x1
// on the 1080p frame; 8x8 ties).
static int tile_tuning(const vrt_render_opts* o, Tuning* t) {
    *t = tuning_of(o);
    if (!o || o->tile_w <= 0 || o->tile_h <= 0) {
        t->tile_w = 8;
        t->tile_h = 16;
    }
    const int n = t->tile_w * t->tile_h;
    if (n % 32 != 0 || n > 128)
        return set_error(VRT_EINVAL, "ray tile %dx%d: tile_w*tile_h must be a multiple of 32 up to 128", t->tile_w,
                         t->tile_h);
    return VRT_OK;
}

// Region distances go to shared memory when they take at most this many bytes
// (16 KiB for 512x256x512, 4 KiB for 256^3); larger worlds read them through L1.
constexpr int kSmemRegionLimit = 32768;

static int launch_mask(vrt_renderer* r, const vrt_world* w, const ViewDev* h_views, int nviews, int total_tiles,
                       const Tuning& t, const ViewDev* d_views, unsigned int* d_counter, cudaStream_t s) {
    MaskParams P;
    std::memset(&P, 0, sizeof(P));
    P.words = w->d_words;
    P.bricks = w->d_bricks;
    P.bdir = w->d_bdir;
    P.rdist = w->d_rdist;
    std::memcpy(P.bb, w->h_aabb, sizeof(P.bb));
    P.one = 1; P.four = 4; P.sixteen = 16;
    P.L = w->L;
    P.views = nviews == 1 ? nullptr : d_views;
    P.nviews = nviews;
    P.total_tiles = total_tiles;
    P.tile_counter = d_counter;
    P.v0 = h_views[0];
    const int region_bytes = w->L.RWp * w->L.RHp * w->L.RWp;
    P.region_bytes16 = (region_bytes + 15) & ~15;
    const bool smem_regions = P.region_bytes16 <= kSmemRegionLimit;
    const size_t smem = (smem_regions ? P.region_bytes16 : 0) + sizeof(uint32_t) * NF * kThreads;
    // 4 CTAs/SM caps registers at 64, 3 CTAs/SM at 85 (no spills); blocks_per_sm picks
    auto kern = t.blocks_per_sm >= 4 ? (smem_regions ? render_mask_kernel<true, 4> : render_mask_kernel<false, 4>)
                                     : (smem_regions ? render_mask_kernel<true, 3> : render_mask_kernel<false, 3>);
    VRT_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    int per_sm = 0;
    VRT_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, kThreads, smem));
    per_sm = std::max(1, std::min(per_sm, t.blocks_per_sm));
    VRT_CUDA(cudaMemsetAsync(d_counter, 0, sizeof(unsigned), s));
    // persistent grid: per_sm CTAs of 8 warps per SM, never more warps than tiles
    const int blocks = std::max(1, std::min(r->num_sms * per_sm, (total_tiles + 7) / 8));
    kern<<<blocks, kThreads, smem, s>>>(P);
    VRT_CUDA(cudaGetLastError());
    return VRT_OK;
}

// How a frame's kernel is launched.  A frame is bound by its longest chains: the SMs stand idle
// from where the first runs out of tiles to the next launch, 5 % of a 1080p frame, 11 % of a
// 4K frame along the ground, 15 of the 54 us of the app's first frame, 4 of the 13 us of a
// 256x256 one, and 2 us of launch each.  So a frame of the world that the stream's last frame
// showed, unchanged since (its stamp), is a programmatic dependent of that one: its CTAs begin
// as soon as all of the frame ahead have begun.  What they read was there before both frames (a
// frame that waits for a change first lets the next begin only behind that wait);
// what they write waits for the end of the frame ahead (cudaGridDependencySynchronize, behind the
// trace), so images, counters and whatever follows on the stream see the frames one after the
// other.  Frames in a row, each alone before: 256x256 16.9 -> 7.4 us, 1080p 192.5 -> 184.2, 4K
// 551 -> 544 (the CTAs that wait hold their places), the app's first frame 58.9 -> 38.4, the
// 800x600 level frame with three lights 65.8 -> 47.8 us.
// Any other frame waits for all ahead.  The word kernel is a dependent then too and waits before
// its first access, as edits do (launch_behind): probe, edit and frame 80.1 -> 77.0 us.  It reads
// the words by plain loads therefore.  (The tile kernel's loads stay on the read-only path.)
// A captured launch is a plain one, and is not taken for the stream's last frame; the streams
// of cudaStreamPerThread share a handle, so theirs overlap nothing.
enum { kPlainFrame, kOverlappedFrame, kCapturedFrame };
static int frame_launch(vrt_renderer* r, const vrt_world* w, cudaStream_t s) {
    cudaStreamCaptureStatus capture = cudaStreamCaptureStatusNone;
    if (cudaStreamIsCapturing(s, &capture) != cudaSuccess || capture != cudaStreamCaptureStatusNone) {
        cudaGetLastError();
        return kCapturedFrame;
    }
    if (w->stamp == 0 || s == cudaStreamPerThread) return kPlainFrame;
    std::lock_guard<std::mutex> lock(r->seen_mu);
    return r->seen_stamp == w->stamp && r->seen_stream == s ? kOverlappedFrame : kPlainFrame;
}

template <class... Params, class... Args>
static cudaError_t launch_frame(vrt_renderer* r, const vrt_world* w, int how, bool behind, void (*kern)(Params...),
                                dim3 grid, int threads, cudaStream_t s, const Args&... args) {
    const cudaError_t e = launch_behind(behind, kern, grid, threads, s, args...);
    if (how != kCapturedFrame) {
        std::lock_guard<std::mutex> lock(r->seen_mu);
        r->seen_stamp = e == cudaSuccess ? w->stamp : 0;
        r->seen_stream = s;
    }
    return e;
}

// Tile kernel launch over the views' tile space (1 view: h_views[0] as a parameter).
static int launch_tiles(const vrt_world* w, const ViewDev* h_views, int nviews, int total_tiles,
                        const ViewDev* d_views, int threads, cudaStream_t s, int tile0 = 0, int ntiles = -1,
                        bool count_lookups = true, vrt_renderer* frame_of = nullptr) {
    MaskParams P;
    std::memset(&P, 0, sizeof(P));
    P.words = w->d_words;
    P.bricks = w->d_bricks;
    P.bdir = w->d_bdir;
    P.rdist = w->d_rdist;
    std::memcpy(P.bb, w->h_aabb, sizeof(P.bb));
    P.one = 1; P.four = 4; P.sixteen = 16;
    P.L = w->L;
    P.views = nviews == 1 ? nullptr : d_views;
    P.nviews = nviews;
    P.total_tiles = total_tiles;
    P.v0 = h_views[0];
    bool exact = false;
    for (int i = 0; i < nviews; i++) exact |= h_views[i].exact != 0;
    const int dims[3] = {w->L.W, w->L.H, w->L.W};
    for (int a = 0; a < 3; a++) {
        P.cl[a] = exact ? 0 : std::max(0, std::min(P.bb[a], dims[a]));
        P.cl[3 + a] = exact ? dims[a] : std::min(dims[a], std::max(P.bb[3 + a] + 1, P.cl[a]));
    }
    for (int t = 0; t < 27; t++) {
        const int sx = t % 3 - 1, sy = (t / 3) % 3 - 1, sz = t / 9 - 1;
        P.clip_k[t] = make_int4(sx > 0 ? P.cl[3] - 1 : (sx < 0 ? -P.cl[0] : INT_MAX),
                                sy > 0 ? P.cl[4] - 1 : (sy < 0 ? -P.cl[1] : INT_MAX),
                                sz > 0 ? P.cl[5] - 1 : (sz < 0 ? -P.cl[2] : INT_MAX),
                                (sx > 0) | ((sy > 0) << 1) | ((sz > 0) << 2));
    }
    const int mx = 4 * P.L.BWp, my = 4 * P.L.BHp;
    for (int o = 0; o < 8; o++) {
        const bool x = o & 1, y = o & 2, z = o & 4;
        P.oct_k[o] = make_int4(x ? P.cl[3] - 1 : mx - 1 - P.cl[0], y ? P.cl[4] - 1 : my - 1 - P.cl[1],
                               z ? P.cl[5] - 1 : mx - 1 - P.cl[2],
                               (x ? 0 : P.L.BWp - 1) + (y ? 0 : P.L.BWp * (P.L.BHp - 1)) +
                                   (z ? 0 : P.L.BWp * P.L.BHp * (P.L.BWp - 1)));
        P.oct_k[8 + o] = make_int4(x ? 0 : mx - P.L.W, y ? 0 : my - P.L.H, z ? 0 : mx - P.L.W,
                                   (x ? 3 : 0) | (y ? 12 : 0) | (z ? 48 : 0));
    }
    // DEBUG launches store side outputs and count box lookups: any view with a debug output
    // or counters (whoever reads no more of the counters than rays, hits and pixels can do
    // without the lookups: count_lookups)
    bool debug = false;
    for (int i = 0; i < nviews; i++) {
        const vrt_debug_out& d = h_views[i].dbg;
        debug |= d.hit_index || d.cast_mask || d.occ_mask || d.steps || d.primary_steps || d.shade ||
                 (count_lookups && h_views[i].stats != nullptr);
    }
    const bool df = w->has_depth_field != 0;
    if (df) {
        // the stop masks are a cache of the words, rebuilt here after any change
        const int st = refresh_stop(const_cast<vrt_world*>(w), s);
        if (st) return st;
        P.bricks = w->d_stop;
        P.bdir = w->d_sdir;
    }
    using Kern = void (*)(MaskParams);
    static const Kern kernels[2][2][2] = {
        {{render_tiles_kernel<false, false, false>, render_tiles_kernel<false, false, true>},
         {render_tiles_kernel<false, true, false>, render_tiles_kernel<false, true, true>}},
        {{render_tiles_kernel<true, false, false>, render_tiles_kernel<true, false, true>},
         {render_tiles_kernel<true, true, false>, render_tiles_kernel<true, true, true>}}};
    const Kern kern = kernels[exact][debug][df];
    P.tile0 = tile0;
    if (ntiles < 0) ntiles = total_tiles - tile0;
    if (frame_of) {  // a renderer's whole frame
        const int how = frame_launch(frame_of, w, s);
        VRT_CUDA(launch_frame(frame_of, w, how, how == kOverlappedFrame, kern, dim3(ntiles), threads, s, P));
        return VRT_OK;
    }
    if (ntiles > 0) kern<<<ntiles, threads, 0, s>>>(P);
    VRT_CUDA(cudaGetLastError());
    return VRT_OK;
}

static void fill_view(ViewDev& v, const vrt_uniforms& u, int width, int height, uint8_t* rgba,
                      const vrt_debug_out* dbg, uint64_t* stats, const Tuning& t, int tile_begin) {
    std::memset(&v, 0, sizeof(v));
    v.u = u;
    v.width = width;
    v.height = height;
    v.map = tile_map(width, height, t.tile_w, t.tile_h);
    v.refill_min = t.refill_min;
    v.tile_begin = tile_begin;
    v.rgba = rgba;
    if (dbg) v.dbg = *dbg;
    v.stats = reinterpret_cast<unsigned long long*>(stats);
    v.exact = t.exact_steps || u.viewDepthField == 1 || (dbg && (dbg->steps || dbg->primary_steps));
}

static inline int tiles_of(int width, int height, const Tuning& t) {
    return ((width + t.tile_w - 1) / t.tile_w) * ((height + t.tile_h - 1) / t.tile_h);
}

static int ensure_views(vrt_renderer* r, int n) {
    if (n <= r->views_cap) return VRT_OK;
    if (r->d_views) cudaFree(r->d_views);
    r->d_views = nullptr;
    r->views_cap = 0;
    cudaError_t e = cudaMalloc(&r->d_views, sizeof(ViewDev) * (size_t)n);
    if (e != cudaSuccess) return set_error(VRT_ENOMEM, "views: %s", cudaGetErrorString(e));
    r->views_cap = n;
    return VRT_OK;
}

extern "C" {

// Fill g_div255 on the current device once; every tile-kernel launch goes through a renderer.
static int ensure_div255(int device) {
    static std::mutex mu;
    static bool done[64] = {};
    std::lock_guard<std::mutex> lock(mu);
    if (device >= 0 && device < 64 && done[device]) return VRT_OK;
    init_div255_kernel<<<1, 256>>>();
    VRT_CUDA(cudaGetLastError());
    VRT_CUDA(cudaDeviceSynchronize());  // later launches may run on any stream
    if (device >= 0 && device < 64) done[device] = true;
    return VRT_OK;
}

int vrt_renderer_create(vrt_renderer** out) {
    if (!out) return set_error(VRT_EINVAL, "out is NULL");
    *out = nullptr;
    vrt_renderer* r = new vrt_renderer();
    cudaError_t e = cudaGetDevice(&r->device);
    if (e == cudaSuccess) e = cudaDeviceGetAttribute(&r->num_sms, cudaDevAttrMultiProcessorCount, r->device);
    if (e == cudaSuccess) e = cudaMalloc(&r->d_counter, 256);
    if (e == cudaSuccess) e = cudaMemset(r->d_counter, 0, 256);
    if (e != cudaSuccess) {
        cudaFree(r->d_counter);
        delete r;
        return cuda_error(e, "vrt_renderer_create");
    }
    const int st = ensure_div255(r->device);
    if (st) {
        cudaFree(r->d_counter);
        delete r;
        return st;
    }
    *out = r;
    return VRT_OK;
}

int vrt_renderer_destroy(vrt_renderer* r) {
    if (!r) return VRT_OK;
    cudaFree(r->d_views);
    cudaFree(r->d_counter);
    cudaFree(r->d_staging);
    cudaFree(r->d_class_count);
    cudaFree(r->d_class_list);
    if (r->copy_stream) cudaStreamDestroy(r->copy_stream);
    for (cudaStream_t b : r->band_stream)
        if (b) cudaStreamDestroy(b);
    for (cudaEvent_t e : r->band_done)
        if (e) cudaEventDestroy(e);
    if (r->start) cudaEventDestroy(r->start);
    if (r->copies_done) cudaEventDestroy(r->copies_done);
    delete r;
    return VRT_OK;
}

// The tile-order buffers of a word-kernel launch over grid g.  Frame f of a grid reads the
// classes frame f-1 wrote (count buffer f%3, lists f%2), appends to count buffer (f+1)%3
// and lists (f+1)%2, and clears count buffer (f+2)%3 for frame f+1: that buffer was last
// read by frame f-1, which ended before frame f began (one stream per renderer).  These are the
// frames that begin when all before has ended.  One that overlaps the frame ahead goes by the
// same classes as the last of these, which are not written to until the next, and records
// none; every 32nd frame at least is a whole one, so that the classes follow a moving camera.
// The order only speeds frames up: without room for its buffers, and captured into a graph
// (whose runs would append to the same lists), the launch runs in row order.
static int word_tile_order(vrt_renderer* r, dim3 g, cudaStream_t s, int* how, WordParams* p) {
    const int nt = (int)(g.x * g.y);
    p->tiles = nt;
    p->class_count_in = nullptr;
    p->class_list_in = nullptr;
    p->class_count_out = nullptr;
    p->class_list_out = nullptr;
    p->class_count_clear = nullptr;
    if (*how == kCapturedFrame) return VRT_OK;
    if (nt > r->tile_cap) {
        cudaFree(r->d_class_count);
        cudaFree(r->d_class_list);
        r->d_class_list = nullptr;
        r->tile_cap = 0;
        cudaError_t e = cudaMalloc(&r->d_class_count, 3 * kTileClasses * sizeof(int));
        if (e == cudaSuccess) e = cudaMalloc(&r->d_class_list, (size_t)2 * kTileClasses * nt * sizeof(int));
        if (e != cudaSuccess) {
            cudaGetLastError();
            cudaFree(r->d_class_count);
            cudaFree(r->d_class_list);
            r->d_class_count = nullptr;
            r->d_class_list = nullptr;
            r->tile_gx = r->tile_gy = 0;
            return VRT_OK;  // row order
        }
        r->tile_cap = nt;
        r->tile_gx = r->tile_gy = 0;
    }
    if (r->tile_gx != (int)g.x || r->tile_gy != (int)g.y) {  // a new grid: no classes yet
        VRT_CUDA(cudaMemsetAsync(r->d_class_count, 0, 3 * kTileClasses * sizeof(int), s));
        r->tile_gx = (int)g.x;
        r->tile_gy = (int)g.y;
        r->tile_frames = 0;
    }
    int* counts = r->d_class_count;
    int* lists = r->d_class_list;
    const size_t list = (size_t)kTileClasses * nt;
    if (*how == kOverlappedFrame && (r->tile_frames < 2 || r->tile_reuses >= kClassReuses)) *how = kPlainFrame;
    // an overlapped frame reads what the last plain one read, which was whole before that one began
    const uint64_t f = *how == kOverlappedFrame ? r->tile_frames - 1 : r->tile_frames;
    p->class_count_in = f > 0 ? counts + (f % 3) * kTileClasses : nullptr;
    p->class_list_in = f > 0 ? lists + (f % 2) * list : nullptr;
    if (*how == kOverlappedFrame) return VRT_OK;
    p->class_count_out = counts + ((f + 1) % 3) * kTileClasses;
    p->class_list_out = lists + ((f + 1) % 2) * list;
    p->class_count_clear = counts + ((f + 2) % 3) * kTileClasses;
    return VRT_OK;
}

int vrt_render(vrt_renderer* r, const vrt_world* w, const vrt_uniforms* u, int32_t width, int32_t height,
               uint8_t* d_rgba, const vrt_debug_out* dbg, uint64_t* d_stats, const vrt_render_opts* opts,
               void* stream) {
    if (!r || !w || !d_rgba) return set_error(VRT_EINVAL, "NULL renderer, world or image");
    if ((uintptr_t)d_rgba & 3)
        return set_error(VRT_EINVAL, "image address not 4-byte aligned (one 32-bit store per pixel)");
    int st = check_uniforms(u);
    if (st) return st;
    if (width < 1 || height < 1 || width > 32768 || height > 32768)
        return set_error(VRT_EINVAL, "image %d x %d out of range", width, height);
    int kernel = opts ? opts->kernel : VRT_KERNEL_AUTO;
    if (kernel == VRT_KERNEL_AUTO) kernel = w->has_depth_field ? VRT_KERNEL_WORD : VRT_KERNEL_MASK_PIXEL;
    if (kernel == VRT_KERNEL_BITMASK && w->has_depth_field)
        return set_error(VRT_ESTATE, "the world holds depth-field words, which only the word kernel follows");
    if (kernel == VRT_KERNEL_WORD) {
        WordParams p;
        std::memset(&p, 0, sizeof(p));
        p.u = *u;
        p.width = width;
        p.height = height;
        p.rgba = d_rgba;
        if (dbg) p.dbg = *dbg;
        p.stats = reinterpret_cast<unsigned long long*>(d_stats);
        std::memcpy(p.bb, w->h_aabb, sizeof(p.bb));
        p.exact = (opts && opts->exact_steps) || u->viewDepthField == 1 || (dbg && (dbg->steps || dbg->primary_steps));
        // 16x8 pixels per CTA unless the options name another tile (a multiple of 32 threads, at most 128)
        const int tw = opts && opts->tile_w > 0 && opts->tile_h > 0 ? opts->tile_w : 16;
        const int th = opts && opts->tile_w > 0 && opts->tile_h > 0 ? opts->tile_h : 8;
        const int threads = tw * th;
        if (threads % 32 != 0 || threads > 128)
            return set_error(VRT_EINVAL, "pixel tile %dx%d: tile_w*tile_h must be a multiple of 32 up to 128", tw, th);
        p.map = tile_map(width, height, tw, th);
        dim3 grid((width + tw - 1) / tw, (height + th - 1) / th);
        // the z-major copy of the words is a cache of them, brought up to date here
        st = refresh_words_z(const_cast<vrt_world*>(w), S(stream));
        if (st) return st;
        p.words = w->d_words;
        p.words_z = w->d_words_z;
        int how = frame_launch(r, w, S(stream));
        st = word_tile_order(r, grid, S(stream), &how, &p);
        if (st) return st;
        p.wait_first = how == kPlainFrame;
        const bool debug = dbg && (dbg->hit_index || dbg->cast_mask || dbg->occ_mask || dbg->steps ||
                                   dbg->primary_steps || dbg->shade);
        const cudaError_t le = launch_frame(r, w, how, how != kCapturedFrame && w->stamp != 0, debug ? render_word_kernel<true> : render_word_kernel<false>,
                                            grid, threads, S(stream), (const int32_t*)w->d_words, w->L, p);
        if (le != cudaSuccess) {
            cudaGetLastError();
            r->tile_gx = r->tile_gy = 0;  // the classes of this frame were not written
            return cuda_error(le, "render_word_kernel");
        }
        if (how == kOverlappedFrame) {
            r->tile_reuses++;
        } else if (how == kPlainFrame) {
            r->tile_frames++;
            r->tile_reuses = 0;
        }
        return VRT_OK;
    }
    if (kernel == VRT_KERNEL_MASK_PIXEL) {  // follows depth-field jumps too
        Tuning t;
        int st = tile_tuning(opts, &t);
        if (st) return st;
        ViewDev v;
        fill_view(v, *u, width, height, d_rgba, dbg, d_stats, t, 0);
        return launch_tiles(w, &v, 1, tiles_of(width, height, t), nullptr, t.tile_w * t.tile_h, S(stream), 0, -1, true, r);
    }
    if (kernel != VRT_KERNEL_BITMASK) return set_error(VRT_EINVAL, "unknown kernel %d", kernel);
    Tuning t = tuning_of(opts);
    ViewDev v;
    fill_view(v, *u, width, height, d_rgba, dbg, d_stats, t, 0);
    return launch_mask(r, w, &v, 1, tiles_of(width, height, t), t, nullptr, r->d_counter, S(stream));
}

int vrt_host_alloc(size_t bytes, void** out) {
    if (!out) return set_error(VRT_EINVAL, "out is NULL");
    *out = nullptr;
    if (bytes == 0) return VRT_OK;
    cudaError_t e = cudaMallocHost(out, bytes);
    if (e != cudaSuccess) {
        *out = nullptr;
        return e == cudaErrorMemoryAllocation ? set_error(VRT_ENOMEM, "pinned host buffer of %zu bytes", bytes)
                                              : cuda_error(e, "cudaMallocHost");
    }
    return VRT_OK;
}

int vrt_host_free(void* p) {
    if (p) VRT_CUDA(cudaFreeHost(p));
    return VRT_OK;
}

// The streams and events of the banded host render, made on first use.
static int ensure_band_resources(vrt_renderer* r) {
    if (r->copy_stream) return VRT_OK;
    for (cudaStream_t& b : r->band_stream) VRT_CUDA(cudaStreamCreateWithFlags(&b, cudaStreamNonBlocking));
    for (cudaEvent_t& e : r->band_done) VRT_CUDA(cudaEventCreateWithFlags(&e, cudaEventDisableTiming));
    VRT_CUDA(cudaEventCreateWithFlags(&r->start, cudaEventDisableTiming));
    VRT_CUDA(cudaEventCreateWithFlags(&r->copies_done, cudaEventDisableTiming));
    VRT_CUDA(cudaStreamCreateWithFlags(&r->copy_stream, cudaStreamNonBlocking));  // last: marks the set made
    return VRT_OK;
}

int vrt_render_to_host(vrt_renderer* r, const vrt_world* w, const vrt_uniforms* u, int32_t width, int32_t height,
                       uint8_t* host_rgba, const vrt_render_opts* opts, void* stream) {
    if (!r || !w || !host_rgba) return set_error(VRT_EINVAL, "NULL renderer, world or image");
    if (width < 1 || height < 1 || width > 32768 || height > 32768)
        return set_error(VRT_EINVAL, "image %d x %d out of range", width, height);
    int st = check_uniforms(u);
    if (st) return st;
    const cudaStream_t s = S(stream);
    if (!opts || opts->host_bands <= 0) {
        // Page-locked host memory is mapped into the device's address space (unified
        // addressing): the kernel stores the image into it over the host link as it renders,
        // with no staging buffer and no copy after the render.
        cudaPointerAttributes pa;
        if (cudaPointerGetAttributes(&pa, host_rgba) != cudaSuccess) {
            (void)cudaGetLastError();  // not a pointer the runtime knows: pageable memory
            pa.type = cudaMemoryTypeUnregistered;
        }
        if (pa.type == cudaMemoryTypeHost && pa.devicePointer && ((uintptr_t)pa.devicePointer & 3) == 0) {
            st = vrt_render(r, w, u, width, height, static_cast<uint8_t*>(pa.devicePointer), nullptr, nullptr, opts,
                            stream);
            if (st) return st;
            VRT_CUDA(cudaStreamSynchronize(s));
            return VRT_OK;
        }
    }
    size_t bytes = (size_t)width * height * 4;
    if (bytes > r->staging_bytes) {
        cudaFree(r->d_staging);
        r->d_staging = nullptr;
        r->staging_bytes = 0;
        cudaError_t e = cudaMalloc(&r->d_staging, bytes);
        if (e != cudaSuccess) return set_error(VRT_ENOMEM, "staging image: %s", cudaGetErrorString(e));
        r->staging_bytes = bytes;
    }
    int kernel = opts ? opts->kernel : VRT_KERNEL_AUTO;
    if (kernel == VRT_KERNEL_AUTO && !w->has_depth_field) kernel = VRT_KERNEL_MASK_PIXEL;
    int bands = 1;
    Tuning t{};
    if (kernel == VRT_KERNEL_MASK_PIXEL) {
        st = tile_tuning(opts, &t);
        if (st) return st;
        const int tiles_y = (height + t.tile_h - 1) / t.tile_h;
        // automatic: one band per 128 rows, up to 8, so that only the last band's copy is
        // exposed (1080p: 8 bands, 0.292 -> 0.265 ms per frame to pinned host memory)
        bands = opts && opts->host_bands > 0 ? opts->host_bands : std::max(1, std::min(8, height / 128));
        bands = std::max(1, std::min({bands, tiles_y, 8}));
    }
    if (bands == 1) {
        st = vrt_render(r, w, u, width, height, r->d_staging, nullptr, nullptr, opts, stream);
        if (st) return st;
        VRT_CUDA(cudaMemcpyAsync(host_rgba, r->d_staging, bytes, cudaMemcpyDeviceToHost, s));
        VRT_CUDA(cudaStreamSynchronize(s));
        return VRT_OK;
    }
    st = ensure_band_resources(r);
    if (st) return st;
    ViewDev v;
    fill_view(v, *u, width, height, r->d_staging, nullptr, nullptr, t, 0);
    const int tiles_x = v.map.tiles_x, tiles_y = (height + t.tile_h - 1) / t.tile_h;
    const int total = tiles_x * tiles_y;
    const size_t row_bytes = (size_t)width * 4;
    // Each band renders on its own stream, with no order among the bands: the launches run
    // back to back like one grid (a band's last wave overlaps the next band's first), and
    // each band's copy starts as soon as that band is done.  Every band is queued before
    // the first copy, because a copy to pageable host memory blocks the calling thread.
    VRT_CUDA(cudaEventRecord(r->start, s));
    for (int b = 0; b < bands; b++) {
        const int r0 = (int)((int64_t)tiles_y * b / bands), r1 = (int)((int64_t)tiles_y * (b + 1) / bands);
        VRT_CUDA(cudaStreamWaitEvent(r->band_stream[b], r->start, 0));
        st = launch_tiles(w, &v, 1, total, nullptr, t.tile_w * t.tile_h, r->band_stream[b], r0 * tiles_x,
                          (r1 - r0) * tiles_x);
        if (st) return st;
        VRT_CUDA(cudaEventRecord(r->band_done[b], r->band_stream[b]));
    }
    for (int b = 0; b < bands; b++) {
        const int r0 = (int)((int64_t)tiles_y * b / bands), r1 = (int)((int64_t)tiles_y * (b + 1) / bands);
        VRT_CUDA(cudaStreamWaitEvent(r->copy_stream, r->band_done[b], 0));
        const int y0 = r0 * t.tile_h, y1 = std::min(height, r1 * t.tile_h);
        VRT_CUDA(cudaMemcpyAsync(host_rgba + (size_t)y0 * row_bytes, r->d_staging + (size_t)y0 * row_bytes,
                                 (size_t)(y1 - y0) * row_bytes, cudaMemcpyDeviceToHost, r->copy_stream));
    }
    VRT_CUDA(cudaEventRecord(r->copies_done, r->copy_stream));
    VRT_CUDA(cudaStreamWaitEvent(s, r->copies_done, 0));  // later work on the stream follows the copies
    VRT_CUDA(cudaEventSynchronize(r->copies_done));
    return VRT_OK;
}

// Checks a batch's views and fills its view table hv (room for count entries, host
// memory): every view renders the one world, has a 4-byte aligned image of a valid size
// and valid uniforms, and may pick its own tile shape of the launch's thread count; the
// views' tiles are laid end to end in the launch's tile space.  Every batch entry point
// goes through here, so all of them check and lay out views alike.
// allow_df: the launch follows depth-field jumps (the tile kernel, launched now rather
// than replayed from a graph that would keep stale stop masks after an edit).
static int build_batch(const vrt_view* views, int32_t count, const Tuning& t, bool tile_kernel, ViewDev* hv,
                       const vrt_world** world_out, int* total_out, bool allow_df) {
    if (!views || count < 1) return set_error(VRT_EINVAL, "empty batch");
    const vrt_world* w = views[0].world;
    if (!w) return set_error(VRT_EINVAL, "view 0 has no world");
    if (w->has_depth_field && !allow_df)
        return set_error(VRT_ESTATE, "the world holds depth-field words: render it with vrt_render or vrt_render_batch "
                                     "and the tile kernel");
    int tiles = 0;
    for (int i = 0; i < count; i++) {
        const vrt_view& v = views[i];
        if (v.world != w) return set_error(VRT_EINVAL, "view %d renders another world; one batch = one world", i);
        if (!v.d_rgba || ((uintptr_t)v.d_rgba & 3) || v.width < 1 || v.height < 1 || v.width > 32768 ||
            v.height > 32768)
            return set_error(VRT_EINVAL, "view %d: bad image (NULL, not 4-byte aligned, or out of range)", i);
        int st = check_uniforms(&v.uniforms);
        if (st) return st;
        Tuning tv = t;  // a view may choose its own tile shape (the tile kernel: of the launch's tile size)
        if (v.tile_w > 0 || v.tile_h > 0) {
            if (v.tile_w < 1 || v.tile_h < 1 ||
                (tile_kernel ? v.tile_w * v.tile_h != t.tile_w * t.tile_h : v.tile_w * v.tile_h > 1024))
                return set_error(VRT_EINVAL, "view %d: tile %dx%d %s", i, v.tile_w, v.tile_h,
                                 tile_kernel ? "does not have the launch's thread count" : "exceeds 1024 pixels");
            tv.tile_w = v.tile_w;
            tv.tile_h = v.tile_h;
        }
        if (v.refill_min < 0 || v.refill_min > 32)
            return set_error(VRT_EINVAL, "view %d: refill_min %d outside 0-32", i, v.refill_min);
        if (v.refill_min > 0) tv.refill_min = v.refill_min;
        fill_view(hv[i], v.uniforms, v.width, v.height, v.d_rgba, nullptr, v.d_stats, tv, tiles);
        tiles += tiles_of(v.width, v.height, tv);
    }
    *world_out = w;
    *total_out = tiles;
    return VRT_OK;
}

// Batches run the tile kernel (AUTO, MASK_PIXEL) or the persistent kernel (BITMASK).
static int batch_tuning(const vrt_render_opts* opts, Tuning* t, bool* tiles) {
    const int kernel = opts ? opts->kernel : VRT_KERNEL_AUTO;
    if (kernel == VRT_KERNEL_BITMASK) {
        *tiles = false;
        *t = tuning_of(opts);
        return VRT_OK;
    }
    if (kernel != VRT_KERNEL_AUTO && kernel != VRT_KERNEL_MASK_PIXEL)
        return set_error(VRT_EINVAL, "batches render with the occupancy-mask kernels, not kernel %d", kernel);
    *tiles = true;
    return tile_tuning(opts, t);
}

static int launch_batch(vrt_renderer* r, const vrt_world* w, const ViewDev* hv, int count, int total,
                        const Tuning& t, bool tiles, const ViewDev* d_views, unsigned* d_counter, cudaStream_t s,
                        bool count_lookups = true) {
    if (tiles) return launch_tiles(w, hv, count, total, d_views, t.tile_w * t.tile_h, s, 0, -1, count_lookups);
    return launch_mask(r, w, hv, count, total, t, d_views, d_counter, s);
}

static int render_batch(vrt_renderer* r, const vrt_view* views, int32_t count, const vrt_render_opts* opts,
                        void* stream, bool count_lookups) {
    if (!r) return set_error(VRT_EINVAL, "NULL renderer");
    Tuning t;
    bool tiles = true;
    int st = batch_tuning(opts, &t, &tiles);
    if (st) return st;
    std::vector<ViewDev> hv((size_t)std::max(count, 1));
    const vrt_world* w = nullptr;
    int total = 0;
    st = build_batch(views, count, t, tiles, hv.data(), &w, &total, tiles);
    if (st) return st;
    if (count > 1) {
        st = ensure_views(r, count);
        if (st) return st;
        // pageable source: the copy is staged before the call returns, so hv may go
        VRT_CUDA(cudaMemcpyAsync(r->d_views, hv.data(), sizeof(ViewDev) * count, cudaMemcpyHostToDevice, S(stream)));
    }
    return launch_batch(r, w, hv.data(), count, total, t, tiles, r->d_views, r->d_counter, S(stream), count_lookups);
}

int vrt_render_batch(vrt_renderer* r, const vrt_view* views, int32_t count, const vrt_render_opts* opts,
                     void* stream) {
    return render_batch(r, views, count, opts, stream, true);
}

// Capture a batch graph's launch as the world stands, and make or update the executable graph.  Runs
// in flight or queued keep what they were launched with.
static int capture_batch(vrt_batch_graph* g) {
    VRT_CUDA(cudaStreamBeginCapture(g->capture_stream, cudaStreamCaptureModeThreadLocal));
    const int st = launch_batch(&g->shape, g->world, g->views.data(), (int)g->views.size(), g->total, g->t, g->tiles,
                                g->d_views, g->d_counter, g->capture_stream);
    cudaGraph_t graph = nullptr;
    cudaError_t e = cudaStreamEndCapture(g->capture_stream, &graph);
    if (st || e != cudaSuccess) {
        if (graph) cudaGraphDestroy(graph);
        return st ? st : cuda_error(e, "cudaStreamEndCapture");
    }
    if (g->graph) cudaGraphDestroy(g->graph);
    g->graph = graph;
    cudaGraphExecUpdateResultInfo info;
    if (!g->exec || cudaGraphExecUpdate(g->exec, g->graph, &info) != cudaSuccess) {
        cudaGetLastError();
        if (g->exec) cudaGraphExecDestroy(g->exec);
        g->exec = nullptr;
        VRT_CUDA(cudaGraphInstantiate(&g->exec, g->graph, 0));
    }
    std::memcpy(g->box, g->world->h_aabb, sizeof(g->box));
    return VRT_OK;
}

int vrt_batch_graph_create(vrt_renderer* r, const vrt_view* views, int32_t count, const vrt_render_opts* opts,
                           void* stream, vrt_batch_graph** out) {
    if (!r || !out) return set_error(VRT_EINVAL, "NULL argument");
    *out = nullptr;
    Tuning t;
    bool tiles = true;
    int st = batch_tuning(opts, &t, &tiles);
    if (st) return st;
    std::vector<ViewDev> hv((size_t)std::max(count, 1));
    const vrt_world* w = nullptr;
    int total = 0;
    st = build_batch(views, count, t, tiles, hv.data(), &w, &total, false);
    if (st) return st;
    vrt_batch_graph* g = new vrt_batch_graph();
    g->world = w;
    g->views = std::move(hv);
    g->total = total;
    g->t = t;
    g->tiles = tiles;
    g->shape.device = r->device;
    g->shape.num_sms = r->num_sms;
    cudaError_t e = cudaMalloc(&g->d_views, sizeof(ViewDev) * (size_t)count);
    if (e == cudaSuccess) e = cudaMalloc(&g->d_counter, 256);
    if (e == cudaSuccess)
        e = cudaMemcpyAsync(g->d_views, g->views.data(), sizeof(ViewDev) * count, cudaMemcpyHostToDevice, S(stream));
    if (e == cudaSuccess) e = cudaStreamSynchronize(S(stream));
    if (e == cudaSuccess) e = cudaStreamCreateWithFlags(&g->capture_stream, cudaStreamNonBlocking);
    if (e != cudaSuccess) {
        vrt_batch_graph_destroy(g);
        return cuda_error(e, "vrt_batch_graph_create");
    }
    st = capture_batch(g);
    if (st) {
        vrt_batch_graph_destroy(g);
        return st;
    }
    *out = g;
    return VRT_OK;
}

int vrt_batch_graph_launch(vrt_batch_graph* g, void* stream) {
    if (!g || !g->exec) return set_error(VRT_EINVAL, "NULL graph");
    // Rays end at the solid box, so one that edits have grown goes into the launch again.  (One that
    // shrank may stay as it is.)
    bool grown = false;
    for (int a = 0; a < 3; a++)
        grown |= g->world->h_aabb[a] < g->box[a] || g->world->h_aabb[3 + a] > g->box[3 + a];
    if (grown) {
        const int st = capture_batch(g);
        if (st) return st;
    }
    VRT_CUDA(cudaGraphLaunch(g->exec, S(stream)));
    return VRT_OK;
}

int vrt_batch_graph_destroy(vrt_batch_graph* g) {
    if (!g) return VRT_OK;
    if (g->exec) cudaGraphExecDestroy(g->exec);
    if (g->graph) cudaGraphDestroy(g->graph);
    if (g->capture_stream) cudaStreamDestroy(g->capture_stream);
    cudaFree(g->d_views);
    cudaFree(g->d_counter);
    delete g;
    return VRT_OK;
}

int vrt_probe_l2_read_gbs(uint64_t bytes, int32_t iters, double* gbs_out) {
    if (!gbs_out || bytes < 4096 || iters < 1) return set_error(VRT_EINVAL, "bad probe arguments");
    bytes &= ~(uint64_t)15;
    void* buf = nullptr;
    unsigned* sink = nullptr;
    VRT_CUDA(cudaMalloc(&buf, bytes));
    VRT_CUDA(cudaMalloc(&sink, sizeof(unsigned)));
    VRT_CUDA(cudaMemset(buf, 1, bytes));
    int dev = 0, sms = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    cudaEvent_t a, b;
    cudaEventCreate(&a);
    cudaEventCreate(&b);
    l2_read_kernel<<<sms * 4, 512>>>(reinterpret_cast<const uint4*>(buf), bytes / 16, 2, sink);  // warm
    cudaEventRecord(a);
    l2_read_kernel<<<sms * 4, 512>>>(reinterpret_cast<const uint4*>(buf), bytes / 16, iters, sink);
    cudaEventRecord(b);
    cudaError_t e = cudaEventSynchronize(b);
    float ms = 0.0f;
    cudaEventElapsedTime(&ms, a, b);
    cudaEventDestroy(a);
    cudaEventDestroy(b);
    cudaFree(buf);
    cudaFree(sink);
    if (e != cudaSuccess) return cuda_error(e, "l2 probe");
    *gbs_out = (double)bytes * iters / (ms * 1e-3) / 1e9;
    return VRT_OK;
}

}  // extern "C"

int vrt::render_batch_rays(vrt_renderer* r, const vrt_view* views, int32_t count, void* stream) {
    return render_batch(r, views, count, nullptr, stream, false);
}

// ====================================================================== batch without allocation

// vrt_render_batch_noalloc keeps its scratch -- the tile counter the persistent warps
// draw tiles from, and the table of views they read -- in this file-scope array instead
// of device memory that a renderer allocates.  Every GPU that loads the library holds it
// (about 46 KiB) until the process exits.  Host code cannot use the array's name as a
// device address: the address comes from cudaGetSymbolAddress, once per device, below.
constexpr int kNoAllocMaxViews = VRT_NOALLOC_MAX_VIEWS;
constexpr size_t kNoAllocCounterBytes = 256;
constexpr size_t kNoAllocBytes = kNoAllocCounterBytes + sizeof(ViewDev) * kNoAllocMaxViews;
static __device__ __align__(256) unsigned char g_noalloc_scratch[kNoAllocBytes];

constexpr int kNoAllocMaxDevices = 64;
static std::mutex g_noalloc_mutex;
static void* g_noalloc_address[kNoAllocMaxDevices];

// Device address of the scratch array on the current device, looked up on the first call
// made with that device current.
static int noalloc_scratch(void** out) {
    int dev = 0;
    VRT_CUDA(cudaGetDevice(&dev));
    if (dev < 0 || dev >= kNoAllocMaxDevices) return set_error(VRT_ERANGE, "device %d beyond %d", dev, kNoAllocMaxDevices);
    std::lock_guard<std::mutex> lock(g_noalloc_mutex);
    if (!g_noalloc_address[dev]) {
        void* p = nullptr;
        cudaError_t e = cudaGetSymbolAddress(&p, g_noalloc_scratch);
        if (e != cudaSuccess) return cuda_error(e, "cudaGetSymbolAddress(g_noalloc_scratch)");
        g_noalloc_address[dev] = p;
    }
    *out = g_noalloc_address[dev];
    return VRT_OK;
}

// The view table reaches the scratch array inside the parameters of copy kernels, up to
// kViewsPerCopy views a launch (a launch's parameters hold at most 32764 bytes): the
// runtime copies a launch's parameters when it is queued, so nothing queued by a call
// refers to the caller's host memory or to this file's stack after the call returns.
constexpr int kViewsPerCopy = 32;
struct ViewChunk {
    ViewDev v[kViewsPerCopy];
};
static_assert(sizeof(ViewChunk) + 16 <= 32764, "a view chunk must fit in one launch's parameters");
static_assert(sizeof(ViewDev) % 4 == 0, "views are copied as 32-bit words");

__global__ void copy_views_kernel(ViewDev* __restrict__ dst, const __grid_constant__ ViewChunk c, int n) {
    const uint32_t* src = reinterpret_cast<const uint32_t*>(c.v);
    uint32_t* out = reinterpret_cast<uint32_t*>(dst);
    const int words = n * (int)(sizeof(ViewDev) / 4);
    for (int i = threadIdx.x; i < words; i += blockDim.x) out[i] = src[i];
}

extern "C" int vrt_render_batch_noalloc(const vrt_view* views, int32_t count, const vrt_render_opts* opts,
                                        void* stream) {
    if (!views || count < 1) return set_error(VRT_EINVAL, "empty batch");
    if (count > kNoAllocMaxViews)
        return set_error(VRT_ERANGE, "%d views exceed the %d the static scratch holds; split the batch", count,
                         kNoAllocMaxViews);
    Tuning t;
    bool tile_kernel = true;  // as vrt_render_batch: the tile kernel unless the persistent one is asked for
    int st = batch_tuning(opts, &t, &tile_kernel);
    if (st) return st;
    // The view checks and tile layout of vrt_render_batch; worlds with depth-field words
    // are refused (VRT_ESTATE): their stop masks are allocated on first use.
    ViewDev hv[kNoAllocMaxViews];  // host view table, on the stack
    const vrt_world* w = nullptr;
    int tiles = 0;
    st = build_batch(views, count, t, tile_kernel, hv, &w, &tiles, false);
    if (st) return st;
    void* scratch = nullptr;
    st = noalloc_scratch(&scratch);
    if (st) return st;
    unsigned int* d_counter = reinterpret_cast<unsigned int*>(scratch);
    ViewDev* d_views = reinterpret_cast<ViewDev*>(static_cast<unsigned char*>(scratch) + kNoAllocCounterBytes);
    if (count > 1) {  // a single view travels in the render launch's own parameters
        ViewChunk chunk{};
        for (int first = 0; first < count; first += kViewsPerCopy) {
            const int n = std::min(kViewsPerCopy, count - first);
            std::memcpy(chunk.v, hv + first, sizeof(ViewDev) * n);
            copy_views_kernel<<<1, 256, 0, S(stream)>>>(d_views + first, chunk, n);
            VRT_CUDA(cudaGetLastError());
        }
    }
    vrt_renderer shape;  // only its device and SM count are read
    VRT_CUDA(cudaGetDevice(&shape.device));
    if (tile_kernel) {
        st = ensure_div255(shape.device);  // once per device, like the scratch address
        if (st) return st;
        return launch_tiles(w, hv, count, tiles, d_views, t.tile_w * t.tile_h, S(stream));
    }
    VRT_CUDA(cudaDeviceGetAttribute(&shape.num_sms, cudaDevAttrMultiProcessorCount, shape.device));
    return launch_mask(&shape, w, hv, count, tiles, t, d_views, d_counter, S(stream));  // zeroes the counter
}
