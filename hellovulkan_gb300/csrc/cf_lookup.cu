// cf_lookup.cu — the consumer side of the culled lists: Scene.frag's cluster
// lookup (HelloVulkan/Shaders/ClusteredForward/Scene.frag:54-78) for every
// pixel of a depth buffer, as a check that the (offset, count) cells and the
// index list drop into the reference's fragment pass, and the pass's direct
// clustered lighting (Radiance.glsl) over a G-buffer.
//
// Per pixel: LinearDepth of its depth, the exponential slice index from log2
// (pinned: cf_log2_pinned), the tile from the pixel centre, then the cluster's
// cell.  The fragment's view-space position is reconstructed the way
// AABBGenerator.comp's ScreenToView unprojects a screen point, and every listed
// light is tested for containing it (the lights a shading loop over the list
// would find in range).  In check mode the lights of the whole set that contain
// it are counted as well, to count the ones the list lacks.
//
// Both passes take a CTA per square tile of pixels and sort the tile's pixels
// by depth first, so that the 32 pixels of a warp read the same one or two
// lists: with every pixel at its own depth, unsorted warps had 5 to 10 of 32
// lanes active.  A sorted warp's fragments also lie in a small box, which few
// lights of the whole set reach.  1920x1080, 1024 lights, every pixel at its own
// depth, one thread per unsorted pixel against sorted tiles: lookup 120 -> 43 us,
// shading 1113 -> 121 us; 480x270 with 3000 lights and the all-lights check
// 812 -> 40 us.
#include <cuda_runtime.h>

#include <cmath>

#include "cf_device.cuh"
#include "cf_launch.cuh"
#include "cf_pinned_math.h"
#include "cf_runtime_internal.h"
#include "cfcull.h"

namespace {

// p = the view-space position of light L (cameraView * position, pinned order).
__device__ __forceinline__ void light_view(const float* V, const CfLightData* __restrict__ L, float p[3], float* r2)
{
    const float4 q = __ldg(reinterpret_cast<const float4*>(&L->position[0]));
    p[0] = cf_mat4_row(V, 0, q.x, q.y, q.z, q.w);
    p[1] = cf_mat4_row(V, 1, q.x, q.y, q.z, q.w);
    p[2] = cf_mat4_row(V, 2, q.x, q.y, q.z, q.w);
    const float r = __ldg(&L->radius);
    *r2 = cf_fmul(r, r);
}

// Scene.frag:54-71 for the fragment at pixel (x, y) with window depth z: the
// linear depth and, when it lies inside the grid, the cluster index.
// xf, yf: its tile coordinates, gl_FragCoord.xy / (screenSize / sliceCount).
__device__ __forceinline__ bool fragment_cluster(const CfClusterForwardUBO& u, float xf, float yf, float z,
                                                 uint32_t* cluster, float* linear_depth)
{
    const float n = u.cameraNear, f = u.cameraFar;
    // LinearDepth (Scene.frag:54-57): near * far / (far + z * (near - far))
    const float lin = cf_fdiv(cf_fmul(n, f), cf_fadd(f, cf_fmul(z, cf_fsub(n, f))));
    // zIndex (Scene.frag:63): max(log2(linDepth) * sliceScaling + sliceBias, 0)
    const float zf = cf_glsl_max(cf_fadd(cf_fmul(cf_log2_pinned(lin), u.sliceScaling), u.sliceBias), 0.0f);
    *linear_depth = lin;
    // NaN compares false: a NaN index leaves the grid too
    if (!(zf < (float)u.sliceCountZ && xf < (float)u.sliceCountX && yf < (float)u.sliceCountY)) return false;
    *cluster = (uint32_t)xf + (uint32_t)yf * u.sliceCountX + (uint32_t)zf * u.sliceCountX * u.sliceCountY;
    return true;
}

// |f - c|^2 < r^2, summed x, y, z in order.
__device__ __forceinline__ bool contains(const float f[3], const float c[3], float r2)
{
    const float dx = cf_fsub(f[0], c[0]), dy = cf_fsub(f[1], c[1]), dz = cf_fsub(f[2], c[2]);
    return cf_fadd(cf_fadd(cf_fmul(dx, dx), cf_fmul(dy, dy)), cf_fmul(dz, dz)) < r2;
}

// ---------------------------------------------------------------------------
// Tiles of pixels, sorted by depth.
// ---------------------------------------------------------------------------
constexpr uint32_t kDepthBins = 128;  // of each of a tile's cluster columns, up to four
constexpr uint32_t kBins = 4 * kDepthBins + 1;  // the last one: past the image
constexpr uint32_t kNoPixel = 0xffffu;

struct Image {
    uint32_t width, height, n_pixels;
    uint32_t tiles_x;  // 0: too narrow for square tiles, a tile is a run of pixels in row-major order
    float tile_w, tile_h;  // pixels per cluster (screenSize / sliceCount)
};

// The CTA's tile of kSide * kSide pixels.
template <uint32_t kSide>
struct Tile {
    uint32_t x0, y0;  // of a run: x0 is its first pixel
    __device__ __forceinline__ explicit Tile(const Image& im)
        : x0(im.tiles_x ? blockIdx.x % im.tiles_x * kSide : blockIdx.x * kSide * kSide),
          y0(im.tiles_x ? blockIdx.x / im.tiles_x * kSide : 0u)
    {
    }
    // Pixel i of the tile; false past the image.
    __device__ __forceinline__ bool at(const Image& im, uint32_t i, uint32_t& x, uint32_t& y) const
    {
        if (im.tiles_x) {
            x = x0 + i % kSide;
            y = y0 + i / kSide;
            return x < im.width && y < im.height;
        }
        const uint32_t p = x0 + i;  // below 2^31 + 1024
        x = p % im.width;
        y = p / im.width;
        return p < im.n_pixels;
    }
};

// What a pixel's column and row give, which a square tile's pixels share: the
// cluster tile coordinate and the clip coordinate of the pixel centre (a run's
// pixels compute them where they are used).
template <uint32_t kSide>
struct TileAxes {
    float tile[2][kSide], clip[2][kSide];
};
// gl_FragCoord / (screenSize / sliceCount) (Scene.frag:64-70)
__device__ __forceinline__ float tile_coord(uint32_t p, float pixels) { return cf_fdiv((float)p + 0.5f, pixels); }
// ScreenToView's clip coordinate of the pixel centre
__device__ __forceinline__ float clip_coord(uint32_t p, float size)
{
    return cf_fsub(cf_fmul(cf_fdiv((float)p + 0.5f, size), 2.0f), 1.0f);
}
template <uint32_t kSide>
__device__ __forceinline__ void fill_axes(const CfClusterForwardUBO& u, const Image& im, const Tile<kSide>& tile,
                                          TileAxes<kSide>& a)
{
    if (im.tiles_x == 0 || threadIdx.x >= 2 * kSide) return;
    const uint32_t axis = threadIdx.x / kSide, i = threadIdx.x % kSide, p = (axis ? tile.y0 : tile.x0) + i;
    a.tile[axis][i] = tile_coord(p, axis ? im.tile_h : im.tile_w);
    a.clip[axis][i] = clip_coord(p, u.screenSize[axis]);
}

// A pixel's depth bin: an eighth of an octave of the denominator of
// LinearDepth, so of the linear depth itself.  It orders the work and nothing
// else; a depth outside [0, 1] or a NaN gets some bin.
__device__ __forceinline__ uint32_t depth_bin(const CfClusterForwardUBO& u, float z)
{
    const float t = u.cameraFar + z * (u.cameraNear - u.cameraFar);
    const int b = ((int)__float_as_uint(t) - (int)__float_as_uint(u.cameraNear)) >> 20;
    return (uint32_t)min(max(b, 0), (int)kDepthBins - 1);
}

struct TileSort {
    uint32_t start[(kBins + 31) / 32 * 32];
    uint32_t next;  // unit not yet taken
};

// order[]: the tile's pixels by cluster column, if asked (left or right of the
// first boundary in the tile, above or below it), and depth bin, those past the
// image (kNoPixel) last.  `depth(q, p)` gives the depth of pixel p, the thread's
// q-th of the tile.  Every thread of the CTA takes part.
template <bool kColumns, uint32_t kSide, uint32_t kThreads, typename Depth>
__device__ __forceinline__ void sort_tile(const CfClusterForwardUBO& u, const Image& im, const Tile<kSide>& tile,
                                          const TileAxes<kSide>& axes, TileSort& s, uint16_t* order, Depth depth)
{
    constexpr uint32_t kPer = kSide * kSide / kThreads;
    const uint32_t tid = threadIdx.x, lane = tid & 31;
    constexpr uint32_t kSlots = sizeof(s.start) / sizeof(s.start[0]);
    for (uint32_t b = tid; b < kSlots; b += kThreads) s.start[b] = 0;
    uint32_t bin[kPer], rank[kPer];
#pragma unroll
    for (uint32_t q = 0; q < kPer; ++q) {
        uint32_t x, y;
        const uint32_t i = q * kThreads + tid;
        bin[q] = tile.at(im, i, x, y) ? depth_bin(u, depth(q, y * im.width + x)) : kBins - 1;
    }
    __syncthreads();  // also the axes'
    if (kColumns && im.tiles_x) {
        const float x1 = floorf(axes.tile[0][0]) + 1.0f, y1 = floorf(axes.tile[1][0]) + 1.0f;
#pragma unroll
        for (uint32_t q = 0; q < kPer; ++q) {
            const uint32_t i = q * kThreads + tid;
            if (bin[q] != kBins - 1)
                bin[q] += (axes.tile[0][i % kSide] >= x1 ? kDepthBins : 0u) + (axes.tile[1][i / kSide] >= y1 ? 2 * kDepthBins : 0u);
        }
    }
#pragma unroll
    for (uint32_t q = 0; q < kPer; ++q) {  // the order within a bin is of no account
        if (__all_sync(cfk::kFull, bin[q] == __shfl_sync(cfk::kFull, bin[q], 0))) {  // a surface: one count for the warp
            if (lane == 0) rank[q] = atomicAdd(&s.start[bin[q]], 32u);
            rank[q] = __shfl_sync(cfk::kFull, rank[q], 0) + lane;
        } else {
            rank[q] = atomicAdd(&s.start[bin[q]], 1u);
        }
    }
    __syncthreads();
    if (tid < 32) {
        constexpr uint32_t kEach = kSlots / 32;
        uint32_t n = 0, c[kEach];
#pragma unroll
        for (uint32_t b = 0; b < kEach; ++b) n += c[b] = s.start[kEach * tid + b];
        n = cfk::warp_inclusive_scan(n, tid) - n;
#pragma unroll
        for (uint32_t b = 0; b < kEach; ++b) {
            s.start[kEach * tid + b] = n;
            n += c[b];
        }
        if (tid == 0) s.next = 0;
    }
    __syncthreads();
#pragma unroll
    for (uint32_t q = 0; q < kPer; ++q)
        order[s.start[bin[q]] + rank[q]] = (uint16_t)(bin[q] == kBins - 1 ? kNoPixel : q * kThreads + tid);
    __syncthreads();
}

// The next 32 pixels of the sorted tile, as units are taken by the CTA's warps
// one after another: a tile's long lists lie at neighbouring depths, so fixed
// shares would leave them to one warp.
__device__ __forceinline__ uint32_t next_unit(TileSort& s, uint32_t lane)
{
    uint32_t unit = 0;
    if (lane == 0) unit = atomicAdd(&s.next, 1u);
    return __shfl_sync(cfk::kFull, unit, 0);
}

// ---------------------------------------------------------------------------
// Lookup.
// ---------------------------------------------------------------------------
constexpr uint32_t kTableLights = 1024;  // view-space lights kept in shared memory at a time

struct LookupArgs {
    CfClusterForwardUBO u;
    Image im;
    const float* depth;
    const CfLightCell* cells;
    const uint32_t* indices;
    uint64_t index_count;
    const CfLightData* lights;
    const float4* aabbs;
    CfFragmentSample* out;
    uint32_t light_count, cap;
    int out_aligned;
};

// Lights [first, first + n) of the set in view space: (x, y, z, r^2).
__device__ __forceinline__ void fill_table(const LookupArgs& A, float4* table, uint32_t first, uint32_t n)
{
    for (uint32_t i = threadIdx.x; i < n; i += blockDim.x) {
        float p[3], r2;
        light_view(A.u.cameraView, &A.lights[first + i], p, &r2);
        table[i] = make_float4(p[0], p[1], p[2], r2);
    }
}

// The view-space position of the fragment at clip coordinates (cx, cy) with
// window depth z: ScreenToView of (x / width, y / height, z, 1).
__device__ __forceinline__ void fragment_view(const CfClusterForwardUBO& u, float cx, float cy, float z, float frag[3])
{
    const float* IP = u.cameraInverseProjection;
    const float vw = cf_mat4_row(IP, 3, cx, cy, z, 1.0f);
    frag[0] = cf_fdiv(cf_mat4_row(IP, 0, cx, cy, z, 1.0f), vw);
    frag[1] = cf_fdiv(cf_mat4_row(IP, 1, cx, cy, z, 1.0f), vw);
    frag[2] = cf_fdiv(cf_mat4_row(IP, 2, cx, cy, z, 1.0f), vw);
}

// How many lights of table[0, n) contain each lane's fragment.  The warp's
// fragments lie in the box [lo, hi]; a light that does not reach it contains
// none of them (its distance to the box is never larger than to a fragment in
// it, rounded operation by rounded operation).
__device__ __forceinline__ uint32_t count_containing(const float4* table, uint32_t n, const float frag[3], const float lo[3],
                                                     const float hi[3], uint32_t lane)
{
    using namespace cfk;
    const f2 lx = f2_pack(lo[0], lo[0]), ly = f2_pack(lo[1], lo[1]), lz = f2_pack(lo[2], lo[2]), hx = f2_pack(hi[0], hi[0]),
             hy = f2_pack(hi[1], hi[1]), hz = f2_pack(hi[2], hi[2]);
    uint32_t count = 0;
    // two lights per lane, in packed operations: a filter of one took a third
    // more instructions (480x270, 3000 lights: 45.7 -> 40.1 us)
    for (uint32_t c = 0; c < n; c += 64) {
        const bool in0 = c + lane < n, in1 = c + 32 + lane < n;
        const float4 a = table[in0 ? c + lane : c], b = table[in1 ? c + 32 + lane : c];
        bool reach0, reach1;
        hit_pair_twice_rounded(f2_pack(a.x, b.x), f2_pack(a.y, b.y), f2_pack(a.z, b.z), a.w, b.w, lx, ly, lz, hx, hy, hz,
                               reach0, reach1);
        const uint32_t m0 = __ballot_sync(kFull, in0 && reach0), m1 = __ballot_sync(kFull, in1 && reach1);
#pragma unroll
        for (uint32_t h = 0; h < 2; ++h)
            for (uint32_t m = h ? m1 : m0; m; m &= m - 1) {
                const float4 q = table[c + 32 * h + __ffs(m) - 1];
                const float p[3] = {q.x, q.y, q.z};
                count += contains(frag, p, q.w) ? 1u : 0u;
            }
    }
    return count;
}

// 32 lights of a list in view space, one array per component so that four
// lights' x are one 16-byte read.
struct ListWarp {
    float x[32], y[32], z[32], r2[32];
};

// Mask of the first n lights of w that contain the fragment (those past them,
// to a multiple of four, reach nothing).  Four lights per step, two per packed
// operation; the products are rounded before scalar additions.
__device__ __forceinline__ uint32_t containing(const ListWarp& w, uint32_t n, const float frag[3])
{
    const cfk::f2 fx = cfk::f2_pack(frag[0], frag[0]), fy = cfk::f2_pack(frag[1], frag[1]),
                  fz = cfk::f2_pack(frag[2], frag[2]);
    uint32_t word = 0;
#pragma unroll 2
    for (uint32_t j = 0; j < n; j += 4) {
        const float4 x = *reinterpret_cast<const float4*>(&w.x[j]);
        const float4 y = *reinterpret_cast<const float4*>(&w.y[j]);
        const float4 z = *reinterpret_cast<const float4*>(&w.z[j]);
        const float4 r2 = *reinterpret_cast<const float4*>(&w.r2[j]);
        float xx[4], yy[4], zz[4];
        cfk::f2 d = cfk::f2_sub(fx, cfk::f2_pack(x.x, x.y));
        cfk::f2_unpack(cfk::f2_mul(d, d), xx[0], xx[1]);
        d = cfk::f2_sub(fx, cfk::f2_pack(x.z, x.w));
        cfk::f2_unpack(cfk::f2_mul(d, d), xx[2], xx[3]);
        d = cfk::f2_sub(fy, cfk::f2_pack(y.x, y.y));
        cfk::f2_unpack(cfk::f2_mul(d, d), yy[0], yy[1]);
        d = cfk::f2_sub(fy, cfk::f2_pack(y.z, y.w));
        cfk::f2_unpack(cfk::f2_mul(d, d), yy[2], yy[3]);
        d = cfk::f2_sub(fz, cfk::f2_pack(z.x, z.y));
        cfk::f2_unpack(cfk::f2_mul(d, d), zz[0], zz[1]);
        d = cfk::f2_sub(fz, cfk::f2_pack(z.z, z.w));
        cfk::f2_unpack(cfk::f2_mul(d, d), zz[2], zz[3]);
        const float lim[4] = {r2.x, r2.y, r2.z, r2.w};
        uint32_t m = 0;
#pragma unroll
        for (int e = 0; e < 4; ++e) m |= cf_fadd(cf_fadd(xx[e], yy[e]), zz[e]) < lim[e] ? 1u << e : 0u;
        word |= m << j;
    }
    return word;
}

// The lookup of a warp's pixels, whose fragments are at frag; with the check,
// `missing` of s holds the lights of the whole set that contain the fragment.
// The warp reads the list of each cluster that its pixels lie in together: a
// lane fetches and transforms an entry; then each pixel of the cluster tests
// 32 of them, or, where the cluster has few of the warp's pixels, the lanes
// test their entries against one pixel after another.  A warp of many clusters
// or short lists has each pixel walk its own list, kOwnStep entries at a time
// with the next ones' indices on their way.
constexpr uint32_t kFewPixels = 3;  // entries per pixel from which a pixel's turn is cheaper than four entries' test
// Where all lists of a warp's pixels are this short, each pixel walks its own
// (1920x1080, scattered: 49.5 -> 46.9 us), and where they lie in so many clusters
// that the longest list has at most kOwnPerList entries for each: a cluster after
// another is then a chain of round trips for a pixel or two each.  One thread
// per unsorted pixel / only short lists walked / this rule, in us:
//   96x64,    32x18x48, 16384 lights, scattered    45.3 / 59.5 / 14.5
//   480x270,  64x64x64, 2000 lights, scattered     18.6 / 30.0 / 14.6
//   480x270, 128x72x24, 4000 lights, surfaces      22.7 / 24.3 / 20.7
//   20x20000, 16x9x24,  1024 lights, scattered     22.6 / 38.5 / 15.7
//   1920x1080, 64x64x64, 2000 lights, scattered   107   / 114  / 64
// With the check: 1855x69, 42x34x50, 48 lights that reach all 45.0 / 58.5 / 30.2 (one
// thread per pixel / no pixel walks its own / this rule), 17x56, 122x61x2, 27 lights of
// radius 20 to 60 12.4 / 21.6 / 12.1.
// A launch of many tiles is bound by issue and takes 4 entries per cluster
// (6 / 8 / 12: the reference view's surfaces 46.4 -> 48.5 / 50.0 / 52.3), two at
// a time; one of a tile per SM or less by latency: 12, four at a time.
// From kOwnClusters on a step of the lists side by side has more pixels at work
// than a round of one list, however long: 31x7444, 57x51x3, 2124 lights in one place
// 84 / - / 145 without this, 86 with it (with the check 701 / - / 215 and 126).
constexpr uint32_t kShortLookup = 4, kOwnClusters = 24;
constexpr uint32_t kBoxList = 8;    // a list up to this long is not worth a box
template <bool kCheck, uint32_t kOwnStep, uint32_t kOwnPerList>
__device__ __forceinline__ void look_up(const LookupArgs& A, const float4* table, bool whole, ListWarp& w, uint32_t lane,
                                        bool valid, float xf, float yf, float z, const float frag[3], CfFragmentSample& s)
{
    const CfClusterForwardUBO& u = A.u;
    uint32_t c = 0, off = 0, cnt = 0, in_list = 0;
    const bool inside = fragment_cluster(u, xf, yf, z, &c, &s.linear_depth) && valid;
    s.view_z = frag[2];
    s.covering = 0;
    s.flags = 0;
    s.cluster = c;
    if (inside) {
        const CfLightCell cell = A.cells[c];
        off = cell.offset;
        cnt = cell.count;
        if ((uint64_t)off + cnt > A.index_count) {  // not a cell of this index list: read nothing through it
            s.flags |= CF_FRAGMENT_BAD_CELL;
            cnt = 0;
        }
        if (cnt >= A.cap) s.flags |= CF_FRAGMENT_CAPPED;
        if (A.aabbs) {
            const float4 lo = __ldg(&A.aabbs[2 * (size_t)c]), hi = __ldg(&A.aabbs[2 * (size_t)c + 1]);
            if (frag[0] < lo.x || frag[1] < lo.y || frag[2] < lo.z || frag[0] > hi.x || frag[1] > hi.y || frag[2] > hi.z)
                s.flags |= CF_FRAGMENT_OUTSIDE_AABB;
        }
    } else {
        s.cluster = 0xFFFFFFFFu;
        s.flags |= CF_FRAGMENT_OUTSIDE_GRID;
    }
    const uint32_t longest = __reduce_max_sync(cfk::kFull, cnt);
    bool own = longest <= kShortLookup;
    if (!own) {
        const uint32_t same = __match_any_sync(cfk::kFull, cnt ? c : ~0u);
        const uint32_t clusters = __popc(__ballot_sync(cfk::kFull, cnt && (same & ((1u << lane) - 1u)) == 0));
        own = longest <= kOwnPerList * clusters || clusters >= kOwnClusters;
    }
    if (own) {
        uint32_t next[kOwnStep], before = 0;
        bool walked = true;  // with the check: none of the entries so far ended the list's part (see below)
#pragma unroll
        for (uint32_t e = 0; e < kOwnStep; ++e) next[e] = e < cnt ? __ldg(&A.indices[off + e]) : 0u;
        for (uint32_t j = 0; j < longest; j += kOwnStep) {
            float4 q[kOwnStep];
            float r[kOwnStep];
            bool in_part[kOwnStep];
#pragma unroll
            for (uint32_t e = 0; e < kOwnStep; ++e) {
                const bool has = j + e < cnt, light = has && next[e] < A.light_count;
                if (has && !light) s.flags |= CF_FRAGMENT_BAD_CELL;
                const CfLightData* l = &A.lights[next[e]];
                q[e] = light ? __ldg(reinterpret_cast<const float4*>(&l->position[0])) : make_float4(0.f, 0.f, 0.f, 0.f);
                r[e] = light ? __ldg(&l->radius) : __uint_as_float(0x7fffffffu);  // NaN: contains nothing
                if (kCheck) {
                    in_part[e] = walked = walked && light && (j + e == 0 || next[e] > before);
                    before = next[e];
                }
                next[e] = j + kOwnStep + e < cnt ? __ldg(&A.indices[off + j + kOwnStep + e]) : 0u;
            }
#pragma unroll
            for (uint32_t e = 0; e < kOwnStep; ++e) {
                const float* V = u.cameraView;
                const float p[3] = {cf_mat4_row(V, 0, q[e].x, q[e].y, q[e].z, q[e].w),
                                    cf_mat4_row(V, 1, q[e].x, q[e].y, q[e].z, q[e].w),
                                    cf_mat4_row(V, 2, q[e].x, q[e].y, q[e].z, q[e].w)};
                const uint32_t hit = contains(frag, p, cf_fmul(r[e], r[e])) ? 1u : 0u;
                s.covering += hit;
                if (kCheck) in_list += in_part[e] ? hit : 0u;
            }
        }
    }
    for (uint32_t todo = own ? 0u : __ballot_sync(cfk::kFull, cnt != 0); todo;) {
        const uint32_t leader = __ffs(todo) - 1;
        const uint32_t list_c = __shfl_sync(cfk::kFull, c, leader), list = __shfl_sync(cfk::kFull, off, leader),
                       n = __shfl_sync(cfk::kFull, cnt, leader);
        const bool mine = cnt != 0 && c == list_c;
        const uint32_t pixels = __ballot_sync(cfk::kFull, mine);
        const uint32_t n_pixels = __popc(pixels);
        // the box of the cluster's fragments, where the list is worth it
        const float inf = __uint_as_float(0x7f800000u);
        float lo[3] = {-inf, -inf, -inf}, hi[3] = {inf, inf, inf};
        if (n > kBoxList) {
#pragma unroll
            for (int a = 0; a < 3; ++a) {  // a NaN coordinate is in no sphere: the reductions pass it over
                lo[a] = cfk::warp_min(mine ? frag[a] : inf);
                hi[a] = cfk::warp_max(mine ? frag[a] : -inf);
            }
        }
        todo &= ~pixels;
        // A light is missing when it is not in the part of the list that a
        // walk over all lights in order would match: the entries up to the
        // first that does not ascend or is no light.
        uint32_t walked = ~0u, before = 0;
        uint32_t li = lane < n ? __ldg(&A.indices[list + lane]) : 0u;
        for (uint32_t j = 0;; j += 32) {
            const bool has = lane < n - j, more = n - j > 32, light = has && li < A.light_count;
            const uint32_t here = li;
            float p[3] = {0.0f, 0.0f, 0.0f}, r2 = __uint_as_float(0xff800000u);  // no light: reaches nothing
            if (light) {
                if (whole) {
                    const float4 L = table[here];
                    p[0] = L.x;
                    p[1] = L.y;
                    p[2] = L.z;
                    r2 = L.w;
                } else {
                    light_view(u.cameraView, &A.lights[here], p, &r2);
                }
            }
            if (more && lane < n - j - 32) li = __ldg(&A.indices[list + j + 32 + lane]);  // for the next round
            if (__any_sync(cfk::kFull, has && !light) && mine) s.flags |= CF_FRAGMENT_BAD_CELL;
            if (kCheck) {
                uint32_t prev = __shfl_up_sync(cfk::kFull, here, 1);
                if (lane == 0) prev = before;
                const uint32_t out = __ballot_sync(cfk::kFull, !light || (j + lane != 0 && here <= prev));
                if (walked) walked = out ? (out & (0u - out)) - 1u : ~0u;  // those before the first such entry
                before = __shfl_sync(cfk::kFull, here, 31);
            }
            // A light that does not reach the box contains none of the fragments.
            const bool reach = light && (n <= kBoxList || cfk::hit_fast(make_float4(p[0], p[1], p[2], r2), lo, hi));
            const uint32_t reached = __ballot_sync(cfk::kFull, reach), ns = __popc(reached);
            if (kFewPixels * n_pixels < ns) {
                for (uint32_t m = pixels; m; m &= m - 1) {
                    const uint32_t t = __ffs(m) - 1;
                    const float f[3] = {__shfl_sync(cfk::kFull, frag[0], t), __shfl_sync(cfk::kFull, frag[1], t),
                                        __shfl_sync(cfk::kFull, frag[2], t)};
                    const uint32_t hits = __ballot_sync(cfk::kFull, contains(f, p, r2));
                    if (lane == t) {
                        s.covering += __popc(hits);
                        if (kCheck) in_list += __popc(hits & walked);
                    }
                }
            } else if (ns) {
                const uint32_t lower = (1u << lane) - 1u;
                const uint32_t at = reach ? __popc(reached & lower) : ns + __popc(~reached & lower);
                w.x[at] = p[0];  // the others follow, and reach nothing
                w.y[at] = p[1];
                w.z[at] = p[2];
                w.r2[at] = reach ? r2 : -inf;
                __syncwarp();
                if (mine) {
                    const uint32_t hits = containing(w, ns, frag);
                    s.covering += __popc(hits);
                    // the walked ones are the first of those that reach
                    if (kCheck) in_list += __popc(hits & (uint32_t)((1ull << __popc(reached & walked)) - 1));
                }
                __syncwarp();
            }
            if (kCheck && walked != ~0u) walked = 0u;
            if (!more) break;
        }
    }
    s.offset = off;
    s.count = (s.flags & CF_FRAGMENT_BAD_CELL) ? 0u : cnt;
    if (kCheck) s.missing -= in_list;
}

// One CTA per tile.  Bound by issue (72% of the slots at 1920x1080): some 300
// instructions a pixel apart from its list, five of them IEEE divisions.  A
// warp's lists cost a transform per 32 entries and a test per entry that
// reaches its fragments' box; when each lane walked its own list the lookup of
// that image took 59 us, with 3000 lights on surfaces 193 us (now 72).  With
// the check, lights come from the table where the whole set fits it; the check
// runs the set through the table in pieces, 32 lights at a time against the box
// of the warp's fragments.
template <uint32_t kSide, uint32_t kThreads, bool kCheck>
__global__ void __launch_bounds__(kThreads, kSide == 16 ? 2 : 5 * 256 / kThreads) lookup_kernel(const __grid_constant__ LookupArgs A)
{
    constexpr uint32_t kPixels = kSide * kSide, kUnits = kPixels / 32;
    __shared__ __align__(16) float4 table[kCheck ? kTableLights : 1];
    __shared__ __align__(16) ListWarp lists[kThreads / 32];
    __shared__ uint32_t missing[kCheck ? kPixels : 1];  // by place in the order, between pieces
    __shared__ uint16_t order[kPixels];
    __shared__ TileSort sort;
    __shared__ TileAxes<kSide> axes;
    const uint32_t lane = threadIdx.x & 31;
    const CfClusterForwardUBO& u = A.u;
    const Tile<kSide> tile(A.im);
    const bool whole = kCheck && A.light_count <= kTableLights;  // the set fits the table
    cfk::grid_dependency_wait();
    cfk::launch_dependents();
    if (whole) fill_table(A, table, 0, A.light_count);
    fill_axes(u, A.im, tile, axes);
    sort_tile<!kCheck, kSide, kThreads>(u, A.im, tile, axes, sort, order, [&](uint32_t, uint32_t p) { return __ldg(&A.depth[p]); });
    const uint32_t pieces = kCheck ? (A.light_count + kTableLights - 1) / kTableLights : 0u;
    for (uint32_t piece = 0; piece < max(pieces, 1u); ++piece) {
        const uint32_t n = pieces ? min(kTableLights, A.light_count - piece * kTableLights) : 0u;
        if (!whole && pieces) {
            if (piece) {
                __syncthreads();
                if (threadIdx.x == 0) sort.next = 0;
            }
            fill_table(A, table, piece * kTableLights, n);
            __syncthreads();
        }
        for (uint32_t unit; (unit = next_unit(sort, lane)) < kUnits;) {
            const uint32_t i = order[unit * 32 + lane];
            const bool valid = i != kNoPixel;
            if (!__any_sync(cfk::kFull, valid)) continue;
            uint32_t x = 0, y = 0;
            float z = 0.0f, cx = 0.0f, cy = 0.0f, xf = 0.0f, yf = 0.0f;
            if (valid) {
                tile.at(A.im, i, x, y);
                z = __ldg(&A.depth[y * A.im.width + x]);
                if (A.im.tiles_x) {
                    cx = axes.clip[0][i % kSide];
                    cy = axes.clip[1][i / kSide];
                    xf = axes.tile[0][i % kSide];
                    yf = axes.tile[1][i / kSide];
                } else {
                    cx = clip_coord(x, u.screenSize[0]);
                    cy = clip_coord(y, u.screenSize[1]);
                    xf = tile_coord(x, A.im.tile_w);
                    yf = tile_coord(y, A.im.tile_h);
                }
            }
            float frag[3];
            fragment_view(u, cx, cy, z, frag);
            CfFragmentSample s;
            s.missing = 0;
            if (kCheck && pieces) {
                const float inf = __uint_as_float(0x7f800000u);
                float lo[3], hi[3];
#pragma unroll
                for (int a = 0; a < 3; ++a) {  // a NaN coordinate is in no sphere: the reductions pass it over
                    lo[a] = cfk::warp_min(valid ? frag[a] : inf);
                    hi[a] = cfk::warp_max(valid ? frag[a] : -inf);
                }
                s.missing = count_containing(table, n, frag, lo, hi, lane) + (piece ? missing[unit * 32 + lane] : 0u);
                if (piece + 1 < pieces) {
                    missing[unit * 32 + lane] = s.missing;
                    continue;
                }
            }
            constexpr bool kMany = kSide == 32 && kThreads <= 512;  // tiles
            look_up<kCheck, kMany ? 2 : 4, kMany ? 4 : 12>(A, table, whole, lists[threadIdx.x >> 5], lane, valid, xf, yf, z, frag, s);
            if (!valid) continue;
            CfFragmentSample* out = &A.out[y * A.im.width + x];
            if (A.out_aligned) {
                // a whole sector; the samples of a large image pass through L2,
                // and should leave it first
                asm volatile("st.global.L1::no_allocate.L2::evict_first.v8.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};"
                             ::"l"(out), "r"(s.cluster), "r"(s.offset), "r"(s.count), "r"(s.covering), "r"(s.missing),
                             "r"(s.flags), "r"(__float_as_uint(s.view_z)), "r"(__float_as_uint(s.linear_depth))
                             : "memory");
            } else {
                *out = s;
            }
        }
    }
}

// ---------------------------------------------------------------------------
// Shading.
// ---------------------------------------------------------------------------
struct V3 {
    float x, y, z;
};

__device__ __forceinline__ V3 v3_sub(V3 a, V3 b) { return {cf_fsub(a.x, b.x), cf_fsub(a.y, b.y), cf_fsub(a.z, b.z)}; }
__device__ __forceinline__ V3 v3_add(V3 a, V3 b) { return {cf_fadd(a.x, b.x), cf_fadd(a.y, b.y), cf_fadd(a.z, b.z)}; }
__device__ __forceinline__ float v3_dot(V3 a, V3 b)
{
    return cf_fadd(cf_fadd(cf_fmul(a.x, b.x), cf_fmul(a.y, b.y)), cf_fmul(a.z, b.z));
}
// normalize(v) = v / sqrt(dot(v, v)), componentwise division
__device__ __forceinline__ V3 v3_normalize(V3 v)
{
    const float l = cf_fsqrt(v3_dot(v, v));
    return {cf_fdiv(v.x, l), cf_fdiv(v.y, l), cf_fdiv(v.z, l)};
}

constexpr float kPi = 3.14159265358979323846f;  // PBRHeader.glsl's PI as a GLSL float

// What Radiance reads of a texel, one array per field over the texels of a warp.
enum TexelField { kPx, kPy, kPz, kNx, kNy, kNz, kVx, kVy, kVz, kAx, kAy, kAz, kFx, kFy, kFz, kA2, kAlphaR, kGv, kNoV4, kKm,
                  kTexelFields };

// Shared memory of one shading warp.
struct ShadeWarp {
    float f[kTexelFields][32];
    uint32_t light[64];    // ring of (light, texel) pairs to evaluate
    uint32_t texel[64];
    union {
        struct {
            float term[3][32];   // what the pairs being evaluated add
            uint32_t pairs[32];  // ... and which of them are a texel's
        };
        struct {
            float x[32], y[32], z[32], e[32];  // a list's lights as out_of_reach sees them
        };
    };
};

// Radiance (Radiance.glsl:2-57) of one light at texel t of w, in the shader's
// operation order, plus the zero its Lo starts from.
__device__ __forceinline__ void radiance(const CfLightData* __restrict__ light, const ShadeWarp& w, uint32_t t,
                                         const CfPBRPushConstant& pc, float out[3])
{
    const float4 q = __ldg(reinterpret_cast<const float4*>(&light->position[0]));
    const float4 col = __ldg(reinterpret_cast<const float4*>(&light->color[0]));
    const float radius = __ldg(&light->radius);
    const V3 N = {w.f[kNx][t], w.f[kNy][t], w.f[kNz][t]}, V = {w.f[kVx][t], w.f[kVy][t], w.f[kVz][t]};
    const V3 d = v3_sub(V3{q.x, q.y, q.z}, V3{w.f[kPx][t], w.f[kPy][t], w.f[kPz][t]});
    const V3 L = v3_normalize(d);
    const V3 H = v3_normalize(v3_add(V, L));
    const float NoH = cf_glsl_max(v3_dot(N, H), 0.0f);
    const float NoL = cf_glsl_max(v3_dot(N, L), 0.0f);
    const float HoV = cf_glsl_max(v3_dot(H, V), 0.0f);
    const float dist = cf_fsqrt(v3_dot(d, d));
    const float att = cf_fdiv(cf_glsl_max(cf_fsub(1.0f, cf_fdiv(dist, radius)), 0.0f), cf_pow_pinned(dist, pc.lightFalloff));
    const float rad[3] = {cf_fmul(cf_fmul(col.x, att), pc.lightIntensity), cf_fmul(cf_fmul(col.y, att), pc.lightIntensity),
                          cf_fmul(cf_fmul(col.z, att), pc.lightIntensity)};
    // DistributionGGX (PBRHeader.glsl:17-28)
    const float a2 = w.f[kA2][t];
    const float den0 = cf_fadd(cf_fmul(cf_fmul(NoH, NoH), cf_fsub(a2, 1.0f)), 1.0f);
    const float D = cf_fdiv(a2, cf_fmul(cf_fmul(kPi, den0), den0));
    // GeometrySchlickGGX (PBRHeader.glsl:41-46); the texel's factor is kGv
    const float alpha_r = w.f[kAlphaR][t];
    const float G = cf_fmul(cf_fdiv(NoL, cf_fadd(cf_fmul(NoL, cf_fsub(1.0f, alpha_r)), alpha_r)), w.f[kGv][t]);
    // FresnelSchlick (PBRHeader.glsl:50-53)
    const float p5 = cf_pow_pinned(cf_glsl_min(cf_glsl_max(cf_fsub(1.0f, HoV), 0.0f), 1.0f), 5.0f);
    const float DG = cf_fmul(D, G);
    const float denom = cf_fadd(cf_fmul(w.f[kNoV4][t], NoL), 0.0001f);
    const float km = w.f[kKm][t];
#pragma unroll
    for (int c = 0; c < 3; ++c) {
        const float f0 = w.f[kFx + c][t];
        const float F = cf_fadd(f0, cf_fmul(cf_fsub(1.0f, f0), p5));
        const float spec = cf_fdiv(cf_fmul(DG, F), denom);
        const float kd = cf_fmul(cf_fsub(1.0f, F), km);
        const float diff = cf_fdiv(cf_fmul(kd, w.f[kAx + c][t]), kPi);
        // Radiance's own Lo starts at vec3(0.0) (Radiance.glsl:13,55): the
        // term is added to zero before Scene.frag adds it to its Lo, which
        // turns a -0 term into +0
        out[c] = cf_fadd(0.0f, cf_fmul(cf_fmul(cf_fadd(diff, spec), rad[c]), NoL));
    }
}

// A light as the tests of out_of_reach see it: its position and the squared
// distance from which it is out of reach, +inf for a light whose colour or
// radius rules the tests out.
struct ReachLimits {
    float dd_min, dd_max;  // squared distances between which pow(dist, falloff) is in [2^-20, 2^20]; dd_max < 0: none
};
constexpr float kMost = 1048576.0f;     // 2^20: largest colour component and intensity the tests take
constexpr float kMostTexel = 1024.0f;   // ... and largest albedo, F0 and metallic
__device__ __forceinline__ float4 reach_entry(const CfLightData* __restrict__ light)
{
    const float4 q = __ldg(reinterpret_cast<const float4*>(&light->position[0]));
    const float4 col = __ldg(reinterpret_cast<const float4*>(&light->color[0]));
    const float r = __ldg(&light->radius);
    const bool plain = r > 0.0f && r <= 1e18f && fabsf(col.x) <= kMost && fabsf(col.y) <= kMost && fabsf(col.z) <= kMost;
    // a little above r^2: the product is rounded
    return make_float4(q.x, q.y, q.z, plain ? r * r * 1.000001f : __uint_as_float(0x7f800000u));
}

// Whether a light adds exactly +0 to a texel.  Its term is ((diff + spec) *
// rad) * NoL with rad = (color * att) * intensity and att = max(1 - dist /
// radius, 0) / pow(dist, falloff).
//   At or beyond the radius the numerator is +0 and att +0: rad is a zero.
//   Behind the texel's surface, N.d below zero by more than rounding can turn
//   (the shader's N.L is within 1e-6 of it), NoL is +0.
// Either way the term is a zero, as long as every other factor is finite, and
// Radiance's 0 + term is +0.  They are: the distance is inside the limits, so
// att is at most 2^20 and rad at most 2^60; the light is not opposite the
// camera, so V + L keeps a length of at least 0.1 and H is a unit vector up to
// rounding; and the texel is `tame` (see shade_kernel), which bounds diff + spec.
// With d from the texel to the light: dd = d.d, vd = V.d, nd = N.d; e: the
// light's reach_entry squared distance.
__device__ __forceinline__ bool out_of_reach(float e, const ReachLimits& lim, float dd, float vd, float nd)
{
    const bool far = dd >= e, behind = nd < 0.0f && nd * nd > 1e-10f * dd && e <= 3e38f;
    return (far || behind) && dd >= lim.dd_min && dd <= lim.dd_max && (vd >= 0.0f || vd * vd <= 0.98f * dd);
}

// The same for the first n lights of w (n up to 32, rounded up to four) at one
// texel: a mask of those that may add something.  Two lights per packed
// operation, and fused ones: the test's margins are wider than any rounding.
__device__ __forceinline__ uint32_t within_reach(const ShadeWarp& w, uint32_t n, const ReachLimits& lim, V3 P, V3 V, V3 N)
{
    using namespace cfk;
    const f2 px = f2_pack(P.x, P.x), py = f2_pack(P.y, P.y), pz = f2_pack(P.z, P.z), vx = f2_pack(V.x, V.x),
             vy = f2_pack(V.y, V.y), vz = f2_pack(V.z, V.z), nx = f2_pack(N.x, N.x), ny = f2_pack(N.y, N.y),
             nz = f2_pack(N.z, N.z);
    uint32_t word = 0;
    for (uint32_t j = 0; j < n; j += 4) {
        const float4 x = *reinterpret_cast<const float4*>(&w.x[j]);
        const float4 y = *reinterpret_cast<const float4*>(&w.y[j]);
        const float4 z = *reinterpret_cast<const float4*>(&w.z[j]);
        const float4 e = *reinterpret_cast<const float4*>(&w.e[j]);
        const float far[4] = {e.x, e.y, e.z, e.w};
        float dd[4], vd[4], nd[4];
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            const f2 dx = f2_sub(h ? f2_pack(x.z, x.w) : f2_pack(x.x, x.y), px),
                     dy = f2_sub(h ? f2_pack(y.z, y.w) : f2_pack(y.x, y.y), py),
                     dz = f2_sub(h ? f2_pack(z.z, z.w) : f2_pack(z.x, z.y), pz);
            f2_unpack(f2_fma(dz, dz, f2_fma(dy, dy, f2_mul(dx, dx))), dd[2 * h], dd[2 * h + 1]);
            f2_unpack(f2_fma(vz, dz, f2_fma(vy, dy, f2_mul(vx, dx))), vd[2 * h], vd[2 * h + 1]);
            f2_unpack(f2_fma(nz, dz, f2_fma(ny, dy, f2_mul(nx, dx))), nd[2 * h], nd[2 * h + 1]);
        }
        uint32_t m = 0;
#pragma unroll
        for (int q = 0; q < 4; ++q) m |= out_of_reach(far[q], lim, dd[q], vd[q], nd[q]) ? 0u : 1u << q;
        word |= m << j;
    }
    return word;
}

struct ShadeArgs {
    CfClusterForwardUBO u;
    Image im;
    CfPBRPushConstant pc;
    float cam[3];
    ReachLimits lim;
    const CfGBufferTexel* gbuf;
    const CfLightCell* cells;
    const uint32_t* indices;
    uint64_t index_count;
    const CfLightData* lights;
    float4* out;
    uint32_t light_count;
};

// Evaluates the ring's pairs [at, at + n) and adds their terms to the texels'
// sums (lane i: texel i's), each texel's in the ring's order.
__device__ __forceinline__ void evaluate_pairs(const ShadeArgs& A, ShadeWarp& w, uint32_t at, uint32_t n, uint32_t lane,
                                               float lo[3])
{
    w.pairs[lane] = 0;
    __syncwarp();
    const uint32_t t = lane < n ? w.texel[(at + lane) & 63u] : 32u;
    const uint32_t same = __match_any_sync(cfk::kFull, t);
    if (lane < n) {
        float term[3];
        radiance(&A.lights[w.light[(at + lane) & 63u]], w, t, A.pc, term);
#pragma unroll
        for (int c = 0; c < 3; ++c) w.term[c][lane] = term[c];
        w.pairs[t] = same;
    }
    __syncwarp();
    for (uint32_t m = w.pairs[lane]; m; m &= m - 1) {
        const uint32_t k = __ffs(m) - 1;
#pragma unroll
        for (int c = 0; c < 3; ++c) lo[c] = cf_fadd(lo[c], w.term[c][k]);
    }
    __syncwarp();
}

// One CTA per tile of texels.  Bound by issue (80% of the slots on surfaces):
// some 600 instructions per 32 lights evaluated, with eighteen IEEE divisions
// and two square roots.  Most listed lights add nothing (of 20 listed on
// surfaces 3 reach the texel), so each is tested first: the lanes of a warp
// fetch the entries of each cluster that its texels lie in, 32 at a time, and
// each of the cluster's texels tests them four at a time (21 instructions an
// entry), or, where the cluster has few of the texels, the lanes test their
// entries against one texel after another.  The pairs that may add something
// are gathered per warp and evaluated 32 at a time, so that no lane idles while
// others evaluate.  1920x1080, 1024 lights, surfaces with 20 listed lights a
// texel: every light evaluated 776 us, tested one by one from each texel's own
// list 228 us, so 164 us (2400 instructions per 32 texels, two thirds of them in
// 3.7 evaluations); every texel at its own depth 1113 / 139 / 121 us.
// A cluster's pairs are gathered entry by entry or, where it has few of the
// texels, texel by texel: entry by entry, lists that all reach took a step for
// each pair (5804x17, 35x14x33, 2903 lights that reach everything: one thread
// per texel 1264 us, entry by entry 4103, texel by texel 2098; 354x27, 79x47x8,
// 104 lights: 114 / 235 / 165).
// Lists up to kShortList each texel walks itself, as the lists of many clusters
// one after another cost more than they save: 27x4x55, four lights a list,
// scattered depths 62 us against 76; with a limit of 4 / 8 / 16 the surfaces above take
// 164 / 166 / 172 us.
// In the smaller images, bound by the latency of a cluster's round trips, also
// lists of up to kOwnEntries entries for each of the warp's clusters: 96x64,
// 40x24x56, 8000 lights, scattered depths: one thread per texel 132 us, without
// this rule 150, with 1 / 2 / 4 entries 149 / 149 / 68.
// The tile's clusters are looked up before it is sorted: a tile of unlit ones is
// not sorted, and its texels ask for nothing but their albedo.  1920x1080 without
// a light in sight: one thread per texel 28.7 us, all tiles sorted 40.2, this 29.7;
// 100 lights, surfaces 36.9 / 55.0 / 47.4.  (Leaving tiles of short lists unsorted
// too costs scattered depths more than it saves surfaces: 100 lights 46.5 -> 54.0
// against 46.0 -> 45.4.)
constexpr uint32_t kShortList = 6, kOwnEntries = 4;
constexpr uint32_t kNoCluster = ~0u;
constexpr uint32_t kFewTexels = 2;  // entries per texel from which a texel's turn is cheaper than four entries' test
template <uint32_t kSide, uint32_t kThreads>
__global__ void __launch_bounds__(kThreads) shade_kernel(const __grid_constant__ ShadeArgs A)
{
    constexpr uint32_t kPixels = kSide * kSide, kUnits = kPixels / 32;
    __shared__ uint16_t order[kPixels];
    __shared__ uint32_t clusters[kPixels];  // kNoCluster: outside of the grid
    __shared__ TileSort sort;
    __shared__ TileAxes<kSide> axes;
    __shared__ __align__(16) ShadeWarp warps[kThreads / 32];
    const uint32_t lane = threadIdx.x & 31, lt_mask = (1u << lane) - 1u;
    ShadeWarp& w = warps[threadIdx.x >> 5];
    const Tile<kSide> tile(A.im);
    cfk::grid_dependency_wait();
    cfk::launch_dependents();
    fill_axes(A.u, A.im, tile, axes);
    __syncthreads();
    bool any_lit = false;
    float z[kPixels / kThreads];
#pragma unroll
    for (uint32_t q = 0; q < kPixels / kThreads; ++q) {
        uint32_t x, y;
        z[q] = tile.at(A.im, q * kThreads + threadIdx.x, x, y) ? __ldg(&A.gbuf[y * A.im.width + x].position[3]) : 0.0f;
    }
#pragma unroll
    for (uint32_t q = 0; q < kPixels / kThreads; ++q) {
        const uint32_t i = q * kThreads + threadIdx.x;
        uint32_t x, y, c = kNoCluster;
        if (tile.at(A.im, i, x, y)) {
            const float xf = A.im.tiles_x ? axes.tile[0][i % kSide] : tile_coord(x, A.im.tile_w);
            const float yf = A.im.tiles_x ? axes.tile[1][i / kSide] : tile_coord(y, A.im.tile_h);
            float lin;
            if (fragment_cluster(A.u, xf, yf, z[q], &c, &lin)) any_lit = any_lit || A.cells[c].count != 0;
        }
        clusters[i] = c;
    }
    if (__syncthreads_or(any_lit)) {
        sort_tile<true, kSide, kThreads>(A.u, A.im, tile, axes, sort, order, [&](uint32_t q, uint32_t) { return z[q]; });
    } else {
        for (uint32_t i = threadIdx.x; i < kPixels; i += kThreads) {
            uint32_t x, y;
            order[i] = (uint16_t)(tile.at(A.im, i, x, y) ? i : kNoPixel);
        }
        if (threadIdx.x == 0) sort.next = 0;
        __syncthreads();
    }
    for (uint32_t unit; (unit = next_unit(sort, lane)) < kUnits;) {
        const uint32_t i = order[unit * 32 + lane];
        const bool valid = i != kNoPixel;
        if (!__any_sync(cfk::kFull, valid)) continue;
        uint32_t x = 0, y = 0, off = 0, cnt = 0;
        float alpha = 0.0f;
        if (valid) {
            tile.at(A.im, i, x, y);
            const uint32_t c = clusters[i];
            if (c != kNoCluster) {
                const CfLightCell cell = A.cells[c];
                if ((uint64_t)cell.offset + cell.count <= A.index_count) {
                    alpha = 1.0f;
                    off = cell.offset;
                    cnt = cell.count;
                }
            }
        }
        const uint32_t pix = y * A.im.width + x;
        const float4* t = reinterpret_cast<const float4*>(&A.gbuf[pix]);
        const float4 alb = __ldg(&t[2]);
        const float al[3] = {alb.x, alb.y, alb.z};
        float lo[3];
#pragma unroll
        for (int k = 0; k < 3; ++k) lo[k] = cf_fmul(al[k], A.pc.albedoMultipler);
        const uint32_t longest = __reduce_max_sync(cfk::kFull, cnt);
        if (longest == 0) {  // the texels of unlit clusters: nothing else is asked of them
            if (valid) A.out[pix] = make_float4(lo[0], lo[1], lo[2], alpha);
            continue;
        }
        const float4 pos = __ldg(&t[0]), nrm = __ldg(&t[1]);
        const V3 P = {pos.x, pos.y, pos.z}, N = {nrm.x, nrm.y, nrm.z};
        const float metallic = nrm.w, roughness = alb.w;
        // Scene.frag:82-115: V, NoV, F0 = mix(baseReflectivity, albedo, metallic), Lo = albedo * albedoMultipler
        const V3 V = v3_normalize(v3_sub(V3{A.cam[0], A.cam[1], A.cam[2]}, P));
        const float NoV = cf_glsl_max(v3_dot(N, V), 0.0f);
        const float mi = cf_fsub(1.0f, metallic);
        const float r1 = cf_fadd(roughness, 1.0f);
        const float alpha_r = cf_fdiv(cf_fmul(r1, r1), 8.0f);  // AlphaDirectLighting (PBRHeader.glsl:32-37)
        const float a = cf_fmul(roughness, roughness), a2 = cf_fmul(a, a);
        w.f[kPx][lane] = P.x, w.f[kPy][lane] = P.y, w.f[kPz][lane] = P.z;
        w.f[kNx][lane] = N.x, w.f[kNy][lane] = N.y, w.f[kNz][lane] = N.z;
        w.f[kVx][lane] = V.x, w.f[kVy][lane] = V.y, w.f[kVz][lane] = V.z;
        bool colours = true;
#pragma unroll
        for (int c = 0; c < 3; ++c) {
            const float f0 = cf_fadd(cf_fmul(A.pc.baseReflectivity, mi), cf_fmul(al[c], metallic));
            w.f[kAx + c][lane] = al[c];
            w.f[kFx + c][lane] = f0;
            colours = colours && fabsf(al[c]) <= kMostTexel && fabsf(f0) <= kMostTexel;
        }
        w.f[kA2][lane] = a2;
        w.f[kAlphaR][lane] = alpha_r;
        w.f[kGv][lane] = cf_fdiv(NoV, cf_fadd(cf_fmul(NoV, cf_fsub(1.0f, alpha_r)), alpha_r));
        w.f[kNoV4][lane] = cf_fmul(4.0f, NoV);
        w.f[kKm][lane] = mi;
        // Tame: diff + spec is bounded.  V is a unit vector up to rounding, N
        // hardly longer than one, roughness in [0, 1.8] (alpha_r in [1/8, 1),
        // so both factors of G are at most 8), colours and metallic moderate
        // (diff at most 2^31).  NoH^2 is at most nn * (1 + 1.1e-6)
        // for any unit H, so DistributionGGX's denominator NoH^2 * (a2 - 1) + 1
        // stays above 3e-6 by the last condition, D below 2^39 and spec below
        // 2^70.  (All false for NaN.)
        const float vv = v3_dot(V, V), nn = v3_dot(N, N);
        const bool tame = colours && vv >= 0.999f && vv <= 1.001f && nn <= 1.0001f && roughness >= 0.0f &&
                          roughness <= 1.8f && fabsf(metallic) <= kMostTexel && a2 * nn + (1.0f - nn * 1.000002f) > 4e-6f;
        __syncwarp();
        bool lit = false;  // a light of the list is one of the set
        uint32_t put = 0, done = 0;
        // Rounds of up to 32 entries' tests.  Where all lists of the warp's texels
        // are short, a round is one entry of each texel's own; else 32 entries of
        // the list of one cluster after another, an entry fetched by each lane and
        // tested by each texel of the cluster.  (One loop over all rounds, so that
        // the evaluation is there once: it is half of the kernel's instructions.)
        bool own = longest <= kShortList;
        if (kSide == 16 && !own) {
            const uint32_t same = __match_any_sync(cfk::kFull, cnt ? off : ~0u);
            own = longest <= kOwnEntries * __popc(__ballot_sync(cfk::kFull, cnt && (same & lt_mask) == 0));
        }
        uint32_t todo = own ? 0u : __ballot_sync(cfk::kFull, cnt != 0), texels = 0, n_texels = 0, list = 0, left = 0, li = 0;
        if (own && cnt) li = __ldg(&A.indices[off]);
        uint32_t step = 0;
        bool mine = false;
        for (bool more = true; more;) {
            bool few = false;  // the cluster has few of the texels
            uint32_t any = 0, need = 0, here = 0;  // need: bit q: entry q may add something to the lane's texel
            if (own) {
                more = step < longest;
                if (more) {
                    const bool has = step < cnt;
                    here = li;
                    if (step + 1 < cnt) li = __ldg(&A.indices[off + step + 1]);  // for the next round
                    const bool light = has && here < A.light_count;
                    if (has && !light) alpha = 0.0f;  // an entry that is no light
                    if (light) {
                        lit = true;
                        const float4 e = reach_entry(&A.lights[here]);
                        const V3 d = v3_sub(V3{e.x, e.y, e.z}, P);
                        need = tame && out_of_reach(e.w, A.lim, v3_dot(d, d), v3_dot(V, d), v3_dot(N, d)) ? 0u : 1u;
                    }
                    any = __any_sync(cfk::kFull, need) ? 1u : 0u;
                    ++step;
                }
            } else {
                if (left == 0) {  // the next list
                    more = todo != 0;
                    if (more) {
                        const uint32_t leader = __ffs(todo) - 1;
                        list = __shfl_sync(cfk::kFull, off, leader);
                        left = __shfl_sync(cfk::kFull, cnt, leader);
                        mine = off == list && cnt == left;
                        texels = __ballot_sync(cfk::kFull, mine);
                        n_texels = __popc(texels);
                        todo &= ~texels;
                        li = lane < left ? __ldg(&A.indices[list + lane]) : 0u;
                    }
                }
                if (more) {
                    const uint32_t n = min(32u, left);
                    here = li;
                    const bool light = lane < n && here < A.light_count;
                    left -= n;
                    list += n;
                    if (lane < left) li = __ldg(&A.indices[list + lane]);  // for the next round
                    const float4 e = light ? reach_entry(&A.lights[here]) : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
                    const uint32_t lights = __ballot_sync(cfk::kFull, light);
                    if (mine) {
                        lit = lit || lights;
                        if (lights != (n < 32 ? (1u << n) - 1u : ~0u)) alpha = 0.0f;  // an entry that is no light
                    }
                    few = kFewTexels * n_texels < n;
                    if (few) {
                        for (uint32_t m = texels; m; m &= m - 1) {
                            const uint32_t t = __ffs(m) - 1;
                            const V3 d = v3_sub(V3{e.x, e.y, e.z}, V3{w.f[kPx][t], w.f[kPy][t], w.f[kPz][t]});
                            const float vd = v3_dot(V3{w.f[kVx][t], w.f[kVy][t], w.f[kVz][t]}, d);
                            const float nd = v3_dot(V3{w.f[kNx][t], w.f[kNy][t], w.f[kNz][t]}, d);
                            const uint32_t reach = __ballot_sync(cfk::kFull, !out_of_reach(e.w, A.lim, v3_dot(d, d), vd, nd));
                            if (lane == t) need = (tame ? reach : ~0u) & lights;
                        }
                    } else {
                        w.x[lane] = e.x;
                        w.y[lane] = e.y;
                        w.z[lane] = e.z;
                        w.e[lane] = e.w;
                        __syncwarp();
                        if (mine) need = (tame ? within_reach(w, n, A.lim, P, V, N) : ~0u) & lights;
                        __syncwarp();  // the next entries take these ones' place
                    }
                    any = __reduce_or_sync(cfk::kFull, need);
                }
            }
            // The pairs: of one entry after another and each texel, or of one texel
            // after another and each entry.
            uint32_t turns = 0;
            if (few && any) {
                turns = __ballot_sync(cfk::kFull, need != 0);
                any = 0;
            }
            for (;;) {
                if (any | turns) {
                    bool pair;
                    uint32_t light = here, texel = lane;
                    if (turns) {
                        texel = __ffs(turns) - 1;
                        turns &= turns - 1;
                        pair = (__shfl_sync(cfk::kFull, need, texel) >> lane) & 1u;
                    } else {
                        const uint32_t q = __ffs(any) - 1, from = __shfl_sync(cfk::kFull, here, q);
                        any &= any - 1;
                        pair = (need >> q) & 1u;
                        if (!own) light = from;
                    }
                    const uint32_t m = __ballot_sync(cfk::kFull, pair);
                    if (pair) {
                        const uint32_t at = (put + __popc(m & lt_mask)) & 63u;
                        w.light[at] = light;
                        w.texel[at] = texel;
                    }
                    put += __popc(m);
                }
                if (put - done >= 32 || (!more && put != done)) {
                    const uint32_t n = min(32u, put - done);
                    evaluate_pairs(A, w, done, n, lane, lo);
                    done += n;
                }
                if (!(any | turns)) break;
            }
        }
        __syncwarp();
        if (valid) {
            // the lights out of reach added +0, which turns a -0 sum into +0
#pragma unroll
            for (int k = 0; k < 3; ++k) lo[k] = lit ? cf_fadd(lo[k], 0.0f) : lo[k];
            A.out[pix] = make_float4(lo[0], lo[1], lo[2], alpha);
        }
        __syncwarp();
    }
}

// A tile of 32x32 pixels, whose sorted warps read one or two lists each, and as
// many threads as the image's tiles need to fill the GPU: 256 where there are
// four tiles per SM, 512 down to one, 1024 below that.  A lookup of less than a
// quarter of a tile per SM takes 16x16.  Lookup without the check, one thread
// per unsorted pixel / 1024 threads / 512 / tiles of 16x16, in us:
//   960x540, every pixel at its own depth, 3000 lights    75.4 / 41.2 / 32.8 / 45.5
//   960x540, surfaces                                     65.9 / 32.2 / 29.3 / 24.9
//   480x270, every pixel at its own depth                 43.5 / 25.5 / 25.1 / 36.5
//   480x270, the all-lights check                          812 / 53.1 / 57.9 / 76.4
// Shading's smaller images take 16x16: its warps need 3.5 KB of shared memory
// each.  Between four and eight tiles per SM, 512 threads a tile leave the last
// wave shorter: 940x1000, surfaces 44.0 -> 39.8 and 62.8 -> 53.4 us (scattered
// depths 83.5 -> 91.7, which gains from warps of few lists); above, 1920x1080
// takes 163 us with 256, 168 with 512.
constexpr uint64_t kLargePixels = 152ull * 4 * 1024, kMiddlePixels = 152ull * 1024, kSmallPixels = 152ull * 256;

Image image_of(const CfClusterForwardUBO& u, uint32_t width, uint32_t height, uint32_t side)
{
    Image im;
    im.width = width;
    im.height = height;
    im.n_pixels = width * height;
    im.tiles_x = width >= side && height >= side ? (width + side - 1) / side : 0u;
    im.tile_w = u.screenSize[0] / (float)u.sliceCountX;
    im.tile_h = u.screenSize[1] / (float)u.sliceCountY;
    return im;
}

unsigned image_blocks(const Image& im, uint32_t side)
{
    const uint64_t n = (uint64_t)side * side;
    return im.tiles_x ? im.tiles_x * ((im.height + side - 1) / side) : (unsigned)((im.n_pixels + n - 1) / n);
}

// Squared distances between which pow(dist, falloff) is in [2^-20, 2^20]:
// |log2 dist| <= k with k * |falloff| <= 20.
ReachLimits reach_limits(const CfPBRPushConstant& pc)
{
    const float f = std::fabs(pc.lightFalloff);
    if (!(f <= 20.0f) || !(std::fabs(pc.lightIntensity) <= kMost)) return {0.0f, -1.0f};
    const int k = f * 62.0f <= 20.0f ? 62 : (int)(20.0f / f);
    return {std::ldexp(1.0f, -2 * k), std::ldexp(1.0f, 2 * k)};
}

// A tile per CTA; the launch overlaps with the end of the stream's previous one.
template <typename Args>
cudaError_t launch_tiles(void (*kernel)(Args), const Args& A, uint32_t side, uint32_t threads, cudaStream_t stream)
{
    return cfk::launch_kernel(true, kernel, dim3(image_blocks(A.im, side)), dim3(threads), 0, stream, A);
}

template <bool kCheck>
cudaError_t launch_lookup(const LookupArgs& A, cudaStream_t stream)
{
    const uint64_t n = A.im.n_pixels;
    if (n >= kLargePixels) return launch_tiles(lookup_kernel<32, 256, kCheck>, A, 32, 256, stream);
    if (n >= kMiddlePixels) return launch_tiles(lookup_kernel<32, 512, kCheck>, A, 32, 512, stream);
    if (n >= kSmallPixels) return launch_tiles(lookup_kernel<32, 1024, kCheck>, A, 32, 1024, stream);
    return launch_tiles(lookup_kernel<16, 256, kCheck>, A, 16, 256, stream);
}

}  // namespace

extern "C" int cf_shade_clusters(const CfClusterForwardUBO* ubo, const float camera_position[3],
                                 const CfPBRPushConstant* pc, const CfGBufferTexel* d_gbuffer, uint32_t width,
                                 uint32_t height, const CfLightCell* d_cells, const uint32_t* d_indices,
                                 uint64_t index_count, const CfLightData* d_lights, uint32_t light_count,
                                 float* d_out, void* stream)
{
    using namespace cfrt;
    if (!ubo || !camera_position || !pc || !d_gbuffer || !d_cells || !d_out || (light_count && !d_lights) ||
        (index_count && !d_indices))
        return fail(CF_ERROR_INVALID_ARGUMENT, "cf_shade_clusters: null argument");
    uint32_t C = 0;
    const int st = validate_grid(ubo->sliceCountX, ubo->sliceCountY, ubo->sliceCountZ, 1, &C);
    if (st) return st;
    if ((float)width != ubo->screenSize[0] || (float)height != ubo->screenSize[1])
        return fail(CF_ERROR_INVALID_ARGUMENT, "G-buffer %ux%u does not match the UBO's screen %gx%g", width, height,
                    (double)ubo->screenSize[0], (double)ubo->screenSize[1]);
    const uint64_t n = (uint64_t)width * height;
    if (n == 0) return CF_SUCCESS;
    if (n > (1ull << 31)) return fail(CF_ERROR_INVALID_ARGUMENT, "G-buffer of %llu texels", (unsigned long long)n);
    if ((reinterpret_cast<uintptr_t>(d_lights) | reinterpret_cast<uintptr_t>(d_gbuffer) |
         reinterpret_cast<uintptr_t>(d_out)) & 15)
        return fail(CF_ERROR_INVALID_ARGUMENT, "lights, G-buffer and output must be 16-byte aligned");
    const bool large = n >= kLargePixels;
    ShadeArgs A;
    A.u = *ubo;
    A.im = image_of(*ubo, width, height, large ? 32 : 16);
    A.pc = *pc;
    for (int i = 0; i < 3; ++i) A.cam[i] = camera_position[i];
    A.lim = reach_limits(*pc);
    A.gbuf = d_gbuffer;
    A.cells = d_cells;
    A.indices = d_indices;
    A.index_count = index_count;
    A.lights = d_lights;
    A.out = reinterpret_cast<float4*>(d_out);
    A.light_count = light_count;
    const cudaStream_t on = (cudaStream_t)stream;
    const cudaError_t e = n >= 2 * kLargePixels ? launch_tiles(shade_kernel<32, 256>, A, 32, 256, on)
                          : large               ? launch_tiles(shade_kernel<32, 512>, A, 32, 512, on)
                                                : launch_tiles(shade_kernel<16, 256>, A, 16, 256, on);
    return e == cudaSuccess ? CF_SUCCESS : cuda_fail(e, "clustered shading launch");
}

extern "C" int cf_lookup_clusters(const CfClusterForwardUBO* ubo, const float* d_depth, uint32_t width, uint32_t height,
                                  const CfLightCell* d_cells, const uint32_t* d_indices, uint64_t index_count,
                                  const CfLightData* d_lights, uint32_t light_count, uint32_t cap,
                                  const CfAABB* d_aabbs, int check_all_lights, CfFragmentSample* d_out, void* stream)
{
    using namespace cfrt;
    if (!ubo || !d_depth || !d_cells || !d_out || (light_count && !d_lights) || (index_count && !d_indices))
        return fail(CF_ERROR_INVALID_ARGUMENT, "cf_lookup_clusters: null argument");
    uint32_t C = 0;
    const int st = validate_grid(ubo->sliceCountX, ubo->sliceCountY, ubo->sliceCountZ, cap ? cap : 1, &C);
    if (st) return st;
    if ((float)width != ubo->screenSize[0] || (float)height != ubo->screenSize[1])
        return fail(CF_ERROR_INVALID_ARGUMENT, "depth buffer %ux%u does not match the UBO's screen %gx%g", width, height,
                    (double)ubo->screenSize[0], (double)ubo->screenSize[1]);
    const uint64_t n = (uint64_t)width * height;
    if (n == 0) return CF_SUCCESS;
    if (n > (1ull << 31)) return fail(CF_ERROR_INVALID_ARGUMENT, "depth buffer of %llu pixels", (unsigned long long)n);
    if (reinterpret_cast<uintptr_t>(d_lights) & 15 || reinterpret_cast<uintptr_t>(d_aabbs) & 15)
        return fail(CF_ERROR_INVALID_ARGUMENT, "lights and AABBs must be 16-byte aligned");
    LookupArgs A;
    A.u = *ubo;
    A.im = image_of(*ubo, width, height, n < kSmallPixels ? 16 : 32);
    A.depth = d_depth;
    A.cells = d_cells;
    A.indices = d_indices;
    A.index_count = index_count;
    A.lights = d_lights;
    A.aabbs = reinterpret_cast<const float4*>(d_aabbs);
    A.out = d_out;
    A.light_count = light_count;
    A.cap = cap ? cap : 0xFFFFFFFFu;
    A.out_aligned = (reinterpret_cast<uintptr_t>(d_out) & 31) == 0;
    const cudaError_t e = check_all_lights ? launch_lookup<true>(A, (cudaStream_t)stream)
                                           : launch_lookup<false>(A, (cudaStream_t)stream);
    return e == cudaSuccess ? CF_SUCCESS : cuda_fail(e, "cluster lookup launch");
}
