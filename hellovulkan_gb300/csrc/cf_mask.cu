// cf_mask.cu — binned culling with hit masks (LightCulling.comp:26-87): five
// launches from lights and AABBs to cells and the packed index list, for one
// view or for every view of a batch.
//
//   box_kernel     one CTA per depth slice: the union box of the slice and of
//                  each group of 32 consecutive clusters, and the reset of
//                  the words that the later launches count in
//   list_kernel    one CTA per segment of lights and block of slices:
//                  transforms its lights (posView = cameraView * position,
//                  r^2) and writes, per slice, those whose sphere reaches the
//                  slice's box, in light order, into the segment's own part of
//                  the slice's list.  No segment needs another's count.  A list
//                  ends where lights that reach the whole slice have filled its
//                  clusters' lists (see list_covering).
//   scan_kernel    warps take units, each a run of a slice's candidates against
//                  one group: the warp keeps the lights that reach the group's
//                  union box and tests each of them against 32 clusters, one
//                  per lane; a lane's results for 32 lights are one mask word
//                  in shared memory.  The masks and the lights' indices go to
//                  the view's pool.  No warp waits for another, and a dense
//                  group's work spreads over many.
//   sum_kernel     one CTA per group, or 32: adds up the units' counts
//   emit_kernel    warps write the groups' cells, and the units' hits from
//                  their masks straight to their places in the packed list
//
// Why this split.  A view's hits are concentrated: on the 2560x1600 view with
// 16384 lights one group of 864 has a twentieth of all (light, group) pairs, and
// half the slices none.  CTAs that own a group and take its candidates in
// tiles (cull_pipe_kernel) are bound by the longest ones; here the longest unit
// is 128 candidates, units of one group go to different SMs, and slices that
// nothing reaches cost nothing.  What is left is latency: the five launches of
// a single view overlap by programmatic dependent launch, and each is a chain
// of two to five L2 round trips (0.5 us each) with 0.9 us to the next launch.
// Batches are bound by issue (1.9 to 2.9 of 4 instructions per cycle in the
// list, scan and write launches).  Measured, back-to-back passes, against the
// staged path: that view 33.8 -> 21.9 us; 65536 lights 77.4 -> 35.5 us; 64 views
// of the benchmark's mix 371 -> 106 us; 256 animated views of 4096 lights
// 1485 -> 234 us.
//
// The tests are the ones of cf_device.cuh; pruning by union box is exact: per
// axis the distance to a box that contains another is never larger, and the
// rounded squares and sums are monotonic.  A NaN bound makes a union infinite.
#include "cf_kernels.cuh"
#include "cf_device.cuh"
#include "cf_launch.cuh"

#include <algorithm>

#include "cf_pinned_math.h"

namespace cfk {
namespace {

constexpr uint32_t kGroup = kMaskGroup;  // clusters per group: one per lane

// ---------------------------------------------------------------------------
// Slice and group boxes.
// ---------------------------------------------------------------------------
// threads per slice: a view's own launch reduces up to 1024 clusters in one
// step; a batch has slices enough to fill the GPU with smaller CTAs, whose
// warps wait less for one another (256 animated views: 359 us with 256 threads,
// 350 with 128, 346 with 64)
constexpr uint32_t kBoxThreads = 1024, kBoxThreadsBatch = 64;

__device__ __forceinline__ float4 min4(float4 a, float4 b)
{
    return make_float4(fminf(a.x, b.x), fminf(a.y, b.y), fminf(a.z, b.z), 0.f);
}
__device__ __forceinline__ float4 max4(float4 a, float4 b)
{
    return make_float4(fmaxf(a.x, b.x), fmaxf(a.y, b.y), fmaxf(a.z, b.z), 0.f);
}

// The union of the lanes' boxes, in every lane: six instructions, for sixty of a
// butterfly of shuffles.
__device__ __forceinline__ void warp_union(float4& lo, float4& hi)
{
    lo = make_float4(warp_min(lo.x), warp_min(lo.y), warp_min(lo.z), 0.f);
    hi = make_float4(warp_max(hi.x), warp_max(hi.y), warp_max(hi.z), 0.f);
}

constexpr uint32_t kBoxIlp = 4;  // groups a warp has loads in flight for (256 views: 43 -> 34 us, the traffic's 19)

template <uint32_t kThreads>
__device__ __forceinline__ void box_body(const ViewCull& v, uint32_t k)
{
    constexpr uint32_t kWarps = kThreads / 32;
    __shared__ float4 s_lo[kWarps], s_hi[kWarps];
    const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const uint32_t xy = v.slice_clusters, gps = (xy + kGroup - 1) / kGroup;
    const float inf = __uint_as_float(0x7f800000u);
    const uint32_t blocks = (v.groups + kGroup - 1) / kGroup;
    for (uint32_t u = k + v.slices * threadIdx.x; u < blocks; u += v.slices * kThreads) v.block_total[u] = 0u;
    if (threadIdx.x == 0) {
        v.slice_total[k] = make_uint2(0u, 0u);
        v.slice_stop[k] = ~0u;
        if (k == 0) *v.pool_head = 0ull;
    }
    float4 lo = make_float4(inf, inf, inf, 0.f), hi = make_float4(-inf, -inf, -inf, 0.f);
    for (uint32_t g0 = warp; g0 < gps; g0 += kBoxIlp * kWarps) {
        float4 a[kBoxIlp], b[kBoxIlp];
#pragma unroll
        for (uint32_t e = 0; e < kBoxIlp; ++e) {
            const uint32_t c = (g0 + e * kWarps) * kGroup + lane;
            a[e] = make_float4(inf, inf, inf, 0.f);
            b[e] = make_float4(-inf, -inf, -inf, 0.f);
            if (c < xy) {
                a[e] = __ldg(&v.aabbs[2 * ((size_t)k * xy + c)]);
                b[e] = __ldg(&v.aabbs[2 * ((size_t)k * xy + c) + 1]);
            }
        }
#pragma unroll
        for (uint32_t e = 0; e < kBoxIlp; ++e) {
            const uint32_t g = g0 + e * kWarps;
            if (g >= gps) break;
            const bool odd = g * kGroup + lane < xy && !(a[e].x <= b[e].x && a[e].y <= b[e].y && a[e].z <= b[e].z);
            warp_union(a[e], b[e]);
            if (__any_sync(kFull, odd)) {  // a NaN, or bounds the wrong way round (see covers)
                a[e] = make_float4(-inf, -inf, -inf, 0.f);
                b[e] = make_float4(inf, inf, inf, 0.f);
            }
            lo = min4(lo, a[e]);
            hi = max4(hi, b[e]);
            if (lane < 2) v.group_boxes[2 * ((size_t)k * gps + g) + lane] = lane ? b[e] : a[e];
        }
    }
    if (lane == 0) {
        s_lo[warp] = lo;
        s_hi[warp] = hi;
    }
    __syncthreads();
    if (warp == 0) {
        lo = s_lo[lane % kWarps];
        hi = s_hi[lane % kWarps];
        warp_union(lo, hi);
        if (lane == 0) {
            v.slice_boxes[2 * k] = lo;
            v.slice_boxes[2 * k + 1] = hi;
        }
    }
}

template <uint32_t kThreads>
__global__ void __launch_bounds__(kThreads) box_kernel(const ViewJob* __restrict__ jobs,
                                                            const uint32_t* __restrict__ prefix, uint32_t n_views,
                                                            const __grid_constant__ ViewJob single)
{
    grid_dependency_wait();
    // after the wait: the list launch starts once every earlier launch has
    // finished, so it may read the lights before its own wait
    launch_dependents();
    if (jobs) {
        const uint32_t vi = find_view(prefix, n_views, blockIdx.x);
        box_body<kThreads>(jobs[vi].v, blockIdx.x - __ldg(&prefix[vi]));
    } else {
        box_body<kThreads>(single.v, blockIdx.x);
    }
}

// ---------------------------------------------------------------------------
// Candidate lists.
// ---------------------------------------------------------------------------
// Most slices per CTA: its lights are read and transformed once for all of them
// (256 animated views: 289 us with 16, 279 with 32).
constexpr uint32_t kListSlices = 32;

__device__ __forceinline__ bool reaches(const float4& L, const float4& lo, const float4& hi)
{
    const float mn[3] = {lo.x, lo.y, lo.z}, mx[3] = {hi.x, hi.y, hi.z};
    return hit_fast(L, mn, mx);
}

// Whether a light reaches every cluster of a slice whose boxes lie in [lo, hi],
// by a test that may say no when it does: per axis a box is no further from it
// than the further side of the union, rounded operation by rounded operation
// (see box_body for boxes of which that does not hold).
__device__ __forceinline__ bool covers(const float4& L, const float4& lo, const float4& hi)
{
    const float dx = max3f(cf_fsub(hi.x, L.x), cf_fsub(L.x, lo.x), 0.0f), dy = max3f(cf_fsub(hi.y, L.y), cf_fsub(L.y, lo.y), 0.0f),
                dz = max3f(cf_fsub(hi.z, L.z), cf_fsub(L.z, lo.z), 0.0f);
    return cf_fadd(cf_fadd(cf_fmul(dx, dx), cf_fmul(dy, dy)), cf_fmul(dz, dz)) < L.w;
}

// A slice's list ends where its clusters' lists are full for certain: with the
// segment in which the covering lights reach the cap.  The higher half of a
// seg_count word is how many of the segment's lights cover the slice, that of
// slice_total their number in all segments; where one segment has as many as the
// cap, slice_stop is the first such segment and the lights it lists up to the
// last one that is needed.  Without an end, the many lights of full lists were
// all scanned, where the staged kernels stop at a cluster's cap; staged / without
// / with it, in us:
//   46x51x9,  39359 lights that reach all, cap 150    54 /  622 / 115
//   32x18x48, 24181 of radius 20 to 60, cap 255       75 /  247 /  97
//   22 views of 36x10x53, 18698 that reach all       814 / 6500 / 1021
//   24x14x32, 10658 that reach all, cap 150           33 /  128 /  36
constexpr uint32_t kCountMask = 0xffffu;
constexpr uint32_t kStopShift = 11;
static_assert(kMaxSegLights < 1u << kStopShift);
// Lights of a warp that reach a slice from which they are tested for covering
// it: the second view above 143 us with 16, 97 with 8 or 4, and views whose lists
// are not full take as long.
constexpr uint32_t kCoverMin = 8;

// Counts the covering lights of a list CTA's segment (slices z0 to z0 + nz, boxes
// and masks as list_body has them; `most`: the slices to test the warp's lights
// for).  Every thread of the CTA takes part.  Out of line: its registers would
// be every CTA's, and few segments have such lights.
__device__ __noinline__ void list_covering(const ViewCull& v, float4 L, uint32_t most, const float4* s_box,
                                           const uint32_t (*s_mask)[32], uint32_t seg, uint32_t z0, uint32_t nz)
{
    __shared__ uint32_t s_covers[kListSlices][32];
    const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
    for (uint32_t q = 0; q < nz; ++q) {
        uint32_t n = 0;
        if ((most >> q) & 1u) n = __popc(__ballot_sync(kFull, covers(L, s_box[2 * q], s_box[2 * q + 1])));
        if (lane == 0) s_covers[q][warp] = n;
    }
    __syncthreads();
    for (uint32_t q = warp; q < nz; q += nw) {
        const uint32_t covering = warp_inclusive_scan(lane < nw ? s_covers[q][lane] : 0u, lane);
        const uint32_t listed = warp_inclusive_scan(lane < nw ? __popc(s_mask[q][lane]) : 0u, lane);
        if (lane == 31 && covering) {
            v.seg_count[(size_t)(z0 + q) * v.segs + seg] = listed | covering << 16;
            atomicAdd(&v.slice_total[z0 + q].y, covering);
        }
        const uint32_t enough = __ballot_sync(kFull, covering >= v.cap);
        if (enough && lane == __ffs(enough) - 1) atomicMin(&v.slice_stop[z0 + q], seg << kStopShift | listed);
    }
}

__device__ __forceinline__ void list_body(const ViewJob& j, uint32_t blk)
{
    __shared__ uint32_t s_mask[kListSlices][32];
    __shared__ uint32_t s_off[kListSlices][32];
    __shared__ float4 s_box[2 * kListSlices], s_quad[2 * kListSlices / 4];
    const ViewCull& v = j.v;
    const uint32_t tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, nw = blockDim.x >> 5;
    const uint32_t seg = blk % v.segs, z0 = (blk / v.segs) * v.list_slices;
    const uint32_t nz = min(v.list_slices, v.slices - z0);
    const uint32_t i = seg * v.seg_lights + tid;
    float4 L = make_float4(0.0f, 0.0f, 0.0f, __uint_as_float(0xff800000u));  // past the lights: reaches nothing
    if (i < j.light_count) {
        // Read before the wait below: the box launch lets this one start only
        // once every earlier launch has finished.  From L2, not from an L1
        // that may hold the lights of an earlier frame.
        const float4 p = __ldcg(reinterpret_cast<const float4*>(&j.lights[i].position[0]));
        const float r = __ldcg(&j.lights[i].radius);
        L.x = cf_mat4_row(j.view, 0, p.x, p.y, p.z, p.w);
        L.y = cf_mat4_row(j.view, 1, p.x, p.y, p.z, p.w);
        L.z = cf_mat4_row(j.view, 2, p.x, p.y, p.z, p.w);
        L.w = cf_fmul(r, r);
    }
    grid_dependency_wait();  // the boxes
    launch_dependents();
    if (tid < 2 * nz) s_box[tid] = v.slice_boxes[2 * z0 + tid];
    __syncthreads();
    if (tid < (nz + 3) / 4) {  // the union of every four slices
        float4 lo = s_box[8 * tid], hi = s_box[8 * tid + 1];
        for (uint32_t q = 4 * tid + 1; q < min(4 * tid + 4, nz); ++q) {
            lo = min4(lo, s_box[2 * q]);
            hi = max4(hi, s_box[2 * q + 1]);
        }
        s_quad[2 * tid] = lo;
        s_quad[2 * tid + 1] = hi;
    }
    __syncthreads();
    // The warp's masks; a light that does not reach four slices' union reaches
    // none of them (most warps reach few slices of the near half).
    uint32_t reached = 0;  // bit q: slice q lists a light of the warp
    if (seg * v.seg_lights + warp * 32 < j.light_count)
        for (uint32_t q0 = 0; q0 < nz; q0 += 4) {
            if (!__any_sync(kFull, reaches(L, s_quad[q0 / 2], s_quad[q0 / 2 + 1]))) continue;
            for (uint32_t q = q0; q < min(q0 + 4, nz); ++q) {
                const uint32_t m = __ballot_sync(kFull, reaches(L, s_box[2 * q], s_box[2 * q + 1]));
                if (m) {
                    reached |= 1u << q;
                    if (lane == 0) s_mask[q][warp] = m;
                }
            }
        }
    if (lane < nz && !((reached >> lane) & 1u)) s_mask[lane][warp] = 0u;
    __syncthreads();
    for (uint32_t q = warp; q < nz; q += nw) {
        const uint32_t c = lane < nw ? __popc(s_mask[q][lane]) : 0u;
        const uint32_t incl = warp_inclusive_scan(c, lane);
        s_off[q][lane] = incl - c;
        if (lane == 31) {
            v.seg_count[(size_t)(z0 + q) * v.segs + seg] = incl;
            if (incl) atomicAdd(&v.slice_total[z0 + q].x, incl);
        }
    }
    __syncthreads();
    uint32_t most = 0;  // bit q: slice q lists kCoverMin of the warp's lights or more
    for (; reached; reached &= reached - 1) {
        const uint32_t q = __ffs(reached) - 1, m = s_mask[q][warp];
        if (__popc(m) >= kCoverMin) most |= 1u << q;
        if ((m >> lane) & 1u) {
            const size_t at = (size_t)(z0 + q) * v.lpad + seg * v.seg_lights + s_off[q][warp] +
                              __popc(m & ((1u << lane) - 1u));
            v.slice_lights[at] = L;
            v.slice_idx[at] = i;
        }
    }
    bool any = false;
    for (uint32_t b = most; b; b &= b - 1) {
        const uint32_t q = __ffs(b) - 1;
        any = any || covers(L, s_box[2 * q], s_box[2 * q + 1]);
    }
    if (__syncthreads_or(any)) list_covering(v, L, most, s_box, s_mask, seg, z0, nz);
    if (v.work && tid == 0) atomicAdd(&v.work[0], (unsigned long long)nz * blockDim.x);
}

// Segments of up to 512 lights have CTAs of their own size, four to an SM.
constexpr uint32_t kSmallSegLights = 512, kSmallListCtas = 4;
template <uint32_t kThreads, uint32_t kCtas>
__global__ void __launch_bounds__(kThreads, kCtas) list_kernel(const ViewJob* __restrict__ jobs,
                                                            const uint32_t* __restrict__ prefix, uint32_t n_views,
                                                            const __grid_constant__ ViewJob single)
{
    if (jobs) {
        const uint32_t vi = find_view(prefix, n_views, blockIdx.x);
        list_body(jobs[vi], blockIdx.x - __ldg(&prefix[vi]));
    } else {
        list_body(single, blockIdx.x);
    }
}

// ---------------------------------------------------------------------------
// Scanning.
// ---------------------------------------------------------------------------

// Per-thread asynchronous copies: a thread waits only for its own.
__device__ __forceinline__ void async16(void* dst, const void* src)
{
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src)
                 : "memory");
}
__device__ __forceinline__ void async4(void* dst, const void* src)
{
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src)
                 : "memory");
}
__device__ __forceinline__ void async_wait_all() { asm volatile("cp.async.wait_all;" ::: "memory"); }

constexpr uint32_t kBank = kMaskMaxRun / 32;  // most chunks of 32 candidates per unit

// Shared memory of one warp: the unit's candidates (each lane copies and reads
// only its own), its pending survivors (a ring of 64, one array per component
// so that four lights' x are one 16-byte read), the light indices of its
// survivors and their mask words.
struct ScanWarp {
    float4 in[kBank][32];
    float x[64], y[64], z[64], r2[64], zz[64];
    uint32_t in_idx[kBank][32];
    uint32_t idx[32 * kBank];
    uint32_t word[kBank][32];
};

// One lane's cluster box, each x and y bound in both halves of a packed pair.
struct LaneBox {
    f2 mnx, mny, mxx, mxy;
};

// Mask of the n pending survivors from ring position `at` that reach this
// lane's box, one of a group whose boxes share their z bounds: the ring holds
// each light's squared z distance.  Four lights per step, two per packed
// operation; the ring is padded with never-hit lights to a multiple of four.
__device__ __forceinline__ uint32_t test_pending(const ScanWarp& s, uint32_t at, uint32_t n, const LaneBox& b)
{
    uint32_t word = 0;
#pragma unroll 2
    for (uint32_t j = 0; j < n; j += 4) {
        const uint32_t p = (at + j) & 63u;  // `at` is a multiple of 32
        const float4 x = *reinterpret_cast<const float4*>(&s.x[p]);
        const float4 y = *reinterpret_cast<const float4*>(&s.y[p]);
        const float4 zz = *reinterpret_cast<const float4*>(&s.zz[p]);
        const float4 r2 = *reinterpret_cast<const float4*>(&s.r2[p]);
        bool h0, h1, h2, h3;
        hit_pair_flat(f2_pack(x.x, x.y), f2_pack(y.x, y.y), zz.x, zz.y, r2.x, r2.y, b.mnx, b.mny, b.mxx, b.mxy, h0, h1);
        hit_pair_flat(f2_pack(x.z, x.w), f2_pack(y.z, y.w), zz.z, zz.w, r2.z, r2.w, b.mnx, b.mny, b.mxx, b.mxy, h2, h3);
        word |= ((h0 ? 1u : 0u) | (h1 ? 2u : 0u) | (h2 ? 4u : 0u) | (h3 ? 8u : 0u)) << j;
    }
    return word;
}

// The same for any boxes and lights, with the shader's branchy test if `exact`
// (survivors that include a non-finite coordinate).  Out of line and reading
// the lane's box again: rare, and its registers would be every unit's.
__device__ __noinline__ uint32_t test_pending_general(const ScanWarp& s, uint32_t at, uint32_t n,
                                                      const float4* __restrict__ box, bool exact)
{
    const float4 lo = __ldg(box), hi = __ldg(box + 1);
    const float mn[3] = {lo.x, lo.y, lo.z}, mx[3] = {hi.x, hi.y, hi.z};
    uint32_t word = 0;
    for (uint32_t j = 0; j < n; ++j) {
        const uint32_t p = (at + j) & 63u;
        const float4 L = make_float4(s.x[p], s.y[p], s.z[p], s.r2[p]);
        if (exact ? hit_exact(L, mn, mx) : hit_fast(L, mn, mx)) word |= 1u << j;
    }
    return word;
}

// Writes the hits of 32 lights (`word`: the lane's cluster's mask, idx: the
// lights' indices) in light order at the lane's next place `pos`, up to `lim`,
// four at a time; returns the place after them.  (All lanes walking the lights
// of dense words is no faster: a word's fullest lane has 7 to 11 hits.)
__device__ __forceinline__ uint32_t emit_word(uint32_t word, const uint32_t* idx, uint32_t* __restrict__ out,
                                              uint32_t pos, uint32_t lim)
{
    const uint32_t n = min((uint32_t)__popc(word), lim - min(pos, lim));
    for (uint32_t t = 0; t < n; t += 4) {
        uint32_t x[4];
#pragma unroll
        for (uint32_t e = 0; e < 4; ++e) {
            x[e] = idx[(__ffs(word) - 1) & 31];
            word &= word - 1;
        }
#pragma unroll
        for (uint32_t e = 0; e < 4; ++e)
            if (t + e < n) out[pos + t + e] = x[e];
    }
    return pos + n;
}

// One group as a warp sees it: lane i holds cluster i.
struct GroupLane {
    float4 ulo, uhi;  // the group's union box
    LaneBox box;
    const float4* at;  // the lane's box (the group's first one past the slice)
    bool present;
    bool flat;  // the group's boxes share their z bounds (generated clusters of one slice do)
};

__device__ __forceinline__ GroupLane load_group(const ViewCull& v, uint32_t g, uint32_t k, uint32_t lane)
{
    const uint32_t xy = v.slice_clusters, gps = (xy + kGroup - 1) / kGroup;
    const uint32_t c0 = k * xy + (g - k * gps) * kGroup;
    GroupLane q;
    q.present = c0 + lane < (k + 1) * xy;
    q.at = &v.aabbs[2 * (size_t)(q.present ? c0 + lane : c0)];
    const float4 lo = __ldg(q.at), hi = __ldg(q.at + 1);
    q.ulo = __ldg(&v.group_boxes[2 * (size_t)g]);
    q.uhi = __ldg(&v.group_boxes[2 * (size_t)g + 1]);
    q.box = LaneBox{f2_pack(lo.x, lo.x), f2_pack(lo.y, lo.y), f2_pack(hi.x, hi.x), f2_pack(hi.y, hi.y)};
    q.flat = __all_sync(kFull, lo.z == q.ulo.z && hi.z == q.uhi.z);
    return q;
}

// Starts the copies of candidates [t0, t0 + n) of slice k's list, n <= kMaskMaxRun,
// into s.  The list is one part per segment: lane i of a window of 32 segments
// holds segment i's first position in the list as a whole, and each lane finds
// its candidates' segments by a binary search over the lanes.
__device__ __forceinline__ void fetch_candidates(const ViewCull& v, ScanWarp& s, uint32_t k, uint32_t t0, uint32_t n,
                                                 uint32_t lane)
{
    const uint32_t* __restrict__ counts = v.seg_count + (size_t)k * v.segs;
    const float4* __restrict__ lists = v.slice_lights + (size_t)k * v.lpad;
    const uint32_t* __restrict__ lists_i = v.slice_idx + (size_t)k * v.lpad;
    uint32_t base = 0;  // candidates before the window
    for (uint32_t w0 = 0; w0 < v.segs && base < t0 + n; w0 += 32) {
        const uint32_t c = w0 + lane < v.segs ? __ldg(&counts[w0 + lane]) & kCountMask : 0u;
        const uint32_t incl = warp_inclusive_scan(c, lane);
        const uint32_t first = base + incl - c, end = base + __shfl_sync(kFull, incl, 31);
        if (end > t0) {
#pragma unroll
            for (uint32_t b = 0; b < kBank; ++b) {
                if (b * 32 >= n) break;
                const uint32_t t = t0 + b * 32 + lane;
                uint32_t i = 0;  // the last segment of the window that starts at or before t
#pragma unroll
                for (uint32_t step = 16; step; step >>= 1)
                    if (__shfl_sync(kFull, first, i + step) <= t) i += step;
                const uint32_t start = __shfl_sync(kFull, first, i);
                if (b * 32 + lane < n && t >= base && t < end) {
                    const uint32_t at = (w0 + i) * v.seg_lights + (t - start);
                    async16(&s.in[b][lane], &lists[at]);
                    async4(&s.in_idx[b][lane], &lists_i[at]);
                }
            }
        }
        base = end;
    }
    // the last chunk's absent lanes: lights that reach nothing
    const uint32_t b = n / 32;
    if (lane >= n % 32 && n % 32) s.in[b][lane] = make_float4(0.f, 0.f, 0.f, __uint_as_float(0xff800000u));
}

// A warp's pass over the unit of n candidates in s (see fetch_candidates).
//   kEmit false  counts the lane's hits (no more than lim are needed) and keeps
//                the mask words and indices
//   kEmit true   writes the hits to out from place `count` up to lim
// Returns the number of survivors tested.
template <bool kEmit>
__device__ __forceinline__ uint32_t scan_candidates(ScanWarp& s, uint32_t n, uint32_t lane, const GroupLane& q,
                                                    uint32_t& count, uint32_t lim, uint32_t* __restrict__ out)
{
    const float inf = __uint_as_float(0x7f800000u);
    const float umn[3] = {q.ulo.x, q.ulo.y, q.ulo.z}, umx[3] = {q.uhi.x, q.uhi.y, q.uhi.z};
    const uint32_t lt_mask = (1u << lane) - 1u;
    uint32_t ns = 0, done = 0;
    bool full = __all_sync(kFull, count >= lim);  // every lane has as many hits as its cluster can list
    auto flush = [&](uint32_t m) {
        // pad to a multiple of four with lights that reach nothing
        if ((m & 3u) && lane < 4u - (m & 3u)) {
            const uint32_t p = (done + m + lane) & 63u;
            s.x[p] = s.y[p] = s.z[p] = s.zz[p] = 0.0f;
            s.r2[p] = -inf;
        }
        __syncwarp();
        const uint32_t r = (done + lane) & 63u;
        const bool bad = lane < m && !(finite_bits(s.x[r]) && finite_bits(s.y[r]) && finite_bits(s.z[r]));
        const bool exact = __any_sync(kFull, bad);
        uint32_t word = exact || !q.flat ? test_pending_general(s, done, m, q.at, exact) : test_pending(s, done, m, q.box);
        if (!q.present) word = 0;
        if constexpr (kEmit) {
            count = emit_word(word, &s.idx[done], out, count, lim);
        } else {
            s.word[done / 32][lane] = word;
            count += __popc(word);
        }
        full = __all_sync(kFull, count >= lim);
        __syncwarp();
        done += m;
    };
    async_wait_all();
    for (uint32_t b = 0; b * 32 < n && !full; ++b) {
        const float4 L = s.in[b][lane];
        const bool pass = hit_fast(L, umn, umx);
        const uint32_t m = __ballot_sync(kFull, pass);
        if (!m) continue;
        if (pass) {
            const uint32_t p = ns + __popc(m & lt_mask);
            s.x[p & 63u] = L.x;
            s.y[p & 63u] = L.y;
            s.z[p & 63u] = L.z;
            s.r2[p & 63u] = L.w;
            const float dz = max3f(cf_fsub(q.ulo.z, L.z), cf_fsub(L.z, q.uhi.z), 0.0f);
            s.zz[p & 63u] = cf_fmul(dz, dz);
            s.idx[p] = s.in_idx[b][lane];
        }
        ns += __popc(m);
        if (ns - done >= 32) flush(32);
    }
    if (ns > done && !full) flush(ns - done);
    return done;
}

// unit_run: the unit's first batch in the pool and, from bit kBatchShift, its
// batches less one; or a mark.  A batch is the 32 mask words (one per cluster)
// of 32 survivors and the survivors' indices.
constexpr uint32_t kBatchShift = 28;
constexpr uint32_t kNoHits = 0xffffffffu;  // the unit has no hit
constexpr uint32_t kNoRun = 0xfffffffeu;   // ... has hits, but the pool had no room for them
constexpr uint32_t kBatchWords = 64;
constexpr int kScanWarps = 4;

// A unit: group g of slice k, n candidates from t0 of the slice's list.
struct Unit {
    uint32_t u, k, g, t0, n;
};

// A warp's unit u: the n candidates in s against group g of slice k.
__device__ __forceinline__ void scan_unit(const ViewCull& v, uint32_t u, uint32_t g, uint32_t k, uint32_t n, ScanWarp& s,
                                          uint32_t lane)
{
    const uint32_t cap = v.cap;
    const GroupLane q = load_group(v, g, k, lane);
    uint32_t count = q.present ? 0u : cap;
    const uint32_t survivors = scan_candidates<false>(s, n, lane, q, count, cap, nullptr);
    if (v.work && lane == 0) {
        atomicAdd(&v.work[0], (unsigned long long)((n + 31) & ~31u));
        atomicAdd(&v.work[1], 32ull * survivors);
    }
    const uint32_t mine = q.present ? min(count, cap) : 0u;
    const bool hits = __any_sync(kFull, mine != 0);
    v.unit_count[(size_t)u * kGroup + lane] = (uint8_t)mine;  // at most kMaskMaxRun
    const uint32_t batches = (survivors + 31) / 32;
    uint32_t run = kNoHits;
    if (lane == 0) {
        if (hits) {
            const unsigned long long at = atomicAdd(v.pool_head, (unsigned long long)batches);
            run = at + batches <= v.pool_batches ? (uint32_t)at | (batches - 1) << kBatchShift : kNoRun;
        }
        v.unit_run[u] = run;
    }
    run = __shfl_sync(kFull, run, 0);
    if (hits && run != kNoRun) {
        uint32_t* out = v.pool + (size_t)(run & ((1u << kBatchShift) - 1)) * kBatchWords + lane;
        for (uint32_t b = 0; b < batches; ++b, out += kBatchWords) {
            out[0] = s.word[b][lane];
            out[32] = s.idx[b * 32 + lane];  // past the survivors: never read
        }
    }
    __syncwarp();  // the next unit overwrites the masks
}

// The runs of a view: slice k's total[k] candidates (up to its list's end, see
// list_covering) in runs of kMaskMaxRun, numbered from first[k]; first[slices]
// is their number.  A run and a group of
// its slice are a unit: first[k] * groups per slice + group * runs of the
// slice + run.  Every block of the scan makes the same plan; the first one
// leaves it in the workspace (slice_first, slice_kept) for the later launches.
struct Plan {
    uint32_t first[kMaskMaxSlices + 1];
    uint32_t total[kMaskMaxSlices];
    uint32_t warp_runs[kScanWarps];
};

// The lights that slice k, of at least the cap's covering lights, lists up to its
// end (see list_covering).
__device__ __forceinline__ uint32_t list_end(const ViewCull& v, uint32_t k)
{
    const uint32_t stop = __ldg(&v.slice_stop[k]);
    uint32_t total = 0, covering = 0;
    for (uint32_t q = 0; q < v.segs && covering < v.cap; ++q) {
        if (q == stop >> kStopShift) return total + (stop & ((1u << kStopShift) - 1));
        const uint32_t c = __ldg(&v.seg_count[(size_t)k * v.segs + q]);
        total += c & kCountMask;
        covering += c >> 16;
    }
    return total;
}

__device__ __forceinline__ void make_plan(const ViewCull& v, Plan& p, bool keep)
{
    constexpr uint32_t kThreads = kScanWarps * 32;
    const uint32_t tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    uint32_t base = 0;
    for (uint32_t k0 = 0; k0 < v.slices; k0 += kThreads) {
        const uint32_t k = k0 + tid;
        const uint2 listed = k < v.slices ? __ldg(&v.slice_total[k]) : make_uint2(0u, 0u);
        const uint32_t total = listed.y < v.cap ? listed.x : list_end(v, k);
        const uint32_t n = (total + kMaskMaxRun - 1) / kMaskMaxRun, incl = warp_inclusive_scan(n, lane);
        if (lane == 31) p.warp_runs[warp] = incl;
        __syncthreads();
        uint32_t at = base + incl - n;
#pragma unroll
        for (uint32_t q = 0; q < (uint32_t)kScanWarps; ++q) {
            at += q < warp ? p.warp_runs[q] : 0u;
            base += p.warp_runs[q];
        }
        if (k < v.slices) {
            p.first[k] = at;
            p.total[k] = total;
        }
        __syncthreads();
    }
    if (tid == 0) p.first[v.slices] = base;
    __syncthreads();
    if (keep)
        for (uint32_t k = tid; k <= v.slices; k += kThreads) {
            v.slice_first[k] = p.first[k];
            if (k < v.slices) v.slice_kept[k] = p.total[k];
        }
}

// The slice of run r (of all).
__device__ __forceinline__ uint32_t slice_of(const ViewCull& v, const Plan& p, uint32_t r)
{
    uint32_t k = 0, hi = v.slices;  // first[k] <= r < first[hi]
    while (hi - k > 1) {
        const uint32_t mid = (k + hi) >> 1;
        if (p.first[mid] <= r) k = mid;
        else hi = mid;
    }
    return k;
}

__device__ __forceinline__ Unit unit_of(const ViewCull& v, uint32_t gps, const Plan& p, uint32_t u)
{
    const uint32_t k = slice_of(v, p, u / gps), runs = p.first[k + 1] - p.first[k], at = u - p.first[k] * gps;
    const uint32_t gl = at / runs, t0 = (at - gl * runs) * kMaskMaxRun;
    return Unit{u, k, k * gps + gl, t0, min(kMaskMaxRun, p.total[k] - t0)};
}

// Lane i's unit, in every lane.
__device__ __forceinline__ Unit unit_from(const Unit& a, uint32_t i)
{
    return Unit{__shfl_sync(kFull, a.u, i), __shfl_sync(kFull, a.k, i), __shfl_sync(kFull, a.g, i),
                __shfl_sync(kFull, a.t0, i), __shfl_sync(kFull, a.n, i)};
}

// A block of a view's scan: every warp takes each `step`th item, a run of
// candidates against v.scan_groups neighbouring groups.  Neighbouring items, of
// the same dense groups, so go to different SMs.  The lanes look up 32 items at
// once.
template <bool kBatch>
__device__ __forceinline__ void scan_body(const ViewCull& v, uint32_t blk, uint32_t blocks, ScanWarp* sm, Plan& p)
{
    const uint32_t warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const uint32_t gps = (v.slice_clusters + kGroup - 1) / kGroup;
    const uint32_t per = kBatch ? v.scan_groups : 1u, parts = (gps + per - 1) / per;  // items per run
    make_plan(v, p, blk == 0);
    const uint32_t items = p.first[v.slices] * parts, step = kScanWarps * blocks;
    for (uint32_t w0 = blk + warp * blocks; w0 < items; w0 += 32 * step) {
        // the lane's item: part `part` of the groups, run r of slice k
        const uint32_t w = min(w0 + lane * step, items - 1), k = slice_of(v, p, w / parts);
        const uint32_t runs = p.first[k + 1] - p.first[k], at = w - p.first[k] * parts, part = at / runs, r = at - part * runs;
        for (uint32_t i = 0; i < 32 && w0 + i * step < items; ++i) {
            const uint32_t ik = __shfl_sync(kFull, k, i), ir = __shfl_sync(kFull, r, i);
            const uint32_t g0 = __shfl_sync(kFull, part, i) * per, g1 = min(g0 + per, gps);
            const uint32_t iruns = p.first[ik + 1] - p.first[ik], u0 = p.first[ik] * gps + ir;
            const uint32_t in = min(kMaskMaxRun, p.total[ik] - ir * kMaskMaxRun);
            fetch_candidates(v, sm[warp], ik, ir * kMaskMaxRun, in, lane);
            if constexpr (kBatch) {
                for (uint32_t g = g0; g < g1; ++g)
                    scan_unit(v, u0 + g * iruns, ik * gps + g, ik, in, sm[warp], lane);
            } else {
                scan_unit(v, u0 + g0 * iruns, ik * gps + g0, ik, in, sm[warp], lane);
            }
        }
    }
}

constexpr int kScanCtas = 8;
__global__ void __launch_bounds__(kScanWarps * 32, kScanCtas) scan_kernel(const ViewJob* __restrict__ jobs,
                                                               const uint32_t* __restrict__ prefix, uint32_t n_views,
                                                               const __grid_constant__ ViewJob single)
{
    __shared__ __align__(16) ScanWarp sm[kScanWarps];
    __shared__ Plan plan;
    grid_dependency_wait();
    launch_dependents();
    if (jobs) {
        const uint32_t vi = find_view(prefix, n_views, blockIdx.x), b0 = __ldg(&prefix[vi]);
        scan_body<true>(jobs[vi].v, blockIdx.x - b0, __ldg(&prefix[vi + 1]) - b0, sm, plan);
    } else {
        scan_body<false>(single.v, blockIdx.x, gridDim.x, sm, plan);
    }
}

// ---------------------------------------------------------------------------
// Group totals.
// ---------------------------------------------------------------------------
constexpr uint32_t kSumWarps = 4;
constexpr uint32_t kSumIlp = 8;       // loads in flight per warp
constexpr uint32_t kSumAlone = 16;    // most units that a warp of a batch adds up by itself
constexpr uint32_t kSumPerWarp = 8;   // most groups per warp of a batch

// One warp's part of a group's sums: units [j0, j1) of those whose counts start
// at `counts`.  load() gives the lane's cluster's hits in kSumIlp of them, all
// asked for at once.
struct GroupUnits {
    const uint8_t* __restrict__ counts;
    uint16_t* __restrict__ before;
    uint32_t j0, j1;

    __device__ __forceinline__ void load(uint32_t j, uint32_t x[kSumIlp]) const
    {
#pragma unroll
        for (uint32_t e = 0; e < kSumIlp; ++e) x[e] = j + e < j1 ? __ldg(&counts[(j + e) * kGroup]) : 0u;
    }
    __device__ __forceinline__ uint32_t sum(uint32_t x[kSumIlp]) const
    {
        uint32_t s = 0;
        for (uint32_t j = j0; j < j1; j += kSumIlp) {
            load(j, x);
#pragma unroll
            for (uint32_t e = 0; e < kSumIlp; ++e) s += x[e];
        }
        return s;
    }
    // Writes the hits before each unit, `at` before the first one; returns the
    // hits of all.  `loaded`: x is as the last load left it.
    __device__ __forceinline__ uint32_t write_before(uint32_t x[kSumIlp], uint32_t at, uint32_t cap, bool loaded) const
    {
        for (uint32_t j = j0; j < j1; j += kSumIlp) {
            if (!loaded || j1 - j0 > kSumIlp) load(j, x);  // else still in registers
#pragma unroll
            for (uint32_t e = 0; e < kSumIlp; ++e) {
                if (j + e < j1) before[(j + e) * kGroup] = (uint16_t)min(at, cap);
                at += x[e];
            }
        }
        return at;
    }
};

// A group's units: the first one, and how many.
__device__ __forceinline__ uint2 group_units(const ViewCull& v, uint32_t g, uint32_t gps)
{
    if (!v.segs) return make_uint2(0u, 0u);
    const uint32_t k = g / gps, first = __ldg(&v.slice_first[k]), runs = __ldg(&v.slice_first[k + 1]) - first;
    return make_uint2(first * gps + (g - k * gps) * runs, runs);
}

// Group g by all warps of the CTA.
__device__ __forceinline__ void sum_group(const ViewCull& v, uint32_t g, uint2 units, uint32_t lane, uint32_t warp)
{
    __shared__ uint32_t s_sum[kSumWarps][32];
    const GroupUnits a = {v.unit_count + (size_t)units.x * kGroup + lane, v.unit_before + (size_t)units.x * kGroup + lane,
                          warp * units.y / kSumWarps, (warp + 1) * units.y / kSumWarps};
    uint32_t x[kSumIlp];
    s_sum[warp][lane] = a.sum(x);
    __syncthreads();
    uint32_t at = 0, all = 0;
#pragma unroll
    for (uint32_t w = 0; w < kSumWarps; ++w) {
        at += w < warp ? s_sum[w][lane] : 0u;
        all += s_sum[w][lane];
    }
    if (warp == 0) {
        all = min(all, v.cap);
        v.group_count[(size_t)g * kGroup + lane] = (uint16_t)all;
        const uint32_t total = warp_sum(all);
        if (lane == 0) {
            v.group_total[g] = total;
            if (total) atomicAdd(&v.block_total[g / kGroup], total);
        }
    }
    a.write_before(x, at, v.cap, true);
}

// A block of a batch's groups.  Where most have a unit or two, or none, each warp
// takes eight, whose first units' counts it asks for at once; the block shares
// the groups of many units.  A block for each group was mostly its own start: the
// sum launch of 256 animated views 67 us, 26 with this.
__device__ __forceinline__ void sum_block(const ViewCull& v, uint32_t blk)
{
    __shared__ uint32_t s_large[kSumWarps];
    const uint32_t warp = threadIdx.x >> 5, lane = threadIdx.x & 31, cap = v.cap;
    const uint32_t gps = (v.slice_clusters + kGroup - 1) / kGroup;
    const uint32_t g0 = (blk * kSumWarps + warp) * v.sum_groups;
    const uint32_t n = g0 < v.groups ? min(v.sum_groups, v.groups - g0) : 0u;
    const uint2 mine = lane < n ? group_units(v, g0 + lane, gps) : make_uint2(0u, 0u);  // lane e: of group g0 + e
    const uint32_t large = __ballot_sync(kFull, mine.y > kSumAlone);
    uint32_t first[kSumPerWarp], x[kSumIlp], total = 0;
#pragma unroll
    for (uint32_t e = 0; e < kSumPerWarp; ++e) {
        if (e >= v.sum_groups) break;
        const uint32_t u = __shfl_sync(kFull, mine.x, e), runs = __shfl_sync(kFull, mine.y, e);
        first[e] = runs ? __ldg(&v.unit_count[(size_t)u * kGroup + lane]) : 0u;
    }
#pragma unroll
    for (uint32_t e = 0; e < kSumPerWarp; ++e) {
        if (e >= n) break;
        const uint32_t u = __shfl_sync(kFull, mine.x, e), runs = __shfl_sync(kFull, mine.y, e);
        if (runs > kSumAlone) continue;
        uint32_t all = first[e];
        if (runs > 1) {  // (that none is before the first unit need not be written)
            const GroupUnits a = {v.unit_count + (size_t)u * kGroup + lane, v.unit_before + (size_t)u * kGroup + lane, 1, runs};
            all = a.write_before(x, all, cap, false);
        }
        all = min(all, cap);
        v.group_count[(size_t)(g0 + e) * kGroup + lane] = (uint16_t)all;
        const uint32_t sum = warp_sum(all);
        if (lane == e) total = sum;
    }
    if (lane < n && !((large >> lane) & 1u)) v.group_total[g0 + lane] = total;
    const uint32_t sum = warp_sum(total);
    if (lane == 0) {
        if (sum) atomicAdd(&v.block_total[g0 / kGroup], sum);
        s_large[warp] = large;
    }
    __syncthreads();
    for (uint32_t w = 0; w < kSumWarps; ++w)
        for (uint32_t m = s_large[w]; m; m &= m - 1) {
            const uint32_t g = (blk * kSumWarps + w) * v.sum_groups + __ffs(m) - 1;
            sum_group(v, g, group_units(v, g, gps), lane, warp);
            __syncthreads();  // s_sum is the next group's
        }
}

__global__ void __launch_bounds__(kSumWarps * 32) sum_kernel(const ViewJob* __restrict__ jobs,
                                                          const uint32_t* __restrict__ prefix, uint32_t n_views,
                                                          const __grid_constant__ ViewJob single)
{
    grid_dependency_wait();
    launch_dependents();
    if (jobs) {
        const uint32_t vi = find_view(prefix, n_views, blockIdx.x);
        sum_block(jobs[vi].v, blockIdx.x - __ldg(&prefix[vi]));
    } else {
        const uint32_t gps = (single.v.slice_clusters + kGroup - 1) / kGroup;
        sum_group(single.v, blockIdx.x, group_units(single.v, blockIdx.x, gps), threadIdx.x & 31, threadIdx.x >> 5);
    }
}

// ---------------------------------------------------------------------------
// Writing.
// ---------------------------------------------------------------------------
constexpr int kEmitWarps = kScanWarps;

// The sum of the totals of the groups before g, in every lane: block sums, then
// the groups of g's own block of 32.
__device__ __forceinline__ uint32_t group_base(const ViewCull& v, uint32_t g, uint32_t lane)
{
    uint32_t sum = lane < g % kGroup ? __ldg(&v.group_total[g - g % kGroup + lane]) : 0u;
    for (uint32_t b = lane; b < g / kGroup; b += 32) sum += __ldg(&v.block_total[b]);
    return warp_sum(sum);
}

// Writes the hits of a unit whose masks were not kept by scanning it again.
// (Not inlined: the registers it needs would be every warp's.)
__device__ __noinline__ void emit_unkept(const ViewCull& v, const Unit a, ScanWarp& s, uint32_t lane, uint32_t pos,
                                         uint32_t lim)
{
    fetch_candidates(v, s, a.k, a.t0, a.n, lane);
    scan_candidates<true>(s, a.n, lane, load_group(v, a.g, a.k, lane), pos, lim, v.indices);
    __syncwarp();
}

// Moves the hits of a unit to their places.
__device__ __forceinline__ void emit_unit(const ViewCull& v, const Unit& a, uint32_t run, ScanWarp& s, uint32_t lane)
{
    const uint32_t before = a.t0 ? __ldg(&v.unit_before[(size_t)a.u * kGroup + lane]) : 0u;  // of the first run: none
    const uint32_t all = __ldg(&v.group_count[(size_t)a.g * kGroup + lane]);
    // the masks are asked for with the counts: one round trip
    const bool kept = run != kNoRun;
    const uint32_t batches = kept ? (run >> kBatchShift) + 1 : 0u;
    const uint32_t* __restrict__ in = v.pool + (kept ? (size_t)(run & ((1u << kBatchShift) - 1)) * kBatchWords : 0) + lane;
    uint32_t word[kBank], idx[kBank];
#pragma unroll
    for (uint32_t b = 0; b < kBank; ++b) {
        word[b] = b < batches ? __ldg(&in[b * kBatchWords]) : 0u;
        idx[b] = b < batches ? __ldg(&in[b * kBatchWords + 32]) : 0u;
    }
    const uint32_t first = group_base(v, a.g, lane) + warp_inclusive_scan(all, lane) - all;
    uint32_t pos = first + before;
    if (__all_sync(kFull, before >= all)) return;  // past the cap in every cluster
    if (!kept) {  // the pool had no room
        emit_unkept(v, a, s, lane, pos, first + all);
        return;
    }
#pragma unroll
    for (uint32_t b = 0; b < kBank; ++b) s.idx[b * 32 + lane] = idx[b];
    __syncwarp();
#pragma unroll
    for (uint32_t b = 0; b < kBank; ++b) {
        if (b >= batches) break;
        pos = emit_word(word[b], &s.idx[b * 32], v.indices, pos, first + all);
    }
    __syncwarp();
}

// A block of a view's writing: every warp takes each `step`th unit that has
// hits, and each `step`th run of kCellGroups groups, for their cells: the base
// of a group is a sum over all before it, which eight groups share.
constexpr uint32_t kCellGroups = 8;
__device__ __forceinline__ void emit_body(const ViewCull& v, uint32_t blk, uint32_t blocks, ScanWarp* sm, Plan& p)
{
    const uint32_t warp = threadIdx.x >> 5, lane = threadIdx.x & 31, step = kEmitWarps * blocks;
    const uint32_t gps = (v.slice_clusters + kGroup - 1) / kGroup;
    uint32_t units = 0;
    if (v.segs) {  // without lights there was no scan
        for (uint32_t k = threadIdx.x; k <= v.slices; k += kEmitWarps * 32) {
            p.first[k] = __ldg(&v.slice_first[k]);
            if (k < v.slices) p.total[k] = __ldg(&v.slice_kept[k]);
        }
        __syncthreads();
        units = p.first[v.slices] * gps;
    }
    for (uint32_t u0 = blk + warp * blocks; u0 < units; u0 += 32 * step) {
        const uint32_t u = u0 + lane * step, run = u < units ? __ldg(&v.unit_run[u]) : kNoHits;
        const Unit mine = unit_of(v, gps, p, min(u, units - 1));
        for (uint32_t m = __ballot_sync(kFull, run != kNoHits); m; m &= m - 1) {
            const uint32_t i = __ffs(m) - 1;
            emit_unit(v, unit_from(mine, i), __shfl_sync(kFull, run, i), sm[warp], lane);
        }
    }
    for (uint32_t g0 = (blk + warp * blocks) * kCellGroups; g0 < v.groups; g0 += step * kCellGroups) {
        uint32_t all[kCellGroups];
#pragma unroll
        for (uint32_t e = 0; e < kCellGroups; ++e)
            all[e] = g0 + e < v.groups ? __ldg(&v.group_count[(size_t)(g0 + e) * kGroup + lane]) : 0u;
        uint32_t base = group_base(v, g0, lane), k = g0 / gps, in_slice = g0 - k * gps;
#pragma unroll
        for (uint32_t e = 0; e < kCellGroups; ++e) {
            if (g0 + e >= v.groups) break;
            const uint32_t incl = warp_inclusive_scan(all[e], lane), i = in_slice * kGroup + lane;
            if (i < v.slice_clusters) v.cells[k * v.slice_clusters + i] = CfLightCell{base + incl - all[e], all[e]};
            base += __shfl_sync(kFull, incl, 31);
            if (++in_slice == gps) {
                in_slice = 0;
                ++k;
            }
        }
        if (g0 + kCellGroups >= v.groups && lane == 0 && v.total) *v.total = base;
    }
}

constexpr int kEmitCtas = 8;  // per SM, as in the scan
__global__ void __launch_bounds__(kEmitWarps * 32, kEmitCtas) emit_kernel(const ViewJob* __restrict__ jobs,
                                                               const uint32_t* __restrict__ prefix, uint32_t n_views,
                                                               const __grid_constant__ ViewJob single)
{
    __shared__ __align__(16) ScanWarp sm[kEmitWarps];
    __shared__ Plan plan;
    grid_dependency_wait();
    launch_dependents();
    if (jobs) {
        const uint32_t vi = find_view(prefix, n_views, blockIdx.x), b0 = __ldg(&prefix[vi]);
        emit_body(jobs[vi].v, blockIdx.x - b0, __ldg(&prefix[vi + 1]) - b0, sm, plan);
    } else {
        emit_body(single.v, blockIdx.x, gridDim.x, sm, plan);
    }
}

}  // namespace

MaskLayout mask_layout(uint32_t clusters, uint32_t slice_clusters, uint32_t slices, uint32_t lights, uint32_t cap,
                       uint32_t seg_lights)
{
    auto al = [](size_t x) { return (x + 255) & ~(size_t)255; };
    const uint32_t lpad = pad_lights(lights), groups = group_count(clusters, slice_clusters, slices, kMaskGroup, kModeBinned);
    MaskLayout m{};
    // The status words, then the words of a one-launch pass over the same
    // workspace: small counts left there would pass for its tagged totals.
    size_t off = 256 + al(kOneLaunchMaxCtas * sizeof(unsigned long long));
    auto take = [&](size_t bytes) {
        const size_t at = off;
        off += al(bytes);
        return at;
    };
    m.group_total = take((size_t)groups * sizeof(uint32_t));
    m.group_count = take((size_t)groups * kMaskGroup * sizeof(uint16_t));
    m.block_total = take((size_t)(groups + kMaskGroup - 1) / kMaskGroup * sizeof(uint32_t));
    m.group_boxes = take((size_t)groups * 2 * sizeof(float4));
    m.slice_boxes = take((size_t)slices * 2 * sizeof(float4));
    m.seg_count = take((size_t)slices * mask_segments(lpad, seg_lights) * sizeof(uint32_t));
    const size_t units = (size_t)groups * ((lpad + kMaskMaxRun - 1) / kMaskMaxRun);
    m.pool_head = take(sizeof(unsigned long long));
    m.slice_total = take((size_t)slices * sizeof(uint2));
    m.slice_stop = take((size_t)slices * sizeof(uint32_t));
    m.slice_kept = take((size_t)slices * sizeof(uint32_t));
    m.slice_first = take((size_t)(slices + 1) * sizeof(uint32_t));
    m.unit_run = take(units * sizeof(uint32_t));
    m.unit_count = take(units * kMaskGroup * sizeof(uint8_t));
    m.unit_before = take(units * kMaskGroup * sizeof(uint16_t));
    // Batches of 32 survivors that all units may keep, as many as fit a third
    // of the largest index list; a unit past that is scanned a second time
    // when the lists are written.
    m.pool_batches = lights ? (uint32_t)std::min<uint64_t>(((uint64_t)clusters * cap / 3 + 4096) / kBatchWords, 1u << 27) : 0u;
    m.pool = take((size_t)m.pool_batches * kBatchWords * sizeof(uint32_t));
    m.slice_lights = take((size_t)slices * lpad * sizeof(float4));
    m.slice_idx = take((size_t)slices * lpad * sizeof(uint32_t));
    m.bytes = off;
    return m;
}

// A view alone has a warp for each unit.  In a batch a warp takes a run of
// candidates against four groups: a third of a unit's instructions were the
// look-up and copy of its candidates (256 animated views: 251 us with one
// group, 237 with two, 234 with four, 236 with eight).
constexpr uint32_t kScanGroupsBatch = 4;
// Lights up to which a group of a batch mostly has few units, and a summing warp
// takes eight groups; past it, one (64 views of up to 65536 lights: 113 us with
// eight for all, 106 with this line; 8192 or 32768 make no difference there).
constexpr uint32_t kSumManyLights = 8192;

static uint32_t mask_list_slices(uint32_t segs, uint32_t slices, uint32_t views)
{
    // as few slices per CTA as keep the launch to one wave of two CTAs per SM
    const uint64_t n = ((uint64_t)segs * slices * views + 303) / 304;
    const uint32_t most = (uint32_t)std::min<uint64_t>(std::max<uint64_t>(n, 4), kListSlices);
    const uint32_t blocks = (slices + most - 1) / most;
    return (slices + blocks - 1) / blocks;
}

void mask_bind(ViewCull& v, const MaskLayout& m, unsigned char* ws, uint32_t seg_lights, uint32_t views)
{
    v.group_total = reinterpret_cast<uint32_t*>(ws + m.group_total);
    v.group_count = reinterpret_cast<uint16_t*>(ws + m.group_count);
    v.block_total = reinterpret_cast<uint32_t*>(ws + m.block_total);
    v.group_boxes = reinterpret_cast<float4*>(ws + m.group_boxes);
    v.slice_boxes = reinterpret_cast<float4*>(ws + m.slice_boxes);
    v.seg_count = reinterpret_cast<uint32_t*>(ws + m.seg_count);
    v.pool_head = reinterpret_cast<unsigned long long*>(ws + m.pool_head);
    v.slice_total = reinterpret_cast<uint2*>(ws + m.slice_total);
    v.slice_stop = reinterpret_cast<uint32_t*>(ws + m.slice_stop);
    v.slice_kept = reinterpret_cast<uint32_t*>(ws + m.slice_kept);
    v.slice_first = reinterpret_cast<uint32_t*>(ws + m.slice_first);
    v.unit_run = reinterpret_cast<uint32_t*>(ws + m.unit_run);
    v.unit_count = ws + m.unit_count;
    v.unit_before = reinterpret_cast<uint16_t*>(ws + m.unit_before);
    v.pool = reinterpret_cast<uint32_t*>(ws + m.pool);
    v.pool_batches = m.pool_batches;
    v.slice_lights = reinterpret_cast<float4*>(ws + m.slice_lights);
    v.slice_idx = reinterpret_cast<uint32_t*>(ws + m.slice_idx);
    v.seg_lights = seg_lights;
    v.segs = mask_segments(v.lpad, seg_lights);
    v.scan_groups = views > 1 ? kScanGroupsBatch : 1;
    v.sum_groups = v.lpad <= kSumManyLights ? kSumPerWarp : 1;
    v.list_slices = mask_list_slices(v.segs, v.slices, views);
}

// A view alone: as many CTAs as keep the launch to about a wave.  A batch has
// CTAs enough, and half the threads wait half as long at its barriers: 64
// views of the benchmark's mix 140.9 us with 1024 lights per segment, 137.6
// with 512.
uint32_t mask_seg_lights(uint32_t lights, uint32_t views)
{
    return lights <= 4096 ? 256u : lights <= 8192 || views > 1 ? 512u : 1024u;
}
uint32_t mask_list_blocks(const ViewCull& v) { return v.segs * ((v.slices + v.list_slices - 1) / v.list_slices); }

// Scan CTAs per view.  Each makes the view's plan first, so few are better once
// there are enough for the GPU: a view gets its share of one resident wave
// (8 CTAs on each of 152 SMs), and more only where the units that its lights
// could make (every light a candidate in every slice; with 16384 lights the
// 2560x1600 view has one in 50) would leave a warp with more than this many.
// Measured with 200 / 400 / 800 / 1600: 64 mixed views 142.8 / 140.9 / 152.2 /
// 206.4 us, 256 views of 4096 lights 367.6 / 358.8 / 357.2 / 354.4 us.
constexpr uint64_t kUnitsPerWarp = 400;

uint32_t mask_scan_blocks(const ViewCull& v, uint32_t views)
{
    const uint64_t most = (uint64_t)v.groups * ((v.lpad + kMaskMaxRun - 1) / kMaskMaxRun);
    if (most == 0) return 0;
    const uint64_t wave = 152u * 8u, one_each = (most + kScanWarps - 1) / kScanWarps;
    const uint64_t share = std::max((wave + views - 1) / views, one_each / kUnitsPerWarp);
    return (uint32_t)std::min(std::min(share, one_each), wave);
}
uint32_t mask_emit_blocks(const ViewCull& v, uint32_t views)
{
    const uint32_t per = kCellGroups * kEmitWarps;  // groups whose cells a CTA writes in one step
    return std::max(mask_scan_blocks(v, views), std::min((v.groups + per - 1) / per, 152u * 8u));
}

static auto list_function(uint32_t seg_lights)
{
    return seg_lights <= kSmallSegLights ? list_kernel<kSmallSegLights, kSmallListCtas> : list_kernel<kMaxSegLights, 2>;
}

cudaError_t launch_mask_lists(const ViewJob& j, cudaStream_t stream)
{
    cudaError_t e = launch_kernel(true, box_kernel<kBoxThreads>, dim3(j.v.slices), dim3(kBoxThreads), 0, stream,
                                  static_cast<const ViewJob*>(nullptr), static_cast<const uint32_t*>(nullptr), 0u, j);
    const uint32_t blocks = mask_list_blocks(j.v);
    if (e == cudaSuccess && blocks)
        e = launch_kernel(true, list_function(j.v.seg_lights), dim3(blocks), dim3(j.v.seg_lights), 0, stream,
                          static_cast<const ViewJob*>(nullptr), static_cast<const uint32_t*>(nullptr), 0u, j);
    return e;
}

cudaError_t launch_mask_scan(const ViewJob& j, cudaStream_t stream)
{
    if (j.v.segs == 0) return cudaSuccess;
    return launch_kernel(true, scan_kernel, dim3(mask_scan_blocks(j.v, 1)), dim3(kScanWarps * 32), 0, stream,
                         static_cast<const ViewJob*>(nullptr), static_cast<const uint32_t*>(nullptr), 0u, j);
}

cudaError_t launch_mask_emit(const ViewJob& j, cudaStream_t stream)
{
    const cudaError_t e = launch_kernel(true, sum_kernel, dim3(j.v.groups), dim3(kSumWarps * 32),
                                        0, stream, static_cast<const ViewJob*>(nullptr),
                                        static_cast<const uint32_t*>(nullptr), 0u, j);
    if (e != cudaSuccess) return e;
    return launch_kernel(true, emit_kernel, dim3(mask_emit_blocks(j.v, 1)), dim3(kEmitWarps * 32), 0, stream,
                         static_cast<const ViewJob*>(nullptr), static_cast<const uint32_t*>(nullptr), 0u, j);
}

cudaError_t launch_mask_batch(const MaskBatch& b, cudaStream_t stream)
{
    if (b.n_views == 0) return cudaSuccess;
    const ViewJob none{};
    const uint32_t n = b.n_views, *p = b.prefix;
    cudaError_t e = launch_kernel(false, box_kernel<kBoxThreadsBatch>, dim3(b.blocks[kMaskBox]), dim3(kBoxThreadsBatch), 0,
                                  stream, b.jobs, p, n, none);
    if (e == cudaSuccess && b.blocks[kMaskList])
        e = launch_kernel(false, list_function(b.seg_lights), dim3(b.blocks[kMaskList]), dim3(b.seg_lights), 0, stream, b.jobs,
                          p + kMaskList * (n + 1), n, none);
    if (e == cudaSuccess && b.blocks[kMaskScan])
        e = launch_kernel(false, scan_kernel, dim3(b.blocks[kMaskScan]), dim3(kScanWarps * 32), 0, stream, b.jobs,
                          p + kMaskScan * (n + 1), n, none);
    if (e == cudaSuccess)
        e = launch_kernel(false, sum_kernel, dim3(b.blocks[kMaskSum]), dim3(kSumWarps * 32), 0, stream, b.jobs,
                          p + kMaskSum * (n + 1), n, none);
    if (e == cudaSuccess)
        e = launch_kernel(false, emit_kernel, dim3(b.blocks[kMaskEmit]), dim3(kEmitWarps * 32), 0, stream, b.jobs,
                          p + kMaskEmit * (n + 1), n, none);
    return e;
}

uint32_t mask_batch_blocks(const ViewCull& v, MaskStage stage, uint32_t views)
{
    switch (stage) {
    case kMaskBox: return v.slices;
    case kMaskList: return mask_list_blocks(v);
    case kMaskScan: return mask_scan_blocks(v, views);
    case kMaskSum: return (v.groups + kSumWarps * v.sum_groups - 1) / (kSumWarps * v.sum_groups);
    default: return mask_emit_blocks(v, views);
    }
}

}  // namespace cfk
