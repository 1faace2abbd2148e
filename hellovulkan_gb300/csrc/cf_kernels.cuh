// cf_kernels.cuh — launch interface of the clustered-forward CUDA kernels.
//
// Data layout in device memory for one view (all 256-byte aligned):
//   aabbs     C x CfAABB (32 B)            written by the AABB generator, reused
//                                          while the projection is unchanged
//   vlights   lpad x float4 (16 B)         view-space light (x, y, z, r^2); lpad is
//                                          the light count rounded up to 32 and
//                                          the pad entries are (0, 0, 0, -inf),
//                                          which fail every test
//   nonfinite ceil(lpad / 256) x uint32    1 where a 256-light granule holds a
//                                          light whose view-space position is not
//                                          finite (those granules take the exact
//                                          branchy test)
//   counts    C x uint32                   capped hit count per cluster (plain path)
//   staging   C x cap x uint32             each cluster's hits in ascending order
//   cells     C x CfLightCell              output
//   indices   >= sum(counts) x uint32      output, packed in cluster order
// and, on the binned path, per depth slice a candidate list (slice_*).
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

#include "cf_types.h"

namespace cfk {

constexpr uint32_t kLightPad = 32;       // view-space light arrays are padded to this
constexpr uint32_t kFlagGranule = 256;   // lights per non-finite flag word


// Device error codes (OR-ed into the context's error word).
constexpr uint32_t kErrFullWaitTimeout = 1u << 0;   // a consumer waited too long for a light tile
constexpr uint32_t kErrEmptyWaitTimeout = 1u << 1;  // the producer waited too long for a free stage
constexpr uint32_t kErrLookbackTimeout = 1u << 2;   // a one-launch CTA waited too long for an earlier CTA's total

// Culling modes (CullConfig::binned).
constexpr int kModeBruteForce = 0;  // transform, every light against every cluster, copy
constexpr int kModeBinned = 1;      // transform, slice binning, persistent culling of the candidates, copy
constexpr int kModeOneLaunch = 2;   // everything in one launch (cf_fused.cu), views of up to kOneLaunchMaxLights

inline uint32_t pad_lights(uint32_t n) { return (n + kLightPad - 1) / kLightPad * kLightPad; }
inline uint32_t granules(uint32_t lpad) { return (lpad + kFlagGranule - 1) / kFlagGranule; }
// Start of a slice list's second segment (see ViewCull): half the padded
// lights, rounded up to a multiple of 32.
__host__ __device__ inline uint32_t list_split(uint32_t lpad) { return (lpad / 32 + 1) / 2 * 32; }

struct ViewCull {
    const float4* vlights;
    const uint32_t* nonfinite;
    const float4* aabbs;
    uint32_t* counts;
    uint32_t* staging;
    CfLightCell* cells;
    uint32_t* indices;
    uint32_t* total;  // may be null
    // binned path: per depth slice, a candidate list of lpad entries
    float4* slice_lights;
    uint32_t* slice_idx;
    // A slice's list is two segments, each in ascending light order and
    // padded to a multiple of 32: the candidates among lights [0, S) at the
    // list's start, those among [S, lpad) from entry S (S = list_split(lpad));
    // the list is the first followed by the second.  A single view bins the
    // two with separate CTAs; a batch writes everything to the first.
    uint32_t* slice_count;      // [2k + h]: padded length of segment h of slice k
    uint32_t* slice_nonfinite;  // [2k + h]: 1 when segment h lists a light with a non-finite coordinate
    float4* group_boxes;        // per cluster group, the union of its AABBs (lo, hi; NaN bound: infinite)
    // optional work counters (profiling only, null otherwise): [0] sphere-box
    // tests against slice slabs and warp union boxes, [1] sphere-box tests
    // against cluster boxes
    unsigned long long* work;
    // cluster groups: the clusters one culling CTA owns.  Plain: group b is
    // [b*gw, min((b+1)*gw, C)); binned: group b is slice b / gps, clusters
    // [k*XY + (b % gps)*gw, min(.. + gw, (k+1)*XY)).
    uint32_t* group_sums;     // capped hit count of each group (plain path)
    uint32_t* group_offsets;  // exclusive scan of group_sums (plain path)
    uint32_t* queue;          // single-view binned launch: item counter, zeroed by the binning launch
    // hit-mask path (cf_mask.cu): slice_lights / slice_idx hold, per slice, one
    // part per segment of seg_lights lights, from entry segment * seg_lights
    float4* slice_boxes;             // per slice: the union of its boxes (lo, hi)
    uint32_t* seg_count;             // [slice * segs + segment]: lights listed
    uint2* slice_total;              // per slice: lights listed, lights that cover it (see list_covering)
    uint32_t* slice_stop;            // per slice: where its list may end
    uint32_t* slice_kept;            // per slice: lights listed up to there
    uint32_t* slice_first;           // the scan's plan (see Plan)
    uint32_t* group_total;           // per group: hits
    uint16_t* group_count;           // per group and cluster: hits
    uint32_t* block_total;           // per 32 groups: hits
    uint32_t* unit_run;              // per unit: its batches in the pool, or a mark
    uint8_t* unit_count;             // per unit and cluster: hits (at most kMaskMaxRun)
    uint16_t* unit_before;           // ... and the hits in the group's earlier units, cut at the cap
    uint32_t* pool;                  // the units' masks and light indices, in batches
    unsigned long long* pool_head;   // batches asked for
    uint32_t pool_batches;
    uint32_t seg_lights;
    uint32_t segs;
    uint32_t list_slices;            // slices a list CTA takes
    uint32_t scan_groups;            // groups a scanning warp tests a run of candidates against
    uint32_t sum_groups;             // groups whose units a warp of a batch adds up
    uint32_t lpad;
    uint32_t clusters;
    uint32_t cap;
    uint32_t slice_clusters;  // X * Y
    uint32_t slices;          // Z
    uint32_t group_width;     // gw = warps * clusters per warp (<= 32)
    uint32_t groups;
    uint32_t binned;
};

// One view of a batch: its culling state plus the inputs of the per-view
// stages, and where its blocks start in each batched launch.
struct ViewJob {
    ViewCull v;
    const CfLightData* lights;
    uint32_t light_count;
    uint32_t pad_[3];
    float view[16];  // cameraView, column-major
};

// First cluster and end of group b (see ViewCull).
__host__ __device__ inline void group_range(const ViewCull& v, uint32_t b, uint32_t* first, uint32_t* end)
{
    if (v.binned) {
        const uint32_t gps = (v.slice_clusters + v.group_width - 1) / v.group_width;
        const uint32_t k = b / gps;
        *first = k * v.slice_clusters + (b % gps) * v.group_width;
        const uint32_t e = *first + v.group_width, se = (k + 1) * v.slice_clusters;
        *end = e < se ? e : se;
    } else {
        *first = b * v.group_width;
        const uint32_t e = *first + v.group_width;
        *end = e < v.clusters ? e : v.clusters;
    }
}

inline uint32_t group_count(uint32_t clusters, uint32_t slice_clusters, uint32_t slices, uint32_t gw, int mode)
{
    return mode == kModeBinned ? slices * ((slice_clusters + gw - 1) / gw) : (clusters + gw - 1) / gw;
}

// One culling configuration: clusters per warp, consumer warps per CTA,
// lights per shared-memory stage, number of stages, mode.  A one-launch
// configuration reads them as clusters per CTA, warps per CTA, the most
// lights it takes (32 per warp and chunk), and 1.
struct CullConfig {
    int clusters_per_warp;
    int warps;
    int tile;
    int stages;
    int binned;  // kModeBruteForce, kModeBinned or kModeOneLaunch
};

// Clusters one culling CTA owns (a cluster group).
inline uint32_t group_width(const CullConfig& c)
{
    return c.binned == kModeOneLaunch ? (uint32_t)c.clusters_per_warp : (uint32_t)(c.warps * c.clusters_per_warp);
}

// The hit-mask path (cf_mask.cu) as a configuration of the binned mode: 32
// clusters per group, 32 lights per mask, no staging (1 stage).
constexpr CullConfig kMaskConfig{4, 8, 32, 1, kModeBinned};
constexpr CullConfig kStagedConfig{2, 8, 1024, 2, kModeBinned};  // the staged binned path's own default
// Most groups the automatic choice gives the hit-mask path: a group reads the
// totals of earlier groups as sums of 32, so their number grows with the view.
constexpr uint32_t kMaskMaxGroups = 32768;
constexpr uint32_t kMaskMaxSlices = 256;  // slices whose first units a scanning CTA keeps in shared memory
constexpr uint32_t kMaskMaxRun = 128;      // most candidates per scanning unit
constexpr uint32_t kMaskGroup = 32;      // clusters per group
constexpr uint32_t kMaxSegLights = 1024; // most lights per list segment
inline bool is_mask_config(const CullConfig& c)
{
    return c.clusters_per_warp == kMaskConfig.clusters_per_warp && c.warps == kMaskConfig.warps &&
           c.tile == kMaskConfig.tile && c.stages == kMaskConfig.stages && c.binned == kMaskConfig.binned;
}
inline uint32_t mask_segments(uint32_t lpad, uint32_t seg_lights) { return (lpad + seg_lights - 1) / seg_lights; }

// Scratch of one view on the hit-mask path.
struct MaskLayout {
    size_t slice_first, group_total, group_count, block_total, group_boxes, slice_boxes, seg_count, pool_head, slice_total, slice_stop, slice_kept,
        unit_run, unit_count, unit_before, pool, slice_lights, slice_idx, bytes;
    uint32_t pool_batches;
};
MaskLayout mask_layout(uint32_t clusters, uint32_t slice_clusters, uint32_t slices, uint32_t lights, uint32_t cap,
                       uint32_t seg_lights);
// Points v's hit-mask buffers into a workspace (v.lpad set).
void mask_bind(ViewCull& v, const MaskLayout& m, unsigned char* ws, uint32_t seg_lights, uint32_t views);
// Lights per list segment for a view of `lights` (a batch: the most of its views).
uint32_t mask_seg_lights(uint32_t lights, uint32_t views);

// Workspace carve-up for one view (cf_cull_lights).  A one-launch view needs
// only the status block and one 8-byte word per CTA (`partials`).
struct WorkspaceLayout {
    size_t vlights, nonfinite, counts, staging, group_sums, group_offsets, slice_lights, slice_idx, slice_count,
        slice_nonfinite, group_boxes, partials, bytes;
};
constexpr size_t kQueueWord = 64;   // byte offset, in a workspace's status block, of the single-view item counter
constexpr size_t kEpochWord = 128;  // byte offset of the one-launch kernel's epoch (see FusedCull)
// Scratch of one view; `groups` = group_count(...) of the configuration used.
WorkspaceLayout workspace_layout(uint32_t clusters, uint32_t lights, uint32_t cap, uint32_t slices, int mode,
                                 uint32_t groups);

inline bool mask_fits(uint32_t clusters, uint32_t slice_clusters, uint32_t slices)
{
    return slices <= kMaskMaxSlices && group_count(clusters, slice_clusters, slices, kMaskGroup, kModeBinned) <= kMaskMaxGroups;
}
// Whether the automatic choices may give the hit-mask path a view of that many
// lights.  A unit (128 lights of every group) has 100 bytes of its workspace:
// they may be half a gigabyte, or twice the slice lists, which the staged path
// has too (128x128x64 with 65536 lights would take 1.8 GB where that takes
// 0.3).  And a scanning warp steps over the windows of 32 segments (32768
// lights) before its candidates; units times windows, hit masks against staged:
//   16x9x24,  4 M lights   457 M   1175 against  2088 us
//   40x24x56, 1 M lights   400 M    666 against   880 us
//   8x8x16,  16 M lights  1950 M   6009 against 10674 us (few groups: staged is slow)
//   32x18x48, 4 M lights  3300 M   3419 against  2074 us
//   16x9x24, 16 M lights  7300 M  10575 against  8166 us
// Of less than four slices a list hardly prunes, and its end (see list_covering)
// seldom comes: 61x51x3 with 51841 lights of radius 20 to 60 166 us with hit masks,
// 47 staged; 40x40x2 with 2304 of them 35, 12.5 by brute force; with 4096 lights of
// radius 1 to 5 30 and 35.
constexpr uint32_t kMaskMinSlices = 4;
constexpr uint64_t kMaskUnitBytes = 100, kMaskMaxUnitBytes = 512ull << 20, kMaskMaxWindowSteps = 2000ull << 20;
inline bool mask_pays(uint32_t clusters, uint32_t slice_clusters, uint32_t slices, uint32_t lights)
{
    if (slices < kMaskMinSlices || !mask_fits(clusters, slice_clusters, slices)) return false;
    const uint64_t lpad = pad_lights(lights), groups = group_count(clusters, slice_clusters, slices, kMaskGroup, kModeBinned);
    const uint64_t units = groups * ((lpad + kMaskMaxRun - 1) / kMaskMaxRun), lists = 20ull * slices * lpad;
    const uint64_t windows = (lpad + 32 * kMaxSegLights - 1) / (32 * kMaxSegLights);
    const uint64_t most = 2 * lists > kMaskMaxUnitBytes ? 2 * lists : kMaskMaxUnitBytes;
    return kMaskUnitBytes * units <= most && units * windows <= kMaskMaxWindowSteps;
}

// One-launch culling of a small view (cf_fused.cu): light transform,
// LightCulling.comp's test for every (cluster, light) pair, the capped
// ordered lists, the cluster-order offsets and the packed output, all in one
// cooperative launch.  CTA b owns clusters [b*per_cta, (b+1)*per_cta); its
// warps transform their share of the lights into registers and test them
// against the CTA's clusters; each test's 32 results are one ballot mask.
// The CTA's capped hit total goes to partials[b] as (tag << 32) | total, and
// each CTA sums the totals of the CTAs before it: that is its output offset.
// The tag is *epoch + 1, read at kernel start; the last CTA stores it back
// into *epoch once every CTA has published (so each CTA has read the old
// value), and words from earlier launches never carry the current tag.  The
// workspace must be zero-filled once after allocation.
struct FusedCull {
    const CfLightData* lights;
    const float4* aabbs;
    CfLightCell* cells;
    uint32_t* indices;
    uint32_t* total;                // may be null
    unsigned long long* partials;   // ctas words
    uint32_t* epoch;
    unsigned long long* work;       // optional work counters (see ViewCull)
    float view[16];                 // cameraView, column-major
    uint32_t light_count;
    uint32_t clusters;
    uint32_t cap;
    uint32_t per_cta;               // clusters per CTA, <= kOneLaunchMaxClustersPerCta
    uint32_t ctas;
};
constexpr uint32_t kOneLaunchMaxLights = 2048;
constexpr uint32_t kOneLaunchMaxClustersPerCta = 32;
constexpr uint32_t kOneLaunchMaxCtas = 256;
// The compiled one-launch shapes: (warps per CTA, most lights) = (32, 1024), (16, 2048), (16, 1024).
bool one_launch_shape_supported(int warps, int max_lights);
// CTAs of that shape that can be resident at once on the current device.
cudaError_t one_launch_resident_ctas(int warps, int max_lights, int* ctas);
// The one-launch configuration for a view, if one fits (false otherwise).
bool one_launch_config(uint32_t clusters, uint32_t lights, CullConfig* cfg);
cudaError_t launch_one_launch(const FusedCull& f, int warps, int max_lights, uint32_t* dev_error, cudaStream_t stream);

bool cull_config_supported(const CullConfig& c);
CullConfig default_cull_config(uint32_t clusters, uint32_t lights, uint32_t slices);
CullConfig unmasked_cull_config(uint32_t clusters, uint32_t lights, uint32_t slices);  // ... without the hit masks

// Test knobs of the culling kernels on the current device (cf_device.cuh):
// the bounded-wait limit and the injected stall bits, per translation unit.
cudaError_t set_test_knobs_kernels(uint64_t wait_limit_ns, uint32_t inject);
cudaError_t set_test_knobs_one_launch(uint64_t wait_limit_ns, uint32_t inject);

cudaError_t launch_aabb(const CfClusterForwardUBO& ubo, CfAABB* aabbs, cudaStream_t stream);
cudaError_t launch_light_xform(const CfLightData* lights, uint32_t count, const float view[16], float4* vlights,
                               uint32_t* nonfinite, cudaStream_t stream);
cudaError_t launch_bin(const ViewCull& v, cudaStream_t stream);
cudaError_t launch_cull(const ViewCull& v, const CullConfig& cfg, uint32_t* dev_error, cudaStream_t stream);
cudaError_t launch_finalize(const ViewCull& v, cudaStream_t stream);
// Hit-mask path of one view: union boxes and candidate lists; the tests; the output.
cudaError_t launch_mask_lists(const ViewJob& j, cudaStream_t stream);
cudaError_t launch_mask_scan(const ViewJob& j, cudaStream_t stream);
cudaError_t launch_mask_emit(const ViewJob& j, cudaStream_t stream);
// total, cells and min(total, capacity) indices of one view into device-addressable host memory
cudaError_t launch_readback(const CfLightCell* cells, uint32_t clusters, const uint32_t* indices,
                            const uint32_t* d_total, uint64_t capacity, CfLightCell* h_cells, uint32_t* h_indices,
                            uint32_t* h_total, cudaStream_t stream);
// Jitters of many light sets in as few launches as possible (one per run of
// tasks none of which reads another's output), in task order: each task's
// dst = src with positions moved by sigma * (Irwin-Hall variate) from (seed,
// light, axis).
struct JitterTask {
    const CfLightData* src;
    CfLightData* dst;
    uint64_t seed;
    uint32_t n;
    float sigma;
};
constexpr uint32_t kMaxJitterTasks = 32;  // tasks per launch (passed by value)
cudaError_t launch_jitter_tasks(const JitterTask* tasks, uint32_t n, cudaStream_t stream);
// Copies of many buffers from device-mapped pinned host memory (16-byte
// aligned, whole 16-byte words) in as few launches as possible.
struct UploadTask {
    const uint4* src;  // the host buffer's device-side address
    uint4* dst;
    uint32_t words;    // 16-byte words
};
constexpr uint32_t kMaxUploadTasks = 48;  // tasks per launch (passed by value)
cudaError_t launch_upload_tasks(const UploadTask* tasks, uint32_t n, cudaStream_t stream);
// Every light `frames` steps along its orbit, in place (CfLightOrbit).
cudaError_t launch_orbits(CfLightData* lights, CfLightOrbit* orbits, uint64_t n, uint32_t frames, cudaStream_t stream);

// AABBs of many views in one launch: view v owns blocks [prefix[v], prefix[v+1])
// of 256 clusters each.
struct AabbJob {
    CfClusterForwardUBO ubo;
    CfAABB* out;
    uint64_t _pad;
};
cudaError_t launch_batch_aabb(const AabbJob* jobs, const uint32_t* prefix, uint32_t n_views, uint32_t blocks,
                              cudaStream_t stream);

// Batches: every stage of many views in one launch (the culling stage once per
// shape bucket).  `prefix` arrays hold, per view, the first block of that view
// in the launch; `blocks` is the launch's total.
struct BatchCull {
    const ViewJob* jobs;
    const uint2* items;  // (view, group) in the order the queue hands them out
    uint32_t n_items;
    uint32_t* queue;     // reset to 0 by launch_batch_xform
};
constexpr uint32_t kMaxBatchQueues = 256;  // queues a batch_xform launch resets (<= its block size)
cudaError_t launch_batch_xform(const ViewJob* jobs, const uint32_t* prefix, uint32_t n_views, uint32_t blocks,
                               uint32_t* queues, uint32_t n_queues, cudaStream_t stream);
// order (optional): view index per block range, prefix then follows that order
cudaError_t launch_batch_bin(const ViewJob* jobs, const uint32_t* prefix, const uint32_t* order, uint32_t n_views,
                             uint32_t blocks, cudaStream_t stream);
cudaError_t launch_batch_cull(const BatchCull& b, const CullConfig& cfg, int ctas, uint32_t* dev_error,
                              cudaStream_t stream);
// The hit-mask path of many views: per stage, view v owns blocks
// [prefix[v], prefix[v + 1]) of the launch (n_views + 1 entries per stage).
enum MaskStage { kMaskBox, kMaskList, kMaskScan, kMaskSum, kMaskEmit, kMaskStages };
struct MaskBatch {
    const ViewJob* jobs;
    const uint32_t* prefix;
    uint32_t n_views, seg_lights;
    uint32_t blocks[kMaskStages];
};
uint32_t mask_batch_blocks(const ViewCull& v, MaskStage stage, uint32_t views);
cudaError_t launch_mask_batch(const MaskBatch& b, cudaStream_t stream);
cudaError_t batch_cull_resident_ctas(const CullConfig& cfg, int* ctas);
cudaError_t launch_batch_scan(const ViewJob* jobs, uint32_t n_views, cudaStream_t stream);
cudaError_t launch_batch_copy(const ViewJob* jobs, const uint32_t* prefix, uint32_t n_views, uint32_t blocks,
                              cudaStream_t stream);
uint32_t copy_blocks(uint32_t groups);  // blocks of the copy launch for a view of `groups` cluster groups
uint32_t bin_blocks(uint32_t slices);   // blocks of a batched binning launch for a view of `slices` depth slices

}  // namespace cfk
