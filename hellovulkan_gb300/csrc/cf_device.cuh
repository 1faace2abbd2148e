// cf_device.cuh — device helpers shared by the culling kernels: bounded-wait
// limits, the global timer, programmatic dependent launch, warp scans, and
// the two forms of LightCulling.comp's sphere-box test.
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

namespace cfk {

constexpr unsigned kFull = 0xffffffffu;
constexpr uint64_t kWaitLimitNs = 2000000000ull;  // 2 s per bounded wait
constexpr uint32_t kWaitLimitIters = 1u << 26;

// Test knobs (include/cfcull_testing.h), one copy per translation unit that
// includes this header: the library is built without relocatable device
// code, so each file sets its own with set_test_knobs_*.
//   g_wait_limit_ns  the time limit of every bounded wait (kWaitLimitNs
//                    unless a test shortens it)
//   g_inject_stall   0, or kInject* bits that make one CTA withhold a part
//                    so that the others' bounded waits run out
static __device__ unsigned long long g_wait_limit_ns = kWaitLimitNs;
static __device__ unsigned int g_inject_stall = 0;
constexpr unsigned kInjectOneLaunchSkipPublish = 1u;  // the one-launch kernel's CTA 0 does not publish its total
constexpr unsigned kInjectBruteForceSkipTile = 2u;    // the brute-force kernel's CTA 0 producer never sends tile 0

__device__ __forceinline__ uint64_t global_timer_ns()
{
    uint64_t t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    return t;
}

// Programmatic dependent launch.  The kernels of one view's step are launched
// with programmatic stream serialisation, so each may be scheduled while the
// previous kernel of the stream is still running: it runs only its prologue
// (barrier init, parameters) before grid_dependency_wait(), which returns
// once every earlier kernel of the stream has completed and its writes are
// visible.  launch_dependents() lets the next kernel be scheduled early.
// Both are no-ops in a launch without a programmatic dependency.
__device__ __forceinline__ void grid_dependency_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void launch_dependents() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }

__device__ __forceinline__ float max3f(float a, float b, float c)
{
    float r;
    asm("max.f32 %0, %1, %2, %3;" : "=f"(r) : "f"(a), "f"(b), "f"(c));
    return r;
}

__device__ __forceinline__ bool finite_bits(float x)
{
    return (__float_as_uint(x) & 0x7f800000u) != 0x7f800000u;
}

__device__ __forceinline__ uint32_t warp_sum(uint32_t x) { return __reduce_add_sync(kFull, x); }

__device__ __forceinline__ uint32_t warp_inclusive_scan(uint32_t x, uint32_t lane)
{
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t y = __shfl_up_sync(kFull, x, o);
        if (lane >= (uint32_t)o) x += y;
    }
    return x;
}

// The least and greatest of the lanes' values (a NaN only where all are).
// Volatile: a plain asm may be moved into the branch that uses its result, where
// lanes that it names would be missing.
__device__ __forceinline__ float warp_min(float x)
{
    float r;
    asm volatile("redux.sync.min.f32 %0, %1, 0xffffffff;" : "=f"(r) : "f"(x));
    return r;
}
__device__ __forceinline__ float warp_max(float x)
{
    float r;
    asm volatile("redux.sync.max.f32 %0, %1, 0xffffffff;" : "=f"(r) : "f"(x));
    return r;
}

// Index of the view whose range [prefix[v], prefix[v+1]) holds block b.  Every
// lane takes part: each step narrows the range to a 32nd with one load (a
// binary search's eight dependent loads were a quarter of a short block's time).
__device__ __forceinline__ uint32_t find_view(const uint32_t* __restrict__ prefix, uint32_t n_views, uint32_t b)
{
    const uint32_t lane = threadIdx.x & 31;
    uint32_t lo = 0;
    for (uint32_t n = n_views; n > 1;) {  // prefix[lo] <= b < prefix[lo + n]
        const uint32_t stride = (n + 31) / 32, at = lane * stride;
        const uint32_t j = 31 - __clz(__ballot_sync(kFull, at < n && __ldg(&prefix[lo + at]) <= b));
        lo += j * stride;
        n = min(stride, n - j * stride);
    }
    return lo;
}

// Exact for every finite light coordinate against boxes with min <= max on
// each axis (or NaN bounds), which every generated AABB satisfies:
//   v < min:  max3(min - v, v - max, 0) = min - v
//   v > max:  = v - max, and (v - max)^2 == (max - v)^2 bit for bit
//   inside:   both differences are <= 0, so d = 0 and the axis adds +0,
//             which leaves the reference's partial sum unchanged
// NaN bounds are ignored by max.f32 exactly like the reference's false
// comparisons.  Boxes set to +inf on every bound never hit (the capped and
// out-of-range clusters).
__device__ __forceinline__ bool hit_fast(const float4& L, const float* mn, const float* mx)
{
    const float dx = max3f(__fsub_rn(mn[0], L.x), __fsub_rn(L.x, mx[0]), 0.0f);
    const float dy = max3f(__fsub_rn(mn[1], L.y), __fsub_rn(L.y, mx[1]), 0.0f);
    const float dz = max3f(__fsub_rn(mn[2], L.z), __fsub_rn(L.z, mx[2]), 0.0f);
    const float sq = __fadd_rn(__fadd_rn(__fmul_rn(dx, dx), __fmul_rn(dy, dy)), __fmul_rn(dz, dz));
    return sq < L.w;
}

// SquaredDistancePointAABB + TestSphereAABB (LightCulling.comp:26-57) as
// written, for granules holding a non-finite light coordinate.
__device__ __forceinline__ bool hit_exact(const float4& L, const float* mn, const float* mx)
{
    const float v[3] = {L.x, L.y, L.z};
    float sq = 0.0f;
#pragma unroll
    for (int a = 0; a < 3; ++a) {
        if (v[a] < mn[a]) {
            const float d = __fsub_rn(mn[a], v[a]);
            sq = __fadd_rn(sq, __fmul_rn(d, d));
        } else if (v[a] > mx[a]) {
            const float d = __fsub_rn(mx[a], v[a]);
            sq = __fadd_rn(sq, __fmul_rn(d, d));
        }
    }
    return sq < L.w;
}

// ---- packed float pairs ------------------------------------------------------
// sub/mul/add.rn.f32x2: two IEEE binary32 round-to-nearest operations per
// instruction, each the same bits as the scalar one; but a packed product that
// is only used in a packed sum is contracted with it (see hit_pair_twice_rounded).
typedef unsigned long long f2;  // two floats in one 64-bit register pair: (lo, hi)

__device__ __forceinline__ f2 f2_pack(float lo, float hi)
{
    f2 r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi));
    return r;
}
__device__ __forceinline__ void f2_unpack(f2 v, float& lo, float& hi)
{
    asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(v));
}
__device__ __forceinline__ f2 f2_sub(f2 a, f2 b)
{
    f2 r;
    asm("sub.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ f2 f2_fma(f2 a, f2 b, f2 c)
{
    f2 r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
    return r;
}
__device__ __forceinline__ f2 f2_mul(f2 a, f2 b)
{
    f2 r;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}

// hit_fast for two lights against one box, light A in the low halves and light
// B in the high halves, the box bounds in both: the differences and squares packed,
// the sums scalar.  The compiler merges a packed product and a packed sum into
// one packed FMA, rounding once where the shader rounds twice (a light one ulp
// from a box's reach then changes sides), also under -fmad=false and however
// the two are written; a scalar __fadd_rn it leaves alone.
__device__ __forceinline__ void hit_pair_twice_rounded(f2 lx, f2 ly, f2 lz, float ar2, float br2, f2 mnx, f2 mny, f2 mnz,
                                                       f2 mxx, f2 mxy, f2 mxz, bool& ha, bool& hb)
{
    float a0, a1, b0, b1, xa, xb, ya, yb, za, zb;
    f2_unpack(f2_sub(mnx, lx), a0, a1);
    f2_unpack(f2_sub(lx, mxx), b0, b1);
    const f2 dx = f2_pack(max3f(a0, b0, 0.0f), max3f(a1, b1, 0.0f));
    f2_unpack(f2_sub(mny, ly), a0, a1);
    f2_unpack(f2_sub(ly, mxy), b0, b1);
    const f2 dy = f2_pack(max3f(a0, b0, 0.0f), max3f(a1, b1, 0.0f));
    f2_unpack(f2_sub(mnz, lz), a0, a1);
    f2_unpack(f2_sub(lz, mxz), b0, b1);
    const f2 dz = f2_pack(max3f(a0, b0, 0.0f), max3f(a1, b1, 0.0f));
    f2_unpack(f2_mul(dx, dx), xa, xb);
    f2_unpack(f2_mul(dy, dy), ya, yb);
    f2_unpack(f2_mul(dz, dz), za, zb);
    ha = __fadd_rn(__fadd_rn(xa, ya), za) < ar2;
    hb = __fadd_rn(__fadd_rn(xb, yb), zb) < br2;
}

// The same with the lights' squared z distances given.
__device__ __forceinline__ void hit_pair_flat(f2 lx, f2 ly, float za, float zb, float ar2, float br2, f2 mnx, f2 mny, f2 mxx,
                                              f2 mxy, bool& ha, bool& hb)
{
    float a0, a1, b0, b1, xa, xb, ya, yb;
    f2_unpack(f2_sub(mnx, lx), a0, a1);
    f2_unpack(f2_sub(lx, mxx), b0, b1);
    const f2 dx = f2_pack(max3f(a0, b0, 0.0f), max3f(a1, b1, 0.0f));
    f2_unpack(f2_sub(mny, ly), a0, a1);
    f2_unpack(f2_sub(ly, mxy), b0, b1);
    const f2 dy = f2_pack(max3f(a0, b0, 0.0f), max3f(a1, b1, 0.0f));
    f2_unpack(f2_mul(dx, dx), xa, xb);
    f2_unpack(f2_mul(dy, dy), ya, yb);
    ha = __fadd_rn(__fadd_rn(xa, ya), za) < ar2;
    hb = __fadd_rn(__fadd_rn(xb, yb), zb) < br2;
}

}  // namespace cfk
