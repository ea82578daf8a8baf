// Internal interface of the direct-sum kernels (direct.cu, direct_precise.cu).
#pragma once

#include <algorithm>
#include <cmath>
#include <cstddef>
#include <cstdint>
#include <cuda_runtime.h>

#include "common.cuh"

namespace nbg
{
    // One source (sx, sy, sz, sm) applied to two targets held as negated positions; lim is
    // their cutoff radius^2, or eps2.
    template <int LAW>
    __device__ __forceinline__ void interact_pair(const float2 sx, const float2 sy, const float2 sz, const float2 sm,
                                                  const float2 nx, const float2 ny, const float2 nz, const float2 lim,
                                                  float2& ax, float2& ay, float2& az)
    {
        const float2 dx = add2(sx, nx);
        const float2 dy = add2(sy, ny);
        const float2 dz = add2(sz, nz);
        float2 r2 = (LAW == NBODY_LAW_SOFTENED) ? fma2(dx, dx, lim) : mul2(dx, dx);
        r2 = fma2(dy, dy, r2);
        r2 = fma2(dz, dz, r2);
        float2 inv = make_float2(rsqrt_sfu(r2.x), rsqrt_sfu(r2.y));
        if (LAW == NBODY_LAW_CUTOFF)
        {
            // physics.h:38-39: nothing when |d|^2 <= radius^2 (lim holds radius^2)
            inv.x = r2.x > lim.x ? inv.x : 0.f;
            inv.y = r2.y > lim.y ? inv.y : 0.f;
        }
        const float2 inv2 = mul2(inv, inv);
        const float2 mi = mul2(sm, inv);
        const float2 s = mul2(mi, inv2);
        ax = fma2(dx, s, ax);
        ay = fma2(dy, s, ay);
        az = fma2(dz, s, az);
    }

    // Systems small enough for direct_small.cu, and for two targets a lane there (see the kernel).
    constexpr size_t kSmallDirect = 8192, kSmallPair = 2048;
    constexpr int kSmallBlock = 256;
    constexpr int kSmallSplit = 8;      // CTAs a cluster: they share targets and split the sources

    // Launch shape of one direct-sum accelerate.
    struct DirectPlan
    {
        int variant;    // index into the instantiated (targets/thread, block) table; -1 when small
        bool small;     // direct_small.cu's kernel: no scratch, one launch
        int T;          // targets per thread
        int block;      // threads per CTA
        int tile;       // sources per shared-memory tile
        int jsplit;     // source chunks (grid.y); >1 means partials + a fixed-order sum
        int chunk;      // sources per chunk (a multiple of tile * fold)
        int fold;       // tiles per exact fold of the running sums (a function of n only)
        int grid_x;     // target blocks
        int law;
        bool aos;
    };

    // Bytes of j-split scratch one accelerate needs: per chunk and body, the chunk's FP32 sum
    // S and its compensation C (two float4). None without a split.
    inline size_t direct_scratch_bytes(const DirectPlan& plan, const size_t n)
    {
        return plan.jsplit > 1 ? 2 * static_cast<size_t>(plan.jsplit) * n * 16 : 0;
    }

    // The accelerations from the chunk partials of the FP32 direct sum: chunk c of body i
    // holds its (S, C) at S[2 c n + i] and C[2 c n + i] (C = S + n in the scratch layout).
    // The pairs are added over the chunks in chunk order as a double-float sum (TwoSum into
    // a running (s, e), the compensations added to e), then s + e is rounded to FP32 and
    // scaled by G: the same formula for one chunk or many, so the result does not depend on
    // how the sources were split. FP32 only: GB300's FP64 pipe runs at 1/64 of the FP32
    // rate, and a small system's few bodies would put that work on a few SMs.
    // W lanes per body (consecutive lanes of one warp, g = lane % W): lane g sums chunks g,
    // g + W, ... as above, and the lanes' double-float sums are then merged pairwise in a
    // fixed order (the same TwoSum step). Every lane of the warp must call it; the result is
    // lane g = 0's. W = 1 is the plain sequential sum.
    template <int W>
    __device__ __forceinline__ float3 combine_partials_w(const float4* __restrict__ S, const float4* __restrict__ C,
                                                         const int js, const int n, const int i, const int g,
                                                         const float G)
    {
        float sx = 0.f, sy = 0.f, sz = 0.f, ex = 0.f, ey = 0.f, ez = 0.f;
#pragma unroll 4
        for (int c = g; c < js; c += W)
        {
            const size_t k = 2 * static_cast<size_t>(c) * n + i;
            const float4 s = S[k], e = C[k];
            float t, r;
            two_sum(sx, s.x, t, r);
            sx = t;
            ex = __fadd_rn(ex, __fadd_rn(r, e.x));
            two_sum(sy, s.y, t, r);
            sy = t;
            ey = __fadd_rn(ey, __fadd_rn(r, e.y));
            two_sum(sz, s.z, t, r);
            sz = t;
            ez = __fadd_rn(ez, __fadd_rn(r, e.z));
        }
#pragma unroll
        for (int off = W / 2; off > 0; off >>= 1)
        {
            const float osx = __shfl_down_sync(0xffffffffu, sx, off, W), oex = __shfl_down_sync(0xffffffffu, ex, off, W);
            const float osy = __shfl_down_sync(0xffffffffu, sy, off, W), oey = __shfl_down_sync(0xffffffffu, ey, off, W);
            const float osz = __shfl_down_sync(0xffffffffu, sz, off, W), oez = __shfl_down_sync(0xffffffffu, ez, off, W);
            float t, r;
            two_sum(sx, osx, t, r);
            sx = t;
            ex = __fadd_rn(ex, __fadd_rn(r, oex));
            two_sum(sy, osy, t, r);
            sy = t;
            ey = __fadd_rn(ey, __fadd_rn(r, oey));
            two_sum(sz, osz, t, r);
            sz = t;
            ez = __fadd_rn(ez, __fadd_rn(r, oez));
        }
        return make_float3(G * __fadd_rn(sx, ex), G * __fadd_rn(sy, ey), G * __fadd_rn(sz, ez));
    }

    __device__ __forceinline__ float3 combine_partials(const float4* __restrict__ S, const float4* __restrict__ C,
                                                       const int js, const int n, const int i, const float G)
    {
        return combine_partials_w<1>(S, C, js, n, i, 0, G);
    }

    // Lanes per body for the combine: a small system has many chunks and few bodies, so eight
    // lanes a body spread the combine over eight times the SMs. A function of (n, js) only,
    // so the sums do not depend on which kernel combines them.
    inline int combine_width(const int n, const int js) { return (js >= 8 && n <= (1 << 16)) ? 8 : 1; }

    // The split of n sources (units of `unit`, a chunk at least one) over CTAs of `per` targets, tb
    // target blocks: the pairs the fullest of the SMs computes one after another. CTAs end
    // together and are not dealt evenly, which leaves an SM the last of ceil(CTAs / SMs) and on
    // average one and a half more; a CTA's start costs about as much as 8,000 pairs, and the
    // partials n / 16 pairs a chunk. Fitted to 1,500 timings of the FP32 sum (8,193 to 200,000
    // bodies, both laws and layouts, every split): its choice takes 0.7 % longer than the best
    // split, 3 % at worst.
    struct SourceSplit
    {
        size_t tb, per, units, unit, n;
        double sms;

        size_t chunk_units(const size_t js) const { return (units + js - 1) / js; }

        double cost(const size_t js) const
        {
            const size_t c = chunk_units(js);
            const double ctas = static_cast<double>(tb * ((units + c - 1) / c)) / sms;
            return (std::ceil(ctas) + 1.5) * static_cast<double>(c * unit * per) + 8000.0 * ctas
                   + 0.06 * static_cast<double>(n * js);
        }

        double least(const size_t max_js) const
        {
            double v = cost(1);
            for (size_t js = 2; js <= max_js; ++js)
                v = std::min(v, cost(js));
            return v;
        }

        // sources a chunk: the fewest chunks within `slack` of the least cost, for the sake of the scratch
        size_t chunk(const size_t max_js, const double slack) const
        {
            const double bar = slack * least(max_js);
            size_t js = 1;
            while (js < max_js && cost(js) > bar)
                ++js;
            return chunk_units(js) * unit;
        }
    };

    // Pick a launch shape for n bodies. force_variant >= 0 pins the (T, block) entry; the
    // chunk partials stay within split_bytes.
    constexpr size_t kSplitBytes = size_t(256) << 20;
    DirectPlan plan_direct(size_t n, int law, bool aos, int force_variant = -1, size_t split_bytes = kSplitBytes);

    // The instantiated kernel shapes: targets per thread, threads per CTA, packed FP32x2 or not.
    int direct_variant_count();
    void direct_variant_describe(int i, int* T, int* block, int* packed);

    // Queue the accelerate. src is pos_mass (SoA) or the Body array viewed as float4
    // (AoS). Results: acc (SoA) or Body::acc in body_out (AoS). scratch must hold
    // direct_scratch_bytes(plan, n); with reduce == false the partials are left there for
    // the fused integrate to sum.
    cudaError_t launch_direct(const DirectPlan& plan, const float4* src, const float4* vel_radius,
                              float4* acc, float* body_out, float4* scratch, int n, float G,
                              float eps2, unsigned* err, cudaStream_t stream, uint64_t* launches,
                              bool reduce = true);

    // The same for a plan with small set (direct_small.cu).
    cudaError_t launch_direct_small(const DirectPlan& plan, const float4* src, const float4* vel_radius, float4* acc,
                                    float* body_out, int n, float G, float eps2, cudaStream_t stream,
                                    uint64_t* launches);

    cudaError_t launch_reduce(const float4* scratch, int jsplit, int n, float G, float4* acc,
                              float* body_out, cudaStream_t stream, uint64_t* launches);

    // Semi-implicit Euler (integrate.cu). When part != nullptr the accelerations are
    // combine_partials over its jsplit chunks (with G), also written to acc / Body::acc.
    cudaError_t launch_integrate_soa(float4* pos_mass, float4* vel_radius, float4* acc,
                                     const float4* part, int jsplit, int n, float G, float dt,
                                     float size, int wrap, cudaStream_t stream, uint64_t* launches);
    cudaError_t launch_integrate_aos(float* bodies, const float4* part, int jsplit, int n,
                                     float G, float dt, float size, int wrap, cudaStream_t stream,
                                     uint64_t* launches);

    // Body (48 B) <-> split streams (integrate.cu).
    cudaError_t launch_split(const float* bodies, float4* pos_mass, float4* vel_radius,
                             float4* acc, int n, cudaStream_t stream, uint64_t* launches);
    cudaError_t launch_join(const float4* pos_mass, const float4* vel_radius, const float4* acc,
                            float* bodies, int n, cudaStream_t stream, uint64_t* launches);
}
