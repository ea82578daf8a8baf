// Direct-sum accelerations of small systems (the reference's N^2 mode) in one launch, for sm_103a.
//
// Up to 8192 bodies the direct sum is bound by latency: the launch, and the chain of dependent
// steps a thread runs through. So the work is spread as widely as the GPU is:
//   - a cluster of 8 CTAs shares 32 T targets and splits the sources 64 ways, a contiguous
//     slice per warp; every lane of a warp holds T targets as packed pairs and applies the
//     warp's sources to them, staged 32 at a time in the warp's own shared memory as operand
//     pairs ({x,x,y,y}, {z,z,m,m}) while the next 32 are on their way. No warp waits for
//     another until its slice is summed;
//   - a slice is at most 128 sources, where the larger shapes sum runs of 256 in FP32 (direct.cu):
//     more accurate, but not their bits, so a system of up to 8192 bodies gets other bits when a
//     shape is pinned. The eight warps' sums are folded exactly into (S, C) pairs, and the eight
//     CTAs' pairs are added through distributed shared memory as combine_partials adds a
//     split's chunks. No partial goes through global memory and no second launch sums them.
//
// T = 2 up to 2048 bodies, where the CTAs are too few to fill the SMs otherwise (2000 bodies: 8.4
// against 9.3 us a call, 4096: 15.0 against 14.6); T = 4 beyond.
//
// Before (a chunk of 256 sources per 64-thread CTA, then a sum of the partials) and now. One
// accelerate of 1000 body records among others: 12.7 -> 7.0-7.4 us; a sum that is waited for, 4096
// bodies 34 -> 27, 8192 56 -> 52. Steps one after another: 500 bodies 24.7 -> 4.4, 1000 24.7 -> 5.6,
// 2000 24.7 -> 10.0, 3000 25.8 -> 13.2, 4096 18.3 -> 18.7 (replayed 16.7 -> 14.5), 6000 27.8 -> 28.8
// (27.0 -> 24.8), 8192 37.1 -> 36.9 (37.0 -> 39.1). Chunks of one tile (plan_direct) would step 4096 in 14.4
// and 8192 in 33.0 us, but with runs of 256 for twice the error; folded every 64 sources they keep it
// and take 14 % longer for a sum of 4096 that is waited for, 37 % for one of 4400.
#include <cooperative_groups.h>

#include "common.cuh"
#include "direct.cuh"

namespace nbg
{
    namespace
    {
        constexpr int kWarps = kSmallBlock / 32;
        constexpr int kSlices = kSmallSplit * kWarps;
        static_assert(kSmallDirect <= static_cast<size_t>(kSlices) * 256, "a slice is at most one run of the larger shapes");
    }

    template <int T, int LAW, bool AOS>
    __global__ void __cluster_dims__(1, kSmallSplit, 1) __launch_bounds__(kSmallBlock) direct_small_kernel(
        const float4* __restrict__ src, const float4* __restrict__ vel_radius, float4* __restrict__ acc,
        float* __restrict__ body_out, const int n, const float G, const float eps2)
    {
        after_previous();
        namespace cg = cooperative_groups;
        constexpr int P = T / 2;
        constexpr int REC = AOS ? 3 : 1;
        constexpr int TARGETS = 32 * T;
        __shared__ __align__(16) float4 pairs[kWarps][64];
        __shared__ float sums[kWarps][3][TARGETS];
        __shared__ float fold[2][3][TARGETS];       // S, C per component and target
        const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
        const int base = blockIdx.x * TARGETS;
        const int len = (n + kSlices - 1) / kSlices;
        const int j0 = min(n, (static_cast<int>(blockIdx.y) * kWarps + warp) * len), j1 = min(n, j0 + len);

        // past the slice's end a source that adds exactly zero
        auto fetch = [&](const int j) {
            float4 s = no_source<LAW>();
            if (j < j1)
            {
                s = src[static_cast<size_t>(j) * REC];
                if (AOS)
                    s.w = src[static_cast<size_t>(j) * REC + 1].w;
            }
            return s;
        };
        float4 s = fetch(j0 + lane);

        float2 nx[P], ny[P], nz[P], lim[P], ax[P], ay[P], az[P];
#pragma unroll
        for (int p = 0; p < P; ++p)
        {
            float q[2][4];
#pragma unroll
            for (int h = 0; h < 2; ++h)
            {
                const int i = min(base + (2 * p + h) * 32 + lane, n - 1);
                const float4 x = src[static_cast<size_t>(i) * REC];
                q[h][0] = -x.x;
                q[h][1] = -x.y;
                q[h][2] = -x.z;
                const float r = LAW != NBODY_LAW_CUTOFF ? 0.f : (AOS ? x.w : vel_radius[i].w);
                q[h][3] = LAW == NBODY_LAW_CUTOFF ? r * r : eps2;
            }
            nx[p] = make_float2(q[0][0], q[1][0]);
            ny[p] = make_float2(q[0][1], q[1][1]);
            nz[p] = make_float2(q[0][2], q[1][2]);
            lim[p] = make_float2(q[0][3], q[1][3]);
            ax[p] = ay[p] = az[p] = make_float2(0.f, 0.f);
        }

        for (int j = j0; j < j1; j += 32)
        {
            __syncwarp();
            pairs[warp][2 * lane] = make_float4(s.x, s.x, s.y, s.y);
            pairs[warp][2 * lane + 1] = make_float4(s.z, s.z, s.w, s.w);
            __syncwarp();
            s = fetch(j + 32 + lane);
            const int count = (min(32, j1 - j) + 7) & ~7;
            for (int e = 0; e < count; e += 8)
#pragma unroll
                for (int u = 0; u < 8; ++u)
                {
                    const float4 a = pairs[warp][2 * (e + u)], b = pairs[warp][2 * (e + u) + 1];
                    const float2 sx = make_float2(a.x, a.y), sy = make_float2(a.z, a.w);
                    const float2 sz = make_float2(b.x, b.y), sm = make_float2(b.z, b.w);
#pragma unroll
                    for (int p = 0; p < P; ++p)
                        interact_pair<LAW>(sx, sy, sz, sm, nx[p], ny[p], nz[p], lim[p], ax[p], ay[p], az[p]);
                }
        }
#pragma unroll
        for (int p = 0; p < P; ++p)
#pragma unroll
            for (int h = 0; h < 2; ++h)
            {
                const int t = (2 * p + h) * 32 + lane;
                sums[warp][0][t] = h ? ax[p].y : ax[p].x;
                sums[warp][1][t] = h ? ay[p].y : ay[p].x;
                sums[warp][2][t] = h ? az[p].y : az[p].x;
            }
        __syncthreads();
        // the warps' slices in order, exactly
        for (int k = threadIdx.x; k < 3 * TARGETS; k += kSmallBlock)
        {
            const int c = k / TARGETS, t = k % TARGETS;
            float S = 0.f, C = 0.f;
#pragma unroll
            for (int w = 0; w < kWarps; ++w)
            {
                float sum, err;
                two_sum(S, sums[w][c][t], sum, err);
                S = sum;
                C = __fadd_rn(C, err);
            }
            fold[0][c][t] = S;
            fold[1][c][t] = C;
        }
        cg::cluster_group cluster = cg::this_cluster();
        cluster.sync();
        // each CTA finishes its share of the targets: the CTAs' pairs in order, as a
        // double-float sum (combine_partials)
        constexpr int SHARE = TARGETS / kSmallSplit;
        if (threadIdx.x < 3 * SHARE)
        {
            const int c = threadIdx.x / SHARE, t = static_cast<int>(blockIdx.y) * SHARE + static_cast<int>(threadIdx.x) % SHARE;
            float sv[kSmallSplit], cv[kSmallSplit];
#pragma unroll
            for (int r = 0; r < kSmallSplit; ++r)
            {
                sv[r] = *cluster.map_shared_rank(&fold[0][c][t], r);
                cv[r] = *cluster.map_shared_rank(&fold[1][c][t], r);
            }
            float S = 0.f, E = 0.f;
#pragma unroll
            for (int r = 0; r < kSmallSplit; ++r)
            {
                float sum, err;
                two_sum(S, sv[r], sum, err);
                S = sum;
                E = __fadd_rn(E, __fadd_rn(err, cv[r]));
            }
            const int i = base + t;
            if (i < n)
            {
                const float a = G * __fadd_rn(S, E);
                if (AOS)
                    body_out[static_cast<size_t>(i) * 12 + 8 + c] = a;
                else
                    reinterpret_cast<float*>(acc)[static_cast<size_t>(i) * 4 + c] = a;
            }
        }
        else if (!AOS && threadIdx.x < 4 * SHARE)
        {
            const int i = base + static_cast<int>(blockIdx.y) * SHARE + static_cast<int>(threadIdx.x) - 3 * SHARE;
            if (i < n)
                reinterpret_cast<float*>(acc)[static_cast<size_t>(i) * 4 + 3] = 0.f;
        }
        cluster.sync();     // no CTA leaves while its pairs are being read
    }

    cudaError_t launch_direct_small(const DirectPlan& plan, const float4* src, const float4* vel_radius, float4* acc,
                                    float* body_out, const int n, const float G, const float eps2, cudaStream_t stream,
                                    uint64_t* launches)
    {
        using Fn = void (*)(const float4*, const float4*, float4*, float*, int, float, float);
        static const Fn fns[2][2][2] = {        // [T = 4][softened][aos]
            { { direct_small_kernel<2, NBODY_LAW_CUTOFF, false>, direct_small_kernel<2, NBODY_LAW_CUTOFF, true> },
              { direct_small_kernel<2, NBODY_LAW_SOFTENED, false>, direct_small_kernel<2, NBODY_LAW_SOFTENED, true> } },
            { { direct_small_kernel<4, NBODY_LAW_CUTOFF, false>, direct_small_kernel<4, NBODY_LAW_CUTOFF, true> },
              { direct_small_kernel<4, NBODY_LAW_SOFTENED, false>, direct_small_kernel<4, NBODY_LAW_SOFTENED, true> } },
        };
        const dim3 grid(static_cast<unsigned>(plan.grid_x / kSmallSplit), kSmallSplit);
        ++*launches;
        return launch_after(true, fns[plan.T == 4 ? 1 : 0][plan.law == NBODY_LAW_SOFTENED ? 1 : 0][plan.aos ? 1 : 0], grid,
                            kSmallBlock, 0, stream, src, vel_radius, acc, body_out, n, G, eps2);
    }
}
