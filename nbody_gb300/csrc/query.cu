// Tree::query (source/bhtree.cpp:153-173) on the device: many rays at once, a thread or
// eight lanes a ray, over a tree in the reference's node layout (bh::Node, include/nbody/bhtree.h:13-22)
// -- the context's exported Barnes-Hut tree or any node array the caller passes.
//
// The walk is the reference's stackless pre-order over `children` / `next`. A node whose
// bounds the ray meets (Bounds::ray_intersect, include/nbody/bounds.h:64-133) is visited
// and the walk descends to its children, or moves to `next` at a leaf. At a node the ray
// misses, the reference's loop leaves its index where it is and so never ends; here the
// walk moves to that node's `next`, skipping its subtree, which is the only reading under
// which the walk ends. Wherever the reference's walk ends, the two visit the same nodes in
// the same order.
//
// ray_intersect is restated operation for operation, as rounded intrinsics: the box is
// centre +- size on every axis (the node's `size` is its edge, so this is twice the cell),
// a ray whose origin lies in it meets it, and otherwise the three face pairs are tried in
// order x, y, z with the line parameter t of either sign.
//
// Every walk is bounded: each node of a well-formed tree is entered at most once, so a walk
// that takes more steps than there are nodes, or reaches an index outside the array, stops
// and raises DEV_ERR_BOUNDS.
#include <cfloat>

#include "common.cuh"
#include "context.cuh"

namespace nbg
{
    namespace
    {
        constexpr int kBlock = 128;

        struct Ray
        {
            float o[3], d[3];
        };

        // Bounds::ray_intersect: the origin in the box, or a face pair met (each as
        // Bounds::ray_intersect_coord<i> with length = FLT_MAX: the reference only lowers length
        // on a hit, after which it returns). Without branches, so that the three faces'
        // divisions and tests overlap; a face along the ray divides by 1, since by zero is the
        // division's slow path. Face after face with branches took, at eight lanes a
        // ray, 410 against 360 us for 20,011 picking rays among 250,007 bodies and 7.7 against 5.9 ms
        // for 10,000 that meet 1,540 nodes each; at one, among 2^20 bodies, 7.5 against 4.1 ms for 10^6
        // picking rays, 30 against 11 for 100,000 that meet all, 2.03 against 2.12 for 10^6 along an axis.
        __device__ __forceinline__ bool ray_meets(const Ray& r, const float4 b)
        {
            const float c[3] = { b.x, b.y, b.z };
            const float s = b.w;
            float lo[3], hi[3];
            bool inside = true, meets = false;
#pragma unroll
            for (int i = 0; i < 3; ++i)
            {
                lo[i] = __fsub_rn(c[i], s);
                hi[i] = __fadd_rn(c[i], s);
                inside = inside & !((r.o[i] < lo[i]) | (r.o[i] > hi[i]));
            }
#pragma unroll
            for (int i = 0; i < 3; ++i)
            {
                const int j = (i + 1) % 3, k = (i + 2) % 3;
                const bool down = r.d[i] < -FLT_EPSILON;
                const bool along = down | (r.d[i] > FLT_EPSILON);
                const float t = __fdiv_rn(__fsub_rn(down ? hi[i] : lo[i], r.o[i]), along ? r.d[i] : 1.f);
                const float pj = __fadd_rn(r.o[j], __fmul_rn(r.d[j], t));
                const float pk = __fadd_rn(r.o[k], __fmul_rn(r.d[k], t));
                const bool in = (pj > lo[j]) & (pj < hi[j]) & (pk > lo[k]) & (pk < hi[k]);
                meets = meets | (along & (t < FLT_MAX) & in);
            }
            return inside | meets;
        }

        // One thread a ray.
        __global__ void __launch_bounds__(kBlock) query_kernel(const float4* __restrict__ nodes, const uint32_t count,
                                                               const float* __restrict__ rays, const uint32_t nrays,
                                                               const int stop, uint32_t* __restrict__ hits,
                                                               const uint32_t max_hits, uint32_t* __restrict__ counts,
                                                               unsigned* __restrict__ err)
        {
            const uint32_t q = blockIdx.x * kBlock + threadIdx.x;
            if (q >= nrays)
                return;
            Ray r;
            for (int i = 0; i < 3; ++i)
            {
                r.o[i] = rays[6 * static_cast<size_t>(q) + i];
                r.d[i] = rays[6 * static_cast<size_t>(q) + 3 + i];
            }
            uint32_t* out = hits + static_cast<size_t>(q) * max_hits;
            uint32_t idx = 0, visited = 0, steps = 0;
            do
            {
                if (idx >= count || ++steps > count)
                {
                    atomicOr(err, DEV_ERR_BOUNDS);
                    break;
                }
                const float4 bounds = __ldg(&nodes[3 * static_cast<size_t>(idx)]);
                const float4 com = __ldg(&nodes[3 * static_cast<size_t>(idx) + 1]);
                const uint4 links = __ldg(reinterpret_cast<const uint4*>(nodes) + 3 * static_cast<size_t>(idx) + 2);
                if (ray_meets(r, bounds))
                {
                    if (visited < max_hits)
                        out[visited] = idx;
                    ++visited;
                    if (stop == NBODY_QUERY_FIRST_BODY && links.y == 0 && com.w != 0.f)
                        break;      // the visitor returns false
                    idx = links.y ? links.y : links.x;
                }
                else
                    idx = links.x;
            } while (idx != 0);
            counts[q] = visited;
        }

        // Eight lanes a ray. The eight nodes from the one the walk enters are tested at once, a
        // lane each -- a block of siblings when it descends -- and the walk goes on among them
        // by their links, whatever those are, until it leaves them. A walk is a chain of
        // dependent node loads and tests, so its time is its number of such windows; with one
        // thread a ray it is the number of nodes (20,000 rays, 250,000 bodies: 0.42 against
        // 0.34 ms). Nodes that are tested in vain cost throughput once the rays fill the GPU.
        __global__ void __launch_bounds__(kBlock) query_group_kernel(const float4* __restrict__ nodes, const uint32_t count,
                                                               const float* __restrict__ rays, const uint32_t nrays,
                                                               const int stop, uint32_t* __restrict__ hits,
                                                               const uint32_t max_hits, uint32_t* __restrict__ counts,
                                                               unsigned* __restrict__ err)
        {
            const uint32_t q = static_cast<uint32_t>((static_cast<uint64_t>(blockIdx.x) * kBlock + threadIdx.x) / 8);
            const uint32_t lane = threadIdx.x & 7;
            const unsigned group = 0xffu << (threadIdx.x & 24);
            if (q >= nrays)
                return;         // whole groups of eight lanes
            Ray r;
            for (int i = 0; i < 3; ++i)
            {
                r.o[i] = rays[6 * static_cast<size_t>(q) + i];
                r.d[i] = rays[6 * static_cast<size_t>(q) + 3 + i];
            }
            uint32_t* out = hits + static_cast<size_t>(q) * max_hits;
            uint32_t idx = 0, visited = 0, steps = 0, base = 0;
            // the lane's node: its links, and whether it is met, and a leaf with mass
            uint32_t next = 0, children = 0;
            unsigned met = 0, bodies = 0;       // of all eight
            bool fresh = true;
            do
            {
                if (idx >= count || ++steps > count)
                {
                    if (lane == 0)
                        atomicOr(err, DEV_ERR_BOUNDS);
                    break;
                }
                if (fresh || idx - base >= 8u)
                {
                    base = idx;
                    fresh = false;
                    const size_t at = 3 * static_cast<size_t>(min(base + lane, count - 1));
                    const float4 bounds = __ldg(&nodes[at]);
                    const float mass = __ldg(&nodes[at + 1].w);
                    const uint2 links = __ldg(reinterpret_cast<const uint2*>(&nodes[at + 2]));
                    next = links.x;
                    children = links.y;
                    met = __ballot_sync(group, ray_meets(r, bounds)) >> (threadIdx.x & 24);
                    bodies = __ballot_sync(group, links.y == 0 && mass != 0.f) >> (threadIdx.x & 24);
                }
                const uint32_t w = idx - base;
                const uint32_t nx = __shfl_sync(group, next, static_cast<int>(w), 8);
                const uint32_t ch = __shfl_sync(group, children, static_cast<int>(w), 8);
                if ((met >> w) & 1u)
                {
                    if (lane == 0 && visited < max_hits)
                        out[visited] = idx;
                    ++visited;
                    if (stop == NBODY_QUERY_FIRST_BODY && (bodies >> w) & 1u)
                        break;      // the visitor returns false
                    idx = ch ? ch : nx;
                }
                else
                    idx = nx;
            } while (idx != 0);
            if (lane == 0)
                counts[q] = visited;
        }

        int grow(nbody_cuda* ctx, void** p, size_t* cap, const size_t bytes, const char* what)
        {
            if (bytes <= *cap)
                return NBODY_OK;
            if (const int st = before_allocation(ctx))
                return st;
            cudaFreeAsync(*p, ctx->stream);
            *p = nullptr;
            *cap = 0;
            const cudaError_t e = cudaMallocAsync(p, bytes, ctx->stream);
            if (e != cudaSuccess)
                return ctx_cuda_fail(ctx, e, what);
            *cap = bytes;
            return NBODY_OK;
        }
    }

    int reserve_query_nodes(nbody_cuda* ctx, const size_t bytes)
    {
        return grow(ctx, &ctx->query_nodes, &ctx->query_nodes_cap, bytes, "query tree allocation");
    }

    int tree_query(nbody_cuda* ctx, const void* nodes, size_t count, const float* rays, const size_t nrays,
                   const int stop, uint32_t* hits, const size_t max_hits, uint32_t* counts)
    {
        if (stop != NBODY_QUERY_ALL && stop != NBODY_QUERY_FIRST_BODY)
            return ctx_fail(ctx, NBODY_ERR_INVALID, "unknown query stop rule");
        if (nrays && (!rays || !counts || (max_hits && !hits)))
            return ctx_fail(ctx, NBODY_ERR_INVALID, "null query buffers");
        if (nrays > UINT32_MAX || max_hits > UINT32_MAX || (max_hits && nrays > SIZE_MAX / 4 / max_hits))
            return ctx_fail(ctx, NBODY_ERR_INVALID, "query too large");
        if (!nodes)
            if (const int st = tree_on_device(ctx, &count))
                return st;
        if (count > UINT32_MAX)
            return ctx_fail(ctx, NBODY_ERR_INVALID, "tree too large");
        if (!nrays)
            return NBODY_OK;
        if (!count)
        {
            for (size_t q = 0; q < nrays; ++q)
                counts[q] = 0;
            return NBODY_OK;
        }
        if (nodes)
        {
            // a caller's array is uploaded each call
            ctx->query_nodes_id = 0;
            if (const int st = reserve_query_nodes(ctx, count * 48))
                return st;
            if (const int st = h2d(ctx, ctx->query_nodes, nodes, count * 48))
                return st;
        }
        const size_t ray_bytes = nrays * 24, hit_bytes = nrays * max_hits * 4, count_bytes = nrays * 4;
        const size_t at_hits = (ray_bytes + 255) / 256 * 256, at_counts = at_hits + (hit_bytes + 255) / 256 * 256;
        if (const int st = grow(ctx, &ctx->query_buf, &ctx->query_buf_cap, at_counts + count_bytes, "query buffers"))
            return st;
        unsigned char* buf = static_cast<unsigned char*>(ctx->query_buf);
        if (const int st = h2d(ctx, buf, rays, ray_bytes))
            return st;
        // Eight lanes a ray while every ray's lanes are resident at once (38,912 rays), else one.
        // Calls among 2^20 bodies in ms, eight lanes / one, picking: 1,000 rays 0.28 / 0.41, 20,000 0.46 /
        // 0.58, 38,912 0.68 / 0.64, 100,000 1.25 / 0.83, 10^6 9.2 / 4.1; all nodes met: 1,000 6.4 / 10.6,
        // 10,000 7.0 / 9.4, 20,000 9.8 / 9.3, 100,000 36 / 11.
        int sms = 0, threads = 0;
        cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, ctx->device);
        cudaDeviceGetAttribute(&threads, cudaDevAttrMaxThreadsPerMultiProcessor, ctx->device);
        const size_t lanes = nrays * 8 <= static_cast<size_t>(sms) * static_cast<size_t>(threads) ? 8 : 1;
        const auto kernel = lanes == 8 ? query_group_kernel : query_kernel;
        kernel<<<static_cast<unsigned>((nrays * lanes + kBlock - 1) / kBlock), kBlock, 0, ctx->stream>>>(
            static_cast<const float4*>(ctx->query_nodes), static_cast<uint32_t>(count),
            reinterpret_cast<const float*>(buf), static_cast<uint32_t>(nrays), stop,
            reinterpret_cast<uint32_t*>(buf + at_hits), static_cast<uint32_t>(max_hits),
            reinterpret_cast<uint32_t*>(buf + at_counts), ctx->dev_error);
        ++ctx->launches;
        const cudaError_t e = cudaGetLastError();
        if (e != cudaSuccess)
            return ctx_cuda_fail(ctx, e, "query launch");
        if (max_hits)
            if (const int st = d2h(ctx, hits, buf + at_hits, hit_bytes))
                return st;
        if (const int st = d2h(ctx, counts, buf + at_counts, count_bytes))
            return st;
        return check_device_error(ctx);
    }

    void release_query(nbody_cuda* ctx)
    {
        cudaFree(ctx->query_nodes);
        cudaFree(ctx->query_buf);
        ctx->query_nodes = ctx->query_buf = nullptr;
        ctx->query_nodes_cap = ctx->query_buf_cap = 0;
    }
}

extern "C" int nbody_cuda_tree_query(nbody_cuda* ctx, const void* nodes, const size_t count, const float* rays,
                                     const size_t nrays, const int stop, uint32_t* hits, const size_t max_hits,
                                     uint32_t* counts)
{
    if (!ctx)
        return NBODY_ERR_INVALID;
    return nbg::tree_query(ctx, nodes, count, rays, nrays, stop, hits, max_hits, counts);
}
