// The last device tree in the reference's own node layout, for Solver::tree() / Sim::nodes()
// (include/nbody/bhtree.h:13-22): 48-byte nodes {bounds centre, size, com, mass, next,
// children, pad, pad}; a split node owns 8 contiguous children, child q at children + q
// where q is the reference octant (bit set when the coordinate is below the centre,
// bounds.h:31-38); child q's `next` is the next sibling and child 7's is the parent's
// `next`, so the stackless walk of bhtree.cpp:97-138 runs over it unchanged.
//
// The device tree keeps only the cells the traversal needs. Expanding it back:
//   - a cell whose bodies all sit in one octant of the cell above is, in the reference, a
//     chain of single-child cells with the same mass and centre of mass: emitted as such;
//   - octants holding nothing become the reference's empty leaves (mass 0);
//   - a single body becomes a leaf carrying its position and mass;
//   - bodies sharing one finest (level-21) Morton cell, which the reference would keep
//     subdividing down to FLT_EPSILON-sized cells (bhtree.cpp:36-42), become one leaf with
//     their total mass and centre of mass.
// Node order is depth-first (the reference's is insertion order); the links, cells, masses
// and centres of mass describe the same tree.
//
// Where a node goes. A node's block of children is appended when the depth-first walk reaches
// the node, so block r (nodes 1 + 8 r ...) belongs to the r-th split node in the walk's order,
// which takes octants in descending Morton order. A split node is a pair (x, l): the level-l
// cell whose last sorted body is x. It precedes exactly the split nodes that end earlier, and
// those of its own end on deeper levels. Split nodes ending at x exist on the levels above
// the common one of bodies x and x + 1 up to the common one of x - 1 and x (level 20 at most):
// a count per body, whose sum over the bodies after x gives every r without a walk. Each kept
// cell then writes the blocks of its own chain, eight lanes a block.
//
// The expansion ran on the host before, from a copy of the tree: a build, an export and a query
// of 20,000 rays over 250,000 bodies took 23.6 ms, 1.6 ms with it here.
#include <algorithm>
#include <cstring>

#include "bh.cuh"
#include "common.cuh"
#include "context.cuh"
#include "scan.cuh"

namespace nbg
{
    namespace
    {
        struct RefNode
        {
            float cx, cy, cz, size;
            float comx, comy, comz, mass;
            uint32_t next, children, pad0, pad1;
        };
        static_assert(sizeof(RefNode) == 48, "reference node layout");

        constexpr int kLevels = 21;

        __device__ __forceinline__ uint64_t compact1by2(uint64_t v)
        {
            v &= 0x1249249249249249ull;
            v = (v ^ (v >> 2)) & 0x10c30c30c30c30c3ull;
            v = (v ^ (v >> 4)) & 0x100f00f00f00f00full;
            v = (v ^ (v >> 8)) & 0x001f0000ff0000ffull;
            v = (v ^ (v >> 16)) & 0x001f00000000ffffull;
            v = (v ^ (v >> 32)) & 0x1fffffull;
            return v;
        }

        // the deepest octree level whose cell holds both codes
        __device__ __forceinline__ int common_level(const uint64_t a, const uint64_t b)
        {
            return a == b ? kLevels : min(kLevels, (__clzll(static_cast<long long>(a ^ b)) - 1) / 3);
        }

        __device__ __forceinline__ int digit(const uint64_t code, const int level)     // octant at `level` (1 .. 21)
        {
            return static_cast<int>((code >> (3 * (kLevels - level))) & 7u);
        }

        // the level above which split nodes end at x
        __device__ __forceinline__ int level_after(const uint64_t* __restrict__ codes, const int n, const int x)
        {
            return x == n - 1 ? -1 : common_level(codes[x], codes[x + 1]);
        }

        // split nodes that end at body x = n - 1 - k
        __global__ void __launch_bounds__(256) split_count_kernel(const uint64_t* __restrict__ codes, const int n,
                                                                  uint32_t* __restrict__ count)
        {
            const int k = blockIdx.x * 256 + threadIdx.x;
            if (k >= n)
                return;
            const int x = n - 1 - k;
            const int deep = x ? min(kLevels - 1, common_level(codes[x - 1], codes[x])) : -1;
            count[k] = static_cast<uint32_t>(max(0, deep - level_after(codes, n, x)));
        }

        __global__ void __launch_bounds__(256) parent_kernel(const OctNode* __restrict__ nodes, const int cells,
                                                             int* __restrict__ parent)
        {
            const int c = blockIdx.x * 256 + threadIdx.x;
            if (c >= cells)
                return;
            if (c == 0)
                parent[0] = -1;
            const int nchild = nodes[c].nchild;
            for (int k = 0; k < nchild; ++k)
            {
                const int ch = nodes[c].child[k];
                if (ch >= 0)
                    parent[ch] = c;
            }
        }

        // A kept cell as a chain of split nodes: levels above + 1 .. level, or 20 for a bucket
        // (which is a leaf at level 21), all ending at body last.
        struct Chain
        {
            uint64_t code;      // of its first body
            int level, above;   // its own, and its parent cell's
            int parent;
            uint32_t rank0;     // rank of a split node of level l: rank0 + l
        };

        __device__ __forceinline__ Chain chain_of(const TreeView& t, const int* __restrict__ parent,
                                                  const uint32_t* __restrict__ after, const int c)
        {
            Chain h;
            const int first = t.nodes[c].first, last = t.nodes[c].last;
            h.code = t.codes[first];
            h.level = common_level(h.code, t.codes[last]);
            h.parent = parent[c];
            h.above = h.parent < 0 ? -1
                                   : common_level(t.codes[t.nodes[h.parent].first], t.codes[t.nodes[h.parent].last]);
            h.rank0 = after[t.n - 1 - last] - static_cast<uint32_t>(level_after(t.codes, t.n, last) + 1);
            return h;
        }

        __device__ __forceinline__ void put(RefNode* __restrict__ out, const size_t at, const BoxParams& box, const int level,
                                            const uint64_t prefix, const float4 com, const uint32_t next,
                                            const uint32_t children)
        {
            const double cell = box.edge / static_cast<double>(1ull << level);
            // each product is exact (22 bits by at most 24), so contraction changes nothing
            const float cx = static_cast<float>(box.lo[0] + (static_cast<double>(compact1by2(prefix)) + 0.5) * cell);
            const float cy = static_cast<float>(box.lo[1] + (static_cast<double>(compact1by2(prefix >> 1)) + 0.5) * cell);
            const float cz = static_cast<float>(box.lo[2] + (static_cast<double>(compact1by2(prefix >> 2)) + 0.5) * cell);
            float4* o = reinterpret_cast<float4*>(out + at);
            o[0] = make_float4(cx, cy, cz, static_cast<float>(cell));
            o[1] = com;
            o[2] = make_float4(__uint_as_float(next), __uint_as_float(children), 0.f, 0.f);
        }

        // Eight lanes a kept cell: lane q writes child q of each of its split nodes.
        __global__ void __launch_bounds__(256) expand_kernel(const TreeView t, const int cells,
                                                             const int* __restrict__ parent,
                                                             const uint32_t* __restrict__ after, const size_t count,
                                                             RefNode* __restrict__ out, unsigned* __restrict__ err)
        {
            const int c = static_cast<int>((blockIdx.x * 256u + threadIdx.x) / 8);
            const int q = threadIdx.x & 7, d = 7 - q;
            const unsigned group = 0xffu << (threadIdx.x & 24);
            if (c >= cells)
                return;         // whole groups of eight lanes
            const BoxParams& box = *t.box;
            const Chain h = chain_of(t, parent, after, c);
            const int nchild = t.nodes[c].nchild;
            const float4 com = t.nodes[c].com_mass;
            if (c == 0 && q == 0)
                put(out, 0, box, 0, 0, com, 0, 1);
            // where the walk goes after the chain's first split node: past every ancestor that
            // is its parent's last octant
            uint32_t next = 0;
            {
                Chain a = h;
                for (int l = h.above + 1; l > 0; --l)
                {
                    const int o = 7 - digit(h.code, l);
                    if (l - 1 <= a.above)
                        a = chain_of(t, parent, after, a.parent);
                    if (o < 7)
                    {
                        next = 1 + 8 * (a.rank0 + static_cast<uint32_t>(l - 1)) + static_cast<uint32_t>(o) + 1;
                        break;
                    }
                }
            }
            for (int l = h.above + 1; l <= min(h.level, kLevels - 1); ++l)
            {
                const uint32_t block = 1 + 8 * (h.rank0 + static_cast<uint32_t>(l));
                const uint64_t prefix = ((h.code >> (3 * (kLevels - l))) << 3) | static_cast<unsigned>(d);
                float4 content = make_float4(0.f, 0.f, 0.f, 0.f);       // an empty octant: a massless leaf
                uint32_t children = 0;
                if (l < h.level)
                {
                    // every body in one octant
                    if (d == digit(h.code, l + 1))
                    {
                        content = com;
                        children = l + 1 < kLevels ? block + 8 : 0;
                    }
                }
                else
                {
                    const int ch = q < nchild ? t.nodes[c].child[q] : 0;
                    const int first = ch < 0 ? ~ch : t.nodes[ch].first;
                    const int own = q < nchild ? digit(t.codes[first], l + 1) : -1;
                    int mine = 0;
                    bool any = false;
                    for (int k = 0; k < 8; ++k)
                    {
                        const int dk = __shfl_sync(group, own, k, 8), ck = __shfl_sync(group, ch, k, 8);
                        if (dk == d)
                        {
                            mine = ck;
                            any = true;
                        }
                    }
                    if (any && mine < 0)
                        content = t.bodies[~mine];
                    else if (any)
                    {
                        content = t.nodes[mine].com_mass;
                        const int last = t.nodes[mine].last;
                        if (l + 1 < kLevels)
                            children = 1 + 8 * (after[t.n - 1 - last]
                                                + static_cast<uint32_t>(l - level_after(t.codes, t.n, last)));
                    }
                }
                if (block + static_cast<uint32_t>(q) < count)
                    put(out, block + q, box, l + 1, prefix, content, q < 7 ? block + q + 1 : next, children);
                else
                    atomicOr(err, DEV_ERR_BOUNDS);
                // after the chain's next split node, which is one of these children
                const int o = l < h.level ? 7 - digit(h.code, l + 1) : 7;
                if (o < 7)
                    next = block + static_cast<uint32_t>(o) + 1;
            }
        }

        // a lone body: the root is its leaf
        __global__ void lone_root_kernel(const TreeView t, RefNode* __restrict__ out)
        {
            put(out, 0, *t.box, 0, 0, t.bodies[0], 0, 0);
        }
    }

    int tree_on_device(nbody_cuda* ctx, size_t* count)
    {
        if (const uint64_t id = bh_build_id(ctx); id && ctx->query_nodes_id == id)
        {
            *count = ctx->query_nodes_count;
            return NBODY_OK;
        }
        TreeView t;
        if (const int st = bh_view(ctx, &t))
            return st;
        cudaStream_t s = ctx->stream;
        const int n = t.n;
        uint32_t* counts = t.words[0];
        uint32_t* after = t.words[1];
        int* parent = reinterpret_cast<int*>(t.words[2]);
        size_t total = 1;
        int cells = 0;
        cudaError_t e = cudaSuccess;
        if (n >= 2)
        {
            split_count_kernel<<<ceil_div(n, 256), 256, 0, s>>>(t.codes, n, counts);
            ++ctx->launches;
            e = exclusive_scan<uint32_t>(counts, after, static_cast<size_t>(n), static_cast<uint32_t*>(t.temp), s,
                                         &ctx->launches);
            unsigned long long kept = 0;
            uint32_t last[2] = { 0, 0 };
            if (e == cudaSuccess)
                e = cudaMemcpyAsync(&kept, t.cells, sizeof kept, cudaMemcpyDeviceToHost, s);
            if (e == cudaSuccess)
                e = cudaMemcpyAsync(&last[0], counts + n - 1, sizeof(uint32_t), cudaMemcpyDeviceToHost, s);
            if (e == cudaSuccess)
                e = cudaMemcpyAsync(&last[1], after + n - 1, sizeof(uint32_t), cudaMemcpyDeviceToHost, s);
            if (e != cudaSuccess)
                return ctx_cuda_fail(ctx, e, "tree export");
            if (const int st = check_device_error(ctx))     // waits for the copies
                return st;
            cells = static_cast<int>(kept);
            total = 1 + 8 * (static_cast<size_t>(last[0]) + last[1]);
        }
        if (total > UINT32_MAX)
            return ctx_fail(ctx, NBODY_ERR_INVALID, "the tree has more nodes than 32-bit links reach");
        ctx->query_nodes_id = 0;
        if (const int st = reserve_query_nodes(ctx, total * sizeof(RefNode)))
            return st;
        RefNode* out = static_cast<RefNode*>(ctx->query_nodes);
        if (n >= 2)
        {
            parent_kernel<<<ceil_div(cells, 256), 256, 0, s>>>(t.nodes, cells, parent);
            expand_kernel<<<ceil_div(static_cast<size_t>(cells) * 8, 256), 256, 0, s>>>(t, cells, parent, after, total,
                                                                                        out, ctx->dev_error);
            ctx->launches += 2;
        }
        else
        {
            lone_root_kernel<<<1, 1, 0, s>>>(t, out);
            ++ctx->launches;
        }
        e = cudaGetLastError();
        if (e != cudaSuccess)
            return ctx_cuda_fail(ctx, e, "tree export");
        ctx->query_nodes_id = t.build_id;
        ctx->query_nodes_count = total;
        *count = total;
        return NBODY_OK;
    }
}

extern "C" int nbody_cuda_tree_export(nbody_cuda* ctx, void* nodes, const size_t max_nodes, size_t* count)
{
    using namespace nbg;
    if (!ctx || !count)
        return NBODY_ERR_INVALID;
    // A small tree is kept on the host once it was exported: exporting it again needs no device
    // (1,000 bodies 7 us, 35 from the device). A larger one's first export would pay for it
    // (20,000 bodies, 3.7 MB: a build and an export 691 us, 543 without; again 190 and 320).
    constexpr size_t kHostBytes = size_t(1) << 20;
    const uint64_t id = bh_build_id(ctx);
    if (!id || ctx->tree_host_id != id)
    {
        size_t have = 0;
        if (const int st = tree_on_device(ctx, &have))
            return st;
        *count = have;
        if (!nodes || !max_nodes)
            return NBODY_OK;
        const size_t bytes = have * sizeof(RefNode);
        if (bytes > kHostBytes)
            return d2h(ctx, nodes, ctx->query_nodes, std::min(have, max_nodes) * sizeof(RefNode));
        ctx->tree_host_id = 0;
        ctx->tree_host.resize(bytes);
        if (const int st = d2h(ctx, ctx->tree_host.data(), ctx->query_nodes, bytes))
            return st;
        ctx->tree_host_id = ctx->query_nodes_id;
    }
    const size_t have = ctx->tree_host.size() / sizeof(RefNode);
    *count = have;
    if (nodes && max_nodes)
        std::memcpy(nodes, ctx->tree_host.data(), std::min(have, max_nodes) * sizeof(RefNode));
    return NBODY_OK;
}
