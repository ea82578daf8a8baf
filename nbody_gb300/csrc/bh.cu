// Barnes-Hut on the device: the reference's octree (source/bhtree.cpp:14-138) rebuilt from
// sorted 63-bit Morton codes, traversed with the reference's opening criterion.
//
// Pipeline per accelerate (all on the context's stream, no host round trip):
//   1. root box: the reference's fixed box centred at the origin with edge State::size
//      (source/detail/tree.h:20), or the smallest power-of-two cube around the bodies'
//      bounding box (tree_box = 1; an exact FP32 min/max); the same pass finds the
//      largest |m| and |x|, which fix the fixed-point scale of step 4;
//   2. morton_kernel: 21 bits per axis, q = floor((x - lo) * 2^21 / edge), clamped and
//      interleaved x -> bit 0: in integers for power-of-two cells on a cell-aligned corner
//      (always for the fitted box), else with both double operations rounded toward
//      -inf. Either way every body lands in exactly the octant the reference's float
//      centre comparisons choose (bounds.h:31-38), whose octant bit is set when the
//      coordinate is below the centre: reference octant = digit ^ 7;
//   3. radix_sort_pairs over (code, index): stable, so ties keep index order;
//   4. gather_sum_kernel: bodies into Morton order, and exact fixed-point (int64) prefix
//      sums of m and m*x within tiles of sorted bodies, plus a scan of the tile totals:
//      differences of their sums give each cell's mass and COM;
//   5. radix_tree_kernel, from prefix bytes of gather_sum_kernel: binary radix tree over
//      the sorted codes (Karras 2012), duplicates separated by index; each internal node's
//      common-prefix length fixes its octree level floor(prefix / 3) (capped at 21, the
//      last Morton level), and the node is flagged as an octree node here;
//   6. octree nodes = binary nodes whose level exceeds their parent's (plus the root).
//      A reference cell whose bodies all sit in one octant (a chain of single-child
//      cells) has the same centre of mass and mass at every level of the chain, and the
//      smallest cell of the chain is the easiest to accept, so the chain behaves exactly
//      as its deepest cell: that is the node kept. Each node lists its <= 8 children
//      (cells or single bodies); cells at the Morton limit (identical codes) are buckets
//      whose bodies are applied one by one when opened;
//   7. traverse_kernel: a warp walks the tree for 32 to 128 Morton-consecutive targets, opening
//      one cell at a time for the targets that rejected it. Every target applies the
//      reference test -- accept when |com - x|^2 > size^2 * theta^2 (bhtree.cpp:117-125), leaves
//      always applied, massless nodes skipped -- most often decided for all of them at once by
//      their bounding boxes, exactly; so each target sums exactly the nodes the reference's
//      traversal would, in an order that depends on the target alone (the sums agree bit for
//      bit whatever the walk's width).
#include <algorithm>
#include <cmath>
#include <cstdlib>
#include <cstring>
#include <type_traits>

#include "bh.cuh"
#include "common.cuh"
#include "context.cuh"
#include "scan.cuh"
#include "sort.cuh"

namespace nbg
{
    namespace
    {
        constexpr int kMortonBits = 21;
        constexpr int kMaxLevel = 21;
        // warps per CTA of the walk with H targets per lane: its stack entries carry H lane masks,
        // and the stacks of one CTA stay within 48 KB of static shared memory
        __host__ __device__ constexpr int trav_warps(const int h) { return h > 4 ? 4 : 8; }
        // and CTAs per SM: two targets a lane fit 64 registers (a million bodies: 3 to 7 % over
        // three CTAs of 80; one and four targets a lane were slower so)
        __host__ __device__ constexpr int trav_ctas(const int h) { return h > 4 || h == 2 ? 4 : 3; }
        // cells stacked by a walk: at most 7 stay per level (8 are pushed, 1 is popped), 22 levels
        constexpr int kStack = 164;
        // group walk: warps per CTA, list entries and stacked parent cells per warp (the
        // stack grows by at most 28 parents per tree level, 22 levels: 616 < 768)
        constexpr int kListWarps = 4;
        // interaction-list entries per warp: the long list (8 KB) drains half as often, the short
        // one (4 KB) keeps more warps resident when the groups are too few to fill them
        constexpr int kListLong = 512;
        constexpr int kListShort = 256;
        // CTAs per SM of the group walk with Q target pairs per lane: two pairs want 128 registers
        // for the list's loop (halo of 16.8M bodies: 41.0 ms at five CTAs, 37.8 at four, 40.8 at
        // three of 168), one pair is fastest with more warps (1M-body disk: 344 us at five, 377 at four)
        __host__ __device__ constexpr int list_ctas(const int q, const int cap)
        {
            return q == 4 ? 3 : (q == 2 ? 4 : (cap > kListShort ? 5 : 6));
        }
        constexpr int kGroupStack = 768;
        // parents stacked up to which a round's parents are taken a round ahead: 120 - 1 + 32, and
        // 616 from there, stay within the stack
        constexpr int kGroupAhead = 120;
        constexpr int kRuns = 4;            // runs (own acceptance boxes) per group
        constexpr int kBboxBlocks = 1024;
        constexpr int kBboxVals = 8;    // min x y z, max x y z, max |m|, max |x|
        constexpr int kStatsWords = 8;
        // The Morton sort: radix passes over the top 45 code bits (octree levels 1-15), then
        // each run of codes that agree on them (a level-15 cell) is put in order by the low 18
        // bits. A run longer than kMaxRun (not met by a workload of 16.8M disk and halo
        // bodies, whose longest is 10) instead makes the build finish with a full sort.
        constexpr int kRunShift = 18;
        constexpr int kMaxRun = 32;
        constexpr int kMomThreads = 512;
        constexpr int kMomItems = 4;
        constexpr int kMomTile = kMomThreads * kMomItems;   // bodies per cell-sum tile
    }

    struct BhState
    {
        size_t cap = 0;                 // bodies the buffers hold
        uint64_t* keys[2] = { nullptr, nullptr };
        uint32_t* vals[2] = { nullptr, nullptr };
        float4* spm = nullptr;          // pos_mass in Morton order
        float* srad = nullptr;          // target radius in Morton order
        int2* child = nullptr;          // binary children: >= 0 internal, < 0 ~leaf
        int2* range = nullptr;          // [first, last] of each internal node
        int* prefix = nullptr;          // common-prefix bits of each internal node
        uint8_t* octflag = nullptr;     // 1 for a binary node that is an octree node
        uint32_t* octidx = nullptr;     // octree nodes before each binary node; kIsOct set on one
        uint64_t* numbering = nullptr;  // number_kernel's tile counts (after a ticket word)
        Int64x4* psum = nullptr;        // N + 1 fixed-point sums of {m x, m y, m z, m} over the
                                        // sorted bodies before x within x's cell-sum tile
        OctNode* nodes = nullptr;
        void* temp = nullptr;           // sort and scan temporaries
        size_t temp_bytes = 0;
        BoxParams* box = nullptr;
        float* bbox_part = nullptr;
        unsigned* box_ticket = nullptr; // blocks that have left their bounds; 0 between builds
        SortSetup sort;
        bool small_ready = false;       // box, bbox_part and box_ticket are there
        unsigned long long* stats = nullptr;   // [0] interactions, [1] node visits, [2] octree nodes,
                                               // [3] the traversal's tile counter, [4] the Morton
                                               // sort's full-sort flag (as unsigned)
        const uint32_t* order = nullptr;       // sorted indices of the last build (keys/vals ping-pong)
        const uint64_t* codes = nullptr;
        bool built = false;                    // a whole tree, for built_n bodies, is on the device
        cudaEvent_t ev[3] = { nullptr, nullptr, nullptr };  // build start, traversal start, end
        bool timed = false;                    // ev[] bracket the last accelerate
        size_t built_n = 0;
        uint64_t build_id = 0;
    };

    // ------------------------------------------------------------------------------------
    // 1. root box
    // ------------------------------------------------------------------------------------
    // The exponent e with 0 <= v < 2^e for a finite float v >= 0 (v = M 2^(E - 150) with
    // M < 2^24, so v < 2^(E - 126); subnormals and zero lie below 2^-126).
    __device__ __forceinline__ int bound_exp(const float v)
    {
        const uint32_t E = (__float_as_uint(v) >> 23) & 0xffu;
        return (E ? static_cast<int>(E) : 1) - 126;
    }

    // Order-preserving integers of floats (no NaN among them), for the integer warp reductions.
    __device__ __forceinline__ int ordered(const float v)
    {
        const int i = __float_as_int(v);
        return i ^ ((i >> 31) & 0x7fffffff);
    }

    __device__ __forceinline__ float unordered(const int i) { return __int_as_float(i ^ ((i >> 31) & 0x7fffffff)); }

    // The minima (first three) and maxima of v over a block of 256 threads, into red[.][0]: a warp
    // reduction, then thread a folds the eight warps' values a. min and max are exact.
    __device__ __forceinline__ void reduce_bounds(const float (&v)[kBboxVals], float (&red)[kBboxVals][8])
    {
#pragma unroll
        for (int a = 0; a < kBboxVals; ++a)
        {
            const int o = ordered(v[a]);
            const int r = a < 3 ? __reduce_min_sync(0xffffffffu, o) : __reduce_max_sync(0xffffffffu, o);
            if ((threadIdx.x & 31) == 0)
                red[a][threadIdx.x >> 5] = unordered(r);
        }
        __syncthreads();
        if (threadIdx.x < kBboxVals)
        {
            float r = red[threadIdx.x][0];
#pragma unroll
            for (int w = 1; w < 8; ++w)
                r = threadIdx.x < 3 ? fminf(r, red[threadIdx.x][w]) : fmaxf(r, red[threadIdx.x][w]);
            red[threadIdx.x][0] = r;
        }
        __syncthreads();
    }

    __device__ __forceinline__ double pow2(const int k) { return __hiloint2double((1023 + k) << 20, 0); }

    // One block of 256 threads folds the blocks' partials and writes the root box: lane a of the
    // first warp works out axis a. Bound by its chain of dependent steps: with a shared-memory
    // tree of eight barriers and one thread for all axes and powers, a step of 65,536 bodies took
    // 143.8 us, now 141.9; of 262,144 203.3, now 201.4.
    __device__ void finish_box(const float* part, const int nparts, const int n, const int mode, const float size,
                               float (&red)[kBboxVals][8], BoxParams* __restrict__ box)
    {
        float v[kBboxVals] = { INFINITY, INFINITY, INFINITY, -INFINITY, -INFINITY, -INFINITY, 0.f, 0.f };
        for (int k = threadIdx.x; k < nparts; k += blockDim.x)
        {
#pragma unroll
            for (int a = 0; a < 3; ++a)
                v[a] = fminf(v[a], __ldcg(&part[k * kBboxVals + a]));
#pragma unroll
            for (int a = 3; a < kBboxVals; ++a)
                v[a] = fmaxf(v[a], __ldcg(&part[k * kBboxVals + a]));
        }
        reduce_bounds(v, red);
        if (threadIdx.x >= 32)
            return;
        const int a = min(static_cast<int>(threadIdx.x), 2);
        double lo_a, center, edge;
        if (mode == 0)
        {
            // tree.h:20 / bhtree.h:29: centred at the origin, edge State::size
            edge = static_cast<double>(size);
            lo_a = -0.5 * edge;
            center = 0.0;
        }
        else
        {
            const double lo = red[a][0], hi = red[3 + a][0];
            double ext = 0.0;
#pragma unroll
            for (int c = 0; c < 3; ++c)
                ext = fmax(ext, static_cast<double>(red[3 + c][0]) - static_cast<double>(red[c][0]));
            // the smallest power of two above ext (a difference of floats: ext = f 2^k, f in
            // [0.5, 1), is normal), which keeps the maximum strictly inside the top cell; 1 for a
            // zero or non-finite extent
            int k = ext > 0.0 && isfinite(ext) ? ((__double2hiint(ext) >> 20) & 0x7ff) - 1022 : 0;
            // centre the cube on the bodies, then move its corner down onto the cell grid
            // (a shift of less than one cell); double the edge if that would uncover the
            // maximum. Cells are powers of two, so dividing by one is an exact multiply.
            for (int pass = 0;; ++pass, ++k)
            {
                edge = pow2(k);
                if (pass == 2)
                    break;
                const double c = isfinite(lo) ? 0.5 * (lo + hi) : 0.0;
                lo_a = floor((c - 0.5 * edge) * pow2(kMortonBits - k)) * pow2(k - kMortonBits);
                center = lo_a + 0.5 * edge;
                if (__all_sync(0xffffffffu, !isfinite(hi) || hi < lo_a + edge))
                    break;
            }
        }
        // the integer quantisation applies when the cells are powers of two and the corner
        // sits on their grid (always for the fitted cube)
        int ex = 0;
        const double mant = frexp(edge, &ex);
        const int cell_exp = ex - 1 - kMortonBits;
        const double lc = ldexp(lo_a, -cell_exp);
        const bool exact = __all_sync(0xffffffffu, mant == 0.5 && isfinite(edge) && cell_exp >= -149 && lc == floor(lc) &&
                                                       fabs(lc) < 4.0e15);
        if (threadIdx.x < 3)
        {
            box->lo[a] = lo_a;
            box->center[a] = center;
            box->lo_cells[a] = exact ? static_cast<long long>(lc) : 0;
        }
        if (threadIdx.x != 0)
            return;
        // |m| < 2^em and |x| < 2^ex for every finite value, and n <= 2^cn, so
        // n |m| 2^mass_shift and n |m x| 2^mom_shift stay below 2^61
        const int cn = n > 1 ? 32 - __clz(n - 1) : 0;
        const int m_exp = bound_exp(red[6][0]), x_exp = bound_exp(red[7][0]);
        box->mass_shift = 61 - cn - m_exp;
        box->mom_shift = 61 - cn - m_exp - x_exp;
        box->edge = edge;
        box->inv_cell = static_cast<double>(1u << kMortonBits) / edge;
        box->cell_exp = cell_exp;
        box->exact = exact ? 1 : 0;
        box->edge_f = static_cast<float>(edge);
    }

    // Per block: the box's min and max per axis, and the largest finite |m| and |x| (over
    // all axes), which fix the fixed-point scale of the cell sums. Min and max are exact,
    // so the float fold equals a double one; the partials are widened at the end.
    // The last block to leave its partials folds them into the root box. The grid also zeroes
    // what the kernels after it count in (zero_a and zero_b, in 16-byte units), which as
    // memsets were two more launches.
    __global__ void __launch_bounds__(256) bbox_kernel(const float4* __restrict__ src, const int stride, const int n,
                                                       const int mode, const float size, float* part,
                                                       unsigned* __restrict__ ticket, uint4* __restrict__ zero_a,
                                                       const size_t count_a, uint4* __restrict__ zero_b,
                                                       const size_t count_b, BoxParams* __restrict__ box)
    {
        after_previous();
        for (size_t k = blockIdx.x * 256u + threadIdx.x; k < count_a; k += gridDim.x * 256u)
            zero_a[k] = make_uint4(0u, 0u, 0u, 0u);
        for (size_t k = blockIdx.x * 256u + threadIdx.x; k < count_b; k += gridDim.x * 256u)
            zero_b[k] = make_uint4(0u, 0u, 0u, 0u);
        float v[kBboxVals] = { INFINITY, INFINITY, INFINITY, -INFINITY, -INFINITY, -INFINITY, 0.f, 0.f };
        auto fold = [&](const float4 p, const float m) {
            const float x[3] = { p.x, p.y, p.z };
#pragma unroll
            for (int a = 0; a < 3; ++a)
            {
                v[a] = fminf(v[a], x[a]);
                v[3 + a] = fmaxf(v[3 + a], x[a]);
                if (isfinite(x[a]))
                    v[7] = fmaxf(v[7], fabsf(x[a]));
            }
            if (isfinite(m))
                v[6] = fmaxf(v[6], fabsf(m));
        };
        const int step = gridDim.x * blockDim.x;
        int i = blockIdx.x * blockDim.x + threadIdx.x;
        // four bodies in flight per thread
        for (; static_cast<long long>(i) + 3 * step < n; i += 4 * step)
        {
            float4 p[4];
            float m[4];
#pragma unroll
            for (int u = 0; u < 4; ++u)
            {
                const size_t k = static_cast<size_t>(i + u * step);
                p[u] = src[k * stride];
                m[u] = stride == 3 ? src[k * 3 + 1].w : p[u].w;
            }
#pragma unroll
            for (int u = 0; u < 4; ++u)
                fold(p[u], m[u]);
        }
        for (; i < n; i += step)
        {
            const float4 p = src[static_cast<size_t>(i) * stride];
            fold(p, stride == 3 ? src[static_cast<size_t>(i) * 3 + 1].w : p.w);
        }
        __shared__ float red[kBboxVals][8];
        reduce_bounds(v, red);
        __shared__ bool last;
        if (threadIdx.x < kBboxVals)
        {
            part[blockIdx.x * kBboxVals + threadIdx.x] = red[threadIdx.x][0];
            __threadfence();
        }
        __syncthreads();
        if (threadIdx.x == 0)
            last = atomicAdd(ticket, 1u) == gridDim.x - 1;
        __syncthreads();
        if (!last)
            return;
        __threadfence();
        if (threadIdx.x == 0)
            *ticket = 0;        // for the next build
        finish_box(part, gridDim.x, n, mode, size, red, box);
    }

    // ------------------------------------------------------------------------------------
    // 2. Morton codes
    // ------------------------------------------------------------------------------------
    __device__ __forceinline__ uint64_t spread3(uint64_t v)
    {
        v &= 0x1fffffull;
        v = (v | (v << 32)) & 0x001f00000000ffffull;
        v = (v | (v << 16)) & 0x001f0000ff0000ffull;
        v = (v | (v << 8)) & 0x100f00f00f00f00full;
        v = (v | (v << 4)) & 0x10c30c30c30c30c3ull;
        v = (v | (v << 2)) & 0x1249249249249249ull;
        return v;
    }

    __device__ __forceinline__ uint64_t quantise(const float x, const double lo, const double inv_cell)
    {
        const double t = __dmul_rd(__dsub_rd(static_cast<double>(x), lo), inv_cell);
        const double f = floor(t);
        if (!(f >= 0.0))
            return 0;
        if (f > 2097151.0)
            return 2097151;
        return static_cast<uint64_t>(f);
    }

    // The same cell index with integer operations only, for a box whose cells are 2^cell_exp
    // and whose corner is lo_cells cells from the origin: x = M 2^E exactly (M the 24-bit
    // significand), so floor(x / cell) = floor(M 2^(E - cell_exp)) is a shift (rounding
    // toward -inf for negative x), and the index is that minus lo_cells, clamped. It equals
    // quantise() there: the directed roundings make floor(rd(rd(x - lo) * inv_cell)) the
    // exact floor((x - lo) / cell) when every cell boundary is a double.
    __device__ __forceinline__ uint64_t quantise_exact(const float x, const int cell_exp, const long long lo_cells)
    {
        const uint32_t bits = __float_as_uint(x);
        const uint32_t e = (bits >> 23) & 0xffu;
        const uint32_t frac = bits & 0x7fffffu;
        const bool neg = bits >> 31;
        if (e == 0xffu)
            return (frac == 0 && !neg) ? 2097151u : 0u;     // +inf clamps high; -inf and NaN to 0
        const long long m = e ? static_cast<long long>(frac | 0x800000u) : static_cast<long long>(frac);
        const int s = (e ? static_cast<int>(e) - 150 : -149) - cell_exp;     // x / cell = m 2^s
        long long cells;
        if (s >= 0)
        {
            if (s > 38)     // |x| / cell >= 2^61: far outside the box
                return neg ? 0u : 2097151u;
            cells = neg ? -(m << s) : (m << s);
        }
        else
        {
            const int r = -s;
            if (r >= 62)
                cells = (neg && m) ? -1 : 0;
            else
                cells = neg ? -((m + (1ll << r) - 1) >> r) : (m >> r);
        }
        const long long q = cells - lo_cells;
        return q < 0 ? 0u : (q > 2097151 ? 2097151u : static_cast<uint64_t>(q));
    }

    constexpr int kMortonItems = 4;     // bodies per thread, all loads issued first

    __global__ void __launch_bounds__(256) morton_kernel(const float4* __restrict__ src, const int stride,
                                                         const int n, const BoxParams* __restrict__ box,
                                                         uint64_t* __restrict__ keys, uint32_t* __restrict__ vals)
    {
        after_previous();
        const int base = blockIdx.x * (256 * kMortonItems) + threadIdx.x;
        float4 p[kMortonItems];
#pragma unroll
        for (int j = 0; j < kMortonItems; ++j)
        {
            const int i = base + j * 256;
            p[j] = i < n ? src[static_cast<size_t>(i) * stride] : make_float4(0.f, 0.f, 0.f, 0.f);
        }
        const BoxParams& b = *box;
#pragma unroll
        for (int j = 0; j < kMortonItems; ++j)
        {
            const int i = base + j * 256;
            if (i >= n)
                break;
            uint64_t qx, qy, qz;
            if (b.exact)
            {
                qx = quantise_exact(p[j].x, b.cell_exp, b.lo_cells[0]);
                qy = quantise_exact(p[j].y, b.cell_exp, b.lo_cells[1]);
                qz = quantise_exact(p[j].z, b.cell_exp, b.lo_cells[2]);
            }
            else
            {
                qx = quantise(p[j].x, b.lo[0], b.inv_cell);
                qy = quantise(p[j].y, b.lo[1], b.inv_cell);
                qz = quantise(p[j].z, b.lo[2], b.inv_cell);
            }
            keys[i] = spread3(qx) | (spread3(qy) << 1) | (spread3(qz) << 2);
            vals[i] = static_cast<uint32_t>(i);
        }
    }

    // After the radix passes over bits [kRunShift, 63), the codes are in order of their top
    // bits, and the codes of one run (equal top bits) keep index order. The thread at the
    // start of a run of 2 .. kMaxRun codes puts it in order of the whole code by a stable
    // insertion sort, so ties keep index order: the result is the order by (code, index).
    // A longer run sets *full, and the build sorts everything again by all 63 bits. Other
    // threads read their neighbours' top bits while a run is being reordered: those bits are
    // the same for every code of the run, so what they see does not depend on the moment.
    __global__ void __launch_bounds__(256) run_sort_kernel(uint64_t* __restrict__ keys, uint32_t* __restrict__ vals,
                                                           const int n, unsigned* __restrict__ full)
    {
        after_previous();
        const int i = blockIdx.x * 256 + threadIdx.x;
        if (i >= n)
            return;
        const uint64_t top = keys[i] >> kRunShift;
        if (i > 0 && (keys[i - 1] >> kRunShift) == top)
            return;     // not the first code of its run
        int len = 1;
        while (i + len < n && len <= kMaxRun && (keys[i + len] >> kRunShift) == top)
            ++len;
        if (len == 1)
            return;
        if (len > kMaxRun)
        {
            atomicOr(full, 1u);
            return;
        }
        for (int a = i + 1; a < i + len; ++a)
        {
            const uint64_t k = keys[a];
            const uint32_t v = vals[a];
            int b = a - 1;
            while (b >= i && keys[b] > k)
            {
                keys[b + 1] = keys[b];
                vals[b + 1] = vals[b];
                --b;
            }
            keys[b + 1] = k;
            vals[b + 1] = v;
        }
    }

    // ------------------------------------------------------------------------------------
    // 4. Morton-ordered copies and the fixed-point cell sums
    // ------------------------------------------------------------------------------------
    // A cell's mass and centre of mass come from differences of prefix sums over the sorted
    // bodies. The sums are integers -- each body's m 2^mass_shift and m x 2^mom_shift,
    // rounded once -- so a difference is the exact sum of the cell's rounded terms: no
    // cancellation against the large prefixes before it, and the same bits whatever order
    // the additions run in. A body's term is formed from the float significands with
    // integer multiplies (m x is an exact 48-bit product), without FP64 arithmetic.

    // v = M 2^e with M < 2^24 (the significand, implicit bit included); false for inf/NaN
    __device__ __forceinline__ bool split_float(const float v, uint32_t& M, int& e, bool& neg)
    {
        const uint32_t bits = __float_as_uint(v);
        const uint32_t E = (bits >> 23) & 0xffu;
        neg = (bits >> 31) != 0;
        M = E ? ((bits & 0x7fffffu) | 0x800000u) : (bits & 0x7fffffu);
        e = (E ? static_cast<int>(E) : 1) - 150;
        return E != 0xffu;
    }

    // round(P 2^s), halves away from zero, with the sign applied. P < 2^48; the box's shifts
    // keep P 2^s below 2^61, so a left shift never overflows (and s >= 64 only when P = 0).
    __device__ __forceinline__ long long fixed_round(const uint64_t P, const int s, const bool neg)
    {
        uint64_t q;
        if (s >= 0)
            q = s < 64 ? P << s : 0;
        else if (s > -50)
            q = (P + (1ull << (-s - 1))) >> -s;
        else
            q = 0;      // P 2^s < 2^-2
        return neg ? -static_cast<long long>(q) : static_cast<long long>(q);
    }

    // {m x, m y, m z, m} of one body in the box's fixed-point units. A non-finite mass
    // contributes nothing; a non-finite coordinate contributes no moment on its axis.
    __device__ __forceinline__ Int64x4 body_terms(const float4 pm, const int mass_shift, const int mom_shift)
    {
        uint32_t Mm;
        int em;
        bool nm;
        if (!split_float(pm.w, Mm, em, nm))
            return Int64x4{ 0, 0, 0, 0 };
        const float x[3] = { pm.x, pm.y, pm.z };
        long long q[3];
#pragma unroll
        for (int a = 0; a < 3; ++a)
        {
            uint32_t Mx;
            int ex;
            bool nx;
            q[a] = split_float(x[a], Mx, ex, nx)
                       ? fixed_round(static_cast<uint64_t>(Mm) * Mx, em + ex + mom_shift, nm != nx) : 0;
        }
        return Int64x4{ q[0], q[1], q[2], fixed_round(Mm, em + mass_shift, nm) };
    }

    __device__ __forceinline__ Int64x4 add4(const Int64x4 a, const Int64x4 b)
    {
        return Int64x4{ a.x + b.x, a.y + b.y, a.z + b.z, a.w + b.w };
    }

    // dl[k] = the common prefix of keys k and k + 1 for k < n - 1: 1 .. 95, one byte (64 + the
    // bits that their indices share when they are equal), and smp[k] = the key at 64 k for
    // 64 k < n - 1: those of k0 .. k0 + 3 (k0 a multiple of 4). For sorted keys the common
    // prefix of keys i < j is the least of dl[i .. j - 1].
    __device__ __forceinline__ void adjacent_prefixes(const uint64_t* __restrict__ keys, const int n, const int k0,
                                                      uint8_t* __restrict__ dl, uint64_t* __restrict__ smp)
    {
        if (k0 >= n - 1)
            return;
        uint64_t a[5];
#pragma unroll
        for (int u = 0; u < 5; ++u)
            a[u] = keys[min(k0 + u, n - 1)];
        if ((k0 & 63) == 0)
            smp[k0 >> 6] = a[0];        // every 64th key, for the far nodes' coarse searches
        uint32_t packed = 0;
#pragma unroll
        for (int u = 0; u < 4; ++u)
        {
            const int k = k0 + u;
            const uint32_t v = a[u] != a[u + 1]
                                   ? static_cast<uint32_t>(__clzll(static_cast<long long>(a[u] ^ a[u + 1])))
                                   : 64u + static_cast<uint32_t>(__clz(k ^ (k + 1)));
            packed |= (k < n - 1 ? v : 0u) << (8 * u);
        }
        if (k0 + 4 <= n - 1)
            *reinterpret_cast<uint32_t*>(dl + k0) = packed;
        else
            for (int u = 0; k0 + u < n - 1; ++u)
                dl[k0 + u] = static_cast<uint8_t>(packed >> (8 * u));
    }

    // Bodies into Morton order (pos_mass, and the radius when srad is given: only the cutoff
    // law reads it), and the fixed-point prefix sums within each tile of kMomTile sorted
    // bodies: part[x] = the sum of the terms of the bodies of x's tile before x, for
    // x = 0 .. n (x = n belongs to tile n / kMomTile, which is past the last tile, and has
    // sum 0, when n is a multiple of the tile). Each tile's total goes to tile_sum; the sum
    // of all bodies before x is then tile_prefix[x / kMomTile] + part[x], with tile_prefix
    // the exclusive scan of the totals (a tile past the last has total 0). Tiles need not
    // wait for one another. Four consecutive bodies per thread; every random read is issued
    // before any is used (indices past the end read the last body and are not stored). The
    // adjacent prefixes of the sorted keys, which the radix tree is found from, are formed here
    // too: they depend on the same sort and nothing else.
    __global__ void __launch_bounds__(kMomThreads) gather_sum_kernel(
        const float4* __restrict__ src, const int stride, const float4* __restrict__ vel_radius,
        const uint32_t* __restrict__ order, const int n, const BoxParams* __restrict__ box,
        float4* __restrict__ spm, float* __restrict__ srad, Int64x4* __restrict__ part,
        Int64x4* __restrict__ tile_sum, const uint64_t* __restrict__ keys, uint8_t* __restrict__ dl,
        uint64_t* __restrict__ smp)
    {
        after_previous();
        using Op = ScanOps<Int64x4>;
        if (n <= 0)
            return;
        __shared__ Int64x4 warp_tot[kMomThreads / 32];
        const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
        const int tile = blockIdx.x;
        const int mass_shift = box->mass_shift, mom_shift = box->mom_shift;
        const int base = tile * kMomTile + threadIdx.x * kMomItems;

        uint32_t idx[kMomItems];
        if (base + kMomItems <= n)
        {
            const uint4 o = *reinterpret_cast<const uint4*>(order + base);
            idx[0] = o.x;
            idx[1] = o.y;
            idx[2] = o.z;
            idx[3] = o.w;
        }
        else
        {
#pragma unroll
            for (int k = 0; k < kMomItems; ++k)
                idx[k] = order[min(base + k, n - 1)];
        }
        float4 p[kMomItems];
        float m[kMomItems], r[kMomItems];
#pragma unroll
        for (int k = 0; k < kMomItems; ++k)
        {
            const uint32_t i = idx[k];
            p[k] = src[static_cast<size_t>(i) * stride];
            if (stride == 3)
            {
                m[k] = src[static_cast<size_t>(i) * 3 + 1].w;     // Body: {pos, radius}, {vel, mass}
                r[k] = p[k].w;
            }
            else
            {
                m[k] = p[k].w;
                r[k] = vel_radius ? vel_radius[i].w : 0.f;
            }
        }
        // the radix tree's prefix bytes, while those reads are in flight
        adjacent_prefixes(keys, n, base, dl, smp);
        // the thread's total here; its bodies' terms are formed again for the prefixes below
        // (cheaper than holding four more Int64x4 through the scan)
        Int64x4 run{ 0, 0, 0, 0 };
#pragma unroll
        for (int k = 0; k < kMomItems; ++k)
        {
            const int i = base + k;
            p[k].w = m[k];
            if (i < n)
            {
                spm[i] = p[k];
                if (srad)
                    srad[i] = r[k];
                run = add4(run, body_terms(p[k], mass_shift, mom_shift));
            }
        }

        // the tile's scan: within warps, then over the warps' totals
        Int64x4 incl = run;
#pragma unroll
        for (int d = 1; d < 32; d <<= 1)
        {
            const Int64x4 o = Op::shfl_up(incl, d);
            if (lane >= d)
                incl = add4(incl, o);
        }
        if (lane == 31)
            warp_tot[warp] = incl;
        __syncthreads();
        if (warp == 0)
        {
            constexpr int kWarpsPerTile = kMomThreads / 32;
            Int64x4 wi = lane < kWarpsPerTile ? warp_tot[lane] : Int64x4{ 0, 0, 0, 0 };
#pragma unroll
            for (int d = 1; d < 32; d <<= 1)
            {
                const Int64x4 o = Op::shfl_up(wi, d);
                if (lane >= d)
                    wi = add4(wi, o);
            }
            if (lane < kWarpsPerTile)
                warp_tot[lane] = wi;    // inclusive over warps
            if (lane == 31)
                tile_sum[tile] = wi;    // the tile's total
        }
        __syncthreads();
        Int64x4 off = Op::shfl_up(incl, 1);
        if (lane == 0)
            off = Int64x4{ 0, 0, 0, 0 };
        if (warp > 0)
            off = add4(off, warp_tot[warp - 1]);
#pragma unroll
        for (int k = 0; k < kMomItems; ++k)
        {
            const int i = base + k;
            if (i < n)
            {
                part[i] = off;
                off = add4(off, body_terms(p[k], mass_shift, mom_shift));
            }
        }
        if (base <= n - 1 && n - 1 < base + kMomItems)
        {
            const int past = (n % kMomTile) == 0 ? 1 : 0;    // x = n opens the tile past the last
            part[n] = past ? Int64x4{ 0, 0, 0, 0 } : off;
            tile_sum[tile + 1] = Int64x4{ 0, 0, 0, 0 };      // past the last tile: total 0
        }
    }

    // ------------------------------------------------------------------------------------
    // 5. binary radix tree (Karras 2012)
    // ------------------------------------------------------------------------------------
    // common-prefix length of sorted keys i and j (0 <= i < n), duplicates separated by
    // index (64 + the index bits they share); -1 for j outside [0, n)
    __device__ __forceinline__ int delta(const uint64_t* __restrict__ keys, const int n, const int i, const int j)
    {
        if (j < 0 || j >= n)
            return -1;
        const uint64_t a = keys[i], b = keys[j];
        if (a != b)
            return __clzll(static_cast<long long>(a ^ b));
        return 64 + __clz(static_cast<int>(static_cast<unsigned>(i) ^ static_cast<unsigned>(j)));
    }

    __device__ __forceinline__ int level_of(const int prefix) { return min(kMaxLevel, prefix / 3); }

    // one bit per byte of four 0x00 / 0xff bytes, byte 0 to bit 0
    __device__ __forceinline__ uint32_t movemask4(const uint32_t m) { return ((m & 0x80808080u) * 0x00204081u) >> 28; }

    // One bit for each of four bytes of x below the matching byte of lim (each <= 128),
    // without SIMD instructions, exact for bytes below 128 (every dl byte is at most 95):
    // with bit 7 set in each byte of x first, subtracting a byte of at most 128 borrows from
    // no other byte, and leaves bit 7 clear exactly where x's byte was the smaller.
    __device__ __forceinline__ uint32_t lt_mask4(const uint32_t x, const uint32_t lim)
    {
        return movemask4(~((x | 0x80808080u) - lim));
    }

    // 16 bytes: bit t set where byte t is below each byte of lim / equal to each byte of q
    __device__ __forceinline__ uint32_t lt_mask16(const uint4 w, const uint32_t lim)
    {
        return lt_mask4(w.x, lim) | (lt_mask4(w.y, lim) << 4) | (lt_mask4(w.z, lim) << 8) | (lt_mask4(w.w, lim) << 12);
    }

    __device__ __forceinline__ uint32_t eq_mask16(const uint4 w, const uint32_t q)
    {
        return lt_mask4(w.x ^ q, 0x01010101u) | (lt_mask4(w.y ^ q, 0x01010101u) << 4)
               | (lt_mask4(w.z ^ q, 0x01010101u) << 8) | (lt_mask4(w.w ^ q, 0x01010101u) << 12);
    }

    // The record of binary node i (Karras 2012) with range [lo, hi], split after gamma and
    // common prefix dnode bits, and whether it is an octree node. The range is bounded by
    // two splits, dmin at i's end and dfar at the other (-1 past either end of the array),
    // both below its own; its parent splits at the larger of the two (the smallest range
    // that strictly contains [lo, hi] ends where the shared prefix first shortens), so the
    // parent's prefix is known without a parent array. A node is an octree node when its
    // level exceeds its parent's, or it is the root.
    __device__ __forceinline__ void write_radix_node(const int i, const int lo, const int hi, const int gamma,
                                                     const int dnode, const int dmin, const int dfar,
                                                     int2* __restrict__ child, int2* __restrict__ range,
                                                     int* __restrict__ prefix, uint8_t* __restrict__ flag)
    {
        child[i] = make_int2(lo == gamma ? ~gamma : gamma, hi == gamma + 1 ? ~(gamma + 1) : gamma + 1);
        range[i] = make_int2(lo, hi);
        const int pre = dnode - 1;      // codes are 63-bit: the top key bit is always shared
        prefix[i] = pre;
        const int up = max(dmin, dfar) - 1;
        flag[i] = (i == 0 || level_of(pre) > level_of(up)) ? 1 : 0;
    }

    // Radix-tree nodes whose ranges end within about kNearScan keys (97.5 % of them at 16.8M
    // disk + halo bodies), found without searches. Node i extends in direction d while the
    // adjacent prefixes stay above dmin = delta(i, i - d), so its far end is the first byte
    // of dl beyond i (in that direction) that is <= dmin: 16 bytes are compared at a time.
    // Its split is the one position of its range's least prefix, dnode = delta(i, j): the
    // first byte equal to dnode from the range's low end. A node whose end lies farther is
    // found by eight lanes together (radix_tree_kernel): a lane's own search, 40 dependent
    // loads for the top levels' nodes, cost a second kernel 14 to 20 us at 65,536 to 262,144
    // bodies. In one kernel with the searches shared a step of 65,536 bodies takes 144 us (155),
    // of 262,144 203 (217), of 1,000,003 423 (433), of 16.8M 4,550 (4,533).
    constexpr int kNearScan = 64;
    constexpr int kNearChunks = kNearScan / 16 + 1;

    // Node i by the byte scans: false when its record is written, true when its range ends
    // too far for them
    __device__ __forceinline__ bool near_node(const uint64_t* __restrict__ keys, const uint8_t* __restrict__ dl,
                                              const int n, const int i, int2* __restrict__ child,
                                              int2* __restrict__ range, int* __restrict__ prefix,
                                              uint8_t* __restrict__ flag, unsigned* __restrict__ err)
    {
        const int dr = dl[i];
        const int dlf = i > 0 ? static_cast<int>(dl[i - 1]) : -1;
        const int d = dr - dlf >= 0 ? 1 : -1;
        const int dmin = d > 0 ? dlf : dr;
        int j = -1;
        if (dmin >= 0)
        {
            const uint32_t rep = static_cast<uint32_t>(dmin + 1) * 0x01010101u;     // bytes <= dmin
            if (d > 0)
            {
                // the first p >= i with dl[p] <= dmin, or n - 1 (past the last pair)
                for (int c = 0; c < kNearChunks; ++c)
                {
                    const int base = (i & ~15) + 16 * c;
                    uint32_t mk = base < n - 1 ? lt_mask16(*reinterpret_cast<const uint4*>(dl + base), rep) : 0u;
                    if (c == 0)
                        mk &= ~((1u << (i & 15)) - 1u);
                    const int past = n - 1 - base;      // bytes from here on are past the last pair
                    if (past < 16)
                        mk |= past <= 0 ? 0xffffu : (0xffffu << past) & 0xffffu;
                    if (mk)
                    {
                        j = base + __ffs(mk) - 1;
                        break;
                    }
                }
            }
            else
            {
                // the last p <= i - 1 with dl[p] <= dmin, plus one; or 0 (before the first)
                for (int c = 0; c < kNearChunks; ++c)
                {
                    const int base = ((i - 1) & ~15) - 16 * c;
                    if (base < 0)
                    {
                        j = 0;
                        break;
                    }
                    uint32_t mk = lt_mask16(*reinterpret_cast<const uint4*>(dl + base), rep);
                    if (c == 0)
                        mk &= (2u << ((i - 1) & 15)) - 1u;
                    if (mk)
                    {
                        j = base + (31 - __clz(mk)) + 1;
                        break;
                    }
                    if (base == 0)
                    {
                        j = 0;
                        break;
                    }
                }
            }
        }
        if (j < 0)
            return true;
        const int lo = min(i, j), hi = max(i, j);
        const int dnode = delta(keys, n, i, j);
        const uint32_t rq = static_cast<uint32_t>(dnode) * 0x01010101u;
        int gamma = -1;
        for (int c = 0; c < kNearChunks + 1; ++c)
        {
            const int base = (lo & ~15) + 16 * c;
            if (base > n - 2)
                break;      // past the last pair: the split was not found
            uint32_t mk = eq_mask16(*reinterpret_cast<const uint4*>(dl + base), rq);
            if (c == 0)
                mk &= ~((1u << (lo & 15)) - 1u);
            if (mk)
            {
                gamma = base + __ffs(mk) - 1;
                break;
            }
        }
        if (gamma < lo || gamma >= hi)
        {
            atomicOr(err, DEV_ERR_BOUNDS);      // a range without its split: not sorted keys
            return false;
        }
        const int dfar = d > 0 ? (j < n - 1 ? static_cast<int>(dl[j]) : -1) : (j > 0 ? static_cast<int>(dl[j - 1]) : -1);
        write_radix_node(i, lo, hi, gamma, dnode, dmin, dfar, child, range, prefix, flag);
        return false;
    }

    // The exclusive scan of the cell sums' tile totals by one block of 256 threads: the octree
    // records need it and the radix tree does not, so one block of that kernel has it done
    // before its others end (at 16.8M bodies, 8193 totals).
    __device__ void scan_totals(const Int64x4* __restrict__ in, Int64x4* __restrict__ out, const int count)
    {
        using Op = ScanOps<Int64x4>;
        __shared__ Int64x4 warp_tot[8];
        const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
        Int64x4 carry{ 0, 0, 0, 0 };        // all earlier chunks'
        for (int base = 0; base < count; base += 256)
        {
            const int i = base + threadIdx.x;
            Int64x4 incl = i < count ? in[i] : Int64x4{ 0, 0, 0, 0 };
#pragma unroll
            for (int d = 1; d < 32; d <<= 1)
            {
                const Int64x4 o = Op::shfl_up(incl, d);
                if (lane >= d)
                    incl = add4(incl, o);
            }
            if (lane == 31)
                warp_tot[warp] = incl;
            __syncthreads();
            Int64x4 off = Op::shfl_up(incl, 1);
            if (lane == 0)
                off = Int64x4{ 0, 0, 0, 0 };
            off = add4(off, carry);
#pragma unroll 1
            for (int w = 0; w < 8; ++w)
            {
                if (w < warp)
                    off = add4(off, warp_tot[w]);
                carry = add4(carry, warp_tot[w]);
            }
            if (i < count)
                out[i] = off;
            __syncthreads();
        }
    }

    __device__ __forceinline__ int delta_of(const uint64_t a, const int i, const uint64_t b, const int j)
    {
        return a != b ? __clzll(static_cast<long long>(a ^ b))
                      : 64 + __clz(static_cast<int>(static_cast<unsigned>(i) ^ static_cast<unsigned>(j)));
    }

    // How many of a monotone predicate's values on eight lanes hold: true on the first ones,
    // false from there. Every lane of the warp calls it.
    __device__ __forceinline__ int count_leading(const bool t, const int lane)
    {
        const unsigned b = ~(__ballot_sync(0xffffffffu, t) >> (lane & 24)) & 0xffu;
        return b ? __ffs(b) - 1 : 8;
    }

    // Searches of four nodes by a warp, eight lanes each. For sorted keys dl[ref .. P - 1] > D exactly
    // when the common prefix of keys ref and P exceeds D, so a coarse search over every 64th key
    // (the samples, 1/64 of the keys, stay in the caches) finds the last sample P for which it
    // does: eight powers of two at once, then eight points of the bracket at once. The answer
    // lies in the 64 bytes after it, which the lanes compare 16 each.
    //
    // The first p >= start with dl[p] <= D (n - 1 when none: past the last pair), given
    // dl[ref .. start - 1] > D and kref = key ref.
    __device__ __forceinline__ int first_le_up(const uint64_t* __restrict__ smp, const uint8_t* __restrict__ dl,
                                               const int n, const uint64_t kref, const int ref, const int start,
                                               const int D, const int lane, unsigned* __restrict__ err)
    {
        const int sub = lane & 7, ka = (start >> 6) + 1;
        auto f = [&](const int k) { return k < (n + 62) / 64 && delta_of(kref, ref, smp[k], 64 * k) > D; };
        int e = 0;
        for (bool open = true; __any_sync(0xffffffffu, open);)
        {
            const int c = count_leading(open && e + sub < 25 && f(ka + (1 << (e + sub)) - 1), lane);
            e += open ? c : 0;
            open = open && c == 8;
        }
        int lo = e ? ka + (1 << (e - 1)) - 1 : 0, hi = e ? ka + (1 << e) - 1 : 0;
        while (__any_sync(0xffffffffu, hi - lo > 1))
        {
            const int stride = (hi - lo + 7) / 8, k = lo + (sub + 1) * stride;
            const int held = count_leading(k < hi && f(k), lane);
            hi = min(hi, lo + (held + 1) * stride);
            lo += held * stride;
        }
        const int q0 = e ? 64 * lo : start;
        const int base = (q0 & ~15) + 16 * sub;
        uint32_t mk = base < n - 1
                          ? lt_mask16(*reinterpret_cast<const uint4*>(dl + base), static_cast<uint32_t>(D + 1) * 0x01010101u)
                          : 0u;
        if (sub == 0)
            mk &= ~((1u << (q0 & 15)) - 1u);
        const int past = n - 1 - base;      // bytes from here on are past the last pair
        if (past < 16)
            mk |= past <= 0 ? 0xffffu : (0xffffu << past) & 0xffffu;
        const unsigned any = (__ballot_sync(0xffffffffu, mk != 0u) >> (lane & 24)) & 0xffu;
        if (!any)
            atomicOr(err, DEV_ERR_BOUNDS);      // not sorted keys
        const int p = __shfl_sync(0xffffffffu, base + __ffs(mk) - 1, any ? __ffs(any) - 1 : 0, 8);
        return any ? p : n - 1;
    }

    // The last p <= start with dl[p] <= D (-1 when none), given dl[start + 1 .. ref - 1] > D.
    __device__ __forceinline__ int last_le_down(const uint64_t* __restrict__ smp, const uint8_t* __restrict__ dl,
                                                const uint64_t kref, const int ref, const int start, const int D,
                                                const int lane, unsigned* __restrict__ err)
    {
        const int sub = lane & 7, ka = start >> 6;
        auto f = [&](const int k) { return k >= 0 && delta_of(kref, ref, smp[k], 64 * k) > D; };
        int e = 0;
        for (bool open = true; __any_sync(0xffffffffu, open);)
        {
            const int c = count_leading(open && e + sub < 25 && f(ka - (1 << (e + sub)) + 1), lane);
            e += open ? c : 0;
            open = open && c == 8;
        }
        int hi = e ? ka - (1 << (e - 1)) + 1 : 0, lo = e ? ka - (1 << e) + 1 : 0;
        while (__any_sync(0xffffffffu, hi - lo > 1))
        {
            const int stride = (hi - lo + 7) / 8, k = hi - (sub + 1) * stride;
            const int held = count_leading(k > lo && f(k), lane);
            lo = max(lo, hi - (held + 1) * stride);
            hi -= held * stride;
        }
        const int q0 = e ? 64 * hi - 1 : start;
        const int base = (q0 & ~15) - 16 * sub;
        uint32_t mk = 0;
        if (q0 >= 0 && base >= 0)
        {
            mk = lt_mask16(*reinterpret_cast<const uint4*>(dl + base), static_cast<uint32_t>(D + 1) * 0x01010101u);
            if (sub == 0)
                mk &= (2u << (q0 & 15)) - 1u;
        }
        const unsigned any = (__ballot_sync(0xffffffffu, mk != 0u) >> (lane & 24)) & 0xffu;
        if (!any && q0 >= 128)
            atomicOr(err, DEV_ERR_BOUNDS);      // not sorted keys
        const int p = __shfl_sync(0xffffffffu, base + 31 - __clz(mk), any ? __ffs(any) - 1 : 0, 8);
        return any ? p : -1;
    }

    // Block 0 scans the tile sums, the others take 256 nodes each: near ones a lane each, then
    // the CTA's far ones (six of 256 at 16.8M bodies) four a warp, so that few warps stay for
    // their dependent loads (each warp searching for its own far nodes took 2 % longer there).
    __global__ void __launch_bounds__(256) radix_tree_kernel(
        const uint64_t* __restrict__ keys, const uint8_t* __restrict__ dl, const uint64_t* __restrict__ smp, const int n,
        int2* __restrict__ child, int2* __restrict__ range, int* __restrict__ prefix, uint8_t* __restrict__ flag,
        const Int64x4* __restrict__ tile_sum, Int64x4* __restrict__ tile_prefix, const int tiles,
        unsigned* __restrict__ err)
    {
        after_previous();
        if (blockIdx.x == 0)
        {
            scan_totals(tile_sum, tile_prefix, tiles);
            return;
        }
        const int i = (blockIdx.x - 1) * 256 + threadIdx.x;
        const bool far = i < n - 1 && near_node(keys, dl, n, i, child, range, prefix, flag, err);
        // the CTA's nodes whose ranges end too far for the byte scans, eight lanes each
        __shared__ int far_node[256];
        __shared__ unsigned far_count;
        const int lane = threadIdx.x & 31;
        if (threadIdx.x == 0)
            far_count = 0;
        __syncthreads();
        const unsigned fm = __ballot_sync(0xffffffffu, far);
        if (fm)
        {
            unsigned at = lane == 0 ? atomicAdd(&far_count, static_cast<unsigned>(__popc(fm))) : 0u;
            at = __shfl_sync(0xffffffffu, at, 0);
            if (far)
                far_node[at + __popc(fm & ((1u << lane) - 1u))] = i;
        }
        __syncthreads();
        const unsigned count = far_count;
        for (unsigned q = (threadIdx.x >> 5) * 4; q < count; q += 32)
        {
            // (a group past the last one repeats it, and writes nothing)
            const bool mine = q + (lane >> 3) < count;
            const int node = far_node[min(q + (lane >> 3), count - 1)];
            const int dr = dl[node];
            const int dlf = node > 0 ? static_cast<int>(dl[node - 1]) : -1;
            const int d = dr - dlf >= 0 ? 1 : -1;
            const int dmin = d > 0 ? dlf : dr;
            // every lane makes both searches' calls; a group's other one ends at once
            const uint64_t ki = keys[node];
            const int up = first_le_up(smp, dl, n, ki, node, node, d > 0 ? dmin : 95, lane, err);
            const int down = last_le_down(smp, dl, ki, node, node - 1, d > 0 ? 95 : dmin, lane, err) + 1;
            const int j = d > 0 ? up : down;
            const int lo = min(node, j), hi = max(node, j);
            const int dnode = delta(keys, n, node, j);
            const int gamma = first_le_up(smp, dl, n, keys[lo], lo, lo, dnode, lane, err);
            if (mine && (lane & 7) == 0)
            {
                const int dfar = d > 0 ? (j < n - 1 ? static_cast<int>(dl[j]) : -1)
                                       : (j > 0 ? static_cast<int>(dl[j - 1]) : -1);
                if (gamma < lo || gamma >= hi)
                    atomicOr(err, DEV_ERR_BOUNDS);
                else
                    write_radix_node(node, lo, hi, gamma, dnode, dmin, dfar, child, range, prefix, flag);
            }
        }
    }

    // ------------------------------------------------------------------------------------
    // 6. octree records
    // ------------------------------------------------------------------------------------
    constexpr uint32_t kIsOct = 0x80000000u;
    constexpr int kNumTile = 4096;      // binary nodes per CTA of the numbering

    // octidx[i] = the octree nodes among binary nodes 0 .. i - 1, with kIsOct set when node i is one
    // itself (its index in the record array is then octidx[i] without it). One launch: tiles of
    // 4096 nodes taken in ticket order, the earlier tiles' count found by decoupled look-back
    // (count_before). status[0] is the ticket, status[1 + t] tile t's count, all zero before. A
    // wait that gives up counts nothing before its tile: indices stay in range.
    __global__ void __launch_bounds__(1024) number_kernel(const uint8_t* __restrict__ flag, const int m,
                                                          uint32_t* __restrict__ octidx, uint64_t* __restrict__ status,
                                                          unsigned* __restrict__ err)
    {
        after_previous();
        __shared__ uint32_t warp_tot[32];
        __shared__ uint32_t before_s;
        __shared__ int tile_s;
        const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
        if (threadIdx.x == 0)
            tile_s = static_cast<int>(atomicAdd(reinterpret_cast<unsigned*>(status), 1u));
        __syncthreads();
        const int tile = tile_s;
        const int base = tile * kNumTile + threadIdx.x * 4;
        uint32_t f = 0;     // a byte per node
        if (base + 4 <= m)
            f = *reinterpret_cast<const uint32_t*>(flag + base);
        else
            for (int k = 0; k < 4; ++k)
                f |= base + k < m ? static_cast<uint32_t>(flag[base + k]) << (8 * k) : 0u;
        const uint32_t mine = __popc(f);
        uint32_t incl = mine;
#pragma unroll
        for (int d = 1; d < 32; d <<= 1)
        {
            const uint32_t o = __shfl_up_sync(0xffffffffu, incl, d);
            if (lane >= d)
                incl += o;
        }
        if (lane == 31)
            warp_tot[warp] = incl;
        __syncthreads();
        if (warp == 0)
        {
            const uint32_t w = warp_tot[lane];
            uint32_t wi = w;
#pragma unroll
            for (int d = 1; d < 32; d <<= 1)
            {
                const uint32_t o = __shfl_up_sync(0xffffffffu, wi, d);
                if (lane >= d)
                    wi += o;
            }
            warp_tot[lane] = wi - w;        // before each warp
            const uint32_t total = __shfl_sync(0xffffffffu, wi, 31);
            if (lane == 0)
                store_relaxed(&status[1 + tile], (tile ? kCountOwn : kCountAll) | total);
            const uint32_t before = count_before(status + 1, tile, err);
            if (lane == 0)
            {
                if (tile)
                    store_relaxed(&status[1 + tile], kCountAll | (before + total));
                before_s = before;
            }
        }
        __syncthreads();
        uint32_t at = before_s + warp_tot[warp] + incl - mine;
        uint32_t out[4];
#pragma unroll
        for (int k = 0; k < 4; ++k)
        {
            const uint32_t is = (f >> (8 * k)) & 1u;
            out[k] = at | (is ? kIsOct : 0u);
            at += is;
        }
        if (base + 4 <= m)
            *reinterpret_cast<uint4*>(octidx + base) = make_uint4(out[0], out[1], out[2], out[3]);
        else
            for (int k = 0; k < 4; ++k)
                if (base + k < m)
                    octidx[base + k] = out[k];
    }

    // The children of a cell: walking down through the binary nodes of the cell's own level
    // (at most three splits below it), every leaf body and every node of a deeper level is
    // one child. Right subtrees first, which is the order the traversal has always used.
    // Children are kept in registers (kid[k] selected by a static index) and stored at once.
    __device__ __forceinline__ void emit_child(int (&kid)[8], int& nc, const int v, unsigned* __restrict__ err)
    {
#pragma unroll
        for (int k = 0; k < 8; ++k)
            kid[k] = k == nc ? v : kid[k];
        if (nc >= 8)
            atomicOr(err, DEV_ERR_BOUNDS);
        ++nc;
    }

    template <int DEPTH>
    __device__ __forceinline__ void collect_children(const int c, const int2* __restrict__ child,
                                                     const uint32_t* __restrict__ octidx, int (&kid)[8],
                                                     int& nc, unsigned* __restrict__ err)
    {
        const uint32_t w = c < 0 ? 0u : octidx[c];
        if (c < 0 || (w & kIsOct))
        {
            emit_child(kid, nc, c < 0 ? c : static_cast<int>(w & ~kIsOct), err);
            return;
        }
        if (DEPTH == 0)
        {
            atomicOr(err, DEV_ERR_BOUNDS);      // more than three splits inside one octal level
            return;
        }
        const int2 ch = child[c];
        collect_children<DEPTH ? DEPTH - 1 : 0>(ch.y, child, octidx, kid, nc, err);
        collect_children<DEPTH ? DEPTH - 1 : 0>(ch.x, child, octidx, kid, nc, err);
    }

    // position of the r-th set bit (from 0) of v, for r < popc(v)
    __device__ __forceinline__ int select_bit(unsigned v, int r)
    {
        int pos = 0;
#pragma unroll
        for (int w = 16; w > 0; w >>= 1)
        {
            const int c = __popc(v & ((1u << w) - 1u));
            if (r >= c)
            {
                r -= c;
                v >>= w;
                pos += w;
            }
        }
        return pos;
    }

    // An int64 as float: |v| split into two 32-bit halves, each converted exactly or with one
    // rounding, joined by one FMA (within about an ulp). No FP64 operation: GB300's FP64
    // pipe is its slowest.
    __device__ __forceinline__ float i64_to_float(const long long v)
    {
        const unsigned long long u = v < 0 ? 0ull - static_cast<unsigned long long>(v) : static_cast<unsigned long long>(v);
        const float f = fmaf(static_cast<float>(static_cast<uint32_t>(u >> 32)), 4294967296.0f,
                             static_cast<float>(static_cast<uint32_t>(u)));
        return v < 0 ? -f : f;
    }

    constexpr int kOctSpan = 4;     // binary nodes per lane that one warp scans for octree nodes

    // One octree record per flagged binary node. Latency bound (chains of dependent loads),
    // so a warp first gathers the flagged nodes among 32 * kOctSpan consecutive binary nodes
    // (ballots; about 40 % are flagged) and its lanes then take them in turn, instead of
    // idling on unflagged ones; and full occupancy (32 registers) beats fewer spills.
    __global__ void __launch_bounds__(256, 8) octnode_kernel(const int2* __restrict__ child, const int2* __restrict__ range,
                                   const int* __restrict__ prefix, const uint32_t* __restrict__ octidx, const Int64x4* __restrict__ part,
                                   const Int64x4* __restrict__ tile_prefix, const int m,
                                   const BoxParams* __restrict__ box, const float theta,
                                   OctNode* __restrict__ nodes, unsigned* __restrict__ err,
                                   unsigned long long* __restrict__ stats)
    {
        after_previous();
        const int gt = blockIdx.x * blockDim.x + threadIdx.x;
        if (gt == 0)
            atomicAdd(&stats[2], static_cast<unsigned long long>((octidx[m - 1] & ~kIsOct) + (octidx[m - 1] >> 31)));
        const int lane = threadIdx.x & 31;
        const int first = (gt >> 5) * (32 * kOctSpan);
        if (first >= m)
            return;     // the whole warp
        unsigned mask[kOctSpan];
        int total = 0;
#pragma unroll
        for (int u = 0; u < kOctSpan; ++u)
        {
            const int i = first + u * 32 + lane;
            mask[u] = __ballot_sync(0xffffffffu, i < m && (octidx[i] & kIsOct));
            total += __popc(mask[u]);
        }
        const int shift = box->mass_shift - box->mom_shift;
        for (int q = lane; q < total; q += 32)
        {
            int u = 0, r = q;
#pragma unroll
            for (int k = 0; k < kOctSpan - 1; ++k)
                if (u == k && r >= __popc(mask[k]))
                {
                    r -= __popc(mask[k]);
                    u = k + 1;
                }
            unsigned mu = mask[0];
#pragma unroll
            for (int k = 1; k < kOctSpan; ++k)
                mu = u == k ? mask[k] : mu;
            const int i = first + u * 32 + select_bit(mu, r);
            const int2 rg = range[i];
            const int pre = prefix[i];
            const int lvl = level_of(pre);
            // the sums before the cell's first body and after its last: exact integers
            const Int64x4 hi = add4(tile_prefix[(rg.y + 1) / kMomTile], part[rg.y + 1]);
            const Int64x4 lo = add4(tile_prefix[rg.x / kMomTile], part[rg.x]);
            const long long ms = hi.w - lo.w;   // exact: the cell's own terms
            OctNode* out = nodes + (octidx[i] & ~kIsOct);
            float4 cm = make_float4(0.f, 0.f, 0.f, 0.f);
            if (ms > 0)
            {
                // com = (sum of m x 2^mom_shift) / (sum of m 2^mass_shift) * 2^(mass_shift - mom_shift),
                // in float: the quotient lies in [-1, 1] before the exact power-of-two scaling
                const float fm = i64_to_float(ms);
                const float rm = __frcp_rn(fm);
                cm = make_float4(ldexpf(i64_to_float(hi.x - lo.x) * rm, shift),
                                 ldexpf(i64_to_float(hi.y - lo.y) * rm, shift),
                                 ldexpf(i64_to_float(hi.z - lo.z) * rm, shift), ldexpf(fm, -box->mass_shift));
            }
            // the reference's node size is the root size halved per level, in float
            const float sz = ldexpf(box->edge_f, -lvl);
            const float open_r2 = __fmul_rn(__fmul_rn(sz, sz), __fmul_rn(theta, theta));
            int kid[8] = { 0, 0, 0, 0, 0, 0, 0, 0 };
            int nc = 0;
            if (pre >= 3 * kMaxLevel)
                nc = -1;     // bucket: identical codes, bodies applied one by one
            else
            {
                const int2 ch = child[i];
                collect_children<2>(ch.y, child, octidx, kid, nc, err);
                collect_children<2>(ch.x, child, octidx, kid, nc, err);
                nc = min(nc, 8);
            }
            out->com_mass = cm;
            *reinterpret_cast<int4*>(&out->open_r2) = make_int4(__float_as_int(open_r2), nc, rg.x, rg.y);
            int4* kids = reinterpret_cast<int4*>(out->child);
            kids[0] = make_int4(kid[0], kid[1], kid[2], kid[3]);
            kids[1] = make_int4(kid[4], kid[5], kid[6], kid[7]);
        }
    }

    // ------------------------------------------------------------------------------------
    // 7. traversal
    // ------------------------------------------------------------------------------------
    template <int LAW>
    __device__ __forceinline__ void apply(const float px, const float py, const float pz, const float lim,
                                          const float sx, const float sy, const float sz, const float m,
                                          const bool take, float& ax, float& ay, float& az)
    {
        const float dx = sx - px, dy = sy - py, dz = sz - pz;
        float r2 = (LAW == NBODY_LAW_SOFTENED) ? fmaf(dx, dx, lim) : dx * dx;
        r2 = fmaf(dy, dy, r2);
        r2 = fmaf(dz, dz, r2);
        float inv = rsqrt_sfu(r2);
        if (LAW == NBODY_LAW_CUTOFF)
            inv = r2 > lim ? inv : 0.f;     // physics.h:38-39
        float s = m * inv * inv * inv;
        s = take ? s : 0.f;
        ax = fmaf(dx, s, ax);
        ay = fmaf(dy, s, ay);
        az = fmaf(dz, s, az);
    }

    // Two targets per lane: the packed form of apply(). Both halves run the scalar
    // operations of apply() in the same order (an FP32x2 operation is two correctly rounded
    // FP32 operations), and a half whose target does not take the node gets s = 0, which
    // adds exactly zero. Targets are held as negated positions (d = s + (-x)).
    template <int LAW>
    __device__ __forceinline__ void apply2(const float2 npx, const float2 npy, const float2 npz, const float2 lim,
                                           const float sx, const float sy, const float sz, const float m,
                                           const bool take_a, const bool take_b, float2& ax, float2& ay, float2& az)
    {
        const float2 dx = add2(f2(sx), npx), dy = add2(f2(sy), npy), dz = add2(f2(sz), npz);
        float2 r2 = (LAW == NBODY_LAW_SOFTENED) ? fma2(dx, dx, lim) : mul2(dx, dx);
        r2 = fma2(dy, dy, r2);
        r2 = fma2(dz, dz, r2);
        float2 inv = make_float2(rsqrt_sfu(r2.x), rsqrt_sfu(r2.y));
        if (LAW == NBODY_LAW_CUTOFF)
        {
            inv.x = r2.x > lim.x ? inv.x : 0.f;     // physics.h:38-39
            inv.y = r2.y > lim.y ? inv.y : 0.f;
        }
        float2 sc = mul2(mul2(mul2(f2(m), inv), inv), inv);
        sc.x = take_a ? sc.x : 0.f;
        sc.y = take_b ? sc.y : 0.f;
        ax = fma2(dx, sc, ax);
        ay = fma2(dy, sc, ay);
        az = fma2(dz, sc, az);
    }

    // The bounding boxes of a warp's targets, split into NSG runs at the NSG - 1 largest Morton
    // jumps between neighbours (lane l holds targets 32 h + l, h < H, of the nvalid ones from
    // t0): run[h] is the run of the lane's target h, and lo / hi receive, on every lane, the box
    // of run `mine` (an empty run's box is inverted, +inf to -inf).
    template <int H, int NSG>
    __device__ __forceinline__ void run_boxes(const uint64_t* __restrict__ codes, const int t0, const int nvalid,
                                              const int lane, const float3 (&pos)[H], const int mine, int (&run)[H],
                                              float3& lo, float3& hi)
    {
        unsigned key[H];    // (common prefix bits << 8 | position); 0xffffffff: no boundary
#pragma unroll
        for (int h = 0; h < H; ++h)
        {
            const int b = 32 * h + lane;        // boundary between positions b - 1 and b
            key[h] = 0xffffffffu;
            if (b > 0 && b < nvalid)
                key[h] = (static_cast<unsigned>(__clzll(static_cast<long long>(codes[t0 + b - 1] ^ codes[t0 + b]))) << 8)
                         | static_cast<unsigned>(b);
            run[h] = 0;
        }
#pragma unroll
        for (int s = 0; s < NSG - 1; ++s)
        {
            unsigned m = key[0];
#pragma unroll
            for (int h = 1; h < H; ++h)
                m = min(m, key[h]);
            m = __reduce_min_sync(0xffffffffu, m);
            const int split = m == 0xffffffffu ? 32 * H : static_cast<int>(m & 0xffu);
#pragma unroll
            for (int h = 0; h < H; ++h)
            {
                run[h] += 32 * h + lane >= split ? 1 : 0;
                if (key[h] == m)
                    key[h] = 0xffffffffu;
            }
        }
#pragma unroll
        for (int g = 0; g < NSG; ++g)
        {
            float3 l = make_float3(INFINITY, INFINITY, INFINITY), u = make_float3(-INFINITY, -INFINITY, -INFINITY);
#pragma unroll
            for (int h = 0; h < H; ++h)
                if (32 * h + lane < nvalid && run[h] == g)
                {
                    l = make_float3(fminf(l.x, pos[h].x), fminf(l.y, pos[h].y), fminf(l.z, pos[h].z));
                    u = make_float3(fmaxf(u.x, pos[h].x), fmaxf(u.y, pos[h].y), fmaxf(u.z, pos[h].z));
                }
#pragma unroll
            for (int o = 16; o > 0; o >>= 1)
            {
                l.x = fminf(l.x, __shfl_xor_sync(0xffffffffu, l.x, o));
                l.y = fminf(l.y, __shfl_xor_sync(0xffffffffu, l.y, o));
                l.z = fminf(l.z, __shfl_xor_sync(0xffffffffu, l.z, o));
                u.x = fmaxf(u.x, __shfl_xor_sync(0xffffffffu, u.x, o));
                u.y = fmaxf(u.y, __shfl_xor_sync(0xffffffffu, u.y, o));
                u.z = fmaxf(u.z, __shfl_xor_sync(0xffffffffu, u.z, o));
            }
            if (g == mine)
            {
                lo = l;
                hi = u;
            }
        }
    }

    // Who takes the (up to eight) sources of a cell's children: H bits per source.
    template <int H>
    struct TakeBits
    {
        using Word = typename std::conditional<(H > 4), uint64_t, uint32_t>::type;
        static constexpr Word kOnes = H == 8 ? Word(0x0101010101010101ull) : (H == 4 ? Word(0x11111111u)
                                      : (H == 2 ? Word(0x5555u) : Word(0xffu)));   // the first bit of each
        static __device__ __forceinline__ Word first(const int n)      // the bits of the first n sources
        {
            return n * H >= 8 * static_cast<int>(sizeof(Word)) ? ~Word(0) : (Word(1) << (n * H)) - 1;
        }
        static __device__ __forceinline__ unsigned count(const Word w)
        {
            return H > 4 ? __popcll(w) : __popc(static_cast<unsigned>(w));
        }
    };

    // |d|^2 in the reference's operation order (bhtree.cpp:117-125), every operation rounded on
    // its own
    __device__ __forceinline__ float dist2_rn(const float dx, const float dy, const float dz)
    {
        return __fadd_rn(__fadd_rn(__fmul_rn(dx, dx), __fmul_rn(dy, dy)), __fmul_rn(dz, dz));
    }

    // The per-target walk for 32 H Morton-consecutive targets per warp: lane l holds targets
    // 32 H t + 32 h + l for h < H, as packed pairs (2p, 2p + 1) when H > 1. Every target sums
    // exactly the nodes that the reference's test accepts for it.
    //
    // The walk opens one cell at a time, for the targets that opened it, and decides most of
    // its up to eight children for the whole warp at once: lane l tests child l % 8 against
    // the bounding box of run l / 8 of the targets. The nearest point of a box gives the least
    // distance any of its targets can have, the farthest corner the greatest -- exactly, in the
    // very roundings of the targets' own test, since each operation of it is monotone in the
    // distance per axis. A child beyond its opening distance of every run's nearest point is
    // taken by all who opened the parent; one within it of every run's farthest corner is
    // opened by all of them; only the others are tested target by target.
    //
    // The order of a target's sum: at each cell it opens, the leaves, then the children it
    // takes, both in child order; then the children it opens, the last first, each with its
    // subtree. That depends on the target alone, not on the others of its warp, so every H
    // gives the same bits.
    //
    // Bound by instruction issue and the latency of its short chains (IPC 2.6 of 4 at a million
    // bodies). The walk before it popped one cell at a time and tested all the warp's targets
    // against it. Walk alone, before and now: 4M disk + halo bodies, theta 0.5: 1.45 -> 1.00 ms,
    // theta 2: 22.5 -> 16.8 ms; a 1M-body disk under the cutoff law, theta 0.5:
    // 0.256 -> 0.197 ms; two Plummer spheres of 10,000 bodies, theta 0.5: 70 -> 41 us.
    template <int LAW, int H>
    __global__ void __launch_bounds__(trav_warps(H) * 32, trav_ctas(H)) traverse_kernel(
        const OctNode* __restrict__ nodes, const float4* __restrict__ spm, const float* __restrict__ srad,
        const uint64_t* __restrict__ codes, const uint32_t* __restrict__ order, const int n, const float G,
        const float eps2, float4* __restrict__ acc, float* __restrict__ body_out, unsigned* __restrict__ err,
        unsigned long long* __restrict__ stats)
    {
        after_previous();
        using Takes = typename TakeBits<H>::Word;
        constexpr int P = (H + 1) / 2;              // target pairs per lane (H = 1: one scalar target)
        constexpr int TW = 32 * H;                  // targets per warp
        constexpr int W = trav_warps(H);
        __shared__ float4 src_mem[W][8];            // the children's (com, mass), or a leaf's (x, m)
        __shared__ int stk_cell[W][kStack];         // cells to be opened
        __shared__ uint8_t stk_mine[W][kStack][32]; // by which of each lane's targets, a bit per slot
        const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
        float4* const srcs = src_mem[warp];
        unsigned inter = 0, visits = 0;

        // tiles are handed out in order by a counter (stats[3], zeroed with the statistics at
        // every build), so warps that drew cheap tiles take more of them: a tile from the
        // dense centre of a disk costs many times one from its edge
        auto next_tile = [&]() {
            unsigned long long t = 0;
            if (lane == 0)
                t = atomicAdd(&stats[3], 1ull);
            return static_cast<int>(__shfl_sync(0xffffffffu, t, 0));
        };
        for (int tile = next_tile(); static_cast<long long>(tile) * TW < n; tile = next_tile())
        {
            const int t0 = tile * TW;
            const int nvalid = static_cast<int>(min(static_cast<long long>(TW), static_cast<long long>(n) - t0));
            float2 npx[P], npy[P], npz[P], lim[P], ax[P], ay[P], az[P];     // negated positions
            float3 lo, hi;      // the box of run lane / 8
            unsigned runs = 0;  // the run of the lane's target h, in bits 4 h
            {
                float3 pos[H];
                int run[H];
                bool finite = true;
#pragma unroll
                for (int p = 0; p < P; ++p)
                {
                    float v[2][4];
#pragma unroll
                    for (int e = 0; e < 2; ++e)
                    {
                        const int h = 2 * p + e < H ? 2 * p + e : H - 1;
                        const int k = min(t0 + 32 * h + lane, n - 1);
                        const float4 pk = spm[k];
                        pos[h] = make_float3(pk.x, pk.y, pk.z);
                        finite = finite && isfinite(pk.x) && isfinite(pk.y) && isfinite(pk.z);
                        v[e][0] = -pk.x;
                        v[e][1] = -pk.y;
                        v[e][2] = -pk.z;
                        const float r = LAW == NBODY_LAW_CUTOFF ? srad[k] : 0.f;
                        v[e][3] = LAW == NBODY_LAW_CUTOFF ? r * r : eps2;
                    }
                    npx[p] = make_float2(v[0][0], v[1][0]);
                    npy[p] = make_float2(v[0][1], v[1][1]);
                    npz[p] = make_float2(v[0][2], v[1][2]);
                    lim[p] = make_float2(v[0][3], v[1][3]);
                    ax[p] = ay[p] = az[p] = make_float2(0.f, 0.f);
                }
                run_boxes<H, kRuns>(codes, t0, nvalid, lane, pos, lane >> 3, run, lo, hi);
                if (!__all_sync(0xffffffffu, finite))
                {
                    // min and max pass over a NaN: a box that decides nothing, so that every
                    // target decides for itself
                    lo = make_float3(-INFINITY, -INFINITY, -INFINITY);
                    hi = make_float3(INFINITY, INFINITY, INFINITY);
                }
#pragma unroll
                for (int h = 0; h < H; ++h)
                    runs |= static_cast<unsigned>(run[h]) << (4 * h);
            }
            // the lane's targets that opened the cell at hand, one bit per slot h; at first all, for
            // a parent of the root
            unsigned all = 0;
#pragma unroll
            for (int h = 0; h < H; ++h)
                all |= 32 * h + lane < nvalid ? 1u << h : 0u;
            unsigned mine = all;
            bool full = true;               // all of the warp's targets
            int sp = 0;
            int kid = 0, nchild = 1;        // the lane's child l % 8 of the cell at hand: at first the root
            int next = 0, last = -1;        // bodies of the bucket at hand (identical codes) still to come
            // Each cell is opened at most once, from its one parent (cells < n). The bound only
            // trips on a malformed tree: it records the error and ends this tile.
            int guard = 0;
            const int guard_limit = n + 64;
            for (;;)
            {
                // --- the children of the cell at hand ---
                // runs that are empty, or have no target among those that opened it, decide nothing
                bool idle = lo.x > hi.x;
                if (!full)
                {
                    unsigned active = 0;
#pragma unroll
                    for (int h = 0; h < H; ++h)
                        active |= (mine >> h) & 1u ? 1u << ((runs >> (4 * h)) & 7u) : 0u;
                    active = __reduce_or_sync(0xffffffffu, active);     // every lane's, idle or not
                    idle = idle || !((active >> (lane >> 3)) & 1u);
                }
                const bool has = (lane & 7) < nchild;
                float4 src = make_float4(0.f, 0.f, 0.f, 0.f);
                float open_r2 = 0.f;
                if (has)
                {
                    src = kid < 0 ? spm[~kid] : nodes[kid].com_mass;
                    open_r2 = kid < 0 ? 0.f : nodes[kid].open_r2;
                }
                const float ax0 = __fsub_rn(lo.x, src.x), ax1 = __fsub_rn(src.x, hi.x);
                const float ay0 = __fsub_rn(lo.y, src.y), ay1 = __fsub_rn(src.y, hi.y);
                const float az0 = __fsub_rn(lo.z, src.z), az1 = __fsub_rn(src.z, hi.z);
                const float near2 = dist2_rn(fmaxf(fmaxf(ax0, ax1), 0.f), fmaxf(fmaxf(ay0, ay1), 0.f),
                                             fmaxf(fmaxf(az0, az1), 0.f));
                const float far2 = dist2_rn(fmaxf(fabsf(ax0), fabsf(ax1)), fmaxf(fabsf(ay0), fabsf(ay1)),
                                            fmaxf(fabsf(az0), fabsf(az1)));
                unsigned beyond = __ballot_sync(0xffffffffu, idle || near2 > open_r2);
                unsigned within = __ballot_sync(0xffffffffu, idle || !(far2 > open_r2));
                unsigned cells = __ballot_sync(0xffffffffu, has && kid >= 0) & 0xffu;
                // a source that is not finite (or a target: its tile's boxes are not), by far2 of run
                // 0, which is never empty
                const bool odd = (__ballot_sync(0xffffffffu, !(far2 < INFINITY)) & 0xffu) != 0u;
                // massless nodes are skipped (bhtree.cpp:109-113)
                const unsigned mass = __ballot_sync(0xffffffffu, src.w != 0.f) & 0xffu;
                beyond &= beyond >> 16;
                beyond &= beyond >> 8;
                within &= within >> 16;
                within &= within >> 8;
                // the children that are applied, in the order of the sums: leaves, then cells taken
                // or tested
                const unsigned leaves = mass & ~cells;
                visits += static_cast<unsigned>(__popc(cells));
                cells &= mass;
                unsigned push = cells & within & ~beyond;
                const unsigned tested = cells & ~beyond & ~within;
                const unsigned applied = cells & ~push;
                const int nleaf = __popc(leaves), count = nleaf + __popc(applied);
                const unsigned below = (1u << (lane & 7)) - 1u;
                const int at = kid < 0 ? __popc(leaves & below) : nleaf + __popc(applied & below);
                if (lane < 8 && ((leaves | applied) >> lane) & 1u)
                    srcs[at] = src;
                __syncwarp();
                // who takes each of them: H bits per source, all who opened the parent unless tested
                Takes takes = static_cast<Takes>(mine) * TakeBits<H>::kOnes;
                Takes opens = 0;            // who opens each tested child
                for (unsigned t = tested; t; t &= t - 1)
                {
                    const int b = __ffs(t) - 1, e = __shfl_sync(0xffffffffu, at, b);
                    const float r2 = __shfl_sync(0xffffffffu, open_r2, b);
                    const float4 s = srcs[e];
                    unsigned take = 0;
                    if (H == 1)
                        take = dist2_rn(__fadd_rn(s.x, npx[0].x), __fadd_rn(s.y, npy[0].x), __fadd_rn(s.z, npz[0].x)) > r2
                                   ? 1u : 0u;
                    else
                    {
#pragma unroll
                        for (int p = 0; p < P; ++p)
                        {
                            // sq2 forms the squares so that none is contracted into the sum
                            const float2 dx = add2(f2(s.x), npx[p]), dy = add2(f2(s.y), npy[p]), dz = add2(f2(s.z), npz[p]);
                            const float2 ds = add2(add2(sq2(dx), sq2(dy)), sq2(dz));
                            take |= (ds.x > r2 ? 1u : 0u) << (2 * p) | (ds.y > r2 ? 2u : 0u) << (2 * p);
                        }
                    }
                    const unsigned rest = mine & ~take;
                    takes &= ~(static_cast<Takes>(rest) << (H * e));
                    opens |= static_cast<Takes>(rest) << (H * b);
                    push |= __any_sync(0xffffffffu, rest != 0u) ? 1u << b : 0u;
                }
                takes &= TakeBits<H>::first(count);
                inter += TakeBits<H>::count(takes);
                if (odd)
                {
                    // one target at a time: zero times an infinity, in the half of a pair that
                    // does not take the source, is not zero
                    for (int e = 0; e < count; ++e)
                    {
                        const float4 s = srcs[e];
#pragma unroll
                        for (int h = 0; h < H; ++h)
                            if ((takes >> (H * e + h)) & 1u)
                            {
                                const int p = h / 2;
                                apply<LAW>(-(h & 1 ? npx[p].y : npx[p].x), -(h & 1 ? npy[p].y : npy[p].x),
                                           -(h & 1 ? npz[p].y : npz[p].x), h & 1 ? lim[p].y : lim[p].x, s.x, s.y, s.z,
                                           s.w, true, h & 1 ? ax[p].y : ax[p].x, h & 1 ? ay[p].y : ay[p].x,
                                           h & 1 ? az[p].y : az[p].x);
                            }
                    }
                }
                else if (full && !tested)
                {
#pragma unroll 4
                    for (int e = 0; e < count; ++e)
                    {
                        const float4 s = srcs[e];
                        if (H == 1)
                            apply<LAW>(-npx[0].x, -npy[0].x, -npz[0].x, lim[0].x, s.x, s.y, s.z, s.w, true, ax[0].x,
                                       ay[0].x, az[0].x);
                        else
#pragma unroll
                            for (int p = 0; p < P; ++p)
                                apply2<LAW>(npx[p], npy[p], npz[p], lim[p], s.x, s.y, s.z, s.w, true, true, ax[p],
                                            ay[p], az[p]);
                    }
                }
                else
                {
                    // pair by pair: the lanes that take nothing with either target sit out the loop
#pragma unroll
                    for (int p = 0; p < P; ++p)
                    {
                        Takes t = takes >> (2 * p);
                        if (t & (H == 1 ? TakeBits<H>::kOnes : static_cast<Takes>(3 * TakeBits<H>::kOnes)))
#pragma unroll 4
                            for (int e = 0; e < count; ++e, t >>= H)
                            {
                                const float4 s = srcs[e];
                                if (H == 1)
                                    apply<LAW>(-npx[0].x, -npy[0].x, -npz[0].x, lim[0].x, s.x, s.y, s.z, s.w, t & 1u,
                                               ax[0].x, ay[0].x, az[0].x);
                                else
                                    apply2<LAW>(npx[p], npy[p], npz[p], lim[p], s.x, s.y, s.z, s.w, t & 1u, t & 2u,
                                                ax[p], ay[p], az[p]);
                            }
                    }
                }
                __syncwarp();               // the sources, and the entry popped last, have been read
                if (sp + 8 > kStack)
                {
                    if (lane == 0)
                        atomicOr(err, DEV_ERR_BOUNDS);
                    break;
                }
                for (unsigned t = push; t; t &= t - 1)
                {
                    const int b = __ffs(t) - 1;
                    const unsigned by = (tested >> b) & 1u ? static_cast<unsigned>(opens >> (H * b)) : mine;
                    stk_mine[warp][sp][lane] = static_cast<uint8_t>(by & ((1u << H) - 1u));
                    if (lane == b)
                        stk_cell[warp][sp] = kid;
                    ++sp;
                }
                __syncwarp();
                // --- the next cell to be opened, or eight more bodies of a bucket ---
                if (next > last)
                {
                    if (sp == 0)
                        break;
                    if (++guard > guard_limit)
                    {
                        if (lane == 0)
                            atomicOr(err, DEV_ERR_BOUNDS);
                        break;
                    }
                    --sp;
                    const OctNode* const node = nodes + stk_cell[warp][sp];
                    const int4 meta = *reinterpret_cast<const int4*>(&node->open_r2);   // open_r2, nchild, first, last
                    kid = node->child[lane & 7];
                    mine = stk_mine[warp][sp][lane];
                    full = __all_sync(0xffffffffu, mine == all);
                    nchild = meta.y;
                    if (nchild < 0)
                    {
                        next = meta.z;
                        last = meta.w;
                    }
                }
                if (next <= last)
                {
                    kid = ~(next + (lane & 7));
                    nchild = min(8, last - next + 1);
                    next += 8;
                }
            }
#pragma unroll
            for (int h = 0; h < H; ++h)
            {
                const int k = t0 + 32 * h + lane;
                if (k >= n)
                    continue;
                const uint32_t i = order[k];
                const float2 sx = ax[h / 2], sy = ay[h / 2], sz = az[h / 2];
                const float gx = G * (h & 1 ? sx.y : sx.x), gy = G * (h & 1 ? sy.y : sy.x), gz = G * (h & 1 ? sz.y : sz.x);
                if (body_out)
                {
                    float* o = body_out + static_cast<size_t>(i) * 12 + 8;
                    o[0] = gx;
                    o[1] = gy;
                    o[2] = gz;
                }
                else
                    acc[i] = make_float4(gx, gy, gz, 0.f);
            }
        }
        // per-warp totals
        unsigned long long total = inter;
        for (int o = 16; o > 0; o >>= 1)
            total += __shfl_down_sync(0xffffffffu, total, o);
        if (lane == 0)
        {
            atomicAdd(&stats[0], total);
            atomicAdd(&stats[1], static_cast<unsigned long long>(visits));
        }
    }

    // ------------------------------------------------------------------------------------
    // 7b. group walk with interaction lists (walk = NBODY_WALK_GROUP)
    // ------------------------------------------------------------------------------------
    // One list source applied to two targets (negated positions), both taking it: the direct
    // sum's packed interaction, 3 FADD2 + 3 FFMA2 + 2 MUFU.RSQ + 3 FMUL2 + 3 FFMA2.
    template <int LAW>
    __device__ __forceinline__ void apply_list2(const float2 npx, const float2 npy, const float2 npz, const float2 lim,
                                                const float4 s, float2& ax, float2& ay, float2& az)
    {
        const float2 dx = add2(f2(s.x), npx), dy = add2(f2(s.y), npy), dz = add2(f2(s.z), npz);
        float2 r2 = (LAW == NBODY_LAW_SOFTENED) ? fma2(dx, dx, lim) : mul2(dx, dx);
        r2 = fma2(dy, dy, r2);
        r2 = fma2(dz, dz, r2);
        float2 inv = make_float2(rsqrt_sfu(r2.x), rsqrt_sfu(r2.y));
        if (LAW == NBODY_LAW_CUTOFF)
        {
            inv.x = r2.x > lim.x ? inv.x : 0.f;     // physics.h:38-39
            inv.y = r2.y > lim.y ? inv.y : 0.f;
        }
        const float2 inv2 = mul2(inv, inv);
        const float2 mi = mul2(f2(s.w), inv);
        const float2 sc = mul2(mi, inv2);
        ax = fma2(dx, sc, ax);
        ay = fma2(dy, sc, ay);
        az = fma2(dz, sc, az);
    }

    // Loads that stay where they are written, ahead of the work that hides them.
    __device__ __forceinline__ int load_ahead(const int* p)
    {
        int v;
        asm volatile("ld.global.nc.s32 %0, [%1];" : "=r"(v) : "l"(p));
        return v;
    }

    __device__ __forceinline__ float4 load_ahead(const float4* p)
    {
        float4 v;
        asm volatile("ld.global.nc.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "l"(p));
        return v;
    }

    // The reference's opening test (bhtree.cpp:117-125) for a box of targets: the cell is
    // accepted when the nearest point of the box lies beyond its opening distance,
    // |com - p|^2 > size^2 * theta^2. Every target in the box is at least that far from the
    // centre of mass, so each would accept the cell itself.
    __device__ __forceinline__ bool box_accepts(const float4 cm, const float open_r2, const float4 lo, const float4 hi)
    {
        const float dx = fmaxf(fmaxf(lo.x - cm.x, cm.x - hi.x), 0.f);
        const float dy = fmaxf(fmaxf(lo.y - cm.y, cm.y - hi.y), 0.f);
        const float dz = fmaxf(fmaxf(lo.z - cm.z, cm.z - hi.z), 0.f);
        return fmaf(dz, dz, fmaf(dy, dy, dx * dx)) > open_r2;
    }

    // A warp serves 64 Q Morton-consecutive targets (lane l holds targets 64 Q t + 32 h + l,
    // h < 2Q, as Q packed pairs) with one walk of the tree, the interaction-list walk of GPU
    // tree codes (Barnes 1990's grouping; Bonsai, Bedorf et al. 2012): the walk decides each
    // cell once for the whole group and appends the sources it yields -- accepted cells as
    // (com, mass), leaves and the bodies of opened buckets as (x, m) -- to an interaction list
    // in shared memory, which every CAP entries is applied to every target of the group
    // with the direct sum's packed loop: no selection and no per-target test.
    //
    // The acceptance box. The group is split at the NSG - 1 largest jumps of its Morton codes
    // (the smallest common prefixes of neighbours) into runs, each with its own bounding box,
    // and a cell is accepted only when every run's box lies beyond its opening distance;
    // otherwise it is opened for the whole group. One box over the group would be wrong in
    // shape: a run that crosses from one cell of the tree into a distant one (at the end of a
    // top-level octant the curve jumps across the whole system) has a box spanning everything
    // between, which opens every cell there down to its leaves. Accepting per run instead
    // (some runs taking a cell, the others its children) was measured too: half the list then
    // applies to only some targets, and the walk took 54 against 45 ms at 16.8M bodies.
    //
    // The walk tests up to 32 cells at a time: it pops up to four opened parent cells from a
    // stack, and lane l tests child l % 8 of parent l / 8. The stack grows by at most 28
    // parents per tree level (22 levels: 616 < kGroupStack). A round's parents are popped before
    // the round ahead of it pushes its own, and its cells' records loaded before that one's
    // list is applied, so that only a nearly empty stack waits for its loads; while more than
    // kGroupAhead parents are stacked they are popped after the pushes, which bounds the stack
    // as before. The list's loop is FP32-pipe work (24 instructions a source and two pairs);
    // unrolled 16 times the pipe waits less between its iterations (2 times: 3 to 20 % longer).
    // Walk alone, before and now: 16.8M halo bodies, theta 2: 41.6 -> 37.8 ms; 1M: 2.62 -> 2.30;
    // two Plummer spheres of 131,072 bodies, theta 2: 797 -> 670 us; of 10,000, theta 0.5: 119 -> 78 us.
    //
    // Each target's sources refine the cells the reference's walk accepts for it alone (a
    // cell opened for the group may be one the target would have accepted), so each target
    // is summed at least as finely as in the reference, over more interactions.
    template <int LAW, int Q, int NSG, int CAP>
    __global__ void __launch_bounds__(kListWarps * 32, list_ctas(Q, CAP)) traverse_list_kernel(
        const OctNode* __restrict__ nodes, const float4* __restrict__ spm, const float* __restrict__ srad,
        const uint64_t* __restrict__ codes, const uint32_t* __restrict__ order, const int n, const float G,
        const float eps2, float4* __restrict__ acc, float* __restrict__ body_out, unsigned* __restrict__ err,
        unsigned long long* __restrict__ stats)
    {
        after_previous();
        constexpr int H = 2 * Q;                    // target slots per lane
        constexpr int TW = 32 * H;                  // targets per group
        static_assert(NSG >= 1 && NSG <= 32, "runs per group");
        __shared__ __align__(16) float4 list_mem[kListWarps][CAP];
        __shared__ int stack_mem[kListWarps][kGroupStack];
        __shared__ __align__(16) float4 box_mem[kListWarps][2 * NSG];
        const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
        const unsigned lt = (1u << lane) - 1u;
        float4* list = list_mem[warp];
        int* stk = stack_mem[warp];
        const float4* box = box_mem[warp];
        unsigned long long inter = 0;               // interactions summed by this warp (uniform)
        unsigned iters = 0;

        auto next_tile = [&]() {
            unsigned long long t = 0;
            if (lane == 0)
                t = atomicAdd(&stats[3], 1ull);
            return static_cast<int>(__shfl_sync(0xffffffffu, t, 0));
        };
        for (int tile = next_tile(); static_cast<long long>(tile) * TW < n; tile = next_tile())
        {
            const int t0 = tile * TW;
            const int nvalid = static_cast<int>(min(static_cast<long long>(TW), static_cast<long long>(n) - t0));
            // --- runs: split at the NSG - 1 largest Morton jumps between neighbours ---
            unsigned key[H];    // (common prefix bits << 8 | position); 0xffffffff: no boundary
#pragma unroll
            for (int h = 0; h < H; ++h)
            {
                const int b = 32 * h + lane;        // boundary between positions b - 1 and b
                key[h] = 0xffffffffu;
                if (b > 0 && b < nvalid)
                    key[h] = (static_cast<unsigned>(__clzll(static_cast<long long>(codes[t0 + b - 1] ^ codes[t0 + b])))
                              << 8) | static_cast<unsigned>(b);
            }
            int split[NSG > 1 ? NSG - 1 : 1];
            split[0] = TW;
#pragma unroll
            for (int sidx = 0; sidx < NSG - 1; ++sidx)
            {
                unsigned m = key[0];
#pragma unroll
                for (int h = 1; h < H; ++h)
                    m = min(m, key[h]);
                for (int o = 16; o > 0; o >>= 1)
                    m = min(m, __shfl_xor_sync(0xffffffffu, m, o));
                split[sidx] = m == 0xffffffffu ? TW : static_cast<int>(m & 0xffu);
#pragma unroll
                for (int h = 0; h < H; ++h)
                    if (key[h] == m)
                        key[h] = 0xffffffffu;
            }
            // --- targets and the run boxes ---
            float2 npx[Q], npy[Q], npz[Q], lim[Q], ax[Q], ay[Q], az[Q];
            float4 blo[NSG], bhi[NSG];
#pragma unroll
            for (int g = 0; g < NSG; ++g)
            {
                blo[g] = make_float4(INFINITY, INFINITY, INFINITY, 0.f);
                bhi[g] = make_float4(-INFINITY, -INFINITY, -INFINITY, 0.f);
            }
#pragma unroll
            for (int q = 0; q < Q; ++q)
            {
                float v[2][4];
#pragma unroll
                for (int e = 0; e < 2; ++e)
                {
                    const int pos = 32 * (2 * q + e) + lane;
                    const int k = t0 + pos;
                    const bool valid = k < n;
                    int run = 0;
#pragma unroll
                    for (int sidx = 0; sidx < NSG - 1; ++sidx)
                        run += pos >= split[sidx] ? 1 : 0;
                    const float4 pk = spm[valid ? k : n - 1];
#pragma unroll
                    for (int g = 0; g < NSG; ++g)
                        if (valid && run == g)
                        {
                            blo[g] = make_float4(fminf(blo[g].x, pk.x), fminf(blo[g].y, pk.y), fminf(blo[g].z, pk.z), 0.f);
                            bhi[g] = make_float4(fmaxf(bhi[g].x, pk.x), fmaxf(bhi[g].y, pk.y), fmaxf(bhi[g].z, pk.z), 0.f);
                        }
                    v[e][0] = -pk.x;
                    v[e][1] = -pk.y;
                    v[e][2] = -pk.z;
                    if (LAW == NBODY_LAW_CUTOFF)
                    {
                        const float r = srad[valid ? k : n - 1];
                        v[e][3] = r * r;
                    }
                    else
                        v[e][3] = eps2;
                }
                npx[q] = make_float2(v[0][0], v[1][0]);
                npy[q] = make_float2(v[0][1], v[1][1]);
                npz[q] = make_float2(v[0][2], v[1][2]);
                lim[q] = make_float2(v[0][3], v[1][3]);
                ax[q] = ay[q] = az[q] = make_float2(0.f, 0.f);
            }
#pragma unroll
            for (int g = 0; g < NSG; ++g)
                for (int o = 16; o > 0; o >>= 1)
                {
                    blo[g].x = fminf(blo[g].x, __shfl_xor_sync(0xffffffffu, blo[g].x, o));
                    blo[g].y = fminf(blo[g].y, __shfl_xor_sync(0xffffffffu, blo[g].y, o));
                    blo[g].z = fminf(blo[g].z, __shfl_xor_sync(0xffffffffu, blo[g].z, o));
                    bhi[g].x = fmaxf(bhi[g].x, __shfl_xor_sync(0xffffffffu, bhi[g].x, o));
                    bhi[g].y = fmaxf(bhi[g].y, __shfl_xor_sync(0xffffffffu, bhi[g].y, o));
                    bhi[g].z = fmaxf(bhi[g].z, __shfl_xor_sync(0xffffffffu, bhi[g].z, o));
                }
            __syncwarp();       // the previous group's readers of the boxes are done
            if (lane < 2 * NSG)
            {
                const int g = lane >> 1;
                float4 bv = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
                for (int gg = 0; gg < NSG; ++gg)
                    if (gg == g)
                        bv = (lane & 1) ? bhi[gg] : blo[gg];
                box_mem[warp][lane] = bv;
            }
            __syncwarp();

            int ln = 0;     // list entries (warp-uniform)
            // apply the whole list to every target of the group, then empty it
            auto drain = [&]() {
                __syncwarp();
#pragma unroll 16
                for (int e = 0; e < ln; ++e)
                {
                    const float4 s = list[e];
#pragma unroll
                    for (int q = 0; q < Q; ++q)
                        apply_list2<LAW>(npx[q], npy[q], npz[q], lim[q], s, ax[q], ay[q], az[q]);
                }
                inter += static_cast<unsigned long long>(ln) * nvalid;
                ln = 0;
                __syncwarp();
            };
            // append one source per flagged lane, draining first when the list would overflow
            auto append = [&](const bool take, const float4 src) {
                const unsigned m = __ballot_sync(0xffffffffu, take);
                if (ln + __popc(m) > CAP)
                    drain();
                if (take)
                    list[ln + __popc(m & lt)] = src;
                ln += __popc(m);
            };
            // the bodies of an opened bucket (identical codes), 32 at a time
            auto append_range = [&](const int first, const int last) {
                for (int b0 = first; b0 <= last; b0 += 32)
                {
                    const int bi = b0 + lane;
                    float4 sb = make_float4(0.f, 0.f, 0.f, 0.f);
                    if (bi <= last)
                        sb = spm[bi];
                    append(bi <= last && sb.w != 0.f, sb);
                }
            };
            // every run's box lies beyond the cell's opening distance (an empty run's box is
            // inverted, +inf to -inf, and accepts everything)
            auto accepts = [&](const float4 cm, const float open_r2) {
                bool a = true;
#pragma unroll
                for (int g = 0; g < NSG; ++g)
                    a = a && box_accepts(cm, open_r2, box[2 * g], box[2 * g + 1]);
                return a;
            };

            // the root: accepted, a bucket, or the first parent on the stack
            int sp = 0;
            {
                const float4 cm = nodes[0].com_mass;
                const int4 meta = *reinterpret_cast<const int4*>(&nodes[0].open_r2);
                if (cm.w != 0.f)
                {
                    if (accepts(cm, __int_as_float(meta.x)))
                        append(lane == 0, cm);
                    else if (meta.y < 0)
                        append_range(meta.z, meta.w);
                    else
                    {
                        if (lane == 0)
                            stk[0] = 0;
                        sp = 1;
                    }
                }
            }
            __syncwarp();
            // the lane's child of the next (up to four) parents off the stack; 0: none (cell 0 is
            // the root, never a child)
            auto pop = [&]() {
                const int slot = lane >> 3;
                const int c = slot < sp ? load_ahead(&nodes[stk[sp - 1 - slot]].child[lane & 7]) : 0;
                sp -= min(sp, 4);
                return c;
            };
            float4 src;             // a child's (com, mass), or a leaf's (x, m)
            float4 meta;            // a cell's open_r2, nchild, first, last
            auto load = [&](const int c) {
                src = make_float4(0.f, 0.f, 0.f, 0.f);
                meta = make_float4(0.f, 0.f, 0.f, 0.f);
                if (c < 0)
                    src = load_ahead(spm + ~c);
                else if (c > 0)
                {
                    src = load_ahead(&nodes[c].com_mass);
                    meta = load_ahead(reinterpret_cast<const float4*>(&nodes[c].open_r2));
                }
            };
            bool more = sp > 0;
            int c = more ? pop() : 0;
            load(c);
            // Each cell is pushed at most once per group, so the walk takes at most one
            // round per cell (< n); the bound only trips on a malformed tree.
            int guard = 0;
            const int guard_limit = n + 64;
            while (more)
            {
                if (++guard > guard_limit)
                {
                    if (lane == 0)
                        atomicOr(err, DEV_ERR_BOUNDS);
                    break;
                }
                ++iters;
                const bool ahead = sp > 0 && sp <= kGroupAhead;
                int cn = ahead ? pop() : 0;
                // empty cells are skipped (bhtree.cpp:109-113); a leaf is always applied
                // (bhtree.cpp:115-116)
                const bool cell = c > 0 && src.w != 0.f;
                const bool taken = cell && accepts(src, meta.x);
                const bool bucket = cell && !taken && __float_as_int(meta.y) < 0;
                const bool push = cell && !taken && !bucket;
                const bool take = c < 0 ? src.w != 0.f : taken;
                const float4 from = src;
                const int first = __float_as_int(meta.z), last = __float_as_int(meta.w);
                __syncwarp();           // every parent read before pushes overwrite its slot
                const unsigned pm = __ballot_sync(0xffffffffu, push);
                if (push)
                {
                    const int at = sp + __popc(pm & lt);
                    if (at < kGroupStack)
                        stk[at] = c;
                    else
                        atomicOr(err, DEV_ERR_BOUNDS);
                }
                sp = min(kGroupStack, sp + __popc(pm));
                __syncwarp();
                more = ahead || sp > 0;
                c = !ahead && more ? pop() : cn;
                load(c);
                append(take, from);
                unsigned bm = __ballot_sync(0xffffffffu, bucket);
                while (bm)
                {
                    const int bl = __ffs(bm) - 1;
                    bm &= bm - 1;
                    append_range(__shfl_sync(0xffffffffu, first, bl), __shfl_sync(0xffffffffu, last, bl));
                }
            }
            drain();
#pragma unroll
            for (int q = 0; q < Q; ++q)
#pragma unroll
                for (int e = 0; e < 2; ++e)
                {
                    const int k = t0 + (2 * q + e) * 32 + lane;
                    if (k >= n)
                        continue;
                    const uint32_t i = order[k];
                    const float gx = G * (e ? ax[q].y : ax[q].x), gy = G * (e ? ay[q].y : ay[q].x);
                    const float gz = G * (e ? az[q].y : az[q].x);
                    if (body_out)
                    {
                        float* o = body_out + static_cast<size_t>(i) * 12 + 8;
                        o[0] = gx;
                        o[1] = gy;
                        o[2] = gz;
                    }
                    else
                        acc[i] = make_float4(gx, gy, gz, 0.f);
                }
        }
        if (lane == 0)
        {
            atomicAdd(&stats[0], inter);
            atomicAdd(&stats[1], static_cast<unsigned long long>(iters));
        }
    }

    // ------------------------------------------------------------------------------------
    // host side
    // ------------------------------------------------------------------------------------
    namespace
    {
        template <typename T>
        cudaError_t grow(T** p, const size_t count, cudaStream_t s)
        {
            if (*p)
                cudaFreeAsync(*p, s);
            *p = nullptr;
            return cudaMallocAsync(reinterpret_cast<void**>(p), std::max<size_t>(count, 1) * sizeof(T), s);
        }

        // The words a build counts in: statistics, the numbering's ticket and a word per tile.
        size_t count_bytes(const size_t n)
        {
            const size_t words = kStatsWords + 1 + (n + kNumTile - 1) / kNumTile;
            return (words + 1) / 2 * 16;
        }

        int reserve_bh(nbody_cuda* ctx, const size_t n)
        {
            if (!ctx->bh)
                ctx->bh = new BhState();
            BhState& b = *ctx->bh;
            if (!b.small_ready)
            {
                cudaError_t e = grow(&b.box, 1, ctx->stream);
                if (e == cudaSuccess)
                    e = grow(&b.bbox_part, kBboxBlocks * kBboxVals, ctx->stream);
                if (e == cudaSuccess)
                    e = grow(&b.box_ticket, 1, ctx->stream);
                if (e == cudaSuccess)
                    e = cudaMemsetAsync(b.box_ticket, 0, sizeof(unsigned), ctx->stream);
                if (e != cudaSuccess)
                    return ctx_cuda_fail(ctx, e, "tree allocation");
                b.small_ready = true;
            }
            if (!b.sort.sms)
                if (const cudaError_t e = setup_sort(&b.sort))
                    return ctx_cuda_fail(ctx, e, "radix sort set-up");
            if (n <= b.cap)
                return NBODY_OK;
            if (const int st = before_allocation(ctx))
                return st;
            const size_t cap = std::max(n, b.cap + b.cap / 2);
            const size_t tiles = (cap + kMomTile - 1) / kMomTile;
            // the sort's temporaries; later the cell sums' tile totals and tile prefixes, and a
            // tree export's scan
            const size_t tb = std::max({ sort_temp_bytes(cap), 2 * (tiles + 1) * sizeof(Int64x4),
                                         scan_temp_elems(cap) * sizeof(uint32_t) });
            cudaError_t e = cudaSuccess;
            cudaStream_t s = ctx->stream;
            // the last tree goes with its buffers, also when not all of the new ones can be had
            b.built = false;
            for (int k = 0; k < 2 && e == cudaSuccess; ++k)
            {
                e = grow(&b.keys[k], cap, s);
                if (e == cudaSuccess)
                    e = grow(&b.vals[k], cap, s);
            }
            if (e == cudaSuccess && fault_injected("tree"))
                e = cudaErrorMemoryAllocation;
            if (e == cudaSuccess) e = grow(&b.spm, cap, s);
            if (e == cudaSuccess) e = grow(&b.srad, cap, s);
            if (e == cudaSuccess) e = grow(&b.child, cap, s);
            if (e == cudaSuccess) e = grow(&b.range, cap, s);
            if (e == cudaSuccess) e = grow(&b.prefix, cap, s);
            if (e == cudaSuccess) e = grow(&b.octflag, cap, s);
            if (e == cudaSuccess) e = grow(&b.octidx, cap, s);
            // the statistics, then the numbering's ticket and tile counts: zeroed together
            if (e == cudaSuccess) e = grow(&b.stats, count_bytes(cap) / sizeof(unsigned long long), s);
            b.numbering = reinterpret_cast<uint64_t*>(b.stats) + kStatsWords;
            if (e == cudaSuccess) e = grow(&b.psum, cap + 1, s);
            if (e == cudaSuccess) e = grow(&b.nodes, cap, s);
            if (e == cudaSuccess)
            {
                if (b.temp)
                    cudaFreeAsync(b.temp, s);
                b.temp = nullptr;
                e = cudaMallocAsync(&b.temp, tb, s);
                b.temp_bytes = tb;
            }
            if (e != cudaSuccess)
            {
                b.cap = 0;
                return ctx_cuda_fail(ctx, e, "tree allocation");
            }
            b.cap = cap;
            return NBODY_OK;
        }

        const float4* body_src(const nbody_cuda* ctx, int* stride)
        {
            if (ctx->layout == NBODY_LAYOUT_AOS)
            {
                *stride = 3;
                return reinterpret_cast<const float4*>(ctx->bodies);
            }
            *stride = 1;
            return ctx->pm;
        }
    }

    // Launches overlap with the end of the kernel before (launch_after) for up to 2^19 bodies (an
    // eager build of 262,144 went from 163 to 147 us; of a million, whose kernels fill the GPU,
    // from 256 to 265), and not in a captured graph: replays of its linear chain were slower so
    // (a step of 65,536 bodies 178 against 155 us).
    static bool launch_early(cudaStream_t s, const size_t n)
    {
        if (n > (1u << 19))
            return false;
        cudaStreamCaptureStatus capture = cudaStreamCaptureStatusNone;
        return cudaStreamIsCapturing(s, &capture) == cudaSuccess && capture == cudaStreamCaptureStatusNone;
    }

    int bh_build(nbody_cuda* ctx, const nbody_step_params* p)
    {
        const size_t n = ctx->count;
        if (const int st = reserve_bh(ctx, n))
            return st;
        BhState& b = *ctx->bh;
        b.built = false;    // until all that makes a tree is launched
        cudaStream_t s = ctx->stream;
        int stride = 1;
        const float4* src = body_src(ctx, &stride);
        const int ni = static_cast<int>(n);
        uint64_t& L = ctx->launches;

        const bool early = launch_early(s, n);
        // tree_box = 0 is the reference's fixed root box; it needs a positive size
        const bool auto_box = p->tree_box != 0 || !(p->size > 0.f);
        // the bounds pass runs for the fixed box too: the cell sums' scale comes from it
        launch_after(early, bbox_kernel, std::min<unsigned>(kBboxBlocks, std::max(1u, ceil_div(n, 1024))), 256, 0, s,
                     src, stride, ni, auto_box ? 1 : 0, p->size, b.bbox_part, b.box_ticket,
                     reinterpret_cast<uint4*>(b.stats), count_bytes(n) / 16, static_cast<uint4*>(b.temp),
                     sort_zero_bytes(n) / 16, b.box);
        ++L;
        launch_after(early, morton_kernel, ceil_div(n, 256 * kMortonItems), 256, 0, s, src, stride, ni, b.box, b.keys[0], b.vals[0]);
        ++L;
        bool in_alt = false;
        cudaError_t e = radix_sort_pairs(b.keys[0], b.vals[0], b.keys[1], b.vals[1], n, kRunShift, 63, b.temp, s, &L,
                                         &in_alt, ctx->dev_error, early, b.sort);
        if (e != cudaSuccess)
            return ctx_cuda_fail(ctx, e, "radix sort");
        if (n > 1)
        {
            // runs of equal top bits into order; a run too long for that sorts everything
            // again by all bits, from the current order (its ties are in index order too)
            const int cur = in_alt ? 1 : 0;
            unsigned* full = reinterpret_cast<unsigned*>(b.stats + 4);
            launch_after(early, run_sort_kernel, ceil_div(n, 256), 256, 0, s, b.keys[cur], b.vals[cur], ni, full);
            ++L;
            e = radix_sort_if(b.keys[cur], b.vals[cur], b.keys[1 - cur], b.vals[1 - cur], n, 0, 63, b.temp,
                              (63 - kRunShift + 8) / 9, s, &L, ctx->dev_error, full, b.sort);
            if (e != cudaSuccess)
                return ctx_cuda_fail(ctx, e, "radix sort");
        }
        const uint64_t* keys = b.keys[in_alt ? 1 : 0];
        const uint32_t* order = b.vals[in_alt ? 1 : 0];
        b.order = order;
        b.codes = keys;
        const unsigned tiles = std::max(1u, ceil_div(n, kMomTile));
        // temporaries: tile totals and their exclusive scan (tiles + 1 each: the entry past
        // the last tile gives the sum of all bodies)
        Int64x4* tile_sum = static_cast<Int64x4*>(b.temp);
        Int64x4* tile_prefix = tile_sum + tiles + 1;
        // adjacent prefix lengths and key samples live in the sort's other key buffer, free until
        // the next build
        const int other = in_alt ? 0 : 1;
        uint8_t* dl = reinterpret_cast<uint8_t*>(b.keys[other]);
        // (n rounded up to 8 bytes, then n / 64 + 1 keys: within the buffer's 8 n bytes for n >= 2)
        uint64_t* smp = reinterpret_cast<uint64_t*>(dl + ((n + 7) & ~size_t(7)));
        const bool radius = p->law == NBODY_LAW_CUTOFF;
        launch_after(early, gather_sum_kernel, tiles, kMomThreads, 0, s, src, stride,
                     radius && ctx->layout != NBODY_LAYOUT_AOS ? ctx->vr : nullptr, order, ni, b.box, b.spm,
                     radius ? b.srad : nullptr, b.psum, tile_sum, keys, dl, smp);
        ++L;
        if (n < 2)
        {
            e = cudaGetLastError();
            if (e != cudaSuccess)
                return ctx_cuda_fail(ctx, e, "tree build");
            b.built = true;
            b.built_n = n;
            ++b.build_id;
            return NBODY_OK;
        }
        const int m = ni - 1;
        launch_after(early, radix_tree_kernel, 1 + ceil_div(m, 256), 256, 0, s, keys, dl, smp, ni, b.child, b.range,
                     b.prefix, b.octflag, tile_sum, tile_prefix, static_cast<int>(tiles) + 1, ctx->dev_error);
        ++L;
        launch_after(early, number_kernel, ceil_div(m, kNumTile), 1024, 0, s, b.octflag, m, b.octidx, b.numbering, ctx->dev_error);
        ++L;
        launch_after(early, octnode_kernel, ceil_div(m, 256 * kOctSpan), 256, 0, s, b.child, b.range, b.prefix, b.octidx,
                     b.psum, tile_prefix, m, b.box, p->theta, b.nodes, ctx->dev_error, b.stats);
        ++L;
        e = cudaGetLastError();
        if (e != cudaSuccess)
            return ctx_cuda_fail(ctx, e, "tree build");
        b.built = true;
        b.built_n = n;
        ++b.build_id;
        return NBODY_OK;
    }

    int bh_accelerate(nbody_cuda* ctx, const nbody_step_params* p)
    {
        const size_t n = ctx->count;
        if (!ctx->bh)
            ctx->bh = new BhState();
        // stage timing: three events on the stream, except while it is captured into a graph
        cudaStreamCaptureStatus capture = cudaStreamCaptureStatusNone;
        bool timed = cudaStreamIsCapturing(ctx->stream, &capture) == cudaSuccess && capture == cudaStreamCaptureStatusNone;
        const bool early = launch_early(ctx->stream, n);
        for (int k = 0; k < 3 && timed; ++k)
            timed = ctx->bh->ev[k] || cudaEventCreate(&ctx->bh->ev[k]) == cudaSuccess;
        ctx->bh->timed = false;
        if (timed)
            cudaEventRecord(ctx->bh->ev[0], ctx->stream);
        if (const int st = bh_build(ctx, p))
            return st;
        BhState& b = *ctx->bh;
        cudaStream_t s = ctx->stream;
        if (timed)
            cudaEventRecord(b.ev[1], s);
        const int ni = static_cast<int>(n);
        float4* acc = ctx->layout == NBODY_LAYOUT_AOS ? nullptr : ctx->acc;
        float* body_out = ctx->layout == NBODY_LAYOUT_AOS ? ctx->bodies : nullptr;
        if (n < 2)
        {
            // a lone body feels nothing (its own leaf is cut off / multiplied by d = 0)
            cudaError_t me = cudaSuccess;
            if (acc)
                me = cudaMemsetAsync(acc, 0, n * sizeof(float4), s);
            else
                for (size_t i = 0; i < n && me == cudaSuccess; ++i)
                    me = cudaMemsetAsync(body_out + i * 12 + 8, 0, 3 * sizeof(float), s);
            return me == cudaSuccess ? NBODY_OK : ctx_cuda_fail(ctx, me, "lone-body acceleration");
        }
        int sms = 0;
        cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, ctx->device);
        if (p->walk == NBODY_WALK_GROUP)
        {
            // Group walk: 128 targets per group (4 per lane) while the groups outnumber the
            // warps of six CTAs an SM (five under the cutoff law), else 64. NBODY_CUDA_BH_GROUP (64,
            // 128 or 256) overrides; the group size changes which cells each target applies, not the
            // bar they meet, so the line is fixed and does not follow the kernels' occupancy.
            const bool soft = p->law == NBODY_LAW_SOFTENED;
            using Walk = void (*)(const OctNode*, const float4*, const float*, const uint64_t*, const uint32_t*, int,
                                  float, float, float4*, float*, unsigned*, unsigned long long*);
            // [group 64, 128, 256][short, long list]
            const Walk fns[3][2] = {
                { soft ? traverse_list_kernel<NBODY_LAW_SOFTENED, 1, kRuns, kListShort>
                       : traverse_list_kernel<NBODY_LAW_CUTOFF, 1, kRuns, kListShort>,
                  soft ? traverse_list_kernel<NBODY_LAW_SOFTENED, 1, kRuns, kListLong>
                       : traverse_list_kernel<NBODY_LAW_CUTOFF, 1, kRuns, kListLong> },
                { soft ? traverse_list_kernel<NBODY_LAW_SOFTENED, 2, kRuns, kListShort>
                       : traverse_list_kernel<NBODY_LAW_CUTOFF, 2, kRuns, kListShort>,
                  soft ? traverse_list_kernel<NBODY_LAW_SOFTENED, 2, kRuns, kListLong>
                       : traverse_list_kernel<NBODY_LAW_CUTOFF, 2, kRuns, kListLong> },
                { soft ? traverse_list_kernel<NBODY_LAW_SOFTENED, 4, kRuns, kListShort>
                       : traverse_list_kernel<NBODY_LAW_CUTOFF, 4, kRuns, kListShort>,
                  soft ? traverse_list_kernel<NBODY_LAW_SOFTENED, 4, kRuns, kListLong>
                       : traverse_list_kernel<NBODY_LAW_CUTOFF, 4, kRuns, kListLong> } };
            auto per_sm = [&](Walk fn) {
                int per = 0;
                if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, fn, kListWarps * 32, 0) != cudaSuccess || per < 1)
                    per = 1;
                return per;
            };
            const char* gsel = std::getenv("NBODY_CUDA_BH_GROUP");
            int group = gsel ? std::atoi(gsel) : 0;
            if (group != 64 && group != 128 && group != 256)
                group = static_cast<long long>(ni) >= 128LL * (soft ? 6 : 5) * sms * kListWarps ? 128 : 64;
            const int gi = group == 256 ? 2 : (group == 128 ? 1 : 0);
            const int groups = (ni + group - 1) / group;
            // the long list once the groups are at least twice the warps it leaves resident
            const bool long_list = groups >= 2LL * per_sm(fns[gi][1]) * sms * kListWarps;
            const Walk fn = fns[gi][long_list ? 1 : 0];
            const int per = per_sm(fn);
            const int grid = std::min((groups + kListWarps - 1) / kListWarps, sms * per);
            launch_after(early, fn, grid, kListWarps * 32, 0, s, b.nodes, b.spm, b.srad, b.codes, b.order, ni, p->G, p->eps2, acc,
                                                body_out, ctx->dev_error, b.stats);
            ++ctx->launches;
            if (timed)
                b.timed = cudaEventRecord(b.ev[2], s) == cudaSuccess;
            const cudaError_t eg = cudaGetLastError();
            return eg == cudaSuccess ? NBODY_OK : ctx_cuda_fail(ctx, eg, "group tree walk");
        }
        // Targets per warp: 128 once there are three such tiles a resident warp, 64 once there is
        // one, else 32. A wider walk opens fewer cells in all but leaves fewer tiles to balance,
        // and each takes longer. Walk in ms at 32 / 64 / 128 targets: 20,000 bodies (two Plummer
        // spheres), theta 2: 0.49 / 0.74 / 1.09; 262,144: 1.63 / 1.51 / 1.62, theta 0.5: 0.088 /
        // 0.090 / 0.117; 1M disk, theta 0.5: 0.213 / 0.197 / 0.244; 4M disk + halo, theta 2:
        // 24.9 / 17.6 / 16.8. Where targets have many cells (theta from 1.25) 64 already when 32
        // would take two tiles a resident warp: 262,144 at theta 1.33 / 2, 32 against 64: disk
        // 0.534 / 0.965 and 0.490 / 0.864, disk + halo 0.725 / 1.712 and 0.692 / 1.593, uniform
        // cube 0.461 / 1.049 and 0.479 / 1.057; at theta 1 the disk 0.391 and 0.387, the cube 0.295
        // and 0.322. NBODY_CUDA_BH_TARGETS (32, 64, 128 or 256) overrides; all give the same sums.
        const char* tsel = std::getenv("NBODY_CUDA_BH_TARGETS");
        const int per_warp = tsel ? std::atoi(tsel) : 0;
        const bool soft = p->law == NBODY_LAW_SOFTENED;
        using Walk = void (*)(const OctNode*, const float4*, const float*, const uint64_t*, const uint32_t*, int,
                              float, float, float4*, float*, unsigned*, unsigned long long*);
        // targets per warp 32, 64, 128, 256
        const Walk fns[4] = {
            soft ? traverse_kernel<NBODY_LAW_SOFTENED, 1> : traverse_kernel<NBODY_LAW_CUTOFF, 1>,
            soft ? traverse_kernel<NBODY_LAW_SOFTENED, 2> : traverse_kernel<NBODY_LAW_CUTOFF, 2>,
            soft ? traverse_kernel<NBODY_LAW_SOFTENED, 4> : traverse_kernel<NBODY_LAW_CUTOFF, 4>,
            soft ? traverse_kernel<NBODY_LAW_SOFTENED, 8> : traverse_kernel<NBODY_LAW_CUTOFF, 8>,
        };
        auto per_sm = [&](const int i) {
            int per = 0;
            if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, fns[i], trav_warps(1 << i) * 32, 0) != cudaSuccess || per < 1)
                per = 1;
            return per;
        };
        int fi = 0;
        while (fi < 3 && per_warp > (32 << fi))
            ++fi;
        if (!per_warp)
        {
            auto resident = [&](const int i) { return static_cast<long long>(per_sm(i)) * sms * trav_warps(1 << i); };
            const bool wide = ni >= 64 * resident(1) || (p->theta >= 1.25f && ni >= 2 * 32 * resident(0));
            fi = ni >= 3 * 128 * resident(2) ? 2 : (wide ? 1 : 0);
        }
        // one resident wave of CTAs, each warp drawing tiles until none are left
        const int warps = trav_warps(1 << fi);
        const int tiles = (ni + (32 << fi) - 1) / (32 << fi);
        const int grid = std::min((tiles + warps - 1) / warps, sms * per_sm(fi));
        launch_after(early, fns[fi], grid, warps * 32, 0, s, b.nodes, b.spm, b.srad, b.codes, b.order, ni, p->G, p->eps2, acc, body_out,
                                            ctx->dev_error, b.stats);
        ++ctx->launches;
        if (timed)
            b.timed = cudaEventRecord(b.ev[2], s) == cudaSuccess;
        const cudaError_t e = cudaGetLastError();
        if (e != cudaSuccess)
            return ctx_cuda_fail(ctx, e, "tree traversal");
        return NBODY_OK;
    }

    int bh_stage_ms(nbody_cuda* ctx, float ms[2])
    {
        if (!ctx->bh || !ctx->bh->timed)
            return ctx_fail(ctx, NBODY_ERR_INVALID, "no timed Barnes-Hut accelerate");
        BhState& b = *ctx->bh;
        cudaError_t e = cudaEventSynchronize(b.ev[2]);
        if (e == cudaSuccess)
            e = cudaEventElapsedTime(&ms[0], b.ev[0], b.ev[1]);
        if (e == cudaSuccess)
            e = cudaEventElapsedTime(&ms[1], b.ev[1], b.ev[2]);
        if (e != cudaSuccess)
            return ctx_cuda_fail(ctx, e, "stage timing");
        return check_device_error(ctx);
    }

    void release_bh(nbody_cuda* ctx)
    {
        if (!ctx->bh)
            return;
        BhState& b = *ctx->bh;
        for (int k = 0; k < 2; ++k)
        {
            cudaFree(b.keys[k]);
            cudaFree(b.vals[k]);
        }
        void* ptrs[] = { b.spm, b.srad, b.child, b.range, b.prefix, b.octflag, b.octidx, b.psum,
                         b.nodes, b.temp, b.box, b.bbox_part, b.box_ticket, b.stats };
        for (void* q : ptrs)
            cudaFree(q);
        for (cudaEvent_t ev : b.ev)
            if (ev)
                cudaEventDestroy(ev);
        delete ctx->bh;
        ctx->bh = nullptr;
    }

    int bh_stats(nbody_cuda* ctx, unsigned long long out[3])
    {
        if (!ctx->bh || !ctx->bh->stats)
        {
            out[0] = out[1] = out[2] = 0;
            return NBODY_OK;
        }
        const cudaError_t e = cudaMemcpyAsync(out, ctx->bh->stats, 3 * sizeof(unsigned long long),
                                              cudaMemcpyDeviceToHost, ctx->stream);
        if (e != cudaSuccess)
            return ctx_cuda_fail(ctx, e, "tree statistics readback");
        return check_device_error(ctx);
    }

    uint64_t bh_build_id(const nbody_cuda* ctx)
    {
        return ctx->bh ? ctx->bh->build_id : 0;
    }

    int bh_view(nbody_cuda* ctx, TreeView* out)
    {
        if (!ctx->bh || !ctx->bh->built)
            return ctx_fail(ctx, NBODY_ERR_INVALID, "no Barnes-Hut tree has been built");
        BhState& b = *ctx->bh;
        *out = TreeView{ static_cast<int>(b.built_n), b.build_id, b.nodes, b.codes, b.spm, b.box, &b.stats[2],
                         { b.octidx, reinterpret_cast<uint32_t*>(b.prefix), reinterpret_cast<uint32_t*>(b.child) },
                         b.temp };
        return NBODY_OK;
    }

    int bh_morton(nbody_cuda* ctx, const nbody_step_params* p, uint64_t* codes, uint32_t* order, double box[4])
    {
        if (!ctx->count)
            return NBODY_OK;
        if (const int st = bh_build(ctx, p))
            return st;
        BhState& b = *ctx->bh;
        const size_t n = ctx->count;
        cudaError_t e = cudaSuccess;
        if (codes)
            e = cudaMemcpyAsync(codes, b.codes, n * sizeof(uint64_t), cudaMemcpyDeviceToHost, ctx->stream);
        if (e == cudaSuccess && order)
            e = cudaMemcpyAsync(order, b.order, n * sizeof(uint32_t), cudaMemcpyDeviceToHost, ctx->stream);
        BoxParams hb;
        if (e == cudaSuccess)
            e = cudaMemcpyAsync(&hb, b.box, sizeof hb, cudaMemcpyDeviceToHost, ctx->stream);
        if (e != cudaSuccess)
            return ctx_cuda_fail(ctx, e, "Morton readback");
        if (const int st = check_device_error(ctx))
            return st;
        if (box)
        {
            box[0] = hb.lo[0];
            box[1] = hb.lo[1];
            box[2] = hb.lo[2];
            box[3] = hb.edge;
        }
        return NBODY_OK;
    }
}
