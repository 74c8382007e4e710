// lbvh.cu -- on-device LBVH build, node-for-node identical to the reference's
// CPU build (LuminaGI-CudaRef src/bvh.cpp:164-211).
//
// Why a radix tree reproduces the reference.  build_recursive (bvh.cpp:75-120)
// splits a range of Morton-sorted triangles at the highest bit in which the
// range's codes differ (find_split is a binary search for that bit), stops at
// <= 4 triangles or when all codes in the range are equal, and numbers the
// nodes breadth-first afterwards (relayout_bfs, bvh.cpp:122-162).  The binary
// radix tree over the sorted codes, with duplicate codes made distinct by
// their sorted position (Karras 2012), contains every one of those ranges as
// a node, split the same way.  The reference tree is that radix tree cut off
// below every node whose range has <= 4 triangles or one distinct code:
//   kept(node)      = node is the root, or its parent is not collapsed
//   collapsed(node) = size <= 4 or code[first] == code[last]
// Breadth-first order with left before right is the order of (depth, first
// triangle), so the BFS index is the rank of that key.  Bounding boxes are
// refitted bottom-up; a leaf box scans its triangles in order and a parent
// box starts from the left child and widens by the right child, with the
// reference's strict < / > updates, so the float bits (signed zeros
// included) are the reference's.
//
// Kernels (15 to 17 device operations): scene bounds and centroids; Morton codes and the digit counts of
// the sort; four sort passes; the radix tree, by gap; node depths and counts
// per depth; the counts' scan; BFS indices; one kernel that moves the
// triangles into order, fits the leaf boxes from its shared-memory copy of
// their vertices and refits the nodes whose range lies within the block's 512
// triangles; and the nodes above those, 32 blocks' tops at a time.
//
// A radix-tree node is named by its gap g, the place between sorted triangles
// g and g + 1 where its range splits; the leaf of triangle k is named k.  The
// tree is the Cartesian tree of the gaps' common-prefix lengths: a node's
// parent is whichever of the two gaps just outside its range has the longer
// prefix, so every thread finds its own node's range and parent from the
// codes alone.
//
// What bounds it: 1,050,972 triangles move 244 MB at least (38 us at the copy
// rate); below 100,000 triangles the chain of dependent launches.  One B200,
// lg_build_bvh_device with permutation and triangles, wall time: 339 us for
// 1,050,972 triangles and 95 us for 20,500.  It was 795 and 347 us with a
// second four-pass sort for the BFS order, the refit through L2 at every level
// and one warp per moved triangle (36 operations).
#include <algorithm>
#include <cstdint>
#include <cstring>
#include <mutex>
#include <vector>

#include <cuda_runtime.h>

#include "common.h"
#include "lbvh.cuh"
#include "pdl.cuh"
#include "radix_sort.cuh"

namespace lg
{
namespace
{
constexpr int kTB = 256;

constexpr int kFirstBits = 26;    // up to 2^26 triangles

inline size_t align256(size_t b) { return (b + 255) & ~(size_t)255; }
inline int blocks_for(size_t n, int tb = kTB) { return (int)((n + tb - 1) / tb); }

// Total order key for "first occurrence of the minimum": value (with -0 and
// +0 equal, NaN excluded) in the high word, position in the low word.
__device__ __forceinline__ uint64_t min_key(float f, uint32_t pos)
{
    if (f != f) return ~0ull;  // NaN never wins
    uint32_t u = __float_as_uint(f == 0.0f ? 0.0f : f);
    u = (u & 0x80000000u) ? ~u : (u | 0x80000000u);
    return ((uint64_t)u << 32) | pos;
}
// For the maximum, larger value wins and, among equal values, the smaller position.
__device__ __forceinline__ uint64_t max_key(float f, uint32_t pos)
{
    if (f != f) return 0ull;
    uint32_t u = __float_as_uint(f == 0.0f ? 0.0f : f);
    u = (u & 0x80000000u) ? ~u : (u | 0x80000000u);
    return ((uint64_t)u << 32) | (0xFFFFFFFFu - pos);
}

__device__ __forceinline__ uint64_t warp_max_u64(uint64_t v)
{
    for (int o = 16; o; o >>= 1)
    {
        uint64_t w = __shfl_xor_sync(0xffffffffu, v, o);
        v = w > v ? w : v;
    }
    return v;
}

// bvh.cpp:170-173 -- scene box over every vertex in input order, and the
// centroids (bvh.cpp:185-187, each operation rounded by itself), so the code
// kernel reads 12 bytes a triangle instead of the records again.
// keys[0..2] = largest ~min_key, keys[3..5] = largest max_key (all cleared to
// 0).  The last block to finish turns the winning keys back into the vertex
// values and the normalisation extent (bvh.cpp:176-178: ext <= 0 -> 1):
// box[0..2] = min, box[3..5] = ext.
__global__ void __launch_bounds__(kTB) bounds_kernel(const lg_triangle* __restrict__ tris, int n,
                                                     unsigned long long* keys, unsigned* ticket,
                                                     float* __restrict__ centroids, float* __restrict__ box)
{
    begin_after_predecessors();
    const float third = 1.0f / 3.0f;
    uint64_t mn[3] = {~0ull, ~0ull, ~0ull}, mx[3] = {0, 0, 0};
    for (int t = blockIdx.x * kTB + threadIdx.x; t < n; t += gridDim.x * kTB)
    {
        const lg_triangle& tr = tris[t];
#pragma unroll
        for (int a = 0; a < 3; ++a)
        {
#pragma unroll
            for (int k = 0; k < 3; ++k)
            {
                const uint32_t pos = (uint32_t)t * 3u + (uint32_t)k;
                const float f = tr.v[k][a];
                const uint64_t a0 = min_key(f, pos), a1 = max_key(f, pos);
                mn[a] = a0 < mn[a] ? a0 : mn[a];
                mx[a] = a1 > mx[a] ? a1 : mx[a];
            }
            centroids[3 * (size_t)t + a] = __fmul_rn(__fadd_rn(__fadd_rn(tr.v[0][a], tr.v[1][a]), tr.v[2][a]), third);
        }
    }
    __shared__ uint64_t s[6][kTB / 32];
    __shared__ bool last;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
    for (int a = 0; a < 3; ++a)
    {
        const uint64_t x = warp_max_u64(~mn[a]);
        const uint64_t y = warp_max_u64(mx[a]);
        if (lane == 0) { s[a][warp] = x; s[3 + a][warp] = y; }
    }
    __syncthreads();
    if (threadIdx.x < 6)
    {
        uint64_t v = s[threadIdx.x][0];
        for (int w = 1; w < kTB / 32; ++w) v = s[threadIdx.x][w] > v ? s[threadIdx.x][w] : v;
        atomicMax(&keys[threadIdx.x], (unsigned long long)v);
        __threadfence();
    }
    __syncthreads();
    if (threadIdx.x == 0) last = atomicAdd(ticket, 1u) == gridDim.x - 1;
    __syncthreads();
    if (!last || threadIdx.x >= 3) return;
    __threadfence();
    const int a = threadIdx.x;
    const uint64_t k = ~(uint64_t)__ldcg(&keys[a]), m = __ldcg(&keys[3 + a]);
    float lo = __int_as_float(0x7f800000), hi = __int_as_float(0xff800000);
    if (k != ~0ull)
    {
        const uint32_t pos = (uint32_t)(k & 0xFFFFFFFFu);
        lo = tris[pos / 3].v[pos % 3][a];
    }
    if (m != 0ull)
    {
        const uint32_t pos = 0xFFFFFFFFu - (uint32_t)(m & 0xFFFFFFFFu);
        hi = tris[pos / 3].v[pos % 3][a];
    }
    float e = __fsub_rn(hi, lo);
    if (e <= 0.0f) e = 1.0f;
    box[a] = lo;
    box[3 + a] = e;
}

__device__ __forceinline__ uint32_t spread3(uint32_t v)
{
    v = (v | (v << 16)) & 0x030000FFu;
    v = (v | (v << 8)) & 0x0300F00Fu;
    v = (v | (v << 4)) & 0x030C30C3u;
    v = (v | (v << 2)) & 0x09249249u;
    return v;
}
// bvh.cpp:23-32 quantiser: clamp(f * 1024, 0, 1023) then truncate.
__device__ __forceinline__ uint32_t quant10(float f)
{
    f = __fmul_rn(f, 1024.0f);
    if (f < 0.0f) f = 0.0f;
    if (f > 1023.0f) f = 1023.0f;
    return __float2uint_rz(f);
}

// bvh.cpp:188-191 with every operation rounded individually (no FMA), and the
// digit counts of the four 8-bit sort passes.
__global__ void __launch_bounds__(kTB) morton_kernel(const float* __restrict__ centroids, int n,
                                                     const float* __restrict__ box, uint32_t* __restrict__ codes,
                                                     uint32_t* __restrict__ hist)
{
    begin_after_predecessors();
    __shared__ uint32_t h[4][256];
    for (int i = threadIdx.x; i < 4 * 256; i += kTB) (&h[0][0])[i] = 0;
    __syncthreads();
    for (int t = blockIdx.x * kTB + threadIdx.x; t < n; t += gridDim.x * kTB)
    {
        uint32_t q[3];
#pragma unroll
        for (int a = 0; a < 3; ++a)
            q[a] = quant10(__fdiv_rn(__fsub_rn(centroids[3 * (size_t)t + a], box[a]), box[3 + a]));
        const uint32_t c = (spread3(q[0]) << 2) | (spread3(q[1]) << 1) | spread3(q[2]);
        codes[t] = c;
#pragma unroll
        for (int p = 0; p < 4; ++p) atomicAdd(&h[p][(c >> (8 * p)) & 0xffu], 1u);
    }
    __syncthreads();
    for (int i = threadIdx.x; i < 4 * 256; i += kTB)
    {
        const uint32_t c = (&h[0][0])[i];
        if (c) atomicAdd(&hist[i], c);
    }
}

// Common-prefix length of sorted keys i and j (both in range), duplicates separated by index.
__device__ __forceinline__ int prefix(uint32_t a, uint32_t b, int i, int j)
{
    return a == b ? 32 + __clz((uint32_t)(i ^ j)) : __clz(a ^ b);
}

constexpr int kChunk = 512;          // sorted triangles per block of the tree, depth and emit kernels
constexpr int kNone = 0x3fffffff;    // no parent (the root's)
constexpr int kCollapsed = 1 << 30;  // in gap_parent: this node is collapsed
constexpr int kLeafLeft = 1 << 31;   // in gap_parent[k]: leaf k's parent is gap k (else gap k - 1)
constexpr int kMaxDepths = 32;       // kept nodes split distinct 30-bit codes: depth <= 30
constexpr int kNotKept = 255;

__device__ __forceinline__ int parent_of(int gap_parent_entry) { return gap_parent_entry & kNone; }

// The radix tree, one sorted position k per thread: gap k's range
// [gap_l, gap_r], parent and collapsed flag, and which side leaf k's parent is
// on.  skip[k] leads out
// of the block's chunk in one step: the first ancestor outside it (or kNone
// past the root) and the number of links to it, so the depth kernel's walks
// take a step per chunk instead of one per level.
__global__ void __launch_bounds__(kChunk) tree_kernel(const uint32_t* __restrict__ codes, int n,
                                                      int* __restrict__ gap_l, int* __restrict__ gap_r,
                                                      int* __restrict__ gap_parent, int2* __restrict__ skip)
{
    begin_after_predecessors();
    constexpr int kNear = 4;
    __shared__ uint32_t s_code[kChunk + 2];  // codes base - 1 .. base + kChunk
    __shared__ int s_l[kChunk], s_r[kChunk], s_list[2 * kChunk], s_listed;
    if (threadIdx.x == 0) s_listed = 0;
    const int base = blockIdx.x * kChunk;
    const int k = base + threadIdx.x;
    for (int i = threadIdx.x; i < kChunk + 2; i += kChunk)
    {
        const int g = base - 1 + i;
        if (g >= 0 && g < n) s_code[i] = codes[g];
    }
    __syncthreads();
    // most searches stay among the chunk's own codes
    auto code = [&](int i) {
        const unsigned at = (unsigned)(i - (base - 1));
        return at < (unsigned)(kChunk + 2) ? s_code[at] : __ldg(&codes[i]);
    };
    const int lo_here = max(base - 1, 0), hi_here = min(base + kChunk, n - 1);  // codes in shared memory
    int entry = kNone, dr = -1, l = k, r = k;
    bool left = false;
    const bool gap = k < n - 1;
    if (k < n)
    {
        const uint32_t ck = code(k);
        const int dl = k > 0 ? prefix(code(k - 1), ck, k - 1, k) : -1;  // gap k - 1
        if (gap) dr = prefix(ck, code(k + 1), k, k + 1);                // gap k
        left = dr > dl;
        if (gap)
        {
            r = k + 1;
            // keys left of the split share more than dr bits with key k, those right of it with key k + 1.  Most
            // ranges are short: up to kNear places on either side here
#pragma unroll
            for (int i = 0; i < kNear; ++i)
            {
                if (l == k - i && l > lo_here && prefix(code(l - 1), ck, l - 1, k) > dr) --l;
                if (r == k + 1 + i && r < hi_here && prefix(code(r + 1), code(k + 1), r + 1, k + 1) > dr) ++r;
            }
        }
    }
    // The longer ones are listed and searched by as many threads as there are, so that no warp runs at the pace of
    // its longest range.
    s_l[threadIdx.x] = l;
    s_r[threadIdx.x] = r;
    __syncthreads();
    if (gap && l == k - kNear && l > lo_here) s_list[atomicAdd(&s_listed, 1)] = (int)threadIdx.x;
    if (gap && r == k + 1 + kNear && r < hi_here) s_list[atomicAdd(&s_listed, 1)] = -1 - (int)threadIdx.x;
    __syncthreads();
    for (int i = threadIdx.x; i < s_listed; i += kChunk)
    {
        const int item = s_list[i], t = item < 0 ? -1 - item : item, dir = item < 0 ? 1 : -1;
        const int g = base + t, from = item < 0 ? g + 1 : g, end = item < 0 ? hi_here : lo_here;
        const uint32_t cf = code(from);
        const int bits = prefix(code(g), code(g + 1), g, g + 1);
        auto in = [&](int at) { return (end - at) * dir >= 0 && prefix(code(at), cf, at, from) > bits; };
        int at = kNear, step = kNear;
        while (in(from + dir * (at + step)))
        {
            at += step;
            step <<= 1;
        }
        for (step >>= 1; step > 0; step >>= 1)
            if (in(from + dir * (at + step))) at += step;
        (item < 0 ? s_r : s_l)[t] = from + dir * at;
    }
    // A range that reaches the end of those codes goes on outside: listed again, and searched by a warp with 32
    // probes a step, at doubling distances first (a thread's own search would be a chain of 2 log2(range) loads
    // from L2).
    __syncthreads();
    if (threadIdx.x == 0) s_listed = 0;
    __syncthreads();
    if (gap && s_l[threadIdx.x] == lo_here && lo_here > 0) s_list[atomicAdd(&s_listed, 1)] = (int)threadIdx.x;
    if (gap && s_r[threadIdx.x] == hi_here && hi_here < n - 1)
        s_list[atomicAdd(&s_listed, 1)] = -1 - (int)threadIdx.x;
    __syncthreads();
    for (int i = threadIdx.x >> 5; i < s_listed; i += kChunk / 32)
    {
        const int lane = threadIdx.x & 31;
        const int item = s_list[i], t = item < 0 ? -1 - item : item, dir = item < 0 ? 1 : -1;
        const int g = base + t, from = item < 0 ? g + 1 : g, edge = item < 0 ? hi_here : lo_here;
        const uint32_t cf = code(from);
        const int bits = prefix(code(g), code(g + 1), g, g + 1);
        // the farthest member lies in [in, out] places past the edge; keys are sorted, so the probes that are
        // members come first
        int in = 0, out = item < 0 ? n - 1 - edge : edge, stride = 0;
        while (in < out)
        {
            const long long d = stride ? (long long)stride * (lane + 1) : 1ll << min(lane, 30);
            const int probe = (int)min((long long)in + d, (long long)out);
            const int at = edge + dir * probe;
            const int hits = __popc(__ballot_sync(0xffffffffu, prefix(__ldg(&codes[at]), cf, at, from) > bits));
            const int reached = __shfl_sync(0xffffffffu, probe, max(hits - 1, 0));
            const int missed = __shfl_sync(0xffffffffu, probe, min(hits, 31));
            if (hits < 32) out = missed - 1;
            if (hits > 0) in = reached;
            stride = (out - in + 31) / 32;
        }
        if (lane == 0) (item < 0 ? s_r : s_l)[t] = edge + dir * in;
    }
    __syncthreads();
    l = s_l[threadIdx.x];
    r = s_r[threadIdx.x];
    if (k < n)
    {
        int par = kNone;
        if (gap)
        {
            const int pl = l > 0 ? prefix(code(l - 1), code(l), l - 1, l) : -1;
            const int pr = r < n - 1 ? prefix(code(r), code(r + 1), r, r + 1) : -1;
            if (pl >= 0 || pr >= 0) par = pr > pl ? r : l - 1;
            gap_l[k] = l;
            gap_r[k] = r;
            entry = par | (r - l + 1 <= 4 || dr >= 32 ? kCollapsed : 0) | (left ? kLeafLeft : 0);
            gap_parent[k] = entry;
        }
    }
    // Pointer doubling over the links inside the chunk (s_l: the ancestor reached so far, s_r: the links to it).
    __syncthreads();
    int to = parent_of(entry), hops = to == kNone ? 0 : 1;
    for (;;)
    {
        const int at = to - base;
        const bool more = to != kNone && at >= 0 && at < kChunk;
        s_l[threadIdx.x] = to;
        s_r[threadIdx.x] = hops;
        if (!__syncthreads_or(more)) break;
        if (more)
        {
            to = s_l[at];
            hops += s_r[at];
        }
        __syncthreads();
    }
    if (gap) skip[k] = make_int2(to, hops);
}

// Depths of the kept nodes of gap k and leaf k (kNotKept for the rest), and
// each chunk's count of nodes per depth, counts[depth][chunk].
__global__ void __launch_bounds__(kChunk) depth_kernel(int n, const int* __restrict__ gap_parent,
                                                       const int2* __restrict__ skip, uchar2* __restrict__ depth,
                                                       int* __restrict__ counts, int chunks)
{
    begin_after_predecessors();
    __shared__ int h[kMaxDepths];
    if (threadIdx.x < kMaxDepths) h[threadIdx.x] = 0;
    __syncthreads();
    const int k = blockIdx.x * kChunk + threadIdx.x;
    if (k < n)
    {
        auto depth_of = [&](int gap) {
            int d = 0;
            for (int at = gap; at != kNone;)
            {
                const int2 s = skip[at];
                d += s.y;
                at = s.x;
            }
            return d;
        };
        int dg = kNotKept, dleaf = kNotKept;
        const int entry = k < n - 1 ? gap_parent[k] : 0;
        if (k < n - 1)
        {
            const int p = parent_of(entry);
            if (p == kNone || !(gap_parent[p] & kCollapsed)) dg = depth_of(k);
        }
        const bool left = (entry & kLeafLeft) != 0;
        const int lp = left ? k : k - 1;
        if (!(gap_parent[lp] & kCollapsed)) dleaf = (left ? dg : depth_of(lp)) + 1;
        if (dg != kNotKept) atomicAdd(&h[dg], 1);
        if (dleaf != kNotKept) atomicAdd(&h[dleaf], 1);
        depth[k] = make_uchar2((unsigned char)dg, (unsigned char)dleaf);
    }
    __syncthreads();
    if (threadIdx.x < kMaxDepths) counts[(size_t)threadIdx.x * chunks + blockIdx.x] = h[threadIdx.x];
}

// Exclusive scan of each depth's row of counts, one block per depth, and the row totals.
__global__ void __launch_bounds__(kTB) depth_scan_kernel(int* __restrict__ counts, int chunks, int* __restrict__ totals)
{
    begin_after_predecessors();
    __shared__ int warp_sums[kTB / 32];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    int* row = counts + (size_t)blockIdx.x * chunks;
    int carry = 0;
    for (int base = 0; base < chunks; base += kTB * 4)
    {
        int v[4], sum = 0;
#pragma unroll
        for (int j = 0; j < 4; ++j)
        {
            const int i = base + threadIdx.x * 4 + j;
            v[j] = i < chunks ? row[i] : 0;
            sum += v[j];
        }
        int x = sum;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1)
        {
            const int y = __shfl_up_sync(0xffffffffu, x, o);
            if (lane >= o) x += y;
        }
        if (lane == 31) warp_sums[warp] = x;
        __syncthreads();
        int before = carry, all = 0;
        for (int w = 0; w < kTB / 32; ++w)
        {
            if (w < warp) before += warp_sums[w];
            all += warp_sums[w];
        }
        __syncthreads();
        int run = before + x - sum;
#pragma unroll
        for (int j = 0; j < 4; ++j)
        {
            const int i = base + threadIdx.x * 4 + j;
            if (i < chunks) row[i] = run;
            run += v[j];
        }
        carry += all;
    }
    if (threadIdx.x == 0) totals[blockIdx.x] = carry;
}

// BFS indices: nodes of one depth cover disjoint ranges, so their order by
// first triangle is their order by the position they are named after.  The
// index is the number of nodes less deep, plus those of the same depth at
// lower positions.  *n_nodes = all kept nodes.
__global__ void __launch_bounds__(kChunk) bfs_kernel(int n, const uchar2* __restrict__ depth,
                                                     const int* __restrict__ counts, int chunks,
                                                     const int* __restrict__ totals, int* __restrict__ bfs_gap,
                                                     int* __restrict__ bfs_leaf, int* __restrict__ n_nodes)
{
    begin_after_predecessors();
    constexpr int kWarps = kChunk / 32;
    __shared__ unsigned masks[kWarps][2][kMaxDepths];  // lanes whose gap / leaf has this depth
    __shared__ int first[kWarps][kMaxDepths];          // index of the warp's first node of the depth
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    masks[warp][0][lane] = masks[warp][1][lane] = 0;
    __syncwarp();
    const int k = blockIdx.x * kChunk + threadIdx.x;
    int d[2] = {kNotKept, kNotKept};
    if (k < n)
    {
        const uchar2 v = depth[k];
        d[0] = v.x;
        d[1] = v.y;
    }
#pragma unroll
    for (int j = 0; j < 2; ++j)
    {
        const unsigned peers = __match_any_sync(0xffffffffu, d[j]);
        if (d[j] != kNotKept && lane == __ffs(peers) - 1) masks[warp][j][d[j]] = peers;
    }
    __syncthreads();
    if (warp == 0)
    {
        const int total = totals[lane];
        int x = total;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1)
        {
            const int y = __shfl_up_sync(0xffffffffu, x, o);
            if (lane >= o) x += y;
        }
        if (blockIdx.x == 0 && lane == 31) *n_nodes = x;
        int run = x - total + counts[(size_t)lane * chunks + blockIdx.x];
        for (int w = 0; w < kWarps; ++w)
        {
            first[w][lane] = run;
            run += __popc(masks[w][0][lane]) + __popc(masks[w][1][lane]);
        }
    }
    __syncthreads();
    if (k >= n) return;
    const unsigned lt = (1u << lane) - 1u;
    int at[2] = {-1, -1};
#pragma unroll
    for (int j = 0; j < 2; ++j)
        if (d[j] != kNotKept)
            at[j] = first[warp][d[j]] + __popc(masks[warp][0][d[j]] & lt) + __popc(masks[warp][1][d[j]] & lt);
    bfs_gap[k] = at[0];
    bfs_leaf[k] = at[1];
}

struct FitBox
{
    float mn[3], mx[3];
};
__device__ __forceinline__ FitBox empty_box()
{
    FitBox b;
#pragma unroll
    for (int a = 0; a < 3; ++a)
    {
        b.mn[a] = __int_as_float(0x7f800000);
        b.mx[a] = __int_as_float(0xff800000);
    }
    return b;
}
__device__ __forceinline__ void fit_vertex(FitBox& b, const float* v)
{
#pragma unroll
    for (int a = 0; a < 3; ++a)
    {
        if (v[a] < b.mn[a]) b.mn[a] = v[a];
        if (v[a] > b.mx[a]) b.mx[a] = v[a];
    }
}
// Left box widened by the right one, with the reference's strict comparisons.
__device__ __forceinline__ FitBox join(FitBox l, const FitBox& r)
{
#pragma unroll
    for (int a = 0; a < 3; ++a)
    {
        if (r.mn[a] < l.mn[a]) l.mn[a] = r.mn[a];
        if (r.mx[a] > l.mx[a]) l.mx[a] = r.mx[a];
    }
    return l;
}
// Lane 0 gets the boxes of lanes 0 to 31 joined in lane order.
__device__ __forceinline__ FitBox warp_join(FitBox b)
{
#pragma unroll
    for (int o = 1; o < 32; o <<= 1)
    {
        FitBox r;
#pragma unroll
        for (int a = 0; a < 3; ++a)
        {
            r.mn[a] = __shfl_down_sync(0xffffffffu, b.mn[a], o);
            r.mx[a] = __shfl_down_sync(0xffffffffu, b.mx[a], o);
        }
        b = join(b, r);
    }
    return b;
}
__device__ __forceinline__ void put_node(lg_bvh_node* out, const FitBox& b, int left, int right, int first, int count)
{
#pragma unroll
    for (int a = 0; a < 3; ++a)
    {
        out->bbMin[a] = b.mn[a];
        out->bbMax[a] = b.mx[a];
    }
    out->left = left;
    out->right = right;
    out->firstTri = first;
    out->triCount = count;
}

// Moves the chunk's triangles into sorted order (word by word: whole sectors
// written, nearly whole ones read) and keeps their vertices in shared memory;
// then each kept leaf's thread fits its box and walks up while a node's range
// lies in the chunk, the second child to arrive at a node joining the two
// boxes, all in shared memory.  Arriving at a node exchanges the child's BFS
// index for what was there: 0 for the first child, the sibling's index + 1 for
// the second.  The chunk's topmost finished nodes go on in top_kernel.
// A leaf is wider than its chunk only where codes are equal, and one thread
// that reads it through the permutation takes 0.3 us a triangle, so past
// kWideLeaf triangles the whole block fits it, each thread a run of it, joined in
// order.  One B200, 131,072 triangles in one place 41.5 -> 0.75 ms, in runs of 5,000
// 1.67 -> 0.11, in runs of 100 0.16 -> 0.14; without such runs no difference.
constexpr int kWideLeaf = 16;
constexpr int kGroup = 32;  // chunks (or groups) per block of the top kernel
// Topmost nodes of one chunk or group: their parents' ranges cross its left or
// its right end, and the kept nodes that cross one place are nested, at most
// 30 deep.
constexpr int kTopMax = 64;
struct TopNode
{
    int at, par, right_end;  // BFS index, parent's gap, last triangle
};
struct EmitShared
{
    union
    {
        float verts[kChunk * 9];  // until the leaf boxes are fitted
        FitBox box[kChunk][2];    // then the children's boxes, by gap and side
    };
    int gl[kChunk], gr[kChunk], gp[kChunk], bfs[kChunk];
    int arrived[kChunk];
    union
    {
        uint32_t idx[kChunk];  // while the triangles are moved
        int top[kChunk];       // then the finished nodes whose parents' ranges leave the chunk
    };
    int n_top;
    // threads whose leaves leave the chunk (ranges are disjoint: one across each end at most), and the warps' parts
    int wide[2], n_wide;
    FitBox part[kChunk / 32];
};
struct TopShared
{
    TopNode in[kGroup * kTopMax], left[kTopMax];
    int start[kGroup + 1], n_left;
    int arrived[kGroup * kTopMax];
    int ends[kGroup * kTopMax][2];
    int4 gap[kGroup * kTopMax];  // of the gap at the input's right end: range, parent's gap, BFS index
    FitBox box[kGroup * kTopMax][2];
};
constexpr int kTopThreads = 512;

__global__ void __launch_bounds__(kChunk)
    emit_kernel(const lg_triangle* __restrict__ tris, const uint32_t* __restrict__ idx, int n,
                const int* __restrict__ gap_l, const int* __restrict__ gap_r, const int* __restrict__ gap_parent,
                const int* __restrict__ bfs_gap, const int* __restrict__ bfs_leaf, lg_triangle* __restrict__ tris_out,
                int32_t* __restrict__ perm_out, lg_bvh_node* nodes, TopNode* __restrict__ tops,
                int* __restrict__ n_tops)
{
    begin_after_predecessors();
    extern __shared__ __align__(16) unsigned char emit_mem[];
    EmitShared& sh = *reinterpret_cast<EmitShared*>(emit_mem);
    const int base = blockIdx.x * kChunk, t = threadIdx.x, k = base + t;
    const int cnt = min(kChunk, n - base);
    const bool gap_here = k < n - 1;
    int leaf = -1;
    if (t == 0) sh.n_top = sh.n_wide = 0;
    if (t < cnt)
    {
        const uint32_t src = idx[k];
        sh.idx[t] = src;
        sh.arrived[t] = 0;
        if (perm_out) perm_out[k] = (int32_t)src;
        sh.gl[t] = gap_here ? gap_l[k] : -1;
        sh.gr[t] = gap_here ? gap_r[k] : n;
        sh.gp[t] = gap_here ? gap_parent[k] : 0;
        sh.bfs[t] = bfs_gap[k];
        leaf = bfs_leaf[k];
    }
    __syncthreads();
    const uint32_t* in_words = reinterpret_cast<const uint32_t*>(tris);
    uint32_t* out_words = reinterpret_cast<uint32_t*>(tris_out) + (size_t)base * 25;
    constexpr int kBatch = 9;  // loads in flight per thread
    for (int w0 = t; w0 < cnt * 25; w0 += kChunk * kBatch)
    {
        uint32_t v[kBatch];
#pragma unroll
        for (int j = 0; j < kBatch; ++j)
        {
            const int w = w0 + j * kChunk;
            const int q = w / 25;
            if (w < cnt * 25) v[j] = in_words[(size_t)sh.idx[q] * 25 + (w - 25 * q)];
        }
#pragma unroll
        for (int j = 0; j < kBatch; ++j)
        {
            const int w = w0 + j * kChunk;
            const int q = w / 25, o = w - 25 * q;
            if (w >= cnt * 25) continue;
            out_words[w] = v[j];
            if (o < 9) sh.verts[q * 9 + o] = __uint_as_float(v[j]);
        }
    }
    __syncthreads();

    // the kept leaf named k, if any: triangle k alone, or collapsed gap k's run (never both: triangle k is in gap
    // k's range)
    int at = -1, gap = -1 - k, first = k, last = k, par = kNone;  // gap: the node's name, -1 - k for leaf k
    FitBox b = empty_box();
    if (t < cnt)
    {
        const int entry = sh.gp[t];
        at = leaf;
        if (at >= 0) par = gap_here && (entry & kLeafLeft) ? k : k - 1;
        else if (gap_here && (entry & kCollapsed))
        {
            at = sh.bfs[t];
            par = parent_of(entry);
            gap = k;
            first = sh.gl[t];
            last = sh.gr[t];
        }
    }
    auto fit_run = [&](FitBox& box, int from, int to) {
        for (int i = from; i < to; ++i)
        {
            const bool here = i >= base && i < base + cnt;
            const float* v = here ? &sh.verts[(i - base) * 9] : &tris[idx[i]].v[0][0];
            for (int j = 0; j < 3; ++j) fit_vertex(box, v + 3 * j);
        }
    };
    const bool wide = at >= 0 && last - first >= kWideLeaf && (first < base || last >= base + cnt);
    if (wide) sh.wide[atomicAdd(&sh.n_wide, 1)] = t;
    else if (at >= 0)
    {
        fit_run(b, first, last + 1);
        put_node(&nodes[at], b, -1, -1, first, last - first + 1);
    }
    __syncthreads();
    for (int j = 0; j < sh.n_wide; ++j)
    {
        const int owner = sh.wide[j], from = sh.gl[owner], end = sh.gr[owner] + 1;
        const int per = (end - from + kChunk - 1) / kChunk, mine = from + t * per;
        FitBox run = empty_box();
        fit_run(run, mine, min(mine + per, end));
        run = warp_join(run);
        if ((t & 31) == 0) sh.part[t >> 5] = run;
        __syncthreads();
        if (t == owner)
        {
            for (int w = 0; w < kChunk / 32; ++w) b = join(b, sh.part[w]);
            put_node(&nodes[at], b, -1, -1, first, last - first + 1);
        }
        __syncthreads();
    }
    // up: node `at` (box b) is finished, par its parent's gap
    for (int right_end = last; at >= 0 && par != kNone;)
    {
        const int lp = par - base;
        if (lp < 0 || lp >= cnt || sh.gl[lp] < base || sh.gr[lp] >= base + cnt)
        {
            sh.top[atomicAdd(&sh.n_top, 1)] = gap;
            break;
        }
        const int side = right_end == par ? 0 : 1;
        sh.box[lp][side] = b;
        __threadfence_block();
        const int other = atomicExch(&sh.arrived[lp], at + 1) - 1;
        if (other < 0) break;
        __threadfence_block();
        const volatile FitBox& vb = sh.box[lp][side ^ 1];
        FitBox ob;
#pragma unroll
        for (int a = 0; a < 3; ++a)
        {
            ob.mn[a] = vb.mn[a];
            ob.mx[a] = vb.mx[a];
        }
        b = side ? join(ob, b) : join(b, ob);
        const int me = sh.bfs[lp];
        put_node(&nodes[me], b, side ? other : at, side ? at : other, -1, 0);
        at = me;
        gap = par;
        right_end = sh.gr[lp];
        par = parent_of(sh.gp[lp]);
    }
    __syncthreads();

    if (t < sh.n_top)
    {
        // in order of position, for the kernel that goes on from here
        const int name = sh.top[t];
        TopNode top;
        if (name < 0)
        {
            const int q = -1 - name;
            top.at = bfs_leaf[q];
            top.par = q < n - 1 && (sh.gp[q - base] & kLeafLeft) ? q : q - 1;
            top.right_end = q;
        }
        else
        {
            top.at = sh.bfs[name - base];
            top.par = parent_of(sh.gp[name - base]);
            top.right_end = sh.gr[name - base];
        }
        int rank = 0;  // their ranges are disjoint
        for (int i = 0; i < sh.n_top; ++i)
        {
            const int g = sh.top[i];
            rank += (g < 0 ? -1 - g : sh.gr[g - base]) < top.right_end;
        }
        tops[(size_t)blockIdx.x * kTopMax + rank] = top;
    }
    if (t == 0) n_tops[blockIdx.x] = sh.n_top;
}

// Goes on where kGroup consecutive blocks of the emit kernel (or of this one)
// stopped: their topmost finished nodes in order, joined upwards through
// shared memory while a node's range lies within the group.  The place of a
// node in the group is that of its gap, which is the right end of exactly one
// of the nodes it came with: `hi` of its left child, `lo` - 1 of its right
// child.  What is left goes to the next launch, whose groups are kGroup times
// as wide.  (Going up through the node records with an atomic and two loads
// from L2 per level held each emit block for another 13 us, at most 46.)
__global__ void __launch_bounds__(kTopThreads)
    top_kernel(const TopNode* __restrict__ tops, const int* __restrict__ n_tops, int groups_in, long long span, int n,
               const int* __restrict__ gap_l, const int* __restrict__ gap_r, const int* __restrict__ gap_parent,
               const int* __restrict__ bfs_gap, TopNode* __restrict__ tops_out, int* __restrict__ n_tops_out,
               lg_bvh_node* nodes)
{
    begin_after_predecessors();
    extern __shared__ __align__(16) unsigned char emit_mem[];
    TopShared& sh = *reinterpret_cast<TopShared*>(emit_mem);
    const int first = blockIdx.x * kGroup, have = min(kGroup, groups_in - first);
    const long long begin = (long long)first * span, end = min(begin + kGroup * span, (long long)n);
    if (threadIdx.x < 32)
    {
        const int c = (int)threadIdx.x < have ? n_tops[first + threadIdx.x] : 0;
        int x = c;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1)
        {
            const int y = __shfl_up_sync(0xffffffffu, x, o);
            if ((int)threadIdx.x >= o) x += y;
        }
        sh.start[threadIdx.x + 1] = x;
        if (threadIdx.x == 0) sh.start[0] = sh.n_left = 0;
    }
    __syncthreads();
    const int cnt = sh.start[kGroup];
    for (int i = threadIdx.x; i < have * kTopMax; i += kTopThreads)
    {
        const int g = i / kTopMax, j = i % kTopMax;
        if (j >= sh.start[g + 1] - sh.start[g]) continue;
        const TopNode in = tops[(size_t)(first + g) * kTopMax + j];
        const int i2 = sh.start[g] + j, k = in.right_end;
        sh.in[i2] = in;
        sh.arrived[i2] = 0;
        if (k < n - 1) sh.gap[i2] = make_int4(gap_l[k], gap_r[k], parent_of(gap_parent[k]), bfs_gap[k]);
    }
    __syncthreads();
    for (int i = threadIdx.x; i < cnt; i += kTopThreads)
    {
        TopNode me = sh.in[i];
        int lo = i, hi = i;
        FitBox b;
#pragma unroll
        for (int a = 0; a < 3; ++a)
        {
            b.mn[a] = nodes[me.at].bbMin[a];
            b.mx[a] = nodes[me.at].bbMax[a];
        }
        while (me.par != kNone)
        {
            const int side = me.right_end == me.par ? 0 : 1;
            const int slot = side ? lo - 1 : hi;
            // a parent whose gap is the group's left end has no place here, and its range leaves the group
            const int4 up = slot >= 0 ? sh.gap[slot] : make_int4(-1, 0, 0, 0);
            if (up.x < begin || up.y >= end)
            {
                sh.left[atomicAdd(&sh.n_left, 1)] = me;
                break;
            }
            sh.box[slot][side] = b;
            sh.ends[slot][side] = side ? hi : lo;
            __threadfence_block();
            const int other = atomicExch(&sh.arrived[slot], me.at + 1) - 1;
            if (other < 0) break;
            __threadfence_block();
            const volatile FitBox& vb = sh.box[slot][side ^ 1];
            FitBox ob;
#pragma unroll
            for (int a = 0; a < 3; ++a)
            {
                ob.mn[a] = vb.mn[a];
                ob.mx[a] = vb.mx[a];
            }
            (side ? lo : hi) = *(volatile int*)&sh.ends[slot][side ^ 1];
            b = side ? join(ob, b) : join(b, ob);
            put_node(&nodes[up.w], b, side ? other : me.at, side ? me.at : other, -1, 0);
            me.at = up.w;
            me.par = up.z;
            me.right_end = up.y;
        }
    }
    __syncthreads();
    for (int i = threadIdx.x; i < sh.n_left; i += kTopThreads)
    {
        int rank = 0;
        for (int j = 0; j < sh.n_left; ++j) rank += sh.left[j].right_end < sh.left[i].right_end;
        tops_out[(size_t)blockIdx.x * kTopMax + rank] = sh.left[i];
    }
    if (threadIdx.x == 0) n_tops_out[blockIdx.x] = sh.n_left;
}

// Single-triangle scene: one leaf (bvh.cpp:92-104 with count 1).
__global__ void single_leaf_kernel(const lg_triangle* __restrict__ tris, lg_bvh_node* nodes)
{
    FitBox b = empty_box();
    for (int k = 0; k < 3; ++k) fit_vertex(b, tris[0].v[k]);
    put_node(&nodes[0], b, -1, -1, 0, 1);
}

int chunks_for(size_t n) { return (int)((n + kChunk - 1) / kChunk); }

struct Layout
{
    size_t bytes = 0;
    size_t off_box, off_cent, off_codes, off_idx, off_gl, off_gr, off_gp, off_skip, off_depth,
        off_counts, off_totals, off_bg, off_bl, off_tops, off_tops2, off_ntops, off_ntops2, off_zero, off_sort,
        off_tmp_tris;
};

Layout layout_for(size_t n, bool need_tmp_tris)
{
    Layout L;
    size_t at = 0;
    auto take = [&](size_t b) { size_t o = at; at += align256(b); return o; };
    L.off_box = take(6 * sizeof(float));
    L.off_cent = take(n * 12);
    L.off_codes = take(n * 4);
    L.off_idx = take(n * 4);
    L.off_gl = take(n * 4);
    L.off_gr = take(n * 4);
    L.off_gp = take(n * 4);
    L.off_skip = take(n * 8);
    L.off_depth = take(n * 2);
    L.off_counts = take((size_t)kMaxDepths * chunks_for(n) * 4);
    L.off_totals = take(kMaxDepths * 4);
    L.off_bg = take(n * 4);
    L.off_bl = take(n * 4);
    L.off_tops = take((size_t)chunks_for(n) * kTopMax * sizeof(TopNode));
    L.off_tops2 = take((size_t)(chunks_for(n) + kGroup - 1) / kGroup * kTopMax * sizeof(TopNode));
    L.off_ntops = take((size_t)chunks_for(n) * 4);
    L.off_ntops2 = take((size_t)(chunks_for(n) + kGroup - 1) / kGroup * 4);
    L.off_zero = take(256);  // bounds keys, block ticket, node count
    L.off_sort = take(radix_sort_scratch_bytes(n));
    L.off_tmp_tris = need_tmp_tris ? take(n * sizeof(lg_triangle)) : 0;
    L.bytes = at + 256;
    return L;
}
}  // namespace

size_t lbvh_scratch_bytes(int n_tris, bool tris_in_scratch)
{
    if (n_tris <= 1) return 256;
    return layout_for((size_t)n_tris, tris_in_scratch).bytes;
}

int lbvh_build(const lg_triangle* d_tris, int n, lg_bvh_node* d_nodes, int* n_nodes_host, int32_t* d_perm_out,
               lg_triangle* d_tris_out, void* scratch, size_t scratch_bytes, cudaStream_t stream)
{
    if (n < 0) return set_error(LG_ERR_INVALID, "BuildBVH: negative triangle count");
    if (n > (1 << kFirstBits)) return set_error(LG_ERR_INVALID, "BuildBVH: %d triangles exceeds 2^26", n);
    if (n == 0) { *n_nodes_host = 0; return LG_OK; }
    if (n == 1)
    {
        single_leaf_kernel<<<1, 1, 0, stream>>>(d_tris, d_nodes);
        if (d_tris_out && d_tris_out != d_tris)
            LG_TRY_CUDA(cudaMemcpyAsync(d_tris_out, d_tris, sizeof(lg_triangle), cudaMemcpyDeviceToDevice, stream));
        if (d_perm_out) LG_TRY_CUDA(cudaMemsetAsync(d_perm_out, 0, sizeof(int32_t), stream));
        LG_TRY_CUDA(cudaGetLastError());
        LG_TRY_CUDA(cudaStreamSynchronize(stream));
        *n_nodes_host = 1;
        return LG_OK;
    }
    // The leaf boxes read the triangles in sorted order; they are gathered into
    // scratch when the caller wants them in place or not at all.
    const bool need_tmp = d_tris_out == nullptr || d_tris_out == d_tris;
    const Layout L = layout_for((size_t)n, need_tmp);
    if (scratch_bytes < L.bytes) return set_error(LG_ERR_CAPACITY, "BuildBVH: scratch too small");
    char* base = (char*)(((uintptr_t)scratch + 255) & ~(uintptr_t)255);
    auto at = [&](size_t off) { return (void*)(base + off); };
    float* box = (float*)at(L.off_box);
    float* centroids = (float*)at(L.off_cent);
    uint32_t* codes = (uint32_t*)at(L.off_codes);
    uint32_t* idx = (uint32_t*)at(L.off_idx);
    int* gl = (int*)at(L.off_gl);
    int* gr = (int*)at(L.off_gr);
    int* gp = (int*)at(L.off_gp);
    int2* skip = (int2*)at(L.off_skip);
    uchar2* depth = (uchar2*)at(L.off_depth);
    int* counts = (int*)at(L.off_counts);
    int* totals = (int*)at(L.off_totals);
    int* bfs_gap = (int*)at(L.off_bg);
    int* bfs_leaf = (int*)at(L.off_bl);
    TopNode* tops = (TopNode*)at(L.off_tops);
    TopNode* tops2 = (TopNode*)at(L.off_tops2);
    int* n_tops = (int*)at(L.off_ntops);
    int* n_tops2 = (int*)at(L.off_ntops2);
    unsigned long long* keys = (unsigned long long*)at(L.off_zero);  // 6 bounds keys
    unsigned* ticket = (unsigned*)(keys + 6);
    int* node_count = (int*)(keys + 7);
    const RadixSortScratch rs = radix_sort_bind(at(L.off_sort), (size_t)n);
    const int chunks = chunks_for((size_t)n);

    LG_TRY_CUDA(cudaMemsetAsync(at(L.off_zero), 0, 256, stream));
    LG_TRY_CUDA(cudaMemsetAsync(rs.hist, 0, rs.zero_bytes, stream));
    const int grid = std::min(blocks_for((size_t)n), 148 * 8);
    LG_TRY_CUDA(launch_dependent(bounds_kernel, grid, kTB, 0, stream, d_tris, n, keys, ticket, centroids, box));
    LG_TRY_CUDA(launch_dependent(morton_kernel, std::min(grid, 148 * 4), kTB, 0, stream, centroids, n, box, codes,
                                 rs.hist));
    // 30-bit codes, stable: ties stay in input order
    LG_TRY_CUDA(radix_sort_pairs(codes, idx, (size_t)n, 0, 30, rs, stream, true, true));
    LG_TRY_CUDA(launch_dependent(tree_kernel, chunks, kChunk, 0, stream, codes, n, gl, gr, gp, skip));
    LG_TRY_CUDA(launch_dependent(depth_kernel, chunks, kChunk, 0, stream, n, gp, skip, depth, counts, chunks));
    LG_TRY_CUDA(launch_dependent(depth_scan_kernel, kMaxDepths, kTB, 0, stream, counts, chunks, totals));
    LG_TRY_CUDA(launch_dependent(bfs_kernel, chunks, kChunk, 0, stream, n, depth, counts, chunks, totals, bfs_gap,
                                 bfs_leaf, node_count));
    lg_triangle* tris_sorted = need_tmp ? (lg_triangle*)at(L.off_tmp_tris) : d_tris_out;
    LG_TRY_CUDA(cudaFuncSetAttribute((const void*)emit_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                     (int)sizeof(EmitShared)));
    LG_TRY_CUDA(launch_dependent(emit_kernel, chunks, kChunk, (int)sizeof(EmitShared), stream, d_tris, idx, n, gl,
                                 gr, gp, bfs_gap, bfs_leaf, tris_sorted, d_perm_out, d_nodes, tops, n_tops));
    LG_TRY_CUDA(cudaFuncSetAttribute((const void*)top_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                     (int)sizeof(TopShared)));
    long long span = kChunk;
    for (int groups = chunks; groups > 1;)
    {
        const int out = (groups + kGroup - 1) / kGroup;
        LG_TRY_CUDA(launch_dependent(top_kernel, out, kTopThreads, (int)sizeof(TopShared), stream, tops, n_tops,
                                     groups, span, n, gl, gr, gp, bfs_gap, tops2, n_tops2, d_nodes));
        std::swap(tops, tops2);
        std::swap(n_tops, n_tops2);
        groups = out;
        span *= kGroup;
    }
    if (d_tris_out && need_tmp)
        LG_TRY_CUDA(cudaMemcpyAsync(d_tris_out, tris_sorted, (size_t)n * sizeof(lg_triangle),
                                    cudaMemcpyDeviceToDevice, stream));
    LG_TRY_CUDA(cudaGetLastError());
    int count = 0;
    LG_TRY_CUDA(cudaMemcpyAsync(&count, node_count, sizeof(int), cudaMemcpyDeviceToHost, stream));
    LG_TRY_CUDA(cudaStreamSynchronize(stream));
    *n_nodes_host = count;
    return LG_OK;
}
}  // namespace lg
