// render_tree.cu -- the binary tree the traversal records are built from.
//
// BuildBVH's tree (bit-exact to the reference) is what lg_build_bvh returns
// and what the G-buffer box comes from.  Rays do not need that exact tree:
// any binary tree over the same leaves gives the same closest hits (up to
// exact ties in t).  Two render trees are built here, both in depth order
// (every depth a contiguous range, the root first), which the 4-wide
// collapse relies on:
//   * mode 0: the input tree itself, stably re-sorted by depth (a tree the
//     caller supplies need not be in breadth-first order);
//   * mode 1: the input tree's leaves, regrouped by PLOC -- "Parallel
//     Locally-Ordered Clustering for BVH Construction" (Meister and Bittner,
//     HPG 2018).  Clusters start as the leaves in Morton order (their first
//     triangles); each round, every cluster finds the neighbour within +-R
//     positions whose union box has the smallest surface area, mutual
//     nearest neighbours merge into a new node, and the survivors are
//     compacted in order.  The Morton tree splits at code bits; PLOC groups
//     by actual box sizes, so traversal opens fewer boxes.
//   * mode 2: PLOC over the triangles themselves (in their Morton order),
//     one triangle per leaf: 2T - 1 nodes.  Leaves index the same triangle
//     array, so nothing is reordered; any BVH over the triangles finds the
//     same closest hits (up to exact ties in t).
// Ties in the neighbour search go to the lower position and every numbering
// comes from prefix sums, so both trees are deterministic.
#include <algorithm>
#include <cstdint>
#include <vector>

#include <cuda_runtime.h>

#include "bvh.h"
#include "common.h"
#include "pdl.cuh"
#include "radix_sort.cuh"
#include "render_tree.cuh"

namespace lg
{
namespace
{
constexpr int kTB = 256;
constexpr int kRadius = 8;  // PLOC search radius (positions on either side); 8 measured 1% faster to trace than 16 or 32

size_t a256(size_t b) { return (b + 255) & ~(size_t)255; }

// ---- exclusive scan of int flags/counts (block sums + one-block scan + add) ----
__device__ __forceinline__ int block_excl_scan(int v, int* warp_sums, int& total)
{
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    int x = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1)
    {
        const int y = __shfl_up_sync(0xffffffffu, x, o);
        if (lane >= o) x += y;
    }
    if (lane == 31) warp_sums[warp] = x;
    __syncthreads();
    int before = 0;
    total = 0;
    for (int w = 0; w < kTB / 32; ++w)
    {
        if (w < warp) before += warp_sums[w];
        total += warp_sums[w];
    }
    __syncthreads();
    return before + x - v;
}
__global__ void scan_local_kernel(const int* __restrict__ in, int n, int* __restrict__ out, int* __restrict__ sums)
{
    begin_after_predecessors();
    __shared__ int ws[kTB / 32];
    const int i = blockIdx.x * kTB + threadIdx.x;
    int total;
    const int e = block_excl_scan(i < n ? in[i] : 0, ws, total);
    if (i < n) out[i] = e;
    if (threadIdx.x == 0) sums[blockIdx.x] = total;
}
__global__ void scan_sums_kernel(int* __restrict__ sums, int nb, int* __restrict__ grand_total)
{
    begin_after_predecessors();
    __shared__ int ws[kTB / 32];
    __shared__ int carry;
    if (threadIdx.x == 0) carry = 0;
    __syncthreads();
    for (int b = 0; b < nb; b += kTB)
    {
        const int i = b + threadIdx.x;
        int total;
        const int e = block_excl_scan(i < nb ? sums[i] : 0, ws, total);
        if (i < nb) sums[i] = carry + e;
        __syncthreads();
        if (threadIdx.x == 0) carry += total;
        __syncthreads();
    }
    if (threadIdx.x == 0 && grand_total) *grand_total = carry;
}
__global__ void scan_add_kernel(int* __restrict__ out, int n, const int* __restrict__ sums)
{
    begin_after_predecessors();
    const int i = blockIdx.x * kTB + threadIdx.x;
    if (i < n) out[i] += sums[blockIdx.x];
}
// out = exclusive scan of in (in == out allowed); *total (device) = sum.
cudaError_t excl_scan(const int* in, int n, int* out, int* sums, int* total, cudaStream_t st)
{
    const int nb = (n + kTB - 1) / kTB;
    if (n <= 0) return cudaMemsetAsync(total, 0, sizeof(int), st);
    cudaError_t e = launch_dependent(scan_local_kernel, nb, kTB, 0, st, in, n, out, sums);
    if (e == cudaSuccess) e = launch_dependent(scan_sums_kernel, 1, kTB, 0, st, sums, nb, total);
    if (e == cudaSuccess) e = launch_dependent(scan_add_kernel, nb, kTB, 0, st, out, n, sums);
    return e;
}
// ---- depth order ----
__global__ void parent_of_kernel(const lg_bvh_node* __restrict__ nodes, int n, int* __restrict__ parent)
{
    begin_after_predecessors();
    const int i = blockIdx.x * kTB + threadIdx.x;
    if (i >= n) return;
    const lg_bvh_node nd = nodes[i];
    if (nd.triCount == 0)
    {
        parent[nd.left] = i;
        parent[nd.right] = i;
    }
}
__global__ void depth_of_kernel(int n, int root, const int* __restrict__ parent, uint32_t* __restrict__ depth,
                                uint32_t* __restrict__ ids)
{
    begin_after_predecessors();
    const int i = blockIdx.x * kTB + threadIdx.x;
    if (i >= n) return;
    uint32_t d = 0;
    // nodes no link reaches (possible in a caller's array) stop at parent -1
    for (int a = i; a != root && a >= 0 && a < n && d < 255u; a = parent[a]) ++d;
    depth[i] = d;
    ids[i] = (uint32_t)i;
}
__global__ void rank_kernel(const uint32_t* __restrict__ order, int n, int* __restrict__ newpos)
{
    begin_after_predecessors();
    const int r = blockIdx.x * kTB + threadIdx.x;
    if (r < n) newpos[order[r]] = r;
}
// Nodes in depth order with their links renumbered, word by word (a node is 10
// words): whole sectors written.  One thread per node took 91 us for 2.1 M
// nodes, this 51.
constexpr int kEmitNodes = 256;
__global__ void __launch_bounds__(kTB) emit_kernel(const lg_bvh_node* __restrict__ in, const uint32_t* __restrict__ order,
                                                   const int* __restrict__ newpos, int n, lg_bvh_node* __restrict__ out)
{
    begin_after_predecessors();
    __shared__ uint32_t s_src[kEmitNodes];
    const int base = blockIdx.x * kEmitNodes, cnt = min(kEmitNodes, n - base);
    for (int i = threadIdx.x; i < cnt; i += kTB) s_src[i] = order[base + i];
    __syncthreads();
    const int* words = reinterpret_cast<const int*>(in);
    int* to = reinterpret_cast<int*>(out) + (size_t)base * 10;
#pragma unroll 5
    for (int w = threadIdx.x; w < cnt * 10; w += kTB)
    {
        const int i = w / 10, o = w - 10 * i;
        const size_t at = (size_t)s_src[i] * 10;
        int v = words[at + o];
        if ((o == 6 || o == 7) && words[at + 9] == 0) v = newpos[v];  // left, right of an internal node
        to[w] = v;
    }
}
// Where each depth's nodes begin in depth order, from the sort's counts of the 256 depths; start[256] = n.
__global__ void level_start_kernel(const uint32_t* __restrict__ counts, int n, int* __restrict__ start)
{
    begin_after_predecessors();
    __shared__ int ws[kTB / 32];
    int total;
    const int e = block_excl_scan((int)counts[threadIdx.x], ws, total);
    start[threadIdx.x] = e;
    if (threadIdx.x == 0) start[256] = n;
}

// ---- PLOC ----
struct Box
{
    float4 lo, hi;  // w unused
};
__device__ __forceinline__ float half_area(const Box& b)
{
    const float dx = b.hi.x - b.lo.x, dy = b.hi.y - b.lo.y, dz = b.hi.z - b.lo.z;
    return dx * dy + dy * dz + dz * dx;
}
__device__ __forceinline__ Box join(const Box& a, const Box& b)
{
    Box c;
    c.lo = make_float4(fminf(a.lo.x, b.lo.x), fminf(a.lo.y, b.lo.y), fminf(a.lo.z, b.lo.z), 0.0f);
    c.hi = make_float4(fmaxf(a.hi.x, b.hi.x), fmaxf(a.hi.y, b.hi.y), fmaxf(a.hi.z, b.hi.z), 0.0f);
    return c;
}

// Leaves by first triangle (= Morton order): leaf_at[t] = node whose range starts at t.
__global__ void leaf_at_kernel(const lg_bvh_node* __restrict__ nodes, int n, int* __restrict__ leaf_at,
                               int* __restrict__ flag)
{
    begin_after_predecessors();
    const int i = blockIdx.x * kTB + threadIdx.x;
    if (i >= n) return;
    const lg_bvh_node nd = nodes[i];
    if (nd.triCount > 0)
    {
        leaf_at[nd.firstTri] = i;
        flag[nd.firstTri] = 1;
    }
}
// Cluster k = leaf k in Morton order, node id k of the new tree.
__global__ void init_clusters_kernel(const lg_bvh_node* __restrict__ nodes, const int* __restrict__ leaf_at,
                                     const int* __restrict__ flag, const int* __restrict__ pos, int n_tris,
                                     lg_bvh_node* __restrict__ tn, int* __restrict__ cid, Box* __restrict__ cbox)
{
    begin_after_predecessors();
    const int t = blockIdx.x * kTB + threadIdx.x;
    if (t >= n_tris || !flag[t]) return;
    const int k = pos[t];
    const lg_bvh_node nd = nodes[leaf_at[t]];
    tn[k] = nd;
    cid[k] = k;
    Box b;
    b.lo = make_float4(nd.bbMin[0], nd.bbMin[1], nd.bbMin[2], 0.0f);
    b.hi = make_float4(nd.bbMax[0], nd.bbMax[1], nd.bbMax[2], 0.0f);
    cbox[k] = b;
}
// Cluster t = triangle t (one-triangle leaf, node id t of the new tree).
__global__ void init_tri_clusters_kernel(const lg_triangle* __restrict__ tris, int n_tris,
                                         lg_bvh_node* __restrict__ tn, int* __restrict__ cid, Box* __restrict__ cbox)
{
    begin_after_predecessors();
    const int t = blockIdx.x * kTB + threadIdx.x;
    if (t >= n_tris) return;
    const lg_triangle tr = tris[t];
    lg_bvh_node nd;
    for (int a = 0; a < 3; ++a)
    {
        nd.bbMin[a] = fminf(fminf(tr.v[0][a], tr.v[1][a]), tr.v[2][a]);
        nd.bbMax[a] = fmaxf(fmaxf(tr.v[0][a], tr.v[1][a]), tr.v[2][a]);
    }
    nd.left = -1;
    nd.right = -1;
    nd.firstTri = t;
    nd.triCount = 1;
    tn[t] = nd;
    cid[t] = t;
    Box b;
    b.lo = make_float4(nd.bbMin[0], nd.bbMin[1], nd.bbMin[2], 0.0f);
    b.hi = make_float4(nd.bbMax[0], nd.bbMax[1], nd.bbMax[2], 0.0f);
    cbox[t] = b;
}
// Nearest neighbour within +-kRadius positions by union surface area; ties -> lower position.
// The clustering round's kernels read the cluster count c from device memory
// (the round loop checks it on the host only every few rounds).
__global__ void __launch_bounds__(kTB) nn_kernel(const Box* __restrict__ cbox, const int* __restrict__ dc,
                                                 int* __restrict__ nn)
{
    begin_after_predecessors();
    __shared__ Box sb[kTB + 2 * kRadius];
    const int c = *dc;
    const int base = blockIdx.x * kTB - kRadius;
    for (int j = threadIdx.x; j < kTB + 2 * kRadius; j += kTB)
    {
        const int g = base + j;
        if (g >= 0 && g < c) sb[j] = cbox[g];
    }
    __syncthreads();
    const int i = blockIdx.x * kTB + threadIdx.x;
    if (i >= c) return;
    const Box bi = sb[threadIdx.x + kRadius];
    float best = __int_as_float(0x7f800000);
    int bj = -1;
    const int lo = max(0, i - kRadius), hi = min(c - 1, i + kRadius);
    for (int j = lo; j <= hi; ++j)
    {
        if (j == i) continue;
        const float a = half_area(join(bi, sb[j - base]));
        if (a < best)
        {
            best = a;
            bj = j;
        }
    }
    nn[i] = bj;
}
// A clustering round in four launches: nn_kernel, round_flags_kernel (merge
// and keep flags and their block-local exclusive scans), round_sums_kernel
// (one block: the block offsets, and the next round's state), and
// round_apply_kernel (merge and compact).  State {c, next node id, error}
// is double-buffered, cur -> nxt, so no launch reads a value its round
// changes.  The integer scans give the same positions as the three-kernel
// scans, so the tree does not change.
__global__ void round_flags_kernel(const int* __restrict__ nn, const int* __restrict__ cur, int* __restrict__ mflag,
                                   int* __restrict__ kflag, int* __restrict__ midx, int* __restrict__ kpos,
                                   int* __restrict__ msums, int* __restrict__ ksums)
{
    begin_after_predecessors();
    __shared__ int ws[kTB / 32];
    const int c = cur[0];
    const int i = blockIdx.x * kTB + threadIdx.x;
    int m = 0, k = 0;
    if (i < c)
    {
        const int j = nn[i];
        const bool mutual = j >= 0 && nn[j] == i;
        m = (mutual && i < j) ? 1 : 0;  // i owns the merged node
        k = (mutual && i > j) ? 0 : 1;  // j's partner disappears
        mflag[i] = m;
        kflag[i] = k;
    }
    int tm, tk;
    const int em = block_excl_scan(m, ws, tm);
    const int ek = block_excl_scan(k, ws, tk);
    if (i < c)
    {
        midx[i] = em;
        kpos[i] = ek;
    }
    if (threadIdx.x == 0)
    {
        msums[blockIdx.x] = tm;
        ksums[blockIdx.x] = tk;
    }
}
constexpr int kSumThreads = 1024;
__global__ void __launch_bounds__(kSumThreads) round_sums_kernel(int* __restrict__ msums, int* __restrict__ ksums, int nb,
                                                                 const int* __restrict__ cur, int* __restrict__ nxt)
{
    begin_after_predecessors();
    __shared__ int ws[2][kSumThreads / 32];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int per = (nb + kSumThreads - 1) / kSumThreads;  // consecutive entries per thread
    const int first = min((int)threadIdx.x * per, nb), last = min(first + per, nb);
    int sm = 0, sk = 0;
    for (int i = first; i < last; ++i)
    {
        sm += msums[i];
        sk += ksums[i];
    }
    int xm = sm, xk = sk;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1)
    {
        const int ym = __shfl_up_sync(0xffffffffu, xm, o), yk = __shfl_up_sync(0xffffffffu, xk, o);
        if (lane >= o)
        {
            xm += ym;
            xk += yk;
        }
    }
    if (lane == 31)
    {
        ws[0][warp] = xm;
        ws[1][warp] = xk;
    }
    __syncthreads();
    int bm = xm - sm, bk = xk - sk, merges = 0, kept = 0;
    for (int w = 0; w < kSumThreads / 32; ++w)
    {
        if (w == warp)
        {
            bm += merges;
            bk += kept;
        }
        merges += ws[0][w];
        kept += ws[1][w];
    }
    for (int i = first; i < last; ++i)
    {
        const int m = msums[i], k = ksums[i];
        msums[i] = bm;
        ksums[i] = bk;
        bm += m;
        bk += k;
    }
    if (threadIdx.x == 0)
    {
        nxt[2] = cur[2] | ((cur[0] > 1 && merges == 0) ? 1 : 0);
        nxt[1] = cur[1] + merges;
        nxt[0] = kept;
    }
}
__global__ void round_apply_kernel(const int* __restrict__ nn, const int* __restrict__ cur,
                                   const int* __restrict__ mflag, const int* __restrict__ kflag,
                                   const int* __restrict__ midx, const int* __restrict__ kpos,
                                   const int* __restrict__ msums, const int* __restrict__ ksums, int* __restrict__ cid,
                                   Box* __restrict__ cbox, lg_bvh_node* __restrict__ tn, int* __restrict__ cid2,
                                   Box* __restrict__ cbox2)
{
    begin_after_predecessors();
    const int c = cur[0], node_base = cur[1];
    const int i = blockIdx.x * kTB + threadIdx.x;
    if (i >= c) return;
    int id = cid[i];
    Box b = cbox[i];
    if (mflag[i])
    {
        // merge with the mutual nearest neighbour j > i (j keeps nothing and writes nothing this round)
        const int j = nn[i];
        id = node_base + msums[blockIdx.x] + midx[i];
        const Box bj = cbox[j];
        b = join(b, bj);
        lg_bvh_node nd;
        nd.bbMin[0] = b.lo.x; nd.bbMin[1] = b.lo.y; nd.bbMin[2] = b.lo.z;
        nd.bbMax[0] = b.hi.x; nd.bbMax[1] = b.hi.y; nd.bbMax[2] = b.hi.z;
        nd.left = cid[i];
        nd.right = cid[j];
        nd.firstTri = -1;
        nd.triCount = 0;
        tn[id] = nd;
    }
    if (kflag[i])
    {
        const int pos = ksums[blockIdx.x] + kpos[i];
        cid2[pos] = id;
        cbox2[pos] = b;
    }
}

// Every remaining round at once, in one block, from kTailClusters clusters on:
// the rounds above in shared memory, with the same neighbours, merges and
// numbering.  On the engine scene 40 of the 64 rounds start with fewer clusters
// than that: 189 us here, about 600 us as four launches of 3 to 4 us each.
constexpr int kTailClusters = 4096;
constexpr int kTailThreads = 1024;
constexpr int kTailItems = kTailClusters / kTailThreads;
struct TailShared
{
    float box[6][kTailClusters];
    int nn[kTailClusters], id[kTailClusters];
    int merges[kTailItems * kTailThreads / 32], keeps[kTailItems * kTailThreads / 32];  // per 32 clusters
    int total[2];
};
__global__ void __launch_bounds__(kTailThreads) rounds_tail_kernel(const int* __restrict__ cid, const Box* __restrict__ cbox,
                                                                   int* __restrict__ state, lg_bvh_node* __restrict__ tn,
                                                                   int* __restrict__ root)
{
    begin_after_predecessors();
    extern __shared__ __align__(16) unsigned char tail_mem[];
    TailShared& sh = *reinterpret_cast<TailShared*>(tail_mem);
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const unsigned lt = (1u << lane) - 1u;
    int c = state[0], next_id = state[1];
    if (c > kTailClusters) return;  // the host never launches it so
    auto box_at = [&](int i) {
        Box b;
        b.lo = make_float4(sh.box[0][i], sh.box[1][i], sh.box[2][i], 0.0f);
        b.hi = make_float4(sh.box[3][i], sh.box[4][i], sh.box[5][i], 0.0f);
        return b;
    };
    auto put_box = [&](int i, const Box& b) {
        sh.box[0][i] = b.lo.x;
        sh.box[1][i] = b.lo.y;
        sh.box[2][i] = b.lo.z;
        sh.box[3][i] = b.hi.x;
        sh.box[4][i] = b.hi.y;
        sh.box[5][i] = b.hi.z;
    };
    for (int i = tid; i < c; i += kTailThreads)
    {
        put_box(i, cbox[i]);
        sh.id[i] = cid[i];
    }
    __syncthreads();
    while (c > 1)
    {
        for (int i = tid; i < c; i += kTailThreads)
        {
            const Box bi = box_at(i);
            float best = __int_as_float(0x7f800000);
            int bj = -1;
            const int lo = max(0, i - kRadius), hi = min(c - 1, i + kRadius);
            for (int j = lo; j <= hi; ++j)
            {
                if (j == i) continue;
                const float a = half_area(join(bi, box_at(j)));
                if (a < best)
                {
                    best = a;
                    bj = j;
                }
            }
            sh.nn[i] = bj;
        }
        __syncthreads();
        Box b[kTailItems];
        int id[kTailItems], rank_m[kTailItems], rank_k[kTailItems], partner[kTailItems];
        bool keep[kTailItems];
#pragma unroll
        for (int k = 0; k < kTailItems; ++k)
        {
            const int i = k * kTailThreads + tid;
            bool m = false;
            keep[k] = false;
            partner[k] = -1;
            if (i < c)
            {
                const int j = sh.nn[i];
                const bool mutual = j >= 0 && sh.nn[j] == i;
                m = mutual && i < j;
                keep[k] = !(mutual && i > j);
                if (m) partner[k] = j;
                b[k] = box_at(i);
                id[k] = sh.id[i];
            }
            const unsigned vm = __ballot_sync(0xffffffffu, m), vk = __ballot_sync(0xffffffffu, keep[k]);
            rank_m[k] = __popc(vm & lt);
            rank_k[k] = __popc(vk & lt);
            if (lane == 0)
            {
                sh.merges[k * (kTailThreads / 32) + warp] = __popc(vm);
                sh.keeps[k * (kTailThreads / 32) + warp] = __popc(vk);
            }
        }
        __syncthreads();
        // exclusive scans of the counts of 32: warp 0 the merges, warp 1 the kept clusters
        if (warp < 2)
        {
            int* v = warp == 0 ? sh.merges : sh.keeps;
            int carry = 0;
            for (int at = lane; at < kTailItems * kTailThreads / 32; at += 32)
            {
                const int own = v[at];
                int x = own;
#pragma unroll
                for (int o = 1; o < 32; o <<= 1)
                {
                    const int y = __shfl_up_sync(0xffffffffu, x, o);
                    if (lane >= o) x += y;
                }
                v[at] = carry + x - own;
                carry += __shfl_sync(0xffffffffu, x, 31);
            }
            if (lane == 0) sh.total[warp] = carry;
        }
        __syncthreads();
        const int merges = sh.total[0], kept = sh.total[1];
        if (merges == 0)
        {
            if (tid == 0) state[2] = 1;
            return;
        }
#pragma unroll
        for (int k = 0; k < kTailItems; ++k)
        {
            if (partner[k] < 0) continue;
            const int j = partner[k];
            b[k] = join(b[k], box_at(j));
            lg_bvh_node nd;
            nd.bbMin[0] = b[k].lo.x; nd.bbMin[1] = b[k].lo.y; nd.bbMin[2] = b[k].lo.z;
            nd.bbMax[0] = b[k].hi.x; nd.bbMax[1] = b[k].hi.y; nd.bbMax[2] = b[k].hi.z;
            nd.left = id[k];
            nd.right = sh.id[j];
            nd.firstTri = -1;
            nd.triCount = 0;
            id[k] = next_id + sh.merges[k * (kTailThreads / 32) + warp] + rank_m[k];
            tn[id[k]] = nd;
        }
        __syncthreads();
#pragma unroll
        for (int k = 0; k < kTailItems; ++k)
            if (keep[k])
            {
                const int pos = sh.keeps[k * (kTailThreads / 32) + warp] + rank_k[k];
                put_box(pos, b[k]);
                sh.id[pos] = id[k];
            }
        next_id += merges;
        c = kept;
        __syncthreads();
    }
    if (tid == 0)
    {
        state[0] = c;
        state[1] = next_id;
        *root = sh.id[0];
    }
}

struct Scratch
{
    char* p;
    char* end;
    template <class T>
    T* take(size_t count)
    {
        T* r = (T*)p;
        p += a256(count * sizeof(T));
        return p <= end ? r : nullptr;
    }
};
}  // namespace

int render_tree_nodes(int n_nodes, int n_tris, int mode)
{
    return mode == 2 && n_tris > 0 ? 2 * n_tris - 1 : n_nodes;
}

size_t render_tree_scratch_bytes(int n_nodes, int n_tris)
{
    const size_t t = (size_t)(n_tris > 0 ? n_tris : 1);
    // the larger of the modes: BuildBVH's n_nodes, or 2T - 1 one-triangle-leaf nodes
    const size_t n = std::max((size_t)(n_nodes > 0 ? n_nodes : 1), 2 * t);
    const size_t L = std::max((n + 1) / 2, t);
    size_t b = 0;
    b += a256(n * sizeof(lg_bvh_node));         // tn
    b += 4 * a256(n * 4);                       // parent, depth, ids, newpos
    b += a256(radix_sort_scratch_bytes(n));
    b += 3 * a256(t * 4);                       // leaf_at, flag, pos
    b += 2 * (a256(L * 4) + a256(L * sizeof(Box)));  // cluster arrays (double buffered)
    b += 5 * a256(L * 4);                       // nn, mflag, midx, kflag, kpos
    b += a256(2 * (L / kTB + 2) * 4) + 256;     // block sums (merge and keep flags), totals
    return b + 1024;
}

int build_render_tree(const lg_bvh_node* d_nodes, int n_nodes, const lg_triangle* d_tris, int n_tris, int mode,
                      lg_bvh_node* d_out, int* d_level_start, int* level_start_host, int* levels, void* scratch,
                      size_t scratch_bytes, cudaStream_t st)
{
    if (n_nodes <= 0) return LG_OK;
    const int in_nodes = n_nodes;
    n_nodes = render_tree_nodes(n_nodes, n_tris, mode);
    Scratch s{(char*)(((uintptr_t)scratch + 255) & ~(uintptr_t)255), (char*)scratch + scratch_bytes};
    lg_bvh_node* tn = s.take<lg_bvh_node>((size_t)n_nodes);
    int* parent = s.take<int>((size_t)n_nodes);
    uint32_t* depth = s.take<uint32_t>((size_t)n_nodes);
    uint32_t* ids = s.take<uint32_t>((size_t)n_nodes);
    int* newpos = s.take<int>((size_t)n_nodes);
    char* sort_mem = s.take<char>(radix_sort_scratch_bytes((size_t)n_nodes));
    if (!tn || !parent || !depth || !ids || !newpos || !sort_mem)
        return set_error(LG_ERR_CAPACITY, "render tree: scratch too small");
    const lg_bvh_node* src = d_nodes;
    int root = 0;
    const int g = (n_nodes + kTB - 1) / kTB;

    if ((mode == 1 || mode == 2) && n_nodes > 1)
    {
        const int t = n_tris;
        int* leaf_at = s.take<int>((size_t)t);
        int* flag = s.take<int>((size_t)t);
        int* pos = s.take<int>((size_t)t);
        const int L = (n_nodes + 1) / 2;
        int* cid = s.take<int>((size_t)L);
        Box* cbox = s.take<Box>((size_t)L);
        int* cid2 = s.take<int>((size_t)L);
        Box* cbox2 = s.take<Box>((size_t)L);
        int* nn = s.take<int>((size_t)L);
        int* mflag = s.take<int>((size_t)L);
        int* midx = s.take<int>((size_t)L);
        int* kflag = s.take<int>((size_t)L);
        int* kpos = s.take<int>((size_t)L);
        int* sums = s.take<int>(2 * ((size_t)t / kTB + 2));
        int* totals = s.take<int>(64);
        if (!sums || !totals) return set_error(LG_ERR_CAPACITY, "render tree: scratch too small");
        int c = 0;
        if (mode == 2)
        {
            LG_TRY_CUDA(launch_dependent(init_tri_clusters_kernel, (t + kTB - 1) / kTB, kTB, 0, st, d_tris, t, tn,
                                         cid, cbox));
            LG_TRY_CUDA(cudaGetLastError());
            c = t;
        }
        else
        {
            LG_TRY_CUDA(cudaMemsetAsync(flag, 0, sizeof(int) * (size_t)t, st));
            LG_TRY_CUDA(launch_dependent(leaf_at_kernel, (in_nodes + kTB - 1) / kTB, kTB, 0, st, d_nodes, in_nodes,
                                         leaf_at, flag));
            LG_TRY_CUDA(excl_scan(flag, t, pos, sums, totals, st));
            LG_TRY_CUDA(launch_dependent(init_clusters_kernel, (t + kTB - 1) / kTB, kTB, 0, st, d_nodes, leaf_at,
                                         flag, pos, t, tn, cid, cbox));
            LG_TRY_CUDA(cudaGetLastError());
            LG_TRY_CUDA(cudaMemcpyAsync(&c, totals, sizeof(int), cudaMemcpyDeviceToHost, st));
            LG_TRY_CUDA(cudaStreamSynchronize(st));
            if (c != L) return set_error(LG_ERR_INVALID, "render tree: %d leaves by range start, %d expected", c, L);
        }
        // Rounds run kRoundsPerCheck at a time on a device-held count, grids sized by the last count read back (an
        // upper bound: rounds only merge); the host reads the state between groups.
        constexpr int kRoundsPerCheck = 8;
        int* sbuf[2] = {totals + 8, totals + 16};  // double-buffered state {c, next node id, error}
        int* ksums = sums + ((size_t)t / kTB + 2);  // the keep flags' block sums beside the merge flags'
        int cur = 0;
        int hstate[3] = {c, L, 0};
        LG_TRY_CUDA(cudaMemcpyAsync(sbuf[0], hstate, sizeof(hstate), cudaMemcpyHostToDevice, st));
        while (hstate[0] > kTailClusters)
        {
            const int gc = (hstate[0] + kTB - 1) / kTB;
            for (int k = 0; k < kRoundsPerCheck; ++k)
            {
                const int* sc = sbuf[cur];
                int* sn = sbuf[cur ^ 1];
                LG_TRY_CUDA(launch_dependent(nn_kernel, gc, kTB, 0, st, cbox, sc, nn));
                LG_TRY_CUDA(launch_dependent(round_flags_kernel, gc, kTB, 0, st, nn, sc, mflag, kflag, midx, kpos,
                                             sums, ksums));
                LG_TRY_CUDA(launch_dependent(round_sums_kernel, 1, kSumThreads, 0, st, sums, ksums, gc, sc, sn));
                LG_TRY_CUDA(launch_dependent(round_apply_kernel, gc, kTB, 0, st, nn, sc, mflag, kflag, midx, kpos,
                                             sums, ksums, cid, cbox, tn, cid2, cbox2));
                LG_TRY_CUDA(cudaGetLastError());
                int* ti = cid; cid = cid2; cid2 = ti;
                Box* tb = cbox; cbox = cbox2; cbox2 = tb;
                cur ^= 1;
            }
            LG_TRY_CUDA(cudaMemcpyAsync(hstate, sbuf[cur], sizeof(hstate), cudaMemcpyDeviceToHost, st));
            LG_TRY_CUDA(cudaStreamSynchronize(st));
            if (hstate[2]) return set_error(LG_ERR_DEVICE, "render tree: a clustering round merged nothing");
        }
        int* droot = totals + 24;
        LG_TRY_CUDA(cudaFuncSetAttribute((const void*)rounds_tail_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                         (int)sizeof(TailShared)));
        LG_TRY_CUDA(launch_dependent(rounds_tail_kernel, 1, kTailThreads, (int)sizeof(TailShared), st, cid, cbox,
                                     sbuf[cur], tn, droot));
        LG_TRY_CUDA(cudaGetLastError());
        LG_TRY_CUDA(cudaMemcpyAsync(hstate, sbuf[cur], sizeof(hstate), cudaMemcpyDeviceToHost, st));
        LG_TRY_CUDA(cudaMemcpyAsync(&root, droot, sizeof(int), cudaMemcpyDeviceToHost, st));
        LG_TRY_CUDA(cudaStreamSynchronize(st));
        if (hstate[2]) return set_error(LG_ERR_DEVICE, "render tree: a clustering round merged nothing");
        const int next_id = hstate[1];
        if (next_id != n_nodes) return set_error(LG_ERR_DEVICE, "render tree: %d nodes, %d expected", next_id, n_nodes);
        src = tn;
    }
    // Depth order: a stable sort of node ids by depth (ids ascending within a depth).
    LG_TRY_CUDA(cudaMemsetAsync(parent, 0xff, sizeof(int) * (size_t)n_nodes, st));
    LG_TRY_CUDA(launch_dependent(parent_of_kernel, g, kTB, 0, st, src, n_nodes, parent));
    LG_TRY_CUDA(launch_dependent(depth_of_kernel, g, kTB, 0, st, n_nodes, root, parent, depth, ids));
    LG_TRY_CUDA(cudaGetLastError());
    const RadixSortScratch rs = radix_sort_bind(sort_mem, (size_t)n_nodes);
    LG_TRY_CUDA(radix_sort_pairs(depth, ids, (size_t)n_nodes, 0, 8, rs, st));
    uint32_t max_depth = 0;
    LG_TRY_CUDA(cudaMemcpyAsync(&max_depth, depth + n_nodes - 1, sizeof(uint32_t), cudaMemcpyDeviceToHost, st));
    LG_TRY_CUDA(launch_dependent(rank_kernel, g, kTB, 0, st, ids, n_nodes, newpos));
    LG_TRY_CUDA(launch_dependent(emit_kernel, (n_nodes + kEmitNodes - 1) / kEmitNodes, kTB, 0, st, src, ids, newpos,
                                 n_nodes, d_out));
    LG_TRY_CUDA(launch_dependent(level_start_kernel, 1, kTB, 0, st, rs.hist, n_nodes, d_level_start));
    LG_TRY_CUDA(cudaMemcpyAsync(level_start_host, d_level_start, 257 * sizeof(int), cudaMemcpyDeviceToHost, st));
    LG_TRY_CUDA(cudaGetLastError());
    LG_TRY_CUDA(cudaStreamSynchronize(st));
    if (max_depth >= 255u) return set_error(LG_ERR_CAPACITY, "render tree: depth over 254");
    *levels = (int)max_depth + 1;
    return LG_OK;
}
}  // namespace lg
