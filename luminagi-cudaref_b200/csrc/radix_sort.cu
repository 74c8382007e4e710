// radix_sort.cu -- see radix_sort.cuh.
//
// Bound by latency at the sizes the library sorts (8 MB of pairs stay in L2): a
// pass is one round of key loads, the ranking, the look-back and the writes.
// One B200, 30-bit keys (4 passes, launched one after the other): 59 us for 1,050,972 pairs and 21 us for
// 20,500.  With three launches a pass (per-tile histogram, scan of the
// [digit][tile] table, scatter with a block-wide sync per 256 keys) a pass took 30
// and 20 us.
#include "radix_sort.cuh"

#include <algorithm>

#include "pdl.cuh"

namespace lg
{
namespace
{
constexpr int kHistThreads = 256;

// Keys per tile.  A sort's tiles start together, so each looks back over many
// unfinished ones: work that grows with the square of the tiles, 134 MB of reads a pass
// at 1,050,972 keys in tiles of 2,048.  So the tiles grow with n to stay near one
// per SM: 15 us a pass in tiles of 8,192 there, 22 us in tiles of 2,048.
int tile_keys(size_t n) { return n <= 148 * 1024 ? 1024 : (n <= 148 * 2048 ? 2048 : (n <= 148 * 4096 ? 4096 : 8192)); }
size_t tiles_for(size_t n) { return (n + tile_keys(n) - 1) / tile_keys(n); }
// Most tiles of a sort of n pairs or fewer: just below the size from which tiles are larger there are 148.
size_t tiles_within(size_t n) { return std::max(tiles_for(n), std::min<size_t>((n + 1023) / 1024, 148)); }
size_t align256(size_t b) { return (b + 255) & ~(size_t)255; }

// Digit totals of every pass in one read of the keys.
__global__ void __launch_bounds__(kHistThreads) hist_kernel(const uint32_t* __restrict__ keys, size_t n, int begin_bit,
                                                        int end_bit, uint32_t* __restrict__ hist)
{
    __shared__ uint32_t h[kRadixMaxPasses][256];
    for (int i = threadIdx.x; i < kRadixMaxPasses * 256; i += kHistThreads) (&h[0][0])[i] = 0;
    begin_after_predecessors();
    __syncthreads();
    for (size_t i = (size_t)blockIdx.x * kHistThreads + threadIdx.x; i < n; i += (size_t)gridDim.x * kHistThreads)
    {
        const uint32_t key = keys[i];
        int p = 0;
        for (int shift = begin_bit; shift < end_bit; shift += 8, ++p)
        {
            const int bits = min(8, end_bit - shift);
            atomicAdd(&h[p][(key >> shift) & ((1u << bits) - 1u)], 1u);
        }
    }
    __syncthreads();
    for (int i = threadIdx.x; i < kRadixMaxPasses * 256; i += kHistThreads)
    {
        const uint32_t c = (&h[0][0])[i];
        if (c) atomicAdd(&hist[i], c);
    }
}

// A published count: two flag bits over the value.
constexpr uint32_t kAggregate = 1u << 30;  // this tile's own count of the digit
constexpr uint32_t kInclusive = 2u << 30;  // the count of all tiles up to this one
constexpr uint32_t kValueMask = (1u << 30) - 1u;
constexpr int kLookBack = 8;               // predecessors read at a time

// Exclusive scan over the first 256 threads of one value each (every thread of the block calls it).
__device__ __forceinline__ uint32_t digit_excl(uint32_t v, uint32_t* warp_sums)
{
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    uint32_t x = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1)
    {
        const uint32_t y = __shfl_up_sync(0xffffffffu, x, o);
        if (lane >= o) x += y;
    }
    if (lane == 31) warp_sums[warp] = x;
    __syncthreads();
    uint32_t before = 0;
    for (int w = 0; w < warp; ++w) before += warp_sums[w];
    return before + x - v;
}

template <int kThreads, int kItems>
struct PassShared
{
    static constexpr int kWarps = kThreads / 32;
    uint32_t warp_cnt[kWarps][256];  // per-warp digit counts, then their exclusive prefix across warps
    uint32_t tile_start[256];        // first place of the digit within the tile
    uint32_t global_base[256];       // global place of the digit's first key, less tile_start
    uint32_t sums[2][kWarps];
    uint32_t tile, pad[3];
    uint32_t key[kThreads * kItems], val[kThreads * kItems];
};

template <int kThreads, int kItems, bool kIota>
__global__ void __launch_bounds__(kThreads) pass_kernel(const uint32_t* __restrict__ keys_in,
                                                        const uint32_t* __restrict__ vals_in,
                                                        uint32_t* __restrict__ keys_out,
                                                        uint32_t* __restrict__ vals_out, uint32_t n, int shift,
                                                        int bits, const uint32_t* __restrict__ hist, uint32_t* state,
                                                        uint32_t* ticket, int poll_limit)
{
    constexpr int kTile = kThreads * kItems, kWarps = kThreads / 32;
    static_assert(kThreads >= 256, "one digit per thread");
    extern __shared__ __align__(16) unsigned char pass_mem[];
    PassShared<kThreads, kItems>& sh = *reinterpret_cast<PassShared<kThreads, kItems>*>(pass_mem);
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    for (int i = tid; i < kWarps * 256; i += kThreads) (&sh.warp_cnt[0][0])[i] = 0;
    begin_after_predecessors();
    if (tid == 0) sh.tile = atomicAdd(ticket, 1u);
    const uint32_t digit_total = tid < 256 ? hist[tid] : 0u;
    __syncthreads();
    const uint32_t tile = sh.tile;
    const uint32_t mask = (1u << bits) - 1u;
    const uint32_t base = tile * (uint32_t)kTile;
    const uint32_t count = min((uint32_t)kTile, n - base);
    const uint32_t lt_mask = (1u << lane) - 1u;

    // Keys in (warp, item, lane) order, so a warp ranks its own run of 32 * kItems keys without a block sync.
    uint32_t key[kItems], val[kItems], rank[kItems];
#pragma unroll
    for (int k = 0; k < kItems; ++k)
    {
        const uint32_t i = (uint32_t)(warp * kItems + k) * 32u + lane;
        key[k] = i < count ? keys_in[base + i] : 0u;
        val[k] = kIota ? base + i : (i < count ? vals_in[base + i] : 0u);
    }
#pragma unroll
    for (int k = 0; k < kItems; ++k)
    {
        const uint32_t i = (uint32_t)(warp * kItems + k) * 32u + lane;
        const bool valid = i < count;
        // keys past the end get digit 256, which matches no real one
        const uint32_t digit = valid ? ((key[k] >> shift) & mask) : 256u;
        const uint32_t peers = __match_any_sync(0xffffffffu, digit);
        const uint32_t before = valid ? sh.warp_cnt[warp][digit] : 0u;
        __syncwarp();
        if (valid && (peers & lt_mask) == 0) sh.warp_cnt[warp][digit] = before + __popc(peers);
        __syncwarp();
        rank[k] = before + __popc(peers & lt_mask);
    }
    __syncthreads();

    // One digit per thread: the tile's count, published for the tiles after it.
    uint32_t total = 0;
    volatile uint32_t* mine = state + (size_t)tile * 256 + tid;
    if (tid < 256)
    {
#pragma unroll
        for (int w = 0; w < kWarps; ++w)
        {
            const uint32_t c = sh.warp_cnt[w][tid];
            sh.warp_cnt[w][tid] = total;
            total += c;
        }
        *mine = (tile == 0 ? kInclusive : kAggregate) | total;
    }
    const uint32_t start = digit_excl(total, sh.sums[0]);
    const uint32_t digit_base = digit_excl(digit_total, sh.sums[1]);
    if (tid < 256)
    {
        uint32_t before = 0;
        if (tile > 0)
        {
            // Add up the counts of the tiles before, nearest first, until one has its inclusive count.  Past the
            // poll limit a count that is not there is taken from that tile's keys themselves, which no tile of this
            // pass writes: the sort is right whatever a wait does, and what runs after it may rely on it.
            int j = (int)tile - 1, polls = 0;
            bool done = false;
            while (!done)
            {
                uint32_t v[kLookBack];
#pragma unroll
                for (int b = 0; b < kLookBack; ++b)
                    v[b] = j - b >= 0 ? *(volatile uint32_t*)(state + (size_t)(j - b) * 256 + tid) : 0u;
#pragma unroll
                for (int b = 0; b < kLookBack; ++b)
                {
                    if (done || j < 0 || (v[b] >> 30) == 0) break;
                    before += v[b] & kValueMask;
                    if (v[b] >> 30 == 2) done = true;
                    --j;
                }
                if (!done && polls++ >= poll_limit)
                {
                    polls = poll_limit;
                    const uint32_t* of_tile = keys_in + (size_t)j * kTile;  // a whole tile: it is not the last
                    for (int i = 0; i < kTile; ++i) before += ((of_tile[i] >> shift) & mask) == (uint32_t)tid ? 1u : 0u;
                    done = --j < 0;
                }
            }
            *mine = kInclusive | ((before + total) & kValueMask);
        }
        sh.tile_start[tid] = start;
        sh.global_base[tid] = digit_base + before - start;
    }
    __syncthreads();
#pragma unroll
    for (int k = 0; k < kItems; ++k)
    {
        const uint32_t i = (uint32_t)(warp * kItems + k) * 32u + lane;
        if (i >= count) continue;
        const uint32_t digit = (key[k] >> shift) & mask;
        const uint32_t at = sh.tile_start[digit] + sh.warp_cnt[warp][digit] + rank[k];
        sh.key[at] = key[k];
        sh.val[at] = val[k];
    }
    __syncthreads();
    for (uint32_t i = tid; i < count; i += kThreads)
    {
        const uint32_t k = sh.key[i];
        const uint32_t pos = sh.global_base[(k >> shift) & mask] + i;
        keys_out[pos] = k;
        vals_out[pos] = sh.val[i];
    }
}

struct PassArgs
{
    const uint32_t *ki, *vi;
    uint32_t *ko, *vo;
    uint32_t n;
    int shift, bits;
    const uint32_t* hist;
    uint32_t *state, *ticket;
    int poll_limit;
};
template <int kThreads, int kItems>
cudaError_t launch_pass(const PassArgs& a, bool iota, size_t tiles, cudaStream_t st)
{
    const int smem = (int)sizeof(PassShared<kThreads, kItems>);
    auto k = iota ? pass_kernel<kThreads, kItems, true> : pass_kernel<kThreads, kItems, false>;
    const cudaError_t e = cudaFuncSetAttribute((const void*)k, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
    if (e != cudaSuccess) return e;
    return launch_dependent(k, (unsigned)tiles, kThreads, smem, st, a.ki, a.vi, a.ko, a.vo, a.n, a.shift, a.bits, a.hist,
                            a.state, a.ticket, a.poll_limit);
}
}  // namespace

size_t radix_sort_scratch_bytes(size_t n)
{
    const size_t t = tiles_within(n ? n : 1);
    return align256(n * 4) * 2 + align256(kRadixMaxPasses * 256 * 4 + 64) + kRadixMaxPasses * t * 256 * 4 + 512;
}

RadixSortScratch radix_sort_bind(void* base, size_t n)
{
    char* p = (char*)(((uintptr_t)base + 255) & ~(uintptr_t)255);
    RadixSortScratch s;
    s.keys_alt = (uint32_t*)p;
    p += align256(n * 4);
    s.vals_alt = (uint32_t*)p;
    p += align256(n * 4);
    s.hist = (uint32_t*)p;
    s.tickets = s.hist + kRadixMaxPasses * 256;
    p += align256(kRadixMaxPasses * 256 * 4 + 64);
    s.state = (uint32_t*)p;
    s.zero_bytes = (size_t)((char*)(s.state + kRadixMaxPasses * tiles_within(n ? n : 1) * 256) - (char*)s.hist);
    s.capacity = n;
    return s;
}

cudaError_t radix_sort_pairs(uint32_t* keys, uint32_t* vals, size_t n, int begin_bit, int end_bit,
                             const RadixSortScratch& s, cudaStream_t stream, bool counted, bool iota)
{
    if (n > s.capacity) return cudaErrorInvalidValue;
    if (!counted)
    {
        const cudaError_t e = cudaMemsetAsync(s.hist, 0, s.zero_bytes, stream);
        if (e != cudaSuccess) return e;
    }
    if (n <= 1 || end_bit <= begin_bit)
        return iota && n == 1 ? cudaMemsetAsync(vals, 0, 4, stream) : cudaSuccess;
    if (n >= (1ull << 30) || end_bit - begin_bit > 8 * kRadixMaxPasses) return cudaErrorInvalidValue;
    const size_t tiles = tiles_for(n);
    cudaError_t e = cudaSuccess;
    if (!counted)
    {
        const size_t blocks = (n + kHistThreads * 4 - 1) / (kHistThreads * 4);
        e = launch_dependent(hist_kernel, (unsigned)(blocks < 592 ? blocks : 592), kHistThreads, 0, stream, keys, n,
                             begin_bit, end_bit, s.hist);
        if (e != cudaSuccess) return e;
    }
    uint32_t *ki = keys, *vi = vals, *ko = s.keys_alt, *vo = s.vals_alt;
    int pass = 0;
    for (int shift = begin_bit; shift < end_bit; shift += 8, ++pass)
    {
        const int bits = (end_bit - shift) < 8 ? (end_bit - shift) : 8;
        const PassArgs a{ki, vi, ko, vo, (uint32_t)n, shift, bits, s.hist + pass * 256,
                         s.state + (size_t)pass * tiles * 256, s.tickets + pass, s.poll_limit};
        const bool first = iota && pass == 0;
        switch (tile_keys(n))
        {
            case 1024: e = launch_pass<256, 4>(a, first, tiles, stream); break;
            case 2048: e = launch_pass<256, 8>(a, first, tiles, stream); break;
            case 4096: e = launch_pass<512, 8>(a, first, tiles, stream); break;
            default: e = launch_pass<512, 16>(a, first, tiles, stream); break;
        }
        if (e != cudaSuccess) return e;
        uint32_t* t = ki; ki = ko; ko = t;
        t = vi; vi = vo; vo = t;
    }
    if (ki != keys)
    {
        e = cudaMemcpyAsync(keys, ki, n * 4, cudaMemcpyDeviceToDevice, stream);
        if (e != cudaSuccess) return e;
        e = cudaMemcpyAsync(vals, vi, n * 4, cudaMemcpyDeviceToDevice, stream);
    }
    return e;
}
}  // namespace lg
