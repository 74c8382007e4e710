// radix_sort.cuh -- stable LSD radix sort of (u32 key, u32 value) pairs.
//
// One launch per 8-bit digit ("onesweep": Adinets and Merrill, "Onesweep: A
// Faster Least Significant Digit Radix Sort for GPUs", 2022, on Merrill and
// Garland's decoupled look-back):
//   1. one pass over the keys counts every digit of every pass (a digit's
//      totals do not depend on the order of the keys), or the caller's own
//      kernel has counted them while it wrote the keys;
//   2. per digit, tiles of 1,024 to 8,192 keys, numbered in the order in which they
//      start: a tile ranks its keys in input order (warp match_any peers +
//      per-warp digit counts), publishes its digit counts, adds up the counts
//      of the tiles before it, and writes its keys through shared memory in
//      digit order.
// Stability makes the result a total order on (key, input position), which
// is what the BVH build relies on for a deterministic triangle order.
//
// A tile waits only for tiles that started before it, so every wait ends; it is
// bounded all the same, and a tile whose wait ran out counts the keys it waits
// for itself.
#pragma once
#include <cstddef>
#include <cstdint>

#include <cuda_runtime.h>

namespace lg
{
constexpr int kRadixMaxPasses = 4;
constexpr int kRadixPollLimit = 1 << 22;  // reads of counts not yet published before a tile counts for itself

struct RadixSortScratch
{
    uint32_t* keys_alt = nullptr;
    uint32_t* vals_alt = nullptr;
    // cleared before each sort, contiguous: digit totals per pass (4 x 256), start tickets per pass (4),
    // and per pass and tile the 256 published counts
    uint32_t* hist = nullptr;
    uint32_t* tickets = nullptr;
    uint32_t* state = nullptr;
    size_t zero_bytes = 0;  // of the cleared part, from hist on
    size_t capacity = 0;    // elements
    int poll_limit = kRadixPollLimit;
};

// Bytes of scratch needed for n elements, or any fewer.
size_t radix_sort_scratch_bytes(size_t n);
// Carves the scratch pointers out of `base` (aligned to 256 bytes).
RadixSortScratch radix_sort_bind(void* base, size_t n);

// Sorts keys/vals in place over bits [begin_bit, end_bit), n < 2^30 and at most
// s.capacity.  Returns a CUDA error.  `counted`: the cleared part of the scratch was cleared on `stream`
// and s.hist[pass * 256 + digit] already holds the digit totals.  `iota`:
// vals is written only, the values are the input positions.
cudaError_t radix_sort_pairs(uint32_t* keys, uint32_t* vals, size_t n, int begin_bit, int end_bit,
                             const RadixSortScratch& s, cudaStream_t stream, bool counted = false, bool iota = false);
}  // namespace lg
