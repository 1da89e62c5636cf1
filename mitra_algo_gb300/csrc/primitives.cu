// SPDX-License-Identifier: MPL-2.0
#include "primitives.cuh"

namespace sym {
namespace {

constexpr int kScanThreads = 256;
constexpr int kScanItems = 8;
constexpr int kScanTile = kScanThreads * kScanItems;

// Block-wide exclusive scan of one value per thread; returns the block total.
__device__ uint64_t block_exclusive(uint64_t v, uint64_t &total) {
  __shared__ uint64_t warp_sums[32];
  int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  uint64_t x = v;
  for (int o = 1; o < 32; o <<= 1) {
    uint64_t y = __shfl_up_sync(0xffffffffu, x, o);
    if (lane >= o) x += y;
  }
  if (lane == 31) warp_sums[warp] = x;
  __syncthreads();
  int warps = blockDim.x >> 5;
  if (warp == 0) {
    uint64_t s = lane < warps ? warp_sums[lane] : 0;
    for (int o = 1; o < 32; o <<= 1) {
      uint64_t y = __shfl_up_sync(0xffffffffu, s, o);
      if (lane >= o) s += y;
    }
    if (lane < warps) warp_sums[lane] = s;
  }
  __syncthreads();
  uint64_t before = warp ? warp_sums[warp - 1] : 0;
  total = warp_sums[warps - 1];
  __syncthreads();
  return before + x - v;
}

__global__ void tile_sums(const uint64_t *in, uint64_t n, uint64_t *partial) {
  chained();
  uint64_t base = uint64_t(blockIdx.x) * kScanTile + threadIdx.x * kScanItems;
  uint64_t s = 0;
  for (int k = 0; k < kScanItems; ++k)
    if (base + k < n) s += in[base + k];
  uint64_t total;
  block_exclusive(s, total);
  if (threadIdx.x == 0) partial[blockIdx.x] = total;
}

// One block scans `count` partial sums in place (exclusive) sequentially in
// chunks of blockDim.
__global__ void scan_partials(uint64_t *partial, uint64_t count) {
  chained();
  __shared__ uint64_t carry;
  if (threadIdx.x == 0) carry = 0;
  __syncthreads();
  for (uint64_t at = 0; at < count; at += blockDim.x) {
    uint64_t i = at + threadIdx.x;
    uint64_t v = i < count ? partial[i] : 0, total;
    uint64_t ex = block_exclusive(v, total);
    if (i < count) partial[i] = carry + ex;
    __syncthreads();
    if (threadIdx.x == 0) carry += total;
    __syncthreads();
  }
}

__global__ void tile_scan(const uint64_t *in, uint64_t n, const uint64_t *partial,
                          uint64_t *out) {
  chained();
  uint64_t base = uint64_t(blockIdx.x) * kScanTile + threadIdx.x * kScanItems;
  uint64_t v[kScanItems], s = 0;
  for (int k = 0; k < kScanItems; ++k) {
    v[k] = base + k < n ? in[base + k] : 0;
    s += v[k];
  }
  uint64_t total;
  uint64_t run = block_exclusive(s, total) + partial[blockIdx.x];
  for (int k = 0; k < kScanItems; ++k) {
    if (base + k < n) out[base + k] = run;
    run += v[k];
  }
  if (base < n && base + kScanItems >= n) out[n] = run;  // thread holding the last item
}

// The whole scan in one block, for the short ones (a radix pass over up to
// 81,920 keys scans its histogram of 256 digits per 1,280 keys): warp w takes
// 32 x kBlockItems consecutive values, round by round, and two barriers join the
// warps.  One launch of 4 us in place of three of 2.5 to 4 each.
constexpr int kBlockItems = 16, kBlockScan = 1024 * kBlockItems;
__global__ void __launch_bounds__(1024) scan_block(const uint64_t *in, unsigned n, uint64_t *out) {
  chained();
  __shared__ uint64_t warp_sums[32];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const unsigned per = (n + 1023) / 1024;  // rounds of a warp
  const unsigned base = warp * per * 32 + lane;
  uint64_t v[kBlockItems], run = 0;
#pragma unroll
  for (unsigned r = 0; r < kBlockItems; ++r) {
    const unsigned i = base + r * 32;
    v[r] = r < per && i < n ? in[i] : 0;
  }
#pragma unroll
  for (unsigned r = 0; r < kBlockItems; ++r)
    if (r < per) {  // v becomes the values before it in the warp's share
      uint64_t x = v[r];
      for (int o = 1; o < 32; o <<= 1) {
        const uint64_t y = __shfl_up_sync(0xffffffffu, x, o);
        if (lane >= o) x += y;
      }
      v[r] = run + x - v[r];
      run += __shfl_sync(0xffffffffu, x, 31);
    }
  if (lane == 0) warp_sums[warp] = run;
  __syncthreads();
  if (warp == 0) {
    const uint64_t own = warp_sums[lane];
    uint64_t x = own;
    for (int o = 1; o < 32; o <<= 1) {
      const uint64_t y = __shfl_up_sync(0xffffffffu, x, o);
      if (lane >= o) x += y;
    }
    warp_sums[lane] = x - own;
    if (lane == 31) out[n] = x;
  }
  __syncthreads();
  const uint64_t before = warp_sums[warp];
#pragma unroll
  for (unsigned r = 0; r < kBlockItems; ++r) {
    const unsigned i = base + r * 32;
    if (r < per && i < n) out[i] = before + v[r];
  }
}

// ---------------------------------------------------------------- radix sort
// Keys per block: more make longer runs of a digit (coalescing), fewer leave
// registers and shared memory for more warps, which is what the scatter waits
// for.  2.5e7 votes, a pass's scatter and histogram: 58 us with 4 rounds or 5, 67
// with 8 (2,048 keys), 72 with 12; 4 make the histograms' scan larger.
constexpr int kSortWarps = 8;
constexpr int kSortRounds = 5;                       // 32-key rounds per warp
constexpr int kSortTile = kSortWarps * kSortRounds * 32;  // 1280 keys per block

__global__ void radix_histogram(const uint64_t *keys, uint64_t n, int shift, uint64_t *hist,
                                unsigned blocks) {
  chained();
  __shared__ unsigned counts[256];
  for (int d = threadIdx.x; d < 256; d += blockDim.x) counts[d] = 0;
  __syncthreads();
  uint64_t base = uint64_t(blockIdx.x) * kSortTile;
  for (int i = threadIdx.x; i < kSortTile; i += blockDim.x)
    if (base + i < n) atomicAdd(&counts[(keys[base + i] >> shift) & 0xff], 1u);
  __syncthreads();
  for (int d = threadIdx.x; d < 256; d += blockDim.x)
    hist[uint64_t(d) * blocks + blockIdx.x] = counts[d];
}

// Stable scatter: warp w ranks its 160 keys round by round (in input order),
// warps are then ordered by their index, blocks by the scanned histogram.
// The block's keys are first placed in digit order in shared memory, so the
// global writes of each digit are one consecutive run.
__global__ void __launch_bounds__(kSortWarps * 32) radix_scatter(
    const uint64_t *keys, const int32_t *vals, uint64_t n, int shift, const uint64_t *offsets,
    unsigned blocks, uint64_t *keys_out, int32_t *vals_out) {
  chained();
  __shared__ unsigned warp_count[kSortWarps][256];
  __shared__ unsigned digit_start[256];
  __shared__ uint64_t skey[kSortTile];
  __shared__ int32_t sval[kSortTile];
  int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  for (int d = threadIdx.x; d < kSortWarps * 256; d += blockDim.x)
    (&warp_count[0][0])[d] = 0;
  __syncthreads();
  uint64_t base = uint64_t(blockIdx.x) * kSortTile + uint64_t(warp) * kSortRounds * 32;
  uint64_t key[kSortRounds];
  int32_t val[kSortRounds];
  unsigned rank[kSortRounds];
  unsigned lt = (1u << lane) - 1;
  for (int r = 0; r < kSortRounds; ++r) {
    uint64_t i = base + r * 32 + lane;
    bool live = i < n;
    key[r] = live ? keys[i] : 0;
    val[r] = live ? vals[i] : 0;
    unsigned digit = live ? unsigned((key[r] >> shift) & 0xff) : 256u;
    unsigned peers = __match_any_sync(0xffffffffu, digit);
    unsigned before = digit < 256 ? warp_count[warp][digit] : 0;
    rank[r] = before + __popc(peers & lt);
    __syncwarp();
    if (live && (peers & lt) == 0) warp_count[warp][digit] = before + __popc(peers);
    __syncwarp();
  }
  __syncthreads();
  // per digit: each warp's start among the block's keys of that digit, and
  // the digit's count; then the digits' starts in the block
  unsigned digit_total = 0;
  if (threadIdx.x < 256) {
    const int d = threadIdx.x;
    for (int w = 0; w < kSortWarps; ++w) {
      unsigned c = warp_count[w][d];
      warp_count[w][d] = digit_total;
      digit_total += c;
    }
  }
  uint64_t all;
  const uint64_t start = block_exclusive(digit_total, all);  // blockDim.x == 256
  if (threadIdx.x < 256) digit_start[threadIdx.x] = unsigned(start);
  __syncthreads();
  for (int r = 0; r < kSortRounds; ++r) {
    uint64_t i = base + r * 32 + lane;
    if (i >= n) continue;
    unsigned digit = unsigned((key[r] >> shift) & 0xff);
    unsigned pos = digit_start[digit] + warp_count[warp][digit] + rank[r];
    skey[pos] = key[r];
    sval[pos] = val[r];
  }
  __syncthreads();
  const uint64_t block_base = uint64_t(blockIdx.x) * kSortTile;
  const unsigned count = unsigned(n - block_base < uint64_t(kSortTile) ? n - block_base : kSortTile);
  for (unsigned j = threadIdx.x; j < count; j += blockDim.x) {
    const uint64_t k = skey[j];
    const unsigned digit = unsigned((k >> shift) & 0xff);
    const uint64_t dst = offsets[uint64_t(digit) * blocks + blockIdx.x] + (j - digit_start[digit]);
    keys_out[dst] = k;
    vals_out[dst] = sval[j];
  }
}

// The whole sort in one block for up to kBlockSort keys, kept in registers
// (ITEMS per thread, warp w the 32 x ITEMS consecutive ones of its share) and
// exchanged through shared memory after every pass; a pass whose digit all
// keys share is skipped.  The padding behind the last key has the largest key
// and stays last.  Bound by its barriers and the rank of each key; a pass takes 3
// to 9 us by the number of keys, where the three launches of a pass over the
// whole device take some 16: 2,000 64-bit keys 27 us, 2,562 41, 8,192 68, all
// some 130 by passes over the device, which cost the same up to here and are
// the better ones for more.
constexpr int kBlockSort = 8192;
template <int ITEMS>
__global__ void __launch_bounds__(1024) sort_block(const uint64_t *keys, const int32_t *vals, unsigned n,
                                                   int begin_bit, int end_bit, uint64_t *keys_out,
                                                   int32_t *vals_out) {
  chained();
  constexpr int kWarps = 32;
  extern __shared__ __align__(16) uint8_t sort_smem[];
  uint64_t *skey = reinterpret_cast<uint64_t *>(sort_smem);                        // 1024 x ITEMS
  int32_t *sval = reinterpret_cast<int32_t *>(sort_smem + size_t(1024) * ITEMS * 8);
  unsigned *counts = reinterpret_cast<unsigned *>(sort_smem + size_t(1024) * ITEMS * 12);  // [warp][256]
  unsigned *start = counts + kWarps * 256;
  __shared__ unsigned long long varies;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const unsigned base = warp * 32 * ITEMS + lane, lt = (1u << lane) - 1;
  uint64_t key[ITEMS];
  int32_t val[ITEMS];
  if (threadIdx.x == 0) varies = 0;
  __syncthreads();
  const uint64_t first = keys[0];
  uint64_t differ = 0;
#pragma unroll
  for (int r = 0; r < ITEMS; ++r) {
    const unsigned i = base + r * 32;
    key[r] = i < n ? keys[i] : ~0ull;
    val[r] = i < n ? vals[i] : 0;
    if (i < n) differ |= key[r] ^ first;
  }
  for (int o = 16; o; o >>= 1) differ |= __shfl_xor_sync(0xffffffffu, differ, o);
  if (lane == 0) atomicOr(&varies, (unsigned long long)differ);
  __syncthreads();
  const uint64_t bits = varies;
  for (int shift = begin_bit; shift < end_bit; shift += 8) {
    if (!((bits >> shift) & 0xff)) continue;
    for (unsigned d = threadIdx.x; d < kWarps * 256; d += 1024) counts[d] = 0;
    __syncthreads();
    unsigned rank[ITEMS];
    unsigned *mine = counts + warp * 256;
#pragma unroll
    for (int r = 0; r < ITEMS; ++r) {
      const unsigned digit = unsigned(key[r] >> shift) & 0xff;
      const unsigned peers = __match_any_sync(0xffffffffu, digit);
      const unsigned before = mine[digit];
      rank[r] = before + __popc(peers & lt);
      __syncwarp();
      if ((peers & lt) == 0) mine[digit] = before + __popc(peers);
      __syncwarp();
    }
    __syncthreads();
    unsigned total = 0;
    if (threadIdx.x < 256)
      for (int w = 0; w < kWarps; ++w) {
        const unsigned c = counts[w * 256 + threadIdx.x];
        counts[w * 256 + threadIdx.x] = total;
        total += c;
      }
    uint64_t all;
    const uint64_t before = block_exclusive(total, all);
    if (threadIdx.x < 256) start[threadIdx.x] = unsigned(before);
    __syncthreads();
#pragma unroll
    for (int r = 0; r < ITEMS; ++r) {
      const unsigned digit = unsigned(key[r] >> shift) & 0xff;
      const unsigned pos = start[digit] + mine[digit] + rank[r];
      skey[pos] = key[r], sval[pos] = val[r];
    }
    __syncthreads();
#pragma unroll
    for (int r = 0; r < ITEMS; ++r) key[r] = skey[base + r * 32], val[r] = sval[base + r * 32];
  }
#pragma unroll
  for (int r = 0; r < ITEMS; ++r) {
    const unsigned i = base + r * 32;
    if (i < n) keys_out[i] = key[r], vals_out[i] = val[r];
  }
}

template <int ITEMS>
void launch_sort_block(Call &call, const uint64_t *keys, const int32_t *values, uint64_t *keys_out,
                       int32_t *values_out, uint64_t n, int begin_bit, int end_bit) {
  constexpr size_t smem = size_t(1024) * ITEMS * 12 + (32 + 1) * 256 * sizeof(unsigned);
  call.allow_shared(sort_block<ITEMS>, smem);
  launch_chained(call.stream(), sort_block<ITEMS>, 1, 1024, smem, keys, values, unsigned(n), begin_bit, end_bit,
                 keys_out, values_out);
  call.launched();
}

__global__ void flags_to_counts(const uint8_t *flags, uint64_t n, uint64_t *counts) {
  chained();
  uint64_t i = uint64_t(blockIdx.x) * blockDim.x + threadIdx.x;
  if (i < n) counts[i] = flags[i] != 0;
}

__global__ void scatter_flagged(const uint8_t *flags, const int32_t *values, uint64_t n,
                                const uint64_t *pos, int32_t *out, uint64_t *count) {
  chained();
  uint64_t i = uint64_t(blockIdx.x) * blockDim.x + threadIdx.x;
  if (i < n && flags[i]) out[pos[i]] = values ? values[i] : int32_t(i);
  if (i == 0) *count = pos[n];
}

}  // namespace

void exclusive_scan(Call &call, const uint64_t *in, uint64_t *out, uint64_t n) {
  if (n == 0) {
    SYM_CUDA(cudaMemsetAsync(out, 0, sizeof(uint64_t), call.stream()));
    return;
  }
  if (n <= kBlockScan) {
    launch_chained(call.stream(), scan_block, 1, 1024, 0, in, unsigned(n), out);
    call.launched();
    return;
  }
  unsigned tiles = static_cast<unsigned>((n + kScanTile - 1) / kScanTile);
  uint64_t *partial = call.alloc<uint64_t>(tiles);
  launch_chained(call.stream(), tile_sums, tiles, kScanThreads, 0, in, n, partial);
  launch_chained(call.stream(), scan_partials, 1, 1024, 0, partial, tiles);
  launch_chained(call.stream(), tile_scan, tiles, kScanThreads, 0, in, n, partial, out);
  call.launched(3);
}

void radix_sort_pairs(Call &call, const uint64_t *keys, const int32_t *values,
                      uint64_t *keys_out, int32_t *values_out, uint64_t n, int key_bits, int first_bit) {
  if (n == 0) return;
  const int passes = (key_bits - first_bit + 7) / 8;
  if (n <= kBlockSort) {
    const auto sort = n <= 1024   ? launch_sort_block<1>
                      : n <= 2048 ? launch_sort_block<2>
                      : n <= 4096 ? launch_sort_block<4>
                                  : launch_sort_block<8>;
    return sort(call, keys, values, keys_out, values_out, n, first_bit, first_bit + 8 * passes);
  }
  unsigned blocks = static_cast<unsigned>((n + kSortTile - 1) / kSortTile);
  uint64_t hist_n = uint64_t(blocks) * 256;
  uint64_t *hist = call.alloc<uint64_t>(hist_n);
  uint64_t *offsets = call.alloc<uint64_t>(hist_n + 1);
  uint64_t *kbuf = call.alloc<uint64_t>(n);
  int32_t *vbuf = call.alloc<int32_t>(n);
  // ping-pong so that the last pass writes keys_out/values_out
  const uint64_t *ksrc = keys;
  const int32_t *vsrc = values;
  for (int p = 0; p < passes; ++p) {
    bool last_to_out = ((passes - 1 - p) % 2) == 0;
    uint64_t *kdst = last_to_out ? keys_out : kbuf;
    int32_t *vdst = last_to_out ? values_out : vbuf;
    int shift = first_bit + 8 * p;
    launch_chained(call.stream(), radix_histogram, blocks, 256, 0, ksrc, n, shift, hist, blocks);
    exclusive_scan(call, hist, offsets, hist_n);
    launch_chained(call.stream(), radix_scatter, blocks, kSortWarps * 32, 0, ksrc, vsrc, n, shift, offsets,
                   blocks, kdst, vdst);
    call.launched(2);
    ksrc = kdst;
    vsrc = vdst;
  }
}

void compact_values(Call &call, const uint8_t *flags, const int32_t *values, uint64_t n,
                    int32_t *out, uint64_t *count) {
  if (n == 0) {
    SYM_CUDA(cudaMemsetAsync(count, 0, sizeof(uint64_t), call.stream()));
    return;
  }
  uint64_t *counts = call.alloc<uint64_t>(n);
  uint64_t *pos = call.alloc<uint64_t>(n + 1);
  launch_chained(call.stream(), flags_to_counts, blocks_for(n), kThreads, 0, flags, n, counts);
  exclusive_scan(call, counts, pos, n);
  launch_chained(call.stream(), scatter_flagged, blocks_for(n), kThreads, 0, flags, values, n, pos, out, count);
  call.launched(2);
}

void compact_indices(Call &call, const uint8_t *flags, uint64_t n, int32_t *out,
                     uint64_t *count) {
  compact_values(call, flags, nullptr, n, out, count);
}

}  // namespace sym
