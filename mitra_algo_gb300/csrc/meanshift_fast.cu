// SPDX-License-Identifier: MPL-2.0
// SIMT mean-shift (FP32 and FP64) over a Morton-chunked 6-D vote set.
#include "chunk_lists.cuh"
#include "meanshift_fast.cuh"
#include "primitives.cuh"

#include <algorithm>
#include <cmath>

namespace sym {
namespace {

// ------------------------------------------------------------ vote sort
__global__ void box_partials(const float *desc, uint64_t q, float *partial) {
  __shared__ float lo[6][256], hi[6][256];
  float l[6], h[6];
  for (int k = 0; k < 6; ++k) l[k] = INFINITY, h[k] = -INFINITY;
  for (uint64_t v = uint64_t(blockIdx.x) * blockDim.x + threadIdx.x; v < q;
       v += uint64_t(gridDim.x) * blockDim.x)
    for (int k = 0; k < 6; ++k) {
      float x = desc[v * 8 + k];
      l[k] = fminf(l[k], x), h[k] = fmaxf(h[k], x);
    }
  for (int k = 0; k < 6; ++k) lo[k][threadIdx.x] = l[k], hi[k][threadIdx.x] = h[k];
  __syncthreads();
  for (int s = 128; s; s >>= 1) {
    if (threadIdx.x < s)
      for (int k = 0; k < 6; ++k) {
        lo[k][threadIdx.x] = fminf(lo[k][threadIdx.x], lo[k][threadIdx.x + s]);
        hi[k][threadIdx.x] = fmaxf(hi[k][threadIdx.x], hi[k][threadIdx.x + s]);
      }
    __syncthreads();
  }
  if (threadIdx.x == 0)
    for (int k = 0; k < 6; ++k)
      partial[blockIdx.x * 12 + k] = lo[k][0], partial[blockIdx.x * 12 + 6 + k] = hi[k][0];
}

__global__ void box_final(const float *partial, int n, float *box) {
  int k = threadIdx.x;
  if (k >= 12) return;
  float v = k < 6 ? INFINITY : -INFINITY;
  for (int i = 0; i < n; ++i) v = k < 6 ? fminf(v, partial[i * 12 + k]) : fmaxf(v, partial[i * 12 + k]);
  box[k] = v;
}

// Morton key of a 6-D point over `bits` bits per coordinate (cells of
// 1/2^bits of the box; at most 10).
__device__ __forceinline__ uint64_t morton6(const float *x, const float *box, int bits = 10) {
  uint64_t key = 0;
  const int cells = 1 << bits;
  for (int k = 0; k < 6; ++k) {
    float lo = box[k], span = box[6 + k] - lo;
    float t = span > 0 ? (x[k] - lo) / span : 0.f;
    uint64_t cell = uint64_t(min(cells - 1, max(0, int(t * float(cells)))));
    for (int b = 0; b < bits; ++b) key |= ((cell >> b) & 1ull) << (6 * b + k);
  }
  return key;
}

// Votes are ordered by `bits` bits per coordinate (8 by default: a cell of
// the vote space is then ~1/256 of its extent, well under the bandwidth on
// the benchmark workloads, and the 48-bit key sorts in six radix passes).
__global__ void morton_keys(const float *desc, uint64_t q, const float *box, int bits,
                            uint64_t *keys, int32_t *idx) {
  uint64_t v = uint64_t(blockIdx.x) * blockDim.x + threadIdx.x;
  if (v >= q) return;
  keys[v] = morton6(desc + v * 8, box, bits);
  idx[v] = int32_t(v);
}

// dst row v = src row order[v]; rows of 8 values (32 or 64 bytes, and the
// buffers 16-byte aligned), moved as 16-byte words.
template <typename T>
__global__ void permute(const T *src, const int32_t *order, uint64_t q, T *dst) {
  uint64_t v = uint64_t(blockIdx.x) * blockDim.x + threadIdx.x;
  if (v >= q) return;
  uint64_t from = uint64_t(uint32_t(order[v]));
  constexpr int kWords = 8 * sizeof(T) / 16;
  const uint4 *s = reinterpret_cast<const uint4 *>(src + from * 8);
  uint4 w[kWords];
  for (int k = 0; k < kWords; ++k) w[k] = s[k];
  uint4 *d = reinterpret_cast<uint4 *>(dst + v * 8);
  for (int k = 0; k < kWords; ++k) d[k] = w[k];
}

__global__ void invert(const int32_t *order, uint64_t q, int32_t *rank) {
  uint64_t v = uint64_t(blockIdx.x) * blockDim.x + threadIdx.x;
  if (v < q) rank[order[v]] = int32_t(v);
}

// One warp per chunk: the chunk's box [lo0..lo5, hi0..hi5] and the boxes
// of its runs of kSubVotes votes (a run past q gets an empty box, lo = +inf
// and hi = -inf).  Lane l holds vote 32 r + l in round r, so a run is a
// group of consecutive lanes of one round.
__global__ void chunk_boxes(const float *desc, uint64_t q, uint64_t nchunks, float *cbox,
                            float *sbox) {
  uint64_t c = (uint64_t(blockIdx.x) * blockDim.x + threadIdx.x) >> 5;
  int lane = threadIdx.x & 31;
  if (c >= nchunks) return;
  float l[6], h[6];
  for (int k = 0; k < 6; ++k) l[k] = INFINITY, h[k] = -INFINITY;
  for (int r = 0; r < kChunk / 32; ++r) {
    const int j = 32 * r + lane;
    const uint64_t v = c * kChunk + j;
    const bool in = v < q;
    float a[6], b[6];
    for (int k = 0; k < 6; ++k) {
      const float x = in ? desc[v * 8 + k] : 0.f;
      a[k] = in ? x : INFINITY, b[k] = in ? x : -INFINITY;
    }
    for (int o = kSubVotes / 2; o; o >>= 1)
      for (int k = 0; k < 6; ++k) {
        a[k] = fminf(a[k], __shfl_xor_sync(0xffffffffu, a[k], o));
        b[k] = fmaxf(b[k], __shfl_xor_sync(0xffffffffu, b[k], o));
      }
    if (lane % kSubVotes == 0) {
      float *s = sbox + (c * kSubs + j / kSubVotes) * 12;
      for (int k = 0; k < 6; ++k) s[k] = a[k], s[6 + k] = b[k];
    }
    for (int k = 0; k < 6; ++k) l[k] = fminf(l[k], a[k]), h[k] = fmaxf(h[k], b[k]);
  }
  for (int o = 16; o >= kSubVotes; o >>= 1)
    for (int k = 0; k < 6; ++k) {
      l[k] = fminf(l[k], __shfl_xor_sync(0xffffffffu, l[k], o));
      h[k] = fmaxf(h[k], __shfl_xor_sync(0xffffffffu, h[k], o));
    }
  if (lane == 0)
    for (int k = 0; k < 6; ++k) cbox[c * 12 + k] = l[k], cbox[c * 12 + 6 + k] = h[k];
}

// One block per run of kBlockChunks chunks: the union of their boxes.
__global__ void __launch_bounds__(kBlockChunks) block_boxes(const float *cbox, uint64_t nchunks,
                                                            float *bbox) {
  __shared__ float part[kBlockChunks / 32][12];
  const uint64_t c = uint64_t(blockIdx.x) * kBlockChunks + threadIdx.x;
  const bool live = c < nchunks;
  float v[12];
  for (int k = 0; k < 12; ++k) v[k] = live ? cbox[c * 12 + k] : (k < 6 ? INFINITY : -INFINITY);
  for (int o = 16; o; o >>= 1)
    for (int k = 0; k < 12; ++k) {
      const float w = __shfl_xor_sync(0xffffffffu, v[k], o);
      v[k] = k < 6 ? fminf(v[k], w) : fmaxf(v[k], w);
    }
  if ((threadIdx.x & 31) == 0)
    for (int k = 0; k < 12; ++k) part[threadIdx.x >> 5][k] = v[k];
  __syncthreads();
  if (threadIdx.x < 12) {
    const int k = threadIdx.x;
    float r = part[0][k];
    for (int w = 1; w < kBlockChunks / 32; ++w) r = k < 6 ? fminf(r, part[w][k]) : fmaxf(r, part[w][k]);
    bbox[uint64_t(blockIdx.x) * 12 + k] = r;
  }
}

// ------------------------------------------------------------ mean shift
// Summation layout of one iteration: the chunks are cut into `splits` runs of
// `cps`, and a seed's sums are its splits' partial sums added in the fixed
// order of ms_reduce.  touched: one bit per (tile, split) that had a chunk to
// evaluate, kGroups x words 32-bit words per tile (split p: bit p / kGroups of
// group p % kGroups); an untouched split has no partial sums -- they would be
// zeros, which change no sum -- and is skipped by ms_reduce.
constexpr int kGroups = 8;
struct Grid {
  uint64_t tiles, splits, cps, slots;
  uint32_t words;  // 32-bit words of `touched` per group of a tile
};

// The layout for `nactive` seeds; without seeds all zero.
__device__ inline Grid grid_for(uint64_t nactive, uint64_t nchunks, int blocks_per_sm) {
  Grid g{};
  if (!nactive) return g;
  g.tiles = (nactive + kChunk - 1) / kChunk;
  const uint64_t want = (uint64_t(blocks_per_sm) * 152 + g.tiles - 1) / g.tiles;
  g.splits = max(uint64_t(1), min(nchunks, want));
  g.cps = (nchunks + g.splits - 1) / g.splits;
  g.splits = (nchunks + g.cps - 1) / g.cps;
  g.slots = g.tiles * kChunk;
  g.words = uint32_t(((g.splits + kGroups - 1) / kGroups + 31) / 32);
  return g;
}

// What retile leaves behind for a SIMT iteration: its layout, and `clear`
// zeroed (the iteration's work counters, touched and chunk bits).
struct Plan {
  Grid *grid = nullptr;
  uint64_t nchunks = 0;
  int blocks_per_sm = 0;
  uint32_t *clear = nullptr;
  uint64_t clear_words = 0;
};

__device__ __forceinline__ bool touch(uint32_t *touched, uint32_t words, uint32_t tile, uint32_t p) {
  uint32_t *w = touched + (uint64_t(tile) * kGroups + p % kGroups) * words + (p / kGroups) / 32;
  const uint32_t bit = 1u << ((p / kGroups) % 32);
  return !(atomicOr(w, bit) & bit);
}

__device__ __forceinline__ float mul_rn(float a, float b) { return __fmul_rn(a, b); }
__device__ __forceinline__ double mul_rn(double a, double b) { return __dmul_rn(a, b); }
__device__ __forceinline__ float add_rn(float a, float b) { return __fadd_rn(a, b); }
__device__ __forceinline__ double add_rn(double a, double b) { return __dadd_rn(a, b); }

// Work items of the SIMT kernel.  split_items: for every tile, the chunks
// within the bandwidth of some of its seeds (bits[t * bwords + c / 32]) and
// the (tile, split) pairs that hold one (pairs, in no particular order).
// weigh_items: an item (quarter of the tile, split) per quarter with active
// seeds, queued by the split's number of chunks, so the warps of ms_tile draw
// the longest items first (a warp that meets one of them last keeps the launch
// waiting: the first Newton iteration of the 20,000-sample motif sphere took
// 4.0 ms in the list's order, 3.0 with the longest first).
// bits, touched and work are zeroed before.  CTAs shared among the tiles.
constexpr int kQueues = 8;  // queue k: items of more than (kQueues - 1 - k) / kQueues of cps chunks
enum { kWorkPairs = 0, kWorkNext = 1, kWorkQueue = 2, kWorkSize = 2 + kQueues };
template <typename T>
__global__ void __launch_bounds__(kListThreads) split_items(
    const float *boxes, const T *means, const int32_t *ids, const unsigned *nact, const float *cbox,
    const float *bbox, uint32_t nchunks, const uint32_t *sblk, const uint32_t *nsurv, uint32_t nblk,
    float skip_gap2, const Grid *grid, uint32_t bwords, uint32_t *bits, uint32_t *touched, uint2 *pairs,
    uint32_t *work) {
  chained();
  __shared__ TileSeeds seeds;
  uint32_t t, sub, per;
  if (!list_share(nact, t, sub, per)) return;
  const uint32_t ns = nsurv[t];
  if (sub >= ns) return;
  load_tile(seeds, t, nact[0], boxes, means, ids);
  const uint32_t cps = uint32_t(grid->cps), words = grid->words;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  for (uint32_t j = sub; j < ns; j += per) {
    const uint32_t blk = sblk[uint64_t(t) * nblk + j];
    const bool keep = chunk_needed(seeds, blk, bbox, cbox, nchunks, skip_gap2);
    const unsigned bal = __ballot_sync(0xffffffffu, keep);
    if (lane == 0) bits[uint64_t(t) * bwords + blk * (kBlockChunks / 32) + warp] = bal;
    if (keep) {  // the first kept chunk of each split in the warp lists it
      const uint32_t p = (blk * kBlockChunks + threadIdx.x) / cps;
      const unsigned peers = __match_any_sync(bal, p);
      if (lane == __ffs(int(peers)) - 1 && touch(touched, words, t, p))
        pairs[atomicAdd(&work[kWorkPairs], 1u)] = make_uint2(t, p);
    }
  }
}

__global__ void __launch_bounds__(256) weigh_items(const uint2 *pairs, const unsigned *nact,
                                                   const uint32_t *bits, uint32_t bwords,
                                                   const Grid *grid, uint32_t nchunks, uint32_t room,
                                                   uint2 *items, uint32_t *work) {
  chained();
  const uint32_t cps = uint32_t(grid->cps);
  const uint32_t n = work[kWorkPairs];
  for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    const uint32_t t = pairs[i].x, p = pairs[i].y;
    const uint32_t c0 = p * cps, c1 = min(nchunks, c0 + cps);
    uint32_t weight = 0;
    for (uint32_t base = c0 & ~31u; base < c1; base += 32) {
      uint32_t word = bits[uint64_t(t) * bwords + base / 32];
      if (base < c0) word &= ~0u << (c0 - base);
      if (c1 - base < 32) word &= (1u << (c1 - base)) - 1u;
      weight += __popc(word);
    }
    const uint32_t k = kQueues - 1 - min(uint32_t(kQueues - 1), (weight - 1) * kQueues / cps);
    const uint32_t quarters = min((nact[0] - t * kChunk + 31) / 32, uint32_t(kChunk / 32));
    const uint32_t at = atomicAdd(&work[kWorkQueue + k], quarters);
    for (uint32_t x = 0; x < quarters; ++x)
      items[uint64_t(k) * room + at + x] = make_uint2(t * (kChunk / 32) + x, p);
  }
}

// Two values at once: packed FP32 arithmetic rounds each like the scalar
// instruction.
template <typename T>
struct Two {
  T x, y;
};
__device__ __forceinline__ unsigned long long bits_of(Two<float> a) {
  unsigned long long r;
  memcpy(&r, &a, 8);
  return r;
}
__device__ __forceinline__ Two<float> two_of(unsigned long long r) {
  Two<float> a;
  memcpy(&a, &r, 8);
  return a;
}
__device__ __forceinline__ Two<float> add2(Two<float> a, Two<float> b) {
  unsigned long long r;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(bits_of(a)), "l"(bits_of(b)));
  return two_of(r);
}
__device__ __forceinline__ Two<float> mul2(Two<float> a, Two<float> b) {
  unsigned long long r;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(bits_of(a)), "l"(bits_of(b)));
  return two_of(r);
}
__device__ __forceinline__ Two<float> fma2(Two<float> a, Two<float> b, Two<float> c) {
  unsigned long long r;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(bits_of(a)), "l"(bits_of(b)), "l"(bits_of(c)));
  return two_of(r);
}
__device__ __forceinline__ Two<double> add2(Two<double> a, Two<double> b) {
  return {add_rn(a.x, b.x), add_rn(a.y, b.y)};
}
__device__ __forceinline__ Two<double> mul2(Two<double> a, Two<double> b) {
  return {mul_rn(a.x, b.x), mul_rn(a.y, b.y)};
}
__device__ __forceinline__ Two<double> fma2(Two<double> a, Two<double> b, Two<double> c) {
  return {fma(a.x, b.x, c.x), fma(a.y, b.y, c.y)};
}

// A run of kSubVotes votes in shared memory: coordinate d of vote j at
// (j / 2) * kPairStride + 2 d + j % 2, so a pair's coordinates are adjacent
// (packed arithmetic) and lanes reading different votes meet different banks.
constexpr int kPairStride = 20, kRunValues = kSubVotes / 2 * kPairStride;

// A warp takes 32 active seeds (a quarter of a tile of kChunk, a lane each) and
// one split of the chunk range: each lane accumulates, for its seed, sum
// w (v - x) and sum w over the split's votes in order, and for a kNear seed
// also the unweighted in-window sums of d = v - x and d d^T (the Jacobian of
// the Newton step).
// COUNT: the votes within the bandwidth of each seed are added to
// counts[seed] instead.
// NEWTON: some seed of the launch is kNear; its 27 sums are kept in shared
// memory (in-window votes are rare, and registers would halve the warps).
// GAUSS: the shifted Gaussian weights instead of Epanechnikov's.
// With `items`, the warps draw (quarter, split) items of split_items' list
// and take the chunks whose bits are set; without, block
// (tile, split) takes every chunk of its split, a quarter per warp, or, where they
// are counted, those that some seed of the quarter can reach.
// evals gains the seed-vote pairs of the (tile, chunk) pairs taken: a chunk
// within the bandwidth of some seed of the tile, whichever quarter's, counts once.
//
// Of the chunks, the lanes test the boxes of four chunks' runs of kSubVotes
// votes (kSubs each) against the box of the warp's seeds at once; a run that
// passes is tested against each seed and then evaluated: first which of the
// votes lie within the bandwidth of the lane's seed (two votes per packed
// instruction, a bit each, no branches), then every lane takes its own
// members in turn.  Votes outside the bandwidth add nothing, so no test
// changes a sum.  Which products of a sum are rounded before they are
// added is spelt out, so every instance rounds alike whatever the compiler
// would contract.
//
// No barrier joins the warps: a form whose four warps shared each chunk
// through shared memory spent 10 to 14 issue slots of stall per instruction
// at its barriers, with 40% of the issue slots used and a third of the time in
// the tail of its CTAs (first Newton iteration of the 20,000-sample motif
// sphere, 2,048 seeds, 2.5e7 votes: 5.2 ms, 2.9 ms here).  The next run's
// 512 bytes are loaded while the current one is evaluated.
constexpr uint64_t kListedPairs = 32768;  // (tile, chunk) pairs from which the items pay (listed)
// words that hold the chunks of a direct split: at least 152 / tiles splits, so at
// most kListedPairs / 152 chunks (rounded up), starting anywhere in a word
constexpr int kDirectWords = (31 + int((kListedPairs + 151) / 152) + 31) / 32;
template <typename T, bool COUNT, bool NEWTON, bool GAUSS>
__global__ void __launch_bounds__(kChunk, sizeof(T) == 4 ? 8 : 2)
    ms_tile(const T *desc, const float *cbox, const float *sbox, uint32_t nchunks, uint64_t q, const T *means,
            const uint8_t *state, const int32_t *ids, const unsigned *nact, T h2, Window<T> win, T gk, float skip_gap2,
            const Grid *plan, uint32_t *touched, const uint32_t *bits, uint32_t bwords, const uint2 *items,
            uint32_t room, uint32_t *work, T *partial, unsigned long long *counts, unsigned long long *evals) {
  chained();
  const Grid grid = *plan;
  const uint32_t nactive = nact[0];
  if (!nactive) return;
  constexpr int kWords = int(sizeof(T)) / 4;  // 16-byte words per lane of a run
  __shared__ __align__(16) T runs[kChunk / 32][2][kRunValues];
  __shared__ T nsum[NEWTON ? 27 * kChunk : 1];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  uint32_t queue_end[kQueues];  // items of the queues up to and including each
  for (int k = 0; k < kQueues; ++k)
    queue_end[k] = (k ? queue_end[k - 1] : 0u) + (items ? work[kWorkQueue + k] : 0u);
  __shared__ uint32_t counted[kDirectWords];  // chunks of the direct split in evals already
  if (!items) {
    if (threadIdx.x < kDirectWords) counted[threadIdx.x] = 0;
    __syncthreads();
  }
  T *const ns = nsum + threadIdx.x;
  const T floor_w = GAUSS ? exp2(-gk) : T(0);
  for (;;) {
    uint32_t tile = blockIdx.x % uint32_t(grid.tiles), split = blockIdx.x / uint32_t(grid.tiles), quarter = warp;
    if (items) {
      uint32_t it = 0;
      if (lane == 0) it = atomicAdd(&work[kWorkNext], 1u);
      it = __shfl_sync(0xffffffffu, it, 0);
      if (it >= queue_end[kQueues - 1]) return;
      uint64_t at = it;
      for (int k = 1; k < kQueues; ++k)
        if (it >= queue_end[k - 1]) at = uint64_t(k) * room + (it - queue_end[k - 1]);
      const uint2 x = items[at];
      tile = x.x / (kChunk / 32), quarter = x.x % (kChunk / 32), split = x.y;
    } else if (split >= grid.splits) {
      return;
    }
    const uint32_t slot = tile * kChunk + quarter * 32 + lane;
    const bool live = slot < nactive;
    if (!__any_sync(0xffffffffu, live)) return;  // without items only
    const int32_t seed = live ? ids[slot] : 0;
    const bool newton = NEWTON && !COUNT && live && is_near(state[seed]);
    T m[6];
    float mf[6], lo[6], hi[6];
    for (int d = 0; d < 6; ++d) {
      m[d] = live ? means[uint64_t(seed) * 8 + d] : T(0);
      mf[d] = float(m[d]);
      lo[d] = live ? mf[d] : INFINITY;
      hi[d] = live ? mf[d] : -INFINITY;
    }
    for (int o = 16; o; o >>= 1)
      for (int d = 0; d < 6; ++d) {
        lo[d] = fminf(lo[d], __shfl_xor_sync(0xffffffffu, lo[d], o));
        hi[d] = fmaxf(hi[d], __shfl_xor_sync(0xffffffffu, hi[d], o));
      }
    T acc[7] = {0, 0, 0, 0, 0, 0, 0};
    unsigned members = 0;
    if (NEWTON)
      for (int j = 0; j < 27; ++j) ns[j * kChunk] = T(0);
    const uint32_t c0 = split * uint32_t(grid.cps);
    const uint32_t c1 = c0 + uint32_t(grid.cps) < nchunks ? c0 + uint32_t(grid.cps) : nchunks;
    const uint32_t *mine = items ? bits + uint64_t(tile) * bwords : nullptr;
    unsigned long long done = 0;

    uint4 held[kWords];
    uint32_t held_run = 0;
    auto fetch = [&](uint32_t run) {
      const uint4 *src = reinterpret_cast<const uint4 *>(desc);
      const uint64_t first = uint64_t(run) * 32 * kWords, last = q * 2 * kWords;
      for (int k = 0; k < kWords; ++k) {
        const uint64_t w = first + uint64_t(lane) * kWords + k;
        held[k] = w < last ? src[w] : make_uint4(0, 0, 0, 0);
      }
      held_run = run;
    };
    // the run in `held` goes to shared memory (lane: half a vote), then is evaluated
    int buf = 0;
    auto store = [&]() {
      T v[4];
      memcpy(v, held, 4 * sizeof(T));
      T *dst = runs[warp][buf] + (lane >> 2) * kPairStride + (lane & 1) * 8 + ((lane >> 1) & 1);
      for (int k = 0; k < 4; ++k) dst[2 * k] = v[k];
      __syncwarp();
    };
    auto eval = [&](uint32_t run, const T *vs) {
      const uint64_t rest = q - uint64_t(run) * kSubVotes;
      unsigned in = 0;
#pragma unroll
      for (int p = 0; p < kSubVotes / 2; ++p) {
        Two<T> v[6], d2{T(0), T(0)};
        memcpy(v, __builtin_assume_aligned(vs + p * kPairStride, 16), 6 * sizeof(Two<T>));
#pragma unroll
        for (int d = 0; d < 6; ++d) {
          const Two<T> e = add2(v[d], Two<T>{-m[d], -m[d]});
          d2 = NEWTON && !GAUSS ? add2(d2, mul2(e, e)) : fma2(e, e, d2);
        }
        in |= unsigned(d2.x < h2) << (2 * p) | unsigned(d2.y < h2) << (2 * p + 1);
      }
      if (rest < uint64_t(kSubVotes)) in &= (1u << unsigned(rest)) - 1u;
      if (!live) in = 0;
      if (COUNT) {
        members += __popc(in);
        return;
      }
      // the lane's members, in vote order, the weights of kAhead at a time (their
      // latencies overlap; past the last member it stands in again, unused)
      constexpr int kAhead = NEWTON ? 2 : 4;
      while (in) {
        T w[kAhead];
        int at[kAhead];
        const int n = __popc(in);
#pragma unroll
        for (int k = 0; k < kAhead; ++k) {
          const int j = __ffs(int(in)) - 1;
          if (k + 1 < n || k + 1 == kAhead) in &= in - 1;
          at[k] = (j >> 1) * kPairStride + (j & 1);
          T d2 = 0;
#pragma unroll
          for (int d = 0; d < 6; ++d) {
            const T e = vs[at[k] + 2 * d] - m[d];
            d2 = NEWTON && !GAUSS ? add_rn(d2, mul_rn(e, e)) : fma(e, e, d2);
          }
          const T x = over(d2, win);
          w[k] = GAUSS ? exp2(-gk * x) - floor_w : T(1) - x;
          if (k >= n) w[k] = T(0);  // adds nothing
        }
        if (n <= kAhead) in = 0;
#pragma unroll
        for (int k = 0; k < kAhead; ++k) {
          // sums of w (v - x), not of w v: the step m - x comes out without
          // the cancellation of a mean of large coordinates (votes moved
          // to their own cell of vote space lie up to 14 from the origin)
          T e[6];
#pragma unroll
          for (int d = 0; d < 6; ++d) {
            e[d] = vs[at[k] + 2 * d] - m[d];
            acc[d] = fma(w[k], e[d], acc[d]);
          }
          acc[6] += w[k];
          if (NEWTON && newton && k < n) {  // Epanechnikov: unweighted sums; Gaussian: by 2^(-k d^2/h^2)
            const T wn = w[k] + floor_w;
            int i = 6;
#pragma unroll
            for (int d = 0; d < 6; ++d) {
              const T we = GAUSS ? wn * e[d] : e[d];
              ns[d * kChunk] += we;
#pragma unroll
              for (int l = d; l < 6; ++l, ++i) {
                T &sum = ns[i * kChunk];
                sum = !GAUSS && l == d ? add_rn(sum, mul_rn(we, we)) : fma(we, e[l], sum);
              }
            }
          }
        }
      }
    };
    bool pending = false;
    auto finish = [&](bool more, uint32_t run) {  // evaluates the held run, with the next one on its way
      const uint32_t cur = held_run;
      if (pending) store();
      if (more) fetch(run);
      if (pending) {
        if (__any_sync(0xffffffffu, live && point_gap2_16(mf, sbox + uint64_t(cur) * 12) <= skip_gap2))
          eval(cur, runs[warp][buf]);
        buf ^= 1;
      }
      pending = more;
    };
    for (uint32_t base = c0 & ~31u; base < c1; base += 32) {
      uint32_t word = mine ? mine[base / 32] : ~0u;  // the chunks to take
      if (base < c0) word &= ~0u << (c0 - base);
      if (c1 - base < 32) word &= (1u << (c1 - base)) - 1u;
      uint32_t fresh = quarter == 0 ? word : 0u;  // those of them to count
      if (!mine && evals) {  // a chunk per lane against the box of the warp's seeds, then each seed
        const uint32_t c = base + lane;
        bool near = false;
        if (c >= c0 && c < c1) {
          const float4 *b4 = reinterpret_cast<const float4 *>(cbox + uint64_t(c) * 12);
          const float4 x = b4[0], y = b4[1], z = b4[2];
          const float box[12] = {x.x, x.y, x.z, x.w, y.x, y.y, y.z, y.w, z.x, z.y, z.z, z.w};
          near = box_gap2(lo, hi, box) <= skip_gap2;
        }
        word = __ballot_sync(0xffffffffu, near);
        for (uint32_t rest = word; rest; rest &= rest - 1) {
          const int k = __ffs(int(rest)) - 1;
          const bool reach = live && point_gap2_16(mf, cbox + uint64_t(base + k) * 12) <= skip_gap2;
          if (!__any_sync(0xffffffffu, reach)) word &= ~(1u << k);
        }
        fresh = 0;
        if (lane == 0 && word) fresh = word & ~atomicOr(&counted[(base - (c0 & ~31u)) / 32], word);
      }
      if (evals && lane == 0 && fresh) {
        done += uint64_t(__popc(fresh)) * kChunk;
        if (c1 == nchunks && c1 - base <= 32 && (fresh >> (nchunks - 1 - base) & 1u) && q % kChunk)
          done -= kChunk - q % kChunk;  // the last chunk is not full
      }
      while (word) {  // four chunks at a time: a run box per lane
        uint32_t w = word;
        for (int k = 0; k < 3; ++k) w = k < (lane >> 3) ? w & (w - 1) : w;
        for (int k = 0; k < 4; ++k) word &= word - 1;
        bool keep = false;
        uint32_t run = 0;
        if (w) {
          run = (base + uint32_t(__ffs(int(w)) - 1)) * kSubs + (lane & 7);
          if (uint64_t(run) * kSubVotes < q) {
            const float4 *b4 = reinterpret_cast<const float4 *>(sbox + uint64_t(run) * 12);
            const float4 a = b4[0], b = b4[1], c = b4[2];
            const float box[12] = {a.x, a.y, a.z, a.w, b.x, b.y, b.z, b.w, c.x, c.y, c.z, c.w};
            keep = box_gap2(lo, hi, box) <= skip_gap2;
          }
        }
        for (unsigned todo = __ballot_sync(0xffffffffu, keep); todo; todo &= todo - 1)
          finish(true, __shfl_sync(0xffffffffu, run, __ffs(int(todo)) - 1));
      }
    }
    finish(false, 0);
    if (COUNT) {
      if (live && members) atomicAdd(&counts[seed], (unsigned long long)members);
    } else if (live) {
      // split-major layout: value d of slot s of split p at (p * kPartial + d) *
      // slots + s, so the reduction reads consecutive seeds contiguously
      T *out = partial + uint64_t(split) * kPartial * grid.slots + slot;
      for (int d = 0; d < 7; ++d) out[d * grid.slots] = acc[d];
      if (newton)
        for (int j = 0; j < 27; ++j) out[(8 + j) * grid.slots] = ns[j * kChunk];
    }
    if (done) atomicAdd(evals, done * (unsigned long long)kChunk);
    if (!items) {
      if (!COUNT && quarter == 0 && lane == 0) touch(touched, grid.words, tile, split);
      return;
    }
  }
}

// b <- M^-1 b by Gaussian elimination with partial pivoting; false when a
// pivot is below `tiny` (singular system).
template <typename T>
__device__ bool solve6(T (&M)[6][6], T (&b)[6], T tiny) {
  for (int c = 0; c < 6; ++c) {
    int piv = c;
    T best = fabs(M[c][c]);
    for (int r = c + 1; r < 6; ++r)
      if (fabs(M[r][c]) > best) best = fabs(M[r][c]), piv = r;
    if (!(best > tiny)) return false;
    if (piv != c) {
      for (int j = 0; j < 6; ++j) {
        T t = M[c][j];
        M[c][j] = M[piv][j], M[piv][j] = t;
      }
      T t = b[c];
      b[c] = b[piv], b[piv] = t;
    }
    for (int r = c + 1; r < 6; ++r) {
      T f = quotient(M[r][c], M[c][c]);
      for (int j = c; j < 6; ++j) M[r][j] -= f * M[c][j];
      b[r] -= f * b[c];
    }
  }
  for (int c = 5; c >= 0; --c) {
    T s = b[c];
    for (int j = c + 1; j < 6; ++j) s -= M[c][j] * b[j];
    b[c] = quotient(s, M[c][c]);
  }
  return true;
}

// One step of a seed from its summed values (ms_reduce): the
// mean-shift step m - x for a kMoving seed, the safeguarded Newton step
// (I - J)^-1 (m - x) for a kNear seed, where for Epanechnikov weights
//   J = dm/dx = 2 / (h^2 sum w) * (sum d d^T - (m - x) (sum d)^T),
// d = v - x over the votes within the bandwidth, and for the shifted
// Gaussian w = g - 2^-k, g = 2^(-k d^2 / h^2) (dw/dx = 2 k ln2 g d / h^2)
//   J = 2 k ln2 / (h^2 sum w) * (sum g d d^T - (m - x) (sum g d)^T).  Stopping rules: exhausted
// when the weight is <= 1e-14 (reference, src/cpu/clustering.cpp:169-181),
// converged when a Newton step^2 < kNewtonStop2 h^2, settled (plain step
// taken) when the Newton step is rejected, or when an accepted Newton step
// is still too long at polish iteration kNewtonCap (polish_it, -1 in the
// approach phase).

// Sum of the splits of one value of a tile's seeds: block (tile, j, g) adds
// value d = j (j < 7) or j + 1 (the Newton sums) over split group g (splits
// g, g + kGroups, ...), one thread per seed slot, so each split's row of 128
// values is read contiguously.  The i-th split of the group goes into the
// sum i % 2, and only the touched splits are read: their positions come
// from the set bits of the group's words.  red[(g * kPartial + d) * slots +
// slot] = the group's sum; ms_update adds the groups in order.  Each half of
// the block takes one of the two sums.  Bound by the latency of the loads: 16
// are in flight per thread.  (Reading every split, two loads in flight, took
// 148 us per iteration on the 5.1e6-pair torus with 256 seeds, 70 MB of zeros
// mostly; 21 us now.)
constexpr int kReduceWords = 32;  // words of touched splits listed at a time
template <typename T>
__global__ void __launch_bounds__(2 * kChunk) ms_reduce(const T *partial, const Grid *plan,
                                                        const unsigned *nact, const uint32_t *touched,
                                                        T *red) {
  chained();
  const Grid grid = *plan;
  if (blockIdx.x >= grid.tiles) return;
  const unsigned nactive = nact[0];
  __shared__ uint16_t list[2][kReduceWords * 16];
  __shared__ int count[2];
  __shared__ T other[kChunk];
  const int half = threadIdx.x >= kChunk, t = threadIdx.x % kChunk, lane = threadIdx.x & 31;
  const uint64_t slot = uint64_t(blockIdx.x) * kChunk + t;
  const int d = blockIdx.y < 7 ? int(blockIdx.y) : int(blockIdx.y) + 1;
  const uint64_t g = blockIdx.z;
  const T *in = partial + (g * kPartial + uint64_t(d)) * grid.slots + slot;
  const uint64_t step = uint64_t(kGroups) * kPartial * grid.slots;
  const uint32_t *words = touched + (uint64_t(blockIdx.x) * kGroups + g) * grid.words;
  const bool live = slot < nactive;
  T sum = 0;
  for (uint32_t w0 = 0; w0 < grid.words; w0 += kReduceWords) {
    if (t < 32) {  // one warp per half lists its touched splits, ascending
      const uint32_t i = w0 + lane;
      uint32_t m = (i < grid.words ? words[i] : 0u) & (half ? 0xAAAAAAAAu : 0x55555555u);
      const int n = __popc(m);
      int incl = n;
      for (int o = 1; o < 32; o <<= 1) {
        const int y = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= o) incl += y;
      }
      for (int at = incl - n; m; m &= m - 1) list[half][at++] = uint16_t(lane * 32 + __ffs(int(m)) - 1);
      if (lane == 31) count[half] = incl;
    }
    __syncthreads();
    const int n = count[half];
    const T *base = in + uint64_t(w0) * 32 * step;
    constexpr int kAhead = 16;  // loads in flight per thread
    if (live)
      for (int k = 0; k < n; k += kAhead) {
        T v[kAhead];
#pragma unroll
        for (int a = 0; a < kAhead; ++a) v[a] = k + a < n ? base[list[half][k + a] * step] : T(0);
#pragma unroll
        for (int a = 0; a < kAhead; ++a) sum += v[a];  // past the end: zeros, which change nothing
      }
    __syncthreads();
  }
  if (half) other[t] = sum;
  __syncthreads();
  if (!half && live) red[(g * kPartial + d) * grid.slots + slot] = sum + other[t];
}

// One thread per seed: the step from the summed values (ms_reduce).
template <typename T>
__global__ void __launch_bounds__(kChunk) ms_update(T *means, const T *red, const Grid *grid,
                                                    const int32_t *ids, const unsigned *nact, T h2,
                                                    T gk, int polish_it, uint8_t *state) {
  chained();
  const uint64_t slots = grid->slots;
  const unsigned nactive = nact[0];
  const uint64_t slot = uint64_t(blockIdx.x) * kChunk + threadIdx.x;
  if (slot >= nactive) return;
  const int32_t s = ids[slot];
  const uint8_t st_s = state[s];
  const bool near = is_near(st_s);
  T acc[7] = {0, 0, 0, 0, 0, 0, 0}, ns[27];
  for (int g = 0; g < kGroups; ++g)
    for (int d = 0; d < 7; ++d) acc[d] += red[(uint64_t(g) * kPartial + d) * slots + slot];
  if (near)
    for (int j = 0; j < 27; ++j) {
      ns[j] = 0;
      for (int g = 0; g < kGroups; ++g) ns[j] += red[(uint64_t(g) * kPartial + 8 + j) * slots + slot];
    }
  if (acc[6] <= T(1e-14)) {
    state[s] = kExhausted;
    return;
  }
  T x[6], delta[6], move = 0;
  for (int d = 0; d < 6; ++d) {
    x[d] = means[uint64_t(s) * 8 + d];
    delta[d] = quotient(acc[d], acc[6]);  // m - x from the sums of w (v - x)
    move += delta[d] * delta[d];
  }
  if (!near) {
    for (int d = 0; d < 6; ++d) means[uint64_t(s) * 8 + d] = x[d] + delta[d];
    if (move < T(kSwitch2) * h2) state[s] = kNear;
    return;
  }
  const T *sd = ns, *sdd = ns + 6;
  T M[6][6], step[6];
  const T g = (gk > T(0) ? T(2) * gk * T(0.69314718055994531) : T(2)) / (h2 * acc[6]);
  for (int d = 0, at = 0; d < 6; ++d)
    for (int l = d; l < 6; ++l, ++at) M[d][l] = M[l][d] = sdd[at];
  for (int d = 0; d < 6; ++d) {
    for (int l = 0; l < 6; ++l) M[d][l] = (d == l ? T(1) : T(0)) - g * (M[d][l] - delta[d] * sd[l]);
    step[d] = delta[d];
  }
  bool ok = solve6(M, step, T(sizeof(T) == 4 ? 1e-6 : 1e-12));
  T len = 0, along = 0;
  for (int d = 0; d < 6; ++d) len += step[d] * step[d], along += step[d] * delta[d];
  ok = ok && isfinite(len) && len <= T(kTrust * kTrust) * h2 &&
       (along > T(0) || len < T(kNewtonStop2) * h2);
  if (ok) {
    for (int d = 0; d < 6; ++d) means[uint64_t(s) * 8 + d] = x[d] + step[d];
    if (len < T(kNewtonStop2) * h2) state[s] = kConverged;
    else if (polish_it >= kNewtonCap) state[s] = kSettled;
  } else {  // rejected: the plain step, and Newton once more (settled at the second rejection)
    for (int d = 0; d < 6; ++d) means[uint64_t(s) * 8 + d] = x[d] + delta[d];
    state[s] = polish_it < kNewtonCap && st_s == kNear ? kNearRetry1 : kSettled;
  }
}

// Active seeds (kMoving, and kNear when include_near): in seed order, sorted
// by the Morton key of their current mean (ties by seed id) when k <= kRetile.
// The number of active seeds and what else `progress` holds goes there; `plan` as
// above.
//
// Runs in every iteration between two kernels that wait for it, so its own
// latency counts.  A block lists the active seeds for itself from their state
// bytes.  Sorted, it makes every key and places kRankSeeds seeds by counting
// the keys below each, a part of the keys per warp, where a bitonic network in
// one block had up to 66 dependent steps (2,048 seeds: 15 us, 128: 5; the
// network took 30 and 10).  Not sorted, a block places kRetile
// seeds behind the active ones it counts before them.
constexpr int kRetile = 2048;  // seeds a block lists
constexpr int kRetileThreads = 256, kRankSeeds = 32;
static_assert(kRetile == kRetileThreads * 8, "eight state bytes per thread");
unsigned retile_blocks(uint64_t k) {
  const uint64_t per = k <= kRetile ? kRankSeeds : kRetile;
  return unsigned(std::max<uint64_t>(1, (k + per - 1) / per));  // one reports that there are none
}

template <typename T>
__global__ void __launch_bounds__(kRetileThreads) retile(const T *means, const uint8_t *state, uint64_t k,
                                                         const float *box, bool include_near,
                                                         int32_t *ids, Progress *progress, Plan plan) {
  constexpr int kWarps = kRetileThreads / 32;
  __shared__ unsigned long long keys[kRetile];
  __shared__ uint16_t seeds[kRetile];
  __shared__ unsigned warp_active[kWarps], warp_near[kWarps], below[kWarps][kRankSeeds];
  chained();
  for (uint64_t i = uint64_t(blockIdx.x) * kRetileThreads + threadIdx.x; i < plan.clear_words;
       i += uint64_t(gridDim.x) * kRetileThreads)
    plan.clear[i] = 0;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const bool sort = k <= kRetile;
  // a block that looks at every seed reports; its loads come ahead of its stores
  const bool reports = threadIdx.x == 0 && blockIdx.x == (sort ? 0 : gridDim.x - 1);
  unsigned done = 0;
  unsigned long long served = 0, began = 0, ended = 0, busy = 0;
  if (reports)
    done = progress->iterations, served = progress->seeds, began = progress->began, ended = progress->ended,
    busy = progress->busy;
  const uint64_t first = sort ? 0 : uint64_t(blockIdx.x) * kRetile;
  // the states of seeds s..s + 7 (zero bits: not active), `near` of them
  unsigned mask = 0, near = 0, before = 0;
  auto look = [&](uint64_t s, unsigned &m) {
    for (int j = 0; j < 8; ++j)
      if (s + j < k) {
        const uint8_t st = state[s + j];
        const bool close = include_near && is_near(st);
        m |= unsigned(st == kMoving || close) << j;
        near += close;
      }
  };
  for (uint64_t s = threadIdx.x * 8; s < first; s += kRetile) {  // (not sorted: the blocks before)
    unsigned m = 0;
    look(s, m);
    before += __popc(m);
  }
  look(first + threadIdx.x * 8, mask);
  // exclusive scan of the counts, with those of the blocks before on top
  unsigned incl = __popc(mask);
  const unsigned mine = incl;
  for (int o = 1; o < 32; o <<= 1) {
    const unsigned y = __shfl_up_sync(0xffffffffu, incl, o);
    if (lane >= o) incl += y;
  }
  if (lane == 31) warp_active[warp] = incl;
  for (int o = 16; o; o >>= 1) {
    near += __shfl_xor_sync(0xffffffffu, near, o);
    before += __shfl_xor_sync(0xffffffffu, before, o);
  }
  if (lane == 0) warp_near[warp] = near, below[0][warp] = before;
  __syncthreads();
  unsigned at = incl - mine, total = 0;
  before = near = 0;
  for (int w = 0; w < kWarps; ++w) {
    if (w < warp) at += warp_active[w];
    total += warp_active[w], near += warp_near[w], before += below[0][w];
  }
  const unsigned n = before + total;
  if (reports) {
    progress->nact[0] = n, progress->nact[1] = near;
    if (plan.grid) *plan.grid = grid_for(n, plan.nchunks, plan.blocks_per_sm);
    if (n) {
      if (done < kTraced) progress->trace[done] = n;
      progress->iterations = done + 1, progress->seeds = served + n;
    }
    if (ended) progress->busy = busy + (ended - began);
    progress->began = ~0ull, progress->ended = 0;
  }
  if (!sort) {
    at += before;
    for (unsigned m = mask; m; m &= m - 1)
      ids[at++] = int32_t(first + threadIdx.x * 8 + __ffs(int(m)) - 1);
    return;
  }
  const unsigned r0 = blockIdx.x * kRankSeeds;
  if (r0 >= n) return;  // the whole block
  for (unsigned m = mask; m; m &= m - 1) seeds[at++] = uint16_t(threadIdx.x * 8 + __ffs(int(m)) - 1);
  __syncthreads();
  for (unsigned i = threadIdx.x; i < n; i += kRetileThreads) {
    const uint64_t s = seeds[i];
    float x[6];
    for (int d = 0; d < 6; ++d) x[d] = float(means[s * 8 + d]);
    keys[i] = morton6(x, box);
  }
  __syncthreads();
  const unsigned i = r0 + lane;
  const unsigned long long key = i < n ? keys[i] : 0;
  const unsigned part = (n + kWarps - 1) / kWarps, j0 = warp * part, j1 = min(n, j0 + part);
  unsigned count = 0;
  for (unsigned j = j0; j < j1; ++j) {
    const unsigned long long other = keys[j];
    count += other < key || (other == key && j < i);  // equal keys: the listed order is seed order
  }
  below[warp][lane] = count;
  __syncthreads();
  if (warp == 0 && i < n) {
    unsigned rank = 0;
    for (int w = 0; w < kWarps; ++w) rank += below[w][lane];
    ids[rank] = int32_t(seeds[i]);
  }
}

template <typename T>
__global__ void gather_seeds(const T *desc, const int64_t *pos, uint64_t k, T *means) {
  uint64_t i = uint64_t(blockIdx.x) * blockDim.x + threadIdx.x;
  if (i >= k) return;
  for (int d = 0; d < 8; ++d) means[i * 8 + d] = desc[uint64_t(pos[i]) * 8 + d];
}

// Whether an iteration draws its work from split_items' list: with few
// (tile, chunk) pairs the direct grid's own tests cost less than the three list
// kernels.  Us per approach iteration, direct and listed: 23 and 34 at 40 pairs
// (mirror planes), on the motif sphere 24 and 37 at 2,800, 48 and 65 at 18,900, 68
// and 84 at 38,000, 147 and 169 at 170,000; on the 1e7-vote Gaussian torus, whose
// tiles reach fewer of their chunks, 50 and 51 at 7,300, 68 and 62 at 11,400, 85 and
// 79 at 45,600.  The line lies between the two.  The sums are the same either way.
bool listed(uint64_t tiles, uint64_t nchunks) { return tiles * nchunks >= kListedPairs; }

// Scratch of the SIMT iterations, sized for `k` seeds.
struct TileWork {
  uint32_t *work = nullptr;     // [items, next item], then `touched`, then `bits`: zeroed together
  uint32_t *touched = nullptr, *bits = nullptr;
  Grid *grid = nullptr;         // of the iteration, by retile
  uint32_t bwords = 0, nblk = 0;
  uint64_t max_splits = 0;      // tiles x splits never exceeds it
  float *boxes = nullptr;
  uint32_t *sblk = nullptr, *nsurv = nullptr;
  uint2 *pairs = nullptr, *items = nullptr;
  unsigned list_ctas = 0;
};

template <typename T>
TileWork tile_work(Call &call, const VoteSet &v, uint64_t k) {
  TileWork w;
  const uint64_t tiles = (k + kChunk - 1) / kChunk;
  w.nblk = uint32_t(v.nblocks);
  w.bwords = w.nblk * (kBlockChunks / 32);
  // splits <= blocks * 152 / tiles + 1 each; a group's words round up
  w.max_splits = uint64_t(v.tuning.simt_blocks_per_sm) * 152 + 2 * tiles;
  const uint64_t touch_words = w.max_splits / 32 + (tiles + 1) * kGroups * 2;
  w.work = call.alloc<uint32_t>(kWorkSize + touch_words + tiles * w.bwords);
  w.touched = w.work + kWorkSize;
  w.bits = w.touched + touch_words;
  w.grid = call.alloc<Grid>(1);
  w.boxes = call.alloc<float>(tiles * kBoxFloats);
  w.sblk = call.alloc<uint32_t>(tiles * w.nblk);
  w.nsurv = call.alloc<uint32_t>(tiles);
  w.pairs = call.alloc<uint2>(w.max_splits);
  w.items = call.alloc<uint2>(w.max_splits * (kChunk / 32) * kQueues);
  static const int per_sm = [] {
    int a = 0;
    SYM_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&a, split_items<T>, kListThreads, 0));
    return std::max(1, a);
  }();
  w.list_ctas = unsigned(std::max<uint64_t>(tiles, uint64_t(152) * per_sm));
  return w;
}

// What retile is to prepare for an iteration of at most `tiles` tiles.
template <typename T>
Plan plan_of(const VoteSet &v, const TileWork &w, uint64_t tiles) {
  Plan p;
  p.grid = w.grid, p.nchunks = v.nchunks, p.blocks_per_sm = v.tuning.simt_blocks_per_sm;
  p.clear = w.work;
  p.clear_words = uint64_t(w.bits - w.work) + (listed(tiles, v.nchunks) ? tiles * w.bwords : 0);
  return p;
}

// One ms_tile launch (and, listed, the work items before it) over the active
// seeds, at most `tiles` tiles of them.
template <typename T, bool COUNT, bool NEWTON, bool GAUSS>
void run_tiles(Call &call, const VoteSet &v, const T *desc, const T *means, const uint8_t *state,
               const int32_t *ids, const unsigned *nact, uint64_t tiles, double h2, const TileWork &w,
               T *partial, unsigned long long *counts, unsigned long long *evals) {
  cudaStream_t st = call.stream();
  const float gap = float(std::sqrt(h2)) + 1e-6f, gap2 = gap * gap;
  const T k = T(v.kernel_k);
  // (tile, split) pairs of any number of tiles up to that: tiles x splits
  const uint64_t pairs =
      std::min<uint64_t>(tiles * v.nchunks, uint64_t(v.tuning.simt_blocks_per_sm) * 152 + tiles);
  if (!listed(tiles, v.nchunks)) {
    launch_chained(st, ms_tile<T, COUNT, NEWTON, GAUSS>, unsigned(pairs), kChunk, 0, desc, v.cbox, v.sbox,
                   uint32_t(v.nchunks), v.q, means, state, ids, nact, T(h2), window(T(h2)), k, gap2, w.grid, w.touched,
                   nullptr, 0u, nullptr, 0u, nullptr, partial, counts, evals);
    call.launched();
    return;
  }
  launch_chained(st, tile_boxes<T>, unsigned(tiles), kCullThreads, 0, means, ids, nact, v.bbox, w.nblk, gap2,
                 w.boxes, w.sblk, w.nsurv, nullptr);
  launch_chained(st, split_items<T>, w.list_ctas, kListThreads, 0, w.boxes, means, ids, nact, v.cbox, v.bbox,
                 uint32_t(v.nchunks), w.sblk, w.nsurv, w.nblk, gap2, w.grid, w.bwords, w.bits, w.touched,
                 w.pairs, w.work);
  const uint32_t room = uint32_t(w.max_splits * (kChunk / 32));
  launch_chained(st, weigh_items, blocks_for(pairs), kThreads, 0, w.pairs, nact, w.bits, w.bwords, w.grid,
                 uint32_t(v.nchunks), room, w.items, w.work);
  static const int per_sm = [] {
    int a = 0;
    SYM_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&a, ms_tile<T, COUNT, NEWTON, GAUSS>,
                                                           kChunk, 0));
    return std::max(1, a);
  }();
  const unsigned ctas = unsigned(std::min<uint64_t>(pairs, uint64_t(152) * per_sm));
  launch_chained(st, ms_tile<T, COUNT, NEWTON, GAUSS>, ctas, kChunk, 0, desc, v.cbox, v.sbox, uint32_t(v.nchunks), v.q,
                 means, state, ids, nact, T(h2), window(T(h2)), k, gap2, w.grid, w.touched, w.bits, w.bwords, w.items, room,
                 w.work, partial, counts, evals);
  call.launched(4);
}

// Iterations are launched back to back: the number of active seeds and the
// layout that goes with it stay on the device, and an iteration that finds no
// active seed returns at once.  The number only falls, so the last one the
// host saw bounds the launches; it looks before the first iteration and after
// every kShiftCheck (an iteration of the mirror planes' approach: 34 us with a
// look at each, 25 now).  A polish with kMoving seeds
// left looks at each: the instance without Newton sums serves an iteration
// without kNear seeds, and rounds distances otherwise.
constexpr int kShiftCheck = 4, kPolishCheck = 2;  // (a polish ends after a few)
template <typename T>
int shift_impl(Call &call, const VoteSet &v, const T *desc, T *means, uint8_t *state, uint64_t k,
               double h2, int max_iter, bool polish, double *seed_iterations,
               unsigned long long *evals, uint32_t *trace = nullptr, int trace_len = 0) {
  cudaStream_t st = call.stream();
  int32_t *ids = call.alloc<int32_t>(k);
  Progress *progress = call.alloc<Progress>(1), seen{};
  const unsigned *const nact = progress->nact;  // on the device
  // partial capacity: splits x slots is at most ~blocks*152*kChunk (+ one tile)
  const int bps = v.tuning.simt_blocks_per_sm;
  uint64_t cap = (uint64_t(bps) * 152 + 2) * uint64_t(kChunk) + std::max<uint64_t>(k, kChunk) * 2;
  T *partial = call.alloc<T>(cap * kPartial);
  T *red = call.alloc<T>(uint64_t(kGroups) * kPartial * std::max<uint64_t>(k, kChunk) * 2);
  TileWork work = tile_work<T>(call, v, k);
  SYM_CUDA(cudaMemsetAsync(progress, 0, sizeof(Progress), st));
  uint64_t tiles = (k + kChunk - 1) / kChunk;  // at most, as the host knows
  const unsigned *const counts = seen.nact;
  const bool gauss = v.kernel_k > 0;
  bool finished = false;
  auto look = [&]() {
    call.d2h(&seen, progress, sizeof(Progress));
    call.sync();
  };
  const int check = polish ? kPolishCheck : kShiftCheck;
  for (int it = 0; it < max_iter; ++it) {
    launch_chained(st, retile<T>, retile_blocks(k), kRetileThreads, 0, means, state, k, v.gbox, polish, ids,
                   progress, plan_of<T>(v, work, tiles));
    call.launched();
    if (it % check == 0 || (polish && counts[1] != counts[0])) {
      look();
      finished = !counts[0];
      if (finished) break;
      tiles = (counts[0] + kChunk - 1) / kChunk;
    }
    if ((uint64_t(bps) * 152 + tiles) * kChunk > cap || uint64_t(bps) * 152 + tiles > work.max_splits)
      fail(SYM_RUNTIME_ERROR, "mean-shift partial buffer too small");
    const auto run = counts[1] ? (gauss ? run_tiles<T, false, true, true> : run_tiles<T, false, true, false>)
                               : (gauss ? run_tiles<T, false, false, true> : run_tiles<T, false, false, false>);
    run(call, v, desc, means, state, ids, nact, tiles, h2, work, partial, nullptr, evals);
    launch_chained(st, ms_reduce<T>, dim3(unsigned(tiles), counts[1] ? 34u : 7u, kGroups), 2 * kChunk, 0,
                   partial, work.grid, nact, work.touched, red);
    launch_chained(st, ms_update<T>, unsigned(tiles), kChunk, 0, means, red, work.grid, ids, nact, T(h2),
                   T(v.kernel_k), polish ? it : -1, state);
    call.launched(2);
  }
  if (!finished) look();
  if (seed_iterations) *seed_iterations += double(seen.seeds);
  for (int i = 0; trace && i < std::min(trace_len, kTraced) && i < int(seen.iterations); ++i) trace[i] = seen.trace[i];
  return int(seen.iterations);
}

}  // namespace

VoteSet build_vote_set(Call &call, const float *desc_raw, const double *desc64_raw, uint64_t q,
                       const Tuning &tuning) {
  cudaStream_t st = call.stream();
  if (tuning.vote_bits < 1 || tuning.vote_bits > 10 || tuning.simt_blocks_per_sm < 1 ||
      tuning.simt_blocks_per_sm > 256 || tuning.tc_ctas_per_sm < 1 || tuning.tc_ctas_per_sm > 8 ||
      tuning.check_interval < 1)
    fail(SYM_INVALID_ARGUMENT, "tuning parameter out of range");
  VoteSet v;
  v.tuning = tuning;
  v.q = q;
  v.nchunks = (q + kChunk - 1) / kChunk;
  const int kBoxBlocks = 256;
  float *bpart = call.alloc<float>(kBoxBlocks * 12);
  v.gbox = call.alloc<float>(12);
  box_partials<<<kBoxBlocks, 256, 0, st>>>(desc_raw, q, bpart);
  check_launch();
  box_final<<<1, 32, 0, st>>>(bpart, kBoxBlocks, v.gbox);
  check_launch();
  uint64_t *keys = call.alloc<uint64_t>(q), *skeys = call.alloc<uint64_t>(q);
  int32_t *idx = call.alloc<int32_t>(q);
  v.order = call.alloc<int32_t>(q);
  v.rank = call.alloc<int32_t>(q);
  morton_keys<<<blocks_for(q), kThreads, 0, st>>>(desc_raw, q, v.gbox, tuning.vote_bits, keys, idx);
  check_launch();
  radix_sort_pairs(call, keys, idx, skeys, v.order, q, 6 * tuning.vote_bits);
  invert<<<blocks_for(q), kThreads, 0, st>>>(v.order, q, v.rank);
  check_launch();
  v.desc = call.alloc<float>(q * 8);
  permute<float><<<blocks_for(q), kThreads, 0, st>>>(desc_raw, v.order, q, v.desc);
  check_launch();
  if (desc64_raw) {
    v.desc64 = call.alloc<double>(q * 8);
    permute<double><<<blocks_for(q), kThreads, 0, st>>>(desc64_raw, v.order, q, v.desc64);
    check_launch();
  }
  v.cbox = call.alloc<float>(v.nchunks * 12);
  v.sbox = call.alloc<float>(v.nchunks * kSubs * 12);
  chunk_boxes<<<blocks_for(v.nchunks * 32), kThreads, 0, st>>>(v.desc, q, v.nchunks, v.cbox,
                                                                v.sbox);
  check_launch();
  v.nblocks = (v.nchunks + kBlockChunks - 1) / kBlockChunks;
  v.bbox = call.alloc<float>(v.nblocks * 12);
  if (v.nblocks) {
    block_boxes<<<unsigned(v.nblocks), kBlockChunks, 0, st>>>(v.cbox, v.nchunks, v.bbox);
    check_launch();
  }
  call.launched(desc64_raw ? 9 : 8);
  return v;
}

void init_means(Call &call, const VoteSet &v, const int64_t *seed_rank, uint64_t k, float *means) {
  gather_seeds<float><<<blocks_for(k), kThreads, 0, call.stream()>>>(v.desc, seed_rank, k, means);
  check_launch();
  call.launched();
}

void init_means(Call &call, const VoteSet &v, const int64_t *seed_rank, uint64_t k, double *means) {
  gather_seeds<double><<<blocks_for(k), kThreads, 0, call.stream()>>>(v.desc64, seed_rank, k, means);
  check_launch();
  call.launched();
}

int shift(Call &call, const VoteSet &v, float *means, uint8_t *state, uint64_t k, double h2,
          int max_iter, bool polish, double *seed_iterations, unsigned long long *evals,
          uint32_t *trace, int trace_len) {
  return shift_impl<float>(call, v, v.desc, means, state, k, h2, max_iter, polish, seed_iterations,
                           evals, trace, trace_len);
}

int shift(Call &call, const VoteSet &v, double *means, uint8_t *state, uint64_t k, double h2,
          int max_iter, bool polish, double *seed_iterations, unsigned long long *evals) {
  return shift_impl<double>(call, v, v.desc64, means, state, k, h2, max_iter, polish,
                            seed_iterations, evals);
}

void active_seeds_async(Call &call, const VoteSet &v, const float *means, const uint8_t *state,
                        uint64_t k, int32_t *ids, Progress *progress) {
  launch_chained(call.stream(), retile<float>, retile_blocks(k), kRetileThreads, 0, means, state, k, v.gbox,
                 false, ids, progress, Plan());
  call.launched();
}

void count_within(Call &call, const VoteSet &v, const float *points, uint64_t nm, double h2,
                  unsigned long long *counts) {
  if (!nm) return;
  cudaStream_t st = call.stream();
  uint8_t *state = call.alloc<uint8_t>(nm);
  SYM_CUDA(cudaMemsetAsync(state, 0, nm, st));
  int32_t *ids = call.alloc<int32_t>(nm);
  Progress *progress = call.alloc<Progress>(1);
  SYM_CUDA(cudaMemsetAsync(progress, 0, sizeof(Progress), st));
  const unsigned *const nact = progress->nact;  // on the device
  const uint64_t tiles = (nm + kChunk - 1) / kChunk;
  TileWork work = tile_work<float>(call, v, nm);
  SYM_CUDA(cudaMemsetAsync(counts, 0, nm * sizeof(*counts), st));
  launch_chained(st, retile<float>, retile_blocks(nm), kRetileThreads, 0, points, state, nm, v.gbox, false, ids,
                 progress, plan_of<float>(v, work, tiles));
  run_tiles<float, true, false, false>(call, v, v.desc, points, nullptr, ids, nact, tiles, h2, work,
                                       static_cast<float *>(nullptr), counts, nullptr);
  call.launched();
}

}  // namespace sym
