// SPDX-License-Identifier: MPL-2.0
// Which chunks of a vote set a tile of seeds can reach: the tests shared by
// the tensor kernel's chunk lists (meanshift_tc.cu) and the SIMT kernel's
// work items (meanshift_fast.cu).  Exact for weights that vanish beyond the
// bandwidth: every vote of a chunk left out is farther than the bandwidth from
// every seed of the tile, and a box holds its seeds' coordinates, so in FP32
// too its gap (monotone in every operation) is never above a seed's.
#pragma once
#include "meanshift_fast.cuh"

namespace sym {
namespace {

__device__ __forceinline__ float box_gap2(const float *lo, const float *hi, const float *b) {
  float g = 0;
  for (int k = 0; k < 6; ++k) {
    float d = fmaxf(fmaxf(b[k] - hi[k], lo[k] - b[6 + k]), 0.f);
    g += d * d;
  }
  return g;
}

// Squared distance of a point to a box.
__device__ __forceinline__ float point_gap2(const float *x, const float *b) {
  float g = 0;
  for (int d = 0; d < 6; ++d) {
    const float e = fmaxf(fmaxf(b[d] - x[d], x[d] - b[6 + d]), 0.f);
    g += e * e;
  }
  return g;
}

// The same with the box's 12 floats on a 16-byte boundary.
__device__ __forceinline__ float point_gap2_16(const float *x, const float *b) {
  const float4 *b4 = reinterpret_cast<const float4 *>(b);
  const float4 p = b4[0], q = b4[1], r = b4[2];
  const float box[12] = {p.x, p.y, p.z, p.w, q.x, q.y, q.z, q.w, r.x, r.y, r.z, r.w};
  return point_gap2(x, box);
}

// The number of active seeds n = nact[0] is read on the device by every
// kernel of an iteration, so the host never waits for it: grids are sized
// for all k seeds and blocks past the active tiles return at once.
__device__ __forceinline__ uint32_t active_tiles(const unsigned *nact) {
  return (nact[0] + kChunk - 1) / kChunk;
}

// boxes[t * kBoxFloats ..]: the box of tile t's active seeds (12 floats:
// lo, hi), then the boxes of its eight groups of 16 seeds (one block per
// tile).  Then the block cull: sblk[t * nblk ..] lists, in ascending order,
// the blocks of kBlockChunks chunks whose box lies within the bandwidth of
// the tile's box and of some group's box, and nsurv[t] counts them; with
// bcount, their counts bcount[t * nblk + j] are zeroed.
constexpr int kGroupSeeds = 16, kBoxFloats = 12 * (1 + kChunk / kGroupSeeds);
constexpr int kCullThreads = 512;  // threads of tile_boxes (the first kChunk hold the seeds)
template <typename T>
__global__ void __launch_bounds__(kCullThreads) tile_boxes(const T *means, const int32_t *ids,
                                                           const unsigned *nact, const float *bbox,
                                                           uint32_t nblk, float skip_gap2,
                                                           float *boxes, uint32_t *sblk,
                                                           uint32_t *nsurv, uint32_t *bcount) {
  __shared__ float part[kChunk / kGroupSeeds][12];
  __shared__ float tb[kBoxFloats];
  __shared__ uint32_t warp_cnt[kCullThreads / 32], base_s;
  chained();
  if (blockIdx.x >= active_tiles(nact)) return;
  if (threadIdx.x < kChunk) {  // whole warps
    const uint64_t slot = uint64_t(blockIdx.x) * kChunk + threadIdx.x;
    const bool live = slot < nact[0];
    float lo[6], hi[6];
    for (int d = 0; d < 6; ++d) {
      float m = live ? float(means[uint64_t(ids[slot]) * 8 + d]) : 0.f;
      lo[d] = live ? m : INFINITY, hi[d] = live ? m : -INFINITY;
    }
    for (int o = kGroupSeeds / 2; o; o >>= 1)  // within each group of 16 lanes
      for (int d = 0; d < 6; ++d) {
        lo[d] = fminf(lo[d], __shfl_xor_sync(0xffffffffu, lo[d], o));
        hi[d] = fmaxf(hi[d], __shfl_xor_sync(0xffffffffu, hi[d], o));
      }
    const int group = threadIdx.x / kGroupSeeds;
    if (threadIdx.x % kGroupSeeds == 0)
      for (int d = 0; d < 6; ++d) part[group][d] = lo[d], part[group][6 + d] = hi[d];
  }
  if (threadIdx.x == 0) base_s = 0;
  __syncthreads();
  float *out = boxes + uint64_t(blockIdx.x) * kBoxFloats;
  constexpr int kGroups = kChunk / kGroupSeeds;
  if (threadIdx.x < 12) {
    float v = part[0][threadIdx.x];
    for (int w = 1; w < kGroups; ++w)
      v = threadIdx.x < 6 ? fminf(v, part[w][threadIdx.x]) : fmaxf(v, part[w][threadIdx.x]);
    out[threadIdx.x] = v, tb[threadIdx.x] = v;
  } else if (threadIdx.x < kBoxFloats) {
    const float v = part[(threadIdx.x - 12) / 12][(threadIdx.x - 12) % 12];
    out[threadIdx.x] = v, tb[threadIdx.x] = v;
  }
  __syncthreads();
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  uint32_t *mine = sblk + uint64_t(blockIdx.x) * nblk;
  for (uint32_t b0 = 0; b0 < nblk; b0 += kCullThreads) {
    const uint32_t b = b0 + threadIdx.x;
    bool keep = false;
    if (b < nblk) {
      float bb[12];
      for (int d = 0; d < 12; ++d) bb[d] = bbox[uint64_t(b) * 12 + d];
      if (box_gap2(tb, tb + 6, bb) <= skip_gap2)
        for (int g = 0; g < kGroups && !keep; ++g)
          keep = box_gap2(tb + 12 + 12 * g, tb + 18 + 12 * g, bb) <= skip_gap2;
    }
    const uint32_t bal = __ballot_sync(0xffffffffu, keep);
    if (lane == 0) warp_cnt[warp] = __popc(bal);
    __syncthreads();
    uint32_t before = base_s, total = 0;
    for (int w = 0; w < kCullThreads / 32; ++w) {
      if (w < warp) before += warp_cnt[w];
      total += warp_cnt[w];
    }
    if (keep) {
      const uint32_t at = before + __popc(bal & ((1u << lane) - 1u));
      mine[at] = b;
      if (bcount) bcount[uint64_t(blockIdx.x) * nblk + at] = 0;  // tile_count adds the block's kept chunks
    }
    __syncthreads();
    if (threadIdx.x == 0) base_s += total;
    __syncthreads();
  }
  if (threadIdx.x == 0) nsurv[blockIdx.x] = base_s;
}

// The CTAs of a list kernel's grid shared among the active tiles: CTA i
// serves tile i % tiles and takes every per-th of its surviving blocks,
// starting at i / tiles (per = CTAs / tiles); false for a CTA left over.
__device__ __forceinline__ bool list_share(const unsigned *nact, uint32_t &t, uint32_t &sub,
                                           uint32_t &per) {
  const uint32_t tiles = active_tiles(nact), i = blockIdx.x;
  if (!tiles) return false;
  per = gridDim.x / tiles;
  if (!per || i >= per * tiles) return false;
  t = i % tiles, sub = i / tiles;
  return true;
}

constexpr int kListThreads = 256;  // chunks per block of the list kernels
static_assert(kListThreads == kBlockChunks, "one thread per chunk of a block box");

// A tile's seeds and their boxes in shared memory, for a CTA of
// kListThreads threads that tests the chunks of the tile's surviving blocks.
constexpr int kQuads = kChunk / 4;
struct TileSeeds {
  float seed[kChunk * 6];
  float gb[kBoxFloats];
  float qb[kQuads * 12];
  bool alive[kChunk];
  uint32_t reach[kChunk / 32];  // seeds within the bandwidth of the block's box
};

template <typename T>
__device__ __forceinline__ void load_tile(TileSeeds &s, uint32_t t, unsigned nactive,
                                          const float *boxes, const T *means, const int32_t *ids) {
  for (int i = threadIdx.x; i < kChunk; i += blockDim.x) {
    const uint64_t slot = uint64_t(t) * kChunk + i;
    const bool live = slot < nactive;
    s.alive[i] = live;
    for (int d = 0; d < 6; ++d)
      s.seed[i * 6 + d] = live ? float(means[uint64_t(ids[slot]) * 8 + d]) : 1e30f;
  }
  if (threadIdx.x < kBoxFloats) s.gb[threadIdx.x] = boxes[uint64_t(t) * kBoxFloats + threadIdx.x];
  __syncthreads();
  if (threadIdx.x < kQuads) {  // a quad without live seeds gets an empty box (gap infinite)
    float lo[6], hi[6];
    for (int d = 0; d < 6; ++d) lo[d] = INFINITY, hi[d] = -INFINITY;
    for (int i = 4 * threadIdx.x; i < 4 * int(threadIdx.x) + 4; ++i)
      if (s.alive[i])
        for (int d = 0; d < 6; ++d)
          lo[d] = fminf(lo[d], s.seed[i * 6 + d]), hi[d] = fmaxf(hi[d], s.seed[i * 6 + d]);
    for (int d = 0; d < 6; ++d)
      s.qb[threadIdx.x * 12 + d] = lo[d], s.qb[threadIdx.x * 12 + 6 + d] = hi[d];
  }
  __syncthreads();
}

// Whether some seed of the tile lies within the bandwidth of chunk c's box,
// for chunk c = blk * kBlockChunks + threadIdx.x of a surviving block:
// tested against the tile's box, each group's box (16 seeds), each quad's
// box (4 consecutive seeds), then the quad's seeds, among the seeds within
// the bandwidth of the block's box only (a seed beyond the bandwidth of the
// block's box is beyond it for each of its chunks: their boxes lie inside
// it).  Called by the whole CTA; two barriers.
__device__ __forceinline__ bool chunk_needed(TileSeeds &s, uint32_t blk, const float *bbox,
                                             const float *cbox, uint64_t nchunks, float skip_gap2) {
  __syncthreads();  // the previous block's mask is no longer read
  if (threadIdx.x < kChunk) {  // whole warps
    bool ok = false;
    if (s.alive[threadIdx.x])
      ok = point_gap2(s.seed + threadIdx.x * 6, bbox + uint64_t(blk) * 12) <= skip_gap2;
    const unsigned bal = __ballot_sync(0xffffffffu, ok);
    if ((threadIdx.x & 31) == 0) s.reach[threadIdx.x >> 5] = bal;
  }
  __syncthreads();
  const uint64_t c = uint64_t(blk) * kBlockChunks + threadIdx.x;
  bool keep = false;
  if (c < nchunks) {
    float cb[12];
    for (int d = 0; d < 12; ++d) cb[d] = cbox[c * 12 + d];
    if (box_gap2(s.gb, s.gb + 6, cb) <= skip_gap2)
      for (int g = 0; g < kChunk / kGroupSeeds && !keep; ++g) {
        const uint32_t gm = (s.reach[g >> 1] >> ((g & 1) * kGroupSeeds)) & 0xffffu;
        if (!gm) continue;
        const float *b = s.gb + 12 + 12 * g;
        if (box_gap2(b, b + 6, cb) > skip_gap2) continue;
        for (int qd = 4 * g; qd < 4 * g + 4 && !keep; ++qd) {
          const uint32_t qm = (gm >> (4 * (qd - 4 * g))) & 0xfu;
          if (!qm) continue;
          if (box_gap2(s.qb + 12 * qd, s.qb + 12 * qd + 6, cb) > skip_gap2) continue;
          for (int i = 4 * qd; i < 4 * qd + 4 && !keep; ++i)
            if ((qm >> (i - 4 * qd)) & 1u) keep = point_gap2(s.seed + i * 6, cb) <= skip_gap2;
        }
      }
  }
  return keep;
}

}  // namespace
}  // namespace sym
