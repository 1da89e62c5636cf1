// SPDX-License-Identifier: MPL-2.0
// BF16 tensor-core mean-shift bulk iterations on sm_103a (tcgen05 + TMEM).
//
// Flash-style, per (tile of 128 seeds, chunk of 128 votes), in units of the
// bandwidth h with the vote set's centre c_g and the chunk centre c_c:
//   u = (s - c_g)/h per seed, as a BF16 value + residue (once per tile)
//   E = (c_c - c_g)/h per chunk, v = (x - c_c)/h per vote, and the per-vote
//       constant f = -2 E.v as a BF16 value + residue (the chunk image)
//   MMA1  D[128x128] = [2u_hi, 1, 1 | 2u_lo, 1, 1] . [v, -|v|^2 | v, f]^T
//                    = 2 (u - E).v - |v|^2                 (tcgen05.mma K=16)
//   epilogue: w = relu(D + 1 - |u - E|^2) = max(0, 1 - |s - x|^2/h^2),
//           one packed FP32 add and one cvt.rn.relu.bf16x2 per two weights,
//           written as BF16 into shared memory
//   MMA2  ACC[128x16] += W[128x128] . [x_hi, 1, 0, x_lo]  (sum w x, sum w)
// The seed offsets are represented to ~2^-17 by their BF16 pairs and the
// epilogue uses the same represented values, so the large offsets cancel
// exactly; v is chunk-relative (small) and rounds once.  MMA2 uses the
// uncentred x split into BF16 value and residue plus a ones column, so sum
// w x and sum w come out of TMEM directly.
// The chunk image is laid out in the canonical no-swizzle K-major
// core-matrix order (8 rows x 16 bytes per core matrix), so one TMA bulk copy
// (cp.async.bulk + mbarrier complete_tx) stages a chunk.  Every mbarrier wait
// is bounded; on timeout the CTA records a status, drains its copies and
// MMAs, and frees its TMEM.
#include "chunk_lists.cuh"
#include "meanshift_fast.cuh"
#include "primitives.cuh"

#include <cuda_bf16.h>

#include <algorithm>
#include <cmath>
#include <vector>

namespace sym {
namespace {

// --------------------------------------------------------------- PTX glue
__device__ __forceinline__ uint32_t smem_u32(const void *p) {
  return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}

__device__ __forceinline__ void mbar_init(uint64_t *bar, uint32_t count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count) : "memory");
}

__device__ __forceinline__ void fence_mbar_init() {
  asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
}

__device__ __forceinline__ void mbar_expect_tx(uint64_t *bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)),
               "r"(bytes)
               : "memory");
}

// A waiting thread is suspended by the hardware until the phase completes
// (or kSuspendNs pass), so waiting warps take no issue slots from the
// working ones.
constexpr uint32_t kSuspendNs = 20000;
constexpr uint64_t kWaitLimitNs = 2000000000ull;  // a wait gives up after 2 s

__device__ __forceinline__ bool mbar_try_wait(uint64_t *bar, uint32_t parity) {
  uint32_t ok;
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2, %3;\n\t"
      "selp.u32 %0, 1, 0, p;\n\t}"
      : "=r"(ok)
      : "r"(smem_u32(bar)), "r"(parity), "r"(kSuspendNs)
      : "memory");
  return ok != 0;
}

__device__ __forceinline__ uint64_t global_ns() {
  uint64_t t;
  asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
  return t;
}

// Bounded wait: false when the barrier phase did not complete within
// limit_ns.
__device__ __forceinline__ bool mbar_wait(uint64_t *bar, uint32_t parity,
                                          uint64_t limit_ns = kWaitLimitNs) {
  if (mbar_try_wait(bar, parity)) return true;
  const uint64_t t0 = global_ns();
  do {
    if (mbar_try_wait(bar, parity)) return true;
  } while (global_ns() - t0 < limit_ns);
  return false;
}

// Bounded wait whose outcome is the same in every lane of the warp (each
// lane polls, so each performs the acquire; all agree on success).
__device__ __forceinline__ bool warp_wait(uint64_t *bar, uint32_t parity) {
  return __all_sync(0xffffffffu, mbar_wait(bar, parity));
}

__device__ __forceinline__ void tma_bulk_load(void *dst, const void *src, uint32_t bytes,
                                              uint64_t *bar) {
  asm volatile(
      "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
          smem_u32(dst)),
      "l"(src), "r"(bytes), "r"(smem_u32(bar))
      : "memory");
}

__device__ __forceinline__ void fence_async_smem() {
  asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
}
__device__ __forceinline__ void tc_fence_before() {
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
}
__device__ __forceinline__ void tc_fence_after() {
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
}

// Whole warp: allocate `cols` TMEM columns, address written to shared memory.
__device__ __forceinline__ void tmem_alloc(uint32_t *dst, uint32_t cols) {
  asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(
                   smem_u32(dst)),
               "r"(cols)
               : "memory");
  asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void tmem_dealloc(uint32_t taddr, uint32_t cols) {
  asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(taddr), "r"(cols)
               : "memory");
}

// Shared-memory matrix descriptor (sm_100 family): start address, leading
// (K-direction core-matrix) byte offset, stride (M/N-direction 8-row group)
// byte offset, descriptor version 1, no swizzle.
__device__ __forceinline__ uint64_t smem_desc(const void *p, uint32_t lbo, uint32_t sbo) {
  uint64_t d = (uint64_t(smem_u32(p)) >> 4) & 0x3FFFull;
  d |= uint64_t((lbo >> 4) & 0x3FFFu) << 16;
  d |= uint64_t((sbo >> 4) & 0x3FFFu) << 32;
  d |= uint64_t(1) << 46;
  return d;
}

// Instruction descriptor of kind::f16: F32 accumulator, BF16 A and B, both
// K-major, N >> 3 at bit 17, M >> 4 at bit 24.
__host__ __device__ constexpr uint32_t idesc_bf16(uint32_t m, uint32_t n) {
  return (1u << 4) | (1u << 7) | (1u << 10) | ((n >> 3) << 17) | ((m >> 4) << 24);
}

__device__ __forceinline__ void mma_bf16(uint32_t d_tmem, uint64_t a, uint64_t b, uint32_t idesc,
                                         uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}" ::"r"(d_tmem),
      "l"(a), "l"(b), "r"(idesc), "r"(accumulate)
      : "memory");
}

// Same, with the A operand (M x 16 BF16) read from TMEM at column a_tmem:
// row m in lane m, two K-consecutive elements per 32-bit column (the lower
// K index in the low half).
__device__ __forceinline__ void mma_bf16_ts(uint32_t d_tmem, uint32_t a_tmem, uint64_t b,
                                            uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n\t}" ::"r"(d_tmem),
      "r"(a_tmem), "l"(b), "r"(idesc), "r"(accumulate)
      : "memory");
}

__device__ __forceinline__ void mma_commit(uint64_t *bar) {
  asm volatile(
      "tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(
          smem_u32(bar))
      : "memory");
}

// 32 consecutive FP32 columns of this thread's TMEM lane.
__device__ __forceinline__ void tmem_ld32(uint32_t taddr, float (&v)[32]) {
  uint32_t r[32];
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x32.b32 "
      "{%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,"
      "%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31}, [%32];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]),
        "=r"(r[7]), "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]),
        "=r"(r[14]), "=r"(r[15]), "=r"(r[16]), "=r"(r[17]), "=r"(r[18]), "=r"(r[19]),
        "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]), "=r"(r[24]), "=r"(r[25]),
        "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
      : "r"(taddr));
  asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
  for (int i = 0; i < 32; ++i) v[i] = __uint_as_float(r[i]);
}

// This thread's TMEM lane, 32 (or 8) consecutive 32-bit columns from
// registers; tmem_wait_st makes them visible before the next handshake.
__device__ __forceinline__ void tmem_st32(uint32_t taddr, const uint32_t (&r)[32]) {
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x32.b32 [%0], "
      "{%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16,"
      "%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31,%32};" ::"r"(taddr),
      "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]),
      "r"(r[8]), "r"(r[9]), "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]),
      "r"(r[15]), "r"(r[16]), "r"(r[17]), "r"(r[18]), "r"(r[19]), "r"(r[20]), "r"(r[21]),
      "r"(r[22]), "r"(r[23]), "r"(r[24]), "r"(r[25]), "r"(r[26]), "r"(r[27]), "r"(r[28]),
      "r"(r[29]), "r"(r[30]), "r"(r[31])
      : "memory");
}
__device__ __forceinline__ void tmem_st16(uint32_t taddr, const uint32_t (&r)[16]) {
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], "
      "{%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16};" ::"r"(taddr),
      "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]),
      "r"(r[8]), "r"(r[9]), "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]),
      "r"(r[15])
      : "memory");
}
__device__ __forceinline__ void tmem_st8(uint32_t taddr, const uint32_t (&r)[8]) {
  asm volatile("tcgen05.st.sync.aligned.32x32b.x8.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8};" ::"r"(
                   taddr),
               "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]),
               "r"(r[7])
               : "memory");
}
__device__ __forceinline__ void tmem_wait_st() {
  asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
}

// tcgen05.ld of 32 columns without the wait (pair with tmem_wait_ld).
__device__ __forceinline__ void tmem_ld32_async(uint32_t taddr, uint32_t (&r)[32]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x32.b32 "
      "{%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,"
      "%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31}, [%32];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]),
        "=r"(r[7]), "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]),
        "=r"(r[14]), "=r"(r[15]), "=r"(r[16]), "=r"(r[17]), "=r"(r[18]), "=r"(r[19]),
        "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]), "=r"(r[24]), "=r"(r[25]),
        "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
      : "r"(taddr));
}
__device__ __forceinline__ void tmem_wait_ld() {
  asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
}

// ------------------------------------------------------------- layouts
// Canonical no-swizzle K-major tile of 16-bit elements: core matrices of 8
// rows x 8 elements (16 bytes per row), `lbo` bytes between K-adjacent core
// matrices, `sbo` bytes between row groups.
__host__ __device__ constexpr uint32_t kmajor_offset(uint32_t row, uint32_t k, uint32_t lbo,
                                                     uint32_t sbo) {
  return (row / 8) * sbo + (k / 8) * lbo + (row % 8) * 16 + (k % 8) * 2;
}

// Chunk image (one TMA bulk copy), built per mean-shift call for 1/h:
//   B1   128 votes x 16, K-major (LBO 128, SBO 256): v = (x - c_c)/h in k
//        0..5 and again in k 8..13; -|v|^2 of the rounded v as a BF16 value
//        and residue in k 6, 7 (-1e30 for padding votes, which then get
//        w = 0); f = -2 E.v as a BF16 value and residue in k 14, 15
//   B2   16 features x 128 votes, K-major (LBO 128, SBO 2048): BF16(x) in
//        features 0..5, ones in 6, the BF16 residue x - BF16(x) in 8..13
//   CEN  E = (c_c - c_g)/h (8 floats)
constexpr uint32_t kB1Bytes = 4096, kB2Bytes = 4096, kCenBytes = 32;
constexpr uint32_t kImage = kB1Bytes + kB2Bytes + kCenBytes;  // 8224
static_assert(kImage % 16 == 0, "TMA bulk copies move multiples of 16 bytes");

__device__ __forceinline__ void split_bf16(float x, __nv_bfloat16 &hi, __nv_bfloat16 &lo) {
  hi = __float2bfloat16_rn(x);
  lo = __float2bfloat16_rn(x - __bfloat162float(hi));
}

// Two consecutive BF16 values as one 32-bit TMEM column (first in the low half).
__device__ __forceinline__ uint32_t bf16_pair(const __nv_bfloat16 *p) {
  return uint32_t(__bfloat16_as_ushort(p[0])) | (uint32_t(__bfloat16_as_ushort(p[1])) << 16);
}

__global__ void build_images(const float *desc, uint64_t q, uint64_t nchunks, const float *cbox,
                             const float *gbox, float inv_h, uint8_t *images) {
  // the image is assembled in shared memory (its 2-byte entries lie 16 or
  // 128 bytes apart for neighbouring votes) and written out in 16-byte words
  __shared__ __align__(16) uint8_t img[kImage];
  uint64_t c = blockIdx.x;
  int t = threadIdx.x;  // vote in chunk
  if (c >= nchunks) return;
  const float *b = cbox + c * 12;
  float cen[6], e[6];
  for (int d = 0; d < 6; ++d) {
    cen[d] = 0.5f * (b[d] + b[6 + d]);
    e[d] = (cen[d] - 0.5f * (gbox[d] + gbox[6 + d])) * inv_h;
  }
  uint64_t v = c * kChunk + t;
  bool live = v < q;
  __nv_bfloat16 *b1 = reinterpret_cast<__nv_bfloat16 *>(img);
  __nv_bfloat16 *b2 = reinterpret_cast<__nv_bfloat16 *>(img + kB1Bytes);
  float *ce = reinterpret_cast<float *>(img + kB1Bytes + kB2Bytes);
  if (t < 8) ce[t] = t < 6 ? e[t] : 0.f;
  const __nv_bfloat16 zero = __float2bfloat16_rn(0.f);
  float n2 = 0, f = 0;
  for (int d = 0; d < 6; ++d) {
    float x = live ? desc[v * 8 + d] : 0.f;
    __nv_bfloat16 h = __float2bfloat16_rn(live ? (x - cen[d]) * inv_h : 0.f);
    float r = __bfloat162float(h);
    n2 = fmaf(r, r, n2);
    f = fmaf(-2.f * e[d], r, f);
    b1[kmajor_offset(t, d, 128, 256) / 2] = h;
    b1[kmajor_offset(t, 8 + d, 128, 256) / 2] = h;
    __nv_bfloat16 xh, xl;
    split_bf16(x, xh, xl);
    b2[kmajor_offset(d, t, 128, 2048) / 2] = xh;
    b2[kmajor_offset(8 + d, t, 128, 2048) / 2] = xl;
  }
  __nv_bfloat16 nh, nl, fh, fl;
  split_bf16(live ? -n2 : -1e30f, nh, nl);
  split_bf16(f, fh, fl);
  b1[kmajor_offset(t, 6, 128, 256) / 2] = nh;
  b1[kmajor_offset(t, 7, 128, 256) / 2] = nl;
  b1[kmajor_offset(t, 14, 128, 256) / 2] = fh;
  b1[kmajor_offset(t, 15, 128, 256) / 2] = fl;
  b2[kmajor_offset(6, t, 128, 2048) / 2] = __float2bfloat16_rn(live ? 1.f : 0.f);
  for (int k : {7, 14, 15}) b2[kmajor_offset(k, t, 128, 2048) / 2] = zero;
  __syncthreads();
  const uint4 *src = reinterpret_cast<const uint4 *>(img);
  uint4 *dst = reinterpret_cast<uint4 *>(images + c * kImage);
  for (int w = t; w < int(kImage / 16); w += kChunk) dst[w] = src[w];
}

// ------------------------------------------------- work lists per tile
// need[t * nchunks + c]: some seed of tile t lies within the bandwidth of
// chunk c's box (chunk_needed), for the chunks of tile t's surviving blocks.
// bcount[t * nblk + j] (zeroed by tile_boxes) gains the kept chunks of the
// tile's j-th surviving block, one integer atomic per warp: no barrier
// between blocks, and the counts do not depend on the order.
__global__ void __launch_bounds__(kListThreads) tile_count(const float *boxes, const float *means,
                                                           const int32_t *ids, const unsigned *nact,
                                                           const float *cbox, const float *bbox,
                                                           uint64_t nchunks, const uint32_t *sblk,
                                                           const uint32_t *nsurv, uint32_t nblk,
                                                           float skip_gap2, uint8_t *need,
                                                           uint32_t *bcount) {
  __shared__ TileSeeds seeds;
  chained();
  uint32_t t, sub, per;
  if (!list_share(nact, t, sub, per)) return;
  const uint32_t ns = nsurv[t];
  if (sub >= ns) return;
  load_tile(seeds, t, nact[0], boxes, means, ids);
  const int lane = threadIdx.x & 31;
  uint32_t *bc = bcount + uint64_t(t) * nblk;
  for (uint32_t j = sub; j < ns; j += per) {
    const uint32_t blk = sblk[uint64_t(t) * nblk + j];
    const bool keep = chunk_needed(seeds, blk, bbox, cbox, nchunks, skip_gap2);
    const uint64_t c = uint64_t(blk) * kBlockChunks + threadIdx.x;
    if (c < nchunks) need[uint64_t(t) * nchunks + c] = keep;
    const unsigned bal = __ballot_sync(0xffffffffu, keep);
    if (lane == 0 && bal) atomicAdd(&bc[j], unsigned(__popc(bal)));
  }
}

// Inclusive scan of one value per thread over a block of 1024 threads;
// `total` receives the block's sum.  Uses warp_sum[32] (shared).
__device__ __forceinline__ uint32_t block_scan_1024(uint32_t v, uint32_t *warp_sum, uint32_t &total) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  uint32_t x = v;
  for (int o = 1; o < 32; o <<= 1) {
    const uint32_t y = __shfl_up_sync(0xffffffffu, x, o);
    if (lane >= o) x += y;
  }
  if (lane == 31) warp_sum[warp] = x;
  __syncthreads();
  if (warp == 0) {
    uint32_t w = warp_sum[lane];
    for (int o = 1; o < 32; o <<= 1) {
      const uint32_t y = __shfl_up_sync(0xffffffffu, w, o);
      if (lane >= o) w += y;
    }
    warp_sum[lane] = w;  // inclusive over warps
  }
  __syncthreads();
  const uint32_t r = (warp ? warp_sum[warp - 1] : 0u) + x;
  total = warp_sum[31];
  __syncthreads();
  return r;
}

// One block of 1024 threads.  The surviving (tile, block) entries, tile by
// tile and in block order within a tile, form the list's order: seg[t] =
// exclusive scan of nsurv over the active tiles; boff[t * nblk + j] = the
// list position of entry (t, j)'s first kept chunk (exclusive scan of the
// counts over all entries in that order); offsets[t] = the first list
// entry of tile t (offsets[tiles] = the list length); and the work plan:
// tile t gets pieces[t+1] - pieces[t] CTAs, about len_t * budget / total
// of them (at least one), so every CTA streams a similar number of chunks;
// budget = sms - tiles (at least tiles), so the pieces fill one wave of the
// GPU.  seg holds max_tiles + 1 entries.  A list longer than `cap` (which
// the counts never give) records DS_CAPACITY and leaves an empty plan.
// Every iteration waits for this one block, so it takes few rounds
// (kScanEntries per thread), searches the tile of an entry in shared memory
// and plans with a thread per tile (20,000-sample motif sphere, 16 tiles at
// first: 7.1 us on average; with one entry per thread, the search in device
// memory and a serial plan 9.2).
constexpr int kScanEntries = 4, kScanTiles = 1024;
__global__ void __launch_bounds__(1024) scan_lists(const uint32_t *bcount, const uint32_t *nsurv,
                                                   const unsigned *nact, uint32_t nblk, uint32_t sms,
                                                   uint64_t cap, uint32_t *seg, uint32_t *boff,
                                                   uint64_t *offsets, uint32_t *pieces,
                                                   int *status) {
  __shared__ uint32_t warp_sum[32];
  __shared__ uint32_t seg_s[kScanTiles + 1];
  chained();
  const uint32_t tiles = active_tiles(nact);
  // exclusive scan over the rounds of a loop: the running total stays in a
  // register, the same in every thread
  uint32_t entries = 0;
  const bool near = tiles <= kScanTiles;  // seg fits in shared memory
  for (uint32_t base = 0; base < tiles; base += blockDim.x) {  // segment starts
    const uint32_t t = base + threadIdx.x;
    const uint32_t v = t < tiles ? nsurv[t] : 0u;
    uint32_t total;
    const uint32_t excl = entries + block_scan_1024(v, warp_sum, total) - v;
    if (t < tiles) {
      seg[t] = excl;
      if (near) seg_s[t] = excl;
    }
    entries += total;
  }
  if (threadIdx.x == 0) {
    seg[tiles] = entries;
    if (near) seg_s[tiles] = entries;
  }
  __syncthreads();
  const uint32_t *starts = near ? seg_s : seg;
  uint32_t list_len = 0;
  for (uint32_t base = 0; base < entries; base += blockDim.x * kScanEntries) {  // list positions
    const uint32_t e0 = base + threadIdx.x * kScanEntries;
    uint32_t at[kScanEntries], v[kScanEntries], tile[kScanEntries], sum = 0;
    uint32_t t = 0;
    if (e0 < entries) {  // the tile of entry e0: the last t with starts[t] <= e0
      uint32_t lo = 0, hi = tiles;  // starts[lo] <= e0 < starts[hi]
      while (hi - lo > 1) {
        const uint32_t mid = (lo + hi) >> 1;
        if (starts[mid] <= e0) lo = mid;
        else hi = mid;
      }
      t = lo;
    }
#pragma unroll
    for (int k = 0; k < kScanEntries; ++k) {
      const uint32_t e = e0 + k;
      v[k] = 0, at[k] = 0, tile[k] = t;
      if (e < entries) {
        while (starts[t + 1] <= e) ++t;
        tile[k] = t, at[k] = e - starts[t];
        v[k] = bcount[uint64_t(t) * nblk + at[k]];
      }
      sum += v[k];
    }
    uint32_t total;
    uint32_t run = list_len + block_scan_1024(sum, warp_sum, total) - sum;
#pragma unroll
    for (int k = 0; k < kScanEntries; ++k) {
      if (e0 + k < entries) {
        boff[uint64_t(tile[k]) * nblk + at[k]] = run;
        // a tile's first entry starts it, and the empty tiles before it
        if (at[k] == 0)
          for (uint32_t x = tile[k] + 1; x-- > 0 && starts[x] == e0 + k;) offsets[x] = run;
      }
      run += v[k];
    }
    list_len += total;
  }
  for (uint32_t t = threadIdx.x; t <= tiles; t += blockDim.x)
    if (starts[t] == entries) offsets[t] = list_len;  // the empty tiles at the end, and the end
  __syncthreads();
  if (list_len > cap) {
    for (uint32_t t = threadIdx.x; t <= tiles; t += blockDim.x) offsets[t] = 0, pieces[t] = 0;
    if (threadIdx.x == 0) atomicExch(status, DS_CAPACITY);
    return;
  }
  const uint32_t budget = tiles < sms ? sms - tiles : tiles;
  uint32_t planned = 0;
  for (uint32_t base = 0; base < tiles; base += blockDim.x) {
    const uint32_t t = base + threadIdx.x;
    uint32_t v = 0;
    if (t < tiles) {
      const uint64_t len = offsets[t + 1] - offsets[t];
      const uint64_t want = list_len ? (len * budget + list_len - 1) / list_len : 1;
      v = uint32_t(want ? want : 1);
    }
    uint32_t total;
    const uint32_t excl = planned + block_scan_1024(v, warp_sum, total) - v;
    if (t < tiles) pieces[t] = excl;
    planned += total;
  }
  if (threadIdx.x == 0) pieces[tiles] = planned;
}

// list[boff[t * nblk + j] + r] = t * nchunks + c for the r-th kept chunk c
// (ascending) of tile t's j-th surviving block: per tile, the kept chunks in
// ascending order.  CTAs shared among tiles as tile_count's.
__global__ void __launch_bounds__(kListThreads) scatter_lists(const uint8_t *need,
                                                              const uint32_t *boff,
                                                              const uint32_t *bcount,
                                                              const uint32_t *sblk,
                                                              const uint32_t *nsurv, uint32_t nblk,
                                                              const unsigned *nact,
                                                              uint64_t nchunks, uint64_t cap,
                                                              int32_t *list, int *status) {
  __shared__ uint32_t warp_cnt[kListThreads / 32];
  chained();
  uint32_t t, sub, per;
  if (!list_share(nact, t, sub, per)) return;
  const uint32_t ns = nsurv[t];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  for (uint32_t j = sub; j < ns; j += per) {
    const uint64_t e = uint64_t(t) * nblk + j;
    if (!bcount[e]) continue;  // the same for the whole CTA
    const uint64_t c = uint64_t(sblk[e]) * kBlockChunks + threadIdx.x;
    const bool keep = c < nchunks && need[uint64_t(t) * nchunks + c];
    const uint32_t bal = __ballot_sync(0xffffffffu, keep);
    if (lane == 0) warp_cnt[warp] = __popc(bal);
    __syncthreads();
    uint64_t before = boff[e];
    for (int w = 0; w < warp; ++w) before += warp_cnt[w];
    before += __popc(bal & ((1u << lane) - 1u));
    if (keep && before < cap) list[before] = int32_t(uint64_t(t) * nchunks + c);
    else if (keep) atomicExch(status, DS_CAPACITY);
    __syncthreads();
  }
}

// --------------------------------------------- pipelined tensor kernel
// Warp roles (19 warps):
//   warps 0..15  the epilogue, two pairs of warpgroups taking alternate
//                chunks (pair p = warp / 8 owns the chunks i with
//                i % 2 == p); in a pair, warp w reads TMEM lanes 32(w%4)..
//                and D columns 64((w/4)%2)..+63
//   warp 16      TMA: streams the chunk images through the stage ring
//   warps 17, 18 MMA issue for pair 0 / pair 1 (one lane each): MMA1 of
//                the pair's chunk k + 1 once it landed and D[p] was read,
//                then MMA2 of chunk k once W[p] was written.
//                A single thread issues one tcgen05.mma per ~85 cycles
//                whatever its N, while the tensor pipe takes an N = 16 MMA
//                every ~40 cycles from two issuers (measured on GB300), so
//                each pair drives its own stream of MMAs
//   shared memory  kStagesTc TMA buffers of one chunk image each, ATILE
//                  (A operand of MMA1, once per tile), U
//   TMEM columns   D[p] = 128p (MMA1 accumulators), W[p] = 256 + 64p (the
//                  BF16 weights, A operand of MMA2), ACC[p][q] = 384 + 64p
//                  + 16q for q = 0..3 (pair p's accumulators, K-step q of
//                  MMA2 into ACC[p][q % 4]; zeroed at the start, summed in
//                  a fixed order at the end)
// mbarriers: load_full[s] (TMA bytes), stage_free[s] (MMA2 of the chunk in
// stage s done; arrived at by the pair once its wait for that MMA2 passed), d_full[p] (MMA1 done), d_free[p] (pair p read D[p]),
// w_full[p] (pair p wrote W[p]), w_free[p] (MMA2 done), acc_done[p].  Every
// wait is bounded; on timeout a warp records the status and stops, an MMA
// warp drains its MMAs into acc_done[p], the TMA warp its copies.
constexpr int kStagesTc = 12;
constexpr int kPairWarps = 8, kTmaWarp = 16, kMmaWarp = 17;  // warps 0..15: the two pairs
constexpr int kThreadsTc = 19 * 32;
constexpr uint32_t kTcStage = 0;                                     // kStagesTc x kImage
constexpr uint32_t kTcU = (kStagesTc * kImage + 1023) / 1024 * 1024; // 128 x 8 floats
constexpr uint32_t kTcATile = kTcU + 128 * 8 * 4;                    // 4096, K-major
constexpr uint32_t kTcBars = kTcATile + 4096;                        // 2 kStagesTc + 10
constexpr uint32_t kTcMisc = kTcBars + 48 * 8;                      // TMEM address, K-step masks
constexpr uint32_t kTcSmem = kTcMisc + 64;
static_assert(kImage % 16 == 0, "TMA alignment");
static_assert(kTcATile % 1024 == 0, "descriptor alignment");
static_assert(2 * kStagesTc + 10 <= 48, "barrier slots");
static_assert(kTcSmem <= 227 * 1024, "shared memory per CTA");
constexpr uint32_t kTcCols = 512, kTcColW = 256, kTcColAcc = 384;

struct TcArgs {
  const uint8_t *images;
  uint64_t nchunks;
  const int32_t *list;      // needed (tile, chunk) entries, t * nchunks + c
  const uint64_t *offsets;  // tiles + 1: first list entry of each tile
  const uint32_t *pieces;   // tiles + 1: first piece (CTA) of each tile
  const unsigned *nact;     // nact[0] = active seeds (tiles of kChunk)
  const float *means;
  const int32_t *ids;
  const float *gbox;        // box of all votes; its centre is c_g
  float inv_h;
  float gauss_k2;           // 0: Epanechnikov; k > 0 (a power of 2): 2^(-k d^2/h^2) - 2^-k
  float *partial;
  unsigned long long *evals;
  Progress *progress;
  bool timed;  // began and ended of it
  int *status;
};

__device__ __forceinline__ void mbar_arrive(uint64_t *bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(bar)) : "memory");
}


// d = a * b + c on two FP32 lanes at once.
__device__ __forceinline__ float2 fma2(float2 a, float2 b, float2 c) {
  unsigned long long ra, rb, rc, rd;
  memcpy(&ra, &a, 8), memcpy(&rb, &b, 8), memcpy(&rc, &c, 8);
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(rd) : "l"(ra), "l"(rb), "l"(rc));
  float2 d;
  memcpy(&d, &rd, 8);
  return d;
}

// {relu(lo), relu(hi)} rounded to BF16 and packed, lo in the low half.
__device__ __forceinline__ uint32_t relu_bf16x2(float lo, float hi) {
  uint32_t r;
  asm("cvt.rn.relu.bf16x2.f32 %0, %1, %2;" : "=r"(r) : "f"(hi), "f"(lo));
  return r;
}

// Shifted Gaussian weights 2^a - 2^-k from the exponents a = -k d^2 / h^2
// (the MMA's D with the seed operand scaled by k, plus -k |u - E|^2), two at
// a time: the exponents rounded to BF16, one MUFU BF16x2 base-2
// exponential, one BF16x2 FMA with relu (votes past the cut, a < -k, get 0).
__device__ __forceinline__ uint32_t gauss_bf16x2(float lo, float hi, uint32_t neg_floor2) {
  uint32_t x, e, w;
  asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(x) : "f"(hi), "f"(lo));
  asm("ex2.approx.ftz.bf16x2 %0, %1;" : "=r"(e) : "r"(x));
  asm("fma.rn.relu.bf16x2 %0, %1, %2, %3;" : "=r"(w) : "r"(e), "r"(0x3F803F80u), "r"(neg_floor2));
  return w;
}

// ACC[q % 4] += W[:, 16q..16q+15] . B2[:, 16q..16q+15]^T for the eight
// K-steps q of the chunk (16 votes each); W in TMEM, the accumulators start
// at zero.  Unrolled with constant descriptor offsets: the issuing thread
// waits ~50 cycles per tcgen05.mma, and every instruction between two MMAs
// adds to that (a branch per K-step nearly doubled the cost on GB300).
// Skipping all-zero K-steps saves nothing once the tile's chunk list is
// culled per seed: under 1% of the 16-vote x 128-seed blocks are zero.
__device__ __forceinline__ void mma2_chunk(uint32_t acc, uint32_t w_tmem, const uint8_t *b2) {
  const uint64_t b = smem_desc(b2, 128, 2048);
#pragma unroll
  for (uint32_t q = 0; q < 8; ++q)
    mma_bf16_ts(acc + 16 * (q & 3u), w_tmem + 8 * q, b + 16 * q, idesc_bf16(128, 16), 1u);
}

__global__ void __launch_bounds__(kThreadsTc, 1) ms_tile_tc(TcArgs a) {
  chained();
  extern __shared__ __align__(1024) uint8_t smem[];
  uint8_t *stage = smem + kTcStage;
  float *U = reinterpret_cast<float *>(smem + kTcU);
  uint8_t *ATILE = smem + kTcATile;
  uint64_t *bars = reinterpret_cast<uint64_t *>(smem + kTcBars);
  uint64_t *load_full = bars, *stage_free = bars + kStagesTc;
  uint64_t *d_full = bars + 2 * kStagesTc, *d_free = d_full + 2, *w_full = d_full + 4;
  uint64_t *w_free = d_full + 6, *acc_done = d_full + 8;  // acc_done[2]
  uint32_t *tmem_slot = reinterpret_cast<uint32_t *>(smem + kTcMisc);

  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  // piece -> (tile, share of the tile's list)
  const uint32_t piece = blockIdx.x;
  const uint32_t ntiles = active_tiles(a.nact);
  if (piece >= a.pieces[ntiles]) return;
  // the launch's own time: its first CTA's start to its last CTA's end by the
  // device's clock (events around the launch kept it from being chained and cost
  // 9 us per iteration)
  if (tid == 0 && a.timed) atomicMin(&a.progress->began, (unsigned long long)global_ns());
  const uint64_t nactive = a.nact[0];
  uint64_t lo_t = 0, hi_t = ntiles;  // last tile whose first piece is <= piece
  while (hi_t - lo_t > 1) {
    uint64_t mid = (lo_t + hi_t) / 2;
    if (a.pieces[mid] <= piece) lo_t = mid;
    else hi_t = mid;
  }
  const uint64_t tile = lo_t;
  const uint64_t k = piece - a.pieces[tile], np = a.pieces[tile + 1] - a.pieces[tile];
  const uint64_t lt0 = a.offsets[tile], len = a.offsets[tile + 1] - lt0;
  const uint64_t e0 = lt0 + len * k / np, e1 = lt0 + len * (k + 1) / np;
  const uint32_t n = uint32_t(e1 - e0);
  const uint64_t tbase = tile * a.nchunks;

  // u = (s - c_g)/h of this tile's seeds: U (FP32 sums of the BF16 pairs)
  // and ATILE rows [2u_hi, 1, 1 | 2u_lo, 1, 1] in shared memory
  if (tid < kChunk) {
    uint64_t slot = tile * kChunk + tid;
    bool live = slot < nactive;
    int32_t sd = live ? a.ids[slot] : 0;
    __align__(16) __nv_bfloat16 k0[8], k1[8];
    // Gaussian weights: the whole operand scaled by the power of two k
    // (exact in BF16), so D comes out as k times the Epanechnikov D
    const float kscale = a.gauss_k2 > 0.f ? a.gauss_k2 : 1.f;
    const __nv_bfloat16 kone = __float2bfloat16_rn(kscale);
    for (int d = 0; d < 6; ++d) {
      float cg = 0.5f * (a.gbox[d] + a.gbox[6 + d]);
      float u = live ? (a.means[uint64_t(sd) * 8 + d] - cg) * a.inv_h : 0.f;
      __nv_bfloat16 hi, lo;
      split_bf16(u, hi, lo);
      U[tid * 8 + d] = __bfloat162float(hi) + __bfloat162float(lo);
      k0[d] = __float2bfloat16_rn(2.f * kscale * __bfloat162float(hi));  // exact
      k1[d] = __float2bfloat16_rn(2.f * kscale * __bfloat162float(lo));
    }
    k0[6] = k0[7] = k1[6] = k1[7] = kone;
    *reinterpret_cast<uint4 *>(ATILE + kmajor_offset(tid, 0, 128, 256)) = *reinterpret_cast<uint4 *>(k0);
    *reinterpret_cast<uint4 *>(ATILE + kmajor_offset(tid, 8, 128, 256)) = *reinterpret_cast<uint4 *>(k1);
  }
  if (tid == 0) {
    for (int s = 0; s < kStagesTc; ++s) mbar_init(&load_full[s], 1), mbar_init(&stage_free[s], 1);
    for (int p = 0; p < 2; ++p) {
      mbar_init(&d_full[p], 1), mbar_init(&w_free[p], 1);
      mbar_init(&d_free[p], kPairWarps), mbar_init(&w_full[p], kPairWarps);
    }
    mbar_init(&acc_done[0], 1), mbar_init(&acc_done[1], 1);
    fence_mbar_init();
  }
  if (warp == 0 && n) tmem_alloc(tmem_slot, kTcCols);
  fence_async_smem();  // ATILE written by the generic proxy, read by the MMA
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = n ? *tmem_slot : 0;
  auto stage_of = [&](uint32_t i) { return stage + (i % kStagesTc) * kImage; };
  if (n && warp < 4) {  // ACC starts at zero (MMA2 always accumulates)
    uint32_t z[32];
    for (int j = 0; j < 32; ++j) z[j] = 0u;
    for (int q2 = 0; q2 < 4; ++q2) tmem_st32(tmem + (uint32_t(warp * 32) << 16) + kTcColAcc + 32 * q2, z);
    tmem_wait_st();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();

  if (warp == kTmaWarp) {
    // ------------------------------------------------ TMA producer
    // chunk ids of the work list, 32 per batch, lane l holding entry
    // 32 * batch + l; the next batch is loaded one batch ahead, so no
    // global-load latency sits on the issue path.  chunk_of is called by the
    // whole warp with non-decreasing i.
    auto load_batch = [&](uint32_t batch) -> uint32_t {
      uint32_t idx = batch * 32 + lane;
      return idx < n ? uint32_t(uint64_t(a.list[e0 + idx]) - tbase) : 0u;
    };
    uint32_t cur = load_batch(0), nxt = load_batch(1), cur_batch = 0;
    auto chunk_of = [&](uint32_t i) -> uint64_t {
      while (i / 32 != cur_batch) {
        cur = nxt;
        nxt = load_batch(++cur_batch + 1);
      }
      return __shfl_sync(0xffffffffu, cur, i % 32);
    };
    bool ok = true;
    uint32_t issued = 0;
    for (; issued < n && issued < uint32_t(kStagesTc); ++issued) {
      const uint64_t c = chunk_of(issued);
      if (lane == 0) {
        mbar_expect_tx(&load_full[issued], kImage);
        tma_bulk_load(stage + issued * kImage, a.images + c * kImage, kImage, &load_full[issued]);
      }
    }
    // chunk j + kStagesTc reuses the stage of chunk j once MMA2(j) is done
    for (uint32_t j = 0; j + kStagesTc < n; ++j) {
      const uint64_t c = chunk_of(j + kStagesTc);
      ok = warp_wait(&stage_free[j % kStagesTc], (j / kStagesTc) & 1);
      if (!ok) break;
      if (lane == 0) {
        mbar_expect_tx(&load_full[j % kStagesTc], kImage);
        tma_bulk_load(stage_of(j), a.images + c * kImage, kImage, &load_full[j % kStagesTc]);
      }
      ++issued;
    }
    if (!ok && lane == 0) {
      atomicExch(a.status, DS_SPIN_LIMIT);
      // drain: wait (bounded) for every copy issued, so none lands after exit
      for (uint32_t c = 0; c < issued; ++c) mbar_wait(&load_full[c % kStagesTc], (c / kStagesTc) & 1);
    }
  } else if (warp >= kMmaWarp) {
    // ------------------------------------------------ MMA issue, pair p
    const uint32_t p = uint32_t(warp - kMmaWarp);
    const uint32_t np = n > p ? (n - p + 1) / 2 : 0;  // chunks 2k + p of the pair
    if (lane == 0 && n) {
      bool ok = true;
      const uint32_t dcol = tmem + 128 * p, wcol = tmem + kTcColW + 64 * p;
      const uint32_t acc = tmem + kTcColAcc + 64 * p;
      // MMA1 of the pair's chunk k (chunk 2k + p) once it landed and the
      // pair read D[p] for chunk k - 1
      auto mma1 = [&](uint32_t k) -> bool {
        const uint32_t i = 2 * k + p;
        if (!mbar_wait(&load_full[i % kStagesTc], (i / kStagesTc) & 1)) return false;
        if (k > 0 && !mbar_wait(&d_free[p], (k - 1) & 1)) return false;
        tc_fence_after();
        mma_bf16(dcol, smem_desc(ATILE, 128, 256), smem_desc(stage_of(i), 128, 256),
                 idesc_bf16(128, 128), 0);
        mma_commit(&d_full[p]);
        return true;
      };
      // the pair reads D for chunk k before it writes W for chunk k, so
      // MMA1(k + 1) is always ready before MMA2(k): the issuer takes them in
      // that order, sleeping in each wait
      if (np) ok = mma1(0);
      for (uint32_t k = 0; ok && k < np; ++k) {
        if (k + 1 < np && !(ok = mma1(k + 1))) break;
        if (!(ok = mbar_wait(&w_full[p], k & 1))) break;  // the pair wrote W[p]
        tc_fence_after();
        mma2_chunk(acc, wcol, stage_of(2 * k + p) + kB1Bytes);
        mma_commit(&w_free[p]);  // W[p] and the chunk's stage are free again
      }
      if (!ok) atomicExch(a.status, DS_SPIN_LIMIT);
      mma_commit(&acc_done[p]);  // once every MMA issued has completed
    }
    __syncwarp();
  } else {
    // ------------------------------------------------ pair p
    // row `row`, D columns 64h..64h+63:  w = relu(D + 1 - |u - E|^2)
    const int p = warp / kPairWarps, quad = warp & 3, h = (warp >> 2) & 1, row = quad * 32 + lane;
    const float *u = U + row * 8;
    const float2 one2 = make_float2(1.f, 1.f);
    const uint32_t lane_base = uint32_t(quad * 32) << 16;
    const uint32_t dcol = tmem + 128 * p + 64 * h, wcol = tmem + kTcColW + 64 * p + 32 * h;
    const bool gauss = a.gauss_k2 > 0.f;
    uint32_t neg_floor2 = 0;  // -2^-k in both BF16 halves
    if (gauss) {
      const uint32_t h16 = __bfloat16_as_ushort(__float2bfloat16_rn(-exp2f(-a.gauss_k2)));
      neg_floor2 = h16 | (h16 << 16);
    }
    bool ok = true;
    uint32_t kth = 0;  // index of chunk i among the pair's chunks
    for (uint32_t i = p; i < n; i += 2, ++kth) {
      if (!warp_wait(&d_full[p], kth & 1) ||
          !warp_wait(&load_full[i % kStagesTc], (i / kStagesTc) & 1)) {
        ok = false;
        break;
      }
      tc_fence_after();
      const float *E = reinterpret_cast<const float *>(stage_of(i) + kB1Bytes + kB2Bytes);
      float rowc = 1.f;
      for (int d = 0; d < 6; ++d) {
        float r = u[d] - E[d];
        rowc = fmaf(-r, r, rowc);
      }
      uint32_t w[16], w2[16];
      {
        uint32_t d0[32], d1[32];
        tmem_ld32_async(lane_base + dcol, d0);
        tmem_ld32_async(lane_base + dcol + 32, d1);
        tmem_wait_ld();
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(&d_free[p]);  // D[p] may be overwritten
        if (gauss) {  // a = k D - k |u - E|^2 = -k d^2 / h^2
          const float rowg = a.gauss_k2 * (rowc - 1.f);
          const float2 rowg2 = make_float2(rowg, rowg);
          for (int j = 0; j < 16; ++j) {
            float2 t = fma2(make_float2(__uint_as_float(d0[2 * j]), __uint_as_float(d0[2 * j + 1])),
                            one2, rowg2);
            w[j] = gauss_bf16x2(t.x, t.y, neg_floor2);
          }
          for (int j = 0; j < 16; ++j) {
            float2 t = fma2(make_float2(__uint_as_float(d1[2 * j]), __uint_as_float(d1[2 * j + 1])),
                            one2, rowg2);
            w2[j] = gauss_bf16x2(t.x, t.y, neg_floor2);
          }
        } else {
          const float2 rowc2 = make_float2(rowc, rowc);
          for (int j = 0; j < 16; ++j) {
            float2 t = fma2(make_float2(__uint_as_float(d0[2 * j]), __uint_as_float(d0[2 * j + 1])),
                            one2, rowc2);
            w[j] = relu_bf16x2(t.x, t.y);
          }
          for (int j = 0; j < 16; ++j) {
            float2 t = fma2(make_float2(__uint_as_float(d1[2 * j]), __uint_as_float(d1[2 * j + 1])),
                            one2, rowc2);
            w2[j] = relu_bf16x2(t.x, t.y);
          }
        }
      }
      if (kth > 0) {
        if (!warp_wait(&w_free[p], (kth - 1) & 1)) {  // MMA2(i-2) read W[p]
          ok = false;
          break;
        }
        // MMA2(i-2) also finished reading chunk i-2's stage, and the pair
        // read its centre before w_full: the TMA warp may refill it (the
        // last two chunks of a pair are never refilled)
        if (quad == 0 && h == 0 && lane == 0) mbar_arrive(&stage_free[(i - 2) % kStagesTc]);
      }
      tc_fence_after();
      tmem_st16(lane_base + wcol, w);
      tmem_st16(lane_base + wcol + 16, w2);
      tmem_wait_st();
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(&w_full[p]);
    }
    if (!ok && lane == 0) atomicExch(a.status, DS_SPIN_LIMIT);
  }
  __syncthreads();
  if (warp < 4) {  // warpgroup 0 writes the tile's partial sums
    const int quad = warp & 3, row = quad * 32 + lane;
    float acc[16];
    for (int j = 0; j < 16; ++j) acc[j] = 0.f;
    if (n && warp_wait(&acc_done[0], 0) && warp_wait(&acc_done[1], 0)) {
      tc_fence_after();
      for (int q2 = 0; q2 < 4; ++q2) {  // ACC[0][0..3], ACC[1][0..3], two per load
        float v[32];
        tmem_ld32(tmem + (uint32_t(quad * 32) << 16) + kTcColAcc + 32 * q2, v);
        for (int j = 0; j < 16; ++j) acc[j] += v[j];
        for (int j = 0; j < 16; ++j) acc[j] += v[16 + j];
      }
    }
    // piece-major: value d of row r of piece p at (p * 8 + d) * 128 + r
    float *out = a.partial + uint64_t(piece) * 8 * kChunk + row;
    for (int d = 0; d < 6; ++d) out[d * kChunk] = acc[d] + acc[8 + d];  // BF16 x + its residue
    out[6 * kChunk] = acc[6];
  }
  if (tid == 0 && n && a.evals) atomicAdd(a.evals, uint64_t(n) * uint64_t(kChunk * kChunk));
  tc_fence_before();
  __syncthreads();
  if (warp == 0 && n) tmem_dealloc(tmem, kTcCols);
  if (tid == 0 && a.timed) atomicMax(&a.progress->ended, (unsigned long long)global_ns());
}

// ------------------------------------------------------ tensor self-test
// One tile: D = A1 . B1^T (128 x 128 x 16) and ACC = A2 . B2^T (128 x 16 x
// 128) from row-major BF16 inputs, through the same paths as ms_tile_tc: B
// operands in the canonical shared-memory layout staged by one TMA bulk
// copy, A operands written to TMEM with tcgen05.st, tcgen05.mma with A from
// TMEM, results read with tcgen05.ld.
constexpr uint32_t kSelfB2 = 4096;
constexpr uint32_t kOffStage = 0, kOffBars = 8192, kOffMisc = kOffBars + 64;
constexpr uint32_t kSmemRequest = 16 * 1024;
constexpr uint32_t kTmemCols = 256, kColD = 0, kColAcc = 128, kColA1 = 160, kColA2 = 192;

__global__ void __launch_bounds__(256, 1) tc_selftest(const __nv_bfloat16 *a1, const __nv_bfloat16 *b1,
                                                      const __nv_bfloat16 *a2, const __nv_bfloat16 *b2,
                                                      uint8_t *scratch, float *d_out, float *acc_out,
                                                      int *status) {
  extern __shared__ __align__(1024) uint8_t smem[];
  uint8_t *S = smem + kOffStage;
  uint64_t *bar = reinterpret_cast<uint64_t *>(smem + kOffBars);
  uint32_t *tmem_slot = reinterpret_cast<uint32_t *>(smem + kOffMisc);
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, quad = warp & 3, wg = warp >> 2;
  const int row = quad * 32 + lane;
  // stage B1 | B2 in global scratch in the canonical layout, then TMA it in
  if (tid < 128) {
    __nv_bfloat16 *g1 = reinterpret_cast<__nv_bfloat16 *>(scratch);
    __nv_bfloat16 *g2 = reinterpret_cast<__nv_bfloat16 *>(scratch + kB1Bytes);
    for (int k = 0; k < 16; ++k) {
      g1[kmajor_offset(tid, k, 128, 256) / 2] = b1[tid * 16 + k];
      g2[kmajor_offset(k, tid, 128, 2048) / 2] = b2[k * 128 + tid];
    }
    asm volatile("fence.proxy.async.global;" ::: "memory");
  }
  if (tid == 0) {
    mbar_init(&bar[0], 1);
    mbar_init(&bar[1], 1);
    fence_mbar_init();
  }
  if (warp == 0) tmem_alloc(tmem_slot, kTmemCols);
  __threadfence();
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = *tmem_slot;
  if (wg == 0) {  // A1 and A2 rows into TMEM, lane = row
    const uint32_t lane_base = uint32_t(quad * 32) << 16;
    uint32_t r8[8], r32[32];
    for (int c = 0; c < 8; ++c) r8[c] = bf16_pair(a1 + row * 16 + 2 * c);
    tmem_st8(tmem + lane_base + kColA1, r8);
    for (int half = 0; half < 2; ++half) {
      for (int c = 0; c < 32; ++c) r32[c] = bf16_pair(a2 + row * 128 + 64 * half + 2 * c);
      tmem_st32(tmem + lane_base + kColA2 + 32 * half, r32);
    }
    tmem_wait_st();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  bool ok = true;
  if (tid == 0) {
    asm volatile("fence.proxy.async.global;" ::: "memory");
    mbar_expect_tx(&bar[0], kB1Bytes + kSelfB2);
    tma_bulk_load(S, scratch, kB1Bytes + kSelfB2, &bar[0]);
  }
  ok = __syncthreads_and(mbar_wait(&bar[0], 0));
  if (ok && tid == 0) {
    tc_fence_after();
    mma_bf16_ts(tmem + kColD, tmem + kColA1, smem_desc(S, 128, 256), idesc_bf16(128, 128), 0);
    for (uint32_t s = 0; s < 8; ++s)
      mma_bf16_ts(tmem + kColAcc, tmem + kColA2 + 8 * s, smem_desc(S + kB1Bytes + s * 256, 128, 2048),
                  idesc_bf16(128, 16), s > 0);
    mma_commit(&bar[1]);
  }
  if (ok) ok = __syncthreads_and(mbar_wait(&bar[1], 0));
  tc_fence_after();
  if (ok) {
    for (int half = 0; half < 2; ++half) {
      float v[32];
      uint32_t col = 64 * wg + 32 * half;
      tmem_ld32(tmem + (uint32_t(quad * 32) << 16) + kColD + col, v);
      for (int j = 0; j < 32; ++j) d_out[row * 128 + col + j] = v[j];
    }
    if (wg == 0) {
      float v[32];
      tmem_ld32(tmem + (uint32_t(quad * 32) << 16) + kColAcc, v);
      for (int j = 0; j < 16; ++j) acc_out[row * 16 + j] = v[j];
    }
  }
  if (!ok && tid == 0) atomicExch(status, DS_SPIN_LIMIT);
  tc_fence_before();
  __syncthreads();
  if (warp == 0) tmem_dealloc(tmem, kTmemCols);
}

// The kernels' bounded wait made to run out: one warp holds TMEM as the
// mean-shift kernel does, waits with mbar_wait on a barrier nothing arrives
// at, with a limit of limit_ns instead of 2 s, then records DS_SPIN_LIMIT,
// frees its TMEM and returns -- the path a real kernel takes when a copy or
// an MMA never completes.  No copy or MMA is issued.
__global__ void __launch_bounds__(32, 1) wait_selftest(uint64_t limit_ns, int *status) {
  __shared__ __align__(8) uint64_t bar;
  __shared__ uint32_t tmem_slot;
  if (threadIdx.x == 0) {
    mbar_init(&bar, 1);
    fence_mbar_init();
  }
  tmem_alloc(&tmem_slot, 32);
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = tmem_slot;
  const bool ok = __all_sync(0xffffffffu, mbar_wait(&bar, 0, limit_ns));
  if (!ok && threadIdx.x == 0) atomicExch(status, DS_SPIN_LIMIT);
  tc_fence_before();
  __syncthreads();
  tmem_dealloc(tmem, 32);
}

// Sum of a seed's pieces (fixed order), then the mean-shift step; a seed
// leaves the bulk (kNear: the FP32 polish takes it on with Newton steps)
// when its squared move falls under kSwitch2 h^2.
// A block serves kUpdateSeeds neighbouring seeds: thread (y, x) adds the
// pieces y, y + 32, ... of seed x, so eight threads read one 32-byte sector of
// the partial sums and kUpdateAhead rounds of loads are in flight; then
// through shared memory warp x takes seed x, the lanes its 32 sums, and a
// fixed butterfly adds them.  Latency-bound: 4 us at 128 seeds and 152 pieces, 6
// at 2,048; a warp per seed, whose lanes read one float of 32 pieces each and
// which stored each coordinate before it loaded the next, took 19 and 37.
constexpr int kUpdateSeeds = 8, kUpdateAhead = 8;
__global__ void __launch_bounds__(32 * kUpdateSeeds) ms_update_bulk(float *means, const float *partial,
                                                                    const uint32_t *pieces,
                                                                    const int32_t *ids,
                                                                    const unsigned *nact, float h2,
                                                                    uint8_t *state) {
  __shared__ float sums[7][32][kUpdateSeeds + 1];
  chained();
  const uint64_t slot0 = uint64_t(blockIdx.x) * kUpdateSeeds;
  const unsigned n = nact[0];
  if (slot0 >= n) return;  // the whole block
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const uint64_t tile = slot0 / kChunk;
  float acc[7] = {0, 0, 0, 0, 0, 0, 0};
  const uint32_t x = threadIdx.x % kUpdateSeeds, y = threadIdx.x / kUpdateSeeds;
  const uint32_t p1 = pieces[tile + 1];
  const float *in = partial + slot0 % kChunk + x;
  for (uint32_t p = pieces[tile] + y; p < p1; p += 32 * kUpdateAhead) {
    float v[kUpdateAhead][7];
#pragma unroll
    for (int r = 0; r < kUpdateAhead; ++r)
      if (p + 32 * r < p1)
#pragma unroll
        for (int d = 0; d < 7; ++d) v[r][d] = in[(uint64_t(p + 32 * r) * 8 + d) * kChunk];
#pragma unroll
    for (int r = 0; r < kUpdateAhead; ++r)
      if (p + 32 * r < p1)
#pragma unroll
        for (int d = 0; d < 7; ++d) acc[d] += v[r][d];
  }
  for (int d = 0; d < 7; ++d) sums[d][y][x] = acc[d];
  __syncthreads();
  const uint64_t slot = slot0 + warp;
  if (slot >= n) return;  // whole warp
  const int32_t s = ids[slot];
  for (int d = 0; d < 7; ++d) acc[d] = sums[d][lane][warp];
  for (int d = 0; d < 7; ++d)
    for (int o = 16; o; o >>= 1) acc[d] += __shfl_xor_sync(0xffffffffu, acc[d], o);
  if (lane != 0) return;
  if (acc[6] <= 1e-14f) {
    state[s] = kExhausted;
    return;
  }
  // every load before the first store: a load behind a store to its own line
  // waits for it (a store per coordinate between the loads took 14 us more)
  float *mean = means + uint64_t(s) * 8;
  float old[6], nx[6], move = 0;
  for (int d = 0; d < 6; ++d) old[d] = mean[d];
  for (int d = 0; d < 6; ++d) {
    nx[d] = quotient(acc[d], acc[6]);
    const float e = old[d] - nx[d];
    move += e * e;
  }
  for (int d = 0; d < 6; ++d) mean[d] = nx[d];
  if (move < float(kSwitch2) * h2) state[s] = kNear;
}

}  // namespace

bool meanshift_bf16_bulk(Call &call, const VoteSet &v, float *means, uint8_t *state, uint64_t k,
                         double h2, int max_iter, int *iterations, double *evaluations,
                         uint32_t *trace, int trace_len, double *kernel_ms,
                         uint64_t *kernel_launches, double *seed_iterations) {
  *iterations = 0;
  *evaluations = 0;
  if (kernel_ms) *kernel_ms = 0;
  if (kernel_launches) *kernel_launches = 0;
  if (!k || !v.q) return false;
  const uint64_t max_tiles = (k + kChunk - 1) / kChunk;
  if (max_tiles * v.nchunks >= (uint64_t(1) << 31)) return false;  // list entries are int32
  cudaStream_t st = call.stream();
  call.allow_shared(ms_tile_tc, kTcSmem);
  uint8_t *images = call.alloc<uint8_t>(v.nchunks * kImage);
  build_images<<<unsigned(v.nchunks), kChunk, 0, st>>>(v.desc, v.q, v.nchunks, v.cbox, v.gbox,
                                                       float(1.0 / std::sqrt(h2)), images);
  check_launch();
  int32_t *ids = call.alloc<int32_t>(k);
  float *boxes = call.alloc<float>(max_tiles * kBoxFloats);
  const uint32_t nblk = uint32_t(v.nblocks);
  uint8_t *need = call.alloc<uint8_t>(max_tiles * v.nchunks);
  uint32_t *bcount = call.alloc<uint32_t>(max_tiles * nblk), *boff = call.alloc<uint32_t>(max_tiles * nblk);
  uint32_t *sblk = call.alloc<uint32_t>(max_tiles * nblk), *nsurv = call.alloc<uint32_t>(max_tiles);
  uint32_t *seg = call.alloc<uint32_t>(max_tiles + 1);
  const uint64_t list_cap = max_tiles * v.nchunks;
  int32_t *list = call.alloc<int32_t>(list_cap);
  // CTAs of the list kernels, shared among the active tiles at run time:
  // one full wave of the GPU at their occupancy
  static const int list_per_sm = [] {
    int a = 0, b = 0;
    SYM_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&a, tile_count, kListThreads, 0));
    SYM_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&b, scatter_lists, kListThreads, 0));
    return std::max(1, std::min(a, b));
  }();
  const unsigned list_ctas = unsigned(std::max<uint64_t>(max_tiles, uint64_t(152) * list_per_sm));
  uint64_t *offsets = call.alloc<uint64_t>(max_tiles + 1);
  uint32_t *pieces = call.alloc<uint32_t>(max_tiles + 1);
  // budget + tiles CTAs: tc_ctas_per_sm waves of the 152 SMs
  const uint32_t sms = 152 * uint32_t(v.tuning.tc_ctas_per_sm);
  const uint64_t max_grid = std::max<uint64_t>(sms, 2 * max_tiles);
  float *partial = call.alloc<float>(max_grid * kChunk * 8);
  Progress *progress = call.alloc<Progress>(1);
  const unsigned *const nact = progress->nact;  // on the device
  unsigned long long *evals = call.alloc<unsigned long long>(1);
  SYM_CUDA(cudaMemsetAsync(evals, 0, 8, st));
  SYM_CUDA(cudaMemsetAsync(progress, 0, sizeof(Progress), st));
  const float gap = float(std::sqrt(h2)) + 1e-6f;
  call.launched();
  TcArgs args{images, v.nchunks, list, offsets, pieces, nact, means, ids, v.gbox,
              float(1.0 / std::sqrt(h2)), float(v.kernel_k), partial, evals, progress, kernel_ms != nullptr,
              call.status()};
  // Iterations are launched back to back: each reads the active-seed count
  // that the previous one left on the device, and one whose count is zero
  // returns at once.  The host looks at the count every kCheck iterations.
  const int kCheck = v.tuning.check_interval;
  int it = 0;
  for (; it < max_iter; ++it) {
    active_seeds_async(call, v, means, state, k, ids, progress);
    launch_chained(st, tile_boxes<float>, unsigned(max_tiles), kCullThreads, 0, means, ids, nact, v.bbox, nblk,
                   gap * gap, boxes, sblk, nsurv, bcount);
    launch_chained(st, tile_count, list_ctas, kListThreads, 0, boxes, means, ids, nact, v.cbox, v.bbox,
                   v.nchunks, sblk, nsurv, nblk, gap * gap, need, bcount);
    launch_chained(st, scan_lists, 1, 1024, 0, bcount, nsurv, nact, nblk, sms, list_cap, seg, boff, offsets,
                   pieces, call.status());
    launch_chained(st, scatter_lists, list_ctas, kListThreads, 0, need, boff, bcount, sblk, nsurv, nblk, nact,
                   v.nchunks, list_cap, list, call.status());
    launch_chained(st, ms_tile_tc, unsigned(max_grid), kThreadsTc, kTcSmem, args);
    launch_chained(st, ms_update_bulk, unsigned((k + kUpdateSeeds - 1) / kUpdateSeeds), 32 * kUpdateSeeds, 0,
                   means, partial, pieces, ids, nact, float(h2), state);
    call.launched(6);
    if (it % kCheck == kCheck - 1) {
      unsigned n = 0;
      call.d2h(&n, nact, sizeof(unsigned));
      call.sync();
      if (!n) {
        ++it;
        break;
      }
    }
  }
  call.check_status("mean_shift (tensor)");
  unsigned long long ev = 0;
  Progress seen;
  call.d2h(&ev, evals, 8);
  call.d2h(&seen, progress, sizeof(seen));
  call.sync();
  *iterations = int(seen.iterations);
  *evaluations = double(ev);
  for (int i = 0; trace && i < std::min(trace_len, kTraced) && i < int(seen.iterations); ++i) trace[i] = seen.trace[i];
  if (seed_iterations) *seed_iterations += double(seen.seeds);
  if (kernel_ms) *kernel_ms = double(seen.busy + (seen.ended ? seen.ended - seen.began : 0)) * 1e-6;
  if (kernel_launches) *kernel_launches = kernel_ms ? seen.iterations : 0;
  return true;
}

void wait_selftest_host(Call &call, uint64_t limit_ns) {
  wait_selftest<<<1, 32, 0, call.stream()>>>(limit_ns, call.status());
  check_launch();
  call.launched();
  call.check_status("tensor-kernel wait self-test");
}

void tc_selftest_host(Call &call, const uint16_t *a1, const uint16_t *b1, const uint16_t *a2,
                      const uint16_t *b2, float *d_out, float *acc_out) {
  call.allow_shared(tc_selftest, kSmemRequest);
  auto up = [&](const uint16_t *p, size_t n) {
    return reinterpret_cast<const __nv_bfloat16 *>(call.upload(p, n));
  };
  const __nv_bfloat16 *da1 = up(a1, 128 * 16), *db1 = up(b1, 128 * 16), *da2 = up(a2, 128 * 128),
                      *db2 = up(b2, 16 * 128);
  uint8_t *scratch = call.alloc<uint8_t>(kB1Bytes + kSelfB2);
  float *dd = call.alloc<float>(128 * 128), *dacc = call.alloc<float>(128 * 16);
  tc_selftest<<<1, 256, kSmemRequest, call.stream()>>>(da1, db1, da2, db2, scratch, dd, dacc,
                                                       call.status());
  check_launch();
  call.launched();
  call.d2h(d_out, dd, 128 * 128 * 4);
  call.d2h(acc_out, dacc, 128 * 16 * 4);
  call.check_status("tensor self-test");
}

}  // namespace sym
