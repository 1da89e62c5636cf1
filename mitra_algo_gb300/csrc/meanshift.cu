// SPDX-License-Identifier: MPL-2.0
// Stage (c): mean-shift clustering in transformation space, reference
// semantics (Epanechnikov weights, 4-D reflection / 12-D rigid descriptors,
// random seeding until every vote is visited).
//
// Reference: src/cpu/clustering.cpp:32-208 (driver + evaluator),
// src/cuda/clustering.cu (the existing GPU path: one block per trajectory,
// launched thousands of times from the host driver).
//
// GB300 design.  A trajectory is a pure function of its seed vote (the
// reference evaluator only reads the seed descriptor and the vote set), so:
//   1. one launch runs the trajectory of EVERY vote as a seed, a warp per
//      seed, and records its final mean, its converged/exhausted flags and
//      its support (the same-kind votes that some iteration counted);
//   2. the host replays the reference's host loop verbatim (RNG draw per seed,
//      visited set, merge test, budgets) on those results - no device round
//      trip per trajectory;
//   3. the hits (iterations that counted a vote) of the trajectories the host
//      loop used are added up per cluster, and each vote takes the cluster with
//      the most (the first cluster on ties).
// Distances, weights and products are the reference's FP64 expressions (no
// FMA contraction), and the weighted sums add the members' contributions in
// vote order, as the reference's serial loop does: each lane evaluates one
// vote of a group of 32, then a lane per sum adds the members' values in
// order.  The means are therefore the reference's bit for bit, and so is every
// decision that depends on them (d^2 < h^2, the stop test, the merge test): no
// rounding band exists to be checked.
// Memory: every device array whose size grows with the square of the votes or
// with the supports fits kBatchBytes.  Where a row of hit counts for every seed
// of a kind does, step 1 writes those, and step 3 adds the used ones; above
// that (16,384 votes of a kind) step 1 writes rows of bits, batch by batch, and
// step 3 runs the used trajectories again.  The supports go to the host as lists,
// piece by piece, and the clusters' hit counts are made batch by batch.
#include "common.cuh"
#include "primitives.cuh"
#include "rng.hpp"

#include <algorithm>
#include <cmath>
#include <vector>

namespace sym {
namespace {

constexpr double kExhausted = 1e-14;  // clustering.cpp:15,169

// AoS descriptors of one kind: out[j*D + k] = lanes[k][ids[j]].
template <int D>
__global__ void gather_desc(const double *lanes, uint64_t q, const int32_t *ids, uint64_t n,
                            double *out) {
  uint64_t j = uint64_t(blockIdx.x) * blockDim.x + threadIdx.x;
  if (j >= n) return;
  int32_t v = ids[j];
  for (int k = 0; k < D; ++k) out[j * D + k] = lanes[uint64_t(k) * q + v];
}

// Lanes of the descriptors rounded to FP32: out[k * n + j] = desc[j * D + k].
template <int D>
__global__ void round_desc(const double *desc, uint64_t n, float *out) {
  const uint64_t j = uint64_t(blockIdx.x) * blockDim.x + threadIdx.x;
  if (j >= n) return;
  for (int k = 0; k < D; ++k) out[uint64_t(k) * n + j] = float(desc[j * D + k]);
}

// Trajectories, a warp each: the i-th from vote seeds[i] (or first + i), into
// row rows[i] (or i) of `out`, `pitch` words apart.  BITS: bit j of the row is
// set when some iteration had vote j within the bandwidth; else word j of the row
// gains the number of iterations that had.  final_mean and flags may be null.
//
// Culling: `lanes32` holds the descriptors rounded to FP32 and `reach` the
// bandwidth plus a bound on how far an FP32 distance can fall below the FP64
// one (the rounding of the mean and of every coordinate, D times 2^-22 of the
// largest coordinate magnitude, and of the FP32 arithmetic).  A vote whose
// FP32 squared distance exceeds reach^2 lies outside the bandwidth in FP64
// as well; only the others take the reference's FP64 test.
//
// A mean moves little, so the votes are not all tested in every iteration: the
// warp lists, in vote order, those within reach + `slack` of the mean in FP32, and
// a vote within the bandwidth of a later mean is among them as long as that mean
// is within `slack` of the listed one; then the list is made anew (a list longer
// than kListed is not kept: every vote is tested).  The listed votes that pass
// the FP32 test are gathered 32 at a time, so FP64 (1/64 of the FP32 rate) runs
// with full warps: each lane makes one vote's distance, weight and products,
// then lane d adds the d-th sum's members in vote order -- one addition per
// member and warp, where every lane adding every sum took D + 1.
// (8,900 votes of the mirrored 128 x 128 height field, 1,500 of them planes:
// trajectories and counts 15.7 ms, 1.0 ms now.)
constexpr int kListed = 1024, kTrajWarps = 4;
template <int D, bool BITS>
__global__ void __launch_bounds__(32 * kTrajWarps) trajectories(
    const double *desc, const float *lanes32, float reach, float slack, uint64_t n, const int32_t *seeds,
    uint64_t first, const int32_t *rows, uint64_t nseeds, double h2, int max_iter, double *final_mean,
    uint8_t *flags, uint32_t *out, uint64_t pitch) {
  __shared__ uint32_t list_s[kTrajWarps][kListed];
  __shared__ uint32_t near_s[kTrajWarps][64];
  __shared__ double term_s[kTrajWarps][32 * (D + 1)];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const uint64_t si = uint64_t(blockIdx.x) * kTrajWarps + warp;
  if (si >= nseeds) return;
  uint32_t *list = list_s[warp], *near = near_s[warp];
  double *term = term_s[warp];
  const uint64_t from = seeds ? uint64_t(seeds[si]) : first + si;
  uint32_t *row = out + (rows ? uint64_t(rows[si]) : si) * pitch;
  double mean[D];  // the same in every lane, as `converged` and `exhausted`
  float mean32[D], listed32[D];
  for (int k = 0; k < D; ++k) mean[k] = desc[from * D + k], listed32[k] = INFINITY;
  bool converged = false, exhausted = false;
  const double stop = 1e-6 * h2;
  const float reach2 = reach * reach, wide = (reach + slack) * (1 + 1e-5f), wide2 = wide * wide;
  const float slack2 = slack * slack * (1 - 1e-4f);
  uint64_t listed = 0;  // entries; n: every vote, no list
  for (int it = 0; it < max_iter; ++it) {
    float moved = 0;
    for (int k = 0; k < D; ++k) {
      mean32[k] = float(mean[k]);
      const float e = mean32[k] - listed32[k];
      moved += e * e;
    }
    if (!(moved < slack2)) {  // list the votes around the mean
      listed = 0;
      for (int k = 0; k < D; ++k) listed32[k] = mean32[k];
      __syncwarp();
      for (uint64_t base = 0; base < n; base += 32) {
        const uint64_t j = base + lane;
        float d32 = j < n ? 0.f : INFINITY;
        constexpr int kSome = D < 6 ? D : 3;  // the last ones (a rigid vote's translation) first
        if (j < n)
          for (int k = D - kSome; k < D; ++k) {
            const float e = mean32[k] - lanes32[uint64_t(k) * n + j];
            d32 += e * e;
          }
        if (!__any_sync(0xffffffffu, j < n && !(d32 > wide2))) continue;
        if (kSome < D && j < n && !(d32 > wide2))
          for (int k = 0; k < D - kSome; ++k) {
            const float e = mean32[k] - lanes32[uint64_t(k) * n + j];
            d32 += e * e;
          }
        const unsigned keep = __ballot_sync(0xffffffffu, !(d32 > wide2) && j < n);
        if (listed + __popc(keep) > kListed) {
          listed = n;
          break;
        }
        if (keep >> lane & 1u) list[listed + __popc(keep & ((1u << lane) - 1u))] = uint32_t(j);
        listed += __popc(keep);
      }
      if (listed == n && n > kListed) {
        for (int k = 0; k < D; ++k) listed32[k] = INFINITY;  // no list: try again next time
      }
      __syncwarp();
    }
    const bool all = listed == n && n > kListed;
    double sum = 0;  // lane 0: the weights; lane d: coordinate d - 1 of the weighted sum
    int pending = 0;
    auto take = [&](int count) {  // the first `count` gathered votes
      const bool mine = lane < count;
      const uint64_t j = mine ? near[lane] : 0;
      bool in = false;
      if (mine) {
        double x[D], dist = 0;
        for (int k = 0; k < D; ++k) {
          x[k] = desc[j * D + k];
          const double d = mean[k] - x[k];
          dist += d * d;
        }
        if (dist < h2) {
          in = true;
          const double w = 1 - dist / h2;
          term[lane * (D + 1)] = w;
          for (int k = 0; k < D; ++k) term[lane * (D + 1) + 1 + k] = w * x[k];
          if (!BITS) atomicAdd(&row[j], 1u);
        }
      }
      const unsigned bits = __ballot_sync(0xffffffffu, in);
      if (BITS && in) {  // the lanes of one word set it together
        const unsigned peers = __match_any_sync(bits, uint32_t(j >> 5));
        const uint32_t set = __reduce_or_sync(peers, 1u << (j & 31));
        if (lane == __ffs(int(peers)) - 1) atomicOr(&row[j >> 5], set);
      }
      __syncwarp();
      for (unsigned m = bits; m; m &= m - 1)  // in vote order
        if (lane <= D) sum += term[(__ffs(int(m)) - 1) * (D + 1) + lane];
      __syncwarp();
    };
    for (uint64_t base = 0; base < listed; base += 32) {
      uint64_t j = base + lane;
      float d32 = INFINITY;
      if (j < listed) {
        if (!all) j = list[j];
        d32 = 0;
        for (int k = 0; k < D; ++k) {
          const float e = mean32[k] - lanes32[uint64_t(k) * n + j];
          d32 += e * e;
        }
      }
      const bool close = base + lane < listed && !(d32 > reach2);
      const unsigned bits = __ballot_sync(0xffffffffu, close);
      if (close) near[pending + __popc(bits & ((1u << lane) - 1u))] = uint32_t(j);
      pending += __popc(bits);
      __syncwarp();
      if (pending >= 32) {
        take(32);
        const uint32_t rest = lane < pending - 32 ? near[32 + lane] : 0u;
        __syncwarp();
        near[lane] = rest;
        pending -= 32;
        __syncwarp();
      }
    }
    if (pending) take(pending);
    const double wt = __shfl_sync(0xffffffffu, sum, 0);
    if (wt <= kExhausted) {
      exhausted = true;
      break;
    }
    double next = lane && lane <= D ? sum / wt : 0.0, movement = 0;
    for (int k = 0; k < D; ++k) {
      const double to = __shfl_sync(0xffffffffu, next, k + 1);
      const double d = mean[k] - to;
      movement += d * d;
      mean[k] = to;
    }
    if (movement < stop) {
      converged = true;
      break;
    }
  }
  if (lane == 0 && final_mean) {
    for (int k = 0; k < D; ++k) final_mean[si * D + k] = mean[k];
    flags[si] = uint8_t((converged ? 1 : 0) | (exhausted ? 2 : 0));
  }
}

// Row s of the supports (bits, or hit counts) as a list: the votes in it,
// ascending; a warp per row.  size[s] (members null), or members[off[s] - off[0]
// ..].
template <bool BITS>
__global__ void list_support(const uint32_t *rows, uint64_t pitch, uint64_t n, uint64_t nseeds,
                             uint64_t *size, const uint64_t *off, uint32_t *members) {
  const uint64_t s = (uint64_t(blockIdx.x) * blockDim.x + threadIdx.x) >> 5;
  const int lane = threadIdx.x & 31;
  if (s >= nseeds) return;
  const uint32_t *row = rows + s * pitch;
  uint64_t at = members ? off[s] - off[0] : 0;
  if (BITS) {
    for (uint64_t base = 0; base < pitch; base += 32) {
      uint32_t word = base + lane < pitch ? row[base + lane] : 0u;
      const uint32_t mine = __popc(word);
      uint32_t incl = mine;
      for (int o = 1; o < 32; o <<= 1) {
        const uint32_t y = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= o) incl += y;
      }
      if (members)
        for (uint64_t to = at + incl - mine; word; word &= word - 1)
          members[to++] = uint32_t((base + lane) * 32) + __ffs(int(word)) - 1;
      at += __shfl_sync(0xffffffffu, incl, 31);
    }
  } else {
    for (uint64_t base = 0; base < n; base += 32) {
      const uint64_t j = base + lane;
      const bool in = j < n && row[j];
      const unsigned bits = __ballot_sync(0xffffffffu, in);
      if (members && in) members[at + __popc(bits & ((1u << lane) - 1u))] = uint32_t(j);
      at += __popc(bits);
    }
  }
  if (!members && lane == 0) size[s] = at;
}

// counts[cluster[i] * n ..] += the hit counts of seed seeds[i]; a block each.
__global__ void add_hits(const uint32_t *rows, uint64_t n, const int32_t *seeds, const int32_t *cluster,
                         uint32_t *counts) {
  const uint32_t *row = rows + uint64_t(seeds[blockIdx.x]) * n;
  uint32_t *sum = counts + uint64_t(cluster[blockIdx.x]) * n;
  for (uint64_t j = threadIdx.x; j < n; j += blockDim.x)
    if (const uint32_t hits = row[j]) atomicAdd(&sum[j], hits);
}

// Per vote the cluster with the most hits among kPick of a batch's, the earliest
// on ties: best[j] = the count, then the complement of the cluster's id, so a
// plain maximum decides over all of them.
constexpr int kPick = 64;
__global__ void pick_cluster(const uint32_t *counts, uint64_t nclusters, uint64_t n,
                             const int32_t *cluster_id, unsigned long long *best) {
  const uint64_t j = uint64_t(blockIdx.x) * blockDim.x + threadIdx.x;
  if (j >= n) return;
  const uint64_t c0 = uint64_t(blockIdx.y) * kPick, c1 = c0 + kPick < nclusters ? c0 + kPick : nclusters;
  unsigned long long most = 0;
  for (uint64_t c = c0; c < c1; ++c)
    if (const uint32_t hits = counts[c * n + j]) {
      const unsigned long long x = (unsigned long long)hits << 32 | (0xffffffffu - uint32_t(cluster_id[c]));
      most = x > most ? x : most;
    }
  if (most) atomicMax(&best[j], most);
}

// Device bytes of one batch of seeds' rows, of a piece of their lists, and of one
// batch of clusters' hit counts.  It also draws the line between the two forms of
// the rows, at 16,384 votes of a kind: counts, without a second run, take 7.6 ms
// for 8,900 votes of a height field where bits take 8.1, and 10.9 for 14,500 where
// bits take 11.7, but 6.5 and 6.8 for 16,384 votes of one kind where bits take 5.8:
// their rows are 32 times larger.
constexpr uint64_t kBatchBytes = uint64_t(1) << 30;

struct KindData {
  int dim = 0;
  uint64_t n = 0;
  std::vector<int32_t> ids;          // global vote id of each local index
  double *desc = nullptr;            // device AoS
  float *lanes32 = nullptr;          // the same rounded to FP32, lane-major
  float reach = 0;                   // the culling radius (trajectories)
  std::vector<double> mean;          // n x dim final means
  std::vector<uint8_t> flags;        // bit0 converged, bit1 exhausted
  std::vector<uint64_t> sup_off;     // n + 1: each seed's support (kind-local
  std::vector<uint32_t> sup;         //   member ids, ascending)
  uint32_t *hits = nullptr;          // device: every seed's hit counts (n x n), where they fit
};

float slack_of(double h2) { return float(0.5 * std::sqrt(h2)); }

template <int D>
void run_all_seeds(Call &call, KindData &k, double h2, int max_iter) {
  if (!k.n) return;
  cudaStream_t st = call.stream();
  const bool counted = k.n * k.n * 4 <= kBatchBytes;
  const uint64_t pitch = counted ? k.n : (k.n + 31) / 32;
  const uint64_t batch = std::max<uint64_t>(1, std::min<uint64_t>(k.n, kBatchBytes / (pitch * 4)));
  if (counted) k.hits = call.alloc<uint32_t>(k.n * k.n);
  const Arena::Mark kept = call.ctx->arena.mark();  // the rest is given back
  uint32_t *rows = counted ? k.hits : call.alloc<uint32_t>(batch * pitch);
  double *mean = call.alloc<double>(batch * D);
  uint8_t *flags = call.alloc<uint8_t>(batch);
  uint64_t *size = call.alloc<uint64_t>(batch), *off = call.alloc<uint64_t>(batch + 1);
  k.mean.resize(k.n * D);
  k.flags.resize(k.n);
  k.sup_off.assign(1, 0);
  k.sup.clear();
  const auto run = counted ? trajectories<D, false> : trajectories<D, true>;
  const auto list = counted ? list_support<false> : list_support<true>;
  std::vector<uint64_t> hoff(batch + 1);
  for (uint64_t first = 0; first < k.n; first += batch) {
    const Arena::Mark before = call.ctx->arena.mark();
    const uint64_t cnt = std::min(batch, k.n - first);
    SYM_CUDA(cudaMemsetAsync(rows, 0, cnt * pitch * 4, st));
    run<<<blocks_for(cnt, kTrajWarps), 32 * kTrajWarps, 0, st>>>(k.desc, k.lanes32, k.reach, slack_of(h2), k.n,
                                                                 nullptr, first, nullptr, cnt, h2, max_iter,
                                                                 mean, flags, rows, pitch);
    check_launch();
    list<<<blocks_for(cnt * 32), kThreads, 0, st>>>(rows, pitch, k.n, cnt, size, nullptr, nullptr);
    check_launch();
    exclusive_scan(call, size, off, cnt);
    call.d2h(hoff.data(), off, (cnt + 1) * 8);
    call.d2h(k.mean.data() + first * D, mean, cnt * D * 8);
    call.d2h(k.flags.data() + first, flags, cnt);
    call.sync();
    call.launched(2);
    const uint64_t at = k.sup.size(), room = std::min(hoff[cnt], std::max(kBatchBytes / 4, k.n));
    uint32_t *members = call.alloc<uint32_t>(room);
    k.sup.resize(at + hoff[cnt]);
    for (uint64_t s = 0; s < cnt; ++s) k.sup_off.push_back(at + hoff[s + 1]);
    for (uint64_t s0 = 0, s1; s0 < cnt; s0 = s1) {  // as many rows as fit the piece; one always does
      s1 = uint64_t(std::upper_bound(hoff.begin() + s0, hoff.begin() + cnt + 1, hoff[s0] + room) - hoff.begin()) - 1;
      if (hoff[s1] == hoff[s0]) continue;
      list<<<blocks_for((s1 - s0) * 32), kThreads, 0, st>>>(rows + s0 * pitch, pitch, k.n, s1 - s0, nullptr,
                                                            off + s0, members);
      check_launch();
      call.launched();
      call.d2h(k.sup.data() + at + hoff[s0], members, (hoff[s1] - hoff[s0]) * 4);
    }
    call.sync();
    call.ctx->arena.rewind(before);
  }
  call.ctx->arena.rewind(kept);
}

struct Center {
  double v[12];
  int kind;                    // index into kinds[]
  std::vector<uint64_t> keys;  // union of supports, kind-local bitmask (from the second seed on)
  uint64_t key_count = 0;
  std::vector<int32_t> seeds;  // kind-local seeds merged into this cluster
};

template <int D>
void count_members(Call &call, const KindData &k, const std::vector<Center> &centers, int kind_index,
                   double h2, int max_iter, std::vector<int32_t> &winner_global) {
  std::vector<int32_t> cluster_ids;
  for (size_t c = 0; c < centers.size(); ++c)
    if (centers[c].kind == kind_index) cluster_ids.push_back(int32_t(c));
  if (cluster_ids.empty()) return;
  cudaStream_t st = call.stream();
  const uint64_t batch = std::max<uint64_t>(1, std::min<uint64_t>(cluster_ids.size(),
                                                                   kBatchBytes / (k.n * 4)));
  const Arena::Mark before = call.ctx->arena.mark();
  uint32_t *counts = call.alloc<uint32_t>(batch * k.n);
  unsigned long long *best = call.alloc<unsigned long long>(k.n);
  int32_t *dids = call.upload(cluster_ids.data(), cluster_ids.size());
  SYM_CUDA(cudaMemsetAsync(best, 0, k.n * 8, st));
  std::vector<int32_t> seeds, cluster;  // kept until the copies are done
  for (uint64_t first = 0; first < cluster_ids.size(); first += batch) {
    const Arena::Mark per_batch = call.ctx->arena.mark();
    const uint64_t nc = std::min<uint64_t>(batch, cluster_ids.size() - first);
    if (first) call.sync();
    seeds.clear(), cluster.clear();
    for (uint64_t c = 0; c < nc; ++c)
      for (int32_t s : centers[cluster_ids[first + c]].seeds) seeds.push_back(s), cluster.push_back(int32_t(c));
    SYM_CUDA(cudaMemsetAsync(counts, 0, nc * k.n * 4, st));
    const int32_t *dseeds = call.upload(seeds.data(), seeds.size());
    const int32_t *dcluster = call.upload(cluster.data(), cluster.size());
    if (k.hits)
      add_hits<<<unsigned(seeds.size()), kThreads, 0, st>>>(k.hits, k.n, dseeds, dcluster, counts);
    else
      trajectories<D, false><<<blocks_for(seeds.size(), kTrajWarps), 32 * kTrajWarps, 0, st>>>(
          k.desc, k.lanes32, k.reach, slack_of(h2), k.n, dseeds, 0, dcluster, seeds.size(), h2, max_iter,
          nullptr, nullptr, counts, k.n);
    check_launch();
    pick_cluster<<<dim3(blocks_for(k.n), blocks_for(nc, kPick)), kThreads, 0, st>>>(counts, nc, k.n, dids + first,
                                                                                    best);
    check_launch();
    call.launched(2);
    call.ctx->arena.rewind(per_batch);
  }
  std::vector<unsigned long long> local(k.n);
  call.d2h(local.data(), best, k.n * 8);
  call.sync();
  call.ctx->arena.rewind(before);
  for (uint64_t j = 0; j < k.n; ++j)
    winner_global[k.ids[j]] = local[j] >> 32 ? int32_t(0xffffffffu - uint32_t(local[j])) : -1;
}

// Index of the centers for the merge test (clustering.cpp:68-73: the first
// center, in creation order, of the same kind within h/2).  A center within
// h/2 lies within h/2 in every coordinate, so on three coordinates it falls
// in one of the 27 cells of pitch slightly above h/2 around the mean; the
// lowest-numbered center among those that pass the reference's test is the
// reference's choice.  Centers with coordinates too large for the grid stay
// in a list that every query scans.
// The cells are hashed into chains of center numbers (an array each of chain
// heads, links and cells: 27 probes per query are 27 array reads).
class CenterGrid {
public:
  CenterGrid(double h, const int dims[3]) : scale_(2.0 / h * (1 - 1e-9)), head_(1024, -1) {
    for (int i = 0; i < 3; ++i) dims_[i] = dims[i];
  }
  void insert(int32_t id, const double *v) {
    uint64_t key;
    if (!cell(v, 0, 0, 0, key)) {
      loose_.push_back(id);
      return;
    }
    if (size_t(id) >= cells_.size()) cells_.resize(id + 1), links_.resize(id + 1, -1);
    if (++count_ > head_.size()) {  // twice the heads, the chains made anew
      std::vector<int32_t> ids;
      for (int32_t at : head_)
        for (; at >= 0; at = links_[at]) ids.push_back(at);
      head_.assign(2 * head_.size(), -1);
      for (int32_t at : ids) link(at);
    }
    cells_[id] = key;
    link(id);
  }
  void erase(int32_t id, const double *v) {
    uint64_t key;
    if (!cell(v, 0, 0, 0, key)) {
      loose_.erase(std::find(loose_.begin(), loose_.end(), id));
      return;
    }
    int32_t *at = &head_[slot(key)];
    while (*at != id) at = &links_[*at];
    *at = links_[id];
    --count_;
  }
  template <class Test>
  int32_t first(const double *v, Test &&passes) const {
    int32_t best = -1;
    for (int32_t id : loose_)
      if ((best < 0 || id < best) && passes(id)) best = id;
    uint64_t key;
    for (int a = -1; a <= 1; ++a)
      for (int b = -1; b <= 1; ++b)
        for (int c = -1; c <= 1; ++c)
          if (cell(v, a, b, c, key))
            for (int32_t id = head_[slot(key)]; id >= 0; id = links_[id])
              if (cells_[id] == key && (best < 0 || id < best) && passes(id)) best = id;
    return best;
  }

private:
  bool cell(const double *v, int a, int b, int c, uint64_t &key) const {
    const int off[3] = {a, b, c};
    key = 0;
    for (int i = 0; i < 3; ++i) {
      const double x = std::floor(v[dims_[i]] * scale_);
      if (!(std::fabs(x) < double(1 << 20))) return false;
      key = (key << 21) | uint64_t(int64_t(x) + off[i] + (1 << 20));
    }
    return true;
  }
  size_t slot(uint64_t key) const {  // splitmix64's finaliser
    key = (key ^ (key >> 30)) * 0xBF58476D1CE4E5B9ull;
    key = (key ^ (key >> 27)) * 0x94D049BB133111EBull;
    return size_t(key ^ (key >> 31)) & (head_.size() - 1);
  }
  void link(int32_t id) {
    int32_t &head = head_[slot(cells_[id])];
    links_[id] = head, head = id;
  }
  double scale_;
  int dims_[3];
  size_t count_ = 0;
  std::vector<int32_t> head_, links_, loose_;
  std::vector<uint64_t> cells_;
};

double desc_d2(const double *a, const double *b, int dim) {
  double s = 0;
  for (int i = 0; i < dim; ++i) {
    double d = a[i] - b[i];
    s += d * d;
  }
  return s;
}

}  // namespace

void clustering_host(Call &call, const sym_votes_view &votes, const sym_model_context &ctx,
                     const sym_options &o, sym_rng *rng, sym_clusters &out,
                     void *(*allocate)(size_t)) {
  const uint64_t q = votes.count;
  const double h = o.bandwidth, h2 = h * h;
  if (o.max_iterations < 1) fail(SYM_INVALID_ARGUMENT, "Invalid parameter range; see --help");
  KindData kinds[2];  // 0: reflection (4-D), 1: rigid (12-D)
  kinds[0].dim = 4, kinds[1].dim = 12;
  std::vector<uint8_t> kind_of(q);
  std::vector<int32_t> local_of(q);
  for (uint64_t i = 0; i < q; ++i) {
    int k = votes.kind[i] == SYM_REFLECTION ? 0 : 1;
    kind_of[i] = uint8_t(k);
    local_of[i] = int32_t(kinds[k].ids.size());
    kinds[k].ids.push_back(int32_t(i));
  }
  for (auto &k : kinds) k.n = k.ids.size();
  if (q) {
    double *lanes = call.alloc<double>(12 * q);
    for (int k = 0; k < 12; ++k) call.h2d(lanes + uint64_t(k) * q, votes.descriptor[k], q * 8);
    for (int t = 0; t < 2; ++t) {
      KindData &k = kinds[t];
      if (!k.n) continue;
      int32_t *ids = call.upload(k.ids.data(), k.n);
      k.desc = call.alloc<double>(k.n * k.dim);
      if (k.dim == 4)
        gather_desc<4><<<blocks_for(k.n), kThreads, 0, call.stream()>>>(lanes, q, ids, k.n, k.desc);
      else
        gather_desc<12><<<blocks_for(k.n), kThreads, 0, call.stream()>>>(lanes, q, ids, k.n, k.desc);
      check_launch();
      k.lanes32 = call.alloc<float>(k.n * k.dim);
      if (k.dim == 4)
        round_desc<4><<<blocks_for(k.n), kThreads, 0, call.stream()>>>(k.desc, k.n, k.lanes32);
      else
        round_desc<12><<<blocks_for(k.n), kThreads, 0, call.stream()>>>(k.desc, k.n, k.lanes32);
      check_launch();
      call.launched(2);
      // the culling radius: h plus the FP32 shortfall of a distance (rounding
      // of mean and coordinates, 2^-24 of the largest magnitude each, and of
      // the FP32 sums), each term taken 4 times over
      double mag = 0;
      for (uint64_t j = 0; j < k.n; ++j)
        for (int c = 0; c < k.dim; ++c) mag = std::max(mag, std::fabs(votes.descriptor[c][k.ids[j]]));
      const double reach = h + k.dim * std::ldexp(mag, -22) + (k.dim + 2) * std::ldexp(h, -22);
      k.reach = std::isfinite(mag) && mag < 1e15 ? float(reach * (1 + 1e-6)) : INFINITY;
    }
    run_all_seeds<4>(call, kinds[0], h2, o.max_iterations);
    run_all_seeds<12>(call, kinds[1], h2, o.max_iterations);
    call.sync();
  }

  // ---- the reference driver (clustering.cpp:44-96), replayed on the host
  auto engine = load_rng(rng);
  std::vector<uint64_t> visited((q + 63) / 64, 0);
  uint64_t unvisited = q, support_entries = 0;
  int limited = 0;
  std::vector<Center> centers;
  const int refl_dims[3] = {1, 2, 3}, rigid_dims[3] = {9, 10, 11};
  CenterGrid grids[2] = {CenterGrid(h, refl_dims), CenterGrid(h, rigid_dims)};
  auto visit = [&](uint64_t i) {
    uint64_t &w = visited[i >> 6];
    uint64_t bit = 1ull << (i & 63);
    if (!(w & bit)) w |= bit, --unvisited;
  };
  while (unvisited) {
    uint64_t r = engine() % unvisited;
    uint64_t seed = 0;
    for (uint64_t w = 0;; ++w) {  // r-th unvisited vote, ascending
      uint64_t free_bits = ~visited[w];
      if ((w + 1) * 64 > q) free_bits &= (q % 64 ? (1ull << (q % 64)) - 1 : ~0ull);
      uint64_t c = __builtin_popcountll(free_bits);
      if (r < c) {
        for (; r; --r) free_bits &= free_bits - 1;
        seed = w * 64 + __builtin_ctzll(free_bits);
        break;
      }
      r -= c;
    }
    int t = kind_of[seed];
    KindData &k = kinds[t];
    uint64_t s = uint64_t(local_of[seed]);
    const uint32_t *members = k.sup.data() + k.sup_off[s];
    const uint64_t size = k.sup_off[s + 1] - k.sup_off[s];
    for (uint64_t m = 0; m < size; ++m) visit(uint64_t(k.ids[members[m]]));
    bool converged = k.flags[s] & 1, exhausted = k.flags[s] & 2;
    if (exhausted) visit(seed);
    if (!converged) ++limited;
    const double *mean = &k.mean[s * k.dim];
    const int merge = grids[t].first(mean, [&](int32_t c) {
      return desc_d2(mean, centers[c].v, k.dim) < h2 / 4;
    });
    auto add_keys = [&](Center &c, uint64_t seed_of) {  // a support's members into the union
      uint64_t added = 0;
      for (uint64_t m = k.sup_off[seed_of]; m < k.sup_off[seed_of + 1]; ++m) {
        uint64_t &w = c.keys[k.sup[m] >> 6];
        const uint64_t bit = uint64_t(1) << (k.sup[m] & 63);
        if (!(w & bit)) w |= bit, ++added;
      }
      return added;
    };
    if (merge < 0) {
      Center c;
      for (int i = 0; i < 12; ++i) c.v[i] = i < k.dim ? mean[i] : 0;
      c.kind = t;
      c.key_count = size;
      c.seeds.push_back(int32_t(s));
      support_entries += c.key_count;
      grids[t].insert(int32_t(centers.size()), c.v);
      centers.push_back(std::move(c));
    } else {
      Center &c = centers[merge];
      double old = double(c.key_count), now = double(size);
      if (old + now > 0) {
        grids[t].erase(merge, c.v);
        for (int i = 0; i < k.dim; ++i) c.v[i] = (old * c.v[i] + now * mean[i]) / (old + now);
        grids[t].insert(merge, c.v);
      }
      if (c.keys.empty()) {
        c.keys.assign((k.n + 63) / 64, 0);
        add_keys(c, uint64_t(c.seeds[0]));
      }
      const uint64_t added = add_keys(c, s);
      c.key_count += added;
      support_entries += added;
      c.seeds.push_back(int32_t(s));
    }
    if (support_entries > 5000000)
      fail(SYM_RUNTIME_ERROR, "Mean-shift support budget exceeded; lower --sample-ratio");
    if (centers.size() > 20000)
      fail(SYM_RUNTIME_ERROR, "Too many mean-shift modes; increase --bandwidth or lower --sample-ratio");
  }
  store_rng(engine, rng);

  // ---- support counts and winners (clustering.cpp:97-108) on the GPU
  std::vector<int32_t> winner(q, -1);
  count_members<4>(call, kinds[0], centers, 0, h2, o.max_iterations, winner);
  count_members<12>(call, kinds[1], centers, 1, h2, o.max_iterations, winner);
  std::vector<std::vector<int32_t>> members(centers.size());
  for (uint64_t i = 0; i < q; ++i)
    if (winner[i] >= 0) members[winner[i]].push_back(int32_t(i));

  // ---- decode (clustering.cpp:109-141), stable sort, truncate
  struct Row {
    sym_cluster_record rec;
    std::vector<int32_t> votes;
  };
  std::vector<Row> rows;
  D3 origin{ctx.center[0], ctx.center[1], ctx.center[2]};
  for (size_t c = 0; c < centers.size(); ++c) {
    if (members[c].empty()) continue;
    Row row{};
    row.rec.reflection = centers[c].kind == 0;
    row.votes = std::move(members[c]);
    const double *d = centers[c].v;
    if (row.rec.reflection) {
      D3 n{d[0], d[1], d[2]};
      double length = norm(n);
      D3 pn = unit(n);
      double offset = d[3] * ctx.box_size / length - dot(pn, origin);
      M3 r = mirror(pn);
      D3 t = pn * (-2 * offset);
      for (int i = 0; i < 9; ++i) row.rec.rotation[i] = r.m[i];
      row.rec.translation[0] = t.x, row.rec.translation[1] = t.y, row.rec.translation[2] = t.z;
      row.rec.plane_normal[0] = pn.x, row.rec.plane_normal[1] = pn.y, row.rec.plane_normal[2] = pn.z;
      row.rec.plane_offset = offset;
    } else {
      M3 m;
      for (int i = 0; i < 9; ++i) m.m[i] = d[i] * 2;
      D3 c0{m.m[0], m.m[3], m.m[6]}, c1{m.m[1], m.m[4], m.m[7]};
      D3 a = unit(c0), b = unit(c1 - a * dot(a, c1));
      if (norm(a) < 0.5 || norm(b) < 0.5) {
        int32_t first = row.votes[0];
        for (int i = 0; i < 9; ++i) m.m[i] = votes.rotation[i][first];
      } else {
        m = columns(a, b, cross(a, b));
      }
      D3 t{d[9], d[10], d[11]};
      D3 tr = t * ctx.box_size + origin - mul(m, origin);
      for (int i = 0; i < 9; ++i) row.rec.rotation[i] = m.m[i];
      row.rec.translation[0] = tr.x, row.rec.translation[1] = tr.y, row.rec.translation[2] = tr.z;
    }
    rows.push_back(std::move(row));
  }
  std::stable_sort(rows.begin(), rows.end(),
                   [](const Row &a, const Row &b) { return a.votes.size() > b.votes.size(); });
  if (rows.size() > size_t(o.max_clusters)) rows.resize(o.max_clusters);
  uint64_t total = 0;
  for (auto &r : rows) total += r.votes.size();
  size_t nrec = rows.size();
  size_t bytes = nrec * sizeof(sym_cluster_record) + (nrec + 1) * 8 + total * 4 + 64;
  char *block = static_cast<char *>(allocate(bytes));
  if (!block) fail(SYM_RUNTIME_ERROR, "host allocation failed");
  out.storage = block;
  out.records = reinterpret_cast<sym_cluster_record *>(block);
  out.vote_offsets = reinterpret_cast<uint64_t *>(block + nrec * sizeof(sym_cluster_record));
  out.vote_indices = reinterpret_cast<int32_t *>(out.vote_offsets + nrec + 1);
  out.count = nrec;
  out.limited_iterations = limited;
  out.vote_offsets[0] = 0;
  for (size_t c = 0; c < nrec; ++c) {
    out.records[c] = rows[c].rec;
    std::copy(rows[c].votes.begin(), rows[c].votes.end(), out.vote_indices + out.vote_offsets[c]);
    out.vote_offsets[c + 1] = out.vote_offsets[c] + rows[c].votes.size();
  }
}

}  // namespace sym
