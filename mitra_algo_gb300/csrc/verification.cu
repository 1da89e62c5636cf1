// SPDX-License-Identifier: MPL-2.0
// Stage (d): verification of every cluster by closest-point tests and
// region growing.
//
// Reference: src/cpu/verification.cpp:22-110, src/cpu/surface.h:12-96,
// src/core/math.cpp:72-112 (CPU); src/cuda/verification.cu (existing GPU
// path: one launch per cluster and a host-driven label propagation loop).
//
// GB300 design:
//  * the median-split BVH is built exactly as the reference builds it
//    (std::nth_element on face centroids, leaves of <= 8 faces), so the
//    near-first, strict-< traversal returns the same face on distance ties
//    and the normal test agrees; the traversal itself runs on the GPU;
//  * ONE launch covers every cluster, both directions and every vertex;
//  * rms / coverage are the reference's serial sums bit for bit, computed in
//    parallel (serial_sum);
//  * patches are connected components grown on the GPU with lock-free
//    union-find that always links the larger root under the smaller one, so
//    a component's root is its smallest vertex; a stable sort by (cluster,
//    side, root) then yields the reference's breadth-first patch order
//    (patches by smallest vertex, members ascending), which the device writes
//    in the result's layout (20 clusters of an 80,000-vertex torus, 1.6e6
//    members: building the lists on the host took some 35 ms of the call's 58).
#include "common.cuh"
#include "face32.cuh"
#include "primitives.cuh"
#include "verification.cuh"

#include <algorithm>
#include <cmath>
#include <cstdlib>
#include <functional>
#include <limits>
#include <numeric>
#include <system_error>
#include <utility>
#include <vector>

namespace sym {

// The reference's build (surface.h:16-50) gives its nodes in preorder and
// halves every range by count, so the number of nodes, of leaves and the depth of
// a subtree follow from its number of faces alone: each subtree knows where its
// nodes and leaves go, and the subtrees build at the same time on host threads.
// std::nth_element sees the same comparisons as the reference's (of the same
// centroids, made once per face and laid out next to the ids it permutes), so it
// leaves the same permutation.  (One thread that formed centroids and boxes
// from the vertices at every comparison kept the first detection on a
// 1e6-triangle torus waiting: 454 ms, 110 ms now.)
namespace {

struct SubtreeSize {
  int64_t nodes, leaves;
  int depth;
};
SubtreeSize joined(const SubtreeSize &l, const SubtreeSize &r) {
  return {1 + l.nodes + r.nodes, l.leaves + r.leaves, 1 + std::max(l.depth, r.depth)};
}
// of n faces and of n + 1: the halves of both are n / 2 and n / 2 + 1 faces
std::pair<SubtreeSize, SubtreeSize> subtree_sizes(int64_t n) {
  const SubtreeSize one{1, 1, 0};
  if (n + 1 <= 8) return {one, one};
  const auto h = subtree_sizes(n / 2);
  const SubtreeSize odd = joined(h.first, h.second);
  if (n & 1) return {odd, joined(h.second, h.second)};
  return {n <= 8 ? one : joined(h.first, h.first), odd};
}
SubtreeSize subtree_size(int64_t n) { return subtree_sizes(n).first; }

// f on a thread of its own, or here when there is none to be had
template <class F>
std::future<void> launch(F f) {
  try {
    return std::async(std::launch::async, f);
  } catch (const std::system_error &) {
    f();
    return {};
  }
}

struct FaceBox {
  double lo[3], hi[3];
};

struct BvhBuilder {
  HostBvh &t;
  std::vector<FaceBox> box;
  std::vector<double> centroid[3];
  struct Keyed {
    double at;
    int32_t face;
  };
  std::vector<Keyed> keyed;  // each subtree works in its own range

  // the subtrees that get a thread: at most 2^kSpawnLevels, of at least kSpawn faces
  static constexpr int64_t kSpawn = 2048;
  static constexpr int kSpawnLevels = 5;

  void run(int64_t n, int64_t grain, const std::function<void(int64_t, int64_t)> &part) {
    std::vector<std::future<void>> jobs;
    for (int64_t at = grain; at < n; at += grain) {
      const int64_t end = std::min(n, at + grain);
      jobs.push_back(launch([&part, at, end] { part(at, end); }));
    }
    part(0, std::min(n, grain));
    for (auto &j : jobs)
      if (j.valid()) j.get();
  }

  FaceBox bounds(int64_t begin, int64_t end) const {
    FaceBox b{{1e300, 1e300, 1e300}, {-1e300, -1e300, -1e300}};
    for (int64_t i = begin; i < end; ++i) {
      const FaceBox &f = box[t.ids[i]];
      for (int k = 0; k < 3; ++k) b.lo[k] = std::min(b.lo[k], f.lo[k]), b.hi[k] = std::max(b.hi[k], f.hi[k]);
    }
    return b;
  }

  // chain[0 .. level): the ancestors; path: their steps
  void build(int64_t begin, int64_t end, int level, int64_t index, int64_t leaf, uint32_t path,
             int32_t *chain) {
    const FaceBox b = bounds(begin, end);
    BvhNode n;
    for (int k = 0; k < 3; ++k) n.lo[k] = b.lo[k], n.hi[k] = b.hi[k];
    n.begin = int32_t(begin), n.end = int32_t(end), n.left = -1, n.right = -1;
    chain[level] = int32_t(index);
    if (end - begin <= 8) {
      t.nodes[index] = n;
      for (int64_t i = begin; i < end; ++i) t.order[t.ids[i]] = FaceOrder{path, int32_t(leaf), int32_t(i), 0};
      std::copy(chain, chain + level + 1, t.ancestors.begin() + leaf * 32);
      return;
    }
    const double ext[3] = {n.hi[0] - n.lo[0], n.hi[1] - n.lo[1], n.hi[2] - n.lo[2]};
    int axis = ext[1] > ext[0] ? 1 : 0;
    if (ext[2] > ext[axis]) axis = 2;
    const int64_t mid = (begin + end) / 2;
    for (int64_t i = begin; i < end; ++i) keyed[i] = {centroid[axis][t.ids[i]], t.ids[i]};
    std::nth_element(keyed.begin() + begin, keyed.begin() + mid, keyed.begin() + end,
                     [](const Keyed &x, const Keyed &y) { return x.at < y.at; });
    for (int64_t i = begin; i < end; ++i) t.ids[i] = keyed[i].face;
    const SubtreeSize l = subtree_size(mid - begin);
    n.left = int32_t(index + 1), n.right = int32_t(index + 1 + l.nodes);
    t.nodes[index] = n;
    const uint32_t right_path = path | (1u << (31 - level));
    auto right = [&, right_path](int32_t *c) {
      build(mid, end, level + 1, n.right, leaf + l.leaves, right_path, c);
    };
    if (level < kSpawnLevels && end - begin >= 2 * kSpawn) {
      int32_t other[32];
      std::copy(chain, chain + level + 1, other);
      auto job = launch([&] { right(other); });
      build(begin, mid, level + 1, n.left, leaf, path, chain);
      if (job.valid()) job.get();
    } else {
      build(begin, mid, level + 1, n.left, leaf, path, chain);
      right(chain);
    }
  }
};

}  // namespace

HostBvh::HostBvh(const sym_mesh_view &m) {
  const int64_t nf = int64_t(m.faces.count);
  ids.resize(nf);
  for (int64_t i = 0; i < nf; ++i) ids[i] = int32_t(i);
  if (!nf) return;
  const SubtreeSize size = subtree_size(nf);
  depth = size.depth;
  if (depth > 31) throw Error(SYM_RUNTIME_ERROR, "verification: BVH too deep");
  nodes.resize(size.nodes);
  order.resize(nf);
  ancestors.assign(size_t(size.leaves) * 32, -1);
  BvhBuilder build{*this, std::vector<FaceBox>(nf), {}, std::vector<BvhBuilder::Keyed>(nf)};
  for (auto &c : build.centroid) c.resize(nf);
  const int32_t *cols[3] = {m.faces.v0, m.faces.v1, m.faces.v2};
  const double *axes[3] = {m.vertices.x, m.vertices.y, m.vertices.z};
  build.run(nf, 1 << 16, [&](int64_t begin, int64_t end) {
    for (int64_t f = begin; f < end; ++f)
      for (int k = 0; k < 3; ++k) {
        const double a = axes[k][cols[0][f]], b = axes[k][cols[1][f]], c = axes[k][cols[2][f]];
        build.box[f].lo[k] = std::min(std::min(std::min(1e300, a), b), c);
        build.box[f].hi[k] = std::max(std::max(std::max(-1e300, a), b), c);
        build.centroid[k][f] = (a + b + c) / 3;
      }
  });
  int32_t chain[32];
  build.build(0, nf, 0, 0, 0, 0, chain);
}

// boxes32 of RefBvh: the boxes of a node's children in FP32 (an inner node's).
__global__ void ref_boxes32(const BvhNode *nodes, uint64_t n, float4 *out) {
  const uint64_t i = uint64_t(blockIdx.x) * blockDim.x + threadIdx.x;
  if (i >= n || nodes[i].left < 0) return;
  const BvhNode &l = nodes[nodes[i].left], &r = nodes[nodes[i].right];
  out[3 * i] = make_float4(float(l.lo[0]), float(l.lo[1]), float(l.lo[2]), float(l.hi[0]));
  out[3 * i + 1] = make_float4(float(l.hi[1]), float(l.hi[2]), float(r.lo[0]), float(r.lo[1]));
  out[3 * i + 2] = make_float4(float(r.lo[2]), float(r.hi[0]), float(r.hi[1]), float(r.hi[2]));
}

RefBvh ref_bvh_upload(const HostBvh &bvh, cudaStream_t stream) {
  RefBvh b;
  b.depth = bvh.depth;
  auto pad = [](size_t x) { return (x + 255) & ~size_t(255); };
  const size_t nn = bvh.nodes.size(), nf = bvh.ids.size(), na = bvh.ancestors.size();
  const size_t s_nodes = pad(nn * sizeof(BvhNode)), s_ids = pad(nf * 4),
               s_order = pad(nf * sizeof(FaceOrder)), s_anc = pad(na * 4);
  SYM_CUDA(cudaMalloc(&b.block, s_nodes + s_ids + s_order + s_anc + nn * 48 + 256));
  char *at = b.block;
  auto put = [&](const void *src, size_t bytes, size_t room) {
    if (bytes) SYM_CUDA(cudaMemcpyAsync(at, src, bytes, cudaMemcpyHostToDevice, stream));
    char *here = at;
    at += room;
    return here;
  };
  b.nodes = reinterpret_cast<const BvhNode *>(put(bvh.nodes.data(), nn * sizeof(BvhNode), s_nodes));
  b.ids = reinterpret_cast<const int32_t *>(put(bvh.ids.data(), nf * 4, s_ids));
  b.order = reinterpret_cast<const FaceOrder *>(put(bvh.order.data(), nf * sizeof(FaceOrder), s_order));
  b.ancestors = reinterpret_cast<const int32_t *>(put(bvh.ancestors.data(), na * 4, s_anc));
  b.boxes32 = reinterpret_cast<const float4 *>(at);
  if (nn) {
    ref_boxes32<<<blocks_for(nn), kThreads, 0, stream>>>(b.nodes, nn, reinterpret_cast<float4 *>(at));
    check_launch();
  }
  SYM_CUDA(cudaStreamSynchronize(stream));
  return b;
}

void ref_bvh_free(RefBvh &b) {
  if (b.block) cudaFree(b.block);
  b = RefBvh{};
}

void RefBvhSource::start(std::vector<double> xyz, std::vector<int32_t> faces, uint64_t nv,
                         uint64_t nf) {
  pending = std::async(std::launch::async, [x = std::move(xyz), f = std::move(faces), nv, nf]() {
    const sym_mesh_view mv{{x.data(), x.data() + nv, x.data() + 2 * nv, nv},
                           {f.data(), f.data() + nf, f.data() + 2 * nf, nf}};
    return std::make_unique<HostBvh>(mv);
  });
}

void RefBvhSource::release() {
  if (pending.valid()) pending.wait();
  ref_bvh_free(dev);
}

namespace {

// The reference-order search (nearest_face) with its FP64 tests made in FP32
// where that decides them: `face` are the faces' FP32 records, boxes32 the
// nodes' children's boxes (RefBvh), um = u M.  The outcome of every decision is
// FP64's: a box is skipped, or a face left out, in FP32 only when its distance is
// above the best by more than the errors of both; children are ordered in FP32
// only when their distances differ by more; the rest goes to FP64, which runs at
// 1/64 of the rate.  (16 boxes and some 30 faces per query were FP64: 8.7 ms for 8
// clusters of the 128 x 128 height field, 1.8 ms now; 2.0 when each face within
// reach went to FP64 in turn, without a look at the rest of its leaf.)
constexpr int kLeafFaces = 8;
__device__ double nearest_face_f(const Surface &s, const float4 *face32, const float4 *boxes32,
                                 float um, D3 p, double limit, int32_t &face, int *status) {
  double best = limit;
  face = -1;
  const F3 pf{float(p.x), float(p.y), float(p.z)};
  const float margin = 32.f * um;
  float reach, reach2;  // of a face's FP32 distance that can still be below the best
  auto bound = [&]() {
    reach = best > 1e-30 && best < 1e30 ? sqrtf(float(best)) * (1.f + 2e-6f) + 64.f * um : INFINITY;
    reach2 = reach * reach;
  };
  bound();
  struct __align__(8) Entry {
    int32_t node;
    float d;  // box_distance_f; -1: for FP64 to decide
  };
  Entry stack[kRefStack];
  int top = 0;
  stack[top++] = {0, -1.f};
  while (top) {
    const Entry at = stack[--top];
    if (at.d > reach) continue;
    const BvhNode &n = s.nodes[at.node];
    // within `reach` by the errors' width, or undecided
    if ((at.d < 0.f || !(at.d <= reach - 128.f * um - 4e-6f * reach)) && box_d2(p, n) > best) continue;
    const int32_t left = n.left;
    if (left < 0) {
      // FP32 distances (or lower bounds) of up to kLeafFaces of the leaf's faces at
      // a time; those that another of them beats by more than the errors are out
      // as well: in order they could be the best only until that one's turn
      const int32_t end = n.end;
      for (int32_t i0 = n.begin; i0 < end; i0 += kLeafFaces) {
        float d2[kLeafFaces], least = INFINITY;
#pragma unroll
        for (int k = 0; k < kLeafFaces; ++k) {
          d2[k] = INFINITY;
          if (i0 + k >= end) continue;
          const Face r = load_face(face32, s.ids[i0 + k]);
          d2[k] = 0.f;
          if (r.reach != 0.f && face_d2n(pf, r, um, reach2, d2[k])) least = fminf(least, d2[k]);
        }
        float within2 = reach2;
        if (least > 1e-30f && least < 1e30f) {
          const float within = sqrtf(least) * (1.f + 2e-6f) + 128.f * um;
          within2 = fminf(reach2, within * within);
        }
#pragma unroll
        for (int k = 0; k < kLeafFaces; ++k) {
          if (i0 + k >= end || d2[k] > within2 || d2[k] > reach2) continue;
          const int32_t f = s.ids[i0 + k];
          const double d = triangle_d2(p, corner(s, f, 0), corner(s, f, 1), corner(s, f, 2));
          if (d < best) best = d, face = f, bound();
        }
      }
    } else {
      const int32_t right = n.right;
      const float4 *r = boxes32 + 3 * int64_t(at.node);
      const float4 x = r[0], y = r[1], z = r[2];
      const float lb[6] = {x.x, x.y, x.z, x.w, y.x, y.y}, rb[6] = {y.z, y.w, z.x, z.y, z.z, z.w};
      const float dl = box_distance_f(pf.x, pf.y, pf.z, lb, margin),
                  dr = box_distance_f(pf.x, pf.y, pf.z, rb, margin);
      if (top + 2 > kRefStack) {
        atomicExch(status, DS_CAPACITY);
        return best;
      }
      const bool swap = right_nearer(dl, dr, margin, [&] {
        return box_d2(p, s.nodes[left]) > box_d2(p, s.nodes[right]);
      });
      stack[top++] = swap ? Entry{left, dl} : Entry{right, dr};
      stack[top++] = swap ? Entry{right, dr} : Entry{left, dl};
    }
  }
  return best;
}

// flags[(c * 2 + dir) * nv + i], err[c * nv + i] (forward direction).
// Query (c, direction, j) takes vertex i = order[j], the vertices in Morton
// order of their position, so a warp walks neighbouring vertices through
// nearly the same BVH nodes; flags and errors stay per vertex (row).
__global__ void __launch_bounds__(kThreads, 3)
    verify_vertices(Surface s, const float4 *face32, const float4 *boxes32, float scale,
                                const double *vn, const int32_t *order,
                                const ClusterMotion *clusters, uint64_t nc, double tau,
                                double limit, uint8_t *flags, double *err, int *status) {
  const uint64_t qid = uint64_t(blockIdx.x) * blockDim.x + threadIdx.x;
  const uint64_t nv = s.nv;
  if (qid >= nc * 2 * nv) return;
  const uint64_t c = qid / (2 * nv), rem = qid % (2 * nv);
  const bool inverse = rem >= nv;
  const uint64_t i = uint64_t(order[rem % nv]), row = qid - rem % nv + i;
  flags[row] = 0;
  if (!inverse) err[c * nv + i] = 0;
  double d = 0;
  const bool ok = exact_query_by(s, vn, clusters[c], inverse, i, tau, d, [&](D3 q, int32_t &face) {
    const float mag = fmaxf(fabsf(float(q.x)), fmaxf(fabsf(float(q.y)), fabsf(float(q.z))));
    const bool finite = isfinite(q.x) && isfinite(q.y) && isfinite(q.z);
    const float um = finite ? kUnit * fmaxf(scale, mag) : INFINITY;
    return nearest_face_f(s, face32, boxes32, um, q, limit, face, status);
  });
  if (!ok) return;
  flags[row] = 1;
  if (!inverse) err[c * nv + i] = d;
}

// The serial sum s = ((x0 + x1) + x2) + ... in parallel, bit for bit.  While
// the running sum stays in one binade [2^E, 2^(E+1)) it is an integer S times
// u = 2^(E - 52), and adding x >= 0 turns S into S + k + c: k = floor(x / u), and
// c = 1 when the rest of x / u exceeds a half, 0 when it is less, and for a
// tie the parity of S + k (round half to even).  So an addend is a map that
// depends only on the parity of S, two increments (even, odd), and such maps
// compose associatively: a block-wide scan gives every prefix of a tile of
// addends.  The first addend whose exact sum leaves the binade (S + k >= 2^53) is
// added as it is, and the rest of the tile starts over from there: one more
// round per binade the sum passes.  Addends that are negative or not finite, and
// sums without a binade (infinite, not a number, next to zero), are added one by
// one, kSerial at a time.
struct Increment {
  long long even, odd;  // what S gains, by its parity; at most kBeyond
};
constexpr long long kBeyond = 1ll << 54;  // past the end of any binade
__device__ __forceinline__ Increment then(Increment a, Increment b) {
  const long long even = a.even + (a.even & 1 ? b.odd : b.even);
  const long long odd = a.odd + (a.odd & 1 ? b.even : b.odd);
  return {even < kBeyond ? even : kBeyond, odd < kBeyond ? odd : kBeyond};
}

// floor(x / u) and the increment of x >= 0 in the binade of exponent E
// (biased, normal).
__device__ __forceinline__ Increment increment(double x, int E, long long &k) {
  const unsigned long long bits = (unsigned long long)__double_as_longlong(x) & ~(1ull << 63);
  const int e = int(bits >> 52);
  const unsigned long long m = (bits & ((1ull << 52) - 1)) | (e ? 1ull << 52 : 0ull);
  const int d = E - (e ? e : 1);  // x / u = m 2^-d
  if (d <= 0) {
    k = d > -2 ? (long long)(m << -d) : kBeyond;
    return {k, k};
  }
  if (d > 53) {
    k = 0;
    return {0, 0};
  }
  k = (long long)(m >> d);
  const unsigned long long rest = m & ((1ull << d) - 1), half = 1ull << (d - 1);
  if (rest == half) return {k + (k & 1), k + ((k + 1) & 1)};
  const long long up = rest > half;
  return {k + up, k + up};
}

constexpr int kSumThreads = 1024, kSumItems = 4, kSumTile = kSumThreads * kSumItems, kSerial = 256;

// The serial sum of value(0), ..., value(n - 1) by a block of kSumThreads.
template <class Value>
__device__ double serial_sum(uint64_t n, Value &&value) {
  __shared__ Increment warp_sum[kSumThreads / 32];
  __shared__ double s_shared;
  __shared__ unsigned event_s;
  __shared__ int rough_s;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  double s = 0;
  int rough = 0;  // the last addend was irregular: go on one by one
  for (uint64_t pos = 0; pos < n;) {
    const unsigned long long sb = (unsigned long long)__double_as_longlong(s);
    const int E = int(sb >> 52);  // sign included: negative sums are not regular
    const bool zero = sb == 0, regular = E > 64 && E < 0x7ff;
    if (rough || !(zero || regular)) {
      if (threadIdx.x == 0) {
        const uint64_t end = pos + kSerial < n ? pos + kSerial : n;
        for (uint64_t j = pos; j < end; ++j) s += value(j);
        s_shared = s;
      }
      __syncthreads();
      s = s_shared;
      pos += kSerial, rough = 0;
      __syncthreads();
      continue;
    }
    // this thread's addends
    const uint64_t first = pos + uint64_t(threadIdx.x) * kSumItems;
    double x[kSumItems];
    long long k[kSumItems];
    Increment each[kSumItems], mine{0, 0};
#pragma unroll
    for (int j = 0; j < kSumItems; ++j) {
      x[j] = first + j < n ? value(first + j) : 0.0;
      const bool odd_one = !(x[j] >= 0.0 && x[j] < INFINITY);
      if (zero) k[j] = x[j] != 0.0 || odd_one ? kBeyond : 0, each[j] = {0, 0};
      else if (odd_one) k[j] = kBeyond, each[j] = {0, 0};
      else each[j] = increment(x[j], E, k[j]);
      mine = then(mine, each[j]);
    }
    // exclusive scan over the block
    Increment incl = mine;
    for (int o = 1; o < 32; o <<= 1) {
      const Increment before{__shfl_up_sync(0xffffffffu, incl.even, o),
                             __shfl_up_sync(0xffffffffu, incl.odd, o)};
      if (lane >= o) incl = then(before, incl);
    }
    if (lane == 31) warp_sum[warp] = incl;
    if (threadIdx.x == 0) event_s = kSumTile;
    __syncthreads();
    if (warp == 0) {
      Increment w = warp_sum[lane];
      for (int o = 1; o < 32; o <<= 1) {
        const Increment before{__shfl_up_sync(0xffffffffu, w.even, o),
                               __shfl_up_sync(0xffffffffu, w.odd, o)};
        if (lane >= o) w = then(before, w);
      }
      warp_sum[lane] = w;  // inclusive over warps
    }
    __syncthreads();
    Increment lane_before{__shfl_up_sync(0xffffffffu, incl.even, 1),
                          __shfl_up_sync(0xffffffffu, incl.odd, 1)};
    if (lane == 0) lane_before = {0, 0};
    const Increment before = warp ? then(warp_sum[warp - 1], lane_before) : lane_before;
    const unsigned long long S0 = zero ? 0 : (sb & ((1ull << 52) - 1)) | (1ull << 52);
    // the first addend that leaves the binade
    unsigned long long S = S0 + (unsigned long long)(S0 & 1 ? before.odd : before.even);
    unsigned long long at_event = 0;
    double x_event = 0;
    unsigned event = kSumTile;
#pragma unroll
    for (int j = 0; j < kSumItems; ++j)
      if (event == kSumTile) {
        if (S + (unsigned long long)k[j] >= (1ull << 53))
          event = threadIdx.x * kSumItems + j, at_event = S, x_event = x[j];
        S += (unsigned long long)(S & 1 ? each[j].odd : each[j].even);
      }
    if (event < kSumTile) atomicMin(&event_s, event);
    __syncthreads();
    const double u = __longlong_as_double((long long)(E - 52) << 52);
    if (event_s == kSumTile) {
      if (threadIdx.x == kSumThreads - 1) s_shared = zero ? 0.0 : double(S) * u, rough_s = 0;
    } else if (event == event_s) {
      s_shared = (zero ? 0.0 : double(at_event) * u) + x_event;
      rough_s = !(x_event >= 0.0 && x_event < INFINITY);
    }
    __syncthreads();
    s = s_shared, rough = rough_s;
    pos += event_s == kSumTile ? uint64_t(kSumTile) : uint64_t(event_s) + 1;
    __syncthreads();
  }
  return s;
}

// Block b < nc: the forward errors of cluster b (and their count); block nc + c:
// the supporting weight of cluster c, forward vertices, then inverse ones;
// block 2 nc: the total weight.  A vertex that does not support the cluster
// adds zero, which leaves a sum as it is.
__global__ void __launch_bounds__(kSumThreads) ordered_sums(const uint8_t *flags, const double *err,
                                                            const double *w, uint64_t nv, uint64_t nc,
                                                            double *error, double *area,
                                                            uint64_t *count, double *total) {
  const uint64_t b = blockIdx.x;
  if (b == 2 * nc) {
    const double t = serial_sum(nv, [&](uint64_t i) { return w[i]; });
    if (threadIdx.x == 0) *total = t;
  } else if (b >= nc) {
    const uint64_t c = b - nc;
    const uint8_t *f = flags + c * 2 * nv;
    const double a =
        serial_sum(2 * nv, [&](uint64_t i) { return f[i] ? w[i < nv ? i : i - nv] : 0.0; });
    if (threadIdx.x == 0) area[c] = a;
  } else {
    __shared__ unsigned long long n_s;
    const uint8_t *f = flags + b * 2 * nv;
    if (threadIdx.x == 0) n_s = 0;
    __syncthreads();
    unsigned n = 0;
    for (uint64_t i = threadIdx.x; i < nv; i += kSumThreads) n += f[i] != 0;
    n = __reduce_add_sync(0xffffffffu, n);
    if ((threadIdx.x & 31) == 0) atomicAdd(&n_s, (unsigned long long)n);
    const double e = serial_sum(nv, [&](uint64_t i) { return f[i] ? err[b * nv + i] : 0.0; });
    if (threadIdx.x == 0) error[b] = e, count[b] = n_s;
  }
}

}  // namespace

// Latency-bound: some 50 scans of 4,096 addends per sum (20 clusters of an
// 80,000-vertex torus: 0.31 ms; one warp per cluster adding in order, whose
// every addition waits for the one before, 13.9 ms).
void ordered_verification_sums(Call &call, const uint8_t *flags, const double *err,
                               const double *w, uint64_t nv, uint64_t nc, double *error,
                               double *area, uint64_t *count, double *total) {
  ordered_sums<<<unsigned(2 * nc + 1), kSumThreads, 0, call.stream()>>>(flags, err, w, nv, nc, error,
                                                                        area, count, total);
  check_launch();
  call.launched();
}

// Union-find over (set, vertex) rows (find_root: verification.cuh).
// parent index space: (c * 2 + dir) * nv + i ; -1 marks excluded vertices.
__global__ void init_parents(const uint8_t *flags, uint64_t n, int32_t *parent, uint64_t nv) {
  uint64_t k = uint64_t(blockIdx.x) * blockDim.x + threadIdx.x;
  if (k < n) parent[k] = flags[k] ? int32_t(k % nv) : -1;
}

__global__ void unite_edges(const uint64_t *nbr_off, const int32_t *nbr, uint64_t nv, uint64_t sets,
                            int32_t *parent_all, int *status, int retry_limit) {
  uint64_t k = uint64_t(blockIdx.x) * blockDim.x + threadIdx.x;
  if (k >= sets * nv) return;
  uint64_t set = k / nv;
  int32_t i = int32_t(k % nv);
  int32_t *parent = parent_all + set * nv;
  if (parent[i] < 0) return;
  for (uint64_t e = nbr_off[i]; e < nbr_off[i + 1]; ++e) {
    int32_t u = nbr[e];
    if (u <= i || parent[u] < 0) continue;  // each edge once, allowed ends only
    for (int guard = 0;; ++guard) {
      if (guard >= retry_limit) {
        atomicExch(status, DS_SPIN_LIMIT);
        return;
      }
      int32_t a = find_root(parent, i), b = find_root(parent, u);
      if (a < 0 || b < 0) {
        atomicExch(status, DS_SPIN_LIMIT);
        return;
      }
      if (a == b) break;
      if (a > b) {
        int32_t t = a;
        a = b;
        b = t;
      }
      if (atomicCAS(&parent[b], b, a) == b) break;
    }
  }
}

namespace {

// Of the k-th kept row (set * nv + vertex, ascending): its component as set *
// nv + root, and the vertex.
__global__ void root_keys(const int32_t *pos, uint64_t n, int32_t *parent_all, uint64_t nv,
                          uint64_t *keys, int32_t *vals) {
  const uint64_t k = uint64_t(blockIdx.x) * blockDim.x + threadIdx.x;
  if (k >= n) return;
  const uint64_t at = uint64_t(uint32_t(pos[k])), set = at / nv;
  const int32_t i = int32_t(at - set * nv);
  keys[k] = set * nv + uint64_t(uint32_t(find_root(parent_all + set * nv, i)));
  vals[k] = i;
}

// starts[s] = the first kept row of set s, s in [0, sets].
__global__ void set_starts(const int32_t *pos, uint64_t n, uint64_t nv, uint64_t sets,
                           uint64_t *starts) {
  const uint64_t s = uint64_t(blockIdx.x) * blockDim.x + threadIdx.x;
  if (s > sets) return;
  uint64_t lo = 0, hi = n;
  while (lo < hi) {
    const uint64_t mid = (lo + hi) / 2;
    if (uint64_t(uint32_t(pos[mid])) < s * nv) lo = mid + 1;
    else hi = mid;
  }
  starts[s] = lo;
}

// The result's order: the forward sets' members (a) cluster by cluster, then
// the inverse ones' (b).  sides: each set's vertices, ascending; members: the
// same grouped by component (keys and vals sorted by component), with first[k]
// = 1 where a component begins.
__global__ void result_order(const int32_t *pos, const uint64_t *keys, const int32_t *vals,
                             uint64_t n, uint64_t nv, uint64_t sets, const uint64_t *starts,
                             const uint64_t *dest, int32_t *sides, int32_t *members,
                             uint8_t *first) {
  const uint64_t k = uint64_t(blockIdx.x) * blockDim.x + threadIdx.x;
  if (k >= n) return;
  const uint64_t at = uint64_t(uint32_t(pos[k])), set = at / nv;
  const uint64_t to = dest[set] + (k - starts[set]);
  sides[to] = int32_t(at - set * nv);
  members[to] = vals[k];  // a set's rows keep their places in the sort
  first[to] = k == starts[set] || keys[k] != keys[k - 1];
}

// dest[s] = the place of set s's first member in the result's order.
__global__ void set_places(const uint64_t *starts, uint64_t nc, uint64_t *dest) {
  if (threadIdx.x || blockIdx.x) return;
  uint64_t at = 0;
  for (int dir = 0; dir < 2; ++dir)
    for (uint64_t c = 0; c < nc; ++c)
      dest[2 * c + dir] = at, at += starts[2 * c + dir + 1] - starts[2 * c + dir];
}

__global__ void triangle_query(const double *q, uint64_t n, double *out) {
  uint64_t i = uint64_t(blockIdx.x) * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const double *r = q + i * 12;
  out[i] = triangle_d2({r[0], r[1], r[2]}, {r[3], r[4], r[5]}, {r[6], r[7], r[8]}, {r[9], r[10], r[11]});
}

}  // namespace

// The union-find's bounded retry loop on a path of 64 vertices (every
// vertex supporting one set) with `retry_limit` retries: with 0 every union
// gives up at once and the call ends in the device-status error that a
// retry loop running out raises; with the regular limit the path becomes
// one component.  Returns the number of components.
uint64_t unite_selftest_host(Call &call, int retry_limit) {
  constexpr uint64_t n = 64;
  std::vector<uint64_t> off(n + 1);
  std::vector<int32_t> idx;
  for (uint64_t i = 0; i < n; ++i) {
    off[i] = idx.size();
    if (i > 0) idx.push_back(int32_t(i - 1));
    if (i + 1 < n) idx.push_back(int32_t(i + 1));
  }
  off[n] = idx.size();
  std::vector<uint8_t> flags(n, 1);
  cudaStream_t st = call.stream();
  const uint64_t *doff = call.upload(off.data(), n + 1);
  const int32_t *didx = call.upload(idx.data(), idx.size());
  const uint8_t *dflags = call.upload(flags.data(), n);
  int32_t *parent = call.alloc<int32_t>(n);
  init_parents<<<1, 64, 0, st>>>(dflags, n, parent, n);
  check_launch();
  unite_edges<<<1, 64, 0, st>>>(doff, didx, n, 1, parent, call.status(), retry_limit);
  check_launch();
  call.launched(2);
  std::vector<int32_t> h(n);
  call.d2h(h.data(), parent, n * 4);
  call.check_status("union-find self-test");
  uint64_t roots = 0;
  for (uint64_t i = 0; i < n; ++i) roots += h[i] == int32_t(i);
  return roots;
}

void triangle_distances_host(Call &call, const double *queries, uint64_t count, double *out) {
  if (!count) return;
  double *q = call.upload(queries, count * 12);
  double *d = call.alloc<double>(count);
  triangle_query<<<blocks_for(count), kThreads, 0, call.stream()>>>(q, count, d);
  check_launch();
  call.launched();
  call.d2h(out, d, count * 8);
  call.sync();
}

ClusterMotion cluster_motion(const sym_cluster_record &r) {
  ClusterMotion m{};
  for (int k = 0; k < 9; ++k) m.r[k] = r.rotation[k];
  for (int k = 0; k < 3; ++k) m.t[k] = r.translation[k], m.n[k] = r.plane_normal[k];
  m.offset = r.plane_offset;
  m.reflection = r.reflection != 0;
  return m;
}

void finish_verification(Call &call, const uint8_t *flags, const double *err, const double *w,
                         const uint64_t *nbr_off, const int32_t *nbr, uint64_t nv, uint64_t nc,
                         sym_verification_result &out, void *(*allocate)(size_t)) {
  cudaStream_t st = call.stream();
  const uint64_t rows = nc * 2 * nv, sets = 2 * nc;
  uint64_t n = 0, patches = 0;  // members of all sets; their components
  std::vector<uint64_t> starts(sets + 1, 0);
  std::vector<int32_t> begins;  // where the components begin, in the result's order
  int32_t *lists = nullptr, *dbegins = nullptr;
  double *sums = nullptr;
  if (nc) {
    sums = call.alloc<double>(3 * nc + 1);  // error, area, count (as bits), total
    uint64_t *na = reinterpret_cast<uint64_t *>(sums + 2 * nc);
    ordered_verification_sums(call, flags, err, w, nv, nc, sums, sums + nc, na, sums + 3 * nc);
    int32_t *parent = call.alloc<int32_t>(rows), *pos = call.alloc<int32_t>(rows);
    init_parents<<<blocks_for(rows), kThreads, 0, st>>>(flags, rows, parent, nv);
    check_launch();
    unite_edges<<<blocks_for(rows), kThreads, 0, st>>>(nbr_off, nbr, nv, sets, parent, call.status(),
                                                        kUniteRetries);
    check_launch();
    uint64_t *counts = call.alloc<uint64_t>(2), *dstarts = call.alloc<uint64_t>(sets + 1),
             *dest = call.alloc<uint64_t>(sets);
    compact_indices(call, flags, rows, pos, counts);
    call.d2h(&n, counts, 8);
    call.sync();
    call.launched(2);
    set_starts<<<blocks_for(sets + 1), kThreads, 0, st>>>(pos, n, nv, sets, dstarts);
    check_launch();
    set_places<<<1, 32, 0, st>>>(dstarts, nc, dest);
    check_launch();
    call.launched(2);
    call.d2h(starts.data(), dstarts, (sets + 1) * 8);
    if (n) {
      uint64_t *keys = call.alloc<uint64_t>(n), *skeys = call.alloc<uint64_t>(n);
      int32_t *vals = call.alloc<int32_t>(n), *svals = call.alloc<int32_t>(n);
      lists = call.alloc<int32_t>(2 * n), dbegins = call.alloc<int32_t>(n);
      uint8_t *first = call.alloc<uint8_t>(n);
      root_keys<<<blocks_for(n), kThreads, 0, st>>>(pos, n, parent, nv, keys, vals);
      check_launch();
      int bits = 1;
      while (bits < 64 && (rows >> bits)) ++bits;
      radix_sort_pairs(call, keys, vals, skeys, svals, n, bits);
      result_order<<<blocks_for(n), kThreads, 0, st>>>(pos, skeys, svals, n, nv, sets, dstarts, dest,
                                                       lists, lists + n, first);
      check_launch();
      compact_indices(call, first, n, dbegins, counts + 1);
      call.launched(2);
      call.d2h(&patches, counts + 1, 8);
    }
  }
  std::vector<double> hs(3 * nc + 1, 0.0);
  if (nc) call.d2h(hs.data(), sums, hs.size() * 8);
  call.check_status("verification");
  if (patches) {
    begins.resize(patches);
    call.d2h(begins.data(), dbegins, patches * 4);
    call.sync();
  }
  // the result block
  uint64_t na = 0;
  for (uint64_t c = 0; c < nc; ++c) na += starts[2 * c + 1] - starts[2 * c];
  const uint64_t ra = uint64_t(std::lower_bound(begins.begin(), begins.end(), int64_t(na),
                                                [](int32_t x, int64_t y) { return int64_t(uint32_t(x)) < y; }) -
                               begins.begin());
  const uint64_t nb = n - na, rb = patches - ra;
  const size_t bytes = (4 * (nc + 1) + (ra + 1) + (rb + 1)) * 8 + 2 * n * 4 + 2 * nc * 8 + 256;
  char *block = static_cast<char *>(allocate(bytes));
  if (!block) fail(SYM_RUNTIME_ERROR, "host allocation failed");
  out.storage = block;
  out.cluster_count = nc;
  uint64_t *u = reinterpret_cast<uint64_t *>(block);
  out.side_a_offsets = u, u += nc + 1;
  out.side_b_offsets = u, u += nc + 1;
  out.patches_a.groups = u, u += nc + 1;
  out.patches_b.groups = u, u += nc + 1;
  out.patches_a.offsets = u, u += ra + 1;
  out.patches_b.offsets = u, u += rb + 1;
  double *dd = reinterpret_cast<double *>(u);
  out.coverage = dd, dd += nc;
  out.rms = dd, dd += nc;
  int32_t *ii = reinterpret_cast<int32_t *>(dd);
  out.side_a = ii, ii += na;
  out.side_b = ii, ii += nb;
  out.patches_a.indices = ii, ii += na;
  out.patches_b.indices = ii;
  if (n) {
    try {
      call.d2h(out.side_a, lists, 2 * n * 4);  // sides a, b, then members a, b
      call.sync();
    } catch (...) {
      std::free(block);
      out = sym_verification_result{};
      throw;
    }
  }
  auto fill = [&](int dir, uint64_t *off, sym_grouped_csr &pg, uint64_t base, uint64_t first,
                  uint64_t last, uint64_t members) {
    off[0] = 0, pg.groups[0] = 0;
    uint64_t row = first;
    for (uint64_t c = 0; c < nc; ++c) {
      off[c + 1] = off[c] + starts[2 * c + dir + 1] - starts[2 * c + dir];
      while (row < last && uint64_t(uint32_t(begins[row])) - base < off[c + 1]) ++row;
      pg.groups[c + 1] = row - first;
    }
    for (uint64_t k = first; k < last; ++k) pg.offsets[k - first] = uint64_t(uint32_t(begins[k])) - base;
    pg.offsets[last - first] = members;
    pg.rows = last - first;
  };
  fill(0, out.side_a_offsets, out.patches_a, 0, 0, ra, na);
  fill(1, out.side_b_offsets, out.patches_b, na, ra, patches, nb);
  for (uint64_t c = 0; c < nc; ++c) {
    uint64_t count;
    std::memcpy(&count, &hs[2 * nc + c], 8);
    const double total = hs[3 * nc];
    out.rms[c] = count ? std::sqrt(hs[c] / double(count)) : 0;
    out.coverage[c] = total > 0 ? std::min(1.0, hs[nc + c] / total) : 0;
  }
}

// The vertices in Morton order of their position (10 bits per axis over
// the mesh's box, ties in index order): the query order of the
// verification kernels; `scale` receives the largest coordinate magnitude.
static std::vector<int32_t> morton_order(const sym_mesh_view &m, float &scale) {
  const uint64_t nv = m.vertices.count;
  const double *x[3] = {m.vertices.x, m.vertices.y, m.vertices.z};
  double lo[3], ext = 0;
  for (int a = 0; a < 3; ++a) {
    lo[a] = nv ? *std::min_element(x[a], x[a] + nv) : 0.0;
    const double hi = nv ? *std::max_element(x[a], x[a] + nv) : 0.0;
    ext = std::max(ext, hi - lo[a]);
    const double most = std::max(std::fabs(lo[a]), std::fabs(hi));
    scale = std::isfinite(most) ? std::max(scale, float(most) * (1 + 1e-6f)) : INFINITY;
  }
  std::vector<uint64_t> key(nv);
  for (uint64_t v = 0; v < nv; ++v) {
    uint64_t code = 0;
    for (int a = 0; a < 3; ++a) {
      const double u = ext > 0 ? (x[a][v] - lo[a]) / ext * 1024.0 : 0.0;
      const uint64_t cell = uint64_t(std::min(1023.0, std::max(0.0, u)));
      for (int bit = 0; bit < 10; ++bit) code |= ((cell >> bit) & 1u) << (3 * bit + (2 - a));
    }
    key[v] = code << 32 | v;
  }
  std::sort(key.begin(), key.end());
  std::vector<int32_t> order(nv);
  for (uint64_t j = 0; j < nv; ++j) order[j] = int32_t(uint32_t(key[j]));
  return order;
}

// Device core of sym_verification.  Mesh arrays are device pointers; `m` is
// the host mesh (the BVH is built on the host with the reference's
// construction order).
void verification_core(Call &call, const sym_mesh_view &m, const double *xyz, const int32_t *faces,
                       const double *vn, const double *w, const uint64_t *nbr_off,
                       const int32_t *nbr, const sym_cluster_record *records, uint64_t nc,
                       double tau, sym_verification_result &out, void *(*allocate)(size_t)) {
  const uint64_t nv = m.vertices.count, nf = m.faces.count;
  cudaStream_t st = call.stream();
  HostBvh bvh(m);
  if (2 * bvh.depth + 4 > kRefStack) fail(SYM_RUNTIME_ERROR, "verification: BVH too deep");
  Surface s;
  s.xyz = xyz;
  s.nv = nv;
  s.faces = faces;
  s.nf = nf;
  s.nodes = call.upload(bvh.nodes.data(), bvh.nodes.size());
  s.ids = call.upload(bvh.ids.data(), bvh.ids.size());
  float4 *boxes32 = call.alloc<float4>(3 * bvh.nodes.size()), *face32 = call.alloc<float4>(4 * nf);
  ref_boxes32<<<blocks_for(bvh.nodes.size()), kThreads, 0, st>>>(s.nodes, bvh.nodes.size(), boxes32);
  check_launch();
  lbvh_face_records<<<blocks_for(nf), kThreads, 0, st>>>(xyz, nv, faces, nf, face32, nullptr);
  check_launch();
  call.launched(2);
  std::vector<ClusterMotion> motions(nc);
  for (uint64_t c = 0; c < nc; ++c) motions[c] = cluster_motion(records[c]);
  ClusterMotion *dm = call.upload(motions.data(), nc);
  uint64_t rows = nc * 2 * nv;
  uint8_t *flags = call.alloc<uint8_t>(rows);
  double *err = call.alloc<double>(nc * nv);
  double limit = std::nextafter(tau * tau, std::numeric_limits<double>::infinity());
  float scale = 0;
  const std::vector<int32_t> order = morton_order(m, scale);
  const int32_t *dorder = call.upload(order.data(), order.size());
  verify_vertices<<<blocks_for(rows), kThreads, 0, st>>>(s, face32, boxes32, scale, vn, dorder, dm, nc,
                                                         tau, limit, flags, err, call.status());
  check_launch();
  call.launched();
  finish_verification(call, flags, err, w, nbr_off, nbr, nv, nc, out, allocate);
}

void verification_host(Call &call, const sym_mesh_view &m, const sym_topology_view &g,
                       const sym_clusters_view &cl, const sym_model_context &ctx,
                       const sym_options &o, sym_verification_result &out,
                       void *(*allocate)(size_t)) {
  const uint64_t nv = m.vertices.count, nf = m.faces.count, nc = cl.count;
  if (!nc) {
    finish_verification(call, nullptr, nullptr, nullptr, nullptr, nullptr, nv, 0, out, allocate);
  } else {
    if (!nv || !nf) fail(SYM_INVALID_ARGUMENT, "verification requires a nonempty surface");
    if (g.normals.count != nv || g.weight_count != nv || g.neighbors.rows != nv)
      fail(SYM_INVALID_ARGUMENT, "SoA component lengths differ");
    validate_csr(g.neighbors, nv, nv, "neighbors");
    for (uint64_t f = 0; f < nf; ++f)
      if (m.faces.v0[f] < 0 || m.faces.v1[f] < 0 || m.faces.v2[f] < 0 ||
          uint64_t(m.faces.v0[f]) >= nv || uint64_t(m.faces.v1[f]) >= nv ||
          uint64_t(m.faces.v2[f]) >= nv)
        fail(SYM_INVALID_ARGUMENT, "Face index out of range");
    double *xyz = upload_points(call, m.vertices);
    int32_t *faces = upload_faces(call, m.faces);
    double *vn = upload_points(call, g.normals);
    double *w = call.upload(g.weights, nv);
    uint64_t nbr_count = g.neighbors.offsets[nv];
    uint64_t *nbr_off = call.upload(g.neighbors.offsets, nv + 1);
    int32_t *nbr = call.upload(g.neighbors.indices, nbr_count);
    verification_core(call, m, xyz, faces, vn, w, nbr_off, nbr, cl.records, nc,
                      o.verify_threshold * ctx.box_size, out, allocate);
  }
}

}  // namespace sym
