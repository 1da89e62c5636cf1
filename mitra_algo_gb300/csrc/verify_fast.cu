// SPDX-License-Identifier: MPL-2.0
// Stage (d) on the throughput path: verification of resident meshes with a
// linear BVH built on the GPU, FP32 closest-point searches and FP64
// rechecks, with results identical to the reference's.
//
// The tests are the reference's (src/cpu/verification.cpp:22-110): a vertex
// supports a mode in one direction when its image under the mode's motion
// lies at least 2 tau from itself, on the correct side of a reflection
// plane, within tau of the surface, and its transformed normal is within
// 60 degrees of the nearest face's normal; coverage is the supporting
// vertices' weight over the total, rms the root mean square of the forward
// distances; patches are the connected components of the supporting
// vertices (region growing).
//
// How the decisions stay the reference's: the LBVH (Karras 2012: 30-bit
// Morton codes of the face centroids, radix sort, longest-common-prefix
// splits, boxes merged bottom-up, built once per resident mesh) is searched
// in FP32 with a window of 1,024 u M (u the FP32 unit, M the query's magnitude),
// and of the faces met those within 128 u M of the nearest are kept, more than the
// errors of two FP32 distances together (flat_d2 and face_d2n derive them), so the
// face of smallest FP64 distance is always among them.  That holds for any
// motion: a matrix that is not orthonormal widens M by its row sums (motion32).
// What FP32 leaves open is decided in FP64 over those candidates.  Where faces at
// the FP64 minimum disagree on the normal test, the one the reference's BVH visits
// first is found from the tree's order (first_in_reference_order); candidates
// that overflow the list go to a list of 64, and those that overflow that to the
// reference-order search (verification.cuh).  That tree is built on the host
// from the time the mesh is loaded.  Sums are the reference's serial ones.
#include "face32.cuh"
#include "primitives.cuh"
#include "verification.cuh"

#include <algorithm>
#include <cmath>
#include <limits>
#include <vector>

namespace sym {
namespace {

__device__ float segment_d2f(F3 p, F3 a, F3 b) {
  F3 d = b - a;
  float l = dotf(d, d), t = 0;
  if (l > 1e-14f) t = fminf(fmaxf(dotf(p - a, d) / l, 0.f), 1.f);
  F3 e = p - (a + d * t);
  return dotf(e, e);
}

// The region test of triangle_d2 (verification.cu) in FP32.
__device__ float triangle_d2f(F3 p, F3 a, F3 b, F3 c) {
  F3 ab = b - a, ac = c - a, ap = p - a;
  F3 n = crossf(ab, ac);
  if (dotf(n, n) < 1e-28f)
    return fminf(fminf(segment_d2f(p, a, b), segment_d2f(p, a, c)), segment_d2f(p, b, c));
  float d1 = dotf(ab, ap), d2 = dotf(ac, ap);
  if (d1 <= 0 && d2 <= 0) return dotf(ap, ap);
  F3 bp = p - b;
  float d3 = dotf(ab, bp), d4 = dotf(ac, bp);
  if (d3 >= 0 && d4 <= d3) return dotf(bp, bp);
  float vc = d1 * d4 - d3 * d2;
  if (vc <= 0 && d1 >= 0 && d3 <= 0) {
    F3 e = p - (a + ab * (d1 / (d1 - d3)));
    return dotf(e, e);
  }
  F3 cp = p - c;
  float d5 = dotf(ab, cp), d6 = dotf(ac, cp);
  if (d6 >= 0 && d5 <= d6) return dotf(cp, cp);
  float vb = d5 * d2 - d1 * d6;
  if (vb <= 0 && d2 >= 0 && d6 <= 0) {
    F3 e = p - (a + ac * (d2 / (d2 - d6)));
    return dotf(e, e);
  }
  float va = d3 * d6 - d5 * d4;
  if (va <= 0 && (d4 - d3) >= 0 && (d5 - d6) >= 0) {
    F3 e = p - (b + (c - b) * ((d4 - d3) / ((d4 - d3) + (d5 - d6))));
    return dotf(e, e);
  }
  float den = va + vb + vc;
  F3 e = p - (a + ab * (vb / den) + ac * (vc / den));
  return fmaxf(dotf(e, e), 0.f);
}

// --------------------------------------------------------------- LBVH build
__device__ __forceinline__ uint32_t spread3(uint32_t v) {  // 10 bits -> every third of 30
  v &= 0x3ffu;
  v = (v | (v << 16)) & 0x030000FFu;
  v = (v | (v << 8)) & 0x0300F00Fu;
  v = (v | (v << 4)) & 0x030C30C3u;
  v = (v | (v << 2)) & 0x09249249u;
  return v;
}

__global__ void lbvh_vertices(const double *xyz, uint64_t nv, float *xyz32) {
  uint64_t i = uint64_t(blockIdx.x) * blockDim.x + threadIdx.x;
  if (i < 3 * nv) xyz32[i] = float(xyz[i]);
}

// key = Morton code of the face centroid (30 bits) << 32 | face: unique.
__global__ void lbvh_keys(const float *xyz, uint64_t nv, const int32_t *faces, uint64_t nf,
                          float3 lo, float3 inv, uint64_t *keys, int32_t *ids) {
  uint64_t f = uint64_t(blockIdx.x) * blockDim.x + threadIdx.x;
  if (f >= nf) return;
  float c[3] = {0, 0, 0};
  for (int k = 0; k < 3; ++k) {
    int32_t v = faces[uint64_t(k) * nf + f];
    for (int a = 0; a < 3; ++a) c[a] += xyz[uint64_t(a) * nv + v];
  }
  float l[3] = {lo.x, lo.y, lo.z}, s[3] = {inv.x, inv.y, inv.z};
  uint32_t q[3];
  for (int a = 0; a < 3; ++a) {
    float u = (c[a] / 3.f - l[a]) * s[a];
    q[a] = uint32_t(fminf(fmaxf(u * 1024.f, 0.f), 1023.f));
  }
  uint32_t code = (spread3(q[0]) << 2) | (spread3(q[1]) << 1) | spread3(q[2]);
  keys[f] = (uint64_t(code) << 32) | uint64_t(uint32_t(f));
  ids[f] = int32_t(f);
}

// key = Morton code of vertex v (30 bits, the faces' quantisation) << 32 | v.
__global__ void lbvh_vertex_keys(const float *xyz, uint64_t nv, float3 lo, float3 inv,
                                 uint64_t *keys, int32_t *ids) {
  uint64_t v = uint64_t(blockIdx.x) * blockDim.x + threadIdx.x;
  if (v >= nv) return;
  float l[3] = {lo.x, lo.y, lo.z}, s[3] = {inv.x, inv.y, inv.z};
  uint32_t q[3];
  for (int a = 0; a < 3; ++a) {
    float u = (xyz[uint64_t(a) * nv + v] - l[a]) * s[a];
    q[a] = uint32_t(fminf(fmaxf(u * 1024.f, 0.f), 1023.f));
  }
  uint32_t code = (spread3(q[0]) << 2) | (spread3(q[1]) << 1) | spread3(q[2]);
  keys[v] = (uint64_t(code) << 32) | uint64_t(uint32_t(v));
  ids[v] = int32_t(v);
}

__device__ __forceinline__ int lcp(const uint64_t *keys, int64_t n, int64_t i, int64_t j) {
  if (j < 0 || j >= n) return -1;
  return __clzll(keys[i] ^ keys[j]);
}

// Internal node i of n - 1 (Karras 2012): its range, split and children;
// child < 0 encodes the leaf ~sorted position; parent_* = 2 * parent + slot.
// A node is 64 bytes (16 words: the children's boxes lo0 hi0 lo1 hi1, then
// their ids in words 12 and 13), so a traversal step reads it with four
// 16-byte loads instead of 14 4-byte ones.
constexpr int kNodeWords = 16, kNodeChild = 12;
__global__ void lbvh_internal(const uint64_t *keys, int64_t n, int32_t *node, int32_t *parent_in,
                              int32_t *parent_leaf) {
  int64_t i = int64_t(blockIdx.x) * blockDim.x + threadIdx.x;
  if (i >= n - 1) return;
  const int d = lcp(keys, n, i, i + 1) > lcp(keys, n, i, i - 1) ? 1 : -1;
  const int dmin = lcp(keys, n, i, i - d);
  int64_t lmax = 2;
  while (lcp(keys, n, i, i + lmax * d) > dmin) lmax *= 2;
  int64_t l = 0;
  for (int64_t t = lmax / 2; t >= 1; t /= 2)
    if (lcp(keys, n, i, i + (l + t) * d) > dmin) l += t;
  const int64_t j = i + l * d;
  const int dnode = lcp(keys, n, i, j);
  int64_t s = 0, t = l;
  do {
    t = (t + 1) / 2;
    if (lcp(keys, n, i, i + (s + t) * d) > dnode) s += t;
  } while (t > 1);
  const int64_t gamma = i + s * d + (d < 0 ? d : 0);
  const int64_t lo = i < j ? i : j, hi = i < j ? j : i;
  int32_t left = lo == gamma ? ~int32_t(gamma) : int32_t(gamma);
  int32_t right = hi == gamma + 1 ? ~int32_t(gamma + 1) : int32_t(gamma + 1);
  node[i * kNodeWords + kNodeChild] = left, node[i * kNodeWords + kNodeChild + 1] = right;
  if (left < 0) parent_leaf[gamma] = int32_t(2 * i);
  else parent_in[gamma] = int32_t(2 * i);
  if (right < 0) parent_leaf[gamma + 1] = int32_t(2 * i + 1);
  else parent_in[gamma + 1] = int32_t(2 * i + 1);
}

// Boxes bottom-up: every leaf writes its box into its parent's slot; the
// second child to arrive at a node merges both slots into the node's box
// and carries it one level up.  Leaves are renamed from sorted positions to
// face ids on the way.
__global__ void lbvh_boxes(const float *xyz, uint64_t nv, const int32_t *faces, int64_t n,
                           const int32_t *sorted_ids, int32_t *nodes, const int32_t *parent_in,
                           const int32_t *parent_leaf, unsigned *arrivals) {
  int64_t leaf = int64_t(blockIdx.x) * blockDim.x + threadIdx.x;
  if (leaf >= n) return;
  const int32_t f = sorted_ids[leaf];
  float b[6] = {INFINITY, INFINITY, INFINITY, -INFINITY, -INFINITY, -INFINITY};
  for (int k = 0; k < 3; ++k) {
    int32_t v = faces[uint64_t(k) * uint64_t(n) + f];
    for (int a = 0; a < 3; ++a) {
      float x = xyz[uint64_t(a) * nv + v];
      b[a] = fminf(b[a], x), b[3 + a] = fmaxf(b[3 + a], x);
    }
  }
  int32_t node = parent_leaf[leaf] >> 1;
  int slot = parent_leaf[leaf] & 1;
  float *box = reinterpret_cast<float *>(nodes);
  nodes[int64_t(node) * kNodeWords + kNodeChild + slot] = ~f;  // leaves now name faces
  for (int guard = 0; guard < 128; ++guard) {
    volatile float *dst = box + int64_t(node) * kNodeWords + slot * 6;
    for (int k = 0; k < 6; ++k) dst[k] = b[k];
    __threadfence();
    if (atomicAdd(&arrivals[node], 1u) == 0) return;  // the sibling finishes the node
    __threadfence();
    volatile const float *src = box + int64_t(node) * kNodeWords;
    for (int a = 0; a < 3; ++a) {
      b[a] = fminf(src[a], src[6 + a]);
      b[3 + a] = fmaxf(src[3 + a], src[9 + a]);
    }
    if (node == 0) return;
    slot = parent_in[node] & 1;
    node = parent_in[node] >> 1;
  }
}

// ------------------------------------------------------------ verification
constexpr int kStackFast = 96;

__device__ __forceinline__ float box_d2f(F3 p, float lx, float ly, float lz, float hx, float hy,
                                         float hz) {
  float dx = fmaxf(fmaxf(lx - p.x, p.x - hx), 0.f);
  float dy = fmaxf(fmaxf(ly - p.y, p.y - hy), 0.f);
  float dz = fmaxf(fmaxf(lz - p.z, p.z - hz), 0.f);
  return dx * dx + dy * dy + dz * dz;
}

struct BvhView {
  uint64_t nv, nf;
  const int32_t *faces;
  const float *xyz;
  const float4 *node;    // nf - 1 records of four (lbvh_internal)
  const float4 *face;    // nf records of four: (a, inv_ab), (b, inv_bc), (c, inv_ca), (n, reach)
  const float4 *flat;    // nf records of four, for the candidate search (FlatFace)
  const int32_t *order;  // nv: query order of the vertices (Morton order of their position)
  const double *fn64;    // nf x 3: the faces' FP64 unit normals of the normal test
};

__device__ __forceinline__ F3 vtx(const BvhView &b, int32_t v) {
  return {b.xyz[v], b.xyz[b.nv + v], b.xyz[2 * b.nv + v]};
}
__device__ __forceinline__ Face load_face(const BvhView &b, int32_t f) { return sym::load_face(b.face, f); }
__device__ __forceinline__ float face_d2(const BvhView &b, F3 p, int32_t f) {
  const float4 *r = b.face + 4 * int64_t(f);
  const float4 x = r[0], y = r[1], z = r[2];
  return triangle_d2f(p, {x.x, x.y, x.z}, {y.x, y.y, y.z}, {z.x, z.y, z.z});
}

// The children of a node and p's squared distances to their boxes.
struct Children {
  int32_t c0, c1;
  float d0, d1;
};
__device__ __forceinline__ Children load_children(const BvhView &b, F3 p, int32_t node) {
  const float4 *r = b.node + 4 * int64_t(node);
  const float4 x = r[0], y = r[1], z = r[2], w = r[3];
  return {__float_as_int(w.x), __float_as_int(w.y), box_d2f(p, x.x, x.y, x.z, x.w, y.x, y.y),
          box_d2f(p, y.z, y.w, z.x, z.y, z.z, z.w)};
}

// A stack entry: a node and its box's squared distance, moved as one word.
struct __align__(8) Pending {
  int32_t node;
  float d2;
};

// Nearest face within `best` (FP32), near-first; -1 when none.
__device__ int32_t nearest_face_fast(const BvhView &b, F3 p, float &best, int *status) {
  int32_t face = -1;
  if (b.nf == 1) {
    float d = face_d2(b, p, 0);
    if (d < best) best = d, face = 0;
    return face;
  }
  Pending stack[kStackFast];
  int top = 0;
  stack[top++] = {0, 0.f};
  while (top) {
    const Pending at = stack[--top];
    if (at.d2 >= best) continue;
    const Children k = load_children(b, p, at.node);
    if (k.c0 < 0 && k.d0 < best) {
      float d = face_d2(b, p, ~k.c0);
      if (d < best) best = d, face = ~k.c0;
    }
    if (k.c1 < 0 && k.d1 < best) {
      float d = face_d2(b, p, ~k.c1);
      if (d < best) best = d, face = ~k.c1;
    }
    const bool p0 = k.c0 >= 0 && k.d0 < best, p1 = k.c1 >= 0 && k.d1 < best;
    if (top + 2 > kStackFast) {
      atomicExch(status, DS_CAPACITY);
      return face;
    }
    const bool first0 = k.d0 <= k.d1;  // the nearer child is popped first
    if (p0 && !first0) stack[top++] = {k.c0, k.d0};
    if (p1) stack[top++] = {k.c1, k.d1};
    if (p0 && first0) stack[top++] = {k.c0, k.d0};
  }
  return face;
}

// The verification tests of one (mode, vertex, direction) query with the
// FP32 search (the refinement's correspondences): returns the nearest face
// when vertex i supports mode m in that direction (-1 otherwise), its FP32
// squared distance in `best` (entering as tau^2) and the image of the vertex
// in q.  The motion is applied in FP64.
__device__ __forceinline__ int32_t support_query(const BvhView &b, const double *xyz,
                                                 const double *vn, const ClusterMotion &m,
                                                 uint64_t i, bool inverse, double tau, float &best,
                                                 double q[3], int *status) {
  const uint64_t nv = b.nv;
  double r[9];
  for (int k = 0; k < 9; ++k) r[k] = inverse ? m.r[(k % 3) * 3 + k / 3] : m.r[k];
  const double p[3] = {xyz[i], xyz[nv + i], xyz[2 * nv + i]};
  double move2 = 0;
  for (int a = 0; a < 3; ++a) {
    double s = 0;
    for (int k = 0; k < 3; ++k) s += r[a * 3 + k] * (inverse ? p[k] - m.t[k] : p[k]);
    q[a] = inverse ? s : s + m.t[a];
    move2 += (q[a] - p[a]) * (q[a] - p[a]);
  }
  if (move2 < 4 * tau * tau) return -1;
  if (m.reflection) {
    double side = m.n[0] * p[0] + m.n[1] * p[1] + m.n[2] * p[2] + m.offset;
    if (inverse ? side <= tau : side >= -tau) return -1;
  }
  const F3 qf{float(q[0]), float(q[1]), float(q[2])};
  const int32_t face = nearest_face_fast(b, qf, best, status);
  if (face < 0) return -1;
  const Face at = load_face(b, face);
  F3 fn = crossf(at.b - at.a, at.c - at.a);
  float len = sqrtf(dotf(fn, fn));
  if (!(len > 0.f)) return -1;
  const double ni[3] = {vn[i], vn[nv + i], vn[2 * nv + i]};
  float rn[3];
  for (int k = 0; k < 3; ++k)
    rn[k] = float(r[k * 3] * ni[0] + r[k * 3 + 1] * ni[1] + r[k * 3 + 2] * ni[2]);
  if ((rn[0] * fn.x + rn[1] * fn.y + rn[2] * fn.z) / len < 0.5f) return -1;
  return face;
}

// ------------------------------------------- exact decisions, FP32 search
// Error bound of the FP32 search, in distance units: kErr (512 FP32 units u)
// times M, the largest coordinate magnitude of the vertex, its image, the
// translation and the mesh, at least 2 tau, times the motion's gain (motion32).
// A decided FP32 distance is far inside kErr M of the reference's FP64 distance
// whatever the face's shape, 56 u M (flat_d2) to 73 (face_d2n); a face without a usable normal (its FP64
// normal not accurate to well below u: no area, or a corner angle with sin
// below 1e-6), or one that face_d2n leaves undecided (a projection within the
// rounding band of an edge line), enters the candidates by a lower bound and
// leaves the decision to FP64.  The same bound serves as the band of the FP32
// threshold tests (2 tau, the plane side, tau), and kNormalBand (on the cosine)
// as that of the normal test, whose FP32 error is a few u times the gain.
constexpr float kErr = 1.0f / 32768.0f;
constexpr float kNormalBand = 1.0f / 1024.0f;
constexpr int kCandidates = 16;

// A face as the candidate search reads it, 64 bytes: the triangle in its own
// plane.  Corner a, the unit normal n and the unit direction e of ab (both
// rounded from FP64), and with x along e and y along n x e the corners b = (l, 0)
// and c = (cx, cy), the reciprocal lengths of the three edges, and `reach`, a
// bound on the edge lengths; reach 0: no usable normal; reach < 0: a face longer
// than a quarter of the mesh's largest coordinate, or with an edge outside 1e-15 ..
// 1e15, for which face_d2n decides.
struct FlatFace {
  F3 a, n, e;
  float l, cx, cy, rab, rbc, rca, reach;
};
__device__ __forceinline__ FlatFace load_flat(const BvhView &b, int32_t f) {
  const float4 *r = b.flat + 4 * int64_t(f);
  const float4 x = r[0], y = r[1], z = r[2], w = r[3];
  return {{x.x, x.y, x.z}, {y.x, y.y, y.z}, {z.x, z.y, z.z}, x.w, y.w, z.w, w.x, w.y, w.z, w.w};
}
__device__ __forceinline__ float dot_fma(F3 a, F3 b) { return fmaf(a.x, b.x, fmaf(a.y, b.y, a.z * b.z)); }

// FP32 squared distance from p to a face with reach > 0, within 64 u M of its
// FP64 distance; only the plane distance when that is above `lim` already.
// The in-plane distance is 0 when p projects inside the three edge lines by
// more than the rounding of those tests (band), else that to the nearest edge
// segment: of a p that projects inside by less, whose in-plane distance is 0, the
// nearest segment is within two bands.
// Error, with M the largest coordinate magnitude of mesh, image and translation
// and at least 2 tau (times the motion's gain, which the image's share needs), and w
// = p - a, |w| <= tau + reach <= 0.75 M: the image (30
// u M) and a (1.8 u M) move w by 32 u M + u |w|; n, e and n x e are within u,
// u and 4 u of their directions, and the products round by 3 u |w| each, which
// moves (h, x, y) by sqrt(4^2 + 4^2 + 8^2) u |w| <= 8 u M; b and c by 2 u reach
// <= u M; the line tests, 5 u (|x| + |y| + reach) <= 6.5 u M each, enter twice; the
// rest is rounding of the distance, 4 u (0.5 M): 32 + 8 + 1 + 13 + 2 = 56 u M.
// In the plane a distance takes some 45 instructions where face_d2n's, from the
// corners and with a band of its own per edge function, take some 120: verify_fp32
// on the 1e6-triangle torus (2e7 queries) 35 ms, 41 with face_d2n; 31 with five
// CTAs per SM instead of four (it waits for memory most of the time).
__device__ __forceinline__ float flat_d2(F3 p, const FlatFace &f, float lim) {
  const F3 w = p - f.a;
  const float h = dot_fma(f.n, w), h2 = h * h;
  if (h2 > lim) return h2;
  const F3 m{fmaf(f.n.y, f.e.z, -(f.n.z * f.e.y)), fmaf(f.n.z, f.e.x, -(f.n.x * f.e.z)),
             fmaf(f.n.x, f.e.y, -(f.n.y * f.e.x))};
  const float x = dot_fma(f.e, w), y = dot_fma(m, w);
  const float bx = f.cx - f.l, rx = x - f.l;  // b to c, b to p
  const float sbc = fmaf(bx, y, -(f.cy * rx)) * f.rbc, sca = fmaf(f.cy, x, -(f.cx * y)) * f.rca;
  const float band = 5.f * kUnit * (fabsf(x) + fabsf(y) + f.reach);
  if (fminf(y, fminf(sbc, sca)) > band) return h2;
  const float tab = __saturatef(x * f.rab);
  const float tbc = __saturatef(fmaf(rx, bx, y * f.cy) * f.rbc * f.rbc);
  const float tca = __saturatef(fmaf(x, f.cx, y * f.cy) * f.rca * f.rca);
  const float ax = fmaf(-f.l, tab, x);
  const float ux = fmaf(-bx, tbc, rx), uy = fmaf(-f.cy, tbc, y);
  const float vx = fmaf(-f.cx, tca, x), vy = fmaf(-f.cy, tca, y);
  const float g2 = fminf(fmaf(ax, ax, y * y), fminf(fmaf(ux, ux, uy * uy), fmaf(vx, vx, vy * vy)));
  return h2 + g2;
}

// The region of the face p's nearest point seems to lie in (0, 1, 2: nearest to
// the segment ab, bc, ca; 3: inside) and its squared distance `d2` (flat_d2).
__device__ __forceinline__ int flat_region(F3 p, const FlatFace &f, float &d2) {
  d2 = flat_d2(p, f, INFINITY);
  const F3 w = p - f.a;
  const F3 m{fmaf(f.n.y, f.e.z, -(f.n.z * f.e.y)), fmaf(f.n.z, f.e.x, -(f.n.x * f.e.z)),
             fmaf(f.n.x, f.e.y, -(f.n.y * f.e.x))};
  const float x = dot_fma(f.e, w), y = dot_fma(m, w);
  const float sbc = fmaf(f.cx - f.l, y, -(f.cy * (x - f.l))) * f.rbc, sca = fmaf(f.cy, x, -(f.cx * y)) * f.rca;
  const float least = fminf(y, fminf(sbc, sca));
  return least >= 0.f ? 3 : least == y ? 0 : least == sbc ? 1 : 2;
}

// Faces whose FP64 distance to the image can be the smallest: every face
// whose FP32 distance (or, for a face face_d2n leaves undecided or one
// without a usable normal, a lower bound: the face_d2n bound or the box
// distance) is within 2 error bounds of min(best FP32 distance, tau +
// bound) -- the face of smallest FP64 distance is at most 2 bounds farther
// in FP32 than the best FP32 face.  Nodes are pruned with a slightly larger
// radius, for the rounding of their boxes' distances.  The search's window is
// generous; the faces returned are held to the errors of decided distances
// themselves, at most 73 u M too long for one and 51 too short for the other of two:
// within 128 u M of the best (with the search's window, 1,024 u M,
// eight times as many queries found neighbouring faces in it that disagree on
// the normal test, and went to FP64).  Undecided faces are listed as ~face.  Returns the count (N + 1 on
// overflow: faces and keys hold N entries); `best` receives the smallest FP32
// squared distance of a decided face (INFINITY when none lies within tau + 3
// bounds).
template <int N = kCandidates>
__device__ int candidate_faces(const BvhView &b, F3 p, float tau_err, float err, int32_t *faces,
                               float *keys, float &best, int *status) {
  best = INFINITY;
  float radius = tau_err + 2.f * err;
  float lim = radius * radius, lim_box = (radius + err * 0.03125f) * (radius + err * 0.03125f);
  int n = 0;
  bool overflow = false;
  const float um = err * (1.f / 512.f);  // err = kErr M = 512 u M
  auto consider = [&](int32_t f, float box) {
    const FlatFace face = load_flat(b, f);
    float key = box;
    int32_t id = ~f;
    if (face.reach > 0.f) key = flat_d2(p, face, lim), id = f;
    else if (face.reach < 0.f && face_d2n(p, load_face(b, f), um, lim, key)) id = f;
    if (id >= 0) {
      if (key < best) {
        best = key;
        radius = fminf(tau_err, sqrtf(best)) + 2.f * err;
        lim = radius * radius;
        lim_box = (radius + err * 0.03125f) * (radius + err * 0.03125f);
      }
    }
    if (key > lim) return;
    if (n == N) {  // drop entries beyond the current limit
      int m = 0;
      for (int j = 0; j < n; ++j)
        if (keys[j] <= lim) faces[m] = faces[j], keys[m++] = keys[j];
      n = m;
    }
    if (n == N) {
      overflow = true;
      return;
    }
    faces[n] = id, keys[n++] = key;
  };
  if (b.nf == 1) {
    consider(0, 0.f);
  } else {
    Pending stack[kStackFast];
    int top = 0;
    stack[top++] = {0, 0.f};
    while (top) {
      const Pending at = stack[--top];
      if (at.d2 > lim_box) continue;
      const Children k = load_children(b, p, at.node);
      if (k.c0 < 0 && k.d0 <= lim_box) consider(~k.c0, k.d0);
      if (k.c1 < 0 && k.d1 <= lim_box) consider(~k.c1, k.d1);
      const bool p0 = k.c0 >= 0 && k.d0 <= lim_box, p1 = k.c1 >= 0 && k.d1 <= lim_box;
      if (top + 2 > kStackFast) {
        atomicExch(status, DS_CAPACITY);
        return N + 1;
      }
      const bool first0 = k.d0 <= k.d1;  // the nearer child is popped first
      if (p0 && !first0) stack[top++] = {k.c0, k.d0};
      if (p1) stack[top++] = {k.c1, k.d1};
      if (p0 && first0) stack[top++] = {k.c0, k.d0};
    }
  }
  if (overflow) return N + 1;
  // what is left by the errors of two decided distances
  radius = fminf(tau_err, sqrtf(best)) + 128.f * um;
  lim = fminf(lim, radius * radius);
  int m = 0;
  for (int j = 0; j < n; ++j)
    if (keys[j] <= lim) faces[m] = faces[j], keys[m++] = keys[j];
  return m;
}

// A cluster's motion in FP32 (the FP32 decisions).
struct MotionF {
  float r[9], t[3], n[3], offset;
  int32_t reflection;
  float gain;  // the largest row or column sum of |r| (and |n|_1) over an orthonormal one's bound
  float reach;  // the largest magnitude among t and, of a reflection, offset
};

// A record's matrix need not be orthonormal: one whose products cancel brings an
// image of ordinary size with the rounding of large terms.  The error bounds are
// those of row sums up to sqrt(3), an orthonormal matrix's most, and grow with
// the sum beyond.  (A matrix or plane that is not finite keeps them: its
// images are not finite either.)
MotionF motion32(const sym_cluster_record &r) {
  MotionF m{};
  double most = 0;
  for (int k = 0; k < 3; ++k) {
    double row = 0, column = 0;
    for (int j = 0; j < 3; ++j) row += std::fabs(r.rotation[3 * k + j]), column += std::fabs(r.rotation[3 * j + k]);
    most = std::max(most, std::max(row, column));
  }
  m.reflection = r.reflection != 0;
  if (m.reflection)
    most = std::max(most, std::fabs(r.plane_normal[0]) + std::fabs(r.plane_normal[1]) + std::fabs(r.plane_normal[2]));
  m.gain = std::isfinite(most) ? std::max(1.f, float(most / 1.7320508 * (1 - 1e-6))) : 1.f;
  for (int k = 0; k < 9; ++k) m.r[k] = float(r.rotation[k]);
  for (int k = 0; k < 3; ++k) {
    m.t[k] = float(r.translation[k]), m.n[k] = float(r.plane_normal[k]);
    m.reach = std::fmax(m.reach, std::fabs(m.t[k]));
  }
  m.offset = float(r.plane_offset);
  if (m.reflection) m.reach = std::fmax(m.reach, std::fabs(m.offset));
  return m;
}

// Row lists between the verification kernels.
// A row (c, direction, vertex i) holds the flag and error of one query;
// the kernels take the queries qid = (c, direction, j) of vertex order[j],
// the vertices in Morton order of their position, so a warp serves
// neighbouring vertices of one motion and walks nearly the same BVH nodes
// (in the mesh's own vertex order the warps of the benchmark mesh spread
// over 3x more of it).  The FP64 and reference-order queries are marked
// per query and compacted in ascending order (compact_indices), so their
// warps keep that locality; appended in completion order they made every
// load of a warp 32 scattered ones.
constexpr uint32_t kNoSlot = 0xffffffffu;
constexpr uint32_t kWideSlot = 0xfffffffeu;  // overflowed the list: for verify_rows_wide
constexpr int32_t kNoFace = INT32_MIN;  // padding of a candidate list (~f marks an undecided face)

struct RowLists {
  uint32_t *forward;    // accepted forward rows whose FP64 distance is still needed
  int32_t *faces;       // kCandidates faces per forward row (-1 padded)
  uint8_t *mark;        // per query: 1 = left to the next kernel (FP64, then reference order)
  int32_t *fp64;        // queries decided in FP64, ascending
  int32_t *reference;   // queries left to the wide list, then to the reference-order BVH
  // FP64 queries the first FP64 pass leaves to the second: with candidates
  // from the front, without from the back of `capacity` entries
  int32_t *open;
  uint64_t capacity;
  // the FP32 candidates of an FP64 query (kCandidates per slot, kNoFace
  // padded), so the FP64 decisions need no search of their own; slot_of[qid]
  // = kNoSlot for a query sent on before its candidates were known,
  // kWideSlot for one whose candidates overflowed the list
  uint32_t *slot_of;
  int32_t *cand;
  unsigned long long slots;    // capacity of cand, in slots
  unsigned long long *counts;  // [forward, slots used, open with candidates, tie, open without]
};

// Decisions in FP32 (verify_fp32).  The reference's tests are made with
// the FP32 image of the vertex; each threshold test that falls within its
// band of the threshold, a badly shaped face among the candidates,
// candidates that disagree on the normal test, or a candidate overflow send
// the row to the FP64 decisions.  An accepted forward row is listed with its
// candidates, the faces its FP64 distance is the smallest of.
__global__ void __launch_bounds__(kThreads, 5)
    verify_fp32(BvhView b, const float *vn32, const MotionF *motions, uint64_t nc, float tau,
                float scale, uint8_t *flags, double *err, RowLists lists, int *status) {
  // query q = (c, direction, j) takes vertex i = order[j]: the warps walk
  // neighbouring vertices; flags and errors stay per vertex (row)
  const uint64_t qid = uint64_t(blockIdx.x) * blockDim.x + threadIdx.x;
  const uint64_t nv = b.nv;
  if (qid >= nc * 2 * nv) return;
  const uint64_t c = qid / (2 * nv), rem = qid % (2 * nv);
  const bool inverse = rem >= nv;
  const uint64_t i = uint64_t(b.order[rem % nv]);
  const uint64_t row = qid - rem % nv + i;
  flags[row] = 0;
  lists.mark[qid] = 0;
  if (!inverse) err[c * nv + i] = 0.0;
  const MotionF &m = motions[c];
  float r[9];
  for (int k = 0; k < 9; ++k) r[k] = inverse ? m.r[(k % 3) * 3 + k / 3] : m.r[k];
  const F3 p = vtx(b, int32_t(i));
  const F3 u = inverse ? F3{p.x - m.t[0], p.y - m.t[1], p.z - m.t[2]} : p;
  F3 q{r[0] * u.x + r[1] * u.y + r[2] * u.z, r[3] * u.x + r[4] * u.y + r[5] * u.z,
       r[6] * u.x + r[7] * u.y + r[8] * u.z};
  if (!inverse) q = q + F3{m.t[0], m.t[1], m.t[2]};
  const float mag = fmaxf(fmaxf(scale, 2.f * tau), fmaxf(fabsf(q.x), fmaxf(fabsf(q.y), fabsf(q.z))));
  const float e = kErr * m.gain * fmaxf(mag, m.reach);
  auto to_fp64 = [&]() {
    lists.mark[qid] = 1;
    lists.slot_of[qid] = kNoSlot;
  };
  // the image moves at least 2 tau (verification.cpp:64)
  const F3 dq = q - p;
  const float moved = sqrtf(dotf(dq, dq));
  if (fabsf(moved - 2.f * tau) <= 2.f * e) return to_fp64();
  if (moved < 2.f * tau) return;
  if (m.reflection) {  // the vertex lies on the plane's side (verification.cpp:66, :84)
    const float side = m.n[0] * p.x + m.n[1] * p.y + m.n[2] * p.z + m.offset;
    const float at = inverse ? tau : -tau;
    if (fabsf(side - at) <= e) return to_fp64();
    if (inverse ? side <= tau : side >= -tau) return;
  }
  int32_t faces[kCandidates];
  float keys[kCandidates];
  float best;
  const int n = candidate_faces(b, q, tau + e, e, faces, keys, best, status);
  if (n > kCandidates) {  // the same search would overflow again: straight to the wide list
    lists.mark[qid] = 1;
    lists.slot_of[qid] = kWideSlot;
    return;
  }
  // from here on an FP64 row keeps its candidates: they hold every face at
  // the FP64 minimum (the window covers the FP32 error of the FP64 image)
  auto to_fp64_listed = [&]() {
    lists.mark[qid] = 1;
    const unsigned long long k = atomicAdd(&lists.counts[1], 1ull);
    if (k >= lists.slots) {
      lists.slot_of[qid] = kNoSlot;
      return;
    }
    lists.slot_of[qid] = uint32_t(k);
    for (int j = 0; j < kCandidates; ++j) lists.cand[k * kCandidates + j] = j < n ? faces[j] : kNoFace;
  };
  for (int j = 0; j < n; ++j)
    if (faces[j] < 0) return to_fp64_listed();  // an undecided face
  if (!n) return;                        // no face within tau (all farther than tau + 3e)
  const float dbest = sqrtf(best);
  if (dbest - e > tau) return;           // every face farther than tau
  if (dbest + e >= tau) return to_fp64_listed();
  // the normal test of every candidate (verification.cpp:70-73)
  const F3 ni{vn32[i], vn32[nv + i], vn32[2 * nv + i]};
  const F3 rn{r[0] * ni.x + r[1] * ni.y + r[2] * ni.z, r[3] * ni.x + r[4] * ni.y + r[5] * ni.z,
              r[6] * ni.x + r[7] * ni.y + r[8] * ni.z};
  int agree = 0, disagree = 0;
  for (int j = 0; j < n; ++j) {
    // the face's unit normal from its FP64 corners (every candidate here
    // has one): the cosine is good to a few u
    const float4 fn = b.face[4 * int64_t(faces[j]) + 3];
    const float v = dotf(rn, F3{fn.x, fn.y, fn.z});
    if (fabsf(v - 0.5f) <= kNormalBand * m.gain) return to_fp64_listed();
    if (v >= 0.5f) ++agree;
    else ++disagree;
  }
  if (agree && disagree) return to_fp64_listed();
  if (!agree) return;
  flags[row] = 1;
  if (!inverse) {
    const unsigned long long k = atomicAdd(&lists.counts[0], 1ull);
    lists.forward[k] = uint32_t(row);
    for (int j = 0; j < kCandidates; ++j) lists.faces[k * kCandidates + j] = j < n ? faces[j] : -1;
  }
}

// The reference's normal test (verification.cpp:70-73, normal_agrees) with
// the face's unit normal from the per-mesh table: the same FP64 values.
__device__ __forceinline__ bool normal_agrees_t(const BvhView &b, int32_t f, const M3 &r, D3 ni) {
  const D3 fnorm{b.fn64[3 * uint64_t(f)], b.fn64[3 * uint64_t(f) + 1], b.fn64[3 * uint64_t(f) + 2]};
  return !(dot(mul(r, ni), fnorm) < 0.5);
}

// One query of the reference's verification, decided with the FP32
// candidates and FP64 rechecks.  Returns 1 (supports; `d2` = the reference's
// FP64 squared distance), 0 (does not), 3 (the faces at the minimum, listed
// in `tied`, N entries, -1 padded, disagree on the normal test; `d2` = the
// minimum) or 2 (more than N candidates; `d2` = the tau^2 search limit).
//
// The reference keeps the face of strictly smallest FP64 distance, the first
// its BVH visits among faces at exactly that distance (surface.h:52-83).
// The candidates hold every face that can be at the minimum, so their FP64
// minimum is the reference's distance; the normal test of the faces at
// exactly that minimum decides when they all give the same outcome; when
// they do not, the reference's visiting order decides (verify_listed_ref).
template <int N = kCandidates>
__device__ int hybrid_query(const BvhView &b, const Surface &s, const double *vn,
                            const ClusterMotion &m, bool inverse, uint64_t i, double tau,
                            float scale, double &d2, int32_t *tied, int *status) {
  const M3 r = query_rotation(m, inverse);
  const D3 p = vertex(s, int32_t(i));
  D3 q;
  if (query_skipped(m, r, inverse, p, tau, q)) return 0;
  const F3 qf{float(q.x), float(q.y), float(q.z)};
  const float mag = fmaxf(fmaxf(scale, 2.f * float(tau)), fmaxf(fabsf(qf.x), fmaxf(fabsf(qf.y), fabsf(qf.z))));
  const float e = kErr * mag;
  int32_t faces[N];
  float keys[N];
  float best;
  const int n = candidate_faces<N>(b, qf, float(tau) + e, e, faces, keys, best, status);
  if (n > N) {
    d2 = nextafter(tau * tau, double(INFINITY));
    return 2;
  }
  double dmin = INFINITY;
  double dist[N];
  for (int j = 0; j < n; ++j) {
    faces[j] = faces[j] < 0 ? ~faces[j] : faces[j];
    dist[j] = triangle_d2(q, corner(s, faces[j], 0), corner(s, faces[j], 1), corner(s, faces[j], 2));
    dmin = fmin(dmin, dist[j]);
  }
  if (!(dmin <= tau * tau)) return 0;
  const D3 ni{vn[i], vn[s.nv + i], vn[2 * s.nv + i]};
  int agree = 0, disagree = 0, t = 0;
  for (int j = 0; j < n; ++j) {
    if (dist[j] != dmin) continue;
    tied[t++] = faces[j];
    if (normal_agrees_t(b, faces[j], r, ni)) ++agree;
    else ++disagree;
  }
  d2 = dmin;
  if (agree && disagree) {
    for (int j = t; j < N; ++j) tied[j] = -1;
    return 3;
  }
  return agree ? 1 : 0;
}

// u M of a query whose image is q, M as the error of a FlatFace distance has it.
__device__ __forceinline__ float search_unit(const ClusterMotion &m, F3 q, float scale, float tau) {
  const float t = fmaxf(fabsf(float(m.t[0])), fmaxf(fabsf(float(m.t[1])), fabsf(float(m.t[2]))));
  return kUnit * fmaxf(fmaxf(fmaxf(scale, 2.f * tau), t), fmaxf(fabsf(q.x), fmaxf(fabsf(q.y), fabsf(q.z))));
}

// Which corner of the face is the nearest point to p, by the region tests of
// triangle_d2, when FP32 decides them: 0, 1, 2 for a, b, c, else -1.  p is
// within 1.8 u M of its FP64 value, as the corners are, so a product e . (p - v)
// is within 3.6 u M (|e| + |p - v|) of its own and its rounding within 5 u |e|
// |p - v|; the band takes twice that and more, in 1-norms.  A decided corner
// is the nearest point by that margin, and for faces with a usable normal
// (corner angles with sin above 1e-6) the FP64 tests, good to 1e-16 of the same
// products, then choose its region too: the distance is triangle_d2's
// |p - v|^2, the same FP64 expression.
__device__ __forceinline__ int corner_region(F3 p, const Face &f, float um) {
  const F3 ab = f.b - f.a, ac = f.c - f.a, bc = f.c - f.b;
  const F3 ap = p - f.a, bp = p - f.b, cp = p - f.c;
  auto norm1 = [](F3 x) { return fabsf(x.x) + fabsf(x.y) + fabsf(x.z); };
  const float lab = norm1(ab), lac = norm1(ac), lbc = norm1(bc);
  const float lap = norm1(ap), lbp = norm1(bp), lcp = norm1(cp);
  // e . v beyond its band, to the + or the - side
  auto above = [&](float x, float le, float lv) { return x > 8.f * um * (le + lv) + 1e-6f * le * lv; };
  if (above(-dotf(ab, ap), lab, lap) && above(-dotf(ac, ap), lac, lap)) return 0;
  if (above(dotf(ab, bp), lab, lbp) && above(-dotf(bc, bp), lbc, lbp)) return 1;
  if (above(dotf(ac, cp), lac, lcp) && above(dotf(bc, cp), lbc, lcp)) return 2;
  return -1;
}

// FP64 distances of a block's rows, one per thread.  FP64 runs at 1/64 of the
// FP32 rate, and a warp pays for an FP64 operation whether one of its lanes needs
// it or all: FP64 is kept to what FP32 cannot decide, and what is left is sorted
// so that the lanes of a warp need the same.
//  * A face whose nearest point is one of its corners (most of a rough mesh's
//    rows: the faces around a vertex at exactly one distance) takes that vertex's
//    |q - v|^2, eight FP64 operations and none for the next face around the
//    same vertex.
//  * Another face is evaluated only when its FP32 distance does not already put it
//    beyond the smallest of those.
//  * What remains goes by the region its nearest point seems to lie in (an edge
//    of the three, or inside) into one of four lists, and whole warps take 32
//    distances of one list: triangle_d2 returns early for the edges, and its
//    divisions, a fifth of its operations, are those of one region.  A wrong
//    guess costs time only.
constexpr int kRowThreads = 256, kRegions = 4, kRegionItems = 384;
struct RowBlock {
  double q[kRowThreads][3], d[kRegions][kRegionItems];
  unsigned long long dmin[kRowThreads];  // as bits: no distance is negative
  const int32_t *list[kRowThreads];
  unsigned at_min[kRowThreads];
  unsigned count[kRegions];
  uint16_t item[kRegions][kRegionItems];  // row * 16 + candidate
};
static_assert(kCandidates == 16 && kRowThreads * 16 <= 65536, "an item is 16 bits");

// The candidates of a row seen in FP32: bit sets of those at the smallest
// distance so far, in no corner's region, and of the normal test's outcome.
struct RowFaces {
  unsigned at_min = 0, open = 0, agrees = 0, unsure = 0;
  double dmin = INFINITY;
  __device__ __forceinline__ void take(double d, int j) {
    if (d < dmin) dmin = d, at_min = 0;
    if (d == dmin) at_min |= 1u << j;
  }
};
__device__ __forceinline__ int32_t listed_face(int32_t x) { return x < 0 ? ~x : x; }

// The candidates cl (up to `end`) of a row whose image is q: their corner
// distances, and with NORMALS their normal tests (turned normal rn, `band`).
template <bool NORMALS>
__device__ __forceinline__ RowFaces corner_distances(const BvhView &b, const Surface &s, D3 q, F3 qf, float um,
                                                     const int32_t *cl, int32_t end, F3 rn, float band) {
  RowFaces r;
  double dv = 0;
  int32_t at_vertex = -1;  // of which dv is the squared distance
  for (int j = 0; j < kCandidates && cl[j] != end; ++j) {
    const int32_t f = listed_face(cl[j]);
    const Face face = load_face(b, f);
    if (NORMALS) {
      const float cosine = dotf(rn, face.n);
      if (face.reach == 0.f || !(fabsf(cosine - 0.5f) > band)) r.unsure |= 1u << j;
      else if (cosine > 0.5f) r.agrees |= 1u << j;
    }
    const int v = face.reach == 0.f ? -1 : corner_region(qf, face, um);
    if (v < 0) {
      r.open |= 1u << j;
      continue;
    }
    const int32_t id = s.faces[uint64_t(v) * s.nf + f];
    if (id != at_vertex) {
      const D3 e = q - vertex(s, id);
      dv = dot(e, e), at_vertex = id;
    }
    r.take(dv, j);
  }
  return r;
}

// Whether face f is farther than dmin in FP32 already (its decided FP32
// distance is within 64 u M of FP64's); `region`: the list its distance belongs to.
__device__ __forceinline__ bool beyond(const BvhView &b, F3 p, int32_t f, float um, double dmin, int &region) {
  const FlatFace face = load_flat(b, f);
  region = 3;
  if (!(face.reach > 0.f)) return false;
  float key;
  region = flat_region(p, face, key);
  return dmin < INFINITY && sqrtf(key) > sqrtf(float(dmin)) + 128.f * um;
}

// The smallest FP64 distance of the row of each thread (`live` ones) over the
// faces `r` left open and the corners it has, and the candidates at exactly that
// distance (TIES).  Called by the whole block; `cl` and `end` as above.
template <bool TIES>
__device__ __forceinline__ void block_distances(RowBlock &sh, const BvhView &b, const Surface &s, bool live,
                                                D3 q, F3 qf, float um, const int32_t *cl, RowFaces &r) {
  const int t = threadIdx.x;
  if (t < kRegions) sh.count[t] = 0;
  __syncthreads();
  if (live) {
    sh.q[t][0] = q.x, sh.q[t][1] = q.y, sh.q[t][2] = q.z;
    sh.list[t] = cl, sh.at_min[t] = 0;
    for (unsigned rest = r.open; rest; rest &= rest - 1) {
      const int j = __ffs(int(rest)) - 1;
      const int32_t f = listed_face(cl[j]);
      int region;
      if (beyond(b, qf, f, um, r.dmin, region)) continue;
      const unsigned at = atomicAdd(&sh.count[region], 1u);
      if (at < kRegionItems) sh.item[region][at] = uint16_t(t * 16 + j);
      else r.take(triangle_d2(q, corner(s, f, 0), corner(s, f, 1), corner(s, f, 2)), j);  // no room left
    }
    sh.dmin[t] = __double_as_longlong(r.dmin);
  }
  __syncthreads();
  const int lane = t & 31, warp = t >> 5;
  unsigned chunks[kRegions + 1];
  chunks[0] = 0;
  for (int k = 0; k < kRegions; ++k) chunks[k + 1] = chunks[k] + (min(sh.count[k], unsigned(kRegionItems)) + 31) / 32;
  for (unsigned c = warp; c < chunks[kRegions]; c += kRowThreads / 32) {
    int k = 0;
    while (c >= chunks[k + 1]) ++k;
    const unsigned at = (c - chunks[k]) * 32 + lane;
    if (at < min(sh.count[k], unsigned(kRegionItems))) {
      const int row = sh.item[k][at] >> 4;
      const int32_t f = listed_face(sh.list[row][sh.item[k][at] & 15]);
      const D3 x{sh.q[row][0], sh.q[row][1], sh.q[row][2]};
      const double d = triangle_d2(x, corner(s, f, 0), corner(s, f, 1), corner(s, f, 2));
      if (TIES) sh.d[k][at] = d;
      atomicMin(&sh.dmin[row], (unsigned long long)__double_as_longlong(d));
    }
  }
  __syncthreads();
  if (TIES) {
    for (int k = 0; k < kRegions; ++k)
      for (unsigned at = t; at < min(sh.count[k], unsigned(kRegionItems)); at += kRowThreads) {
        const int row = sh.item[k][at] >> 4;
        if ((unsigned long long)__double_as_longlong(sh.d[k][at]) == sh.dmin[row])
          atomicOr(&sh.at_min[row], 1u << (sh.item[k][at] & 15));
      }
    __syncthreads();
  }
  if (live) {
    const double d = __longlong_as_double((long long)sh.dmin[t]);
    if (d < r.dmin) r.dmin = d, r.at_min = 0;
    r.at_min |= sh.at_min[t];
  }
  __syncthreads();  // the lists are free again
}

// The reference's FP64 squared distance of each listed forward row: the
// smallest over its candidate faces (the face it keeps is among them).
// 3.3e6 rows of the 180,000-vertex torus: 1.4 ms (1.6 with two CTAs per SM in
// place of four); a lane per row that evaluated
// every candidate took 2.9.
__global__ void __launch_bounds__(kRowThreads, 4) forward_errors(BvhView b, Surface s, const ClusterMotion *motions,
                                                              RowLists lists, unsigned long long count,
                                                              float scale, float tau, double *err) {
  __shared__ RowBlock sh;
  const uint64_t k = uint64_t(blockIdx.x) * kRowThreads + threadIdx.x;
  const uint64_t nv = s.nv;
  const bool live = k < count;
  uint64_t at = 0;
  D3 q{0, 0, 0};
  F3 qf{0, 0, 0};
  float um = 0;
  RowFaces r;
  const int32_t *cl = nullptr;
  if (live) {
    const uint64_t row = lists.forward[k], c = row / (2 * nv), i = row % (2 * nv);
    const ClusterMotion &m = motions[c];
    at = c * nv + i;
    q = mul(query_rotation(m, false), vertex(s, int32_t(i))) + D3{m.t[0], m.t[1], m.t[2]};
    qf = F3{float(q.x), float(q.y), float(q.z)};
    um = search_unit(m, qf, scale, tau);
    cl = lists.faces + k * kCandidates;
    r = corner_distances<false>(b, s, q, qf, um, cl, -1, F3{0, 0, 0}, 0.f);
  }
  block_distances<false>(sh, b, s, live, q, qf, um, cl, r);
  if (live) err[at] = r.dmin;
}

// A query of the FP64 rows.
struct Query {
  uint64_t c, i, row;
  bool inverse;
};
__device__ __forceinline__ Query query_of(const BvhView &b, uint64_t qid) {
  const uint64_t nv = b.nv, rem = qid % (2 * nv);
  Query x;
  x.c = qid / (2 * nv), x.inverse = rem >= nv;
  x.i = uint64_t(b.order[rem % nv]);
  x.row = qid - rem % nv + x.i;
  return x;
}
// Its vertex's image and the unit of the FP32 search there (verify_fp32 decided
// the 2 tau and side tests of a row with candidates), its turned normal, and the
// band of the normal test.
__device__ __forceinline__ void query_image(const Surface &s, const ClusterMotion *motions,
                                            const MotionF *motions32, const float *vn32, const Query &x,
                                            float scale, float tau, D3 &q, F3 &qf, float &um, F3 &rn,
                                            float &band) {
  const ClusterMotion &m = motions[x.c];
  const M3 r = query_rotation(m, x.inverse);
  const D3 p = vertex(s, int32_t(x.i)), mt{m.t[0], m.t[1], m.t[2]};
  q = x.inverse ? mul(r, p - mt) : mul(r, p) + mt;
  qf = F3{float(q.x), float(q.y), float(q.z)};
  um = search_unit(m, qf, scale, tau);
  const MotionF &mf = motions32[x.c];
  band = kNormalBand * mf.gain;
  float rf[9];
  for (int j = 0; j < 9; ++j) rf[j] = x.inverse ? mf.r[(j % 3) * 3 + j / 3] : mf.r[j];
  const F3 ni{vn32[x.i], vn32[s.nv + x.i], vn32[2 * s.nv + x.i]};
  rn = F3{rf[0] * ni.x + rf[1] * ni.y + rf[2] * ni.z, rf[3] * ni.x + rf[4] * ni.y + rf[5] * ni.z,
          rf[6] * ni.x + rf[7] * ni.y + rf[8] * ni.z};
}
// The decision of a row whose faces at the minimum are known: the normal test of
// those, and where they disagree (`tie`) that of the one the reference's search
// visits first (its visiting order is a total order on the faces for this query).
__device__ __forceinline__ bool decide_row(const BvhView &b, const RefBvh &t, const double *vn,
                                           const ClusterMotion &m, const Query &x, double tau, D3 q, float um,
                                           const int32_t *cl, RowFaces &r, bool &tie) {
  if (!(r.dmin <= tau * tau)) return false;
  for (unsigned rest = r.at_min & r.unsure; rest; rest &= rest - 1) {
    const int j = __ffs(int(rest)) - 1;
    if (normal_agrees_t(b, listed_face(cl[j]), query_rotation(m, x.inverse),
                        D3{vn[x.i], vn[b.nv + x.i], vn[2 * b.nv + x.i]}))
      r.agrees |= 1u << j;
  }
  tie = (r.at_min & r.agrees) && (r.at_min & ~r.agrees);
  if (!tie) return (r.at_min & r.agrees) != 0;
  int jf = __ffs(int(r.at_min)) - 1;
  int32_t first = listed_face(cl[jf]);
  for (unsigned rest = r.at_min & (r.at_min - 1); rest; rest &= rest - 1) {
    const int j = __ffs(int(rest)) - 1;
    const int32_t f = listed_face(cl[j]);
    if (first_in_reference_order_f(t, q, um, first, f) != first) first = f, jf = j;
  }
  return r.agrees >> jf & 1u;
}

// The FP64 decisions of the rows verify_fp32 listed, a lane per row, where the
// corners decide (block_distances); the others, with a face left to evaluate or
// without candidates, are left in lists.open for verify_rows_open, from its two
// ends: the searches of the latter take much longer.  Rows whose candidates
// overflowed stay marked for verify_rows_wide.  On the 1e6-triangle torus 1.1e7
// rows take 3.0 ms and the 3.3e6 left to the second kernel 2.8 (4.2 with a lane per
// row that evaluates its open faces in turn); eight lanes per row, each with its
// own copy of the image, took 17 and 11.  Both wait for the faces' records as much
// as for FP64, so the launch bounds leave room for four and three CTAs per SM (two
// each: 4.3 and 3.4 ms).
__global__ void __launch_bounds__(kThreads, 4) verify_rows_fp64(BvhView b, Surface s, RefBvh t, const double *vn, const float *vn32,
                                 const ClusterMotion *motions, const MotionF *motions32, double tau,
                                 float scale, uint8_t *flags, double *err, RowLists lists,
                                 unsigned long long rows) {
  const uint64_t k = uint64_t(blockIdx.x) * blockDim.x + threadIdx.x;
  const int lane = threadIdx.x & 31;
  int32_t left = -1;      // the row to list for the second kernel
  bool search = false;    // ... which has to search
  bool tie = false;
  if (k < rows) {
    const uint64_t qid = uint64_t(lists.fp64[k]);  // a query, as verify_fp32's
    const uint32_t slot = lists.slot_of[qid];
    if (slot == kNoSlot) {
      left = int32_t(qid), search = true;
    } else if (slot != kWideSlot) {
      const Query x = query_of(b, qid);
      D3 q;
      F3 qf, rn;
      float um, band;
      query_image(s, motions, motions32, vn32, x, scale, float(tau), q, qf, um, rn, band);
      const int32_t *cl = lists.cand + uint64_t(slot) * kCandidates;
      RowFaces r = corner_distances<true>(b, s, q, qf, um, cl, kNoFace, rn, band);
      for (unsigned rest = r.open; rest && left < 0; rest &= rest - 1) {
        int region;
        if (r.dmin == INFINITY || !beyond(b, qf, listed_face(cl[__ffs(int(rest)) - 1]), um, r.dmin, region))
          left = int32_t(qid);
      }
      if (left < 0) {
        const bool ok = decide_row(b, t, vn, motions[x.c], x, tau, q, um, cl, r, tie);
        flags[x.row] = ok;
        if (!x.inverse) err[x.c * b.nv + x.i] = ok ? r.dmin : 0.0;
        lists.mark[qid] = 0;
      }
    }
  }
  const unsigned ties = __ballot_sync(0xffffffffu, tie);
  if (ties && lane == 0) atomicAdd(&lists.counts[3], (unsigned long long)__popc(ties));
  // one atomic per warp and list
  const unsigned rows_left = __ballot_sync(0xffffffffu, left >= 0 && !search),
                 to_search = __ballot_sync(0xffffffffu, left >= 0 && search);
  unsigned long long at = 0;
  if (lane == 0 && rows_left) at = atomicAdd(&lists.counts[2], (unsigned long long)__popc(rows_left));
  if (lane == 1 && to_search) at = atomicAdd(&lists.counts[4], (unsigned long long)__popc(to_search));
  const unsigned long long rows_at = __shfl_sync(0xffffffffu, at, 0),
                           search_at = __shfl_sync(0xffffffffu, at, 1);
  const unsigned lt = (1u << lane) - 1;
  if (left >= 0 && !search) lists.open[rows_at + __popc(rows_left & lt)] = left;
  if (left >= 0 && search) lists.open[lists.capacity - 1 - (search_at + __popc(to_search & lt))] = left;
}

// The rows verify_rows_fp64 left: those that search (whole blocks of them, on one
// lane each), then those with candidates.
__global__ void __launch_bounds__(kRowThreads, 3) verify_rows_open(
    BvhView b, Surface s, RefBvh t, const double *vn, const float *vn32, const ClusterMotion *motions,
    const MotionF *motions32, double tau, float scale, uint8_t *flags, double *err, RowLists lists,
    int *status) {
  __shared__ RowBlock sh;
  const unsigned long long searches = lists.counts[4], open = lists.counts[2];
  const unsigned long long listed_from = (searches + kRowThreads - 1) / kRowThreads * kRowThreads;
  const int lane = threadIdx.x & 31;
  for (uint64_t k0 = uint64_t(blockIdx.x) * kRowThreads; k0 < listed_from + open;
       k0 += uint64_t(gridDim.x) * kRowThreads) {  // whole blocks of one kind
    const uint64_t k = k0 + threadIdx.x;
    bool tie = false;
    if (k0 < listed_from) {
      if (k < searches) {
        const uint64_t qid = uint64_t(lists.open[lists.capacity - 1 - k]);
        const Query x = query_of(b, qid);
        const ClusterMotion &m = motions[x.c];
        double d = 0;
        int32_t tied[kCandidates];
        int v = hybrid_query(b, s, vn, m, x.inverse, x.i, tau, scale, d, tied, status);
        if (v == 3) {
          tie = true;
          const M3 r = query_rotation(m, x.inverse);
          D3 q;
          query_skipped(m, r, x.inverse, vertex(s, int32_t(x.i)), tau, q);
          int32_t first = tied[0];
          for (int j = 1; j < kCandidates && tied[j] >= 0; ++j)
            first = first_in_reference_order(t, q, first, tied[j]);
          v = normal_agrees_t(b, first, r, D3{vn[x.i], vn[b.nv + x.i], vn[2 * b.nv + x.i]}) ? 1 : 0;
        }
        flags[x.row] = v == 1;
        if (!x.inverse) err[x.c * b.nv + x.i] = v == 1 ? d : 0.0;
        if (v != 2) lists.mark[qid] = 0;  // marked queries go on to the reference-order search
      }
    } else {
      const bool live = k < listed_from + open;
      uint64_t qid = 0;
      Query x{};
      D3 q{0, 0, 0};
      F3 qf{0, 0, 0}, rn{0, 0, 0};
      float um = 0, band = 0;
      RowFaces r;
      const int32_t *cl = nullptr;
      if (live) {
        qid = uint64_t(lists.open[k - listed_from]);
        x = query_of(b, qid);
        query_image(s, motions, motions32, vn32, x, scale, float(tau), q, qf, um, rn, band);
        cl = lists.cand + uint64_t(lists.slot_of[qid]) * kCandidates;
        r = corner_distances<true>(b, s, q, qf, um, cl, kNoFace, rn, band);
      }
      block_distances<true>(sh, b, s, live, q, qf, um, cl, r);
      if (live) {
        const bool ok = decide_row(b, t, vn, motions[x.c], x, tau, q, um, cl, r, tie);
        flags[x.row] = ok;
        if (!x.inverse) err[x.c * b.nv + x.i] = ok ? r.dmin : 0.0;
        lists.mark[qid] = 0;
      }
    }
    const unsigned ties = __ballot_sync(0xffffffffu, tie);
    if (ties && lane == 0) atomicAdd(&lists.counts[3], (unsigned long long)__popc(ties));
  }
}

// Queries whose candidates overflowed the list of verify_fp32 and of
// verify_rows_fp64: the same FP32 search and FP64 decision with room for
// kWideCandidates faces (one thread per query; such queries are rare, and
// the reference-order search they would otherwise take walks the
// reference's BVH one FP64 node at a time).  A query that overflows this
// list as well stays marked for verify_listed_ref.
constexpr int kWideCandidates = 64;
__global__ void verify_rows_wide(BvhView b, Surface s, RefBvh t, const double *vn,
                                 const ClusterMotion *motions, double tau, float scale,
                                 uint8_t *flags, double *err, RowLists lists,
                                 unsigned long long count, int *status) {
  const uint64_t k = uint64_t(blockIdx.x) * blockDim.x + threadIdx.x;
  if (k >= count) return;
  const uint64_t qid = uint64_t(lists.reference[k]), nv = b.nv;  // a query, as verify_fp32's
  const uint64_t c = qid / (2 * nv), rem = qid % (2 * nv);
  const bool inverse = rem >= nv;
  const uint64_t i = uint64_t(b.order[rem % nv]);
  const uint64_t row = qid - rem % nv + i;
  double d = 0;
  int32_t tied[kWideCandidates];
  int v = hybrid_query<kWideCandidates>(b, s, vn, motions[c], inverse, i, tau, scale, d, tied,
                                        status);
  if (v == 2) return;  // still marked
  if (v == 3) {
    atomicAdd(&lists.counts[3], 1ull);
    const M3 r = query_rotation(motions[c], inverse);
    D3 q;
    query_skipped(motions[c], r, inverse, vertex(s, int32_t(i)), tau, q);
    int32_t first = tied[0];
    for (int x = 1; x < kWideCandidates && tied[x] >= 0; ++x)
      first = first_in_reference_order(t, q, first, tied[x]);
    v = normal_agrees_t(b, first, r, D3{vn[i], vn[nv + i], vn[2 * nv + i]}) ? 1 : 0;
  }
  flags[row] = v == 1;
  if (!inverse) err[c * nv + i] = v == 1 ? d : 0.0;
  lists.mark[qid] = 0;
}

// Queries whose candidates overflowed the wide list too: the reference's
// search itself (exact_query) with the search limit nextafter(tau^2, inf).
__global__ void verify_listed_ref(Surface s, const double *vn, const int32_t *order,
                                  const ClusterMotion *motions, double tau, RowLists lists,
                                  unsigned long long count, uint8_t *flags, double *err,
                                  int *status) {
  const uint64_t k = uint64_t(blockIdx.x) * blockDim.x + threadIdx.x;
  if (k >= count) return;
  const uint64_t qid = lists.reference[k], nv = s.nv;  // a query, as verify_fp32's
  const uint64_t c = qid / (2 * nv), rem = qid % (2 * nv);
  const bool inverse = rem >= nv;
  const uint64_t i = uint64_t(order[rem % nv]);
  const uint64_t row = qid - rem % nv + i;
  double d = 0;
  const bool ok = exact_query(s, vn, motions[c], inverse, i, tau,
                              nextafter(tau * tau, double(INFINITY)), d, status);
  flags[row] = ok;
  if (!inverse) err[c * nv + i] = ok ? d : 0.0;
}

// Cluster c < nc: sum of the forward errors, supporting weight (both
// directions) and forward count; c == nc: the total weight.  kTreeThreads
// fixed-order strided partials and a fixed tree: reproducible, and within a
// few units of rounding of the reference's serial sums.  A partial is a chain
// of FP64 additions, which one SM runs at 1/64 of its FP32 rate, so the chains
// are spread: a warp of 32 strides takes one of the two sums
// (tree_partials, one-warp blocks), with kTreeAhead elements' loads in flight,
// and the trees follow in a kernel of their own.  1e6-triangle torus, 20
// clusters: 490 us; a block of all 256 strides per cluster took 1,570 us.
constexpr int kTreeThreads = 256, kTreeAhead = 8;

__global__ void __launch_bounds__(32) tree_partials(const uint8_t *flags, const double *err,
                                                    const double *w, uint64_t nv, uint64_t nc,
                                                    double *partial, unsigned *partial_count) {
  const uint64_t c = blockIdx.z, kind = blockIdx.y;  // 0: the errors, 1: the weights
  const unsigned stride0 = blockIdx.x * 32 + threadIdx.x;
  const uint8_t *fa = flags + c * 2 * nv, *fb = fa + nv;
  double sum = 0;
  unsigned n = 0;
  for (uint64_t i0 = stride0; i0 < nv; i0 += kTreeThreads * kTreeAhead) {
    if (c == nc) {
      if (kind == 0) break;
      double v[kTreeAhead];
#pragma unroll
      for (int k = 0; k < kTreeAhead; ++k) {
        const uint64_t i = i0 + uint64_t(k) * kTreeThreads;
        v[k] = i < nv ? w[i] : 0.0;
      }
#pragma unroll
      for (int k = 0; k < kTreeAhead; ++k)
        if (i0 + uint64_t(k) * kTreeThreads < nv) sum += v[k];
      continue;
    }
    bool a[kTreeAhead], b[kTreeAhead];
    double v[kTreeAhead];
#pragma unroll
    for (int k = 0; k < kTreeAhead; ++k) {
      const uint64_t i = i0 + uint64_t(k) * kTreeThreads;
      a[k] = i < nv && fa[i], b[k] = i < nv && kind == 1 && fb[i];
    }
#pragma unroll
    for (int k = 0; k < kTreeAhead; ++k) {
      const uint64_t i = i0 + uint64_t(k) * kTreeThreads;
      v[k] = a[k] || b[k] ? (kind == 0 ? err[c * nv + i] : w[i]) : 0.0;
    }
#pragma unroll
    for (int k = 0; k < kTreeAhead; ++k) {
      if (a[k]) sum += v[k], ++n;
      if (b[k]) sum += v[k];
    }
  }
  const uint64_t at = (c * 2 + kind) * kTreeThreads + stride0;
  partial[at] = sum;
  if (kind == 0) partial_count[c * kTreeThreads + stride0] = n;
}

__global__ void __launch_bounds__(kTreeThreads) tree_sums(const double *partial,
                                                          const unsigned *partial_count, uint64_t nc,
                                                          double *error, double *area,
                                                          uint64_t *count, double *total) {
  __shared__ double se[kTreeThreads], sa[kTreeThreads];
  __shared__ unsigned long long sn[kTreeThreads];
  const uint64_t c = blockIdx.x;
  se[threadIdx.x] = partial[c * 2 * kTreeThreads + threadIdx.x];
  sa[threadIdx.x] = partial[(c * 2 + 1) * kTreeThreads + threadIdx.x];
  sn[threadIdx.x] = partial_count[c * kTreeThreads + threadIdx.x];
  __syncthreads();
  for (int h = kTreeThreads / 2; h; h >>= 1) {
    if (int(threadIdx.x) < h) {
      se[threadIdx.x] += se[threadIdx.x + h];
      sa[threadIdx.x] += sa[threadIdx.x + h];
      sn[threadIdx.x] += sn[threadIdx.x + h];
    }
    __syncthreads();
  }
  if (threadIdx.x == 0) {
    if (c == nc) {
      *total = sa[0];
    } else {
      error[c] = se[0], area[c] = sa[0], count[c] = sn[0];
    }
  }
}

// ------------------------------------------------ FP64 transform refinement
// Closest point of triangle abc to p in FP64: the region tests of Ericson,
// Real-Time Collision Detection, 2005, section 5.1.5, and for a triangle
// without area (|ab x ac|^2 < 1e-28) the nearest of its three segments, the
// rule of the verification's distance (the reference's
// point_triangle_distance2).
__device__ void closest_on_segment(const double p[3], const double a[3], const double b[3],
                                   double out[3]) {
  double d[3], l = 0, t = 0;
  for (int k = 0; k < 3; ++k) d[k] = b[k] - a[k], l += d[k] * d[k];
  if (l > 1e-14) {
    t = ((p[0] - a[0]) * d[0] + (p[1] - a[1]) * d[1] + (p[2] - a[2]) * d[2]) / l;
    t = t < 0.0 ? 0.0 : (1.0 < t ? 1.0 : t);
  }
  for (int k = 0; k < 3; ++k) out[k] = a[k] + d[k] * t;
}

__device__ void closest_point(const double p[3], const double a[3], const double b[3],
                              const double c[3], double out[3]) {
  double ab[3], ac[3], ap[3], bp[3], cp[3];
  for (int k = 0; k < 3; ++k)
    ab[k] = b[k] - a[k], ac[k] = c[k] - a[k], ap[k] = p[k] - a[k], bp[k] = p[k] - b[k],
    cp[k] = p[k] - c[k];
  auto dot3 = [](const double *x, const double *y) { return x[0] * y[0] + x[1] * y[1] + x[2] * y[2]; };
  const double n[3] = {ab[1] * ac[2] - ab[2] * ac[1], ab[2] * ac[0] - ab[0] * ac[2],
                       ab[0] * ac[1] - ab[1] * ac[0]};
  if (dot3(n, n) < 1e-14 * 1e-14) {  // no area: the nearest of the three segments
    double s[3][3], e[3];
    closest_on_segment(p, a, b, s[0]);
    closest_on_segment(p, a, c, s[1]);
    closest_on_segment(p, b, c, s[2]);
    for (int j = 0; j < 3; ++j) {
      const double r[3] = {p[0] - s[j][0], p[1] - s[j][1], p[2] - s[j][2]};
      e[j] = dot3(r, r);
    }
    const int m01 = e[1] < e[0] ? 1 : 0;
    const int pick = e[2] < e[m01] ? 2 : m01;
    for (int k = 0; k < 3; ++k) out[k] = s[pick][k];
    return;
  }
  auto set = [&](const double *base, const double *dir, double t) {
    for (int k = 0; k < 3; ++k) out[k] = base[k] + dir[k] * t;
  };
  const double d1 = dot3(ab, ap), d2 = dot3(ac, ap);
  if (d1 <= 0 && d2 <= 0) return set(a, ab, 0);
  const double d3 = dot3(ab, bp), d4 = dot3(ac, bp);
  if (d3 >= 0 && d4 <= d3) return set(b, ab, 0);
  const double vc = d1 * d4 - d3 * d2;
  if (vc <= 0 && d1 >= 0 && d3 <= 0) return set(a, ab, d1 / (d1 - d3));
  const double d5 = dot3(ab, cp), d6 = dot3(ac, cp);
  if (d6 >= 0 && d5 <= d6) return set(c, ab, 0);
  const double vb = d5 * d2 - d1 * d6;
  if (vb <= 0 && d2 >= 0 && d6 <= 0) return set(a, ac, d2 / (d2 - d6));
  const double va = d3 * d6 - d5 * d4;
  if (va <= 0 && (d4 - d3) >= 0 && (d5 - d6) >= 0) {
    const double bc[3] = {c[0] - b[0], c[1] - b[1], c[2] - b[2]};
    return set(b, bc, (d4 - d3) / ((d4 - d3) + (d5 - d6)));
  }
  const double den = va + vb + vc;
  for (int k = 0; k < 3; ++k) out[k] = a[k] + ab[k] * (vb / den) + ac[k] * (vc / den);
}

struct Origin {
  double x[3];
};

// Forward correspondences: for each vertex i that supports mode c forward
// (the verification's tests), the FP64 closest point of its nearest face to
// the vertex's image, relative to `o`; ok[c * nv + i] says which.
__global__ void refine_pairs(BvhView b, const double *xyz, const double *vn,
                             const ClusterMotion *motions, uint64_t nc, double tau, float tau2, Origin o,
                             double *target, uint8_t *ok, int *status) {
  // query (c, j) takes vertex i = order[j] (neighbouring vertices in a
  // warp); the pairs stay per vertex (row), so the sums keep their order
  const uint64_t qid = uint64_t(blockIdx.x) * blockDim.x + threadIdx.x;
  const uint64_t nv = b.nv;
  if (qid >= nc * nv) return;
  const uint64_t c = qid / nv, i = uint64_t(b.order[qid % nv]), row = c * nv + i;
  ok[row] = 0;
  float best = tau2;
  double q[3];
  const int32_t face = support_query(b, xyz, vn, motions[c], i, false, tau, best, q, status);
  if (face < 0) return;
  double corner[3][3], out[3];
  for (int k = 0; k < 3; ++k) {
    const int32_t v = b.faces[uint64_t(k) * b.nf + face];
    for (int a = 0; a < 3; ++a) corner[k][a] = xyz[uint64_t(a) * nv + v];
  }
  closest_point(q, corner[0], corner[1], corner[2], out);
  for (int a = 0; a < 3; ++a) target[row * 3 + a] = out[a] - o.x[a];
  ok[row] = 1;
}

constexpr int kRefineSums = 28, kRefineThreads = 128, kRefineGroups = 9, kRefineAhead = 4;

// The strided partials of N sums over the correspondences of one cluster: a
// thread takes vertices i0, i0 + kRefineThreads, ... in order.  `terms` adds a
// correspondence's terms from its weight and those of the coordinates of p
// (the vertex) and q (its target) that the masks P and Q name; the loads of
// kRefineAhead vertices are in flight together.
template <unsigned P, unsigned Q, int N, class Terms>
__device__ __forceinline__ void refine_partials(const double *xyz, const double *w, uint64_t nv,
                                                const uint8_t *ok, const double *target,
                                                const Origin &o, uint64_t i0, double *out,
                                                Terms &&terms) {
  double acc[N];
  for (int k = 0; k < N; ++k) acc[k] = 0;
  for (uint64_t at = i0; at < nv; at += kRefineThreads * kRefineAhead) {
    bool use[kRefineAhead];
    double wi[kRefineAhead], p[kRefineAhead][3], q[kRefineAhead][3];
#pragma unroll
    for (int k = 0; k < kRefineAhead; ++k) {
      const uint64_t i = at + uint64_t(k) * kRefineThreads;
      use[k] = i < nv && ok[i];
    }
#pragma unroll
    for (int k = 0; k < kRefineAhead; ++k) {
      if (!use[k]) continue;
      const uint64_t i = at + uint64_t(k) * kRefineThreads;
      wi[k] = w[i];
#pragma unroll
      for (int a = 0; a < 3; ++a) {
        if (P >> a & 1) p[k][a] = xyz[a * nv + i];
        if (Q >> a & 1) q[k][a] = target[i * 3 + a];
      }
    }
#pragma unroll
    for (int k = 0; k < kRefineAhead; ++k) {
      if (!use[k]) continue;
#pragma unroll
      for (int a = 0; a < 3; ++a)
        if (P >> a & 1) p[k][a] -= o.x[a];
      terms(acc, wi[k], p[k], q[k]);
    }
  }
  for (int k = 0; k < N; ++k) out[k * kRefineThreads] = acc[k];
}

// The weighted sums of mode c's correspondences (p the vertex, q its target,
// both relative to o; weights = vertex weights): W, W p, W q, W p q^T
// (row-major), W p p^T and W q q^T (upper triangles), as kRefineThreads
// fixed-order strided partials each; refine_solve adds them by a fixed tree.
// Bound by FP64 additions and products at 1/64 of the FP32 rate, so they are
// spread over the SMs: one-warp blocks (32 strides, one of kRefineGroups
// groups of three or four sums with a common factor, cluster).  16k vertices,
// 8 clusters: 56 us; one block per cluster took 318.
__global__ void __launch_bounds__(32) refine_sums(const double *xyz, const double *w, uint64_t nv,
                                                  const uint8_t *ok_all, const double *target_all,
                                                  Origin o, double *partial) {
  const uint64_t c = blockIdx.z;
  const unsigned stride0 = blockIdx.x * 32 + threadIdx.x;
  const uint8_t *ok = ok_all + c * nv;
  const double *target = target_all + c * nv * 3;
  double *out = partial + c * kRefineSums * kRefineThreads + stride0;
  auto sums_at = [&](int k) { return out + k * kRefineThreads; };
  // w x[A] (y0, y1, y2) into acc[0..2]
  auto row = [](double *acc, double wx, const double *y) {
    for (int e = 0; e < 3; ++e) acc[e] += wx * y[e];
  };
  switch (blockIdx.y) {
    case 0:
      refine_partials<7, 0, 4>(xyz, w, nv, ok, target, o, stride0, sums_at(0),
                               [&](double *acc, double wi, const double *p, const double *) {
                                 acc[0] += wi;
                                 for (int a = 0; a < 3; ++a) acc[1 + a] += wi * p[a];
                               });
      break;
    case 1:
      refine_partials<0, 7, 3>(xyz, w, nv, ok, target, o, stride0, sums_at(4),
                               [&](double *acc, double wi, const double *, const double *q) { row(acc, wi, q); });
      break;
    case 2:
      refine_partials<1, 7, 3>(xyz, w, nv, ok, target, o, stride0, sums_at(7),
                               [&](double *acc, double wi, const double *p, const double *q) { row(acc, wi * p[0], q); });
      break;
    case 3:
      refine_partials<2, 7, 3>(xyz, w, nv, ok, target, o, stride0, sums_at(10),
                               [&](double *acc, double wi, const double *p, const double *q) { row(acc, wi * p[1], q); });
      break;
    case 4:
      refine_partials<4, 7, 3>(xyz, w, nv, ok, target, o, stride0, sums_at(13),
                               [&](double *acc, double wi, const double *p, const double *q) { row(acc, wi * p[2], q); });
      break;
    case 5:
      refine_partials<7, 0, 3>(xyz, w, nv, ok, target, o, stride0, sums_at(16),
                               [&](double *acc, double wi, const double *p, const double *) { row(acc, wi * p[0], p); });
      break;
    case 6:
      refine_partials<6, 0, 3>(xyz, w, nv, ok, target, o, stride0, sums_at(19),
                               [&](double *acc, double wi, const double *p, const double *) {
                                 acc[0] += wi * p[1] * p[1], acc[1] += wi * p[1] * p[2], acc[2] += wi * p[2] * p[2];
                               });
      break;
    case 7:
      refine_partials<0, 7, 3>(xyz, w, nv, ok, target, o, stride0, sums_at(22),
                               [&](double *acc, double wi, const double *, const double *q) { row(acc, wi * q[0], q); });
      break;
    default:
      refine_partials<0, 6, 3>(xyz, w, nv, ok, target, o, stride0, sums_at(25),
                               [&](double *acc, double wi, const double *, const double *q) {
                                 acc[0] += wi * q[1] * q[1], acc[1] += wi * q[1] * q[2], acc[2] += wi * q[2] * q[2];
                               });
  }
}

// Eigen-decomposition of a symmetric 3x3 matrix (row-major) by cyclic
// Jacobi rotations: eigenvalues in `val`, eigenvectors in the columns of
// `vec`, sorted by decreasing eigenvalue.
__device__ void jacobi3(const double m[9], double val[3], double vec[9]) {
  double a[9];
  for (int k = 0; k < 9; ++k) a[k] = m[k], vec[k] = (k % 4 == 0) ? 1 : 0;
  for (int sweep = 0; sweep < 32; ++sweep) {
    const double off = a[1] * a[1] + a[2] * a[2] + a[5] * a[5];
    const double diag = a[0] * a[0] + a[4] * a[4] + a[8] * a[8];
    if (!(off > 1e-40 * diag)) break;
    for (int pi = 0; pi < 2; ++pi)
      for (int qi = pi + 1; qi < 3; ++qi) {
        const double apq = a[pi * 3 + qi];
        if (apq == 0) continue;
        // the rotation that zeroes a[p][q]: tan of its angle is the smaller
        // root of t^2 + 2 theta t - 1 = 0, theta = (a_qq - a_pp) / (2 a_pq)
        const double theta = (a[qi * 4] - a[pi * 4]) / (2 * apq);
        const double t = (theta >= 0 ? 1.0 : -1.0) / (fabs(theta) + sqrt(theta * theta + 1));
        const double cs = 1 / sqrt(t * t + 1), sn = t * cs;
        for (int k = 0; k < 3; ++k) {  // columns p, q of a
          const double akp = a[k * 3 + pi], akq = a[k * 3 + qi];
          a[k * 3 + pi] = cs * akp - sn * akq, a[k * 3 + qi] = sn * akp + cs * akq;
        }
        for (int k = 0; k < 3; ++k) {  // rows p, q
          const double apk = a[pi * 3 + k], aqk = a[qi * 3 + k];
          a[pi * 3 + k] = cs * apk - sn * aqk, a[qi * 3 + k] = sn * apk + cs * aqk;
        }
        for (int k = 0; k < 3; ++k) {
          const double vkp = vec[k * 3 + pi], vkq = vec[k * 3 + qi];
          vec[k * 3 + pi] = cs * vkp - sn * vkq, vec[k * 3 + qi] = sn * vkp + cs * vkq;
        }
      }
  }
  for (int k = 0; k < 3; ++k) val[k] = a[k * 4];
  for (int i = 0; i < 2; ++i)  // sort the columns, largest first
    for (int j = 0; j < 2 - i; ++j)
      if (val[j] < val[j + 1]) {
        double tv = val[j];
        val[j] = val[j + 1], val[j + 1] = tv;
        for (int k = 0; k < 3; ++k) {
          double tc = vec[k * 3 + j];
          vec[k * 3 + j] = vec[k * 3 + j + 1], vec[k * 3 + j + 1] = tc;
        }
      }
}

// A block per mode adds the partials of refine_sums, one thread of it finds
// the least-squares motion of the correspondences.
// Rigid: the rotation R maximising tr(R H), H = sum w (p - pbar)(q - qbar)^T,
// from H's singular vectors (Kabsch: H = U S V^T, R = V diag(1, 1, d) U^T
// with d making det R = +1), t = qbar - R pbar.  Reflection: the plane
// normal is the top eigenvector of sum w (q - p)(q - p)^T (the displacements
// run along it), oriented like the previous one, and the plane passes
// through the weighted mean of the midpoints (p + q) / 2.  A mode with too
// few or degenerate correspondences keeps its motion.
__global__ void __launch_bounds__(kRefineThreads) refine_solve(const double *partial, Origin o,
                                                               ClusterMotion *motions) {
  __shared__ double part[kRefineSums][kRefineThreads];
  const uint64_t c = blockIdx.x;
  for (int k = 0; k < kRefineSums; ++k)
    part[k][threadIdx.x] = partial[(c * kRefineSums + k) * kRefineThreads + threadIdx.x];
  __syncthreads();
  for (int h = kRefineThreads / 2; h; h >>= 1) {
    if (int(threadIdx.x) < h)
      for (int k = 0; k < kRefineSums; ++k) part[k][threadIdx.x] += part[k][threadIdx.x + h];
    __syncthreads();
  }
  if (threadIdx.x) return;
  double s[kRefineSums];
  for (int k = 0; k < kRefineSums; ++k) s[k] = part[k][0];
  const double W = s[0];
  if (!(W > 0)) return;
  double pb[3], qb[3];
  for (int a = 0; a < 3; ++a) pb[a] = s[1 + a] / W, qb[a] = s[4 + a] / W;
  ClusterMotion &m = motions[c];
  if (!m.reflection) {
    double H[9], HtH[9], S2[3], V[9];
    for (int a = 0; a < 3; ++a)
      for (int e = 0; e < 3; ++e) H[a * 3 + e] = s[7 + a * 3 + e] / W - pb[a] * qb[e];
    for (int a = 0; a < 3; ++a)
      for (int e = 0; e < 3; ++e)
        HtH[a * 3 + e] = H[a] * H[e] + H[3 + a] * H[3 + e] + H[6 + a] * H[6 + e];
    jacobi3(HtH, S2, V);
    const double s0 = sqrt(fmax(S2[0], 0.0)), s1 = sqrt(fmax(S2[1], 0.0));
    if (!(s1 > 1e-9 * s0)) return;  // collinear correspondences: rotation undetermined
    double U[9];  // U_k = H V_k / s_k for k = 0, 1; U_2 = U_0 x U_1
    for (int k = 0; k < 2; ++k)
      for (int a = 0; a < 3; ++a)
        U[a * 3 + k] = (H[a * 3] * V[k] + H[a * 3 + 1] * V[3 + k] + H[a * 3 + 2] * V[6 + k]) /
                       (k ? s1 : s0);
    U[2] = U[3] * U[7] - U[6] * U[4];
    U[5] = U[6] * U[1] - U[0] * U[7];
    U[8] = U[0] * U[4] - U[3] * U[1];
    const double detv = V[0] * (V[4] * V[8] - V[5] * V[7]) - V[1] * (V[3] * V[8] - V[5] * V[6]) +
                        V[2] * (V[3] * V[7] - V[4] * V[6]);
    const double d[3] = {1, 1, detv < 0 ? -1.0 : 1.0};
    double R[9];
    for (int a = 0; a < 3; ++a)
      for (int e = 0; e < 3; ++e)
        R[a * 3 + e] = V[a * 3] * d[0] * U[e * 3] + V[a * 3 + 1] * d[1] * U[e * 3 + 1] +
                       V[a * 3 + 2] * d[2] * U[e * 3 + 2];
    for (int k = 0; k < 9; ++k) m.r[k] = R[k];
    for (int a = 0; a < 3; ++a) {
      double rp = 0;
      for (int e = 0; e < 3; ++e) rp += R[a * 3 + e] * (pb[e] + o.x[e]);
      m.t[a] = qb[a] + o.x[a] - rp;
    }
  } else {
    double C[9], val[3], V[9];
    const int up[3][3] = {{0, 1, 2}, {1, 3, 4}, {2, 4, 5}};  // upper-triangle slots
    for (int a = 0; a < 3; ++a)
      for (int e = 0; e < 3; ++e)
        C[a * 3 + e] = (s[22 + up[a][e]] - s[7 + a * 3 + e] - s[7 + e * 3 + a] + s[16 + up[a][e]]) / W;
    jacobi3(C, val, V);
    if (!(val[0] > 0)) return;
    double n[3] = {V[0], V[3], V[6]};
    const double len = sqrt(n[0] * n[0] + n[1] * n[1] + n[2] * n[2]);
    if (!(len > 0)) return;
    const double sgn = (n[0] * m.n[0] + n[1] * m.n[1] + n[2] * m.n[2]) < 0 ? -1.0 : 1.0;
    for (int a = 0; a < 3; ++a) n[a] *= sgn / len;
    double off = 0;
    for (int a = 0; a < 3; ++a) off -= n[a] * (0.5 * (pb[a] + qb[a]) + o.x[a]);
    for (int a = 0; a < 3; ++a) {
      m.n[a] = n[a];
      m.t[a] = -2 * off * n[a];
      for (int e = 0; e < 3; ++e) m.r[a * 3 + e] = (a == e ? 1.0 : 0.0) - 2 * n[a] * n[e];
    }
    m.offset = off;
  }
}

// patches[set] += 1 for every component root of the set.
__global__ void count_roots(int32_t *parent_all, uint64_t nv, uint64_t sets, unsigned *patches) {
  uint64_t k = uint64_t(blockIdx.x) * blockDim.x + threadIdx.x;
  if (k >= sets * nv) return;
  const uint64_t set = k / nv;
  int32_t *parent = parent_all + set * nv;
  const int32_t i = int32_t(k % nv);
  if (parent[i] >= 0 && find_root(parent, i) == i) atomicAdd(&patches[set], 1u);
}

}  // namespace

// Unit normal of every face, (b - a) x (c - a) normalised in FP64 as the
// reference's normal test forms it (src/cpu/verification.cpp:71-75), rounded
// to FP32.  Not usable when that FP64 normal is not accurate to well below
// an FP32 unit (|ab x ac| <= 1e-6 |ab| |ac|: its direction error is about
// 1e-16 / sin of the corner angle), and near the reference's cut-off of
// unit() (a cross product of norm <= 1e-14 becomes the zero vector, which
// fails the test): those faces leave their rows to the FP64 decisions.
// The FP32 record of the face (Face) goes with it: its corners, reciprocal
// squared edge lengths and, where the normal is usable, a bound on its edge
// lengths.
__global__ void lbvh_face_records(const double *xyz, uint64_t nv, const int32_t *faces, uint64_t nf,
                                  float4 *face, double *fn64) {
  const uint64_t f = uint64_t(blockIdx.x) * blockDim.x + threadIdx.x;
  if (f >= nf) return;
  D3 c[3];
  F3 k[3];
  for (int i = 0; i < 3; ++i) {
    const int32_t v = faces[i * nf + f];
    c[i] = D3{xyz[v], xyz[nv + v], xyz[2 * nv + v]};
    k[i] = F3{float(c[i].x), float(c[i].y), float(c[i].z)};
  }
  const D3 ab = c[1] - c[0], ac = c[2] - c[0], n = cross(ab, ac);
  const D3 u = unit(n);  // the normal test's expression (normal_agrees), once per face
  if (fn64) fn64[3 * f] = u.x, fn64[3 * f + 1] = u.y, fn64[3 * f + 2] = u.z;
  const double n2 = dot(n, n), l2 = dot(ab, ab) * dot(ac, ac);
  const bool usable = n2 > 1e-12 * l2 && n2 > 4e-28;
  float inv[3], longest = 0;
  for (int i = 0; i < 3; ++i) {
    const F3 e = k[(i + 1) % 3] - k[i];
    const float l = dotf(e, e);
    inv[i] = l > 0.f ? 1.f / l : 0.f;
    longest = fmaxf(longest, l);
  }
  for (int i = 0; i < 3; ++i) face[4 * f + i] = make_float4(k[i].x, k[i].y, k[i].z, inv[i]);
  face[4 * f + 3] = make_float4(float(u.x), float(u.y), float(u.z),
                                usable ? fmaxf(sqrtf(longest) * 1.0001f, 1e-30f) : 0.f);
}

// The FlatFace records: one thread per face, in FP64 (a face's quotients and
// square roots are some 150 FP64 operations, 0.2 ms for 1e6 faces, once per mesh).
__global__ void lbvh_flat_records(const double *xyz, uint64_t nv, const int32_t *faces, uint64_t nf,
                                  const float4 *face, float longest, float4 *flat) {
  const uint64_t f = uint64_t(blockIdx.x) * blockDim.x + threadIdx.x;
  if (f >= nf) return;
  D3 c[3];
  for (int i = 0; i < 3; ++i) {
    const int32_t v = faces[i * nf + f];
    c[i] = D3{xyz[v], xyz[nv + v], xyz[2 * nv + v]};
  }
  const D3 ab = c[1] - c[0], ac = c[2] - c[0], bc = c[2] - c[1];
  const double lab = norm(ab), lbc = norm(bc), lca = norm(ac);
  const D3 n = unit(cross(ab, ac)), e = div(ab, lab), m = cross(n, e);
  const float4 normal = face[4 * f + 3];
  const bool plain = normal.w <= longest && fmin(lab, fmin(lbc, lca)) > 1e-15 && fmax(lab, fmax(lbc, lca)) < 1e15;
  const float reach = plain ? normal.w : -normal.w;
  flat[4 * f] = make_float4(float(c[0].x), float(c[0].y), float(c[0].z), float(lab));
  flat[4 * f + 1] = make_float4(float(n.x), float(n.y), float(n.z), float(dot(ac, e)));
  flat[4 * f + 2] = make_float4(float(e.x), float(e.y), float(e.z), float(dot(ac, m)));
  flat[4 * f + 3] = make_float4(float(1.0 / lab), float(1.0 / lbc), float(1.0 / lca), reach);
}

Lbvh lbvh_build(Call &call, const double *xyz, const double *vn, uint64_t nv,
                const int32_t *faces, uint64_t nf) {
  Lbvh b;
  b.nv = nv, b.nf = nf, b.faces = faces;
  if (!nf) return b;
  cudaStream_t st = call.stream();
  const uint64_t ni = nf - 1;
  auto pad = [](uint64_t x) { return (x + 255) & ~uint64_t(255); };
  const uint64_t s_xyz = pad(12 * nv), s_node = pad(4 * kNodeWords * (ni + 1)),
                 s_face = pad(64 * nf), s_order = pad(4 * nv), s_fn64 = pad(24 * nf);
  SYM_CUDA(cudaMalloc(&b.block, 2 * s_xyz + s_node + 2 * s_face + s_order + s_fn64));
  char *at = b.block;
  auto take = [&](uint64_t bytes) {
    char *r = at;
    at += bytes;
    return r;
  };
  b.node = reinterpret_cast<float4 *>(take(s_node));
  b.face = reinterpret_cast<float4 *>(take(s_face));
  b.flat = reinterpret_cast<float4 *>(take(s_face));
  b.xyz = reinterpret_cast<float *>(take(s_xyz));
  b.vn = reinterpret_cast<float *>(take(s_xyz));
  b.order = reinterpret_cast<int32_t *>(take(s_order));
  b.fn64 = reinterpret_cast<double *>(take(s_fn64));
  lbvh_vertices<<<blocks_for(3 * nv), kThreads, 0, st>>>(xyz, nv, b.xyz);
  check_launch();
  lbvh_vertices<<<blocks_for(3 * nv), kThreads, 0, st>>>(vn, nv, b.vn);
  check_launch();
  lbvh_face_records<<<blocks_for(nf), kThreads, 0, st>>>(xyz, nv, faces, nf, b.face, b.fn64);
  check_launch();
  // the mesh box, for the Morton quantisation
  std::vector<float> h(3 * nv);
  SYM_CUDA(cudaMemcpyAsync(h.data(), b.xyz, 12 * nv, cudaMemcpyDeviceToHost, st));
  call.sync();
  float lo[3], hi[3];
  for (int a = 0; a < 3; ++a) {
    auto mm = std::minmax_element(h.begin() + a * nv, h.begin() + (a + 1) * nv);
    lo[a] = *mm.first, hi[a] = *mm.second;
  }
  float ext = std::max({hi[0] - lo[0], hi[1] - lo[1], hi[2] - lo[2], 1e-30f});
  for (int a = 0; a < 3; ++a) b.scale = std::max({b.scale, std::fabs(lo[a]), std::fabs(hi[a])});
  lbvh_flat_records<<<blocks_for(nf), kThreads, 0, st>>>(xyz, nv, faces, nf, b.face, 0.25f * b.scale, b.flat);
  check_launch();
  call.launched();
  uint64_t *keys = call.alloc<uint64_t>(nf), *skeys = call.alloc<uint64_t>(nf);
  int32_t *ids = call.alloc<int32_t>(nf), *sids = call.alloc<int32_t>(nf);
  lbvh_keys<<<blocks_for(nf), kThreads, 0, st>>>(b.xyz, nv, faces, nf, make_float3(lo[0], lo[1], lo[2]),
                                                 make_float3(1 / ext, 1 / ext, 1 / ext), keys, ids);
  check_launch();
  // the keys arrive in the order of their low halves, the ids: the codes alone are sorted
  radix_sort_pairs(call, keys, ids, skeys, sids, nf, 62, 32);
  {  // the query order of the verification: neighbouring vertices in a warp
    uint64_t *vkeys = call.alloc<uint64_t>(nv), *svkeys = call.alloc<uint64_t>(nv);
    int32_t *vids = call.alloc<int32_t>(nv);
    lbvh_vertex_keys<<<blocks_for(nv), kThreads, 0, st>>>(
        b.xyz, nv, make_float3(lo[0], lo[1], lo[2]), make_float3(1 / ext, 1 / ext, 1 / ext), vkeys,
        vids);
    check_launch();
    call.launched();
    radix_sort_pairs(call, vkeys, vids, svkeys, b.order, nv, 62, 32);
  }
  if (ni) {
    int32_t *parent_in = call.alloc<int32_t>(ni), *parent_leaf = call.alloc<int32_t>(nf);
    unsigned *arrivals = call.alloc<unsigned>(ni);
    SYM_CUDA(cudaMemsetAsync(arrivals, 0, 4 * ni, st));
    int32_t *nodes = reinterpret_cast<int32_t *>(b.node);
    lbvh_internal<<<blocks_for(ni), kThreads, 0, st>>>(skeys, int64_t(nf), nodes, parent_in,
                                                        parent_leaf);
    check_launch();
    lbvh_boxes<<<blocks_for(nf), kThreads, 0, st>>>(b.xyz, nv, faces, int64_t(nf), sids, nodes,
                                                     parent_in, parent_leaf, arrivals);
    check_launch();
  }
  call.launched(ni ? 8 : 6);
  call.sync();
  return b;
}

void lbvh_free(Lbvh &b) {
  if (b.block) cudaFree(b.block);
  b = Lbvh{};
}

namespace {

BvhView view_of(const Lbvh &b) {
  return {b.nv, b.nf, b.faces, b.xyz, b.node, b.face, b.flat, b.order, b.fn64};
}

// `refine` passes of FP64 least-squares refinement of the nc modes' motions
// against the mesh (ICP: forward correspondences under the current motion,
// then the motion that fits them best), on the device; dm is updated in
// place.  `origin` (a point near the mesh) keeps the sums well conditioned.
void refine_motions(Call &call, const BvhView &view, const double *xyz, const double *vn,
                    const double *w, ClusterMotion *dm, uint64_t nc, double tau, int refine,
                    const double origin[3]) {
  const uint64_t nv = view.nv;
  if (refine <= 0 || !nc || !nv || !view.nf) return;
  cudaStream_t st = call.stream();
  const Origin o{{origin[0], origin[1], origin[2]}};
  double *target = call.alloc<double>(nc * nv * 3);
  double *partial = call.alloc<double>(nc * kRefineSums * kRefineThreads);
  uint8_t *ok = call.alloc<uint8_t>(nc * nv);
  for (int it = 0; it < refine; ++it) {
    refine_pairs<<<blocks_for(nc * nv), kThreads, 0, st>>>(view, xyz, vn, dm, nc, tau,
                                                           float(tau * tau), o, target, ok,
                                                           call.status());
    check_launch();
    refine_sums<<<dim3(kRefineThreads / 32, kRefineGroups, unsigned(nc)), 32, 0, st>>>(
        xyz, w, nv, ok, target, o, partial);
    check_launch();
    refine_solve<<<unsigned(nc), kRefineThreads, 0, st>>>(partial, o, dm);
    check_launch();
    call.launched(3);
  }
}

void store_motion(const ClusterMotion &m, sym_cluster_record &r) {
  for (int k = 0; k < 9; ++k) r.rotation[k] = m.r[k];
  for (int k = 0; k < 3; ++k) r.translation[k] = m.t[k], r.plane_normal[k] = m.n[k];
  r.plane_offset = m.offset;
}

}  // namespace

// The reference-order BVH of a resident mesh on the device: the build the
// mesh's load started on a host thread, or, without one, a build from the
// device's vertices and faces.
void ensure_ref_bvh(Call &call, const ResidentSurface &m) {
  RefBvhSource &src = *m.ref;
  if (src.dev.block) return;
  std::unique_ptr<HostBvh> bvh;
  if (src.pending.valid()) {
    bvh = src.pending.get();
  } else {
    std::vector<double> x(3 * m.nv);
    std::vector<int32_t> f(3 * m.nf);
    call.d2h(x.data(), m.xyz, 24 * m.nv);
    call.d2h(f.data(), m.faces, 12 * m.nf);
    call.sync();
    const sym_mesh_view mv{{x.data(), x.data() + m.nv, x.data() + 2 * m.nv, m.nv},
                           {f.data(), f.data() + m.nf, f.data() + 2 * m.nf, m.nf}};
    bvh = std::make_unique<HostBvh>(mv);
  }
  if (2 * bvh->depth + 4 > kRefStack) fail(SYM_RUNTIME_ERROR, "verification: BVH too deep");
  src.dev = ref_bvh_upload(*bvh, call.stream());
}

uint64_t exact_flags(Call &call, const ResidentSurface &m, const ClusterMotion *dm,
                     const sym_cluster_record *records, uint64_t nc, double tau, uint8_t *flags,
                     double *err, uint64_t *fp64_rows) {
  const uint64_t nv = m.nv, rows = nc * 2 * nv;
  cudaStream_t st = call.stream();
  if (fp64_rows) *fp64_rows = 0;
  if (!rows) return 0;
  if (rows >= (uint64_t(1) << 31)) fail(SYM_INVALID_ARGUMENT, "verification: too many queries");
  if (!m.nf) {
    SYM_CUDA(cudaMemsetAsync(flags, 0, rows, st));
    SYM_CUDA(cudaMemsetAsync(err, 0, nc * nv * 8, st));
    return 0;
  }
  const Lbvh &bvh = *m.lbvh;
  std::vector<MotionF> mf(nc);
  for (uint64_t c = 0; c < nc; ++c) mf[c] = motion32(records[c]);
  const MotionF *dmf = call.upload(mf.data(), nc);
  RowLists lists;
  lists.forward = call.alloc<uint32_t>(nc * nv);
  lists.faces = call.alloc<int32_t>(nc * nv * kCandidates);
  lists.mark = call.alloc<uint8_t>(rows);
  lists.fp64 = call.alloc<int32_t>(rows);
  lists.reference = call.alloc<int32_t>(rows);
  lists.slot_of = call.alloc<uint32_t>(rows);
  lists.slots = std::min<uint64_t>(rows, uint64_t(1) << 24);  // at most 1 GiB of candidates
  lists.cand = call.alloc<int32_t>(lists.slots * kCandidates);
  lists.counts = call.alloc<unsigned long long>(5);
  lists.capacity = rows;
  uint64_t *listed = call.alloc<uint64_t>(2);
  SYM_CUDA(cudaMemsetAsync(lists.counts, 0, 40, st));
  const BvhView view = view_of(bvh);
  Surface s{m.xyz, nv, m.faces, m.nf, nullptr, nullptr};
  verify_fp32<<<blocks_for(rows), kThreads, 0, st>>>(view, bvh.vn, dmf, nc, float(tau), bvh.scale,
                                                      flags, err, lists, call.status());
  check_launch();
  compact_indices(call, lists.mark, rows, lists.fp64, listed);
  unsigned long long counts[4] = {0, 0, 0, 0};
  call.d2h(counts, lists.counts, 8);
  call.d2h(&counts[1], listed, 8);
  call.sync();
  call.launched();
  if (counts[0]) {
    forward_errors<<<blocks_for(counts[0], kRowThreads), kRowThreads, 0, st>>>(view, s, dm, lists, counts[0],
                                                                             bvh.scale, float(tau), err);
    check_launch();
    call.launched();
  }
  if (counts[1]) {
    ensure_ref_bvh(call, m);
    s.nodes = m.ref->dev.nodes, s.ids = m.ref->dev.ids;
    lists.open = lists.reference;  // free until the next compaction
    verify_rows_fp64<<<blocks_for(counts[1]), kThreads, 0, st>>>(view, s, m.ref->dev, m.vn, bvh.vn, dm, dmf, tau,
                                                                 bvh.scale, flags, err, lists, counts[1]);
    check_launch();
    verify_rows_open<<<unsigned(std::min<uint64_t>(blocks_for(counts[1] + kRowThreads, kRowThreads), 152 * 8)),
                       kRowThreads, 0, st>>>(view, s, m.ref->dev, m.vn, bvh.vn, dm, dmf, tau, bvh.scale, flags,
                                             err, lists, call.status());
    check_launch();
    call.launched(2);
    compact_indices(call, lists.mark, rows, lists.reference, listed + 1);
    call.d2h(&counts[2], listed + 1, 8);
    call.d2h(&counts[3], lists.counts + 3, 8);
    call.sync();
    if (counts[2]) {  // overflowed lists: the wider list first
      verify_rows_wide<<<blocks_for(counts[2]), kThreads, 0, st>>>(
          view, s, m.ref->dev, m.vn, dm, tau, bvh.scale, flags, err, lists, counts[2],
          call.status());
      check_launch();
      call.launched();
      compact_indices(call, lists.mark, rows, lists.reference, listed + 1);
      call.d2h(&counts[2], listed + 1, 8);
      call.d2h(&counts[3], lists.counts + 3, 8);
      call.sync();
    }
  }
  if (fp64_rows) *fp64_rows = counts[1];
  if (counts[2]) {
    verify_listed_ref<<<blocks_for(counts[2]), kThreads, 0, st>>>(s, m.vn, bvh.order, dm, tau,
                                                                   lists, counts[2], flags, err,
                                                                   call.status());
    check_launch();
    call.launched();
  }
  return counts[2] + counts[3];
}

// Coverage, rms and patch counts of the nc modes (sym_detect_fast), after
// `refine` FP64 refinement passes of their motions (written back to
// records); the same coverage, rms and patches as the reference's
// verification of the records.
void verification_fast(Call &call, const ResidentSurface &m, sym_cluster_record *records,
                       uint64_t nc, double tau, int refine, const double origin[3],
                       double *coverage, double *rms, uint32_t *patches, uint64_t *undecided,
                       uint64_t *fp64_rows) {
  const uint64_t nv = m.nv;
  if (undecided) *undecided = 0;
  if (fp64_rows) *fp64_rows = 0;
  if (!nc || !nv) {
    for (uint64_t c = 0; c < nc; ++c) coverage[c] = rms[c] = 0, patches[2 * c] = patches[2 * c + 1] = 0;
    return;
  }
  cudaStream_t st = call.stream();
  std::vector<ClusterMotion> motions(nc);
  for (uint64_t c = 0; c < nc; ++c) motions[c] = cluster_motion(records[c]);
  ClusterMotion *dm = call.upload(motions.data(), nc);
  if (refine > 0 && m.nf) {
    const Lbvh &bvh = *m.lbvh;
    const BvhView view = view_of(bvh);
    refine_motions(call, view, m.xyz, m.vn, m.w, dm, nc, tau, refine, origin);
    call.d2h(motions.data(), dm, nc * sizeof(ClusterMotion));
    call.check_status("transform refinement");
    for (uint64_t c = 0; c < nc; ++c) store_motion(motions[c], records[c]);
  }
  const uint64_t rows = nc * 2 * nv;
  uint8_t *flags = call.alloc<uint8_t>(rows);
  double *err = call.alloc<double>(nc * nv);
  const uint64_t n = exact_flags(call, m, dm, records, nc, tau, flags, err, fp64_rows);
  if (undecided) *undecided = n;
  double *error = call.alloc<double>(nc), *area = call.alloc<double>(nc), *total = call.alloc<double>(1);
  uint64_t *na = call.alloc<uint64_t>(nc);
  double *partial = call.alloc<double>((nc + 1) * 2 * kTreeThreads);
  unsigned *partial_count = call.alloc<unsigned>((nc + 1) * kTreeThreads);
  tree_partials<<<dim3(kTreeThreads / 32, 2, unsigned(nc + 1)), 32, 0, st>>>(flags, err, m.w, nv, nc,
                                                                            partial, partial_count);
  check_launch();
  tree_sums<<<unsigned(nc + 1), kTreeThreads, 0, st>>>(partial, partial_count, nc, error, area, na, total);
  check_launch();
  call.launched(2);
  int32_t *parent = call.alloc<int32_t>(rows);
  unsigned *dpatch = call.alloc<unsigned>(2 * nc);
  SYM_CUDA(cudaMemsetAsync(dpatch, 0, 8 * nc, st));
  init_parents<<<blocks_for(rows), kThreads, 0, st>>>(flags, rows, parent, nv);
  check_launch();
  unite_edges<<<blocks_for(rows), kThreads, 0, st>>>(m.nbr_off, m.nbr, nv, 2 * nc, parent,
                                                      call.status(), kUniteRetries);
  check_launch();
  count_roots<<<blocks_for(rows), kThreads, 0, st>>>(parent, nv, 2 * nc, dpatch);
  check_launch();
  call.launched(3);
  std::vector<double> herr(nc), harea(nc);
  std::vector<uint64_t> hna(nc);
  std::vector<unsigned> hp(2 * nc);
  double htotal = 0;
  call.d2h(herr.data(), error, nc * 8);
  call.d2h(harea.data(), area, nc * 8);
  call.d2h(hna.data(), na, nc * 8);
  call.d2h(&htotal, total, 8);
  call.d2h(hp.data(), dpatch, 8 * nc);
  call.check_status("verification");
  for (uint64_t c = 0; c < nc; ++c) {
    rms[c] = hna[c] ? std::sqrt(herr[c] / double(hna[c])) : 0;
    coverage[c] = htotal > 0 ? std::min(1.0, harea[c] / htotal) : 0;
    patches[2 * c] = hp[2 * c], patches[2 * c + 1] = hp[2 * c + 1];
  }
}

// The reference's verification of `records` on a resident mesh: side
// lists, patches, coverage and rms identical to verification_core's.
void verification_resident(Call &call, const ResidentSurface &m, const sym_cluster_record *records,
                           uint64_t nc, double tau, sym_verification_result &out,
                           void *(*allocate)(size_t), uint64_t *undecided) {
  const uint64_t nv = m.nv;
  if (undecided) *undecided = 0;
  uint8_t *flags = nullptr;
  double *err = nullptr;
  if (nc) {
    std::vector<ClusterMotion> motions(nc);
    for (uint64_t c = 0; c < nc; ++c) motions[c] = cluster_motion(records[c]);
    ClusterMotion *dm = call.upload(motions.data(), nc);
    flags = call.alloc<uint8_t>(nc * 2 * nv);
    err = call.alloc<double>(nc * nv);
    const uint64_t n = exact_flags(call, m, dm, records, nc, tau, flags, err, nullptr);
    if (undecided) *undecided = n;
  }
  finish_verification(call, flags, err, m.w, m.nbr_off, m.nbr, nv, nc, out, allocate);
}

}  // namespace sym
