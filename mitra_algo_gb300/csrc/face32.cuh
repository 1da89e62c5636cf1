// SPDX-License-Identifier: MPL-2.0
// A mesh face in FP32 as the closest-point searches read it, and how far an
// FP32 distance to it can be trusted: shared by the exact verification
// (verification.cu), which skips faces by it, and the throughput one
// (verify_fast.cu), which decides by it.  Both units are compiled without FMA
// contraction.
#pragma once
#include "verification.cuh"

namespace sym {

struct F3 {
  float x, y, z;
};
__device__ __forceinline__ F3 operator-(F3 a, F3 b) { return {a.x - b.x, a.y - b.y, a.z - b.z}; }
__device__ __forceinline__ F3 operator+(F3 a, F3 b) { return {a.x + b.x, a.y + b.y, a.z + b.z}; }
__device__ __forceinline__ F3 operator*(F3 a, float s) { return {a.x * s, a.y * s, a.z * s}; }
__device__ __forceinline__ float dotf(F3 a, F3 b) { return a.x * b.x + a.y * b.y + a.z * b.z; }
__device__ __forceinline__ F3 crossf(F3 a, F3 b) {
  return {a.y * b.z - a.z * b.y, a.z * b.x - a.x * b.z, a.x * b.y - a.y * b.x};
}

// A face as the searches read it, 64 bytes: corners a, b, c in FP32, the
// reciprocal squared lengths of the edges ab, bc, ca, the unit normal from the
// FP64 corners and `reach`, a bound on the edge lengths (0: no usable normal).
struct Face {
  F3 a, b, c, n;
  float inv_ab, inv_bc, inv_ca, reach;
};

__device__ __forceinline__ Face load_face(const float4 *faces, int32_t f) {
  const float4 *r = faces + 4 * int64_t(f);
  const float4 x = r[0], y = r[1], z = r[2], w = r[3];
  return {{x.x, x.y, x.z}, {y.x, y.y, y.z}, {z.x, z.y, z.z}, {w.x, w.y, w.z}, x.w, y.w, z.w, w.w};
}

// FP32 unit roundoff, of which the bounds below count multiples (u M: at the
// largest coordinate magnitude M of the mesh and the image).
constexpr float kUnit = 1.0f / 16777216.0f;

// FP32 squared distance from p to a face with a usable normal; um = u M, the
// FP32 unit at the query's magnitude.  The plane distance when p projects
// inside all three edges by more than their rounding band (p then projects
// into the face), the nearest of the edge segments when it projects outside
// one of them by more than its band (the nearest point then lies on an edge p
// is outside of, so edges p is inside of by more than the band need no
// distance).  Otherwise `d2` receives min(plane, segments), a lower bound of
// the distance, and the function returns false; also, with the plane
// distance, when that alone is above `lim` (the caller drops the face).
// Band of an edge function E = (n x e) . (p - v): with |dn| <= u,
// corners within 1.8 u M and the image within 30 u M of their FP64 values,
// and the cross and dot products' rounding, |dE| <= u (11 |e| |p - v| +
// 3.6 M |p - v| + 32 M |e|) <= 42 u M (|p - v| + |e|) for |e| <= 3.5 M; one
// band serves the three, 64 u M (|p - a|_1 + 2 reach) with |p - v| <= |p - a| +
// reach and |e| <= reach (a band too wide only leaves more to FP64): six
// square roots and three divisions fewer per face than bands and segments of
// their own.
// Error of a decided distance, in u M, with I the image's own (30 for one made in
// FP32, 1.8 for one rounded from FP64), corners 1.8, and |p - v| and |e| at most
// 3.5 M.  The plane distance: normal, difference and dot product 5 x 3.5, so I +
// 19.3 either way.  A segment: its rounded differences are the exact ones of a
// point and an end moved by 3.5 each, and with 3.5 for e t the distance is I +
// 12.3 off either way; its foot, off by u (3 |p - v| + 5 |e|), only lengthens it,
// by up to 28.  The last subtraction, the square and the root add 1.5 to 2.5 u of
// the distance itself.  With I = 30 and distances up to 0.6 M (M is at least 2 tau)
// that is at most 73 too long and 51 too short: of two faces the nearer one in
// FP64 is never 128 u M farther here.  With I = 1.8 and any distance it is
// at most 52 too long and 30 too short.
__device__ __forceinline__ bool face_d2n(F3 p, const Face &f, float um, float lim, float &d2) {
  const F3 ap = p - f.a;
  const float h = dotf(f.n, ap), h2 = h * h;
  d2 = h2;
  if (h2 > lim) return false;
  const F3 ab = f.b - f.a, bc = f.c - f.b, ca = f.a - f.c, bp = p - f.b, cp = p - f.c;
  const float band = 64.f * um * (fabsf(ap.x) + fabsf(ap.y) + fabsf(ap.z) + 2.f * f.reach);
  const float ea = dotf(crossf(f.n, ab), ap), eb = dotf(crossf(f.n, bc), bp),
              ec = dotf(crossf(f.n, ca), cp);
  const float least = fminf(ea, fminf(eb, ec));
  if (least > band) return true;  // inside
  float seg = INFINITY;
  auto segment = [&](F3 q, F3 e, float inv) {
    const float t = __saturatef(dotf(q, e) * inv);
    const F3 r = q - e * t;
    seg = fminf(seg, dotf(r, r));
  };
  if (ea <= band) segment(ap, ab, f.inv_ab);
  if (eb <= band) segment(bp, bc, f.inv_bc);
  if (ec <= band) segment(cp, ca, f.inv_ca);
  if (least < -band) {
    d2 = seg;
    return true;
  }
  d2 = fminf(h2, seg);
  return false;
}

// The faces' records, and with `fn64` not null their FP64 unit normals.
__global__ void lbvh_face_records(const double *xyz, uint64_t nv, const int32_t *faces, uint64_t nf,
                                  float4 *face, double *fn64);

}  // namespace sym
