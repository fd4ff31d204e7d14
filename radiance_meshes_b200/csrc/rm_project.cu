// Stage 1 on the GPU: per-tet projection, near-plane clipping, planar/behind
// culling, fp64 circumsphere power (the sort depth), tile rectangle and tile
// count; plus its reverse pass with respect to the vertices.
//
// This translation unit is compiled with -fmad=false: the tile rectangles and
// the sort depth decide the tile lists, which must be bit-identical to the CPU
// restatement of the reference arithmetic, so every fp32/fp64 operation here is
// the plain IEEE operation in the order written.
//
// Reference behaviour reproduced: slang/vertex_shader.slang:20-89,
// slang/camera.slang:103-108,351-508, slang/intersect.slang:76-89,
// slang/stable_power.slang:17-84, slang/utils.slang:85-125.

#include <climits>

#include "rm_common.cuh"

namespace rm {

__device__ __forceinline__ float safe_clipf(float v, float lo, float hi) { return fmaxf(fminf(v, hi), lo); }
__device__ __forceinline__ float safe_divf(float a, float b) {
  const float TINY = 1.0754944e-20f;
  if (fabsf(b) < TINY) return safe_clipf(a / TINY, -1e20f, 1e20f);
  return safe_clipf(a / b, -1e20f, 1e20f);
}
__device__ __forceinline__ f3 normalize3(f3 a) {
  float l = sqrtf(dot(a, a));
  return {a.x / l, a.y / l, a.z / l};
}
__device__ __forceinline__ f3 lerp3(f3 a, f3 b, float t) { return a + (b - a) * t; }

__device__ __forceinline__ float dist_norm2(const DevCam& c) {
  return c.dist[0] * c.dist[0] + c.dist[1] * c.dist[1] + c.dist[2] * c.dist[2] + c.dist[3] * c.dist[3];
}

__device__ __forceinline__ f3 point2camspace(f3 p, const DevCam& c) {
  float h[4];
#pragma unroll
  for (int i = 0; i < 4; ++i)
    h[i] = c.W[4 * i + 0] * p.x + c.W[4 * i + 1] * p.y + c.W[4 * i + 2] * p.z + c.W[4 * i + 3] * 1.0f;
  // A rigid world-to-camera transform has the last row (0, 0, 0, 1): w is exactly 1 and x / 1 is x, so
  // the three guarded divisions reduce to the clip (same bits, far fewer instructions).
  if (h[3] == 1.0f) return {safe_clipf(h[0], -1e20f, 1e20f), safe_clipf(h[1], -1e20f, 1e20f), safe_clipf(h[2], -1e20f, 1e20f)};
  return {safe_divf(h[0], h[3]), safe_divf(h[1], h[3]), safe_divf(h[2], h[3])};
}

__device__ __forceinline__ void distort(float& x, float& y, const DevCam& c) {
  if (dist_norm2(c) < 1e-9f) return;
  float k1 = c.dist[0], k2 = c.dist[1], p1 = c.dist[2], p2 = c.dist[3];
  float r2 = x * x + y * y;
  float radial = r2 * (k1 + r2 * k2);
  float tx = 2.0f * p1 * x * y + p2 * (r2 + 2.0f * x * x);
  float ty = 2.0f * p2 * x * y + p1 * (r2 + 2.0f * y * y);
  float nx = x + x * radial + tx;
  float ny = y + y * radial + ty;
  x = nx;
  y = ny;
}

// Fisheye angle functions with a fixed operation sequence (IEEE double, no contraction), so
// that tile rectangles of fisheye cameras are reproducible bit for bit by any implementation
// that evaluates the same series; the result is rounded to float once.  Library acosf/sinf
// differ between vendors in the last bit.
//   asin(s) = sum_n c_n s^(2n+1), c_0 = 1, c_{n+1} = c_n (2n+1)^2 / ((2n+2)(2n+3)), |s| <= 0.5
//   acos(x) = pi/2 - asin(x) for x < 0.5, 2 asin(sqrt((1 - x)/2)) otherwise        (0 <= x <= 1)
//   sin(t)  = sum_n (-1)^n t^(2n+1)/(2n+1)!,                                        0 <= t <= pi/2
// Both loops are unrolled so that the coefficients are constants: as written in a rolled loop, the 32
// IEEE double divisions of one projection were most of the kernel's time (1M tets, 720 x 720: 2.38 ms).
__device__ __forceinline__ double asin_series(double s) {
  const double s2 = s * s;
  double term = s, sum = s;
#pragma unroll
  for (int n = 0; n < 20; ++n) {
    const double a = double(2 * n + 1);
    term = term * s2 * (a * a / (double(2 * n + 2) * double(2 * n + 3)));
    sum += term;
  }
  return sum;
}
__device__ __forceinline__ float fisheye_acos(float x) {
  const double xd = double(x);
  const bool low = xd < 0.5;
  const double a = asin_series(low ? xd : sqrt((1.0 - xd) * 0.5));
  return float(low ? 1.5707963267948966 - a : 2.0 * a);
}
// x / d for a constant d, rounded as the division rounds: quotient from the correctly rounded reciprocal,
// then one correction with the exact remainder (Markstein, "Computation of elementary functions on the IBM
// RISC System/6000 processor", 1990).  Checked against the division on 3.6e8 random dividends of the twelve
// divisors below; a term so small that the remainder is not exact is far below half an ulp of the sum.
__device__ __forceinline__ double div_by_constant(double x, double d, double reciprocal) {
  const double q = x * reciprocal;
  return fma(fma(-q, d, x), reciprocal, q);
}
__device__ __forceinline__ float fisheye_sin(float t) {
  const double td = double(t), t2 = td * td;
  double term = td, sum = td;
#pragma unroll
  for (int n = 1; n < 13; ++n) {
    const double d = double(2 * n) * double(2 * n + 1);
    term = div_by_constant(-(term * t2), d, 1.0 / d);
    sum += term;
  }
  return float(sum);
}

// theta / sin(theta) for z = cos(theta) in [0, 1], to 1e-6: acos(z) = sqrt(1 - z) P(z) with the polynomial of
// Abramowitz and Stegun 4.4.46, so the quotient is P(z) / sqrt(1 + z), smooth up to the axis.
__device__ __forceinline__ float fisheye_ratio_estimate(float z) {
  float p = -0.0012624911f;
  p = fmaf(p, z, 0.0066700901f);
  p = fmaf(p, z, -0.0170881256f);
  p = fmaf(p, z, 0.0308918810f);
  p = fmaf(p, z, -0.0501743046f);
  p = fmaf(p, z, 0.0889789874f);
  p = fmaf(p, z, -0.2145988016f);
  p = fmaf(p, z, 1.5707963050f);
  return p * rsqrtf(1.0f + z);
}

template <bool FISHEYE>
__device__ __forceinline__ f3 camspace_to_image(f3 p, const DevCam& c) {
  float ux, uy;
  if (FISHEYE) {
    f3 dir = normalize3(p);
    float sat = fminf(fmaxf(dir.z, 0.0f), 1.0f);
    float theta = fisheye_acos(sat);
    float st = fisheye_sin(theta);
    float k = (st < 1e-6f) ? 1.0f : theta / st;
    ux = dir.x * k;
    uy = dir.y * k;
  } else {
    ux = p.x / p.z;
    uy = p.y / p.z;
  }
  distort(ux, uy, c);
  float px = ux * c.K[0] + c.K[2];
  float py = uy * c.K[4] + c.K[5];
  return {px, py, p.z};
}

// samples per edge of the extent search
__device__ __forceinline__ int edge_samples(const DevCam& c) {
  return c.type == 1 ? 4 : (dist_norm2(c) > 1e-9f ? 3 : 2);
}

// Bounds of the projected samples.  FISHEYE: a sample that an estimate puts inside the bounds by more than the
// estimate's error (1e-6 of the ratio and a few roundings, against 0.01 pixel + 1e-5 of the focal length) leaves
// them as they are; its projection, two double series, is not evaluated.  Most samples between the ends of an
// edge are of that kind.
template <bool FISHEYE>
__device__ __forceinline__ void add_sample(f3 s, f3& mn, f3& mx, const DevCam& c) {
  if (FISHEYE && dist_norm2(c) < 1e-9f) {
    const float inv = rsqrtf(s.x * s.x + s.y * s.y + s.z * s.z);
    const float k = inv * fisheye_ratio_estimate(fminf(fmaxf(s.z * inv, 0.0f), 1.0f));
    const float px = fmaf(s.x * k, c.K[0], c.K[2]), py = fmaf(s.y * k, c.K[4], c.K[5]);
    const float ex = 0.01f + 1e-5f * (fabsf(c.K[0]) + fabsf(c.K[2])), ey = 0.01f + 1e-5f * (fabsf(c.K[4]) + fabsf(c.K[5]));
    if (px > mn.x + ex && px < mx.x - ex && py > mn.y + ey && py < mx.y - ey && s.z <= mx.z) return;
  }
  const f3 pv = camspace_to_image<FISHEYE>(s, c);
  mn = {fminf(mn.x, pv.x), fminf(mn.y, pv.y), fminf(mn.z, pv.z)};
  mx = {fmaxf(mx.x, pv.x), fmaxf(mx.y, pv.y), fmaxf(mx.z, pv.z)};
}

template <bool FISHEYE>
__device__ __forceinline__ void update_bounds_from_edge(f3 a, f3 b, f3& mn, f3& mx, const DevCam& c) {
  const int n = edge_samples(c);
  for (int i = 0; i < n; ++i) {
    float t = float(i) / float(n - 1);
    add_sample<FISHEYE>(lerp3(a, b, t), mn, mx, c);
  }
}

// Bounds of a tet's face f, clipped against the near plane; the tet's are those of its four faces together.
template <bool FISHEYE>
__device__ __forceinline__ void extent_of_face(const f3 tet[4], int f, f3& mn, f3& mx, const DevCam& c) {
  const float eps = 1e-4f;
  // faces (0,1,2) (0,2,3) (0,3,1) (1,3,2)
  const f3 fv[3] = {f == 3 ? tet[1] : tet[0], f == 0 ? tet[1] : (f == 1 ? tet[2] : tet[3]),
                    f == 0 ? tet[2] : (f == 1 ? tet[3] : (f == 2 ? tet[1] : tet[2]))};
  f3 out[4];
  int cnt = 0;
#pragma unroll
  for (int j = 0; j < 3; ++j) {
    f3 va = fv[j], vb = fv[(j + 1) % 3];
    bool ain = va.z > eps, bin = vb.z > eps;
    if (ain) {
      bool found = false;
      for (int k = 0; k < cnt; ++k)
        if (out[k].x == va.x && out[k].y == va.y && out[k].z == va.z) found = true;
      if (!found) out[cnt++] = va;
    }
    if (ain != bin) {
      float t = (eps - va.z) / (vb.z - va.z);
      out[cnt++] = lerp3(va, vb, t);
    }
  }
  if (cnt > 1)
    for (int j = 0; j < cnt; ++j) update_bounds_from_edge<FISHEYE>(out[j], out[(j + 1) % cnt], mn, mx, c);
}

// Directed edges of the faces (0,1,2) (0,2,3) (0,3,1) (1,3,2), two bits per end point.
constexpr unsigned kFrom = 0u | (1u << 2) | (2u << 4) | (0u << 6) | (2u << 8) | (3u << 10) | (0u << 12) | (3u << 14) |
                           (1u << 16) | (1u << 18) | (3u << 20) | (2u << 22);
constexpr unsigned kTo = 1u | (2u << 2) | (0u << 4) | (2u << 6) | (3u << 8) | (0u << 10) | (3u << 12) | (1u << 14) |
                         (0u << 16) | (3u << 18) | (2u << 20) | (1u << 22);
__device__ __forceinline__ f3 pick(const f3 v[4], unsigned i) { return i == 0 ? v[0] : (i == 1 ? v[1] : (i == 2 ? v[2] : v[3])); }

// Extent of a tet that lies entirely in front of the near plane, seen by an
// undistorted pinhole camera.  The general routine then clips nothing and samples
// every directed face edge a->b at its two ends, a + (b-a)*0 and a + (b-a)*1.  The
// first is the vertex a itself (up to the sign of a zero, which no later step can
// see).  The second equals b bit for bit unless the subtraction or the addition
// rounded, which happens for about one sample in forty; its projection is then
// already among the four vertex projections.  So the four vertices are projected,
// the twelve end samples are formed and compared with their vertex, and only the
// ones that differ are projected as well: the same minima and maxima as the 24
// projections of the general routine.
__device__ __forceinline__ void find_extent_unclipped(const f3 cs[4], f3& mn, f3& mx, const DevCam& c) {
  const float BIG = 1e20f;
  mn = {BIG, BIG, BIG};
  mx = {-BIG, -BIG, -BIG};
  auto add = [&](f3 p) {
    const float ux = p.x / p.z, uy = p.y / p.z;
    const float px = ux * c.K[0] + c.K[2];
    const float py = uy * c.K[4] + c.K[5];
    mn = {fminf(mn.x, px), fminf(mn.y, py), fminf(mn.z, p.z)};
    mx = {fmaxf(mx.x, px), fmaxf(mx.y, py), fmaxf(mx.z, p.z)};
  };
  add(cs[0]);
  add(cs[1]);
  add(cs[2]);
  add(cs[3]);
  unsigned pending = 0;
#pragma unroll
  for (int e = 0; e < 12; ++e) {
    const f3 a = cs[(kFrom >> (2 * e)) & 3u], b = cs[(kTo >> (2 * e)) & 3u];
    const f3 s_ = lerp3(a, b, 1.0f);
    if (s_.x != b.x || s_.y != b.y || s_.z != b.z) pending |= 1u << e;
  }
  while (pending) {
    const int e = __ffs(pending) - 1;
    pending &= pending - 1;
    add(lerp3(pick(cs, (kFrom >> (2 * e)) & 3u), pick(cs, (kTo >> (2 * e)) & 3u), 1.0f));
  }
}

// The same for a lens with distortion or a fisheye camera, which sample every edge at 3 or 4 points: the four
// vertices, the end samples that differ from their vertex, and the samples between the ends - 16 (lens) or 28
// (fisheye, most of them only estimated) projections where the general routine takes 36 or 48.  Part f of four: vertex f
// and the edges of face f.
template <bool FISHEYE>
__device__ __forceinline__ void extent_of_curved_face(const f3 cs[4], int f, f3& mn, f3& mx, const DevCam& c) {
  add_sample<FISHEYE>(pick(cs, f), mn, mx, c);
  const int n = edge_samples(c);
#pragma unroll 1
  for (int e = 3 * f; e < 3 * f + 3; ++e) {
    const f3 a = pick(cs, (kFrom >> (2 * e)) & 3u), b = pick(cs, (kTo >> (2 * e)) & 3u);
    const f3 end = lerp3(a, b, 1.0f);
    const bool differs = end.x != b.x || end.y != b.y || end.z != b.z;
#pragma unroll 1
    for (int i = 1; i < n; ++i) {
      if (i == n - 1 && !differs) break;
      add_sample<FISHEYE>(lerp3(a, b, float(i) / float(n - 1)), mn, mx, c);
    }
  }
}

__device__ __forceinline__ bool is_planar(const f3 v[4]) {
  f3 n = normalize3(cross(v[1] - v[0], v[2] - v[0]));
  float d = dot(n, v[3] - v[0]);
  return fabsf(d) < 1e-3f;
}

// ---------------------------------------------------------------------------
// Tile rectangle without the reference's arithmetic, for tets entirely in front of the near plane.  The reference's bounds
// (and with them the rectangle) are defined by the rounding of long sequences of IEEE operations: divisions, and for a
// fisheye two double series per sample.  Here the bounds are formed with approximate reciprocals and fused multiply-adds
// and widened by a bound of everything that can differ; where the floors and ceilings that decide the rectangle are the
// same at both ends, the rectangle is the reference's.  Otherwise (one tet in a thousand for a pinhole) the tet is
// deferred to the exact sequence.
// ---------------------------------------------------------------------------
struct Extent {
  float x0, x1, y0, y1;
  __device__ __forceinline__ void clear() { x0 = y0 = 3e38f; x1 = y1 = -3e38f; }
  __device__ __forceinline__ void add(float x, float y) {
    x0 = fminf(x0, x); x1 = fmaxf(x1, x);
    y0 = fminf(y0, y); y1 = fmaxf(y1, y);
  }
};

// false: undecided
__device__ __forceinline__ bool rect_of_extent(const Extent& b, float dx, float dy, const DevCam& c, int4& r) {
  const float iw = c.inv_tile_w, ih = c.inv_tile_h, gw = float(c.grid_w), gh = float(c.grid_h);
  auto clip = [](float v, float hi) { return fmaxf(0.0f, fminf(hi, v)); };
  const float x0 = floorf(clip((b.x0 - dx) * iw, gw)), y0 = floorf(clip((b.y0 - dy) * ih, gh));
  const float x1 = ceilf(clip((b.x1 + dx) * iw, gw)), y1 = ceilf(clip((b.y1 + dy) * ih, gh));
  r = make_int4(int(x0), int(y0), int(x1), int(y1));
  return x0 == floorf(clip((b.x0 + dx) * iw, gw)) && y0 == floorf(clip((b.y0 + dy) * ih, gh)) &&
         x1 == ceilf(clip((b.x1 - dx) * iw, gw)) && y1 == ceilf(clip((b.y1 - dy) * ih, gh));
}

// u = 2^-24 below; the sample at the far end of an edge, a + (b - a), is
// off b by up to 3 u times the largest coordinate.
enum CameraKind { kPinhole, kLens, kFisheye };
template <CameraKind KIND>
__device__ __forceinline__ bool estimate_rect(const f3 cs[4], const DevCam& c, int4& r) {
  const float fx = fabsf(c.K[0]), fy = fabsf(c.K[4]), cx = fabsf(c.K[2]), cy = fabsf(c.K[5]);
  const float mx = fmaxf(fmaxf(fabsf(cs[0].x), fabsf(cs[1].x)), fmaxf(fabsf(cs[2].x), fabsf(cs[3].x)));
  const float my = fmaxf(fmaxf(fabsf(cs[0].y), fabsf(cs[1].y)), fmaxf(fabsf(cs[2].y), fabsf(cs[3].y)));
  const float mz = fmaxf(fmaxf(cs[0].z, cs[1].z), fmaxf(cs[2].z, cs[3].z));
  Extent b;
  b.clear();
  float dx, dy;
  if (KIND == kLens && dist_norm2(c) == 1e-9f) return false;  // distorted, but sampled at the ends only
  if (KIND == kFisheye) {
    if (dist_norm2(c) >= 1e-9f) return false;
    // sixteen samples: the vertices and two points of each edge, whose direction the reference takes both ways
    float near = 0.0f;
    auto add = [&](f3 s) {
      const float inv = rsqrtf(fmaf(s.x, s.x, fmaf(s.y, s.y, s.z * s.z)));
      const float k = inv * fisheye_ratio_estimate(fminf(s.z * inv, 1.0f));
      near = fmaxf(near, inv);
      b.add(fmaf(s.x * k, c.K[0], c.K[2]), fmaf(s.y * k, c.K[4], c.K[5]));
    };
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      add(cs[i]);
#pragma unroll
      for (int j = 0; j < i; ++j) {
        add(cs[i] + (cs[j] - cs[i]) * (1.0f / 3.0f));
        add(cs[i] + (cs[j] - cs[i]) * (2.0f / 3.0f));
      }
    }
    // the ratio to 2e-6 of a half circle; the samples' rounding, seen from the nearest one
    const float m = 1e-6f * (mx + my + mz) * near;
    dx = fmaf(fx, 4e-6f + m, fmaf(1e-6f, cx, 2e-4f));
    dy = fmaf(fy, 4e-6f + m, fmaf(1e-6f, cy, 2e-4f));
  } else {
    float ax = 0.0f, ay = 0.0f, rz = 0.0f;
    auto add = [&](f3 s) {
      const float iz = fast_rcp(s.z);
      float x = s.x * iz, y = s.y * iz;
      ax = fmaxf(ax, fabsf(x));
      ay = fmaxf(ay, fabsf(y));
      rz = fmaxf(rz, iz);
      if (KIND == kLens) distort(x, y, c);
      b.add(fmaf(x, c.K[0], c.K[2]), fmaf(y, c.K[4], c.K[5]));
    };
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      add(cs[i]);
      if (KIND == kLens) {  // and the middle of every edge
#pragma unroll
        for (int j = 0; j < i; ++j) add(cs[i] + (cs[j] - cs[i]) * 0.5f);
      }
    }
    if (KIND == kPinhole) {
      // quotients and affine map: 7 u fx |x|, 6 u |cx|; samples off the vertices: 3 u fx (mx + |x| mz) / min z
      dx = 8e-8f * fmaf(fx, fmaf(13.0f, ax, 3.3f * fmaf(ax, mz, mx) * rz), 6.0f * cx);
      dy = 8e-8f * fmaf(fy, fmaf(13.0f, ay, 3.3f * fmaf(ay, mz, my) * rz), 6.0f * cy);
    } else {
      // the same relative to the largest coordinate, through the polynomial: its terms bound it and, five-fold, its
      // derivative's
      const float m = fmaxf(fmaxf(ax, ay), fmaxf(mx, my) * rz), m2 = 2.0f * m * m;
      const float terms = fmaf(m, fmaf(m2, fabsf(c.dist[0]) + fabsf(c.dist[1]) * m2, 1.0f), 3.0f * m2 * (fabsf(c.dist[2]) + fabsf(c.dist[3])));
      const float d = 4e-7f * terms * fmaf(3.3f * mz, rz, 24.0f);
      dx = fmaf(fx, d, 5e-7f * cx);
      dy = fmaf(fy, d, 5e-7f * cy);
    }
  }
  // four coinciding vertices have no edge to sample: the exact routine then leaves the bounds empty
  if (b.x0 == b.x1 && b.y0 == b.y1) return false;
  return rect_of_extent(b, dx, dy, c, r);
}

// is_planar from an estimate of the distance where that is not within rounding of the threshold
__device__ __forceinline__ bool is_planar_filtered(const f3 v[4]) {
  const f3 n = cross(v[1] - v[0], v[2] - v[0]), e = v[3] - v[0];
  const float nn = fmaf(n.x, n.x, fmaf(n.y, n.y, n.z * n.z));
  const float d = fabsf(fmaf(n.x, e.x, fmaf(n.y, e.y, n.z * e.z))) * rsqrtf(nn);
  const float margin = 2e-6f * (fabsf(e.x) + fabsf(e.y) + fabsf(e.z));
  if (nn > 1e-30f && nn < 1e30f) {
    if (d > 1e-3f + margin) return false;
    if (d < 1e-3f - margin) return true;
  }
  return is_planar(v);
}

// The three quotients of a vector by one double, rounded as the divisions round: quotient from the correctly rounded
// reciprocal, corrected twice with the exact remainder (Markstein, "Computation of elementary functions on the IBM RISC
// System/6000 processor", 1990); outside the range where the remainders are exact, the divisions.
__device__ __forceinline__ d3 divide3(d3 a, double d) {
  auto fits = [](double v) { const double m = fabs(v); return m > 1e-120 && m < 1e120; };
  if (!(fits(a.x) && fits(a.y) && fits(a.z) && fits(d))) return {a.x / d, a.y / d, a.z / d};
  const double r = 1.0 / d;
  auto quotient = [&](double x) {
    double q = x * r;
    q = fma(fma(-q, d, x), r, q);
    return fma(fma(-q, d, x), r, q);
  };
  return {quotient(a.x), quotient(a.y), quotient(a.z)};
}

__device__ __forceinline__ double length3(d3 a) { return sqrt(dot(a, a)); }

// branch: 0 regular, 1 tiny tet (centroid rule), 2 degenerate (-1e20)
__device__ __forceinline__ double power_of_circumsphere(d3 A, d3 B, d3 C, d3 D, d3 P, d3& center, int& branch) {
  d3 a = B - A, b = C - A, c = D - A;
  double aa = dot(a, a), bb = dot(b, b), cc = dot(c, c);
  d3 cbc = cross(b, c), cca = cross(c, a), cab = cross(a, b);
  double denominator = 2.0 * dot(a, cbc);
  double radius;
  if (fabs(denominator) < 1e-10) {
    double m = fmax(length3(B - A),
                    fmax(length3(C - A), fmax(length3(D - A), fmax(length3(C - B), fmax(length3(D - B), length3(D - C))))));
    if (m < 1e-7) {
      center = (A + B + C + D) * 0.25;
      double dA = length3(A - center), dB = length3(B - center), dC = length3(C - center), dD = length3(D - center);
      radius = fmin(dA, fmin(dB, fmin(dC, dD)));
      d3 diff = center - P;
      branch = 1;
      return dot(diff, diff) - radius * radius;
    }
    branch = 2;
    return -1e20;
  }
  d3 num = cbc * aa + cca * bb + cab * cc;
  d3 rel = divide3(num, denominator);
  center = A + rel;
  radius = length3(rel);
  d3 diff = center - P;
  branch = 0;
  return dot(diff, diff) - radius * radius;
}

__device__ __forceinline__ float clipf(float v, float lo, float hi) { return fmaxf(lo, fminf(hi, v)); }

// What is left of a tet once its rectangle over the whole frame is known: band, planar test, sort depth, circumcentre.
// Returns the number of tiles, 0 if it is culled.
struct Projected {
  int4 r;
  float depth;
  f3 cc;
};
__device__ __forceinline__ int finish_tet(const f3 v[4], int4 r, const DevCam& cam, Projected& out) {
  out = {make_int4(0, 0, 0, 0), 0.0f, {0.0f, 0.0f, 0.0f}};
  // band restriction (whole frame: row0 = 0, row1 = grid_h)
  r.y = max(r.y, cam.row0);
  r.w = min(r.w, cam.row1);
  if (r.w < r.y) r.w = r.y;
  const int nt = (r.z - r.x) * (r.w - r.y);
  if (nt == 0 || is_planar_filtered(v)) return 0;
  d3 A = {v[0].x, v[0].y, v[0].z}, B = {v[1].x, v[1].y, v[1].z}, C = {v[2].x, v[2].y, v[2].z},
     D = {v[3].x, v[3].y, v[3].z}, P = {cam.pos[0], cam.pos[1], cam.pos[2]};
  d3 cc = {0, 0, 0};
  int branch;
  const float sort_depth = float(power_of_circumsphere(A, B, C, D, P, cc, branch));
  if (sort_depth < -1e19f) return 0;
  out = {r, fminf(fmaxf(sort_depth, -1e20f), 1e20f), {float(cc.x), float(cc.y), float(cc.z)}};
  return nt;
}

// Where the projection leaves its results; the two kernels below share it.
//   depth_keys[g]  sortable depth bits, 0xFFFFFFFF for culled tets
//   tile_diff      2-D difference array of tile coverage ((gh+1) x (gw+1) int32), diff_copies of them
struct ProjectOut {
  int32_t* tiles_touched;
  int4* rect;
  float *vs_tetra, *circumcenter;
  uint32_t* depth_keys;
  uint8_t* visible;
  int32_t* tile_diff;
  int diff_copies;
  uint32_t* counters;  // visible tets, status bits, deferred tets
  uint32_t* deferred;  // their ids
};
__device__ __forceinline__ void store_tet(const ProjectOut& o, int64_t g, int nt, const Projected& p) {
  o.tiles_touched[g] = nt;
  if (o.visible) o.visible[g] = nt > 0;
  o.rect[g] = p.r;
  o.depth_keys[g] = nt > 0 ? float2sortable_key(p.depth) : 0xFFFFFFFFu;
}
// A small grid comes in several partial arrays (a power of two), so that fewer atomics meet on one address.
__device__ __forceinline__ int32_t* coverage_array(const ProjectOut& o, const DevCam& cam) {
  return o.tile_diff + (blockIdx.x & (o.diff_copies - 1)) * ((cam.grid_w + 1) * (cam.grid_h + 1));
}
// What a rectangle adds to the difference array, at each of its corners.
template <typename F>
__device__ __forceinline__ void for_corners(int4 r, F add) {
  add(r.x, r.y, 1);
  add(r.z, r.y, -1);
  add(r.x, r.w, -1);
  add(r.z, r.w, 1);
}

// The corners of a warp's rectangles, by all lanes of it (on: this lane has one).  The tets of a mesh come in runs of
// neighbours, so that most corners of a warp lie in a few tiles and many on the same: they are added up in a window of
// 16 x 16 cells in shared memory (zero), which leaves as one atomic per cell that is not zero, lanes side by side.  Four
// atomics per tet kept L2 busy for a third of the kernel: 6M tets, 1080p 320 -> 241 us, 21M 1380 -> 785 us, 36M, 2160p
// 2250 -> 1334 us; 2M, where more than half are culled: 70 -> 74 us, and half of a scene of 0.6M 30 -> 32.  In random order the
// corners miss the window: 2M 106.5 -> 109 us, 6.7M 464 -> 465, 21M 1827 -> 1829.
constexpr int kWindow = 16;
__device__ __forceinline__ void add_coverage(const ProjectOut& o, const DevCam& cam, bool on, int4 r, int32_t* window) {
  if (!__any_sync(0xffffffffu, on)) return;
  const int x0 = __reduce_min_sync(0xffffffffu, on ? r.x : INT_MAX), y0 = __reduce_min_sync(0xffffffffu, on ? r.y : INT_MAX);
  const int pitch = cam.grid_w + 1, lane = threadIdx.x & 31;
  int32_t* diff = coverage_array(o, cam);
  if (on) {
    for_corners(r, [&](int x, int y, int v) {
      if (x - x0 < kWindow && y - y0 < kWindow) atomicAdd(&window[(y - y0) * kWindow + x - x0], v);
      else atomicAdd(&diff[y * pitch + x], v);
    });
  }
  __syncwarp();
  int32_t* at = diff + (y0 + lane / kWindow) * pitch + x0 + lane % kWindow;
#pragma unroll
  for (int i = 0; i < kWindow * kWindow; i += 32, at += 32 / kWindow * pitch) {
    const int32_t v = window[i + lane];
    if (v) atomicAdd(at, v);
  }
}

// One thread per tet (and, for the NaN scan, per vertex coordinate).  Bound by instruction issue (6M tets: 70 % of the
// slots; no block barriers, or persistent warps that fetch vertices ahead, are no faster).  The camera sits in shared memory
// (32 loads per thread from global before), a warp's depths and circumcentres leave through shared memory as 16-byte stores,
// and the reference's exact arithmetic is left to k_project_deferred, for the tets whose rectangle an estimate does not
// decide: a few lanes of a warp would hold up the rest for thousands of instructions.  With the exact sequence for every tet
// 6M tets, 1080p took 369 us, with the deferral 290 (238 now, see add_coverage); 1M through a fisheye 436 us with the
// deferred tets done in place, 81 with the deferral (59 now).
constexpr int kProjectThreads = 128;

template <bool FISHEYE>
__global__ void __launch_bounds__(kProjectThreads, 8)
k_project(const int32_t* __restrict__ indices, int64_t T, const float* __restrict__ vertices, int64_t V, RmCamera rcam,
          ProjectOut o) {
  after_previous();
  __shared__ DevCam cam;
  __shared__ __align__(16) float rows[kProjectThreads / 32][2][96];
  __shared__ __align__(16) int32_t windows[kProjectThreads / 32][kWindow * kWindow];
  const int64_t g = (int64_t)blockIdx.x * kProjectThreads + threadIdx.x;
  const int lane = threadIdx.x & 31;
  load_cam_shared(rcam, cam);
  int32_t* window = windows[threadIdx.x >> 5];
#pragma unroll
  for (int i = 0; i < kWindow * kWindow; i += 128) *reinterpret_cast<int4*>(window + i + 4 * lane) = make_int4(0, 0, 0, 0);
  if (g < 3 * V) {
    float v = __ldg(vertices + g);
    if (v != v) atomicOr(o.counters + 1, RM_STATUS_NAN_VERTEX);
  }
  int4 id = make_int4(0, 0, 0, 0);
  bool ids_ok = false;
  if (g < T) {
    id = __ldg(reinterpret_cast<const int4*>(indices) + g);
    // A vertex id outside [0, V) would read out of bounds here and in every later stage: the tet is
    // culled (later stages skip culled tets) and the host is told through the status word.
    ids_ok = (uint32_t)id.x < (uint64_t)V && (uint32_t)id.y < (uint64_t)V && (uint32_t)id.z < (uint64_t)V &&
             (uint32_t)id.w < (uint64_t)V;
    if (!ids_ok) atomicOr(o.counters + 1, RM_STATUS_BAD_INDEX);
  }
  f3 v[4] = {{0.f, 0.f, 0.f}, {0.f, 0.f, 0.f}, {0.f, 0.f, 0.f}, {0.f, 0.f, 0.f}};
  if (ids_ok) {
    v[0] = load3(vertices, id.x);
    v[1] = load3(vertices, id.y);
    v[2] = load3(vertices, id.z);
    v[3] = load3(vertices, id.w);
  }
  __syncthreads();  // the camera is there
  const bool lens = !FISHEYE && dist_norm2(cam) >= 1e-9f;

  int nt = 0;
  Projected p = {make_int4(0, 0, 0, 0), 0.0f, {0.0f, 0.0f, 0.0f}};
  bool defer = false;
  if (ids_ok) {
    f3 cs[4];
#pragma unroll
    for (int k = 0; k < 4; ++k) cs[k] = point2camspace(v[k], cam);
    const float eps = 1e-4f;
    const bool f0 = cs[0].z > eps, f1 = cs[1].z > eps, f2 = cs[2].z > eps, f3_ = cs[3].z > eps;
    // with no vertex in front of the near plane nothing is left of the faces: the extent is empty
    bool seen = f0 || f1 || f2 || f3_;
    const bool front = f0 && f1 && f2 && f3_;
    if (!FISHEYE && !lens && front && (cam.row0 > 0 || cam.row1 < cam.grid_h)) {
      // Band pre-test: a tet whose four projected vertices all lie more than a pixel above the band's
      // first pixel row, or more than a pixel below its last, ends with an empty rectangle after the
      // clamp to the band; it is culled here.  The comparison
      // py < y is made without the division (Z > 0): fy*Y + (cy - y)*Z < 0; its rounding error is far
      // below the one-pixel margin wherever py is near y.
      const float c_lo = cam.K[5] - (float(cam.row0 * cam.tile_h) - 1.0f);
      const float c_hi = cam.K[5] - (float(cam.row1 * cam.tile_h) + 1.0f);
      bool above = true, below = true;
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        const float a = cam.K[4] * cs[k].y;
        above = above && (a + c_lo * cs[k].z < 0.0f);
        below = below && (a + c_hi * cs[k].z > 0.0f);
      }
      seen = !(above || below);
    }
    if (seen) {
      int4 r = make_int4(0, 0, 0, 0);
      bool known = false;
      if (front) {
        if (FISHEYE) known = estimate_rect<kFisheye>(cs, cam, r);
        else if (lens) known = estimate_rect<kLens>(cs, cam, r);
        else known = estimate_rect<kPinhole>(cs, cam, r);
      }
      defer = !known;
      if (known) nt = finish_tet(v, r, cam, p);
    }
  }
  if (g < T) store_tet(o, g, nt, p);
  add_coverage(o, cam, nt > 0, p.r, window);
  {
    const unsigned m = __ballot_sync(0xffffffffu, defer);
    if (m) {
      uint32_t at = 0;
      if (lane == 0) at = atomicAdd(o.counters + 2, (uint32_t)__popc(m));
      at = __shfl_sync(0xffffffffu, at, 0) + __popc(m & ((1u << lane) - 1u));
      if (defer) o.deferred[at] = (uint32_t)g;
    }
  }
  const int64_t g0 = g - lane;
  if (g0 + 32 <= T && ((reinterpret_cast<uintptr_t>(o.vs_tetra) | reinterpret_cast<uintptr_t>(o.circumcenter)) & 15) == 0) {
    float* vs_row = rows[threadIdx.x >> 5][0];
    float* cc_row = rows[threadIdx.x >> 5][1];
    vs_row[3 * lane] = 0.0f;
    vs_row[3 * lane + 1] = 0.0f;
    vs_row[3 * lane + 2] = p.depth;
    cc_row[3 * lane] = p.cc.x;
    cc_row[3 * lane + 1] = p.cc.y;
    cc_row[3 * lane + 2] = p.cc.z;
    __syncwarp();
    if (lane < 24) {
      reinterpret_cast<float4*>(o.vs_tetra + 3 * g0)[lane] = reinterpret_cast<const float4*>(vs_row)[lane];
      reinterpret_cast<float4*>(o.circumcenter + 3 * g0)[lane] = reinterpret_cast<const float4*>(cc_row)[lane];
    }
  } else if (g < T) {
    o.vs_tetra[3 * g + 0] = 0.0f;
    o.vs_tetra[3 * g + 1] = 0.0f;
    o.vs_tetra[3 * g + 2] = p.depth;
    o.circumcenter[3 * g + 0] = p.cc.x;
    o.circumcenter[3 * g + 1] = p.cc.y;
    o.circumcenter[3 * g + 2] = p.cc.z;
  }
  // visible-tet count, one atomic per block: one per warp queued on the one address
  const int n_visible = __syncthreads_count(nt > 0);
  if (threadIdx.x == 0 && n_visible) atomicAdd(o.counters, (uint32_t)n_visible);
}

// The tets whose rectangle the estimate left open, with the reference's arithmetic.  k_project stored them as culled.
// Four lanes per tet, one per face: bound by the length of the sequence, not by its throughput (6M tets, 1080p: 6 thousand
// tets in 27 us with a lane each).
template <bool FISHEYE>
__global__ void __launch_bounds__(kProjectThreads)
k_project_deferred(const int32_t* __restrict__ indices, const float* __restrict__ vertices, RmCamera rcam, ProjectOut o) {
  after_previous();
  __shared__ DevCam cam;
  load_cam_shared(rcam, cam);
  __syncthreads();
  const bool lens = !FISHEYE && dist_norm2(cam) >= 1e-9f;
  const uint32_t n = o.counters[2];
  const int face = threadIdx.x & 3;
  constexpr uint32_t kPerBlock = kProjectThreads / 4;
  for (uint32_t first = blockIdx.x * kPerBlock; first < n; first += gridDim.x * kPerBlock) {
    const uint32_t i = first + threadIdx.x / 4;
    const bool live = i < n;
    const uint32_t g = live ? o.deferred[i] : 0u;
    const int4 id = live ? __ldg(reinterpret_cast<const int4*>(indices) + g) : make_int4(0, 0, 0, 0);
    const f3 v[4] = {load3(vertices, id.x), load3(vertices, id.y), load3(vertices, id.z), load3(vertices, id.w)};
    f3 cs[4];
#pragma unroll
    for (int k = 0; k < 4; ++k) cs[k] = point2camspace(v[k], cam);
    const bool front = cs[0].z > 1e-4f && cs[1].z > 1e-4f && cs[2].z > 1e-4f && cs[3].z > 1e-4f;
    const bool point = cs[0].x == cs[1].x && cs[0].x == cs[2].x && cs[0].x == cs[3].x && cs[0].y == cs[1].y &&
                       cs[0].y == cs[2].y && cs[0].y == cs[3].y && cs[0].z == cs[1].z && cs[0].z == cs[2].z &&
                       cs[0].z == cs[3].z;
    const float BIG = 1e20f;
    f3 mn = {BIG, BIG, BIG}, mx = {-BIG, -BIG, -BIG};
    if (live) {
      if (!FISHEYE && !lens && front) find_extent_unclipped(cs, mn, mx, cam);
      else if (front && !point) extent_of_curved_face<FISHEYE>(cs, face, mn, mx, cam);
      else extent_of_face<FISHEYE>(cs, face, mn, mx, cam);
    }
#pragma unroll
    for (int s = 1; s <= 2; s <<= 1) {
      mn = {fminf(mn.x, __shfl_xor_sync(0xffffffffu, mn.x, s)), fminf(mn.y, __shfl_xor_sync(0xffffffffu, mn.y, s)), mn.z};
      mx = {fmaxf(mx.x, __shfl_xor_sync(0xffffffffu, mx.x, s)), fmaxf(mx.y, __shfl_xor_sync(0xffffffffu, mx.y, s)),
            fmaxf(mx.z, __shfl_xor_sync(0xffffffffu, mx.z, s))};
    }
    if (!live || face != 0 || mx.z <= 0.0f) continue;
    const int4 r = make_int4(int(floorf(clipf(mn.x / float(cam.tile_w), 0.f, float(cam.grid_w)))),
                             int(floorf(clipf(mn.y / float(cam.tile_h), 0.f, float(cam.grid_h)))),
                             int(ceilf(clipf(mx.x / float(cam.tile_w), 0.f, float(cam.grid_w)))),
                             int(ceilf(clipf(mx.y / float(cam.tile_h), 0.f, float(cam.grid_h)))));
    Projected p;
    const int nt = finish_tet(v, r, cam, p);
    if (nt == 0) continue;
    store_tet(o, g, nt, p);
    int32_t* diff = coverage_array(o, cam);
    for_corners(p.r, [&](int x, int y, int v) { atomicAdd(&diff[y * (cam.grid_w + 1) + x], v); });
    o.vs_tetra[3 * (int64_t)g + 2] = p.depth;
    o.circumcenter[3 * (int64_t)g + 0] = p.cc.x;
    o.circumcenter[3 * (int64_t)g + 1] = p.cc.y;
    o.circumcenter[3 * (int64_t)g + 2] = p.cc.z;
    atomicAdd(o.counters, 1u);
  }
}

// Reverse of the sort-depth / circumcentre computation with respect to the
// four vertices, in fp64, accumulated into vertices_grad with fp32 atomics.
__global__ void __launch_bounds__(256)
k_vertex_backward(const int32_t* __restrict__ indices, const float* __restrict__ vertices, int64_t T, RmCamera rcam,
                  const int32_t* __restrict__ tiles_touched, const float* __restrict__ g_vs,
                  const float* __restrict__ g_cc, float* __restrict__ vgrad) {
  int64_t g = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (g >= T) return;
  if (tiles_touched[g] == 0) return;
  float gp_in = __ldg(g_vs + 3 * g + 2);
  float gc0 = __ldg(g_cc + 3 * g), gc1 = __ldg(g_cc + 3 * g + 1), gc2 = __ldg(g_cc + 3 * g + 2);
  if (gp_in == 0.0f && gc0 == 0.0f && gc1 == 0.0f && gc2 == 0.0f) return;
  int4 id = __ldg(reinterpret_cast<const int4*>(indices) + g);
  int vid[4] = {id.x, id.y, id.z, id.w};
  d3 p[4];
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    f3 v = load3(vertices, vid[k]);
    p[k] = {v.x, v.y, v.z};
  }
  d3 P = {__ldg(rcam.cam_pos), __ldg(rcam.cam_pos + 1), __ldg(rcam.cam_pos + 2)};
  d3 center = {0, 0, 0};
  int branch;
  double power = power_of_circumsphere(p[0], p[1], p[2], p[3], P, center, branch);
  float sd = float(power);
  double g_power = (sd > -1e20f && sd < 1e20f) ? double(gp_in) : 0.0;
  d3 g_center = {gc0, gc1, gc2};
  d3 gp[4] = {{0, 0, 0}, {0, 0, 0}, {0, 0, 0}, {0, 0, 0}};
  if (branch == 0) {
    d3 a = p[1] - p[0], b = p[2] - p[0], c = p[3] - p[0];
    double aa = dot(a, a), bb = dot(b, b), cc = dot(c, c);
    d3 X = cross(b, c), Y = cross(c, a), Z = cross(a, b);
    double den = 2.0 * dot(a, X);
    d3 num = X * aa + Y * bb + Z * cc;
    d3 rel = {num.x / den, num.y / den, num.z / den};
    d3 diff = center - P;
    d3 g_ct = g_center + diff * (2.0 * g_power);
    d3 g_rel = g_ct - rel * (2.0 * g_power);
    d3 g_num = {g_rel.x / den, g_rel.y / den, g_rel.z / den};
    double g_den = -dot(g_rel, rel) / den;
    double g_aa = dot(g_num, X), g_bb = dot(g_num, Y), g_cc2 = dot(g_num, Z);
    d3 g_X = g_num * aa + a * (2.0 * g_den);
    d3 g_Y = g_num * bb, g_Z = g_num * cc;
    d3 g_a = X * (2.0 * g_den) + a * (2.0 * g_aa);
    d3 g_b = b * (2.0 * g_bb);
    d3 g_c = c * (2.0 * g_cc2);
    g_b = g_b + cross(c, g_X);  g_c = g_c + cross(g_X, b);
    g_c = g_c + cross(a, g_Y);  g_a = g_a + cross(g_Y, c);
    g_a = g_a + cross(b, g_Z);  g_b = g_b + cross(g_Z, a);
    gp[1] = g_a; gp[2] = g_b; gp[3] = g_c;
    gp[0] = g_ct - g_a - g_b - g_c;
  } else if (branch == 1) {
    d3 diff = center - P;
    d3 g_ct = g_center + diff * (2.0 * g_power);
    int arg = 0;
    double best = length3(p[0] - center);
#pragma unroll
    for (int k = 1; k < 4; ++k) {
      double dk = length3(p[k] - center);
      if (dk < best) { best = dk; arg = k; }
    }
    d3 g_rv = (p[arg] - center) * (-2.0 * g_power);
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      if (k == arg) gp[k] = gp[k] + g_rv;
    }
    g_ct = g_ct - g_rv;
#pragma unroll
    for (int k = 0; k < 4; ++k) gp[k] = gp[k] + g_ct * 0.25;
  }
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    atomicAdd(vgrad + 3 * (int64_t)vid[k] + 0, float(gp[k].x));
    atomicAdd(vgrad + 3 * (int64_t)vid[k] + 1, float(gp[k].y));
    atomicAdd(vgrad + 3 * (int64_t)vid[k] + 2, float(gp[k].z));
  }
}

}  // namespace rm

// ---------------------------------------------------------------------------
// host-side launchers used by rm_api.cu
// ---------------------------------------------------------------------------
int rm_launch_project(const int32_t* indices, int64_t T, const float* vertices, int64_t V, const RmCamera* cam,
                      int32_t* tiles_touched, int32_t* rect, float* vs_tetra, float* circumcenter, uint32_t* depth_keys,
                      int32_t* tile_diff, int diff_copies, uint32_t* counters, uint32_t* deferred, uint8_t* visible,
                      cudaStream_t st) {
  int64_t n = T > 3 * V ? T : 3 * V;
  if (n == 0) return RM_OK;
  const int64_t blocks = (n + rm::kProjectThreads - 1) / rm::kProjectThreads;
  const rm::ProjectOut o = {tiles_touched, reinterpret_cast<int4*>(rect), vs_tetra, circumcenter, depth_keys, visible,
                            tile_diff,     diff_copies,                   counters, deferred};
  const bool fisheye = cam->camera_type == 1;
  {
    RmProfScope prof("k_project", st);
    auto kernel = fisheye ? rm::k_project<true> : rm::k_project<false>;
    RM_CUDA_CHECK(rm_launch(kernel, (unsigned)blocks, rm::kProjectThreads, 0, st, indices, T, vertices, V, *cam, o));
  }
  {
    RmProfScope prof("k_project_deferred", st);
    auto kernel = fisheye ? rm::k_project_deferred<true> : rm::k_project_deferred<false>;
    // How many tets are deferred only the device knows; a block takes 32 of them at a time, one time after the other.  Sixteen
    // blocks for an SM: 1M tets, fisheye, 57.6 us with four, 45.4 with sixteen; 36M, 2160p, 72.0, 59.7; 6.7M 25.0, 20.9; sixty-four
    // cost 4 us where nothing is deferred.  (Sixteen lanes per tet instead of four: fisheye 43.8, but 36M 121.)
    RM_CUDA_CHECK(rm_launch_behind(T, kernel, (unsigned)(blocks < 16 * 148 ? blocks : 16 * 148), rm::kProjectThreads, 0, st, indices,
                                   vertices, *cam, o));
  }
  return RM_OK;
}

int rm_launch_vertex_backward(const int32_t* indices, const float* vertices, int64_t T, const RmCamera* cam,
                              const int32_t* tiles_touched, const float* g_vs, const float* g_cc, float* vgrad,
                              cudaStream_t st) {
  if (T == 0) return RM_OK;
  unsigned blocks = (unsigned)((T + 255) / 256);
  RmProfScope prof("k_vertex_backward", st);
  RM_CUDA_CHECK(rm_launch(rm::k_vertex_backward, blocks, 256, 0, st, indices, vertices, T, *cam, tiles_touched, g_vs, g_cc,
                          vgrad));
  return RM_OK;
}
